"""Graph launches beside the uploads and other graphs of the same device."""
from __future__ import annotations

import numpy as np
import pytest

import irisb200
import workload as W

pytestmark = pytest.mark.gpu


def _engine(dm, peer, n_db, n_q, K=6400):
    e = irisb200.ShareDB(peer, dm, n_db, n_q * 32, K, W.SEEDS[peer])
    e.alloc_db(n_db)
    e.fill_random(peer + 1, n_db)
    return e


def test_uploads_wait_for_every_graph(dm):
    """Two graphs over two engines on two streams: an upload to the engine of
    the first, long one waits for it, not only for the graph launched last."""
    K, n_q, n_db = 6400, 20, 16384
    rng = np.random.default_rng(2)
    long, short = _engine(dm, 0, n_db, n_q), _engine(dm, 1, 64, n_q)
    slots = [(j, 0, 31, j) for j in range(n_q)]
    rows = [rng.integers(0, 1 << 16, (n_q, K), dtype=np.uint16) for _ in range(2)]
    for e in (long, short):
        e.query_upload_slots(rows[0], slots)
    long.dot(0, n_db, 1)
    want = long.fetch_results(n_db)
    dm.synchronize()

    def many():
        for _ in range(40):
            long.dot(0, n_db, 1, dm.stream(0))
    graphs = [irisb200.Graph.capture(dm, many), irisb200.Graph.capture(dm, lambda: short.dot(0, 64, 1, dm.stream(0)))]
    for _ in range(3):
        graphs[0].launch(dm.stream(2))
        graphs[1].launch(dm.stream(1))
        long.query_upload_slots(rows[1], slots)
        dm.synchronize()
        assert np.array_equal(long.fetch_results(n_db), want)
        long.query_upload_slots(rows[0], slots)
    for g in graphs:
        g.close()
    long.close()
    short.close()


def test_graph_launch_beside_an_open_capture(dm):
    """A graph launched on a stream of its own while another one is being
    captured runs, stays out of the capture, and reads the rows uploaded before."""
    K, n_q, n_db = 6400, 20, 4096
    rng = np.random.default_rng(3)
    a, b = _engine(dm, 0, n_db, n_q), _engine(dm, 1, n_db, n_q)
    rows = rng.integers(0, 1 << 16, (n_q, K), dtype=np.uint16)
    slots = [(j, 0, 31, j) for j in range(n_q)]
    want = {}
    for e in (a, b):
        e.query_upload_slots(rows, slots)
        e.dot(0, n_db, 1)
        want[e] = e.fetch_results(n_db)
    first = irisb200.Graph.capture(dm, lambda: a.dot(0, n_db, 1, dm.stream(0)))
    a.query_upload_slots(rows[::-1].copy(), slots)
    a.query_upload_slots(rows, slots)  # in flight when the capture below begins

    def body():
        first.launch(dm.stream(1))
        b.dot(0, n_db, 1, dm.stream(0))
    second = irisb200.Graph.capture(dm, body)
    dm.synchronize()
    assert np.array_equal(a.fetch_results(n_db), want[a])
    second.launch(dm.stream(0))
    dm.synchronize()
    assert np.array_equal(b.fetch_results(n_db), want[b])
    for g in (first, second):
        g.close()
    a.close()
    b.close()
