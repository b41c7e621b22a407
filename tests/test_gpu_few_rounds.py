"""Launches of few rounds of tiles: 64- and 128-row one-SM tiles on engines whose
own tile is wider, and SM pairs where they fill the rounds as well.  Whatever
runs, the dot shares equal the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import irisb200
import workload as W

pytestmark = pytest.mark.gpu


# engines, rows, entries: one round of 64-row tiles (the last one past the rows),
# its edge, one round of 128-row ones, its edge (148 tiles), pairs in one round,
# two rounds of 128-row tiles against two of pairs; rows that 128 or 256 do not divide
@pytest.mark.parametrize("n,rows,entries,gemm", [
    (1, 1984, 300, "one_sm"), (1, 2048, 512, "one_sm"), (1, 1408, 1461, "one_sm"), (1, 512, 4736, "one_sm"),
    (1, 512, 4737, "pair"), (2, 1216, 900, "pair"), (1, 1536, 1900, "pair"), (1, 1792, 3100, "one_sm"),
    (2, 640, 1900, "pair"), (1, 896, 3968, "pair"), (1, 832, 40, "one_sm")])
@pytest.mark.parametrize("tile", [0, 128])
def test_few_rounds(dm, oracle, n, rows, entries, gemm, tile):
    K = 12800
    rng = np.random.default_rng(rows + entries)
    q = rng.integers(0, 1 << 16, (rows, K), dtype=np.uint16)
    engines = [irisb200.ShareDB(p, dm, entries, rows, K, W.SEEDS[p], is_remote=False) for p in range(n)]
    for p, e in enumerate(engines):
        e.alloc_db(entries)
        e.fill_random(p, entries)
        e.query_upload(q)
        e.set_tile(tile)
    pad = engines[0].result_view()[1]
    irisb200.dot_many(engines, [1] * n, 0, entries)
    dm.synchronize()
    ran = engines[0].last_gemm()[0]
    assert ran == ("one_sm" if tile and pad % tile == 0 else gemm)
    at = sorted({0, entries // 2, entries - 1})
    for e in engines:
        got = e.fetch_results(entries)
        rec = np.concatenate([e.fetch_records(i, 1) for i in at])
        assert np.array_equal(got[:, at], oracle.dot_u16(q, rec))
        e.set_tile(64)
        e.dot(0, entries, 1)
        assert e.last_gemm()[0] == "one_sm" and np.array_equal(e.fetch_results(entries), got)
        e.close()
