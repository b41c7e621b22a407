"""The tuners at row counts that no 256-row tile divides reach the two-SM GEMMs,
and so the rotation-structured one where the library runs it untuned."""
from __future__ import annotations

import numpy as np
import pytest

import irisb200
import workload as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_q", [3, 20, 28])
def test_plain_scan_tunes_over_the_two_sm_gemms(dm, n_q):
    from irisb200.scan import PlainScan
    M = 16384
    ce = [irisb200.ShareDB(p, dm, M, 1024, 12800, W.SEEDS[p]) for p in range(3)]
    me = [irisb200.ShareDB(p, dm, M, 1024, 6400, W.SEEDS[p]) for p in range(3)]
    for e in ce + me:
        e.alloc_db(M)
    irisb200.synth_db(ce, me, 5, 0, M)
    c, dc = irisb200.Circuits(dm, W.SEEDS), irisb200.DistanceComparator(dm, n_q, M)
    qc, qm = irisb200.synth_queries(5, 6, n_q, {1: (77, 3)})
    slots = [(j, 0, 31, j) for j in range(n_q)]
    for p in range(3):
        ce[p].query_upload_slots(qc[p], slots)
        me[p].query_upload_slots(qm[p], slots)
    ps = PlainScan(dm, ce, me, c, dc, n_q, M, 16384)

    def bitmap():
        dc.reset()
        ps.scan()
        dm.synchronize()
        return dc.fetch_bitmap(n_q, M)
    want, untuned = bitmap(), ce[0].last_gemm()[0]
    assert untuned == ("quad" if n_q >= 18 else "pair")
    best = ps.tune(passes=1, finalists=2, rounds=1)
    n = len(ps.candidates())
    added = [cd for cd, _ in ps.tune_log[n:-2]]
    assert added == [("pair", 256, 16384), ("pair", 256, 8192), ("split", 0, 16384)]
    assert len(ps.tune_log) == n + 3 + 2 and best in ps.candidates() + added
    for cand in added:
        ps.configure(cand)
        assert np.array_equal(bitmap(), want) and (n_q < 18 or ce[0].last_gemm()[0] == "quad")
    assert ("pair", 256, 8192) not in ps.candidates()
    with pytest.raises(irisb200.IrisError):
        ps.tune(only_path="pair")  # not in the list, as before
    ps.restore()
    ps.close()
    for x in [dc, c] + ce + me:
        x.close()


def test_batched_engine_tunes_over_the_two_sm_gemms(dm):
    from irisb200.batched import BatchedEngine, Request
    M, n = 16384, 18
    ce = [irisb200.ShareDB(p, dm, M, 1024, 12800, W.SEEDS[p]) for p in range(3)]
    me = [irisb200.ShareDB(p, dm, M, 1024, 6400, W.SEEDS[p]) for p in range(3)]
    for e in ce + me:
        e.alloc_db(M)
    irisb200.synth_db(ce, me, 5, 0, M)
    qc, qm = irisb200.synth_queries(5, 6, n, {j: (100 * j, j - 8) for j in range(0, n, 4)})
    reqs = [Request(code=np.ascontiguousarray(qc[:, j]), mask=np.ascontiguousarray(qm[:, j]), n_rot=31) for j in range(n)]
    eng = BatchedEngine(dm, ce, me, irisb200.Circuits(dm, W.SEEDS), max_variants=32, max_reauth=4, seeds=W.SEEDS)
    first = eng.run(reqs)
    assert [r.matches for r in eng.run(reqs)] == [r.matches for r in first]
    assert all(100 * j in first[j].matches for j in range(0, n, 4))
    assert any(cd[0] == "pair" for cd, _ in eng.tune_log[640]) and not any(
        cd[0] == "pair" for cd in BatchedEngine._candidates(640, M))
    eng.close()
    for e in ce + me:
        e.close()
