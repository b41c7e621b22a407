"""Writes into the resident DB between batches: an identity update (a new
record written at an index, write_db_at_index, actor.rs:3547-3600) becomes
matchable, and a deletion (the default-iris record, actor.rs:2641-2680)
removes a match; each pass equals the CPU path on the records read back."""
from __future__ import annotations

import numpy as np
import pytest

import irisb200
import workload as W

pytestmark = pytest.mark.gpu

N_DB, NQ, A = 512, 4, 16384


def _scan(dm, c, ce, me, qc, qm):
    dc = irisb200.DistanceComparator(dm, NQ, N_DB)
    try:
        irisb200.dot_many(ce + me, [1, 1, 1, 2, 2, 2], 0, N_DB)
        dc.compare_threshold_open(c, ce, me, 0, N_DB, NQ, A)
        dm.synchronize()
        return irisb200.bitmap_get(dc.fetch_bitmap(NQ, N_DB), NQ, N_DB)
    finally:
        dc.close()


def test_update_and_delete(dm, oracle):
    codes, masks, cs, ms = W.make_db(oracle, N_DB, 0xAB12)
    qc, qm, plain = W.make_queries(oracle, NQ, codes, masks, 9, {0: (100, 0), 2: (300, 5)})
    ce = [irisb200.ShareDB(p, dm, N_DB, NQ * 32, 12800, W.SEEDS[p]) for p in range(3)]
    me = [irisb200.ShareDB(p, dm, N_DB, NQ * 32, 6400, W.SEEDS[p]) for p in range(3)]
    c = irisb200.Circuits(dm, W.SEEDS)
    slots = [(j, 0, 31, j) for j in range(NQ)]
    try:
        for p in range(3):
            ce[p].alloc_db(N_DB)
            me[p].alloc_db(N_DB)
            ce[p].load_records(0, cs[p])
            me[p].load_records(0, ms[p])
            ce[p].query_upload_slots(qc[p], slots)
            me[p].query_upload_slots(qm[p], slots)
        before = _scan(dm, c, ce, me, qc, qm)
        assert before[0, 100] and before[2, 300]
        # identity update: entry 7 becomes query 1's own iris (fresh shares)
        code1, mask1 = plain[1]
        rc, rm = irisb200.encode_iris(code1, mask1, seed=777)
        for p in range(3):
            ce[p].load_records(7, rc[p][None])
            me[p].load_records(7, rm[p][None])
        # deletion of entry 100
        irisb200.delete_records(ce, me, [100])
        after = _scan(dm, c, ce, me, qc, qm)
        assert after[1, 7] and not after[0, 100] and after[2, 300]
        cs2 = np.stack([ce[p].fetch_records(0, N_DB) for p in range(3)])
        ms2 = np.stack([me[p].fetch_records(0, N_DB) for p in range(3)])
        assert np.array_equal(after, W.expected_bitmap(oracle, qc, qm, cs2, ms2, A))
        assert not after[:, 100].any()  # the deletion record matches none of the queries
    finally:
        c.close()
        for e in ce + me:
            e.close()


def _limbs(rec):
    return ((rec & 0xFF).astype(np.uint8) ^ 0x80).view(np.int8), ((rec >> 8).astype(np.uint8) ^ 0x80).view(np.int8)


# the shortest code, the longest whose limbs fit a block's shared memory, and one that does not
@pytest.mark.parametrize("K", [128, 232448, 232576])
def test_stored_limbs_of_any_length(dm, K):
    rng = np.random.default_rng(K)
    e = irisb200.ShareDB(0, dm, 64, 64, K, W.SEEDS[0])
    e.alloc_db(64)
    rec = rng.integers(0, 1 << 16, (7, K), dtype=np.uint16)
    e.load_records_i8(20, *_limbs(rec))
    assert np.array_equal(e.fetch_records(20, 7), rec)
    assert not e.fetch_records(19, 1).any() and not e.fetch_records(27, 1).any()
    e.load_records(40, rec)
    assert np.array_equal(e.fetch_records(40, 7), rec)
    e.close()


def test_stored_limbs_need_no_free_memory():
    """Records go into the resident database however full the device is."""
    K, n = 6400, 8192
    rng = np.random.default_rng(1)
    rec = rng.integers(0, 1 << 16, (n, K), dtype=np.uint16)
    dm = irisb200.DeviceManager(0)
    e = irisb200.ShareDB(0, dm, 64, 64, K, W.SEEDS[0])
    e.alloc_db(n)
    e.load_records_i8(0, *_limbs(rec[:1]))  # the kernels are loaded
    taken = []
    for step in (1 << 30, 1 << 25):  # less than 64 MB stay free
        while dm.mem_info()[0] > 2 * step:
            taken.append(irisb200.DeviceBuffer(dm, max(step, dm.mem_info()[0] - 2 * step)))
    try:
        e.load_records_i8(0, *_limbs(rec))
        assert np.array_equal(e.fetch_records(0, n), rec)
    finally:
        for b in taken:
            b.free()
        e.close()
        dm.close()


@pytest.mark.parametrize("K,n", [(128, 3), (6400, 70), (12800, 2400)])
def test_random_records_are_the_seeded_words(dm, K, n):
    """fill_random: 64-bit word i of each limb, in record order, is splitmix64 of the seed at i."""
    e = irisb200.ShareDB(0, dm, 64, 64, K, W.SEEDS[0])
    e.alloc_db(n)
    e.fill_random(99, n)

    def limb(seed):
        with np.errstate(over="ignore"):
            z = np.uint64(seed) + np.arange(1, n * K // 8 + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return (z ^ (z >> np.uint64(31))).view(np.uint8).astype(np.uint16).reshape(n, K)
    assert np.array_equal(e.fetch_records(0, n), limb(99) | limb(99 ^ 0x5A5A5A5A5A5A5A5A) << 8)
    e.close()
