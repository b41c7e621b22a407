"""The rotation-structured GEMM (quads of rotations, nine products of a quarter
of K) against the plain limb GEMM on the same engines: dot shares are whole
numbers modulo 2^16 and must be equal, for every form of upload, after every
kind of DB write, and in graph replays whose rows stop being quads."""
from __future__ import annotations

import numpy as np
import pytest

import irisb200
import workload as W

pytestmark = pytest.mark.gpu


def _engine(dm, K, n_db, rows, seed, remote=True, records=None):
    e = irisb200.ShareDB(1, dm, n_db, rows, K, W.SEEDS[1], is_remote=remote)
    e.alloc_db(n_db)
    e.fill_random(seed, records or n_db)
    e.set_batch(7)
    return e


def _both(e, offset, length, mult=1):
    """(quad GEMM, plain GEMM) results of the uploaded rows."""
    e.set_tile(0)
    e.dot(offset, length, mult)
    quad = e.fetch_results(length)
    e.set_tile(64)
    e.dot(offset, length, mult)
    plain = e.fetch_results(length)
    e.set_tile(0)
    return quad, plain


# padded rows of one part-filled quad tile, one full one, several, an uneven
# split over tiles; DB lengths around the 256-entry tile
@pytest.mark.parametrize("n_q,n_db,K,remote,mult", [
    (18, 8192, 6400, True, 2), (20, 9217, 12800, True, 1), (24, 9111, 6400, False, 1), (32, 4095, 12800, True, 2),
    (33, 8220, 6400, True, 1), (64, 2561, 12800, True, 1)])
def test_slots(dm, n_q, n_db, K, remote, mult):
    rng = np.random.default_rng(n_q)
    e = _engine(dm, K, n_db, n_q * 32, n_q, remote)
    base = rng.integers(0, 1 << 16, (n_q, K), dtype=np.uint16)
    slots = []
    for j in range(n_q):  # full slots, and runs of 1..31 rotations from anywhere
        n = 31 if j % 3 else int(rng.integers(1, 32))
        slots.append((int(rng.integers(n_q)), int(rng.integers(0, 32 - n)), n, j))
    e.query_upload_slots(base, slots)
    for offset, length in ((0, n_db), (32, n_db - 33), (0, 1)):
        quad, plain = _both(e, offset, length, mult)
        assert np.array_equal(quad, plain)
    e.close()


def _row_tables(rng, n_rows, n_base):
    """Row tables: aligned runs, runs that break quads, single rows, all empty."""
    out = []
    for kind in range(5):
        d = np.full(n_rows, 0xFFFFFFFF, np.uint32)
        for s in range(0, n_rows, 32):
            src, mir = int(rng.integers(n_base)), 0x80 if rng.random() < 0.5 else 0
            if kind == 0:  # 16 + 8 + 8 rows, aligned: quads
                for first, n in ((0, 16), (16, 8), (24, 8)):
                    src = int(rng.integers(n_base))
                    r0 = int(rng.integers(0, 31 - n + 1))
                    d[s + first:s + first + n] = (src << 8 | mir) + np.arange(r0, r0 + n)
            elif kind == 1:  # unaligned run and another query's row beside it: not quads
                d[s:s + 31] = (src << 8 | mir) + np.arange(31)
                d[s + 31] = (int(rng.integers(n_base)) << 8) + int(rng.integers(31))
            elif kind == 2:  # one row per quad, anywhere in it: quads
                for i in (0, 1, 8, 9, 16, 17, 24, 25):
                    d[s + i + 2 * int(rng.integers(4))] = (int(rng.integers(n_base)) << 8 | mir) + int(rng.integers(31))
            elif kind == 3:  # holes in a run: quads
                d[s:s + 31] = (src << 8 | mir) + np.arange(31)
                d[s + rng.choice(32, 11, replace=False)] = 0xFFFFFFFF
        out.append(d)
    return out


@pytest.mark.parametrize("K", [6400, 12800])
def test_row_tables(dm, K):
    n_db, n_rows, n_base = 8200, 768, 9
    rng = np.random.default_rng(K)
    e = _engine(dm, K, n_db, n_rows, 5)
    base = rng.integers(0, 1 << 16, (n_base, K), dtype=np.uint16)
    for d in _row_tables(rng, n_rows, n_base):
        e.query_upload_rows(base, d)
        quad, plain = _both(e, 0, n_db)
        assert np.array_equal(quad, plain)
        e.query_put_base(0, base)
        e.query_expand_rows(n_base, d)
        assert np.array_equal(_both(e, 0, n_db)[0], plain)
    e.query_upload(rng.integers(0, 1 << 16, (n_rows, K), dtype=np.uint16))  # rows of no structure
    quad, plain = _both(e, 0, n_db)
    assert np.array_equal(quad, plain)
    e.close()


def test_db_writes(dm):
    """The records' sums follow every kind of write, and records read back as written."""
    K, n_db = 6400, 8300
    rng = np.random.default_rng(3)
    e = _engine(dm, K, n_db, 640, 11)
    src = _engine(dm, K, 300, 64, 12)
    base = rng.integers(0, 1 << 16, (20, K), dtype=np.uint16)
    e.query_upload_slots(base, [(j, 0, 31, j) for j in range(20)])
    rec = rng.integers(0, 1 << 16, (300, K), dtype=np.uint16)

    def check():
        quad, plain = _both(e, 0, n_db)
        assert np.array_equal(quad, plain)
        return plain
    before = check()
    e.load_records(1000, rec)
    after = check()
    assert not np.array_equal(before[:, 1000:1300], after[:, 1000:1300])
    assert np.array_equal(e.fetch_records(1000, 300), rec)
    e.query_upload_slots(base, [(j, 0, 31, j) for j in range(20)])  # load_records used the query staging
    lo = ((rec & 0xFF).astype(np.uint8) ^ 0x80).view(np.int8)
    hi = ((rec >> 8).astype(np.uint8) ^ 0x80).view(np.int8)
    e.load_records_i8(2000, lo, hi)
    again = check()
    assert np.array_equal(e.fetch_records(2000, 300), rec)
    assert not np.array_equal(again[:, 2000:], after[:, 2000:])
    e.gather_records(src, np.arange(299, -1, -1, dtype=np.uint32))
    check()
    assert np.array_equal(e.fetch_records(0, 300), src.fetch_records(0, 300)[::-1])
    e.close()
    src.close()


def test_captured_launch_follows_the_uploads(dm):
    """A graph captured on quads replays correctly on rows that are none, and back."""
    K, n_db, n_rows = 6400, 8200, 768
    rng = np.random.default_rng(8)
    e = irisb200.ShareDB(0, dm, n_db, n_rows, K, W.SEEDS[0])
    e.alloc_db(n_db)
    e.fill_random(2, n_db)
    base = rng.integers(0, 1 << 16, (9, K), dtype=np.uint16)
    tables = _row_tables(rng, n_rows, 9)
    e.query_upload_rows(base, tables[0])
    dm.synchronize()
    g = irisb200.Graph.capture(dm, lambda: e.dot(0, n_db, 1, dm.stream(0)))
    for k in (0, 1, 3, 1, 2):
        e.query_upload_rows(base, tables[k])
        g.launch(dm.stream(0))
        got = e.fetch_results(n_db)
        assert np.array_equal(got, _both(e, 0, n_db)[1])
    dm.synchronize()
    g.close()
    e.close()


def test_captured_launch_keeps_its_row_count(dm):
    """A graph captured at one padded row count replays on those rows of a
    longer upload, whose forms lie elsewhere."""
    K, n_db = 6400, 4100
    rng = np.random.default_rng(12)
    e = irisb200.ShareDB(0, dm, n_db, 1024, K, W.SEEDS[0])
    e.alloc_db(n_db)
    e.fill_random(3, n_db)
    base = rng.integers(0, 1 << 16, (32, K), dtype=np.uint16)
    slots = [(j, 0, 31, j) for j in range(32)]
    e.query_upload_slots(base[:20], slots[:20])
    plain = _both(e, 0, n_db)[1]
    dm.synchronize()
    g = irisb200.Graph.capture(dm, lambda: e.dot(0, n_db, 1, dm.stream(0)))
    e.query_upload_slots(base, slots)  # 1024 rows, the first 640 as before
    g.launch(dm.stream(0))
    dm.synchronize()
    e.query_upload_slots(base[20:], slots[:12])
    e.query_upload_slots(base[:20], slots[:20])  # 640 rows again: the replay's result stride
    assert np.array_equal(e.fetch_results(n_db), plain)
    g.launch(dm.stream(0))
    assert np.array_equal(e.fetch_results(n_db), plain)
    dm.synchronize()
    g.close()
    e.close()


def test_small_gather_leaves_the_plain_gemm(dm):
    """A gather of a few records, then of many, then a write: results follow the records."""
    K, n_db = 6400, 8300
    rng = np.random.default_rng(4)
    e = _engine(dm, K, n_db, 640, 21)
    src = _engine(dm, K, 9000, 64, 22)
    base = rng.integers(0, 1 << 16, (20, K), dtype=np.uint16)
    for n in (300, 8200, 40):
        ids = rng.permutation(9000)[:n].astype(np.uint32)
        e.gather_records(src, ids)
        e.query_upload_slots(base, [(j, 0, 31, j) for j in range(20)])
        for offset, length in ((0, n_db), (320, n_db - 320)):
            quad, plain = _both(e, offset, length)
            assert np.array_equal(quad, plain)
    e.close()
    src.close()


@pytest.mark.parametrize("captured", [False, True])
def test_sums_give_way_to_other_allocations(dm, captured):
    """The library's own allocations take the room of the derived sums back,
    and results stay the same, those of a graph that was captured with them
    included."""
    K, n_db = 12800, 200000
    rng = np.random.default_rng(9)
    e = _engine(dm, K, 8192, 640, 31)
    big = irisb200.ShareDB(0, dm, 64, 640, K, W.SEEDS[0])
    big.alloc_db(n_db)  # 5 GB of records, 6.4 GB of sums
    base = rng.integers(0, 1 << 16, (20, K), dtype=np.uint16)
    e.query_upload_slots(base, [(j, 0, 31, j) for j in range(20)])
    before, plain = _both(e, 0, 8192)
    assert np.array_equal(before, plain)
    dm.synchronize()
    g = irisb200.Graph.capture(dm, lambda: e.dot(0, 8192, 1, dm.stream(0))) if captured else None
    taken = []  # mem_info counts what the sums hold as free (the driver may find more in its pools)
    while dm.mem_info()[0] > (4 << 30):
        taken.append(irisb200.DeviceBuffer(dm, dm.mem_info()[0] - (3 << 30)))
    after, _ = _both(e, 0, 8192)
    assert np.array_equal(after, plain)
    if captured:
        for _ in range(2):
            g.launch(dm.stream(0))
            assert np.array_equal(e.fetch_results(8192), plain)
            e.query_upload_slots(base, [(j, 0, 31, j) for j in range(20)])
        dm.synchronize()
        g.close()
    e.query_upload_slots(base, [(j, 0, 31, j) for j in range(20)])
    assert np.array_equal(_both(e, 0, 8192)[0], plain)
    for b in taken:
        b.free()
    big.close()
    e.close()
