"""The rotation-structured GEMM where it runs: every launch here is one that the
library gives to it (asserted), compared with the plain GEMM over all entries
and with the oracle at the edges of its tiles."""
from __future__ import annotations

import numpy as np
import pytest

import irisb200
import workload as W
from test_gpu_quad import _engine, _row_tables

pytestmark = pytest.mark.gpu


def _plain(e, offset, length, mult=1):
    e.set_tile(64)
    e.dot(offset, length, mult)
    assert e.last_gemm()[0] == "one_sm"
    out = e.fetch_results(length)
    e.set_tile(0)
    return out


def _quad(e, offset, length, mult=1):
    e.dot(offset, length, mult)
    assert e.last_gemm()[0] == "quad"
    return e.fetch_results(length)


def _slots(rng, n_q):
    """Full slots, and runs of 1..31 rotations from anywhere."""
    out = []
    for j in range(n_q):
        n = 31 if j % 3 else int(rng.integers(1, 32))
        out.append((int(rng.integers(n_q)), int(rng.integers(0, 32 - n)), n, j))
    return out


def _expected(oracle, rows, records, m0, mult, K, party, batch, remote):
    """The oracle's dot shares of entries m0.. against the given rows."""
    dots = oracle.dot_u16(rows, records).T
    if not remote:
        return (dots.astype(np.uint32) * mult % 65536).astype(np.uint16).T
    dom = oracle.DOM_CODE_DOT if K == 12800 else oracle.DOM_MASK_DOT
    return oracle.mask_dot_shares(dots, m0, rows.shape[0], mult, *W.SEEDS[party], dom, 0, batch).T


# one part-filled tile of quads, a full one, an uneven split over several; both
# code lengths, multipliers, with and without the zero-share mask
@pytest.mark.parametrize("n_q,n_db,K,remote,mult", [
    (18, 16384, 6400, True, 2), (20, 16353, 12800, True, 1), (24, 16384, 12800, False, 1), (26, 9500, 6400, False, 2),
    (32, 9500, 12800, True, 1), (40, 8192, 6400, True, 2), (64, 8129, 12800, True, 1)])
def test_slots(dm, oracle, n_q, n_db, K, remote, mult):
    rng = np.random.default_rng(n_q)
    e = _engine(dm, K, n_db, -(-n_q * 32 // 256) * 256 if n_q > 24 else n_q * 32, n_q, remote)
    base = rng.integers(0, 1 << 16, (n_q, K), dtype=np.uint16)
    slots = _slots(rng, n_q)
    e.query_upload_slots(base, slots)
    quad = _quad(e, 0, n_db, mult)
    assert np.array_equal(quad, _plain(e, 0, n_db, mult))
    rows = np.zeros((quad.shape[0], K), np.uint16)
    for s, (src, lo, n, _) in enumerate(slots):
        for r in range(n):
            rows[32 * s + r] = oracle.rotate_share(base[src], lo + r)
    for m0 in (0, 248, n_db - 24):  # the first and last entries, and the edge of the first tile
        exp = _expected(oracle, rows, e.fetch_records(m0, 24), m0, mult, K, 1, 7, remote)
        assert np.array_equal(quad[:, m0:m0 + 24], exp)
    e.close()


@pytest.mark.parametrize("K", [6400, 12800])
def test_row_tables(dm, oracle, K):
    """Rows with holes, single rows, mirrored bases: quads; unaligned runs and raw rows: not."""
    n_db, n_rows, n_base = 16384, 768, 9
    rng = np.random.default_rng(K)
    e = _engine(dm, K, n_db, n_rows, 5)
    base = rng.integers(0, 1 << 16, (n_base, K), dtype=np.uint16)
    for kind, d in enumerate(_row_tables(rng, n_rows, n_base)):
        e.query_upload_rows(base, d)
        plain = _plain(e, 0, n_db)
        rows = np.zeros((n_rows, K), np.uint16)
        for r in np.nonzero(d != 0xFFFFFFFF)[0]:
            src = base[d[r] >> 8]
            rows[r] = oracle.rotate_share(oracle.mirror_share(src, K == 12800) if d[r] & 0x80 else src, int(d[r] & 0x7F))
        assert np.array_equal(plain[:, 256:280], _expected(oracle, rows, e.fetch_records(256, 24), 256, 1, K, 1, 7, True))
        for upload in (lambda: None, lambda: (e.query_put_base(0, base), e.query_expand_rows(n_base, d))):
            upload()
            if kind == 1:  # another query's row in a quad
                e.dot(0, n_db, 1)
                assert e.last_gemm()[0] == "pair"
                assert np.array_equal(e.fetch_results(n_db), plain)
            else:
                assert np.array_equal(_quad(e, 0, n_db), plain)
    e.query_upload(rng.integers(0, 1 << 16, (n_rows, K), dtype=np.uint16))
    e.dot(0, n_db, 1)
    assert e.last_gemm()[0] == "pair"
    assert np.array_equal(e.fetch_results(n_db), _plain(e, 0, n_db))
    e.close()


def test_db_writes_and_gathers(dm):
    """The records' sums follow every kind of write; those that a gather leaves
    behind are brought in line by the next dot that reads them, outside captures."""
    K, n_db, n_q = 6400, 16384, 20
    rng = np.random.default_rng(3)
    e, src = _engine(dm, K, n_db, n_q * 32, 11), _engine(dm, K, n_db, 64, 12)
    base = rng.integers(0, 1 << 16, (n_q, K), dtype=np.uint16)
    rec = rng.integers(0, 1 << 16, (300, K), dtype=np.uint16)
    lo = ((rec & 0xFF).astype(np.uint8) ^ 0x80).view(np.int8)
    hi = ((rec >> 8).astype(np.uint8) ^ 0x80).view(np.int8)
    seen = []
    for write in (lambda: None, lambda: e.load_records(1000, rec), lambda: e.load_records_i8(2000, lo, hi),
                  lambda: e.gather_records(src, rng.permutation(n_db)[:n_db].astype(np.uint32)),
                  lambda: e.fill_random(77, 3000)):
        write()
        e.query_upload_slots(base, [(j, 0, 31, j) for j in range(n_q)])
        seen.append(_quad(e, 0, n_db))
        assert np.array_equal(seen[-1], _plain(e, 0, n_db))
    for a, b in zip(seen, seen[1:]):
        assert not np.array_equal(a, b)
    for n in (40, n_db):  # a few; and all of them while no rows are there for the quad GEMM
        for captured in (False, True):
            e.query_upload(base[:1])
            e.gather_records(src, rng.permutation(n_db)[:n].astype(np.uint32))
            e.set_db_len(n_db)
            e.query_upload_slots(base, [(j, 0, 31, j) for j in range(n_q)])
            past = _quad(e, 64, n_db - 64) if n == 40 else None  # records past those: no need
            plain = _plain(e, 0, n_db)
            assert past is None or np.array_equal(past, plain[:, 64:])
            if captured:
                dm.synchronize()
                g = irisb200.Graph.capture(dm, lambda: e.dot(0, n_db, 1, dm.stream(0)))
                assert e.last_gemm()[0] == "pair"
                g.launch(dm.stream(2))
                dm.synchronize()
                assert np.array_equal(e.fetch_results(n_db), plain)
                g.close()
            e.dot(0, n_db, 1, dm.stream(2))  # on a stream of its own
            dm.synchronize()
            irisb200.dot_many([e], [1], 0, n_db, dm.stream(1))
            assert e.last_gemm()[0] == "quad"
            dm.synchronize()
            assert np.array_equal(e.fetch_results(n_db), plain)
    e.close()
    src.close()


def test_replays_follow_the_uploads(dm):
    """A graph captured on quads replays on rows that are none, on another row
    count, and back: the device word says which GEMM runs."""
    K, n_db, n_rows = 6400, 16384, 768
    rng = np.random.default_rng(8)
    e = _engine(dm, K, n_db, n_rows, 2)
    base = rng.integers(0, 1 << 16, (9, K), dtype=np.uint16)
    tables = _row_tables(rng, n_rows, 9)
    want = []
    for d in tables:
        e.query_upload_rows(base, d)
        want.append(_plain(e, 0, n_db))
    e.query_upload_rows(base, tables[0])
    dm.synchronize()
    g = irisb200.Graph.capture(dm, lambda: e.dot(0, n_db, 1, dm.stream(0)))
    assert e.last_gemm() == ("captured", n_rows)
    for k in (0, 1, 3, 1, 2):
        e.query_upload_rows(base, tables[k])
        g.launch(dm.stream(0))
        assert e.last_gemm() == ("captured", 0 if k == 1 else n_rows)
        dm.synchronize()
        assert np.array_equal(e.fetch_results(n_db), want[k])
    e.query_upload_rows(base, tables[0][:640])  # fewer rows: the captured ones are no longer what the forms hold
    assert e.last_gemm()[1] == 640
    g.launch(dm.stream(0))
    dm.synchronize()
    e.query_upload_rows(base, tables[0])
    g.launch(dm.stream(0))
    dm.synchronize()
    assert np.array_equal(e.fetch_results(n_db), want[0])
    g.close()
    e.close()


def test_six_engines_and_sums_that_give_way(dm):
    """The six engines of a pass in one launch, direct and captured, before and
    after the library took the memory of their sums for an allocation."""
    n_db, n_q = 3000, 20
    rng = np.random.default_rng(9)
    engines = [irisb200.ShareDB(p % 3, dm, n_db, 640, 12800 if p < 3 else 6400, W.SEEDS[p % 3]) for p in range(6)]
    for k, e in enumerate(engines):
        e.alloc_db(n_db)
        e.fill_random(k, n_db)
        e.query_upload_slots(rng.integers(0, 1 << 16, (n_q, e.code_length), dtype=np.uint16),
                             [(j, 0, 31, j) for j in range(n_q)])
    mults = [1, 1, 1, 2, 2, 2]

    def check(gemm, held):
        irisb200.dot_many(engines, mults, 0, n_db)
        assert [e.last_gemm()[0] for e in engines] == [gemm] * 6 and all(e.has_sums() == held for e in engines)
        dm.synchronize()
        for e, w in zip(engines, want):
            assert np.array_equal(e.fetch_results(n_db), w)
    want = [_plain(e, 0, n_db, m) for e, m in zip(engines, mults)]
    check("quad", True)
    g = irisb200.Graph.capture(dm, lambda: irisb200.dot_many(engines, mults, 0, n_db, dm.stream(0)))
    assert {e.last_gemm() for e in engines} == {("captured", 640)}
    taken = []
    while any(e.has_sums() for e in engines):
        taken.append(irisb200.DeviceBuffer(dm, max(dm.mem_info()[0] - (1 << 30), 1 << 24)))
    check("pair", False)
    g.launch(dm.stream(0))
    dm.synchronize()
    for e, w in zip(engines, want):
        assert e.last_gemm()[1] == 0 and np.array_equal(e.fetch_results(n_db), w)
    g.close()
    for x in taken:
        x.free()
    for e in engines:
        e.close()


def test_runs_quads_tells_what_a_launch_does(dm):
    n_db = 9500
    rng = np.random.default_rng(10)
    engines = [irisb200.ShareDB(p % 3, dm, n_db, 1000, 6400, W.SEEDS[p % 3]) for p in range(6)]
    for e in engines:
        e.alloc_db(n_db)
    seen = set()
    for n_q in (16, 18, 20, 25, 30):
        for e in engines:
            e.query_upload_slots(rng.integers(0, 1 << 16, (n_q, 6400), dtype=np.uint16),
                                 [(j, 0, 31, j) for j in range(n_q)])
        for pair in (False, True):
            for e in engines:
                e.set_pair(pair)
            for some in (engines[:1], engines[:3], engines):
                for length in (96, 1024, 3000, n_db):
                    irisb200.dot_many(some, [1] * len(some), 0, length)
                    ran = some[0].last_gemm()[0] == "quad"
                    assert irisb200.ShareDB.runs_quads(some, 32 * n_q, length, pair) == ran
                    seen.add((n_q, ran))
    assert {q for q, ran in seen if ran} == {18, 20, 25, 30} and (16, False) in seen
    assert not irisb200.ShareDB.runs_quads(engines, 2048, n_db, False)  # above the capacity
    dm.derived_bytes(give_back=True)
    assert not irisb200.ShareDB.runs_quads(engines, 640, n_db, False)
    for e in engines:
        e.close()


def test_a_program_s_own_capture_keeps_the_sums(dm):
    """A dot captured by the program itself, on the engine's own party stream,
    replays on the sums it was captured with: they are not given back."""
    import torch
    K, n_db, n_q = 6400, 16384, 20
    rng = np.random.default_rng(14)
    e = irisb200.ShareDB(0, dm, n_db, n_q * 32, K, W.SEEDS[0])
    e.alloc_db(n_db)
    e.fill_random(6, n_db)
    e.query_upload_slots(rng.integers(0, 1 << 16, (n_q, K), dtype=np.uint16), [(j, 0, 31, j) for j in range(n_q)])
    want = _quad(e, 0, n_db)
    dm.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(dm.stream(0)), capture_error_mode="thread_local"):
        e.dot(0, n_db, 1)
    assert e.last_gemm() == ("captured", n_q * 32)
    dm.derived_bytes(give_back=True)
    assert e.has_sums()
    ptr, stride = e.result_view()
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(e.fetch_results(n_db), want)
    del g
    torch.cuda.synchronize()
    e.close()


def test_records_allocated_anew_start_a_new_generation_of_sums(dm):
    """Records allocated anew have sums and a device word of their own: a graph
    over the first ones (not launched again) keeps a word that no upload writes,
    and one captured over the new ones follows the uploads and the sums."""
    K, n_q = 6400, 20
    rng = np.random.default_rng(15)
    e = irisb200.ShareDB(0, dm, 16384, n_q * 32, K, W.SEEDS[0])
    base = rng.integers(0, 1 << 16, (n_q, K), dtype=np.uint16)
    slots = [(j, 0, 31, j) for j in range(n_q)]
    graphs, want = [], None
    for n_db in (16384, 16000, 16384):
        e.alloc_db(n_db)
        e.fill_random(n_db, n_db)
        e.query_upload_slots(base, slots)
        want = _quad(e, 0, n_db)
        assert np.array_equal(want, _plain(e, 0, n_db))
        dm.synchronize()
        graphs.append(irisb200.Graph.capture(dm, lambda: e.dot(0, n_db, 1, dm.stream(0))))
        assert e.last_gemm() == ("captured", n_q * 32)
        for held in (True, False):
            graphs[-1].launch(dm.stream(0))
            dm.synchronize()
            assert np.array_equal(e.fetch_results(n_db), want)
            dm.derived_bytes(give_back=True)
            assert not e.has_sums() and e.last_gemm()[1] == 0
    for g in graphs:
        g.close()
    e.close()
