"""Host-side logic of the batched launch (no GPU): the row descriptors that
point variants at shared base queries with the mirror bit, and the
expansion rule the device applies to them (rotation of the mirrored share)
checked against the oracle's mirror_share / rotate_share."""
from __future__ import annotations

import numpy as np

from oracle import oracle
from irisb200.batched import attach_bases, centred_rotations, pack


def expand_row(base: np.ndarray, d: int) -> np.ndarray:
    """The row that expand_rows_kernel builds for descriptor d from the base
    queries `base` [n][K], restated with numpy (4-coefficient columns)."""
    K = base.shape[1]
    src, rot, mirror = d >> 8, d & 0x7F, bool(d & 0x80)
    left = 15 - rot
    cols = base[src].reshape(K // 800, 200, 4).astype(np.int64)
    src_col = (np.arange(200) + left) % 200
    if mirror:
        src_col = np.where(src_col < 100, 99 - src_col, 299 - src_col)
    out = cols[:, src_col, :]
    if mirror and K == 12800:
        out[8:] = -out[8:]
    return (out % 65536).astype(np.uint16).reshape(K)


def test_attach_bases_sets_source_and_mirror_bit():
    variants = [list(centred_rotations(n)) for n in (31, 31, 16, 1, 1)]
    base_of = [0, 0, 1, 2, 2]
    mirrored = [False, True, False, False, True]
    lay = pack(variants)
    out = attach_bases(lay, base_of, mirrored)
    assert (lay.row_desc == out.row_desc).sum() == (lay.row_desc == 0xFFFFFFFF).sum() + \
        sum(len(r) for v, r in enumerate(variants) if base_of[v] == v and not mirrored[v])
    for r, d in enumerate(lay.row_desc):
        if d == 0xFFFFFFFF:
            assert out.row_desc[r] == 0xFFFFFFFF
            continue
        v = int(d) >> 8
        e = int(out.row_desc[r])
        assert e >> 8 == base_of[v]
        assert bool(e & 0x80) == mirrored[v]
        assert e & 0x7F == int(d) & 0xFF
    assert np.array_equal(out.seg_query, lay.seg_query) and np.array_equal(out.seg_mask, lay.seg_mask)


def test_device_mirror_rule_matches_oracle():
    rng = np.random.default_rng(11)
    for K, flip in ((12800, True), (6400, False)):
        base = rng.integers(0, 65536, (2, K), dtype=np.uint16)
        mirrored = oracle.mirror_share(base[1], flip)
        for rot in range(31):
            assert np.array_equal(expand_row(base, (1 << 8) | 0x80 | rot), oracle.rotate_share(mirrored, rot))
            assert np.array_equal(expand_row(base, (0 << 8) | rot), oracle.rotate_share(base[0], rot))


class _Obj:
    """Records calls; any method is a no-op."""

    def __init__(self, **kw):
        self.calls = []
        self.__dict__.update(kw)

    def __getattr__(self, name):
        def f(*a, **k):
            self.calls.append(name)
        return f


class _Buf:
    def __init__(self, shape, dtype):
        self.array = np.zeros(shape, dtype)

    def free(self):
        self.array = None


def _fake_engine(monkeypatch):
    """A BatchedEngine over fake device objects: the comparator reports
    variant v of the DB pass as matching entry 100 + v, and reauth variant v
    as matching its target when v is even."""
    import irisb200.batched as B
    from irisb200 import MAX_MATCHES_LEN

    class DM(_Obj):
        def set_host_sync(self, on):
            self.calls.append(("host_sync", bool(on)))

        def error_code(self):
            return 0

    class DC(_Obj):
        def fetch_final_results_into(self, n, final, counters, matches):
            assert not dm.calls or dm.calls[-1] != ("host_sync", True)
            counters[:n] = 1
            matches[:n, 0] = 100 + np.arange(n)

    class SDC(_Obj):
        def row_words(self):
            return 4

        def fetch_rows_into(self, first, n, out):
            out[:n] = 0
            for v in range(0, n, 2):
                out[v, v // 32] |= np.uint32(1 << (v % 32))

    class Graph:
        @staticmethod
        def capture(dm_, fn):
            fn()
            return _Obj()

    dm = DM()
    monkeypatch.setattr(B, "PinnedArray", _Buf)
    monkeypatch.setattr(B, "Event", _Obj)
    monkeypatch.setattr(B, "Graph", Graph)
    monkeypatch.setattr(B, "dot_many", lambda *a, **k: None)
    e = B.BatchedEngine.__new__(B.BatchedEngine)
    e.dm, e.c = dm, _Obj()
    e.ce = [_Obj(query_length=1024) for _ in range(3)]
    e.me = [_Obj(query_length=1024) for _ in range(3)]
    e.sce = [_Obj(query_length=8 * 64) for _ in range(3)]
    e.sme = [_Obj(query_length=8 * 64) for _ in range(3)]
    e.dc, e.sdc = DC(), SDC()
    e.scan = _Obj()  # the native DB pass (irs_scan_*): configure / run are no-ops here
    e.threshold_a, e.max_variants, e.max_reauth, e.db_len = 16384, 16, 8, 4096
    e._pin, e._pinned, e._events, e._inflight, e._par = None, [], None, [None, None], 0
    e.graphs, e.tuned, e.autotune, e.tune_log, e.fixed = {}, {}, False, {}, None
    assert MAX_MATCHES_LEN >= 1
    return e, dm


def test_submit_collect_maps_results_and_reuses_buffers(monkeypatch):
    from irisb200.batched import Request
    e, dm = _fake_engine(monkeypatch)
    z = np.zeros((3, 12800), np.uint16), np.zeros((3, 6400), np.uint16)

    def req(n, mir, kind="uniqueness", t=-1):
        return Request(code=z[0], mask=z[1], n_rot=n, mirrored=mir, kind=kind, target=t)
    batch = [req(31, True), req(16, False), req(1, True, "reauth", 7), req(31, False, "reauth", 9), req(1, False)]
    ta = e.submit(batch)
    tb = e.submit(batch)
    assert ta.par != tb.par and ta.results is None
    tc = e.submit(batch)  # reuses ta's buffers
    assert ta.results is not None and tc.par == ta.par
    for t in (ta, tb, tc):
        res = e.collect(t)
        # uniqueness variants in order: (0, normal), (0, mirror), (1, normal), (4, normal)
        assert res[0].matches == [100] and res[0].mirror_matches == [101]
        assert res[1].matches == [102] and res[4].matches == [103]
        # reauth variants: (2, normal) v0 hit, (2, mirror) v1 miss, (3, normal) v2 hit
        assert res[2].reauth_match is True and res[2].reauth_mirror_match is False
        assert res[3].reauth_match is True
    # every submit ran with host sync off and restored it afterwards
    syncs = [c for c in dm.calls if isinstance(c, tuple)]
    assert syncs == [("host_sync", False), ("host_sync", True)] * 3
    assert dm.calls.count("advance_batch_counter") == 3
    e.close()
    assert e._pin is None


def test_submit_rejects_oversized_batches(monkeypatch):
    import pytest
    from irisb200.batched import Request
    e, dm = _fake_engine(monkeypatch)
    for x in e.ce + e.me:
        x.query_length = 256  # 8 words of 32 rows
    z = np.zeros((3, 12800), np.uint16), np.zeros((3, 6400), np.uint16)
    with pytest.raises(ValueError):
        e.submit([Request(code=z[0], mask=z[1], n_rot=31, mirrored=True) for _ in range(9)])  # 18 variants > 16
    with pytest.raises(ValueError):  # 12 variants fit the count, but need 12 words of rows
        e.submit([Request(code=z[0], mask=z[1], n_rot=31, mirrored=True) for _ in range(6)])
    with pytest.raises(ValueError):  # reauth target outside the DB
        e.submit([Request(code=z[0], mask=z[1], n_rot=1, kind="reauth", target=e.db_len)])
    assert e._inflight == [None, None]
    assert not any(isinstance(c, tuple) for c in dm.calls)  # failed before any device work


def test_submit_edge_batches(monkeypatch):
    """An empty batch, a reauth-only batch and a uniqueness-only batch each
    complete; only the passes a batch needs are enqueued."""
    from irisb200.batched import Request
    e, dm = _fake_engine(monkeypatch)
    z = np.zeros((3, 12800), np.uint16), np.zeros((3, 6400), np.uint16)
    assert e.run([]) == []
    assert "compare_threshold_open_prepared" not in e.sdc.calls and not e.graphs
    res = e.run([Request(code=z[0], mask=z[1], n_rot=1, kind="reauth", target=3)])
    assert res[0].reauth_match is True and res[0].matches == [] and not e.graphs
    res = e.run([Request(code=z[0], mask=z[1], n_rot=16)])
    assert res[0].matches == [100] and res[0].reauth_match is None and e.graphs
    e.close()


def test_autotuner_candidates():
    """The tuner's candidates: the two-launch path at every tile width that
    divides the padded rows (the 64-row tile only up to 768 rows), the two-SM
    GEMM where the 256-row tile applies, the fused scan where the rows are a
    multiple of 128; the two-launch paths at 131,072 down to 8,192-entry
    chunks, the fused scan at the three longest (all capped at the DB)."""
    from irisb200.batched import BatchedEngine
    c = BatchedEngine._candidates(2048, 524288)
    assert ("split", 256, 131072) in c and ("split", 128, 32768) in c
    assert not any(t == 64 for _, t, _ in c)
    assert ("pair", 256, 65536) in c and ("fused", 128, 32768) in c
    assert ("pair", 256, 8192) in c and ("split", 256, 16384) in c and ("fused", 128, 16384) not in c
    assert len(c) == 2 * 5 + 5 + 3
    c = BatchedEngine._candidates(640, 524288)
    assert {t for p, t, _ in c if p == "split"} == {128, 64}
    assert not any(p == "pair" for p, _, _ in c) and any(p == "fused" for p, _, _ in c)
    c = BatchedEngine._candidates(64, 1000)
    assert c == [("split", 64, 1024)]


def _quad_pure(row_desc) -> bool:
    """No quad (rows i, i + 2, i + 4, i + 6 of an octet) holds rows of two
    variants, and a quad's rows keep their rotation distance."""
    for b in range(0, row_desc.size, 8):
        for i in (b, b + 1):
            live = [(int(d) >> 7, (int(d) & 0x7F) - 2 * m) for m, d in enumerate(row_desc[i:i + 8:2])
                    if d != 0xFFFFFFFF]
            if len(set(live)) > 1:
                return False
    return True


def test_pack_quads_keeps_quads_apart_and_every_row():
    from irisb200.batched import QUAD_MIN_ROWS, pack_for, pack_quads
    rng = np.random.default_rng(2)
    for _ in range(60):
        k = int(rng.integers(1, 80))
        rows = [list(centred_rotations(int(n))) for n in rng.choice([1, 2, 7, 8, 9, 16, 25, 31], k)]
        lay = pack_quads(rows)
        assert _quad_pure(lay.row_desc)
        seen = {v: [] for v in range(k)}
        for r, d in enumerate(lay.row_desc):
            if d != 0xFFFFFFFF:
                seen[int(d) >> 8].append((r, int(d) & 0x7F))
        for v, want in enumerate(rows):
            at = [r for r, _ in seen[v]]
            assert [rot for _, rot in seen[v]] == want and at == list(range(at[0], at[0] + len(want)))
            j = int(np.nonzero(lay.seg_query == v)[0][0])
            s = int(np.searchsorted(lay.seg_start, j, side="right")) - 1
            assert s == at[0] // 32 and int(lay.seg_mask[j]) == ((1 << len(want)) - 1) << (at[0] % 32)
        # no room for it, or too few rows to pay: the dense packing
        cap = -(-pack(rows).n_rows // 64) * 64
        small = pack_for(rows, cap)
        assert small.n_rows <= cap
        if lay.n_rows < QUAD_MIN_ROWS - 64:
            assert np.array_equal(pack_for(rows, 1 << 16).row_desc, pack(rows).row_desc)


def _mix(rng, n):
    """Requests of 1, 16 or 31 rotations, half of them mirrored."""
    from irisb200.batched import Request
    z = np.zeros((3, 12800), np.uint16), np.zeros((3, 6400), np.uint16)
    return [Request(code=z[0], mask=z[1], n_rot=int(rng.choice([1, 16, 31])), mirrored=bool(rng.random() < 0.5))
            for _ in range(n)]


def test_rows_are_packed_by_quads_only_where_the_pass_runs_them(monkeypatch):
    """An engine whose pass cannot run the quad GEMM (no sums, a path with a
    tile of its own, launches too short) packs densely; one that can, and gains
    by it, packs by quads."""
    e, _ = _fake_engine(monkeypatch)
    e.max_variants = 128
    asked = []

    class Engine(_Obj):
        runs = True

        def runs_quads(self, engines, n_rows, length, pair):
            asked.append((len(engines), n_rows, length, pair))
            return Engine.runs
    e.ce = [Engine(query_length=4096) for _ in range(3)]
    e.me = [Engine(query_length=4096) for _ in range(3)]
    reqs = _mix(np.random.default_rng(4), 48)
    uniq, _ = e._variants(reqs)
    dense = pack([list(centred_rotations(reqs[i].n_rot)) for i, _ in uniq])

    def rows(path, autotune=False):
        e.fixed, e.autotune = path, autotune
        buf = np.zeros(4096, np.uint32)
        seg = (np.zeros(129, np.uint32), np.zeros(128, np.uint32), np.zeros(128, np.uint32))
        code, mask = np.zeros((3, 128, 12800), np.uint16), np.zeros((3, 128, 6400), np.uint16)
        return e._stage(reqs, uniq, code, mask, buf, seg, 4096, pad=True)[0]
    live = lambda lay: int((lay.row_desc != 0xFFFFFFFF).sum())  # noqa: E731
    for path, autotune in (("pair", False), (None, True), ("pair", True)):
        lay = rows(path, autotune)
        assert _quad_pure(lay.row_desc) and live(lay) == live(dense)
        assert asked[-1][0] == 6 and asked[-1][2] <= e.db_len and asked[-1][3]
    for path, autotune in (("split", False), ("fused", False), (None, False), ("split", True)):
        n = len(asked)
        lay = rows(path, autotune)  # a tile width of its own: not even asked
        assert lay.n_slots == dense.n_slots and not _quad_pure(lay.row_desc) and len(asked) == n
    e.tuned = {k: ("split", 256, 32768) for k in range(64, 4097, 64)}  # what the tuner chose
    assert not _quad_pure(rows(None, True).row_desc)
    e.tuned = {k: ("split", 0, 32768) for k in range(64, 4097, 64)}  # the library's own choice
    assert _quad_pure(rows(None, True).row_desc)
    e.tuned = {}
    Engine.runs = False
    assert not _quad_pure(rows("pair").row_desc)


def test_packing_takes_the_cheaper_pass():
    """Quads kept apart cost padded rows: they are taken where the measured time
    of that many on the quad GEMM is below that of the dense rows."""
    from irisb200.batched import pack_for, pack_quads, padded_rows
    rng = np.random.default_rng(8)
    quad = dict(zip((640, 768, 1024, 1280, 2048), (2.55, 2.85, 3.47, 4.65, 6.55)))
    plain = dict(zip((512, 640, 768, 1024, 1280, 2048), (2.37, 3.2, 3.6, 4.7, 5.95, 9.7)))
    both = set()
    for n in range(17, 60):
        rows = [list(centred_rotations(r.n_rot)) for r in _mix(rng, n) for _ in range(2 if r.mirrored else 1)]
        got = pack_for(rows, 4096)
        dense, apart = pack(rows), pack_quads(rows)
        p, q = padded_rows(dense.n_rows, 4096), padded_rows(apart.n_rows, 4096)
        if p not in plain or q not in quad or dense.n_rows != -(-sum(map(len, rows)) // 32) * 32:
            continue
        pays = quad[q] < plain[p]
        assert np.array_equal(got.row_desc, (apart if pays else dense).row_desc)
        both.add((p, q, pays))
    assert (512, 640, False) in both and any(pays for _, _, pays in both)


def test_the_two_sm_path_takes_every_row_count_it_can_run():
    from irisb200.batched import BatchedEngine
    e = BatchedEngine.__new__(BatchedEngine)
    e.db_len, e.fixed = 65536, "pair"
    assert e._pass_candidates(640) == [("pair", 256, c) for c in (65536, 32768, 16384, 8192)]
    assert e._pass_candidates(2048) == [c for c in BatchedEngine._candidates(2048, 65536) if c[0] == "pair"]
    assert e._pass_candidates(64) == BatchedEngine._candidates(64, 65536)  # no two-SM GEMM there
    e.fixed = None
    assert e._pass_candidates(640) == BatchedEngine._candidates(640, 65536)
