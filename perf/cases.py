"""Performance cases of the iris uniqueness path, through the package's public entry points.

Every case is a call that a program built on irisb200 makes: one batch against the resident share database
(PlainScan), the whole call with its uploads and downloads, a batch of uneven requests (BatchedEngine), the
continuous server, the second-stage re-check of candidates (SubsetPass), the limb dot product of one engine,
and the comparison circuit on flat share vectors with and without its OR tree.  Irises, shares and randomness
are synthetic and seeded: code bits uniform, mask pairs kept with probability 0.9, some queries near-duplicates
of database entries.  All outputs are whole numbers (bits, indices, counts, shares modulo 2^16), so two builds
agree on them exactly and there is no 64-bit value to compare with.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "iris-mpc_b200"))

import irisb200 as I  # noqa: E402
from irisb200.batched import BatchedEngine, Request  # noqa: E402
from irisb200.scan import PlainScan  # noqa: E402
from irisb200.serving import ContinuousServer  # noqa: E402
from irisb200.subset import SubsetPass  # noqa: E402

# (seed0, seed1) of the three parties: party p's second seed is party p-1's own
SEEDS = [([0] * 8, [2] * 8), ([1] * 8, [0] * 8), ([2] * 8, [1] * 8)]
K_CODE, K_MASK = I.IRIS_CODE_LENGTH, I.MASK_CODE_LENGTH
A = I.THRESHOLD_ANON_STATS_A
LARGEST = 64 * 131072  # (query, entry) pairs of the largest case


def listed():
    return [
        # one iris against a small development database: launches and host work
        {"name": "scan_1x1000", "kind": "scan", "queries": 1, "entries": 1000, "path": "default"},
        # one person, both orientations, against a shard: the pass streams the database
        {"name": "scan_2x131072", "kind": "scan", "queries": 2, "entries": 131072, "path": "default"},
        # a part-filled batch and a database that is no multiple of any tile
        {"name": "scan_23x20011", "kind": "scan", "queries": 23, "entries": 20011, "path": "default"},
        # the full 64-query batch on the two-SM GEMM that the tuner picks for it, one shard of the benchmark's database
        {"name": "scan_64x131072", "kind": "scan", "queries": 64, "entries": 131072, "path": "pair"},
        # the same batch as a caller sees it: host shares in, self check, merged results out
        {"name": "e2e_64x32768", "kind": "e2e", "queries": 64, "entries": 32768, "path": "pair"},
        # uneven requests (1, 16 and 31 rotations, mirrored ones, reauths) in one launch
        {"name": "batched_48x65536", "kind": "batched", "requests": 48, "entries": 65536},
        # a burst at the continuous server
        {"name": "serve_24x40000", "kind": "serve", "requests": 24, "entries": 40000},
        # the candidates of a batch checked again at the match ratio
        {"name": "subset_32x700", "kind": "subset", "queries": 32, "ids": 700, "entries": 20000},
        # one party's code dots, the row count of the reference's matmul benchmark
        {"name": "dot_930x32768", "kind": "dot", "rows": 930, "entries": 32768, "mask": False, "remote": True},
        # the comparison circuit alone: a few words, and a whole chunk's worth
        {"name": "compare_4096", "kind": "compare", "elements": 4096, "or_tree": False},
        {"name": "compare_16M", "kind": "compare", "elements": 1 << 24, "or_tree": False},
        # the comparison reduced to one shared bit
        {"name": "or_tree_1M", "kind": "compare", "elements": (1 << 20) + 64, "or_tree": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan", "e2e", "batched", "serve", "subset", "dot", "dot", "compare", "compare"])
    if kind in ("scan", "e2e"):
        q = _log(rng, 1, 64)
        n = min(_log(rng, 500, 131072 if kind == "scan" else 32768), LARGEST // q)
        return {"kind": kind, "queries": q, "entries": n, "path": rng.choice(["default", "pair"])}
    if kind == "batched":
        return {"kind": kind, "requests": _log(rng, 2, 48), "entries": _log(rng, 2000, 65536)}
    if kind == "serve":
        return {"kind": kind, "requests": _log(rng, 2, 24), "entries": _log(rng, 2000, 40000)}
    if kind == "subset":
        return {"kind": kind, "queries": _log(rng, 1, 64), "ids": _log(rng, 8, 4000), "entries": 20000}
    if kind == "dot":
        return {"kind": kind, "rows": _log(rng, 31, 2048), "entries": _log(rng, 500, 65536),
                "mask": rng.random() < 0.4, "remote": rng.random() < 0.8}
    or_tree = rng.random() < 0.3
    return {"kind": kind, "elements": 64 * _log(rng, 1, (1 << 20) // 64 if or_tree else (1 << 24) // 64),
            "or_tree": or_tree}


class _Held:
    """The handles of one state, closed with it."""

    def __init__(self):
        self.dm = I.DeviceManager(0)
        self.own = []

    def keep(self, x):
        self.own.append(x)
        return x

    def __del__(self):
        try:
            self.dm.synchronize()
            for x in reversed(self.own):
                (x.close if hasattr(x, "close") else x.free)()
            self.dm.close()
        except Exception:
            pass


class _View:
    """A device buffer of the library as torch sees it; the tensor keeps its owner alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


def _database(h, seed, entries, rows, result_entries, capacity=None):
    """Six resident engines (three parties, code and mask) over a synthetic database."""
    ce = [h.keep(I.ShareDB(p, h.dm, result_entries, rows, K_CODE, SEEDS[p])) for p in range(3)]
    me = [h.keep(I.ShareDB(p, h.dm, result_entries, rows, K_MASK, SEEDS[p])) for p in range(3)]
    for e in ce + me:
        e.alloc_db(capacity or entries)
    I.synth_db(ce, me, seed, 0, entries)
    return ce, me, h.keep(I.Circuits(h.dm, SEEDS))


def _planted(rng, n, entries):
    """Every third query is a near-duplicate of a database entry, turned by up to 15 columns."""
    at = rng.choice(entries, size=min(n, entries), replace=False)
    return {j: (int(at[j]), int(rng.integers(-15, 16))) for j in range(0, min(n, entries), 3)}


def _requests(rng, seed, n, entries):
    """1, 16 or 31 rotations, half of them mirrored, one in five a reauth."""
    code, mask = I.synth_queries(seed, seed + 1, n, _planted(rng, n, entries))
    out = []
    for j in range(n):
        reauth = rng.random() < 0.2
        out.append(Request(code=np.ascontiguousarray(code[:, j]), mask=np.ascontiguousarray(mask[:, j]),
                           n_rot=int(rng.choice([1, 16, 31])), mirrored=bool(rng.random() < 0.5),
                           kind="reauth" if reauth else "uniqueness",
                           target=int(rng.integers(entries)) if reauth else -1))
    return out


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    h = _Held()
    s = {"case": dict(case), "held": h, "dm": h.dm, "batch": 0}
    if kind in ("scan", "e2e"):
        nq, n = case["queries"], case["entries"]
        chunk = 32768 if case["path"] == "pair" else 65536
        ce, me, c = _database(h, seed, n, nq * 32, max(64, min(chunk, (n + 31) // 32 * 32)))
        dc = h.keep(I.DistanceComparator(h.dm, nq, n))
        ps = h.keep(PlainScan(h.dm, ce, me, c, dc, nq, n, A))
        if case["path"] == "pair":
            ps.configure(("pair", 256, chunk))
        code, mask = I.synth_queries(seed, seed + 1, nq, _planted(rng, nq, n))
        slots = [(j, 0, 31, j) for j in range(nq)]
        rows = np.zeros((nq, dc.row_words()), np.uint32)
        s.update(ce=ce, me=me, c=c, dc=dc, ps=ps, slots=slots, rows=rows)
        if kind == "scan":
            for p in range(3):
                ce[p].query_upload_slots(code[p], slots)
                me[p].query_upload_slots(mask[p], slots)
        else:
            pc, pm = h.keep(I.PinnedArray(code.shape, np.uint16)), h.keep(I.PinnedArray(mask.shape, np.uint16))
            pc.array[:], pm.array[:] = code, mask
            # the batch's own irises as records, for the check of the batch against itself
            sce, sme, _ = _records_of_batch(h, seed, nq, rng, n)
            s.update(pc=pc, pm=pm, sce=sce, sme=sme)
    elif kind == "batched":
        ce, me, c = _database(h, seed, case["entries"], 128 * 32, case["entries"])
        reqs = _requests(rng, seed, case["requests"], case["entries"])
        s.update(engine=h.keep(BatchedEngine(h.dm, ce, me, c, max_variants=128, max_reauth=64, threshold_a=A,
                                             seeds=SEEDS, autotune=False, path="pair")), requests=reqs)
    elif kind == "serve":
        ce, me, c = _database(h, seed, case["entries"], 2048, 32768, capacity=case["entries"] + 64)
        reqs = _requests(rng, seed, case["requests"], case["entries"])
        s.update(server=h.keep(ContinuousServer(h.dm, ce, me, c, row_capacity=2048, max_variants=128, max_reauth=32,
                                                threshold_a=A, seeds=SEEDS)), requests=reqs)
    elif kind == "subset":
        nq, n = case["queries"], case["entries"]
        ce, me, c = _database(h, seed, n, 64, 64)
        planted = _planted(rng, nq, n)
        code, mask = I.synth_queries(seed, seed + 1, nq, planted)
        ids = np.unique(np.concatenate([rng.choice(n, size=case["ids"], replace=False),
                                        np.array([e for e, _ in planted.values()], np.int64)]))
        s.update(subset=h.keep(SubsetPass(h.dm, ce, me, c, max_queries=nq, max_subset=4096, seeds=SEEDS)),
                 code=code, mask=mask, ids=ids)
    elif kind == "dot":
        k = K_MASK if case["mask"] else K_CODE
        db = h.keep(I.ShareDB(0, h.dm, case["entries"], case["rows"], k, SEEDS[0], is_remote=case["remote"]))
        db.alloc_db(case["entries"])
        db.fill_random(seed, case["entries"])
        db.query_upload(rng.integers(0, 1 << 16, (case["rows"], k), dtype=np.uint16))
        ptr, stride = db.result_view()
        s.update(db=db, out=torch.as_tensor(_View(h, ptr, (case["entries"], stride), "<i2"), device="cuda"))
    else:
        n = case["elements"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        shares = [torch.randint(-(1 << 15), 1 << 15, (n,), dtype=torch.int16, device="cuda", generator=g)
                  for _ in range(6)]
        s.update(c=h.keep(I.Circuits(h.dm, SEEDS)), shares=shares, ptr=[x.data_ptr() for x in shares])
        if not case["or_tree"]:
            s["res"] = [torch.empty(n // 64, dtype=torch.int64, device="cuda") for _ in range(6)]
            s["res_ptr"] = [x.data_ptr() for x in s["res"]]
            s["opened"] = I.DeviceBuffer(h.dm, n // 8)
            s["opened_view"] = torch.as_tensor(_View((h, s["opened"]), s["opened"].ptr, (n // 64,), "<i8"), device="cuda")
    torch.cuda.synchronize()
    return s


def _records_of_batch(h, seed, nq, rng, entries):
    """Engines whose records are the batch's irises, as the in-batch check holds them; one iris repeats."""
    sce = [h.keep(I.ShareDB(p, h.dm, max(nq, 32), nq * 32, K_CODE, SEEDS[p])) for p in range(3)]
    sme = [h.keep(I.ShareDB(p, h.dm, max(nq, 32), nq * 32, K_MASK, SEEDS[p])) for p in range(3)]
    code, mask = I.synth_queries(seed, seed + 1, nq, _planted(np.random.default_rng(seed), nq, entries),
                                 preprocess=False)
    for p in range(3):
        sce[p].alloc_db(max(nq, 32))
        sme[p].alloc_db(max(nq, 32))
        sce[p].load_records(0, code[p])
        sme[p].load_records(0, mask[p])
    return sce, sme, None


MULTS = [1, 1, 1, 2, 2, 2]


def _next_batch(s, *handles):
    """A fresh randomness id for the batch, as a program gives every batch."""
    s["batch"] = s["batch"] % 1000000 + 1
    for x in handles:
        x.set_batch(s["batch"])


def _merged(s):
    nq = s["case"]["queries"]
    s["dc"].fetch_rows_into(0, nq, s["rows"])
    return (*s["dc"].fetch_final_results(nq), s["rows"])


def run(s):
    kind = s["case"]["kind"]
    if kind == "scan":
        _next_batch(s, *s["ce"], *s["me"], s["c"])
        s["dc"].reset()
        s["ps"].scan()
        s["dc"].join_db_matches(s["case"]["queries"], s["case"]["entries"])
        return _merged(s)
    if kind == "e2e":
        nq, n = s["case"]["queries"], s["case"]["entries"]
        _next_batch(s, *s["ce"], *s["me"], *s["sce"], *s["sme"], s["c"])
        for p in range(3):
            for code, mask in ((s["ce"][p], s["me"][p]), (s["sce"][p], s["sme"][p])):
                code.query_upload_slots(s["pc"].array[p], s["slots"])
                mask.query_upload_slots(s["pm"].array[p], s["slots"])
        s["dc"].reset()
        I.dot_many(s["sce"] + s["sme"], MULTS, 0, nq)
        s["dc"].compare_threshold_open(s["c"], s["sce"], s["sme"], 0, nq, nq, A, self_check=True)
        s["ps"].scan()
        s["dc"].join_db_matches(nq, n)
        s["dc"].join_batch_matches(nq)
        return _merged(s)
    if kind == "batched":
        return _results(s["engine"].run(s["requests"]))
    if kind == "serve":
        done = s["server"].serve([0.0] * len(s["requests"]), s["requests"])
        return _results([c.result for c in sorted(done, key=lambda c: c.idx)])
    if kind == "subset":
        found = s["subset"].run(s["code"], s["mask"], s["ids"], I.THRESHOLD_A)
        return (np.array([len(x) for x in found]), np.array([e for x in found for e in x], np.int64),
                s["subset"].match_counts)
    if kind == "dot":
        _next_batch(s, s["db"])
        s["db"].dot(0, s["case"]["entries"], 2 if s["case"]["mask"] else 1)
        return s["out"]
    _next_batch(s, s["c"])
    if s["case"]["or_tree"]:
        return s["c"].compare_threshold_masked_many_with_or_tree(s["ptr"][:3], s["ptr"][3:], s["case"]["elements"], A)
    s["c"].compare_threshold_masked_many(s["ptr"][:3], s["ptr"][3:], s["case"]["elements"], A,
                                         res_a=s["res_ptr"][:3], res_b=s["res_ptr"][3:], opened=s["opened"])
    return (*s["res"], s["opened_view"])


def _results(found):
    """One row per request: match counts, the first match and the reauth bits (-1 where there is none)."""
    first = lambda v: v[0] if v else -1  # noqa: E731
    value = lambda v: -1 if v is None else int(v)  # noqa: E731
    return np.array([[value(r.match_count), first(r.matches), value(r.mirror_match_count), first(r.mirror_matches),
                      value(r.reauth_match), value(r.reauth_mirror_match)] for r in found], np.int64)


def work(case):
    """Every share read once and every result written once; a multiply-add per coefficient of each query row and
    entry; per compared element, the keystream that the protocol draws (24 blocks of 592 operations for 32)."""
    kind = case["kind"]
    per_entry = 3 * 2 * (K_CODE + K_MASK)
    if kind == "dot":
        k = K_MASK if case["mask"] else K_CODE
        return {"bytes": 2 * k * (case["entries"] + case["rows"]) + 2 * case["rows"] * case["entries"],
                "flops": 2 * k * case["rows"] * case["entries"]}
    if kind == "compare":
        n = case["elements"]
        return {"bytes": 12 * n + (0 if case["or_tree"] else 7 * n // 8), "flops": 24 * 592 * n // 32}
    if kind == "subset":
        rows, entries = 31 * case["queries"], case["ids"]
    elif kind in ("scan", "e2e"):
        rows, entries = 31 * case["queries"], case["entries"]
    else:  # 1, 16 or 31 rotations, three orientations for two requests, four in five against the database
        rows, entries = int(16 * 1.5 * 0.8 * case["requests"]) + 1, case["entries"]
    return {"bytes": per_entry * entries + per_entry * max(1, rows // 31) + rows * entries // 31 / 8,
            "flops": 3 * (2 * (K_CODE + K_MASK) + 24 * 592 / 32 / 3) * rows * entries}


def exact(case, seed):
    """Whole numbers throughout: shares, bits and indices, equal or wrong."""
    return None
