"""The work a user of the GPU operators has them do, as cases that can be timed.

Each case is one query step on relations that are already in device memory,
through the C ABI (include/pythia_gpu.h) as pythia_gb300.gpu binds it: the
calls a plan's operators make. Relations are arrays of packed tuples of 8-byte
columns: a key, then payload columns. Join rows and groups come in no stated
order, so the cases that return groups sort them by key as an ORDER BY would,
and the joins either aggregate or write the rows of a foreign-key join.
"""
import ctypes

import torch

from pythia_gb300 import gpu

_CTX = None
SPREAD = -7046029254386353131        # odd: maps 1..n to n distinct 64-bit keys all over the domain


def _ctx():
    global _CTX
    if _CTX is None:
        _CTX = gpu.Context(0)
    return _CTX


def listed():
    return [
        # A dimension lookup of a few thousand tuples: launches and round trips.
        dict(name="join_agg_tiny", kind="join_agg", build=1000, probe=10_007, domain="dense", width=16, skew=False),
        # 1M x 16M primary-key join under count and sum.
        dict(name="join_agg", kind="join_agg", build=1 << 20, probe=16 << 20, domain="dense", width=16, skew=False),
        # Keys that are not a compact range (ids, hashes): the hashed table.
        dict(name="join_agg_sparse", kind="join_agg", build=3_000_017, probe=48_000_011, domain="sparse", width=16,
             skew=False),
        # 16M x 256M foreign-key join, every row written.
        dict(name="join_rows_large", kind="join_rows", build=16 << 20, probe=256 << 20),
        # Join feeding an aggregate (the served plans): sum of a dec column per build-side group.
        dict(name="join_group_dec", kind="join_group", build=4 << 20, probe=40 << 20, groups=41_943),
        # 256-way radix partition, the input of partitioned plans.
        dict(name="partition_256", kind="partition", rows=100_000_007, width=16, fn="parammodulo", buckets=256),
        # Page sort of 64M tuples, keys U[0, 16M).
        dict(name="sort_64m", kind="sort", rows=64 << 20, bits=24, width=16),
        # Group-by of 256M rows into a million groups, dec sums.
        dict(name="groupby_dec_large", kind="groupby", rows=256 << 20, groups=1_000_000, domain="dense", val="dec"),
        # Group-by on 64-bit ids: hashed groups, long sums.
        dict(name="groupby_ids", kind="groupby", rows=20_000_003, groups=250_000, domain="sparse", val="long"),
        # Sort-merge join of 64M x 64M, about four duplicates a key on each side, under count and sum.
        dict(name="mpsm_agg", kind="mpsm_agg", build=64 << 20, probe=64 << 20, bits=24),
        # Sort-merge join with its rows written, then summed per build-side category.
        dict(name="mpsm_rows", kind="mpsm_rows", build=16 << 20, probe=16 << 20, bits=22, groups=1000),
        # Scan of 24-byte lines (order, part, price): half pass the filter, two columns are kept.
        dict(name="filter_project", kind="filter_project", rows=50_000_003, width=24, share=0.5),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["join_agg", "join_rows", "join_group", "partition", "sort", "groupby", "mpsm_agg", "mpsm_rows",
                       "filter_project"])
    if kind == "join_agg":
        build = _log(rng, 1000, 4 << 20)
        return dict(kind=kind, build=build, probe=_log(rng, 2 * build, 16 * build) | 1,
                    domain=rng.choice(["dense", "sparse"]), width=rng.choice([16, 16, 24]), skew=rng.random() < 0.3)
    if kind == "join_rows":
        build = _log(rng, 1000, 16 << 20)
        return dict(kind=kind, build=build, probe=_log(rng, build, 8 * build) | 1)
    if kind == "join_group":
        build = _log(rng, 10_000, 4 << 20)
        return dict(kind=kind, build=build, probe=10 * build + rng.randrange(100), groups=max(1, build // 100))
    if kind == "partition":
        fn = rng.choice(["parammodulo", "modulo", "exactrange"])
        return dict(kind=kind, rows=_log(rng, 1000, 64 << 20) | 1, width=rng.choice([16, 16, 24]), fn=fn,
                    buckets=rng.randrange(3, 256) if fn == "exactrange" else 1 << rng.randrange(3, 11))
    if kind == "sort":
        return dict(kind=kind, rows=_log(rng, 1000, 64 << 20) | 1,
                    bits=rng.choice([rng.randrange(16, 32), rng.randrange(44, 62)]), width=rng.choice([16, 16, 24]))
    if kind == "groupby":
        rows = _log(rng, 10_000, 128 << 20) | 1
        return dict(kind=kind, rows=rows, groups=_log(rng, 10, max(20, min(2_000_000, rows // 8))),
                    domain=rng.choice(["dense", "sparse"]), val=rng.choice(["int", "long", "dec"]))
    if kind == "mpsm_agg":
        n = _log(rng, 10_000, 64 << 20)
        return dict(kind=kind, build=n, probe=_log(rng, n // 4 + 1, n) | 1, bits=max(10, n.bit_length() - rng.randrange(0, 4)))
    if kind == "mpsm_rows":
        n = _log(rng, 10_000, 16 << 20)
        probe, bits = _log(rng, n // 4 + 1, n) | 1, max(10, n.bit_length() - rng.randrange(0, 3))
        return dict(kind=kind, build=n, probe=probe, bits=bits,
                    groups=rng.randrange(4, max(6, min(1500, (n * probe >> bits) // 40))))
    return dict(kind=kind, rows=_log(rng, 10_000, 64 << 20) | 1, width=rng.choice([16, 24, 40]),
                share=rng.choice([0.02, 0.3, 0.5, 0.9]))


# ---------------------------------------------------------------- inputs
def _ints(g, n, hi):
    return torch.randint(0, hi, (n,), generator=g, device="cuda", dtype=torch.int64)


def _rows(*cols):
    return torch.stack(cols, dim=1).contiguous()


def _decs(g, n):
    """Prices: [0, 10000) as float64 bit patterns."""
    return (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 1e4).view(torch.int64)


def _build_side(g, n, domain, payload):
    keys = torch.randperm(n, generator=g, device="cuda") + 1
    return _rows(keys * SPREAD if domain == "sparse" else keys, payload)


def _fk(g, R, n, skew=False):
    """n foreign keys into R: uniform, or with log-uniform ranks (Zipf, s = 1)."""
    if not skew:
        return R[_ints(g, n, R.shape[0]), 0]
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    return R[(float(R.shape[0]) ** u).long().clamp_(1, R.shape[0]) - 1, 0]


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    kind = case["kind"]
    if kind in ("join_agg", "join_rows"):
        R = _build_side(g, case["build"], case.get("domain", "dense"), _ints(g, case["build"], 1 << 31))
        n = case["probe"]
        cols = [_fk(g, R, n, case.get("skew", False)), _ints(g, n, 1 << 31)]
        if case.get("width", 16) == 24:                 # (line number, foreign key, value)
            cols.insert(0, torch.arange(n, device="cuda"))
        return R, _rows(*cols)
    if kind == "join_group":
        R = _build_side(g, case["build"], "dense", _ints(g, case["build"], case["groups"]))
        return R, _rows(_fk(g, R, case["probe"]), _decs(g, case["probe"]))
    if kind in ("partition", "sort"):
        n = case["rows"]
        hi = 1 << (case["bits"] if kind == "sort" else 40)
        cols = [_ints(g, n, hi), _ints(g, n, 1 << 31)]
        if case["width"] == 24:
            cols.append(torch.arange(n, device="cuda"))
        return (_rows(*cols),)
    if kind == "groupby":
        n = case["rows"]
        k = _ints(g, n, case["groups"])
        k[torch.randperm(n, generator=g, device="cuda")[: case["groups"]]] = torch.arange(case["groups"], device="cuda")
        v = _decs(g, n) if case["val"] == "dec" else _ints(g, n, 1 << 31)
        return (_rows(k * SPREAD if case["domain"] == "sparse" else k, v),)
    if kind in ("mpsm_agg", "mpsm_rows"):
        hi = 1 << case["bits"]
        R = _rows(_ints(g, case["build"], hi), _ints(g, case["build"], case.get("groups", 1 << 31)))
        return R, _rows(_ints(g, case["probe"], hi), _ints(g, case["probe"], 1 << 31))
    n = case["rows"]
    # Prices below the filter's constant for exactly the stated share of the rows, in random places.
    u, cut = torch.rand(n, generator=g, device="cuda", dtype=torch.float64), 1e4 * case["share"]
    low = torch.randperm(n, generator=g, device="cuda") < int(n * case["share"])
    price = torch.where(low, u * cut, cut + u * (1e4 - cut)).view(torch.int64)
    cols = [torch.arange(n, device="cuda"), _ints(g, n, 1 << 20), price, _ints(g, n, 1 << 31), _ints(g, n, 1 << 31)]
    return (_rows(*(cols[1:3] if case["width"] == 16 else cols[: case["width"] // 8])),)


def _rel(t, key_off=0, key_bytes=8):
    return gpu.Rel(t.data_ptr(), t.shape[0], t.shape[1] * t.element_size(), key_off, key_bytes)


def _empty(n, words=2, dtype=torch.int64):
    return torch.empty((max(int(n), 1), words), dtype=dtype, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    ctx = _ctx()
    t = _inputs(case, seed)
    st = dict(case=case, ctx=ctx, t=t)
    if kind in ("join_agg", "join_rows", "join_group"):
        off = 8 if case.get("width", 16) == 24 else 0
        st["R"], st["S"] = _rel(t[0]), _rel(t[1], off)
        if kind == "join_group":
            st["proj"] = gpu.cols((("B", 8, 8), ("P", 8, 8)))
            st["out"], st["sorted"] = _empty(case["groups"]), _empty(case["groups"])
        else:
            st["proj"] = gpu.cols((("P", off + 8, 8), ("B", 8, 8)))
            if kind == "join_rows":
                st["out"] = _empty(case["probe"])
    elif kind == "partition":
        st["in"], st["out"] = _rel(t[0]), torch.empty_like(t[0])
        st["cfg"] = gpu.hashcfg(case["fn"], case["buckets"], min=0, max=(1 << 40) - 1)
        nb = ctx.nbuckets(st["cfg"])
        st["offs"] = torch.empty(nb + 1, dtype=torch.int64, device="cuda")
    elif kind == "sort":
        st["in"], st["out"] = _rel(t[0]), torch.empty_like(t[0])
    elif kind == "groupby":
        st["in"] = _rel(t[0])
        words, dtype = (3, torch.int32) if case["val"] == "int" else (2, torch.int64)
        st["out"], st["sorted"] = _empty(case["groups"], words, dtype), _empty(case["groups"], words, dtype)
    elif kind in ("mpsm_agg", "mpsm_rows"):
        st["R"], st["S"] = _rel(t[0]), _rel(t[1])
        if kind == "mpsm_rows":
            st["proj"] = gpu.cols((("B", 8, 8), ("P", 8, 8)))
            hi = 1 << case["bits"]
            m = int((torch.bincount(t[0][:, 0], minlength=hi) * torch.bincount(t[1][:, 0], minlength=hi)).sum())
            st["rows"] = _empty(m)
            st["out"], st["sorted"] = _empty(case["groups"]), _empty(case["groups"])
        else:
            st["proj"] = gpu.cols((("P", 8, 8), ("B", 8, 8)))
    else:
        w = case["width"]
        st["in"] = _rel(t[0], 0, 0)
        st["kept"] = torch.empty_like(t[0])
        price = 8 if w == 16 else 16
        st["preds"] = gpu.preds([("dec", "<", price, 1e4 * case["share"])])
        st["cols"] = gpu.cols([(0, price - 8, 8), (0, price, 8)] if w != 16 else [(0, price, 8)])
        st["out"] = _empty(case["rows"], 2 if w != 16 else 1)
    return st


# ---------------------------------------------------------------- the calls
def _groups(ctx, out, dest, ng, key_bytes=8):
    """Groups ordered by key, as (key, aggregate) rows."""
    r = gpu.Rel(out.data_ptr(), ng, out.shape[1] * out.element_size(), 0, key_bytes)
    ctx._check(gpu.lib().pg_sort_pages(ctx.h, ctx.stream, ctypes.byref(r), dest.data_ptr()))
    return dest[:ng]


def run(st):
    case, ctx, L = st["case"], st["ctx"], gpu.lib()
    kind, ref = case["kind"], ctypes.byref
    if kind in ("join_agg", "join_rows", "join_group"):
        c, nc = st["proj"]
        ht, res, ng = ctypes.c_void_p(), gpu.JoinResult(), ctypes.c_uint64()
        ctx._check(L.pg_hashjoin_build(ctx.h, ctx.stream, ref(st["R"]), c, nc, ref(ht)))
        try:
            if kind == "join_agg":
                ctx._check(L.pg_hashjoin_probe(ctx.h, ctx.stream, ht, ref(st["S"]), c, nc, None, 0,
                                               gpu.JOIN_COUNT | gpu.JOIN_SUM, 1, ref(res)))
                return {"rows": res.n_out, "sum": res.sum}
            if kind == "join_rows":
                ctx._check(L.pg_hashjoin_probe(ctx.h, ctx.stream, ht, ref(st["S"]), c, nc, st["out"].data_ptr(),
                                               case["probe"], gpu.JOIN_MATERIALIZE, -1, ref(res)))
                return st["out"][: res.n_out]
            ctx._check(L.pg_hashjoin_groupby(ctx.h, ctx.stream, ht, ref(st["S"]), 8, gpu.VAL["dec"], gpu.AGG["sum"],
                                             st["out"].data_ptr(), case["groups"], ref(ng)))
        finally:
            ctx._check(L.pg_hashtable_free(ctx.h, ht))
        t = _groups(ctx, st["out"], st["sorted"], ng.value)
        return {"keys": t[:, 0], "sums": t.view(torch.float64)[:, 1]}
    if kind == "partition":
        ctx._check(L.pg_partition(ctx.h, ctx.stream, ref(st["in"]), ref(st["cfg"]), st["out"].data_ptr(),
                                  st["offs"].data_ptr()))
        return st["out"], st["offs"]
    if kind == "sort":
        ctx._check(L.pg_sort_pages(ctx.h, ctx.stream, ref(st["in"]), st["out"].data_ptr()))
        return st["out"]
    if kind == "groupby":
        ng = ctypes.c_uint64()
        ctx._check(L.pg_groupby(ctx.h, ctx.stream, ref(st["in"]), 8, gpu.VAL[case["val"]], gpu.AGG["sum"],
                                case["groups"], st["out"].data_ptr(), case["groups"], ref(ng)))
        t = _groups(ctx, st["out"], st["sorted"], ng.value)
        return {"keys": t[:, 0], "sums": t.view(torch.float64)[:, 1]} if case["val"] == "dec" else t
    if kind in ("mpsm_agg", "mpsm_rows"):
        c, nc = st["proj"]
        res, ng = gpu.JoinResult(), ctypes.c_uint64()
        if kind == "mpsm_agg":
            ctx._check(L.pg_mpsm_join(ctx.h, ctx.stream, ref(st["R"]), ref(st["S"]), c, nc, None, 0,
                                      gpu.JOIN_COUNT | gpu.JOIN_SUM, 1, ref(res)))
            return {"rows": res.n_out, "sum": res.sum}
        ctx._check(L.pg_mpsm_join(ctx.h, ctx.stream, ref(st["R"]), ref(st["S"]), c, nc, st["rows"].data_ptr(),
                                  st["rows"].shape[0], gpu.JOIN_MATERIALIZE, -1, ref(res)))
        j = gpu.Rel(st["rows"].data_ptr(), res.n_out, 16, 0, 8)
        ctx._check(L.pg_groupby(ctx.h, ctx.stream, ref(j), 8, gpu.VAL["long"], gpu.AGG["sum"], case["groups"],
                                st["out"].data_ptr(), case["groups"], ref(ng)))
        return {"rows": res.n_out, "groups": _groups(ctx, st["out"], st["sorted"], ng.value)}
    kept = ctypes.c_uint64()
    pr, npr = st["preds"]
    c, nc = st["cols"]
    ctx._check(L.pg_filter(ctx.h, ctx.stream, ref(st["in"]), pr, npr, st["kept"].data_ptr(), ref(kept)))
    k = gpu.Rel(st["kept"].data_ptr(), kept.value, case["width"], 0, 0)
    ctx._check(L.pg_project(ctx.h, ctx.stream, ref(k), c, nc, st["out"].data_ptr()))
    return st["kept"][: kept.value], st["out"][: kept.value]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("join_agg", "mpsm_agg"):
        return dict(bytes=16 * case["build"] + case.get("width", 16) * case["probe"], flops=0)
    if kind == "join_rows":
        return dict(bytes=16 * case["build"] + 32 * case["probe"], flops=0)
    if kind == "join_group":
        return dict(bytes=16 * (case["build"] + case["probe"] + case["groups"]), flops=0)
    if kind in ("partition", "sort"):
        return dict(bytes=2 * case["width"] * case["rows"], flops=0)
    if kind == "groupby":
        return dict(bytes=16 * (case["rows"] + case["groups"]), flops=0)
    if kind == "mpsm_rows":
        pairs = case["build"] * case["probe"] / (1 << case["bits"])
        return dict(bytes=16 * (case["build"] + case["probe"] + 2 * pairs), flops=0)
    w, out = case["width"], 8 if case["width"] == 16 else 16
    return dict(bytes=case["rows"] * (w + case["share"] * (2 * w + out)), flops=0)


def exact(case, seed):
    """Dec sums in 64-bit floating point; everything else is whole numbers."""
    kind = case["kind"]
    if kind == "join_group":
        R, S = _inputs(case, seed)
        group = torch.empty(case["build"] + 1, dtype=torch.int64, device="cuda")
        group[R[:, 0]] = R[:, 1]
        idx, vals, spread = group[S[:, 0]], S[:, 1], False
    elif kind == "groupby" and case["val"] == "dec":
        (T,) = _inputs(case, seed)
        spread = case["domain"] == "sparse"
        inv = pow(SPREAD & ((1 << 64) - 1), -1, 1 << 64)
        idx, vals = (T[:, 0] * (inv - (1 << 64) if inv >> 63 else inv) if spread else T[:, 0]), T[:, 1]
    else:
        return None
    sums = torch.zeros(case["groups"], dtype=torch.float64, device="cuda")
    sums.index_add_(0, idx, vals.contiguous().view(torch.float64))
    present = torch.nonzero(torch.bincount(idx, minlength=case["groups"]))[:, 0]
    if spread:
        present = present[torch.argsort(present * SPREAD)]
    return {"keys": None, "sums": sums[present]}
