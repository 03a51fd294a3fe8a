"""Edges of the tiled and counted kernels: sizes around tile boundaries, widths
that change the copy unit, unaligned bases, key windows at their limits."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc
from pythia_gb300 import datagen as dg
from pythia_gb300 import gpu

pytestmark = pytest.mark.gpu


def _rows(n, width, seed):
    """n rows of `width` bytes whose first int32 is uniform in [0, 1000)."""
    rng = np.random.default_rng(seed)
    a = rng.integers(-(1 << 31), 1 << 31, size=(n, width // 4), dtype=np.int64).astype(np.int32)
    a[:, 0] = rng.integers(0, 1000, size=n)
    return a


# Tiles hold (24 KB / width) rows rounded down to 32, at least 32; over 1024
# bytes a thread copies each tuple.
@pytest.mark.parametrize("width", [4, 8, 12, 16, 24, 40, 136, 1024, 1028])
@pytest.mark.parametrize("shift", [0, 4, 8])
def test_filter_and_project_tile_edges(ctx, width, shift):
    L = gpu.lib()
    tile = max(32, 24 * 1024 // width // 32 * 32)
    for n in (1, 31, 33, tile - 1, tile, tile + 1, 5 * tile + 7):
        rows = _rows(n, width, width * 1000 + n)
        src, dst = ctx.alloc(rows.nbytes + 64), ctx.alloc(rows.nbytes + 64)
        ctx._check(L.pg_h2d(ctx.h, ctx.stream, src.ptr + shift, rows.ctypes.data, rows.nbytes))
        r = gpu.Rel(src.ptr + shift, n, width, 0, 0)
        for limit in (0, 300, 1000):                       # none, some, every row
            pr, npr = gpu.preds([("int", "<", 0, limit)])
            m = ctypes.c_uint64()
            ctx._check(L.pg_filter(ctx.h, ctx.stream, ctypes.byref(r), pr, npr, dst.ptr + shift, ctypes.byref(m)))
            got = np.empty((m.value, width // 4), dtype=np.int32)
            if m.value:
                ctx._check(L.pg_d2h(ctx.h, ctx.stream, got.ctypes.data, dst.ptr + shift, got.nbytes))
                ctx.sync()
            assert np.array_equal(got, rows[rows[:, 0] < limit])
        cols = [(width - 4, 4)] if width < 16 else [(width - 8, 8), (0, 4), (8, 4)]
        c = (gpu.Col * len(cols))(*[gpu.Col(0, o, b) for o, b in cols])
        ctx._check(L.pg_project(ctx.h, ctx.stream, ctypes.byref(r), c, len(cols), dst.ptr + shift))
        want = np.concatenate([rows[:, o // 4:(o + b) // 4] for o, b in cols], axis=1)
        got = np.empty_like(want)
        ctx._check(L.pg_d2h(ctx.h, ctx.stream, got.ctypes.data, dst.ptr + shift, got.nbytes))
        ctx.sync()
        assert np.array_equal(got, want)


def _mpsm(ctx, R, S, **kw):
    proj = (("P", 8, 8), ("B", 8, 8))
    got, n, _ = ctx.mpsm(R, S, proj=proj, **kw)
    want, wn, _ = orc.mergejoin(R, S, proj=proj)
    assert n == wn and np.array_equal(orc.canonical(got), orc.canonical(want))
    for sc in (0, 1):
        _, n2, s2 = ctx.mpsm(R, S, proj=proj, flags=gpu.JOIN_COUNT | gpu.JOIN_SUM, sum_col=sc)
        assert (n2, s2) == orc.mergejoin(R, S, proj=proj, materialise=False, sum_col=sc)[1:]


# Key windows at the counted join's limits (2^24 values whatever the size, 16
# tuples' worth beyond), either side of the scan's blocks, values that do and
# do not fit 4 bytes, and runs either side of the longest one warp writes.
@pytest.mark.parametrize("case", ["one_key", "scan_edge", "widest", "too_wide", "wide_values", "extremes", "run_limit",
                                  "over_run_limit"])
def test_mpsm_counted_window(ctx, case):
    n = 30_000
    R, S = dg.uniform_keys(n, 4096, dg.seed_for(201)), dg.uniform_keys(n, 4096, dg.seed_for(202))
    if case == "one_key":
        R, S = R[:300], S[:200]
        R[:, 0] = S[:, 0] = -7
    elif case == "scan_edge":
        R[0, 0], R[1, 0] = 0, 4096                          # 4097 counts: one in the second block
        S[0, 0] = 4096
    elif case == "widest":
        R[0, 0], R[1, 0] = 0, (1 << 24) - 1
    elif case == "too_wide":
        R[0, 0], R[1, 0] = 0, 1 << 40
        S[5, 0] = 1 << 40
    elif case == "wide_values":
        R[::2, 1] = -R[::2, 1]
        R[0, 1], R[1, 1] = np.iinfo(np.int64).min, np.iinfo(np.int64).max
    elif case == "extremes":
        R[:, 0] += np.iinfo(np.int64).max - 5000
        S[:, 0] += np.iinfo(np.int64).max - 5000
        S[3, 0] = np.iinfo(np.int64).min
    else:
        R[: 16384 + (case == "over_run_limit"), 0] = 99
        S = S[:500]
        S[:3, 0] = 99
    _mpsm(ctx, R, S)


# The rows' values are kept as 2- or 4-byte differences where their span allows;
# a warp takes 64 probe tuples, a block 512.
@pytest.mark.parametrize("span", [0, (1 << 16) - 1, 1 << 16, (1 << 32) - 1, 1 << 32])
@pytest.mark.parametrize("n", [1, 64, 65, 512, 513, 40_003])
def test_mpsm_value_spans(ctx, n, span):
    R, S = dg.uniform_keys(n, n // 3 + 1, dg.seed_for(208)), dg.uniform_keys(n + 1, n // 3 + 1, dg.seed_for(209))
    R[:, 1] = 77 + R[:, 1] % (span + 1)
    R[0, 1], R[-1, 1] = 77, 77 + span
    S[0, 0], S[-1, 0] = R[0, 0], R[-1, 0]
    _mpsm(ctx, R, S)


def test_mpsm_key_outside_the_sampled_window(ctx):
    # Over 4M tuples the window comes from every 1024th; a matching key far from
    # the rest and off the sample must still join.
    n = (1 << 22) + 5
    R, S = dg.uniform_keys(n, 1 << 20, dg.seed_for(203)), dg.uniform_keys(1000, 1 << 20, dg.seed_for(204))
    R[1025, 0] = S[7, 0] = 3 << 20
    _, n2, s2 = ctx.mpsm(R, S, flags=gpu.JOIN_COUNT | gpu.JOIN_SUM, sum_col=0)
    assert (n2, s2) == orc.mergejoin(R, S, materialise=False, sum_col=0)[1:]
    got, n3, _ = ctx.mpsm(R, S)
    want, _, _ = orc.mergejoin(R, S)
    assert n3 == n2 and np.array_equal(orc.canonical(got), orc.canonical(want))


# Rows of over 32M build and 8M probe tuples go by a partition of both sides; a key off
# the sampled window sends them to the exact one.
@pytest.mark.parametrize("far", [False, True])
def test_mpsm_rows_partitioned_first(ctx, far):
    n, m = (32 << 20) + 3, (8 << 20) + 5
    rng = np.random.default_rng(212)
    R = np.stack([rng.permutation(n) - 9, rng.integers(0, 1 << 31, size=n)], axis=1)
    S = np.stack([rng.integers(0, n, size=m) - 9, np.arange(m)], axis=1)
    want = np.empty(n, dtype=np.int64)
    want[R[:, 0] + 9] = R[:, 1]
    want = want[S[:, 0] + 9]
    if far:
        old = R[1025, 0]
        R[1025, 0] = 3 * n
        S[S[:, 0] == old, 0] = 3 * n
        S[5, 0], want[5] = 3 * n, R[1025, 1]
    got, rows, _ = ctx.mpsm(R, S, proj=(("P", 8, 8), ("B", 8, 8)))
    assert rows == m
    got = np.ascontiguousarray(got).view(np.int64).reshape(-1, 2)
    seen = np.full(m, -1, dtype=np.int64)
    seen[got[:, 0]] = got[:, 1]
    assert np.array_equal(seen, want)


# 16-byte tuples and at most 256 buckets: tiles of 3072 rows over two blocks an
# SM. Sizes around one tile, a chunk of several, keys in any word, 4-byte keys
# and every kind of bucket function.
@pytest.mark.parametrize("n", [1, 31, 3071, 3072, 3073, 304 * 3072 + 1, 2 * 304 * 3072 - 5])
@pytest.mark.parametrize("cfg", [("parammodulo", dict(buckets=256)), ("parammodulo", dict(buckets=256, skipbits=28, offset=9)),
                                 ("parammodulo", dict(buckets=128, skipbits=40)), ("modulo", dict(buckets=8)),
                                 ("exactrange", dict(buckets=231, min=-(1 << 40), max=1 << 40)), ("knuth", dict(buckets=64)),
                                 ("alwayszero", dict())])
def test_partition_16_byte_tiles(ctx, n, cfg):
    rows = dg.uniform_keys(n, 1 << 41, dg.seed_for(205))
    rows[:, 0] -= 1 << 40
    fn, kw = cfg
    for key in ((0, 8), (8, 8), (4, 8), (12, 4)):
        if fn == "exactrange" and key != (0, 8):
            continue
        got, offs = ctx.partition(rows, gpu.hashcfg(fn, **kw), *key)
        want, woffs = orc.partition(rows, orc.hashcfg(fn, **kw), key)
        assert np.array_equal(offs, woffs)
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8))


# From 4M tuples the sort's digits come from a sampled key window: an aligned
# one, one that straddles zero, one that a key off the sample refutes, and spans
# over 63 bits. Ties keep input order.
@pytest.mark.parametrize("case", ["aligned", "straddling", "refuted", "power_of_two_edge", "one_value", "full_span"])
def test_sort_key_windows(ctx, case):
    n = (1 << 22) + 77
    rows = dg.uniform_keys(n, 1 << 20, dg.seed_for(206))
    if case == "straddling":
        rows[:, 0] -= 1 << 19
    elif case == "refuted":
        rows[1025, 0], rows[2050, 0] = 1 << 45, -5
    elif case == "power_of_two_edge":
        rows[5, 0] = 1 << 20
    elif case == "one_value":
        rows[:, 0] = 42
    elif case == "full_span":
        rows[:, 0] *= -7046029254386353131
        rows[3, 0], rows[4, 0] = np.iinfo(np.int64).min, np.iinfo(np.int64).max
    want = rows[np.argsort(rows[:, 0], kind="stable")]
    assert np.array_equal(ctx.sort(rows), want)


def _same_join(ctx, R, S, **kw):
    got, n, _ = ctx.hashjoin(R, S, **kw)
    want, wn, _ = orc.hashjoin(R, S, hash=orc.hashcfg("modulo", 1 << 12), **kw)
    assert n == wn and np.array_equal(orc.canonical(got), orc.canonical(want))
    for sc in (0, 1):
        _, n2, s2 = ctx.hashjoin(R, S, flags=gpu.JOIN_COUNT | gpu.JOIN_SUM, sum_col=sc, **kw)
        assert (n2, s2) == orc.hashjoin(R, S, materialise=False, sum_col=sc, hash=orc.hashcfg("modulo", 1 << 12), **kw)[1:]


# Builds of up to 2^20 tuples are one cooperative launch of a block per 2048, which
# makes either layout: dense, or hashed for keys too far apart or repeated; wide
# values and the empty-marker key (-1) beside far keys go back to the exact build.
BUILDS = ["dense", "far", "repeated", "far_repeated", "marker", "marker_far", "wide_values", "extremes"]


@pytest.mark.parametrize("n,case", [(n, c) for n in (1, 2, 33, 2048, 2049, 70_001) for c in BUILDS] +
                         [(n, c) for n in (1 << 20, (1 << 20) + 1) for c in ("dense", "far")])
def test_join_small_builds(ctx, n, case):
    R = dg.build_relation(n, dg.seed_for(207))
    S = dg.probe_uniform(3 * n + 5, R, dg.seed_for(208))
    if case in ("far", "far_repeated", "marker_far"):
        R[:, 0] *= -7046029254386353131
        S[:, 0] *= -7046029254386353131
    if case in ("repeated", "far_repeated"):
        R[n // 2:, 0] = R[: n - n // 2, 0]
    elif case in ("marker", "marker_far"):
        R[n // 3, 0] = S[1, 0] = -1
        if case == "marker":
            R[:, 0] = np.arange(-2, n - 2)
    elif case == "wide_values":
        R[0, 1] = -5
    elif case == "extremes":
        R[0, 0], R[-1, 0] = np.iinfo(np.int64).min, np.iinfo(np.int64).max
        S[0, 0], S[2, 0] = R[0, 0], R[-1, 0]
    S[::5, 0] += 1                                          # some misses
    _same_join(ctx, R, S)


# Hashed counts and sums: one tuple a thread in blocks of 256, 64 blocks an SM.
@pytest.mark.parametrize("m", [1, 255, 257, 152 * 64 * 256 + 3])
def test_join_hashed_agg_sizes(ctx, m):
    R = dg.build_relation(70_000, dg.seed_for(209))
    S = dg.probe_uniform(m, R, dg.seed_for(210))
    R[:, 0] *= -7046029254386353131
    S[:, 0] *= -7046029254386353131
    R[9, 0] = -1
    S[:: max(1, m // 7), 0] = -1
    for sc in (0, 1):
        _, n2, s2 = ctx.hashjoin(R, S, flags=gpu.JOIN_COUNT | gpu.JOIN_SUM, sum_col=sc)
        assert (n2, s2) == orc.hashjoin(R, S, materialise=False, sum_col=sc, hash=orc.hashcfg("modulo", 1 << 16))[1:]


# Up to 2^20 tuples sort in one cooperative launch: one block of 4096 rows, every
# block with four or eight rows a thread, one pass, eight passes, one value; then
# the first size past it. Other widths go by (key, row) records. Ties keep order.
@pytest.mark.parametrize("n", [1, 31, 4096, 4097, 150_000, 152 * 4096, 152 * 4096 + 1, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("bits", [0, 1, 8, 9, 30, 64])
def test_sort_one_launch(ctx, n, bits):
    rows = dg.uniform_keys(n, 1 << min(bits, 40), dg.seed_for(211))
    if bits == 64:
        rows[:, 0] *= -7046029254386353131
        rows[0, 0], rows[-1, 0] = np.iinfo(np.int64).max, np.iinfo(np.int64).min
    else:
        rows[:, 0] -= 1 << bits >> 1
    assert np.array_equal(ctx.sort(rows), rows[np.argsort(rows[:, 0], kind="stable")])
    if n <= 150_000:
        assert np.array_equal(ctx.sort(rows, (8, 8)), rows[np.argsort(rows[:, 1], kind="stable")])
        words = rows.view(np.int32).reshape(n, 4)
        for width, off in ((12, 0), (24, 8), (20, 4)):
            t = np.zeros((n, width // 4), dtype=np.int32)
            t[:, 0], t[:, -1] = np.arange(n), np.arange(n)
            t[:, off // 4:off // 4 + 2] = words[:, :2]
            assert np.array_equal(ctx.sort(t, (off, 8)), t[np.argsort(rows[:, 0], kind="stable")])


# Dense group tables in shared memory: 224 KB a CTA, two CTAs an SM up to half of
# that. Slots of 4 (counts), 5 (int), 9 (long) and 13 bytes (dec, 53 up to 2163 slots
# with the words of small values); larger windows go to the global table. Dec sums
# all of one sign overflow their word, tiny values and zeros need the lazy words.
@pytest.mark.parametrize("val,groups", [("count", 27_000), ("int", 1), ("int", 22_938), ("long", 3), ("long", 12_743),
                                        ("long", 12_744), ("long", 25_486), ("long", 25_487), ("dec", 2), ("dec", 2163),
                                        ("dec", 2164), ("dec", 8822), ("dec", 8823), ("dec", 17_644), ("dec", 17_645)])
def test_groupby_shared_table_sizes(ctx, val, groups):
    n = (1 << 22) - 1                                       # the exact key window
    rng = np.random.default_rng(groups)
    rows = np.empty((n, 2), dtype=np.int64)
    rows[:, 0] = rng.integers(0, groups, size=n) - 5
    rows[:groups, 0] = np.arange(groups) - 5
    if val == "dec":
        v = rng.uniform(0.5, 1.0, size=n) * np.where(rows[:, 0] % 2, 1e4, -1e4)
        v[::37] *= 1e-9
        v[::1001] = 0.0
        v[rows[:, 0] == 1] = 0.0                            # a group that adds nothing
        rows[:, 1] = v.view(np.int64)
        got = np.ascontiguousarray(ctx.groupby(rows, val=(8, "dec"))).view(np.int64).reshape(-1, 2)
        want = orc.groupby_exact(rows).view(np.int64).reshape(-1, 2)
        assert np.array_equal(got[np.argsort(got[:, 0], kind="stable")], want)
        return
    rows[:, 1] = rng.integers(-(1 << 62), 1 << 62, size=n)
    agg, vtype = ("count", "long") if val == "count" else ("sum", val)
    got = ctx.groupby(rows, val=(8, vtype), agg=agg)
    want = orc.groupby(rows, val=(8, vtype), agg=agg, hash=orc.hashcfg("modulo", 1024))
    assert np.array_equal(orc.canonical(got), orc.canonical(want))


# Tuples that are not 16 bytes load key and value apart.
@pytest.mark.parametrize("val", ["int", "long", "dec"])
@pytest.mark.parametrize("n", [1, 1023, 1025, 50_001])
def test_groupby_shared_table_24_byte_rows(ctx, n, val):
    a = dg.groupby_rows(n, 7, 1e4, dg.seed_for(211)) if val == "dec" else dg.uniform_keys(n, 7, dg.seed_for(211))
    rows = np.ascontiguousarray(np.concatenate([a, a[:, :1]], axis=1))
    got = np.ascontiguousarray(ctx.groupby(rows, val=(8, val)))
    if val == "dec":
        g = got.view(np.int64).reshape(-1, 2)
        assert np.array_equal(g[np.argsort(g[:, 0], kind="stable")], orc.groupby_exact(a).view(np.int64).reshape(-1, 2))
    else:
        assert np.array_equal(orc.canonical(got), orc.canonical(orc.groupby(rows, val=(8, val))))


# Join then group-by with each CTA's groups in shared memory, for as many as fit and
# flush fewer slots than there are probe tuples; the global table past that. Sizes
# around a block's 1024 tuples, and probe misses.
@pytest.mark.parametrize("probe,groups", [(1, 1), (1023, 5), (1025, 9), (3_000_000, 2163), (3_000_000, 2164),
                                          (3_000_000, 17_644), (3_000_000, 17_645), (3_000_000, 46_000)])
@pytest.mark.parametrize("swap", [False, True])
def test_hashjoin_groupby_shared_tables(ctx, probe, groups, swap):
    build = 2 * groups + 1
    rng = np.random.default_rng(probe + groups)
    R = np.stack([rng.permutation(build), np.arange(build) % groups + 40], axis=1).astype(np.int64)
    keys = rng.integers(-3, build + 3, size=probe)
    keys[0] = 0
    dec = rng.uniform(0.5, 1.0, size=probe) * np.where(keys % 2, 1e6, -1e6)
    dec[::41] *= 1e-12
    whole = rng.integers(-(1 << 62), 1 << 62, size=probe)
    group = np.full(build, -1, dtype=np.int64)
    group[R[:, 0]] = R[:, 1]
    hit = (keys >= 0) & (keys < build)
    for vtype, v in (("dec", dec.view(np.int64)), ("long", whole), ("int", whole), ("count", whole)):
        cols = [v, keys] if swap else [keys, v]
        S = np.ascontiguousarray(np.stack(cols, axis=1).astype(np.int64))
        pkey, val = ((8, 8), 0) if swap else ((0, 8), 8)
        joined = np.ascontiguousarray(np.stack([group[keys[hit]], v[hit]], axis=1))
        agg, t = ("count", "long") if vtype == "count" else ("sum", vtype)
        got = np.ascontiguousarray(ctx.hashjoin_groupby(R, S, pkey=pkey, val=(val, t), agg=agg))
        want = orc.groupby_exact(joined) if t == "dec" else orc.groupby(joined, val=(8, t), agg=agg)
        assert np.array_equal(orc.canonical(got), orc.canonical(want))


# Windows of up to 8192 keys are counted in shared memory when there are eight tuples
# for each of the blocks' counts and blocks for half the SMs. Either side of both limits,
# counted on either side, 16- and 24-byte tuples, and one key with most of the tuples.
@pytest.mark.parametrize("n,keys", [(620_000, 1), (600_000, 1000), (630_000, 1000), (5_100_000, 8192), (5_100_000, 8193)])
@pytest.mark.parametrize("width", [16, 24])
def test_mpsm_few_keys_counted_in_shared_memory(ctx, n, keys, width):
    rng = np.random.default_rng(keys)
    R = np.stack([rng.integers(0, keys, size=n) - 3] + [rng.integers(-(1 << 62), 1 << 62, size=n)] * (width // 8 - 1), axis=1)
    R[n // 3:n // 2, 0] = -3
    R[0, 0], R[-1, 0] = -3, keys - 4
    S = R[:: n // 700].copy()
    S[:5, 0] = keys - 3                                     # no match
    sums, rows = {}, np.bincount(R[:, 0] + 3, minlength=keys + 1)
    total = np.zeros(keys + 1, dtype=np.uint64)
    np.add.at(total, R[:, 0] + 3, R[:, 1].astype(np.uint64))
    k = S[:, 0] + 3
    want = int(rows[k].sum())
    sums["B"] = int(total[k].sum(dtype=np.uint64).astype(np.int64))
    sums["P"] = int((rows[k].astype(np.uint64) * S[:, 1].astype(np.uint64)).sum(dtype=np.uint64).astype(np.int64))
    for a, b, of in ((R, S, {0: "P", 1: "B"}), (S, R, {0: "B", 1: "P"})):
        for col in (0, 1):
            _, got, s = ctx.mpsm(a, b, proj=(("P", 8, 8), ("B", 8, 8)), flags=gpu.JOIN_COUNT | gpu.JOIN_SUM, sum_col=col)
            assert (got, s) == (want, sums[of[col]])


# A warp's probe tuples (64 or 128 of them) with more than 8192 rows in all are written in
# slices of 2048 rows by a second launch: one row either side of both, tuples of many
# rows among others, more rows than the output takes (counted, not written), and an
# output too small for any slice.
@pytest.mark.parametrize("dup", [1, 5])
@pytest.mark.parametrize("runs", [[8191], [8192], [8193], [10_240, 10_241], [16_384, 16_384, 3], [4000, 4193, 9000], [130] * 64])
def test_mpsm_slices_of_long_runs(ctx, runs, dup):
    rng = np.random.default_rng(sum(runs))
    others = 3000
    R = np.concatenate([np.full(x, i) for i, x in enumerate(runs)] + [np.repeat(np.arange(others) + len(runs), dup)])
    R = np.stack([R, rng.integers(0, 1 << 31, size=R.size)], axis=1).astype(np.int64)
    R = R[rng.permutation(R.shape[0])]
    S = np.concatenate([np.arange(len(runs)), rng.integers(len(runs), len(runs) + others + 5, size=500)])
    S = np.stack([S, np.arange(S.size)], axis=1).astype(np.int64)
    _mpsm(ctx, R, S)
    L, res, n = gpu.lib(), gpu.JoinResult(), 0
    dR, dS = ctx.upload(R), ctx.upload(S)
    rR, rS = ctx.rel(dR, R.shape[0], 16), ctx.rel(dS, S.shape[0], 16)
    c, nc = gpu.cols((("P", 8, 8), ("B", 8, 8)))
    full = int(np.bincount(R[:, 0], minlength=len(runs) + others + 5)[S[:, 0]].sum())
    for cap in (0, 100, 8192, 8193, full // 2, full - 1):
        if cap >= full:
            continue
        out = ctx.alloc(16 * (cap + 64))
        ctx._check(L.pg_memset(ctx.h, ctx.stream, out.ptr, 0xA5, 16 * (cap + 64)))
        rc = L.pg_mpsm_join(ctx.h, ctx.stream, ctypes.byref(rR), ctypes.byref(rS), c, nc, out.ptr, cap,
                            gpu.JOIN_MATERIALIZE, -1, ctypes.byref(res))
        assert rc == gpu.PG_ERR_OUTPUT_FULL and res.n_out == full
        assert (ctx.download(out, 16 * (cap + 64))[16 * cap:] == 0xA5).all()


# Flagged sides: the window comes from the counted side's ends, and a side confirmed
# sorted is not partitioned first. Flags that hold, that do not, and a side whose ends
# do not show that it is not sorted.
@pytest.mark.parametrize("n,m", [(50_001, 20_003), ((32 << 20) + 3, (8 << 20) + 5)])
@pytest.mark.parametrize("case", ["sorted", "build_only", "probe_only", "neither", "wide_inside"])
def test_mpsm_flagged_sides(ctx, n, m, case):
    rng = np.random.default_rng(n)
    keys = np.arange(n) * 2 - 9
    pick = np.sort(rng.integers(0, n, size=m))
    if case in ("probe_only", "neither"):
        keys = keys[rng.permutation(n)]
    if case in ("build_only", "neither"):
        pick = pick[rng.permutation(m)]
    if case == "wide_inside":
        keys[n // 2] = 1 << 45
    R = np.stack([keys, rng.integers(0, 1 << 20, size=n)], axis=1)
    S = np.stack([np.sort(keys)[pick] if case != "wide_inside" else keys[pick], np.arange(m)], axis=1)
    if case in ("build_only", "neither"):
        S[:, 0] = np.sort(keys)[pick]
    order = np.argsort(R[:, 0], kind="stable")
    want = R[order[np.searchsorted(R[order, 0], S[:, 0])], 1]
    flags = gpu.JOIN_BUILD_SORTED | gpu.JOIN_PROBE_SORTED
    proj = (("P", 8, 8), ("B", 8, 8))
    _, count, total = ctx.mpsm(R, S, proj=proj, flags=gpu.JOIN_COUNT | gpu.JOIN_SUM | flags, sum_col=1)
    assert (count, total) == (m, int(want.sum()))
    got, rows, _ = ctx.mpsm(R, S, proj=proj, flags=gpu.JOIN_MATERIALIZE | flags)
    got = np.ascontiguousarray(got).view(np.int64).reshape(-1, 2)
    seen = np.full(m, -1, dtype=np.int64)
    seen[got[:, 0]] = got[:, 1]
    assert rows == m and np.array_equal(seen, want)


# Tuples other than 16 bytes: radix passes over the tuples where the keys need few,
# over (key, row) records where they need more, and one launch up to 2^20 (wide tuples
# again by passes). Either side of each, and of the widths that the passes take.
@pytest.mark.parametrize("n,width,bits", [((1 << 20) + 1, 8, 30), ((1 << 20) + 1, 12, 32), ((1 << 20) + 1, 12, 33),
                                          ((1 << 20) + 1, 24, 24), ((1 << 20) + 1, 24, 25), ((1 << 20) + 1, 40, 16),
                                          ((1 << 20) + 1, 400, 8), ((1 << 20) + 1, 404, 8), (104_857, 400, 8), (104_858, 400, 8),
                                          (104_858, 400, 9), (209_716, 200, 16), (83_000, 512, 8), ((1 << 20) + 1, 24, 0)])
def test_sort_of_other_widths(ctx, n, width, bits):
    rng = np.random.default_rng(width * bits + n)
    rows = np.zeros((n, width // 4), dtype=np.int32)
    rows[:, -1] = np.arange(n)
    kb = 4 if width == 8 else 8
    keys = rng.integers(0, 1 << bits, size=n) - (1 << bits >> 1)
    keys[0], keys[1] = -(1 << bits >> 1), (1 << bits) - 1 - (1 << bits >> 1)
    rows[:, : kb // 4] = keys.astype(np.int64 if kb == 8 else np.int32).view(np.int32).reshape(n, -1)
    assert np.array_equal(ctx.sort(rows, (0, kb)), rows[np.argsort(keys, kind="stable")])


# Tuples over 240 bytes are filtered, and projections of at most a quarter of tuples over
# 128 bytes made, without staging: tiles of 512 rows. Either side of the widths, of the
# quarter and of a tile, rows of more units than a block has threads, bases that are and
# are not aligned to the copies' units.
@pytest.mark.parametrize("width", [132, 240, 244, 256, 400, 1000, 1024, 1028, 3000])
@pytest.mark.parametrize("shift", [(0, 0), (4, 0), (0, 8), (8, 8)])
def test_filter_and_project_of_wide_tuples(ctx, width, shift):
    L, (si, so) = gpu.lib(), shift
    quarter = width // 16 * 4
    for n in (1, 511, 512, 513, 5000):
        rows = _rows(n, width, width + n)
        src, dst = ctx.alloc(rows.nbytes + 64), ctx.alloc(rows.nbytes + 64)
        ctx._check(L.pg_h2d(ctx.h, ctx.stream, src.ptr + si, rows.ctypes.data, rows.nbytes))
        r = gpu.Rel(src.ptr + si, n, width, 0, 0)
        for limit in (0, 20, 500, 1000):
            pr, npr = gpu.preds([("int", "<", 0, limit)])
            m = ctypes.c_uint64()
            ctx._check(L.pg_memset(ctx.h, ctx.stream, dst.ptr, 0xA5, rows.nbytes + 64))
            ctx._check(L.pg_filter(ctx.h, ctx.stream, ctypes.byref(r), pr, npr, dst.ptr + so, ctypes.byref(m)))
            want = rows[rows[:, 0] < limit]
            got = ctx.download(dst, rows.nbytes + 64)
            assert m.value == len(want) and np.array_equal(got[so:so + want.nbytes], want.reshape(-1).view(np.uint8))
            assert (got[:so] == 0xA5).all() and (got[so + want.nbytes:] == 0xA5).all()
        for cols in ([(0, 4)], [(width - 8, 8)], [(4, quarter)], [(4, quarter - 4), (width - 8, 8)], [(0, min(width, 1016))] * 2):
            ow = sum(b for _, b in cols)
            if ow > width:
                cols, ow = cols[:1], cols[0][1]
            c = (gpu.Col * len(cols))(*[gpu.Col(0, o, b) for o, b in cols])
            ctx._check(L.pg_project(ctx.h, ctx.stream, ctypes.byref(r), c, len(cols), dst.ptr + so))
            want = np.concatenate([rows[:, o // 4:(o + b) // 4] for o, b in cols], axis=1)
            got = ctx.download(dst, rows.nbytes + 64)
            assert np.array_equal(got[so:so + want.nbytes], np.ascontiguousarray(want).reshape(-1).view(np.uint8))


# Either side of the lines between the two partitions of 16-byte tuples: few buckets,
# functions that cost more than the ranking.
@pytest.mark.parametrize("fn,kw,n", [("parammodulo", dict(buckets=1), 10_001), ("parammodulo", dict(buckets=2), 3_999_999),
                                     ("parammodulo", dict(buckets=2), 4_000_000), ("modulo", dict(buckets=4), 10_001), ("parammodulo", dict(buckets=1), 400_000),
                                     ("exactrange", dict(buckets=4, min=0, max=(1 << 40) - 1), 400_000),
                                     ("exactrange", dict(buckets=5, min=0, max=(1 << 40) - 1), 10_001),
                                     ("bytes", dict(buckets=4), 399_999), ("bytes", dict(buckets=4), 400_000), ("bytes", dict(buckets=8), 2_499_999),
                                     ("bytes", dict(buckets=8), 2_500_000), ("knuth", dict(buckets=256, skipbits=3), 10_001)])
def test_partition_rules(ctx, fn, kw, n):
    rows = dg.uniform_keys(n, 1 << 40, dg.seed_for(213))
    got, offs = ctx.partition(rows, gpu.hashcfg(fn, **kw))
    want, woffs = orc.partition(rows, orc.hashcfg(fn, **kw))
    assert np.array_equal(offs, woffs) and np.array_equal(got, want)


# Few words of unstaged tuples are projected a thread a row: few tuples, one word, and up
# to four words of tuples of 900 bytes and more; units a thread past each line.
@pytest.mark.parametrize("n,width,keep", [(199_999, 132, 16), (200_000, 132, 16), (200_000, 132, 4), (999_999, 132, 8),
                                          (1_000_000, 132, 8), (1_000_000, 200, 8), (1_000_000, 196, 8),
                                          (200_000, 896, 16), (200_000, 900, 16), (200_000, 900, 20), (1, 900, 4)])
def test_project_few_words(ctx, n, width, keep):
    rows = _rows(n, width, n + keep)
    got = ctx.project(rows, [(width - keep, keep)])
    assert np.array_equal(np.ascontiguousarray(got).view(np.int32).reshape(n, -1), rows[:, (width - keep) // 4:])
