"""Join tables whose first uses come from several threads at once: the order in
which a probe reads a table that another thread settles (on the host, with a fake
table), and probes of fresh tables of repeated keys from threads of their own."""
import ctypes
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

from pythia_gb300 import datagen as dg
from pythia_gb300 import gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_table_settled_between_two_reads_is_never_seen_settled_and_unique(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    so = str(tmp_path / "libtableview.so")
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "pythia_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "tableview_shim.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    for k in range(4):                          # before the first read .. after the last
        v = L.tableview_settled_before(k)
        spec, unique = bool(v & 1), bool(v & 2)
        assert spec or not unique, k            # repeated keys: unique only while the header checks it
        assert not spec or unique, k            # an unsettled table goes by its header


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["dense", "repeated", "far", "wide"])
def test_first_probes_from_several_threads(ctx, case):
    # Every build of 16-byte tuples is first used unsettled: four threads, each on a
    # stream of its own, count and sum a fresh table's matches at once.
    L, threads, n = gpu.lib(), 4, 3000
    R = dg.build_relation(n, dg.seed_for(301))
    S = dg.probe_uniform(2 * n, R, dg.seed_for(302))
    if case == "repeated":
        R[n // 2:, 0] = R[: n // 2, 0]
    elif case == "far":
        R[:, 0] *= -7046029254386353131
        S[:, 0] *= -7046029254386353131
    elif case == "wide":
        R[0, 1] = -5
    order = np.argsort(R[:, 0], kind="stable")
    keys, vals = R[order, 0], R[order, 1].astype(np.uint64)
    lo, hi = np.searchsorted(keys, S[:, 0], "left"), np.searchsorted(keys, S[:, 0], "right")
    pre = np.concatenate([np.zeros(1, np.uint64), np.cumsum(vals, dtype=np.uint64)])
    want = (int((hi - lo).sum()), int((pre[hi] - pre[lo]).sum(dtype=np.uint64).astype(np.int64)))
    dR, dS = ctx.upload(R), ctx.upload(S)
    rR, rS = ctx.rel(dR, n, 16), ctx.rel(dS, 2 * n, 16)
    c, nc = gpu.cols((("P", 8, 8), ("B", 8, 8)))
    streams = []
    for _ in range(threads):
        s = ctypes.c_void_p()
        ctx._check(L.pg_stream_create(ctx.h, ctypes.byref(s)))
        streams.append(s.value)
    bad = []
    gate, done = threading.Barrier(threads + 1), threading.Barrier(threads + 1)
    state = {"ht": None, "rounds": 300}

    def probe(k):
        for _ in range(state["rounds"]):
            gate.wait()
            res = gpu.JoinResult()
            rc = L.pg_hashjoin_probe(ctx.h, streams[k], state["ht"], ctypes.byref(rS), c, nc, None, 0,
                                     gpu.JOIN_COUNT | gpu.JOIN_SUM, 1, ctypes.byref(res))
            if rc or (res.n_out, res.sum) != want:
                bad.append((k, rc, res.n_out, res.sum))
            done.wait()

    workers = [threading.Thread(target=probe, args=(k,), daemon=True) for k in range(threads)]
    for t in workers:
        t.start()
    for _ in range(state["rounds"]):
        ht = ctypes.c_void_p()
        ctx._check(L.pg_hashjoin_build(ctx.h, ctx.stream, ctypes.byref(rR), c, nc, ctypes.byref(ht)))
        state["ht"] = ht.value
        gate.wait()
        done.wait()
        L.pg_hashtable_free(ctx.h, ht)
    for t in workers:
        t.join()
    for s in streams:
        L.pg_stream_destroy(ctx.h, s)
    assert not bad, bad[:5]


def _pool_bytes():
    """Bytes in use in the device's default memory pool."""
    rt = ctypes.CDLL("libcudart.so.13")
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0     # cudaMemPoolAttrUsedMemCurrent
    return used.value


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3000, 1 << 20])
def test_probed_dense_table_keeps_only_its_entries(ctx, n):
    # 2n + n/8 + 4096 entries of 4 bytes and the header; the build's spare hashed
    # slots (up to 32 bytes a tuple twice over) are gone after the second probe.
    R = dg.build_relation(n, dg.seed_for(303))
    S = dg.probe_uniform(1000, R, dg.seed_for(304))
    dR, dS = ctx.upload(R), ctx.upload(S)
    rR, rS = ctx.rel(dR, n, 16), ctx.rel(dS, 1000, 16)
    c, nc = gpu.cols((("P", 8, 8), ("B", 8, 8)))
    L, ht, res = gpu.lib(), ctypes.c_void_p(), gpu.JoinResult()
    ctx.sync()
    before = _pool_bytes()
    ctx._check(L.pg_hashjoin_build(ctx.h, ctx.stream, ctypes.byref(rR), c, nc, ctypes.byref(ht)))
    try:
        for _ in range(2):
            ctx._check(L.pg_hashjoin_probe(ctx.h, ctx.stream, ht, ctypes.byref(rS), c, nc, None, 0, gpu.JOIN_COUNT, -1,
                                           ctypes.byref(res)))
            assert res.n_out == 1000
        ctx.sync()
        kept = _pool_bytes() - before
        assert kept <= 4 * (2 * n + n // 8 + 4096) + 4096, kept
    finally:
        L.pg_hashtable_free(ctx.h, ht)


# Values that span 2^32 or more beside dense keys take 8-byte entries, made by the
# build kernel like the other layouts of up to 2^20 tuples: a join is the build, a
# probe that finds the header and one that finds the table. Sizes around one block's
# 2048 tuples and a word of presence bits.
@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 2048, 2049, 70_001, 1 << 20])
@pytest.mark.parametrize("repeated", [False, True])
def test_small_build_of_wide_values(ctx, n, repeated):
    R = np.stack([np.random.default_rng(n).permutation(n) - 5, np.arange(n) * 7 - 9], axis=1).astype(np.int64)
    R[0, 1], R[-1, 1] = np.iinfo(np.int64).min, np.iinfo(np.int64).max
    if repeated:
        if n == 1:
            return
        R[n // 2, 0] = R[0, 0]
    S = np.stack([np.arange(-9, n + 3), np.arange(n + 12)], axis=1).astype(np.int64)
    vals = {}
    for k, v in R.tolist():
        vals.setdefault(k, []).append(v)
    want = sorted((p, v) for k, p in S.tolist() for v in vals.get(k, ()))
    before = gpu.kernel_launches()
    t = ctx.build_table(R)
    try:
        _, count, total = t.probe(S, flags=gpu.JOIN_COUNT | gpu.JOIN_SUM, sum_col=1)
        assert repeated or gpu.kernel_launches() - before <= 5      # 7 with an exact rebuild
        assert count == len(want) and (total - sum(v for _, v in want)) % (1 << 64) == 0
        got = np.ascontiguousarray(t.probe(S, out_cap=len(want))[0]).view(np.int64).reshape(-1, 2)
        assert sorted(map(tuple, got.tolist())) == want
        if not repeated:                                            # the layout of the exact build
            image = t.serialize()
            ctx.tune(build_spec=2)
            try:
                u = ctx.build_table(R)
                assert np.array_equal(image, u.serialize())
                u.free()
            finally:
                ctx.tune(build_spec=0)
    finally:
        t.free()


# The tuples of a repeated key walk past each other. Over 2^18 tuples, a key that walks
# past a sixteenth of them sends the build to the exact build's kernel instead of holding
# blocks at a barrier, whose wait it could outlast. Without that the first probe makes three
# launches more than the next: the build, and a probe and its tail that find the header.
@pytest.mark.gpu
@pytest.mark.parametrize("n,copies,exact", [(100, 100, False), (9000, 9000, False), (270_000, 8000, False), (270_000, 20_000, True)])
def test_small_build_of_long_walks(ctx, n, copies, exact):
    R = np.stack([np.maximum(np.arange(n), copies), np.arange(n)], axis=1).astype(np.int64)
    R[: copies, 0] = copies
    S = np.stack([np.arange(copies - 1, n + 2), np.zeros(n + 3 - copies)], axis=1).astype(np.int64)
    before = gpu.kernel_launches()
    t = ctx.build_table(R)
    try:
        launches = []
        for _ in range(2):
            _, count, total = t.probe(S, flags=gpu.JOIN_COUNT | gpu.JOIN_SUM, sum_col=1)
            assert (count, total) == (n, n * (n - 1) // 2)
            launches.append(gpu.kernel_launches() - before)
            before += launches[-1]
        assert (launches[0] - launches[1] > 3) == exact
    finally:
        t.free()
