"""Calls whose scratch cannot be allocated. A process of its own loads an allocator
(tests/native/failalloc.c) that fails one chosen pool allocation, and makes the same
call with each of its allocations failing in turn. Whatever happens, no allocation may
stay out afterwards; a call that has a way to do without its larger tables must
take it and give the same result."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu

COMMON = """
import ctypes, sys
import numpy as np
sys.path.insert(0, %r)
from pythia_gb300 import datagen as dg, gpu
F = ctypes.CDLL(None)
F.failalloc_next.argtypes, F.failalloc_next.restype = [ctypes.c_long], None
F.failalloc_failed_bytes.restype = ctypes.c_long
ctx, L, ref = gpu.Context(0), gpu.lib(), ctypes.byref

def each_failing(call, check, must_do_without):
    # `call` returns a code; `check` its result. Allocations of `must_do_without` bytes
    # and more have to be done without.
    assert call() == 0 and check()
    for k in range(200):
        before = F.failalloc_out()
        F.failalloc_next(k)
        rc = call()
        bytes = F.failalloc_failed_bytes()
        F.failalloc_next(-1)
        assert F.failalloc_out() == before, (k, bytes, rc, F.failalloc_out() - before)
        if bytes == 0:
            assert rc == 0 and check()
            print("allocations:", k)
            return
        assert rc in (0, gpu.PG_ERR_OOM), (k, bytes, rc)
        if bytes >= must_do_without:
            assert rc == 0, (k, bytes)
        if rc == 0:
            assert check(), (k, bytes)
        assert call() == 0 and check()                      # and the next call is unharmed
    raise AssertionError("never ran out of allocations")
"""

MPSM = COMMON + """
n, m = %d, %d
rng = np.random.default_rng(n)
R = np.stack([rng.permutation(n) * 3, rng.integers(0, %d, size=n)], axis=1).astype(np.int64)
S = np.stack([rng.integers(0, n, size=m) * 3, np.arange(m)], axis=1).astype(np.int64)
val = np.empty(3 * n, dtype=np.int64)
val[R[:, 0]] = R[:, 1]
want = val[S[:, 0]]
dR, dS, dO = ctx.upload(R), ctx.upload(S), ctx.alloc(16 * m)
rR, rS = ctx.rel(dR, n, 16), ctx.rel(dS, m, 16)
c, nc = gpu.cols((("P", 8, 8), ("B", 8, 8)))
res = gpu.JoinResult()

def rows():
    return L.pg_mpsm_join(ctx.h, ctx.stream, ref(rR), ref(rS), c, nc, dO.ptr, m, gpu.JOIN_MATERIALIZE, -1, ref(res))

def rows_right():
    got = ctx.download(dO, 16 * m).view(np.int64).reshape(-1, 2)
    seen = np.full(m, -1, dtype=np.int64)
    seen[got[:, 0]] = got[:, 1]
    return res.n_out == m and np.array_equal(seen, want)

def agg():
    return L.pg_mpsm_join(ctx.h, ctx.stream, ref(rR), ref(rS), c, nc, None, 0, gpu.JOIN_COUNT | gpu.JOIN_SUM, 1, ref(res))

def agg_right():
    return res.n_out == m and res.sum == int(want.sum())

F.failalloc_next(0)
rows()
assert F.failalloc_failed_bytes() > 0                       # the allocator is the one in use
F.failalloc_next(-1)
each_failing(rows, rows_right, 1 << 14)
each_failing(agg, agg_right, 1 << 14)
"""


def _run(tmp_path, source):
    cc = shutil.which("gcc")
    if not cc:
        pytest.skip("no host C compiler")
    so = str(tmp_path / "failalloc.so")
    subprocess.run([cc, "-O1", "-shared", "-fPIC", os.path.join(ROOT, "tests", "native", "failalloc.c"), "-o", so,
                    "-ldl", "-lpthread"], check=True)
    r = subprocess.run([sys.executable, "-c", source], env=dict(os.environ, LD_PRELOAD=so), cwd=ROOT, timeout=500,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


# The second size partitions both sides first.
@pytest.mark.parametrize("n,m", [(100_003, 50_001), ((32 << 20) + 5, (8 << 20) + 3)])
def test_counted_merge_join(tmp_path, n, m):
    _run(tmp_path, MPSM % (ROOT, n, m, 1 << 31))


SORT = COMMON + """
n, width, bits = %d, %d, %d
rng = np.random.default_rng(n)
rows = rng.integers(0, 1 << 30, size=(n, width // 4)).astype(np.int32)
keys = rng.integers(0, 1 << bits, size=n)
rows[:, :2] = keys.astype(np.int64).view(np.int32).reshape(n, 2)
want = rows[np.argsort(keys, kind="stable")]
dI, dO = ctx.upload(rows), ctx.alloc(rows.nbytes)
r = ctx.rel(dI, n, width)

def call():
    return L.pg_sort_pages(ctx.h, ctx.stream, ref(r), dO.ptr)

def right():
    return np.array_equal(ctx.download(dO, rows.nbytes).view(np.int32).reshape(n, -1), want)

each_failing(call, right, 16 * n)
"""


# One launch of records, passes over the tuples (few digits) and over records (many).
@pytest.mark.parametrize("n,width,bits", [(50_000, 24, 20), ((1 << 20) + 77, 24, 16), ((1 << 20) + 77, 24, 40),
                                          ((1 << 20) + 77, 8, 20)])
def test_sort_of_other_widths(tmp_path, n, width, bits):
    if width == 8:
        source = SORT.replace("rows[:, :2]", "rows")
    else:
        source = SORT
    _run(tmp_path, source % (ROOT, n, width, bits))


# Keys that span too much to be counted: the sort's own scratch.
def test_sorted_merge_join(tmp_path):
    source = (MPSM % (ROOT, 30_001, 20_001, 1 << 31)).replace("dR, dS, dO =", "R[:, 0] <<= 30\nS[:, 0] <<= 30\ndR, dS, dO =")
    _run(tmp_path, source.replace("1 << 14)", "1 << 40)"))
