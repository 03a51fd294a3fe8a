"""The shared-memory adds of the hashed group-by's dec sums and 64-bit words, made of
32-bit adds (pythia_gb300/csrc/pg_fixsum.h), checked on the host against exact integers:
the carry out of every 64-bit add, and the chained words' total whatever the signs,
scales and order of the values."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U64 = ctypes.c_uint64
M64 = (1 << 64) - 1


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    so = str(tmp_path_factory.mktemp("fxh") / "libfxhalves.so")
    subprocess.run([cxx, "-O2", "-fno-strict-aliasing", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "pythia_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "fixsum_halves_shim.cpp"), "-o", so], check=True)
    L = ctypes.CDLL(so)
    L.fx_add_halves.argtypes, L.fx_add_halves.restype = [ctypes.POINTER(ctypes.c_uint32), U64], ctypes.c_uint32
    L.fx_chain_add_halves.argtypes = [ctypes.POINTER(U64), U64, ctypes.POINTER(U64)]
    L.fx_chain_count.argtypes = [ctypes.POINTER(U64), U64, ctypes.POINTER(U64)]
    return L


def test_the_carry_out_of_64_bits(fx):
    edges = [0, 1, 2, (1 << 31), (1 << 32) - 1, 1 << 32, (1 << 32) + 1, (1 << 63) - 1, 1 << 63, M64 - (1 << 32), M64 - 1, M64]
    rng = np.random.default_rng(21)
    edges += [int(x) for x in rng.integers(0, 1 << 63, size=60)]
    for a in edges:
        for b in edges:
            q = (ctypes.c_uint32 * 2)(a & 0xFFFFFFFF, a >> 32)
            carry = fx.fx_add_halves(q, b)
            assert (q[0] | (q[1] << 32)) == (a + b) & M64 and carry == (a + b) >> 64, (a, b)


def test_chained_words_hold_the_exact_sum(fx):
    rng = np.random.default_rng(22)
    top = 1 << 188
    for trial in range(40):
        n, stride = int(rng.integers(1, 2000)), int(rng.integers(1, 5))
        kind = trial % 4
        if kind == 0:                                     # near the bound, one sign: the upper word overflows
            vs = [top - 1 - int(rng.integers(0, 1 << 62)) for _ in range(n)]
        elif kind == 1:
            vs = [-(top - 1 - int(rng.integers(0, 1 << 62))) for _ in range(n)]
        elif kind == 2:                                   # near the bound, both signs
            vs = [(top - 1 - int(rng.integers(0, 1 << 62))) * (1 if rng.random() < 0.5 else -1) for _ in range(n)]
        else:                                             # every scale: carries between the words
            vs = [int(rng.integers(0, 1 << 62)) << int(rng.integers(0, 126)) for _ in range(n)]
            vs = [v if rng.random() < 0.6 else -v for v in vs]
        for order in range(2):
            t, w = (U64 * (4 * stride))(), (U64 * 4)()
            for v in (vs if order == 0 else [vs[i] for i in rng.permutation(n)]):
                u = v & ((1 << 192) - 1)
                fx.fx_chain_add_halves(t, stride, (U64 * 3)(u & M64, (u >> 64) & M64, u >> 128))
            fx.fx_chain_count(t, stride, w)
            got = sum(int(w[k]) << (64 * k) for k in range(4))
            assert (got - (1 << 256) if got >> 255 else got) == sum(vs), (trial, order)
            assert all(t[i] == 0 for i in range(4 * stride) if i % stride)      # the other slots
