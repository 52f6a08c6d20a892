"""The field products every kernel uses (loom_b200/csrc/field.cuh), built with
g++ for the host and compared with Python integers at the edges of their
input ranges.  No GPU needed."""
import ctypes
import os
import shutil
import subprocess

import pytest

from loom_b200 import field as F

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r'''
#include "field.cuh"
extern "C" uint32_t f_mul(uint32_t a, uint32_t b) { return lg::mul(a, b); }
extern "C" uint32_t f_mul_lazy(uint32_t a, uint32_t b) { return lg::mul_lazy(a, b); }
'''
EDGES = [0, 1, 2, F.P // 2, F.P - 1, F.P, F.P + 1, 2 * F.P - 1, (1 << 31) - 1, 1 << 31, (1 << 32) - 1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("field")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "loom_b200", "csrc"),
                    str(d / "shim.cpp"), "-o", str(d / "libfield.so")], check=True)
    L = ctypes.CDLL(str(d / "libfield.so"))
    for f in (L.f_mul, L.f_mul_lazy):
        f.argtypes, f.restype = [ctypes.c_uint32, ctypes.c_uint32], ctypes.c_uint32
    return L


@pytest.mark.parametrize("a", EDGES)
def test_montgomery_products_at_the_edges(lib, a):
    """mul: a anywhere in a word, b below p, result canonical; mul_lazy: the
    same product below 2p."""
    for b in [e for e in EDGES if e < F.P] + [0x12345678, 0x7ABCDEF0 % F.P]:
        want = a * b * F.R_INV % F.P
        assert lib.f_mul(a, b) == want, (a, b)
        lazy = lib.f_mul_lazy(a, b)
        assert lazy < 2 * F.P and lazy % F.P == want, (a, b)
