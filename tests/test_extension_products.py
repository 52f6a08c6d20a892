"""The extension-field products every kernel uses (loom_b200/csrc/field.cuh),
built with g++ for the host and compared with Python integers where their
unreduced sums are largest.  No GPU needed."""
import ctypes
import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

from loom_b200 import field as F

P = F.P
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r'''
#include "field.cuh"
extern "C" void f_mul6(const uint32_t* a, const uint32_t* b, uint32_t* r) {
  lg::E6 x, y;
  for (int i = 0; i < 6; i++) { x.c[i] = a[i]; y.c[i] = b[i]; }
  x = lg::e6_mul(x, y);
  for (int i = 0; i < 6; i++) r[i] = x.c[i];
}
extern "C" void f_inv6(const uint32_t* a, const uint32_t*, uint32_t* r) {
  lg::E6 x;
  for (int i = 0; i < 6; i++) x.c[i] = a[i];
  x = lg::e6_inv(x);
  for (int i = 0; i < 6; i++) r[i] = x.c[i];
}
extern "C" void f_mul2(const uint32_t* a, const uint32_t* b, uint32_t* r) {
  const lg::E2 v = lg::e2_mul(lg::E2{a[0], a[1]}, lg::E2{b[0], b[1]});
  r[0] = v.a0; r[1] = v.a1; r[2] = r[3] = r[4] = r[5] = 0;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("ext")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "loom_b200", "csrc"),
                    str(d / "shim.cpp"), "-o", str(d / "libext.so")], check=True)
    return ctypes.CDLL(str(d / "libext.so"))


def call(f, a, b):
    u = ctypes.c_uint32 * 6
    r = u()
    f(u(*a), u(*b), r)
    return list(r)


def e2(a, b):
    return [(a[0] * b[0] + 3 * a[1] * b[1]) % P, (a[0] * b[1] + a[1] * b[0]) % P]


def e6(x, y):
    c = [[0, 0] for _ in range(5)]
    for i, j in itertools.product(range(3), range(3)):
        t = e2(x[2 * i:2 * i + 2], y[2 * j:2 * j + 2])
        c[i + j] = [(p + q) % P for p, q in zip(c[i + j], t)]
    for k in (3, 4):
        t = e2(c[k], (1, 1))
        c[k - 3] = [(p + q) % P for p, q in zip(c[k - 3], t)]
    return c[0] + c[1] + c[2]


def operands():
    rng = np.random.default_rng(3)
    out = [[P - 1] * 6, [0] * 6, [1] * 6, [P - 1, 0, P - 1, 0, P - 1, 0], [(P + 1) // 2] * 6, [(P - 1) // 3] * 6]
    out += [[P - 1 if k == i else 0 for k in range(6)] for i in range(6)]
    return out + [[int(v) for v in rng.integers(0, P, 6)] for _ in range(20)]


def test_products_and_inverses(lib):
    ops = operands()
    for a, b in itertools.product(ops, ops):
        assert call(lib.f_mul6, a, b) == [v * F.R_INV % P for v in e6(a, b)], (a, b)
        assert call(lib.f_mul2, a, b)[:2] == [v * F.R_INV % P for v in e2(a, b)], (a, b)
    one = [pow(2, 32, P)] + [0] * 5
    for a in ops:
        want = one if any(a) else [0] * 6
        assert call(lib.f_mul6, a, call(lib.f_inv6, a, a)) == want, a
