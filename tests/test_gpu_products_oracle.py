"""Both grand products against the oracle, which shares no code with them, on
both sides of each change of tile shape (2^16 and 2^18 rows) and of the separate
prefix launch (2^21 rows): rows aligned to 8 bytes or not, output over the
numerators, a zero denominator."""
import ctypes
import functools

import numpy as np
import pytest

import oracle
from loom_b200 import _lib, field as F

pytestmark = pytest.mark.gpu
SIZES = [1, 1000, 65536, 65537, 262144, 262145, (1 << 21) + 1]


@functools.lru_cache(maxsize=None)
def case(n, zero):
    rng = np.random.Generator(np.random.PCG64(n))
    num, den = (F.to_mont(rng.integers(0, F.P, (n, 6), dtype=np.uint64).astype(np.uint32)) for _ in range(2))
    want = oracle.grand_product(num, den)
    if zero:  # a ratio is 0 where its denominator is: the rows after it too
        z = n // 2
        want[z + 1:] = 0
        den[z] = 0
    return num, den, want


def run(ctx, n, zero, offset, over, call):
    import torch
    num, den, want = case(n, zero)

    def put(a):
        t = torch.zeros(6 * n + offset, dtype=torch.int32, device="cuda:0")
        t[offset:].copy_(torch.from_numpy(a.reshape(-1).view(np.int32)))
        return t

    a, b = put(num), put(den)
    out = a if over else torch.zeros_like(a)
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr() + 4 * offset) for t in (a, b, out)]
    call(ctx, p, n)
    torch.cuda.synchronize()
    assert np.array_equal(out[offset:].cpu().numpy().view(np.uint32).reshape(n, 6), want)


def product(ctx, p, n):
    ctx._check(ctx.L.lg_grand_product(ctx.h, p[0], p[1], n, p[2], 1))


def product_noalloc(ctx, p, n):
    import torch
    s = torch.cuda.Stream(device=0)
    assert ctx.L.lg_grand_product_noalloc(p[0], p[1], n, p[2], ctypes.c_void_p(s.cuda_stream)) == _lib.LG_OK
    s.synchronize()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("zero", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("over", [False, True])
@pytest.mark.parametrize("call", [product, product_noalloc])
def test_product(ctx, n, zero, offset, over, call):
    run(ctx, n, zero, offset, over, call)
