"""lg_rs_encode on device buffers: encoded in place where input and output are
apart and the output is aligned, through staged copies otherwise; the sizes it
refuses."""
import ctypes

import numpy as np
import pytest

import oracle
from loom_b200 import _lib, field as F

pytestmark = pytest.mark.gpu


def rnd(shape, seed):
    return F.to_mont(np.random.Generator(np.random.PCG64(seed)).integers(0, F.P, shape, dtype=np.uint64).astype(np.uint32))


def words(n):
    import torch
    t = torch.zeros(n + 16, dtype=torch.int32, device="cuda:0")
    torch.cuda.synchronize()
    return t


def put(t, at, a):
    import torch
    t[at:at + a.size].copy_(torch.from_numpy(np.ascontiguousarray(a).reshape(-1).view(np.int32)))
    torch.cuda.synchronize()


def get(t, at, n):
    return t[at:at + n].cpu().numpy().view(np.uint32)


def p(t, at=0):
    return ctypes.c_void_p(t.data_ptr() + 4 * at)


# both sides of each change of transform: radix-2 stages, one block a column,
# the large transforms' splits, and a batch of more than one chunk of them
@pytest.mark.parametrize("logn,cols", [(1, 3), (3, 2), (4, 5), (9, 3), (11, 2), (13, 3), (14, 2), (15, 3), (16, 2), (17, 1),
                                       (18, 17)])
@pytest.mark.parametrize("off_in,off_out", [(0, 0), (1, 0), (0, 3), (2, 4)])
def test_device_columns(ctx, logn, cols, off_in, off_out):
    n = 1 << logn
    a = rnd((cols, n), logn)
    src, dst = words(cols * n), words(4 * cols * n)
    put(src, off_in, a)
    ctx._check(ctx.L.lg_rs_encode(ctx.h, p(src, off_in), n, cols, p(dst, off_out), 1))
    got = get(dst, off_out, 4 * cols * n).reshape(cols, 4 * n)
    for i in range(0, cols, 4):
        assert np.array_equal(got[i], oracle.rs_encode(a[i], 4 * n)), i
    assert np.array_equal(got, ctx.rs_encode(a))
    assert np.array_equal(get(src, off_in, cols * n).reshape(cols, n), a)  # only read
    assert not get(dst, 0, off_out).any() and not get(dst, off_out + 4 * cols * n, 16 - off_out).any()


@pytest.mark.parametrize("logn", [3, 12, 15])
@pytest.mark.parametrize("at", [0, 1, 3])
def test_output_over_its_input(ctx, logn, at):
    """`in` at the front or inside of `out`: staged."""
    n, cols = 1 << logn, 3
    a, t = rnd((cols, n), 50 + logn), words(4 * cols * n)
    put(t, at * n, a)
    ctx._check(ctx.L.lg_rs_encode(ctx.h, p(t, at * n), n, cols, p(t), 1))
    assert np.array_equal(get(t, 0, 4 * cols * n).reshape(cols, 4 * n), ctx.rs_encode(a))


@pytest.mark.parametrize("cols", [0, 1])
def test_refused_sizes(ctx, cols):
    """More than 2^22 rows: refused before anything is read, columns or not."""
    t = words(64)
    for n in (1 << 23, 1 << 40):
        assert ctx.L.lg_rs_encode(ctx.h, p(t), n, cols, p(t, 16), 1) == _lib.LG_ERR_UNSUPPORTED
    for n in (0, 1, 3, 24):
        assert ctx.L.lg_rs_encode(ctx.h, p(t), n, cols, p(t, 16), 1) == _lib.LG_ERR_INVALID
