"""Entry points that read and write the caller's device rows in place: the same
values from aligned and unaligned buffers, and from buffers that overlap
(which take the staged copy), as from host memory."""
import ctypes

import numpy as np
import pytest

import oracle
from loom_b200 import field as F

pytestmark = pytest.mark.gpu


def rnd(shape, seed):
    return F.to_mont(np.random.Generator(np.random.PCG64(seed)).integers(0, F.P, shape, dtype=np.uint64).astype(np.uint32))


class Rows:
    """A device buffer of words with room for an offset of a few words."""

    def __init__(self, words, data=None, offset=0):
        import torch
        self.t = torch.zeros(words + 8, dtype=torch.int32, device="cuda:0")
        self.v = self.t[offset:offset + words]
        if data is not None:
            self.v.copy_(torch.from_numpy(np.ascontiguousarray(data).reshape(-1).view(np.int32)))
        torch.cuda.synchronize()

    def ptr(self, word=0):
        return ctypes.c_void_p(self.v.data_ptr() + 4 * word)

    def get(self, shape, word=0):
        n = int(np.prod(shape))
        return self.v[word:word + n].cpu().numpy().view(np.uint32).reshape(shape)


def u32(a):
    return np.ascontiguousarray(a).ctypes.data_as(ctypes.POINTER(ctypes.c_uint32))


@pytest.mark.parametrize("logn", [1, 2, 9, 12, 13])
@pytest.mark.parametrize("off_in,off_out", [(0, 0), (4, 2), (1, 0), (0, 3)])
def test_fold_rows(ctx, logn, off_in, off_out):
    n, layer, alpha = 1 << logn, rnd((1 << logn, 6), logn), rnd(6, 3)
    src, dst = Rows(6 * n, layer, off_in), Rows(3 * n, offset=off_out)
    ctx._check(ctx.L.lg_fri_fold(ctx.h, src.ptr(), n, u32(alpha), dst.ptr(), 1))
    want = oracle.fri_fold(layer, alpha)
    assert np.array_equal(dst.get((n // 2, 6)), want)
    # over its own input
    ctx._check(ctx.L.lg_fri_fold(ctx.h, src.ptr(), n, u32(alpha), src.ptr(), 1))
    assert np.array_equal(src.get((n // 2, 6)), want)
