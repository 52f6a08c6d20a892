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


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1025, 65536, 65537, 262145])
@pytest.mark.parametrize("offset", [0, 1])
def test_grand_product_rows(ctx, n, offset):
    """Tile shapes change at 2^16 and 2^18 rows; `out` may be `num` itself."""
    num, den = rnd((n, 6), 7 + n), rnd((n, 6), 8 + n)
    want = oracle.grand_product(num, den)
    a, b, out = Rows(6 * n, num, offset), Rows(6 * n, den, offset), Rows(6 * n, offset=offset)
    ctx._check(ctx.L.lg_grand_product(ctx.h, a.ptr(), b.ptr(), n, out.ptr(), 1))
    assert np.array_equal(out.get((n, 6)), want)
    ctx._check(ctx.L.lg_grand_product(ctx.h, a.ptr(), b.ptr(), n, a.ptr(), 1))
    assert np.array_equal(a.get((n, 6)), want)


def test_grand_product_rows_that_overlap(ctx):
    """`out` shifted by rows against `num`: through the staged copy."""
    n, shift = 3000, 5
    num, den = rnd((n, 6), 1), rnd((n, 6), 2)
    a, b = Rows(6 * (n + shift), np.concatenate([num, num[:shift]])), Rows(6 * n, den)
    ctx._check(ctx.L.lg_grand_product(ctx.h, a.ptr(), b.ptr(), n, a.ptr(6 * shift), 1))
    assert np.array_equal(a.get((n, 6), 6 * shift), oracle.grand_product(num, den))


@pytest.mark.parametrize("n,zero", [(300, 0), (300, 299), (70000, 40000), (300000, 123457)])
def test_grand_product_with_a_zero_denominator(ctx, n, zero):
    """A zero denominator makes its ratio zero (as an inversion of zero gives
    zero), whatever rows share its inversion: the rows before it are those of
    the product without it, the rows after it zero."""
    num, den = rnd((n, 6), 3), rnd((n, 6), 4)
    want = oracle.grand_product(num, den)
    want[zero + 1:] = 0
    den[zero] = 0
    assert np.array_equal(ctx.grand_product(num, den), want)


@pytest.mark.parametrize("logr,cols", [(1, 3), (2, 1), (3, 4), (9, 5), (10, 65), (12, 130)])
@pytest.mark.parametrize("offset", [0, 2, 1])
def test_deep_quotient_rows(ctx, logr, cols, offset):
    rows = 1 << logr
    lde, values, alpha, z = rnd((cols, rows), logr), rnd((cols, 6), 60 + cols), rnd(6, 61), rnd(6, 62)
    want = ctx.deep_quotient(lde, alpha, z, values)  # host memory, aligned
    x, v, out = Rows(cols * rows, lde, offset), Rows(6 * cols, values, offset), Rows(6 * rows, offset=offset)
    ctx._check(ctx.L.lg_deep_quotient(ctx.h, x.ptr(), cols, rows, u32(alpha), u32(z), v.ptr(), out.ptr(), 1))
    assert np.array_equal(out.get((rows, 6)), want)
    if cols >= 6:  # over its own columns
        ctx._check(ctx.L.lg_deep_quotient(ctx.h, x.ptr(), cols, rows, u32(alpha), u32(z), v.ptr(), x.ptr(), 1))
        assert np.array_equal(x.get((rows, 6)), want)


def test_deep_quotient_at_a_row_of_the_domain(ctx):
    """z on the domain: that row's denominator is zero and its quotient 0."""
    rows, cols = 16, 3
    lde, values, alpha = rnd((cols, rows), 1), rnd((cols, 6), 2), rnd(6, 3)
    w, row = F.root_of_unity(rows), 6
    z = np.zeros(6, dtype=np.uint32)
    z[0] = pow(w, int(f"{row:04b}"[::-1], 2), F.P)
    got = ctx.deep_quotient(lde, alpha, F.to_mont(z), values)
    assert not got[row].any() and got[[r for r in range(rows) if r != row]].any(axis=1).all()


@pytest.mark.parametrize("shape,offset", [([(1 << 9, 3, 1), (1 << 5, 1, 2)], 0), ([(2, 1, 0), (2, 0, 1)], 1),
                                          ([(1 << 10, 1, 1), (1 << 10, 2, 0), (1 << 15, 1, 0)], 1)])
def test_commit_of_device_columns(ctx, shape, offset):
    """Columns on the device, aligned or not, against the same columns on the
    host; they are left as they were."""
    groups, bufs, data = [], [], []
    for gi, (n, nb, ne) in enumerate(shape):
        base, ext = [rnd(n, 10 * gi + k) for k in range(nb)], [rnd((n, 6), 10 * gi + 5 + k) for k in range(ne)]
        groups.append({"rows": n, "base": base, "ext": ext})
        data += base + ext
        bufs += [Rows(c.size, c, offset) for c in base + ext]
    ptrs = (ctypes.c_void_p * len(bufs))(*[b.ptr().value for b in bufs])
    rows = np.array([s[0] for s in shape], dtype=np.uint64)
    nb, ne = (np.array([s[k] for s in shape], dtype=np.uint32) for k in (1, 2))
    root = np.zeros(8, dtype=np.uint32)
    ctx._check(ctx.L.lg_commit_root(ctx.h, len(shape), rows.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), u32(nb),
                                    u32(ne), ptrs, 1, u32(root)))
    assert np.array_equal(root, ctx.commit_root(groups))
    for b, c in zip(bufs, data):
        assert np.array_equal(b.get(c.shape), c)
