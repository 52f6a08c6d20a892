"""DEEP quotients from host memory, whose weighted values are summed on the
host up to 256 columns, against the oracle and against the same call on device buffers."""
import ctypes

import numpy as np
import pytest

import oracle
from loom_b200 import field as F

pytestmark = pytest.mark.gpu


def rnd(shape, seed):
    return F.to_mont(np.random.Generator(np.random.PCG64(seed)).integers(0, F.P, shape, dtype=np.uint64).astype(np.uint32))


@pytest.mark.parametrize("logr,cols", [(1, 1), (2, 3), (3, 4), (6, 5), (9, 65), (3, 256), (3, 257), (4, 300)])
def test_host_equals_oracle_and_device(ctx, logr, cols):
    import torch
    rows = 1 << logr
    lde, values, alpha, z = rnd((cols, rows), logr), rnd((cols, 6), 70 + cols), rnd(6, 71), rnd(6, 72)
    got = ctx.deep_quotient(lde, alpha, z, values)
    assert np.array_equal(got, oracle.deep_quotient(lde, alpha, z, values))
    d = [torch.from_numpy(a.view(np.int32)).cuda() for a in (lde, values)] + [torch.zeros(rows, 6, dtype=torch.int32).cuda()]
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr()) for t in d]
    u = [np.ascontiguousarray(a).ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)) for a in (alpha, z)]
    ctx._check(ctx.L.lg_deep_quotient(ctx.h, p[0], cols, rows, u[0], u[1], p[1], p[2], 1))
    assert np.array_equal(d[2].cpu().numpy().view(np.uint32), got)
