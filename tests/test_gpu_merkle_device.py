"""lg_merkle_root on device buffers: leaves and injections as the caller holds
them, the injections read in place where they are aligned."""
import ctypes

import numpy as np
import pytest

import oracle
from loom_b200 import field as F

pytestmark = pytest.mark.gpu


def rnd(shape, seed):
    return F.to_mont(np.random.Generator(np.random.PCG64(seed)).integers(0, F.P, shape, dtype=np.uint64).astype(np.uint32))


@pytest.mark.parametrize("log_leaves,widths", [(0, [0]), (3, []), (5, [5, 5, 2]), (9, [9, 8, 8, 0]), (12, [12, 3]),
                                               (14, [14, 13, 13, 5])])
@pytest.mark.parametrize("off_leaves,off_inj", [(0, 0), (1, 0), (0, 4), (0, 3), (5, 2)])
def test_device_digests(ctx, log_leaves, widths, off_leaves, off_inj):
    import torch
    leaves = rnd((1 << log_leaves, 8), log_leaves)
    inj = [rnd((1 << w, 8), 100 + k) for k, w in enumerate(widths)]

    def put(parts, off):
        flat = np.concatenate([a.reshape(-1) for a in parts]) if parts else np.zeros(8, dtype=np.uint32)
        t = torch.zeros(flat.size + off, dtype=torch.int32, device="cuda:0")
        t[off:].copy_(torch.from_numpy(flat.view(np.int32)))
        return t, ctypes.c_void_p(t.data_ptr() + 4 * off)

    (a, pa), (b, pb) = put([leaves], off_leaves), put(inj, off_inj)
    before = a.clone(), b.clone()
    torch.cuda.synchronize()
    w = np.array([1 << x for x in widths] or [1], dtype=np.uint64)
    root = np.zeros(8, dtype=np.uint32)
    ctx._check(ctx.L.lg_merkle_root(ctx.h, pa, 1 << log_leaves, len(widths),
                                    w.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)), pb, 1,
                                    root.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32))))
    assert np.array_equal(root, oracle.merkle_root(leaves, inj))
    assert torch.equal(a, before[0]) and torch.equal(b, before[1])  # only read
