"""Calls that fail part way: nothing of them runs on after the return, and the
context takes the next call."""
import ctypes
import time

import numpy as np
import pytest

import oracle
from loom_b200 import Context, LoomError, _lib, field as F

pytestmark = pytest.mark.gpu


def dev(words, seed):
    import torch
    g = torch.Generator(device="cuda:0").manual_seed(seed)
    t = torch.randint(0, F.P, (words,), dtype=torch.int32, device="cuda:0", generator=g)
    torch.cuda.synchronize()
    return t


def p(t, word=0):
    return ctypes.c_void_p(t.data_ptr() + 4 * word)


def encode(ctx, src, n, cols, dst):
    ctx._check(ctx.L.lg_rs_encode(ctx.h, p(src), n, cols, p(dst), 1))


def test_a_failed_call_leaves_nothing_running():
    """The transforms of a commitment are queued, then its tree exceeds the
    context's budget: the device is idle when the call returns (a fifth of the
    transforms' time is far above a wait for an idle device)."""
    import torch
    n, cols = 1 << 20, 24
    src, dst = dev(cols * n, 1), torch.empty(4 * cols * n, dtype=torch.int32, device="cuda:0")
    roomy = Context(0)
    encode(roomy, src, n, cols, dst)
    t0 = time.perf_counter()
    encode(roomy, src, n, cols, dst)
    transforms = time.perf_counter() - t0
    roomy.close()
    # LDE, coefficients and twiddles fit; a byte short of the tree's digests
    tree = 64 << 21
    ctx = Context(0, hbm_budget=20 * cols * n + 16 * n + tree - 1)
    u32p, u64p = ctypes.POINTER(ctypes.c_uint32), ctypes.POINTER(ctypes.c_uint64)
    one = lambda v, t: np.array([v], dtype=t)
    rows, nb, ne, root = one(n, np.uint64), one(cols, np.uint32), one(0, np.uint32), np.zeros(8, dtype=np.uint32)
    ptrs = (ctypes.c_void_p * cols)(*[src.data_ptr() + 4 * n * i for i in range(cols)])
    waits = []
    for _ in range(5):
        h = ctypes.c_void_p()
        rc = ctx.L.lg_commit(ctx.h, 1, rows.ctypes.data_as(u64p), nb.ctypes.data_as(u32p), ne.ctypes.data_as(u32p),
                             ptrs, 1, ctypes.byref(h), root.ctypes.data_as(u32p))
        t0 = time.perf_counter()
        torch.cuda.synchronize()
        waits.append(time.perf_counter() - t0)
        assert rc == _lib.LG_ERR_OOM and "budget" in ctx.L.lg_last_error(ctx.h).decode()
    assert min(waits) < transforms / 5, (waits, transforms)
    small = F.to_mont(np.arange(1, 17, dtype=np.uint32))
    assert np.array_equal(ctx.rs_encode(small)[0], oracle.rs_encode(small, 64))
    ctx.close()


@pytest.mark.parametrize("logn,cols", [(12, 40), (15, 3), (17, 40), (20, 24)])
def test_an_encoding_that_does_not_fit_leaves_its_output_alone(logn, cols):
    """Device columns are encoded into the caller's buffer; whatever the budget
    refuses, it refuses before the first word is written."""
    import torch
    n = 1 << logn
    src, dst = dev(cols * n, 2), torch.empty(4 * cols * n, dtype=torch.int32, device="cuda:0")
    roomy = Context(0)
    encode(roomy, src, n, cols, dst)
    want, peak = dst.clone(), roomy.mem_usage()[1]
    roomy.close()
    refused = 0
    for part in range(1, 17):
        ctx = Context(0, hbm_budget=max(1, peak * part // 16))
        dst.fill_(-1)
        torch.cuda.synchronize()
        try:
            encode(ctx, src, n, cols, dst)
            assert torch.equal(dst, want)
        except LoomError as e:
            assert e.code == _lib.LG_ERR_OOM
            assert bool((dst == -1).all()), f"refused at {part}/16 of {peak} bytes"
            refused += 1
        ctx.close()
    assert 0 < refused < 16
