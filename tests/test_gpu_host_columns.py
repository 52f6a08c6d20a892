"""Host columns that lie next to one another in memory but not in one
page-locked block: two blocks registered one by one, a registered block beside
pageable memory, and columns that share a block."""
import mmap

import numpy as np
import pytest

from loom_b200 import field as F, plonk

pytestmark = pytest.mark.gpu
PAGE = mmap.PAGESIZE


class Blocks:
    """`pages` pages of memory, the page ranges of `locked` registered one by one."""

    def __init__(self, pages, locked):
        import torch
        self.rt = torch.cuda.cudart()
        torch.zeros(1, device="cuda:0")
        self.mem = mmap.mmap(-1, pages * PAGE)
        self.words = np.frombuffer(self.mem, dtype=np.uint32)
        self.words[:] = 0
        self.at = []
        for first, n in locked:
            a = self.words.ctypes.data + first * PAGE
            assert int(self.rt.cudaHostRegister(a, n * PAGE, 0)) == 0
            self.at.append(a)

    def close(self):
        for a in self.at:
            assert int(self.rt.cudaHostUnregister(a)) == 0


def lay_out(blocks, columns):
    out, off = [], 0
    for c in columns:
        v = blocks.words[off:off + c.size].reshape(c.shape)
        v[:] = c
        out.append(v)
        off += c.size
    return out


# columns of one page each: page-locked blocks and the pageable rest
LAYOUTS = [[(0, 4), (4, 4)], [(0, 1), (1, 2), (3, 5)], [(0, 3)], [(4, 4)], [(2, 3)], [(0, 8)], []]


@pytest.mark.parametrize("locked", LAYOUTS)
def test_commit(ctx, locked):
    n = PAGE // 4
    rng = np.random.default_rng(len(locked))
    cols = [F.to_mont(rng.integers(0, F.P, n, dtype=np.uint64).astype(np.uint32)) for _ in range(8)]
    want = ctx.commit_root([{"rows": n, "base": [c.copy() for c in cols[:3]]}, {"rows": n, "base": [c.copy() for c in cols[3:]]}])
    b = Blocks(8, locked)
    try:
        v = lay_out(b, cols)
        assert np.array_equal(ctx.commit_root([{"rows": n, "base": v[:3]}, {"rows": n, "base": v[3:]}]), want)
    finally:
        b.close()


@pytest.mark.parametrize("locked", LAYOUTS)
def test_prove(ctx, locked):
    compiled, wit = plonk.build(1, PAGE // 4, seed=5)
    mont = [F.to_mont(w) for w in wit]
    want = ctx.prove(compiled.words, mont, 8)
    b = Blocks(max(8, len(mont)), locked)
    try:
        assert ctx.prove(compiled.words, lay_out(b, mont), 8) == want
    finally:
        b.close()
