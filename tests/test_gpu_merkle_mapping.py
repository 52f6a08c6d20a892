"""Merkle trees across the line between the two permutation mappings (one
thread or six lanes per node): sizes on both sides of it, injections wider and
narrower than it, permutation counts that leave partial groups and warps."""
import numpy as np
import pytest

import oracle
from loom_b200 import field as F

pytestmark = pytest.mark.gpu


def rnd(shape, seed):
    return F.to_mont(np.random.Generator(np.random.PCG64(seed)).integers(0, F.P, shape, dtype=np.uint64).astype(np.uint32))


@pytest.mark.parametrize("log_leaves,widths", [(0, []), (1, [1]), (5, [5, 5]), (6, [0]), (12, [12, 3]), (13, [12]),
                                               (14, [14, 13, 13, 5]), (15, [12, 12]), (16, [13])])
def test_tree_equals_oracle(ctx, log_leaves, widths):
    leaves = rnd((1 << log_leaves, 8), log_leaves)
    inj = [rnd((1 << w, 8), 100 + k) for k, w in enumerate(widths)]
    assert np.array_equal(ctx.merkle_root(leaves, inj), oracle.merkle_root(leaves, inj))


@pytest.mark.parametrize("n", [1, 5, 6, 21, 130])
def test_partial_groups_of_permutations(ctx, n):
    canon = np.random.Generator(np.random.PCG64(n)).integers(0, F.P, (n, 24), dtype=np.uint64).astype(np.uint32)
    canon[0], canon[-1] = F.P - 1, np.where(np.arange(24) % 2, 0, F.P - 1)
    got = F.from_mont(ctx.poseidon2_permute(F.to_mont(canon)))
    for i in range(n):
        assert np.array_equal(got[i], oracle.p2_permute(canon[i], 24)), i
