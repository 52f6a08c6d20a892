"""lg_poseidon2_permute with six lanes a state and with one thread a state:
around the line between them and at partial warps and blocks."""
import numpy as np
import pytest

import oracle
from loom_b200 import Context, field as F

pytestmark = pytest.mark.gpu


def states(n):
    c = np.random.Generator(np.random.PCG64(n)).integers(0, F.P, (n, 24), dtype=np.uint64).astype(np.uint32)
    c[0], c[-1] = F.P - 1, np.where(np.arange(24) % 2, 0, F.P - 1)
    return c


@pytest.mark.parametrize("lanes", [1, 6])
@pytest.mark.parametrize("n", [1, 31, 32, 127, 129, 300])
def test_forms_equal_oracle(lanes, n):
    c = Context(0)
    c.set_leaf_mapping(lanes)
    s = states(n)
    got = F.from_mont(c.poseidon2_permute(F.to_mont(s)))
    c.close()
    for i in range(n):
        assert np.array_equal(got[i], oracle.p2_permute(s[i], 24)), i


def test_around_the_line(ctx):
    import torch
    line = 96 * torch.cuda.get_device_properties(0).multi_processor_count
    for n in (line - 1, line, line + 1):
        s = F.to_mont(states(n))
        got = ctx.poseidon2_permute(s)
        six = Context(0)
        six.set_leaf_mapping(6)
        assert np.array_equal(got, six.poseidon2_permute(s))
        six.close()
