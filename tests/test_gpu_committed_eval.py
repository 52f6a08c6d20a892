"""Evaluations of committed polynomials (lg_committed_eval) at the sizes where
its cut into runs and chunks changes: fewer coefficients than one run, one
run, one block, one chunk and its neighbours, several chunks; base and
extension polynomials, negative and repeated shifts.  The reference value is
P(zeta w^s) by Horner's rule over the coefficients, in Python integers."""
import numpy as np
import pytest

from loom_b200 import field as F

pytestmark = pytest.mark.gpu
P = F.P


def rnd(shape, seed):
    return np.random.Generator(np.random.PCG64(seed)).integers(0, P, shape, dtype=np.uint64).astype(np.uint32)


def e2(a, b):  # F[u]/(u^2 - 3)
    return ((a[0] * b[0] + 3 * a[1] * b[1]) % P, (a[0] * b[1] + a[1] * b[0]) % P)


def e6(x, y):  # E2[v]/(v^3 - (u + 1)), the schoolbook product
    a, b = [x[0:2], x[2:4], x[4:6]], [y[0:2], y[2:4], y[4:6]]
    c = [[0, 0] for _ in range(5)]
    for i in range(3):
        for j in range(3):
            t = e2(a[i], b[j])
            c[i + j] = [(c[i + j][k] + t[k]) % P for k in range(2)]
    for k in (3, 4):  # v^3 = 1 + u
        t = e2(c[k], (1, 1))
        c[k - 3] = [(c[k - 3][q] + t[q]) % P for q in range(2)]
    return tuple(c[0] + c[1] + c[2])


def powers(z, n):
    out = np.zeros((n, 6), dtype=object)
    v = (1, 0, 0, 0, 0, 0)
    for k in range(n):
        out[k] = v
        v = e6(v, z)
    return out


def coefficients(values):
    """Inverse transform of Lagrange values (canonical), O(n log n) over Python-sized words."""
    n = len(values)
    if n == 1:
        return np.array(values, dtype=object)
    w = pow(F.root_of_unity(n), P - 2, P)
    a = np.array(values, dtype=object)

    def rec(x, w):
        if len(x) == 1:
            return x
        e, o = rec(x[0::2], w * w % P), rec(x[1::2], w * w % P)
        t = F.powers(w, len(e)).astype(object) * o % P
        return np.concatenate([(e + t) % P, (e - t) % P])

    return rec(a, w) * pow(n, P - 2, P) % P


@pytest.mark.parametrize("logn,shifts", [(1, [0, 1, -1]), (3, [0]), (4, [0, 3]), (5, [1]), (12, [0, 1]), (13, [0, -2, 0]),
                                         (14, [1])])
def test_committed_eval(ctx, logn, shifts):
    n = 1 << logn
    base, ext, zeta = rnd(n, logn), rnd((n, 6), 50 + logn), tuple(int(x) for x in rnd(6, 90 + logn))
    batch = ctx.commit([{"rows": n, "base": [F.to_mont(base)], "ext": [F.to_mont(ext)]}])
    got = F.from_mont(batch.eval(F.to_mont(np.array(zeta, dtype=np.uint32)), shifts))
    batch.release()
    cb = coefficients([int(x) for x in base])
    ce = [coefficients([int(x) for x in ext[:, w]]) for w in range(6)]
    for k, s in enumerate(shifts):
        f = pow(F.root_of_unity(n), s % n, P)
        zp = powers(tuple(x * f % P for x in zeta), n)
        lane = lambda c: tuple(int(x) for x in (c[:, None] * zp).sum(axis=0) % P)
        assert tuple(int(x) for x in got[0, k]) == lane(cb), (logn, s)
        want = (0,) * 6
        for w in range(6):
            t = e6(lane(ce[w]), tuple(int(q == w) for q in range(6)))
            want = tuple((want[q] + t[q]) % P for q in range(6))
        assert tuple(int(x) for x in got[1, k]) == want, (logn, s)
