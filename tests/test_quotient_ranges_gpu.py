"""The FP64 smoothers divide by a known diagonal through its reciprocal, with
plain divisions where an operand is outside the range in which that rounds
to nearest: coefficients and sources of any magnitude, and zeros, give the
oracle's doubles."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,depth", [(2, 1), (2, 5), (2, 6), (2, 7), (2, 10), (3, 1), (3, 3), (3, 4)])
@pytest.mark.parametrize("alpha,b", [(1.0, 1.0), (1e-160, 1.0), (1e160, 1.0), (1.0, 1e-290), (1.0, 1e290),
                                     (1e-160, 1e-200), (1.0, 0.0), ("wide", 1.0), ("wide", "sparse")])
def test_one_cycle_of_any_magnitude(dim, depth, alpha, b):
    import basilisk_b200 as bmg
    n = 1 << depth
    rng = np.random.default_rng(17 * depth + dim)
    shape = lambda d: tuple(n + 1 if e == d else n for e in range(dim))
    al = [rng.uniform(0.5, 2.0, shape(d)) for d in range(dim)]
    rhs = rng.standard_normal((n,) * dim)
    if alpha == "wide":
        # neighbouring faces up to 100 binary orders apart
        al = [np.ldexp(c, rng.integers(-50, 50, c.shape)) for c in al]
    else:
        al = [alpha * c for c in al]
    if b == "sparse":
        # zeros, and a few values at the ends of the range of doubles
        keep = rng.random(rhs.shape) < 0.02
        rhs = np.where(keep, np.ldexp(rhs, rng.integers(-500, 400, rhs.shape)), 0.0)
    else:
        rhs = b * rhs
    g, o = bmg.Grid(dim, depth), oracle.Grid(dim, depth, relax=oracle.RELAX_RBGS)
    fa = g.scalar()
    for side in range(2 * dim):
        fa.bc(side, "dirichlet", 0.0)
        o.set_bc(side, oracle.DIRICHLET, value=0.0)
    fa.set(np.zeros(rhs.shape))
    o.set_a(np.zeros(rhs.shape))
    o.set_b(rhs)
    o.set_alpha(al)
    o.set_lambda_const(0.0)
    huge = 1e300
    sg = g.poisson(fa, g.scalar(rhs), alpha=g.face_vector(al), tolerance=huge, nrelax=3)
    so = o.poisson(tolerance=huge, nrelax=3)
    assert sg["i"] == so["i"] and sg["resa"] == so["resa"], (sg, so)
    np.testing.assert_array_equal(fa.get(), o.get_a())
    g.close()
