"""The FP64 tiles of constant coefficients: box and periodic sides, different
constants along x and y, lambda, remainders of the sweeps of a launch, the
prolongation in a level's first launch and the correction in the last, bit
for bit against the oracle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,nrelax,sides", [(9, 1, "walls"), (9, 4, "periodic"), (9, 5, "channel"),
                                                (10, 3, "walls"), (11, 6, "channel"), (11, 4, "periodic")])
@pytest.mark.parametrize("alpha,lam", [(1.0, 0.0), (0.3, -2.5), (1e-200, -1e-200)])
def test_one_cycle_bit_identical(depth, nrelax, sides, alpha, lam):
    import basilisk_b200 as bmg
    n = 1 << depth
    rng = np.random.default_rng(depth + nrelax)
    b, a0 = rng.standard_normal((n, n)), rng.standard_normal((n, n))
    g, o = bmg.Grid(2, depth, L0=1.5), oracle.Grid(2, depth, L0=1.5, relax=oracle.RELAX_RBGS, threads=8)
    fa = g.scalar()
    for d in range(2):
        if sides == "periodic" or (sides == "channel" and d == 0):
            g.periodic(2 * d)
            o.set_periodic(d)
        else:
            for s in (2 * d, 2 * d + 1):
                kind = ("dirichlet", "neumann")[s % 2]
                fa.bc(s, kind, 0.5 - s)
                o.set_bc(s, oracle.DIRICHLET if kind == "dirichlet" else oracle.NEUMANN, value=0.5 - s)
    fa.set(a0)
    o.set_a(a0)
    o.set_b(b)
    o.set_alpha_const(alpha)
    o.set_lambda_const(lam)
    falpha = None if alpha == 1.0 else g.const_face_vector(alpha)
    sg = g.poisson(fa, g.scalar(b), alpha=falpha, lambda_=g.const_scalar(lam), tolerance=1e300, nrelax=nrelax)
    so = o.poisson(tolerance=1e300, nrelax=nrelax)
    assert sg["resb"] == so["resb"] and sg["resa"] == so["resa"]
    np.testing.assert_array_equal(fa.get(), o.get_a())
    g.close()
