"""Field values in and out by rows of the contiguous axis (with the ghost
images of a cell field's finest level written by the same launch): every
extent at which a row, a chunk of a row or a block of rows can end."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,depth", [(1, 0), (1, 5), (1, 10), (1, 13), (2, 0), (2, 1), (2, 5), (2, 6),
                                       (2, 7), (2, 10), (3, 0), (3, 1), (3, 3), (3, 5), (3, 7)])
def test_fields_round_trip(dim, depth):
    import basilisk_b200 as bmg
    rng = np.random.default_rng(dim * 100 + depth)
    g = bmg.Grid(dim, depth)
    s, v = g.scalar(), g.face_vector()
    for level in sorted({depth, max(0, depth - 1)}):
        for f in [s] + v.components:
            x = rng.standard_normal(f.shape(level))
            f.set(x, level=level)
            np.testing.assert_array_equal(f.get(level=level), x)
    g.close()


@pytest.mark.parametrize("dim,depth,periodic", [(1, 6, False), (2, 0, False), (2, 0, True), (2, 1, False),
                                                (2, 7, True), (2, 8, False), (3, 0, True), (3, 1, False),
                                                (3, 5, False)])
def test_ghosts_of_a_field_set(dim, depth, periodic):
    """The residual of a field just set reads the ghosts its set wrote (or,
    for conditions given afterwards, the ghosts bc () wrote): the oracle's
    residual bit for bit."""
    import basilisk_b200 as bmg
    rng = np.random.default_rng(depth)
    n = 1 << depth
    a, b = (rng.standard_normal((n,) * dim) for _ in range(2))
    g, o = bmg.Grid(dim, depth), oracle.Grid(dim, depth)
    fa, fb, fr = g.scalar(), g.scalar(), g.scalar()
    o.set_alpha_const(1.0)
    o.set_lambda_const(-0.5)
    lam = g.const_scalar(-0.5)
    conds = [(side, ("dirichlet", "neumann")[side % 2], 0.25 * (side + 1)) for side in range(2 * dim)]
    if periodic:
        for d in range(dim):
            g.periodic(2 * d)
            o.set_periodic(d)
    else:
        for side, kind, value in conds:
            fa.bc(side, kind, value)
            o.set_bc(side, oracle.DIRICHLET if kind == "dirichlet" else oracle.NEUMANN, value=value)
    fa.set(a)
    fb.set(b)
    o.set_a(a)
    o.set_b(b)
    assert g.residual(fa, fb, fr, lambda_=lam) == o.residual()
    np.testing.assert_array_equal(fr.get(), o.get_res())
    if not periodic:
        for side, kind, value in conds:
            fa.bc(side, kind, 2.0 * value)
            o.set_bc(side, oracle.DIRICHLET if kind == "dirichlet" else oracle.NEUMANN, value=2.0 * value)
        assert g.residual(fa, fb, fr, lambda_=lam) == o.residual()
        np.testing.assert_array_equal(fr.get(), o.get_res())
    g.close()
