"""The tiles of the large 2D levels along the sides of the box: stored
coefficients with walls, periodic directions and both, remainders of a
launch's sweeps."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

WALLS = {0: ("dirichlet", 0.5), 1: ("neumann", -0.25), 2: ("neumann", 1.0), 3: ("dirichlet", -1.0)}


def problem(depth, sides, lam, seed):
    per = {"walls": (), "periodic": (0, 1), "channel": (0,), "pipe": (1,)}[sides]
    bc = {s: v for s, v in WALLS.items() if s // 2 not in per}
    p = helpers.random_problem(2, depth, np.random.default_rng(seed), periodic=per, bc=bc, lam=lam)
    for d in per:                                # face n of a periodic direction is face 0
        c = p["alpha"][d]
        c[(slice(None),) * d + (-1,)] = c[(slice(None),) * d + (0,)]
    return p


@pytest.mark.parametrize("depth,nrelax", [(8, 5), (9, 1), (9, 6), (10, 4)])
@pytest.mark.parametrize("sides", ["walls", "periodic", "channel", "pipe"])
@pytest.mark.parametrize("lam", [None, "field"])
def test_stored_coefficients_bit_identical(depth, nrelax, sides, lam):
    from oracle import oracle
    p = problem(depth, sides, lam, depth + nrelax)
    g, a, b, alpha, lam_f = helpers.gpu_grid(p, relax="rbgs")
    o = helpers.oracle_grid(p, relax=oracle.RELAX_RBGS, threads=8)
    sg = g.poisson(a, b, alpha=alpha, lambda_=lam_f, tolerance=1e300, nrelax=nrelax)
    so = o.poisson(tolerance=1e300, nrelax=nrelax)
    assert sg["resb"] == so["resb"] and sg["resa"] == so["resa"]
    np.testing.assert_array_equal(a.get(), o.get_a())
    g.close()


@pytest.mark.parametrize("depth", [9, 10])
@pytest.mark.parametrize("lam", [None, "field"])
def test_mixed_commutes_with_half_a_period(depth, lam):
    """A shift by half the domain along both axes keeps every level's cells
    and colours (minlevel 1) and moves the tiles against them: the solutions
    of the mixed form are the shifted ones, bit for bit."""
    p = problem(depth, "periodic", lam, depth)
    n = 1 << depth
    q = dict(p)
    roll = lambda c: np.roll(c, (n // 2, n // 2), axis=(0, 1))
    q["b"] = roll(p["b"])
    if lam:
        q["lambda"] = roll(p["lambda"])
    faces = []
    for d, c in enumerate(p["alpha"]):
        r = roll(np.delete(c, -1, axis=d))
        faces.append(np.concatenate([r, np.take(r, [0], axis=d)], axis=d))
    q["alpha"] = faces
    out = []
    for prob in (p, q):
        g, a, b, alpha, lam_f = helpers.gpu_grid(prob, relax="rbgs", precision="mixed")
        st = g.poisson(a, b, alpha=alpha, lambda_=lam_f, tolerance=1e300, nrelax=7, minlevel=1)
        out.append((st["resa"], a.get()))
        g.close()
    assert out[0][0] == out[1][0]
    np.testing.assert_array_equal(roll(out[0][1]), out[1][1])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("depth", [9, 10])
@pytest.mark.parametrize("alpha", ["stored", "unit"])
def test_a_solve_repeats_itself(depth, precision, alpha):
    """The same walls, coefficients and right-hand side many times on one grid:
    the same bits each time."""
    p = problem(depth, "walls", None, 3)
    if alpha == "unit":
        p = dict(p, alpha=None)
    g, a, b, al, lam = helpers.gpu_grid(p, relax="rbgs", precision=precision)
    zero = np.zeros((1 << depth, 1 << depth))
    first = None
    for _ in range(12):
        a.set(zero)
        st = g.poisson(a, b, alpha=al, lambda_=lam, tolerance=1e300, nrelax=6)
        if first is None:
            first = (st["resa"], a.get())
        assert st["resa"] == first[0]
        np.testing.assert_array_equal(a.get(), first[1])
    g.close()


@pytest.mark.parametrize("depth", [9, 10])
@pytest.mark.parametrize("sides", ["walls", "channel", "pipe"])
@pytest.mark.parametrize("lam", [None, "field"])
def test_mixed_cycle_is_the_fp64_cycle_to_rounding(depth, sides, lam):
    """One cycle of both forms from the same start.  The sweeps contract, so
    the forms differ by the roundings of the FP32 operations, some ten per
    cell and pass, 2 nrelax passes on each of depth levels: at most
    10 * 12 * 10 * 2^-24 = 7e-5 of the largest value.  A side's ghosts left
    out of one pass change the cells along it by a quarter of their value."""
    p = problem(depth, sides, lam, 17)
    out = []
    for precision in ("fp64", "mixed"):
        g, a, b, alpha, lam_f = helpers.gpu_grid(p, relax="rbgs", precision=precision)
        g.poisson(a, b, alpha=alpha, lambda_=lam_f, tolerance=1e300, nrelax=6, minlevel=1)
        out.append(a.get())
        g.close()
    assert np.abs(out[1] - out[0]).max() <= 7e-5*np.abs(out[0]).max()
