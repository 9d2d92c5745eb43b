"""The decomposed solve (grid/multigrid-mpi.h over blocks) against one grid
covering the same domain.

A domain of dims blocks of depth d equals one grid of depth d + log2 dims[0]
whose levels below log2 dims[0] are never visited: poisson () on the blocks
(minlevel 1 of a block) is the single grid's solve with minlevel
1 + log2 dims[0].  With the boundary exchanged after every pass, the blocks
must give the single grid's mgstats (cycles, nrelax, residuals) and
solution bit for bit in FP64; mgstats.sum is a sum in another order."""
import math

import numpy as np
import pytest

from basilisk_b200 import problems
from basilisk_b200.shard import ShardedGrid
from helpers import gpu_grid

pytestmark = pytest.mark.gpu


def sharded(prob, dims, relax):
    k = int(math.log2(dims[0]))
    sg = ShardedGrid(prob["dim"], prob["depth"] - k, dims=dims, periodic=prob["periodic"],
                     relax=relax)
    a = sg.scalar()
    for side, (kind, val) in prob["bc"].items():
        a.bc(side, kind, float(val))
    a.set(np.zeros(prob["b"].shape))
    b = sg.scalar(prob["b"])
    alpha = sg.face_vector(prob["alpha"]) if prob["alpha"] is not None else None
    lam = prob["lambda"]
    if lam is None:
        lam_f = None
    elif np.isscalar(lam):
        lam_f = sg.const_scalar(float(lam))
    else:
        lam_f = sg.scalar(lam)
    return sg, a, b, alpha, lam_f


def compare(prob, dims, relax, tolerance):
    k = int(math.log2(dims[0]))
    g, a, b, alpha, lam = gpu_grid(prob, relax=relax)
    st = g.poisson(a, b, alpha=alpha, lambda_=lam, tolerance=tolerance, minlevel=1 + k)
    ref = a.get()
    g.close()
    sg, sa, sb, salpha, slam = sharded(prob, dims, relax)
    ss = sg.poisson(sa, sb, alpha=salpha, lambda_=slam, tolerance=tolerance)
    got = sa.get()
    sg.close()
    for key in ("i", "nrelax", "resb", "resa"):
        assert ss[key] == st[key], (key, ss, st)
    assert ss["minlevel"] == 1 and st["minlevel"] == 1 + k
    assert abs(ss["sum"] - st["sum"]) <= 1e-12 * max(1.0, np.abs(prob["b"]).sum())
    np.testing.assert_array_equal(got, ref)
    return ss


@pytest.mark.parametrize("relax", ["rbgs", "jacobi"])
def test_two_phase_2x2_blocks_bit_identical(relax):
    """Dirichlet walls, variable face coefficients (density ratio 1000),
    four blocks of 128^2."""
    compare(problems.two_phase_2d(depth=8, seed=3), (2, 2), relax, 1e-6)


def test_periodic_2x2_blocks_bit_identical():
    """A periodic domain: the blocks' neighbours wrap around."""
    compare(problems.poisson_periodic_2d(depth=8, seed=4), (2, 2), "rbgs", 1e-8)


def test_sixteen_blocks_bit_identical():
    """4 x 4 blocks of 64^2: interior blocks with four neighbours, corner
    ghosts from the diagonal blocks."""
    compare(problems.two_phase_2d(depth=8, seed=6), (4, 4), "rbgs", 1e-6)


def test_mixed_conditions_and_lambda_field_bit_identical():
    """Inhomogeneous Dirichlet on two sides, Neumann on the others (each
    block keeps the condition of the domain's sides it touches), a stored
    lambda field: 2x2 blocks against one grid."""
    import helpers
    rng = np.random.default_rng(21)
    prob = helpers.random_problem(2, 7, rng, bc={0: ("dirichlet", 0.5), 1: ("neumann", -0.25),
                                                 2: ("dirichlet", -1.0), 3: ("neumann", 0.75)},
                                  lam="field")
    compare(prob, (2, 2), "rbgs", 1e-9)


def test_one_block_is_the_grid():
    """dims (1, 1): one block, nothing to exchange (its periodic directions
    are its own), the grid's solve with minlevel 1."""
    compare(problems.poisson_periodic_2d(depth=7, seed=9), (1, 1), "rbgs", 1e-8)


def test_1d_two_blocks_bit_identical():
    """One dimension, two blocks: single-cell ghost slabs."""
    import helpers
    rng = np.random.default_rng(13)
    prob = helpers.random_problem(1, 9, rng, bc={0: ("dirichlet", 1.0), 1: ("dirichlet", -0.5)})
    compare(prob, (2,), "rbgs", 1e-10)


def test_helmholtz_3d_2x2x2_blocks_bit_identical():
    """Periodic 3D Helmholtz (viscosity.h form) on eight blocks of 16^3:
    x slabs, strided y and z slabs."""
    compare(problems.helmholtz_3d(depth=5, seed=7), (2, 2, 2), "rbgs", 1e-8)


def test_two_blocks_rectangular_domain():
    """MPI_Dims_create (2, 2) = (2, 1): a 2:1 domain of two square blocks
    (the reference's rescaled domain, multigrid-mpi.h:115-123), periodic
    along x.  Its solution is symmetric under the shift by one block along
    x when the right-hand side is."""
    n = 64
    rng = np.random.default_rng(8)
    half = rng.standard_normal((n, n))
    half -= half.mean()
    b = np.concatenate([half, half], axis=0)
    sg = ShardedGrid(2, 6, dims=(2, 1), periodic=(0,), relax="rbgs", L0=2.0)
    a = sg.scalar()
    for side in ("top", "bottom"):
        a.bc(side, "dirichlet", 0.0)
    a.set(np.zeros((2 * n, n)))
    bb = sg.scalar(b)
    st = sg.poisson(a, bb, tolerance=1e-8)
    assert st["status"] == 0 and st["resa"] <= 1e-8, st
    sol = a.get()
    sg.close()
    np.testing.assert_array_equal(sol[:n], sol[n:])


@pytest.mark.parametrize("relax", ["rbgs", "jacobi"])
@pytest.mark.parametrize("dim,depth,dims,periodic", [(1, 3, (4,), False), (2, 2, (2, 2), False),
                                                     (2, 3, (4, 4), True), (2, 6, (2, 2), True),
                                                     (2, 7, (2, 2), False), (2, 8, (4, 4), False),
                                                     (3, 2, (2, 2, 2), False), (3, 3, (4, 4, 4), True),
                                                     (3, 5, (2, 2, 2), False)])
def test_blocks_around_the_single_cta_levels_bit_identical(dim, depth, dims, periodic, relax):
    """Blocks of two cells and up, whose levels lie below, at and above the
    cells that one CTA relaxes for all blocks (all their images -- edges and
    corners, box, periodic and neighbouring -- written by the owners)."""
    import helpers
    rng = np.random.default_rng(100 * dim + depth)
    kinds = [("dirichlet", 0.5), ("neumann", -0.25), ("dirichlet", -1.0), ("neumann", 0.75),
             ("neumann", 0.5), ("dirichlet", 0.25)]
    if periodic:
        prob = helpers.random_problem(dim, depth, rng, periodic=tuple(range(dim)), lam="field")
        for d, c in enumerate(prob["alpha"]):    # face n of a periodic direction is face 0
            c[(slice(None),) * d + (-1,)] = c[(slice(None),) * d + (0,)]
    else:
        prob = helpers.random_problem(dim, depth, rng, bc={s: kinds[s] for s in range(2 * dim)}, lam="field")
    compare(prob, dims, relax, 1e-8)


def test_blocks_of_one_cell():
    """2 x 2 blocks of a single cell, Dirichlet 0, alpha = 1: the solution of
    the 4 x 4 system (each cell: -6 a + two neighbours = b Delta^2).  Every
    cell relaxes from the last pass's neighbours and ghosts, which leaves the
    chequered mode undamped: b has none of it."""
    sg = ShardedGrid(2, 0, dims=(2, 2), relax="rbgs")
    a = sg.scalar()
    for side in ("right", "left", "top", "bottom"):
        a.bc(side, "dirichlet", 0.0)
    b = np.array([[6.0, 0.0], [2.0, -4.0]])
    a.set(np.zeros((2, 2)))
    st = sg.poisson(a, sg.scalar(b), tolerance=1e-9)
    assert st["status"] == 0 and st["resa"] <= 1e-9, st
    A = np.array([[-6, 1, 1, 0], [1, -6, 0, 1], [1, 0, -6, 1], [0, 1, 1, -6]], float)
    np.testing.assert_allclose(a.get().ravel(), np.linalg.solve(A, b.ravel() / 4.0), atol=1e-10)
    sg.close()


@pytest.mark.parametrize("dim,dims,periodic", [(1, (4,), False), (2, (2, 2), False), (2, (4, 4), True),
                                               (3, (2, 2, 2), False)])
def test_jacobi_on_blocks_of_one_cell_bit_identical(dim, dims, periodic):
    """Blocks of depth 0 against the one level of a grid of dims cells."""
    import helpers
    k = int(math.log2(dims[0]))
    rng = np.random.default_rng(70 + dim)
    bc = {s: ("dirichlet", 0.5) if s % 3 else ("neumann", -0.25) for s in range(2 * dim)}
    prob = helpers.random_problem(dim, k, rng, periodic=tuple(range(dim)) if periodic else (),
                                  bc=None if periodic else bc, lam="field")
    if periodic:
        for d, c in enumerate(prob["alpha"]):    # face n of a periodic direction is face 0
            c[(slice(None),) * d + (-1,)] = c[(slice(None),) * d + (0,)]
    g, a, b, alpha, lam = helpers.gpu_grid(prob, relax="jacobi")
    st = g.poisson(a, b, alpha=alpha, lambda_=lam, tolerance=1e-9, minlevel=k)
    ref = a.get()
    g.close()
    sg, sa, sb, salpha, slam = sharded(prob, dims, "jacobi")
    ss = sg.poisson(sa, sb, alpha=salpha, lambda_=slam, tolerance=1e-9)
    got = sa.get()
    sg.close()
    assert ss["minlevel"] == 0
    for key in ("status", "i", "nrelax", "resb", "resa"):
        assert ss[key] == st[key], (key, ss, st)
    np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("relax", ["rbgs", "jacobi"])
@pytest.mark.parametrize("dim,depth,dims", [(1, 4, (3,)), (2, 4, (3, 1)), (2, 5, (3, 1)), (2, 3, (5, 3)),
                                            (2, 6, (3, 1)), (2, 5, (5, 3)), (3, 3, (3, 1, 1))])
def test_repeated_blocks_equal_one_block(dim, depth, dims, relax):
    """A periodic domain of equal blocks, their number not a power of two:
    every block is the periodic solve of one block (the coarse levels of all
    of them joined in one CTA)."""
    import helpers
    prob = helpers.random_problem(dim, depth, np.random.default_rng(50 + dim + depth),
                                  periodic=tuple(range(dim)), lam="field")
    for d, c in enumerate(prob["alpha"]):
        c[(slice(None),) * d + (-1,)] = c[(slice(None),) * d + (0,)]
    out = []
    for D in ((1,) * dim, dims):
        sg = ShardedGrid(dim, depth, dims=D, periodic=tuple(range(dim)), relax=relax, L0=float(D[0]))
        faces = []
        for d, c in enumerate(prob["alpha"]):
            inner = np.tile(np.delete(c, -1, axis=d), D)
            faces.append(np.concatenate([inner, np.take(inner, [0], axis=d)], axis=d))
        a = sg.scalar()
        a.set(np.zeros(np.tile(prob["b"], D).shape))
        st = sg.poisson(a, sg.scalar(np.tile(prob["b"], D)), alpha=sg.face_vector(faces),
                        lambda_=sg.scalar(np.tile(prob["lambda"], D)), tolerance=1e-8)
        out.append((st, a.get()))
        sg.close()
    (s1, a1), (sn, an) = out
    for key in ("i", "nrelax", "resb", "resa"):
        assert sn[key] == s1[key], (key, sn, s1)
    np.testing.assert_array_equal(an, np.tile(a1, dims))


def test_tiles_and_passes_bit_identical():
    """Levels on either side of the size up to which tiles take several
    sweeps per launch."""
    import helpers
    prob = helpers.random_problem(2, 10, np.random.default_rng(10), lam="field",
                                  bc={0: ("dirichlet", 0.5), 1: ("neumann", -0.25),
                                      2: ("dirichlet", -1.0), 3: ("neumann", 0.75)})
    compare(prob, (2, 2), "rbgs", 1e-2*np.abs(prob["b"]).max())


def test_coarsest_level_of_tiles():
    """minlevel above the single-CTA levels: the cycle starts from zero on a
    level of tiles.  -laplacian + |lambda| is an M-matrix, whose inverse's
    maximum norm is at most 1/|lambda|: two solutions differ by at most the
    sum of their residuals over |lambda|."""
    sols = []
    lam = 1e4
    b = np.random.default_rng(3).standard_normal((256, 256))
    for minlevel in (7, 1):
        sg = ShardedGrid(2, 7, dims=(2, 2), relax="rbgs")
        a = sg.scalar()
        for side in ("right", "left", "top", "bottom"):
            a.bc(side, "dirichlet", 0.0)
        a.set(np.zeros(b.shape))
        st = sg.poisson(a, sg.scalar(b), lambda_=sg.const_scalar(-lam), tolerance=1e-7, minlevel=minlevel)
        assert st["status"] == 0 and st["resa"] <= 1e-7, st
        sols.append((a.get(), st["resa"]))
        sg.close()
    (a7, r7), (a1, r1) = sols
    assert np.abs(a7 - a1).max() <= (r7 + r1)/lam*(1. + 1e-6)
