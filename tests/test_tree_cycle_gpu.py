"""The quadtree cycle in distributed shared memory against one launch per
operation (a tree built with BMG_NO_TREE_INTERP set), bit for bit: trees from
a single cell to more cells of a level than the shared memory stages, random
refinements, refined corners, coarsest levels inside and above the leaves."""
import math
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


L0 = 1.25


def condition(shape, depth, seed):
    rng = np.random.default_rng(seed)
    picks = {l: rng.random((1 << l, 1 << l)) < 0.35 for l in range(depth + 1)}

    def cond(level, x, y):
        if level >= depth:
            return False
        if shape == "uniform":
            return True
        if level < 2:
            return True
        if shape == "corner":
            return max(x, y) / L0 < 2.5 / (1 << level)
        if shape == "band":
            return level < 4 or abs(math.hypot(x - 0.5, y - 0.5) - 0.3) < 3.0 * L0 / (1 << level)
        n = 1 << level
        return bool(picks[level][int(x / L0 * n), int(y / L0 * n)])
    return cond


def solve(depth, shape, minlevel, nrelax, launches):
    import basilisk_b200 as bmg
    if launches:
        os.environ["BMG_NO_TREE_INTERP"] = "1"
    try:
        g = bmg.TreeGrid(depth, L0=L0)
        g.refine(condition(shape, depth, 3))
    finally:
        os.environ.pop("BMG_NO_TREE_INTERP", None)
    rng = np.random.default_rng(depth)
    a, b, alpha, lam = g.scalar(), g.scalar(), g.face_vector(), g.scalar()
    for s, kind in enumerate(("dirichlet", "neumann", "neumann", "dirichlet")):
        a.bc(s, kind, 0.0)
    for l in range(g.tree_depth + 1):
        n = 1 << l
        b.set(rng.standard_normal((n, n)), level=l)
        a.set(rng.standard_normal((n, n)), level=l)
        lam.set(-rng.uniform(0.1, 1.0, (n, n)), level=l)
        alpha.set([rng.uniform(0.5, 2.0, (n + 1, n)), rng.uniform(0.5, 2.0, (n, n + 1))], level=l)
    st = g.poisson(a, b, alpha=alpha, lambda_=lam, tolerance=1e-7, minlevel=minlevel, nrelax=nrelax)
    out = [np.where(g.leaf_mask(l), a.get(level=l), 0.0) for l in range(g.tree_depth + 1)]
    g.close()
    return st, out


@pytest.mark.parametrize("depth,shape,minlevel,nrelax", [(0, "uniform", 0, 0), (1, "uniform", 0, 0), (5, "uniform", 0, 0),
                                                         (4, "corner", 0, 1), (8, "corner", 3, 0), (6, "band", 0, 0),
                                                         (9, "band", 0, 0), (9, "band", 6, 2), (5, "random", 0, 0),
                                                         (7, "random", 0, 0), (9, "random", 2, 3)])
def test_cycle_bit_identical_to_launches(depth, shape, minlevel, nrelax):
    s1, x1 = solve(depth, shape, minlevel, nrelax, False)
    s0, x0 = solve(depth, shape, minlevel, nrelax, True)
    for key in ("i", "nrelax", "resb", "resa"):
        assert s1[key] == s0[key], (key, s1, s0)
    for u, v in zip(x1, x0):
        np.testing.assert_array_equal(u, v)
