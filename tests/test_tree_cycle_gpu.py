"""The quadtree cycle in distributed shared memory against the interpreter (a
tree built with BMG_NO_TREE_CYCLE set) and one launch per operation
(BMG_NO_TREE_INTERP; FP64 alone has that route), bit for bit: trees from a
single cell to more cells of a level than the shared memory stages, random
refinements, refined corners, coarsest levels inside and above the leaves, and
a tree whose cells fit the slots in FP32 and not in FP64.  Which route ran
shows in the launches: three per iteration, or one interpreted."""
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
        if shape == "half":
            return level < depth - 1 or x < L0 / 2
        if shape == "corner":
            return max(x, y) / L0 < 2.5 / (1 << level)
        if shape == "band":
            return level < 4 or abs(math.hypot(x - 0.5, y - 0.5) - 0.3) < 3.0 * L0 / (1 << level)
        n = 1 << level
        return bool(picks[level][int(x / L0 * n), int(y / L0 * n)])
    return cond


def solve(depth, shape, minlevel, nrelax, off=None, precision="fp64"):
    import basilisk_b200 as bmg
    if off:
        os.environ[off] = "1"
    try:
        g = bmg.TreeGrid(depth, L0=L0, precision=precision)
        g.refine(condition(shape, depth, 3))
    finally:
        if off:
            os.environ.pop(off, None)
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
    g.reset_counters()
    tolerance = 1e-2 if shape == "half" else 1e-7
    st = g.poisson(a, b, alpha=alpha, lambda_=lam, tolerance=tolerance, minlevel=minlevel, nrelax=nrelax)
    out = [np.where(g.leaf_mask(l), a.get(level=l), 0.0) for l in range(g.tree_depth + 1)]
    st = dict(st, launches=g.counters()["launches"])
    g.close()
    return st, out


def same(one, other):
    (s1, x1), (s0, x0) = one, other
    for key in ("i", "nrelax", "resb", "resa"):
        assert s1[key] == s0[key], (key, s1, s0)
    for u, v in zip(x1, x0):
        np.testing.assert_array_equal(u, v)


def few_passes(depth, shape):
    """Full trees of one or two levels at nrelax 4 and below are interpreted
    (depth 1 from minlevel 1)."""
    return shape == "uniform" and depth < 2


TREES = [(0, "uniform", 0, 0), (1, "uniform", 0, 0), (5, "uniform", 0, 0), (4, "corner", 0, 1),
         (8, "corner", 3, 0), (6, "band", 0, 0), (9, "band", 0, 0), (9, "band", 6, 2),
         (5, "random", 0, 0), (7, "random", 0, 0), (9, "random", 2, 3)]


@pytest.mark.parametrize("depth,shape,minlevel,nrelax", TREES + [(10, "half", 0, 0)])
def test_cycle_bit_identical_to_launches(depth, shape, minlevel, nrelax):
    fast = solve(depth, shape, minlevel, nrelax)
    interpreted = solve(depth, shape, minlevel, nrelax, "BMG_NO_TREE_CYCLE")
    same(fast, interpreted)
    same(fast, solve(depth, shape, minlevel, nrelax, "BMG_NO_TREE_INTERP"))
    fits = shape != "half" and not few_passes(depth, shape)
    assert fast[0]["launches"] - interpreted[0]["launches"] == (2 * fast[0]["i"] if fits else 0)


@pytest.mark.parametrize("depth,shape,minlevel,nrelax", TREES + [(10, "half", 0, 0)])
def test_mixed_cycle_bit_identical_to_the_interpreter(depth, shape, minlevel, nrelax):
    fast = solve(depth, shape, minlevel, nrelax, precision="mixed")
    interpreted = solve(depth, shape, minlevel, nrelax, "BMG_NO_TREE_CYCLE", precision="mixed")
    same(fast, interpreted)
    fits = not few_passes(depth, shape)
    assert fast[0]["launches"] - interpreted[0]["launches"] == (2 * fast[0]["i"] if fits else 0)
