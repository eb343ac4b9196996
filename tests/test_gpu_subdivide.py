"""The subdivision of all levels at once against the one that goes level by
level (taken when a leaf predicate is set; this one keeps every node): the same
nodes, ranges and lists, number by number, over leaf capacities, depth limits,
clustered and coincident points, sizes at the edges of a block of places."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def both(aran, run, **kw):
    out = []
    for pred in (None, lambda v: False):
        with aran.Solver3d((-1, -1, -1), (1, 1, 1), order=4, **kw) as s:
            s.set_leaf_predicate(pred)
            pot = run(s)
            out.append((s.tree_info(), s.tree_lists(), pot))
    (ia, la, pa), (ib, lb, pb) = out
    assert ia == ib
    for k in la:
        assert np.array_equal(la[k], lb[k]), k
    assert np.linalg.norm(pa - pb) <= 1e-12 * np.linalg.norm(pb)


@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1024, 1025, 9000])
@pytest.mark.parametrize("maxbox,max_depth", [(1, 0), (1, 2), (7, 1), (20, 0), (64, 4), (5000, 0)])
def test_same_tree(aran, n, maxbox, max_depth):
    for x, q in (W.uniform(n, n), W.plummer(n, n)):
        both(aran, lambda s: s.solve(x, q)[0], maxbox=maxbox, max_depth=max_depth, precision="fp64")


@pytest.mark.parametrize("semifar", [0, 40])
def test_coincident_and_clustered(aran, semifar):
    rng = np.random.default_rng(3)
    x = np.concatenate([np.full((50, 3), 0.3), rng.uniform(-1, 1, (700, 3)),
                        1e-5 * rng.normal(size=(4000, 3)), np.full((9, 3), -1.0)])
    q = rng.uniform(-1, 1, len(x))
    both(aran, lambda s: s.solve(x, q)[0], maxbox=4, max_depth=21, precision="fp64",
         semifar_threshold=semifar)


def test_forest(aran):
    sizes = [0, 1, 3000, 0, 0, 1024, 17, 5000, 0]
    rng = np.random.default_rng(4)
    lo = np.arange(len(sizes))[:, None] * np.array([[2.0, 0.0, 4.0]]) - 1.0
    x = np.concatenate([a + 2.0 * rng.random((n, 3)) ** 2 for a, n in zip(lo, sizes)])
    q = rng.uniform(-1, 1, len(x))
    off = np.concatenate([[0], np.cumsum(sizes)])
    both(aran, lambda s: s.solve_forest(x, q, off, np.hstack([lo, lo + 2.0]))[0], maxbox=9,
         precision="fp64")
