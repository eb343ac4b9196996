"""The subdivision of all levels at once against the one that goes level by
level (taken when a leaf predicate is set; this one keeps every node): the same
nodes, ranges and lists, number by number, over leaf capacities, depth limits,
clustered and coincident points, sizes at the edges of a block of places."""
import ctypes

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


@pytest.mark.parametrize("maxbox,max_depth", [(1, 21), (3, 2), (20, 21), (64, 5), (5000, 21)])
def test_same_tree_2d(aran, maxbox, max_depth):
    """Results to rounding and the same lists (their sizes and the counters)."""
    rng = np.random.default_rng(maxbox)
    sizes = [1, 1023, 1, 6000, 1024, 40]
    x = [rng.uniform(-1, 1, (n, 2)) for n in sizes]
    x[3][:3000] = 0.1 + 1e-4 * rng.normal(size=(3000, 2))
    x[4][:30] = 0.25                                  # coincident
    x = np.concatenate(x)
    q = rng.uniform(-1, 1, len(x))
    off = np.concatenate([[0], np.cumsum(sizes)])
    keep = aran.LEAF_PREDICATE(lambda v, _d: 0)
    out = []
    for pred in (None, keep):
        with aran.Solver2d(maxbox=maxbox, max_depth=max_depth, order=6) as s:
            fn = aran.load().aran_gpu_solver2d_set_leaf_predicate
            assert fn(s._h, ctypes.cast(pred, ctypes.c_void_p) if pred else None, None) == 0
            acc = s.solve(x, q, off)
            out.append((s.tree_info(), s.get_stats(), acc))
    (ia, sa, a), (ib, sb, b) = out
    assert ia == ib and sa == sb
    ok = np.isfinite(b)                               # coincident points divide by zero
    assert np.array_equal(ok, np.isfinite(a)) and ok.sum() >= len(q) - 30
    assert np.linalg.norm((a - b)[ok]) <= 1e-13 * np.linalg.norm(b[ok])
