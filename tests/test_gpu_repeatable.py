"""Solves without heavy near ranges (whose chunks are added as they come) give
the same bits every time, and a system the same bits whatever is solved beside
it."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [2, 12])
@pytest.mark.parametrize("n,maxbox", [(2400, 40), (5000, 96), (700, 700)])
def test_fp64_leaves_over_several_windows(aran, n, maxbox, order):
    """Leaves of 34 points and more lie over three windows of 32 particles."""
    x, q = W.uniform(n, n + order)
    with aran.Solver3d(maxbox=maxbox, order=order, precision="fp64") as s:
        pot, fld = s.solve(x, q)
        mult, _ = s.expansions()
        for _ in range(4):
            p, f = s.solve(x, q)
            assert np.array_equal(p, pot) and np.array_equal(f, fld)
        # behind a system of k points: other places in the windows.  Its root is
        # the first node, the roots come first, and deeper nodes are all of x
        for k in (1, 13, 31):
            xs, qs = np.concatenate([x[:k], x]), np.concatenate([q[:k], q])
            s.solve_forest(xs, qs, np.array([0, k, k + n]), np.tile([0.0] * 3 + [1.0] * 3, (2, 1)))
            assert np.array_equal(s.expansions()[0][1:], mult)


@pytest.mark.parametrize("order,precision,maxbox", [(4, "fp64", 20), (12, "fp64", 40), (26, "fp64", 64),
                                                    (8, "mixed", 20), (12, "mixed", 64),
                                                    (16, "mixed", 40)])
@pytest.mark.parametrize("copies", [2, 40])
def test_alone_and_in_a_forest(aran, order, precision, maxbox, copies):
    """The order of a target's translations does not depend on the parents in the
    pass (FP64 solves, and the FP64 levels of mixed ones from order 16)."""
    n = 3000
    x, q = W.uniform(n, order)
    x = np.round(x * 2.0**40) / 2.0**40          # shifts by whole numbers are exact
    shift = np.arange(copies)[:, None] * np.array([[2.0, 0.0, -4.0]])
    xs = np.concatenate([x[:7]] + [x + h for h in shift])
    boxes = np.hstack([shift, shift + 1.0])
    offs = np.concatenate([[0], 7 + np.arange(copies + 1) * n])
    with aran.Solver3d(maxbox=maxbox, order=order, precision=precision) as s:
        pot, fld = s.solve(x, q)
        fp, ff = s.solve_forest(xs, np.concatenate([q[:7], np.tile(q, copies)]), offs,
                                np.concatenate([boxes[:1], boxes]))
    for k in range(copies):
        a, b = offs[k + 1], offs[k + 2]
        assert np.array_equal(fp[a:b], pot) and np.array_equal(ff[a:b], fld), k
