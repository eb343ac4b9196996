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
