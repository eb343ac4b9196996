"""The FP64 near field: leaves of every size around the block's edges (threads
per target = 128 / n), chunked heavy ranges apart (tests of clustered sets),
against the FP64 direct sum; and its reciprocal square root against
correctly rounded values."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("field", [False, True])
@pytest.mark.parametrize("n", [2, 3, 42, 43, 63, 64, 65, 127, 128, 129, 257, 1000])
def test_one_leaf(aran, oracle, n, field):
    """maxbox n: one leaf, every pair by the near field."""
    x, q = W.uniform(n, n)
    x[n // 2] = x[0]      # coincident points are skipped
    with aran.Solver3d(maxbox=n, order=2, field=field, precision="fp64") as s:
        pot, fld = s.solve(x, q)
    rp, rf = oracle.direct(x, q)
    # n terms of either sign, each good to 4 ulp
    tol = 4 * 2.3e-16 * np.sqrt(n) * 10
    scale = np.linalg.norm(np.abs(rp).max())
    assert np.abs(pot - rp).max() <= tol * max(scale, 1e-300) or n == 2
    if n == 2:
        assert np.all(pot == 0.0)
    elif field:
        assert np.abs(fld - rf).max() <= tol * np.abs(rf).max()


def test_reciprocal_square_root(aran):
    """Pairs of points, one forest system each: the potential of a unit charge
    is 1/r.  dx, dx^2 and the rounding of the last step leave at most 3 ulp."""
    k = 4000
    rng = np.random.default_rng(3)
    r = 10.0 ** rng.uniform(-9, -0.3, k)
    x = np.zeros((2 * k, 3))
    x[0::2] = 0.25
    x[1::2] = 0.25
    x[1::2, 0] += r
    d = x[1::2, 0] - x[0::2, 0]
    boxes = np.tile([0.0, 0.0, 0.0, 1.0, 1.0, 1.0], (k, 1))
    with aran.Solver3d(maxbox=2, order=2, field=False, precision="fp64") as s:
        pot, _ = s.solve_forest(x, np.ones(2 * k), np.arange(0, 2 * k + 1, 2), boxes)
    assert np.abs(pot[0::2] * d - 1.0).max() <= 3 * 2.3e-16
    assert np.array_equal(pot[0::2], pot[1::2])
