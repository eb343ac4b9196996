"""The mixed-precision near field on leaves of every size around the block's
edges (threads per target = 128 / n, tiles of 256 sources), against the FP64
direct sum term by term in size, with close and coincident points."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 13, 22, 24, 25, 42, 43, 64, 65, 127, 128, 129, 255, 257, 700])
def test_one_leaf(aran, n, field):
    """maxbox n: one leaf, every pair by the near field.  An offset is good to
    2^-24 of the leaf (relative to a pair at h/8: 8e-7), the hardware
    reciprocal square root to 2^-22, each of the other operations to 2^-24."""
    x, q = W.uniform(n, n + 1)
    if n > 2:
        x[n // 2] = x[0]                               # coincident: skipped
        x[1] = x[2] + np.array([3e-5, -2e-5, 1e-5])    # closer than h/8
    with aran.Solver3d(maxbox=max(n, 25), order=2, field=field, precision="mixed") as s:
        pot, fld = s.solve(x, q)
    if n <= 24:                     # the blocks of small leaf capacities
        with aran.Solver3d(maxbox=n, order=2, field=field, precision="mixed") as s:
            pot, fld = s.solve(x, q)
    d = x[:, None, :] - x[None, :, :]
    r = np.sqrt((d ** 2).sum(-1))
    with np.errstate(divide="ignore"):
        inv = np.where(r > (1e-5 if field else 0.0), 1.0 / r, 0.0)
    w = q[None, :] * inv
    assert np.all(np.abs(pot - w.sum(1)) <= 2e-6 * np.abs(w).sum(1))
    if field:
        g = (w * inv * inv)[:, :, None] * d
        assert np.all(np.abs(fld + g.sum(1)) <= 5e-6 * np.abs(w * inv).sum(1)[:, None])


def test_many_near_ranges(aran, oracle):
    """A coarse leaf beside finely divided cells has more near ranges than are
    taken together (32), some of them empty, some heavy."""
    rng = np.random.default_rng(5)
    x = np.concatenate([rng.uniform(0.0, 1.0, (300, 3)), 0.5 + 0.02 * rng.normal(size=(9000, 3)),
                        0.26 + 0.01 * rng.normal(size=(4000, 3))]).clip(0, 1 - 1e-9)
    q = rng.uniform(-1, 1, len(x))
    with aran.Solver3d(maxbox=6, order=10, precision="mixed") as s:
        pot, fld = s.solve(x, q)
    with aran.Solver3d(maxbox=6, order=10, precision="fp64") as s:
        p64, f64 = s.solve(x, q)
    assert np.linalg.norm(pot - p64) < 1e-6 * np.linalg.norm(p64)
    assert np.linalg.norm(fld - f64) < 1e-6 * np.linalg.norm(f64)


def test_box_far_from_the_origin(aran):
    """Positions exact in FP64 in either box: only the box's extent counts, so
    results differ by the order of FP64 additions at most."""
    x, q = W.uniform(5000, 3)
    x = np.round(x * 2.0**30) / 2.0**30
    h = np.array([2.0**20, -(2.0**21), 3.0])
    out = []
    for lb in (np.zeros(3), h):
        with aran.Solver3d(tuple(lb), tuple(lb + 1.0), maxbox=40, order=8, precision="mixed") as s:
            out.append(s.solve(x + lb, q))
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b)
