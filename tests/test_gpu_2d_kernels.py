"""The 2D near field on leaves of every size around the block's edges, and the
2D M2L at the orders where its instances change (terms per lane in FP64,
length of the binomial row in mixed precision)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("precision,tol", [("fp64", 4e-15), ("mixed", 4e-6)])
@pytest.mark.parametrize("n", [1, 2, 3, 42, 43, 64, 65, 127, 128, 129, 255, 257, 700])
def test_one_leaf(aran, n, precision, tol):
    """maxbox n: every pair by the near field; errors in units of the sum of the
    terms' sizes (mixed: an offset is good to 2^-24 of the leaf, 8e-7 of a pair
    at h/8, and enters three times; FP64: 10 operations and the sum)."""
    rng = np.random.default_rng(n)
    x, q = rng.uniform(-1, 1, (n, 2)), rng.uniform(-1, 1, n)
    if n > 2:
        x[1] = x[2] + np.array([3e-5, -2e-5])    # closer than h/8
    with aran.Solver2d(maxbox=max(n, 65), order=4, precision=precision) as s:
        acc = s.solve(x, q)
    with aran.Solver2d(maxbox=min(n, 64), order=4, precision=precision) as s:
        leaf = s.solve(x, q)        # a warp per leaf
    if n <= 64:
        assert np.abs(leaf - acc).max() <= 2e-6 * np.abs(acc).max()
    z = x[:, 0] + 1j * x[:, 1]
    d = z[:, None] - z[None, :]
    np.fill_diagonal(d, np.inf)
    w = q[None, :] / d
    assert np.all(np.abs(acc - w.sum(1)) <= tol * max(1.0, np.sqrt(n) / 8) * np.abs(w).sum(1))


@pytest.mark.parametrize("precision,orders", [("fp64", (2, 31, 32, 40, 63, 64)),
                                              ("mixed", (2, 12, 13, 20, 21, 31))])
def test_orders(aran, oracle, precision, orders):
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.uniform(-1, 1, (1500, 2)), 0.3 + 0.02 * rng.normal(size=(1500, 2))])
    x = x.clip(-1, 1)
    q = rng.uniform(-1, 1, len(x))
    for p in orders:
        with aran.Solver2d(maxbox=12, order=p, precision=precision) as s:
            acc = s.solve(x, q)
        ref, _ = oracle.solve2d(x, q, [0, len(q)], [[-1.0, -1.0, 1.0, 1.0]], 12, p)
        assert rel_l2(acc, ref) < (1e-12 if precision == "fp64" else 3e-6), p


def test_box_far_from_the_origin(aran):
    """Positions exact in FP64 in either box: only the box's extent counts, so
    mixed results differ by the order of additions at most."""
    rng = np.random.default_rng(8)
    x = np.round(rng.uniform(-1, 1, (4000, 2)) * 2.0**30) / 2.0**30
    q = rng.uniform(-1, 1, len(x))
    out = []
    for h in (np.zeros(2), np.array([2.0**20, -(2.0**21)])):
        box = np.concatenate([h - 1.0, h + 1.0])[None, :]
        with aran.Solver2d(maxbox=32, order=20, precision="mixed") as s:
            out.append(s.solve(x + h, q, boxes=box))
    assert rel_l2(out[1], out[0]) <= 1e-10
