"""Rounding of the near fields' FP32 sums: charges of one sign in one box of 2 x 2
x 2 (2D: 2 x 2) leaves, every pair by the near field, against the FP64 sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rms(v):
    return float(np.sqrt(np.mean(np.square(v))))


@pytest.mark.parametrize("per", [30, 60, 120])
def test_mixed_3d(aran, per):
    """Sums of 32 terms at a time in plain FP32, compensated beyond: 8 x 120 terms
    1.7e-8 rms by an emulation in FP32, which grows as the root of 1 / terms; half
    as much again is allowed."""
    err = []
    for seed in range(10):
        rng = np.random.default_rng(seed)
        cell = np.array([[i, j, k] for i in (0, 1) for j in (0, 1) for k in (0, 1)])
        x = np.concatenate([0.5 * (c + rng.uniform(0.0, 1.0, (per, 3))) for c in cell])
        q = rng.uniform(0.0, 1.0, len(x))
        r = np.sqrt(((x[:, None] - x[None]) ** 2).sum(-1))
        np.fill_diagonal(r, np.inf)
        with aran.Solver3d(maxbox=per + 10, order=2, field=False, precision="mixed",
                           max_depth=1) as s:
            pot, _ = s.solve(x, q)
        err.append(pot / (q / r).sum(1) - 1.0)
    assert rms(err) <= 1.5 * 1.7e-8 * np.sqrt(120 / per)
