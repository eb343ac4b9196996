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


@pytest.mark.parametrize("per", [60, 70, 120])
def test_mixed_2d(aran, per):
    """Sums of at most 64 terms at a time in plain FP32, compensated beyond: 1.8e-8
    rms of the terms' sum; half as much again is allowed."""
    err = []
    for seed in range(10):
        rng = np.random.default_rng(seed)
        x = np.concatenate([np.array(c) + rng.uniform(0.0, 1.0, (per, 2))
                            for c in ((-1, -1), (0, -1), (-1, 0), (0, 0))])
        q = rng.uniform(0.0, 1.0, len(x))
        z = x[:, 0] + 1j * x[:, 1]
        d = z[:, None] - z[None]
        np.fill_diagonal(d, np.inf)
        with aran.Solver2d(maxbox=per + per // 2, order=8, precision="mixed", max_depth=1) as s:
            e = (s.solve(x, q) - (q / d).sum(1)) / np.abs(q / d).sum(1)
        err.append([e.real, e.imag])
    assert rms(err) <= 1.5 * 1.8e-8


@pytest.mark.parametrize("scale", [1.0, 1e-148, 1e152])
def test_fp64_2d_reciprocal(aran, scale):
    """Pairs of points, one system each, across the ends of the range where the
    reciprocal is made from the hardware's approximation: a unit charge gives
    1 / dx, with a half ulp each from dx^2, the reciprocal (0.01 more), the product
    and the comparison."""
    k = 4000
    rng = np.random.default_rng(5)
    x = np.zeros((2 * k, 2))
    x[0::2] = 0.25 * scale
    x[1::2] = 0.25 * scale
    x[1::2, 0] += scale * 10.0 ** rng.uniform(-3, -0.3, k)
    d = x[1::2, 0] - x[0::2, 0]
    with aran.Solver2d(maxbox=2, order=2, precision="fp64") as s:
        acc = s.solve(x, np.ones(2 * k), np.arange(0, 2 * k + 1, 2), np.array([0.0, 0.0, scale, scale]))
    assert np.abs(acc[1::2].real * d - 1.0).max() <= 4.05 * 2.0**-53
    assert np.array_equal(acc[1::2].real, -acc[0::2].real)
