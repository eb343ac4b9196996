"""Rounding of the 2D FP64 translations at an order whose truncation is far below
it, against sums in extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_fp64_small_leaves(aran):
    """Small leaves: most of the sum by translations.  With Horner's rule, which
    adds the small terms first, the rms error of these twelve sets is 1.56e-16."""
    err = []
    for seed in range(12):
        rng = np.random.default_rng(seed)
        x = rng.uniform(-1, 1, (1500, 2))
        q = rng.uniform(0, 1, 1500)
        z = x[:, 0].astype(np.longdouble) + 1j * x[:, 1].astype(np.longdouble)
        d = z[:, None] - z[None]
        np.fill_diagonal(d, np.inf)
        ref = (q / d).sum(1)
        with aran.Solver2d(maxbox=8, order=40, precision="fp64") as s:
            a = s.solve(x, q)
        err.append(float(np.sqrt((abs(a - ref) ** 2).sum() / (abs(ref) ** 2).sum())))
    assert np.mean(err) <= 1.6e-16
