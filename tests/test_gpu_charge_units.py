"""Mixed solves give the same bits whatever the unit of the charges: a power of two
taken out of every charge comes back in the results, the expansions and, system
by system, in a forest."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu

UNITS = (-900, -130, -100, -60, 60, 100, 130, 900)


@pytest.mark.parametrize("order,semifar", [(4, 0), (8, 0), (9, 20), (12, 0), (16, 20), (18, 0)])
def test_powers_of_two(aran, order, semifar):
    """Orders of the lane-parallel, the sibling and the FP64 root kernels."""
    x, q = W.uniform(4000, order)
    q[::7] = 0.0
    with aran.Solver3d(maxbox=24, order=order, precision="mixed", semifar_threshold=semifar) as s:
        pot, fld = s.solve(x, q)
        mult, loc = s.expansions()
        for k in UNITS:
            u = 2.0**k
            p, f = s.solve(x, q * u)
            assert np.array_equal(p, pot * u) and np.array_equal(f, fld * u), k
            if abs(k) < 500:
                m, lo = s.expansions()
                assert np.array_equal(m, mult * u) and np.array_equal(lo, loc * u), k
        # all in one forest, a system without charges and an empty one among them
        qs = np.concatenate([q * 2.0**k for k in UNITS] + [np.zeros(3), q])
        nu = len(UNITS)
        offs = np.concatenate([np.arange(nu + 1) * len(q), [nu * len(q), nu * len(q) + 3, len(qs)]])
        xs = np.concatenate([x] * nu + [x[:3], x])
        fp, ff = s.solve_forest(xs, qs, offs, np.tile([0.0] * 3 + [1.0] * 3, (nu + 3, 1)))
    for i, k in enumerate(UNITS + (0,)):
        a = i * len(q) + (3 if k == 0 else 0)
        assert np.array_equal(fp[a:a + len(q)], pot * 2.0**k), k
        assert np.array_equal(ff[a:a + len(q)], fld * 2.0**k), k
    assert not fp[nu * len(q):nu * len(q) + 3].any()
