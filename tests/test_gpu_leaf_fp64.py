"""P2M and L2P in FP64 at the edges of the windows of 32 particles (leaves inside
one, across one and over several, a last window that is not full), with and
without the field, against the oracle."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12     # the oracle's FP64 solve, as for the other FP64 tests


@pytest.mark.parametrize("order", [1, 2, 9, 16])
@pytest.mark.parametrize("n,maxbox", [(31, 1), (33, 2), (64, 3), (700, 12), (1025, 33), (4000, 150)])
def test_windows(aran, oracle, n, maxbox, order):
    x, q = W.uniform(n, n + order)
    for field in (False, True):
        with aran.Solver3d(maxbox=maxbox, order=order, field=field, precision="fp64") as s:
            pot, fld = s.solve(x, q)
        ref, _ = oracle.solve(x, q, order=order, maxbox=maxbox, field=False)
        assert np.linalg.norm(pot - ref) < FP64_TOL * np.linalg.norm(ref)
    ref, _ = oracle.solve(x, q, order=order, maxbox=maxbox, field=True)
    assert np.linalg.norm(fld - ref) < FP64_TOL * np.linalg.norm(ref)
