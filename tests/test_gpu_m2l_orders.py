"""The lane-parallel M2L at every order it serves (even orders 4 to 16): few
parents (the offset list split over CTAs, a last group that is not full),
many parents (no split), against the oracle's FP64 solve and the kernel whose
lanes run over the coefficients."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu

MIXED_TOL = 3e-6    # FP32 bulk against the FP64 oracle, as for the other mixed tests
KERNEL_TOL = 1e-6   # two FP32 evaluations of the same operator


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("order", [4, 6, 8, 10, 12, 14, 16])
@pytest.mark.parametrize("n,maxbox,dist", [(700, 8, "uniform"), (6000, 12, "plummer")])
def test_lane_orders_against_oracle(aran, oracle, order, n, maxbox, dist):
    x, q = W.uniform(n, 50 + order) if dist == "uniform" else W.plummer(n, 50 + order)
    lb = (0, 0, 0) if dist == "uniform" else (-1, -1, -1)
    with aran.Solver3d(lb, (1, 1, 1), maxbox=maxbox, order=order, precision="mixed") as s:
        pot, fld = s.solve(x, q)
    opot, _ = oracle.solve(x, q, order=order, maxbox=maxbox, field=False, lb=lb, ub=(1, 1, 1))
    ofld, _ = oracle.solve(x, q, order=order, maxbox=maxbox, field=True, lb=lb, ub=(1, 1, 1))
    assert rel_l2(pot, opot) < MIXED_TOL
    assert rel_l2(fld, ofld) < MIXED_TOL


@pytest.mark.parametrize("order", [6, 12, 16])
def test_lane_kernel_unsplit(aran, order):
    """Enough parents for one CTA per group of them to take the whole list."""
    x, q = W.uniform(60000, 7)
    out = {}
    for kernel in ("lanes", "sibling"):
        with aran.Solver3d(maxbox=2, order=order, precision="mixed") as s:
            s.set_m2l_kernel(kernel)
            out[kernel] = s.solve(x, q)
    for a, b in zip(out["lanes"], out["sibling"]):
        assert rel_l2(a, b) < KERNEL_TOL


def test_lane_kernel_reused_buffers(aran):
    """Solves of different sizes on one solver (the split's workspace and the
    expansions are kept and reused) equal those of fresh solvers."""
    sets = [W.uniform(n, n) for n in (40000, 900, 15000)]
    with aran.Solver3d(maxbox=16, order=10, precision="mixed") as s:
        got = [s.solve(x, q) for x, q in sets]
    for (x, q), (pot, fld) in zip(sets, got):
        with aran.Solver3d(maxbox=16, order=10, precision="mixed") as s:
            p, f = s.solve(x, q)
        assert rel_l2(pot, p) < 1e-12 and rel_l2(fld, f) < 1e-12
