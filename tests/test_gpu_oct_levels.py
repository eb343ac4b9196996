"""M2M and L2L with a thread per part of a coefficient: levels of few nodes take
it in FP32, every level in FP64.  A system alone (few nodes a level) and in a
forest of its copies (many) take different kernels and must agree as forests
do; FP64 orders from the smallest to the largest against the oracle."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FOREST_TOL = 1e-10   # only the order of FP64 additions differs
FP64_TOL = 1e-12     # the oracle's FP64 solve, as for the other FP64 tests


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("order", [4, 8, 10, 12, 16])
@pytest.mark.parametrize("copies", [3, 20])
def test_levels_of_few_and_many_nodes(aran, order, copies):
    x, q = W.plummer(3000, order)
    x = np.round(x * 2.0**40) / 2.0**40          # shifts by whole numbers are exact
    shift = np.arange(copies)[:, None] * np.array([[2.0, 0.0, -4.0]])
    xs = np.concatenate([x + h for h in shift])
    with aran.Solver3d((-1, -1, -1), (1, 1, 1), maxbox=8, order=order, precision="mixed") as s:
        pot, fld = s.solve(x, q)
        fp, ff = s.solve_forest(xs, np.tile(q, copies), np.arange(copies + 1) * len(q),
                                np.hstack([shift - 1.0, shift + 1.0]))
    for p, f in zip(np.split(fp, copies), np.split(ff, copies)):
        assert rel_l2(p, pot) < FOREST_TOL
        assert rel_l2(f, fld) < FOREST_TOL


@pytest.mark.parametrize("order", [1, 2, 3, 13, 30])
def test_fp64_orders(aran, oracle, order):
    x, q = W.plummer(2500, 70 + order)
    lb, ub = (-1, -1, -1), (1, 1, 1)
    with aran.Solver3d(lb, ub, maxbox=6, order=order, precision="fp64") as s:
        pot, _ = s.solve(x, q)
    opot, _ = oracle.solve(x, q, order=order, maxbox=6, field=False, lb=lb, ub=ub)
    assert rel_l2(pot, opot) < FP64_TOL
