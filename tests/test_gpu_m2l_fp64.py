"""The FP64 M2L where its instances and its ways of taking opposite offsets
change (pairs at once up to order 20, read twice from 21, by half CTAs from 24,
singly at 28, pairs again from 29), with sources at both, one or none of an opposite pair, unsplit
and split offset lists, against the oracle."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12     # the oracle's FP64 solve, as for the other FP64 tests


@pytest.mark.parametrize("order", [3, 12, 13, 16, 17, 20, 21, 23, 24, 28, 29])
def test_against_oracle(aran, oracle, order):
    x, q = W.plummer(1500, order)            # dense middle, sparse rim
    lb, ub = (-1, -1, -1), (1, 1, 1)
    with aran.Solver3d(lb, ub, maxbox=5, order=order, precision="fp64") as s:
        pot, _ = s.solve(x, q)
    ref, _ = oracle.solve(x, q, order=order, maxbox=5, field=False, lb=lb, ub=ub)
    assert np.linalg.norm(pot - ref) < FP64_TOL * np.linalg.norm(ref)


def test_many_parents(aran, oracle):
    x, q = W.uniform(20000, 9)
    with aran.Solver3d(maxbox=3, order=6, precision="fp64") as s:
        pot, fld = s.solve(x, q)
    ref, _ = oracle.solve(x, q, order=6, maxbox=3, field=False)
    assert np.linalg.norm(pot - ref) < FP64_TOL * np.linalg.norm(ref)
