"""Rounding of the mixed M2L kernels: the lane-parallel kernel's constants add no
error to every translation alike, so its potentials are as close to the FP64 solve
of the same order as with the sibling kernel."""
import numpy as np
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [6, 8, 10, 12, 14])
def test_lanes_against_sibling(aran, order):
    err = {"lanes": [], "sibling": []}
    for seed in (90, 91, 92):
        x, q = W.plummer(4000, seed)
        kw = dict(lbound=(-1, -1, -1), ubound=(1, 1, 1), maxbox=8, order=order, field=False)
        with aran.Solver3d(precision="fp64", **kw) as s:
            ref, _ = s.solve(x, q)
        with aran.Solver3d(precision="mixed", **kw) as s:
            for kernel in err:
                s.set_m2l_kernel("auto" if kernel == "lanes" else kernel)
                pot, _ = s.solve(x, q)
                err[kernel].append(np.linalg.norm(pot - ref) / np.linalg.norm(ref))
    assert np.mean(err["lanes"]) <= 1.02 * np.mean(err["sibling"]), err
