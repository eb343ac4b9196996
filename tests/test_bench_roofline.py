"""The roofline entry of bench.py names the kernel that ran."""
import os

import bench

CSRC = os.path.join(os.path.dirname(os.path.abspath(bench.__file__)), "aran_gb300", "csrc")


def test_fp64_roofline_names_the_fp64_kernel():
    """launch_m2l sends every FP64 pass to m2l_fp64.cu, whatever the choice."""
    with open(os.path.join(CSRC, "m2l_fp64.cu")) as f:
        assert "k_m2l_fp64(" in f.read()
    for p in (4, 12, 13, 26):
        for choice in ("", "lanes", "sibling", "tc"):
            assert bench.roofline_kernel("fp64", p, choice).split()[0] == "k_m2l_fp64"
    assert bench.roofline_kernel("mixed", 12, "").startswith("k_m2l_lanes<12>")
