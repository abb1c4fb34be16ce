"""Kernels that walk a mesh's arrays: up to 2^31 - 1 items in steps of up to 2^20, so the index must be
wider than an int, which wraps on the last step and would address memory before the array."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hana-softwarerenderer_gb300", "csrc")


def test_walks_over_mesh_arrays_count_in_64_bits():
    found = 0
    for f in glob.glob(os.path.join(CSRC, "*.cu*")):
        s = open(f).read()
        # the signed type's wrap: (2^31 - 1 - 2^20, 2^31 - 1] + 2^20 is negative, and below any count
        assert not re.search(r"for \(int \w+ = (int\()?blockIdx", s), f
        found += len(re.findall(r"for \(size_t i = blockIdx\.x \* \(size_t\)blockDim\.x", s))
    assert found >= 6
