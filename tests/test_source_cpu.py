"""Properties of the CUDA sources that no run can show: an order of memory accesses that holds by accident."""
import glob
import os

from horizon_kernels_b200 import build


def test_no_barrier_takes_its_lanes_from_the_active_mask():
    """__activemask() names the lanes that happen to run together, not those that must meet: merge_kernel's lanes of a row read
    the row's state before one of them replaces it, and name each other"""
    for f in sorted(glob.glob(os.path.join(build.CSRC, "*.cu*"))):
        assert "__activemask" not in open(f).read(), f
