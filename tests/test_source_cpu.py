"""Properties of the CUDA sources that no run can show: an order of memory accesses that holds by accident, registers that
spill."""
import glob
import os
import subprocess

import pytest

from horizon_kernels_b200 import build


def test_no_barrier_takes_its_lanes_from_the_active_mask():
    """__activemask() names the lanes that happen to run together, not those that must meet: merge_kernel's lanes of a row read
    the row's state before one of them replaces it, and name each other"""
    for f in sorted(glob.glob(os.path.join(build.CSRC, "*.cu*"))):
        assert "__activemask" not in open(f).read(), f


def test_no_decode_kernel_spills(tmp_path):
    """what else lives in a decode kernel (the merge above all) must not push its unit loop over the register budget that the
    resident CTAs leave"""
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    r = subprocess.run([nvcc, *[f for f in build.NVCC_FLAGS if f not in ("-shared", "-cudart", "static")], "-Xptxas", "-v", "-c", "-o",
                        str(tmp_path / "decode.o"), os.path.join(build.CSRC, "hkv_decode.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    kernels, name = {}, None
    for line in r.stderr.splitlines():
        if "Function properties for" in line:
            name = line.split()[-1]
        elif "bytes spill stores" in line and "decode_kernel" in name:
            kernels[name] = line.strip()
    assert len(kernels) == 9
    assert all("0 bytes spill stores, 0 bytes spill loads" in k.split("frame, ")[1] and k.startswith("0 bytes") for k in kernels.values()), kernels
