"""Builds the CUDA library (csrc/*.cu) for sm_100a with nvcc into horizon_kernels_b200/lib/libhkv.so, and the host module
(csrc/hkv_host.cpp, torch's C++ API) into lib/hkv_host.so.

nvcc cross-compiles without a GPU. The library exports only the C ABI declared in include/hkv.h and depends on the
CUDA runtime alone (linked statically), not on torch; the host module binds it to torch's tensors."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(OUT_DIR, "libhkv.so")
HOST = os.path.join(OUT_DIR, "hkv_host.so")
SOURCES = ["hkv_write.cu", "hkv_decode.cu", "hkv_dequant.cu", "hkv_prefill.cu", "hkv_probe.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
              "-shared", "-cudart", "static"]


def _newest_source() -> float:
    t = 0.0
    for root in (CSRC, os.path.join(os.path.dirname(HERE), "include")):
        for f in os.listdir(root):
            t = max(t, os.path.getmtime(os.path.join(root, f)))
    return t


def _run(cmd, verbose=False):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        sys.stderr.write(r.stderr)
    if r.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed:\n" + r.stdout + r.stderr)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OUT_DIR, exist_ok=True)
    src = _newest_source()
    if force or not os.path.exists(HOST) or os.path.getmtime(HOST) < src or not _host_loads():
        build_host()
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= src:
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    _run([nvcc, *NVCC_FLAGS, *(["-Xptxas", "-v"] if verbose else []), "-o", LIB,
          *[os.path.join(CSRC, s) for s in SOURCES]], verbose)
    return LIB


def _host_loads() -> bool:
    """whether the built host module is one for the installed torch"""
    from . import _lib
    try:
        _lib.load_host(HOST)
        return True
    except (ImportError, OSError, AttributeError):
        return False


def build_host() -> str:
    import sysconfig

    import torch
    t = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    _run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
          f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          f'-DHKV_TORCH_VERSION="{torch.__version__}"', f"-I{t}/include",
          f"-I{t}/include/torch/csrc/api/include", f"-I{sysconfig.get_paths()['include']}", f"-I{cuda}/include",
          os.path.join(CSRC, "hkv_host.cpp"), "-o", HOST, f"-L{t}/lib", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu",
          "-ltorch_python"])
    return HOST


if __name__ == "__main__":
    print(build(force=True, verbose="-v" in sys.argv))
