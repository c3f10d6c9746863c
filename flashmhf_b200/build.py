"""Build the native code in-tree: the C-ABI library with nvcc for sm_100a, and the torch host module with g++.

    python -m flashmhf_b200.build            # build what is older than its sources
    python -m flashmhf_b200.build --force

The outputs are flashmhf_b200/lib/libflashmhf_b200.so (kernels and C ABI, no torch types) and
flashmhf_b200/lib/_flashmhf_torch.so (the host path from torch tensors to that ABI).  nvcc cross-compiles without a GPU.
"""
import os
import subprocess
import sys
import sysconfig
import tempfile
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libflashmhf_b200.so")
TORCH_PATH = os.path.join(LIB_DIR, "_flashmhf_torch.so")
SOURCES = ["api.cu", "simt_check.cu", "tc_fwd.cu", "tc_bwd.cu", "prologue.cu", "lm_aux.cu", "selftest.cu"]
TORCH_SOURCE = "torch_host.cpp"
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]


def _header():
    return os.path.join(os.path.dirname(PKG), "include", "flashmhf.h")


def _stale(out, inputs):
    return not os.path.exists(out) or any(os.path.getmtime(f) > os.path.getmtime(out) for f in inputs)


def _lib_inputs():
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))] + [_header()]


def is_stale():
    return _stale(LIB_PATH, _lib_inputs()) or _stale(TORCH_PATH, [os.path.join(CSRC, TORCH_SOURCE), _header()])


def _run(cmd, verbose=False):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose:
        print(r.stderr)
    if r.returncode != 0:
        raise RuntimeError("compiler failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)


def _build_lib(tmp, verbose):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = [os.path.join(tmp, s + ".o") for s in SOURCES]
    flags = NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else [])
    with ThreadPoolExecutor(len(SOURCES)) as pool:
        jobs = [pool.submit(_run, [nvcc] + flags + ["-c", os.path.join(CSRC, s), "-o", o], verbose) for s, o in zip(SOURCES, objs)]
        for j in jobs:
            j.result()
    _run([nvcc] + NVCC_FLAGS + ["-shared", "-o", LIB_PATH] + objs)


def _build_torch_module():
    import torch
    from torch.utils import cpp_extension
    inc = cpp_extension.include_paths(device_type="cuda") + [sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_flashmhf_torch",
           "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
    for p in inc:
        cmd += ["-isystem", p]
    cmd += [os.path.join(CSRC, TORCH_SOURCE), "-o", TORCH_PATH, "-L" + os.path.join(os.path.dirname(torch.__file__), "lib")]
    _run(cmd + ["-lc10", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-lc10_cuda", "-ltorch_cuda"])


def build(force=False, verbose=False):
    os.makedirs(LIB_DIR, exist_ok=True)
    with tempfile.TemporaryDirectory() as tmp, ThreadPoolExecutor(2) as pool:
        jobs = []
        if force or _stale(LIB_PATH, _lib_inputs()):
            jobs.append(pool.submit(_build_lib, tmp, verbose))
        if force or _stale(TORCH_PATH, [os.path.join(CSRC, TORCH_SOURCE), _header()]):
            jobs.append(pool.submit(_build_torch_module))
        for j in jobs:
            j.result()
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
