"""In-tree build of the C-ABI library (``libtdb_b200.so``) with nvcc for sm_100a, and of the host extension (``_host.so``)
that the Python operators call."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libtdb_b200.so")
HOST = os.path.join(HERE, "_host.so")
HOST_SOURCES = ["host_ops.cpp"]
SOURCES = ["tdb_api.cu", "tables.cu", "attn_simt.cu", "attn_scores.cu", "attn_small.cu", "attn_umma.cu", "attn_far.cu", "relpos_umma.cu", "encoder.cu", "skinny.cu", "encoder_short.cu"]
HEADERS = ["tdb_internal.h", "ptx_sm100.cuh", "attn_common.cuh", "gelu.cuh", "attn_blocks.cuh", "attn_warp_mma.cuh", os.path.join("..", "..", "include", "tdb_b200.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden"]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; the library must be built where the CUDA toolkit is installed")
    return cand


def needs_build(target: str = LIB, sources=None) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    deps = [os.path.join(CSRC, s) for s in (sources or SOURCES)] + [os.path.normpath(os.path.join(CSRC, h)) for h in HEADERS]
    return any(os.path.getmtime(d) > t for d in deps)


def build_host(verbose: bool = False) -> str:
    """Compile the host extension against torch's headers; it links against the library next to it."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ext
    gxx = shutil.which("g++")
    if gxx is None:
        raise RuntimeError("g++ not found")
    cuda_home = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    inc = [*ext.include_paths(), sysconfig.get_path("include"), os.path.join(cuda_home, "include"), CSRC]
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [gxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *[f"-I{i}" for i in inc], *[os.path.join(CSRC, s) for s in HOST_SOURCES], "-o", HOST,
           f"-L{HERE}", "-l:libtdb_b200.so", "-Wl,-rpath,$ORIGIN", f"-L{torch_lib}", "-ltorch_python", "-ltorch",
           "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", f"-L{os.path.join(cuda_home, 'lib64')}", "-lcudart",
           "-lcublasLt"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if verbose or r.returncode:
        sys.stderr.write(r.stdout)
    if r.returncode:
        raise RuntimeError("g++ failed on the host extension")
    return HOST


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every translation unit for sm_100a and link the shared library next to this file; then the host extension."""
    if force or needs_build():
        _build_lib(verbose)
    if force or needs_build(HOST, HOST_SOURCES):
        build_host(verbose)
    return LIB


def _build_lib(verbose: bool) -> None:
    nvcc = _nvcc()
    objs = []
    flags = list(NVCC_FLAGS)
    if verbose:
        flags = flags + ["-Xptxas", "-v"]
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = os.path.join(HERE, "build", src.replace(".cu", ".o"))
        cmd = [nvcc, *flags, "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode:
            sys.stderr.write(out)
        if pr.returncode:
            raise RuntimeError(f"nvcc failed on {src}")
    cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
    subprocess.run(cmd, check=True)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
