"""Build recipe of the CUDA library (libb200tp.so) for sm_100a and of the torch binding (_b2torch.so) over it.

nvcc cross-compiles without a GPU.  Both are built in-tree under
nano-vllm_b200/lib/ so that they travel with the source tree.
"""
from __future__ import annotations

import hashlib
import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIBDIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIBDIR, "libb200tp.so")
BINDING = os.path.join(LIBDIR, "_b2torch.so")
BINDING_SOURCE = "b2_torch.cpp"
SOURCES = ["b2_ctx.cu", "b2_elementwise.cu", "b2_attention.cu", "b2_stack.cu", "b2_gemm_tile.cu", "b2_gemm.cu"]
HEADERS = ["b2_common.cuh", os.path.join("..", "..", "include", "b200tp.h")]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17"]


def _stamp() -> str:
    h = hashlib.sha256()
    for name in SOURCES + HEADERS + [BINDING_SOURCE]:
        with open(os.path.join(CSRC, name), "rb") as f:
            h.update(f.read())
    h.update(" ".join(NVCC_FLAGS).encode())
    return h.hexdigest()


def _binding_command() -> list[str]:
    """g++ command of the torch binding: it calls the C ABI (found beside it) and torch's C++ tensors."""
    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            os.path.join(CSRC, BINDING_SOURCE), "-o", BINDING, "-I" + sysconfig.get_paths()["include"],
            "-isystem", os.path.join(base, "include"), "-isystem", os.path.join(base, "include", "torch", "csrc", "api", "include"),
            "-isystem", os.path.join(cuda, "include"), "-L" + LIBDIR, "-L" + os.path.join(base, "lib"), "-Wl,-rpath,$ORIGIN",
            "-l:libb200tp.so", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu into objects, link the shared library, compile the torch binding; returns the library's path."""
    os.makedirs(LIBDIR, exist_ok=True)
    stamp_file = os.path.join(LIBDIR, "build.stamp")
    stamp = _stamp()
    if not force and os.path.exists(LIB) and os.path.exists(BINDING) and os.path.exists(stamp_file) and open(stamp_file).read() == stamp:
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(LIBDIR, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, "-Xcompiler", "-fPIC", "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
    cmd = [nvcc, "-shared", "-Wno-deprecated-gpu-targets", "-o", LIB, *objs, "-lcudart"]
    subprocess.check_call(cmd)
    subprocess.check_call(_binding_command())
    with open(stamp_file, "w") as f:
        f.write(stamp)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
