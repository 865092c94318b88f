"""Build libonecomp_b200.so in-tree with nvcc for sm_100a.

    python -m onecompression_b200.build

The library has no dependency beyond the CUDA runtime; the host side loads it
with ctypes (see ``_lib.py``).
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libonecomp_b200.so")

# file -> extra flags.  gptq.cu must not contract a*b-c into an FMA.
SOURCES = {
    "errors.cu": [],
    "gemm.cu": [],
    "gemm_tc.cu": [],
    "gemm_split.cu": [],
    "split.cu": [],
    "factor.cu": [],
    "gptq.cu": ["-fmad=false"],
    "moment_simt.cu": [],
    "moment_tc.cu": [],
    "moment_tc2.cu": [],
    "moment_noalloc.cu": [],
    "pack.cu": [],
    "packed_linear.cu": [],
    "qep.cu": [],
    "rtn.cu": ["-fmad=false"],
    "rmsnorm.cu": [],
    "blockops.cu": ["-fmad=false"],
}

BASE = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA kernels cannot be built")
    return exe


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    objs = []
    procs = []
    for src, extra in SOURCES.items():
        path = os.path.join(CSRC, src)
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(obj, [path] + headers + [os.path.abspath(__file__)]):
            cmd = [nvcc] + BASE + extra + (["-Xptxas", "-v"] if verbose else []) + ["-c", path, "-o", obj]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out.decode())
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
    if force or procs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
        subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
