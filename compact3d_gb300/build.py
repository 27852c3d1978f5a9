"""Build of libc3d.so, the sm_103a CUDA library behind include/c3d.h.

Each translation unit is compiled by nvcc in parallel (one -gencode, sm_103a) and linked
into an in-tree shared library ``compact3d_gb300/libc3d.so``.  No PyTorch, CMake or
Python extension machinery is involved: the library is a plain C-ABI .so.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libc3d.so")
SOURCES = ["c3d_capi.cu", "c3d_step.cu", "c3d_xpass.cu", "c3d_xbatch.cu", "c3d_zpass.cu", "c3d_spec.cu", "c3d_noalloc.cu", "c3d_les.cu", "c3d_ops.cu", "c3d_refine.cu", "c3d_ckpt.cu", "c3d_stats.cu", "c3d_iwm.cu"]
# the kernels of both precisions, compiled once for each (C3D_BITS), which halves the build
SPLIT = {"c3d_xpass.cu", "c3d_xbatch.cu", "c3d_zpass.cu"}
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def flags(extra=()) -> list[str]:
    return ARCH + ["-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr",
                   "-Xcompiler", "-fPIC", "-Xptxas", "-O3"] + list(extra)


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False, ptxas_v: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "c3d.h"))
    nv = nvcc()
    jobs = []
    objs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        for bits in ((32, 64) if src in SPLIT else (None,)):
            o = os.path.join(OBJ, src.replace(".cu", f"_{bits}.o" if bits else ".o"))
            objs.append(o)
            if force or _stale(o, [s] + headers):
                extra = (["-Xptxas", "-v"] if ptxas_v else []) + ([f"-DC3D_BITS={bits}"] if bits else [])
                jobs.append([nv] + flags(extra) + ["-c", s, "-o", o])
    if jobs:
        with cf.ThreadPoolExecutor(max_workers=len(jobs)) as ex:
            futs = [ex.submit(subprocess.run, j, capture_output=True, text=True) for j in jobs]
            for j, f in zip(jobs, futs):
                r = f.result()
                if verbose or r.returncode != 0 or ptxas_v:
                    sys.stderr.write(r.stdout + r.stderr)
                if r.returncode != 0:
                    raise RuntimeError("nvcc failed: " + " ".join(j))
    if force or jobs or _stale(LIB, objs):
        cmd = [nv] + ARCH + ["-shared", "-o", LIB + ".tmp"] + objs + ["-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
        os.replace(LIB + ".tmp", LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True, ptxas_v="-v" in sys.argv)
    print(LIB)
