"""Build liboa_gpu.so (sm_100a) in-tree with nvcc.

    python -m openatom_b200.build [--verbose]

The library is a plain C ABI (include/oa_gpu.h); Python loads it with ctypes.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "liboa_gpu.so")
SOURCES = ["oa_state.cu", "oa_pencil.cu", "oa_pp.cu", "oa_pp_f0.cu", "oa_pp_f1.cu", "oa_pp_f2.cu", "oa_pp_f3.cu", "oa_pp_d0.cu", "oa_pp_d1.cu", "oa_pp_d2.cu", "oa_pp_d3.cu", "oa_pp_ees_f.cu", "oa_pp_ees_d.cu", "oa_rho.cu", "oa_rho_zpass.cu", "oa_rho_zpass_f.cu", "oa_rho_pencil.cu", "oa_pc.cu", "oa_dgemm.cu", "oa_ns.cu", "oa_tgemm.cu", "oa_ozaki.cu", "oa_nl.cu", "oa_ions.cu", "oa_eesl.cu", "oa_step.cu", "oa_noalloc.cu", "oa_abi.cu"]
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def nvcc() -> str:
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if c and (os.path.isabs(c) and os.path.exists(c) or not os.path.isabs(c)):
            return c
    return "nvcc"


def build(verbose: bool = False, force: bool = False) -> str:
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    deps = srcs + [os.path.join(CSRC, h) for h in os.listdir(CSRC) if h.endswith((".cuh", ".h"))]
    deps.append(os.path.join(ROOT, "include", "oa_gpu.h"))
    if not force and os.path.exists(LIB):
        t = os.path.getmtime(LIB)
        if all(os.path.getmtime(d) <= t for d in deps):
            return LIB
    objdir = os.path.join(HERE, "_build")
    os.makedirs(objdir, exist_ok=True)
    flags = ARCH + ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "-rdc=false",
                    "-I", os.path.join(ROOT, "include"), "-I", CSRC]
    if verbose:
        flags += ["-Xptxas", "-v"]

    def compile_one(s):
        o = os.path.join(objdir, os.path.basename(s) + ".o")
        cmd = [nvcc()] + flags + ["-c", s, "-o", o]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
        if r.returncode:
            raise RuntimeError(f"nvcc failed on {s}")
        return o

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        objs = list(pool.map(compile_one, srcs))
    cmd = [nvcc()] + ARCH + ["-shared", "-o", LIB] + objs + ["-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("link failed")
    return LIB


if __name__ == "__main__":
    build(verbose="--verbose" in sys.argv, force=True)
    print(LIB)
