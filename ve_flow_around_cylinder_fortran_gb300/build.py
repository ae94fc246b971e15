"""Build libvefem.so (sm_103a) in-tree with nvcc.

Every translation unit is compiled with ``-fmad=false`` and the host code
with ``-ffp-contract=off``: the FP64 assembly must evaluate the reference's
expressions as separately rounded IEEE operations, in source order, for its
results to match the sequential algorithm bit for bit.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OUT = os.path.join(PKG, "_build")
LIB = os.path.join(OUT, "libvefem.so")
PROBE = os.path.join(OUT, "libvefem_probe.so")
INCLUDE = os.path.join(ROOT, "include")

SOURCES = ["vefem_fd64.cu", "vefem_gather.cu", "vefem_capi.cu", "vefem_opcount.cpp",
           "vefem_noalloc.cu", "vefem_exact.cu", "vefem_mlp.cu", "vefem_batch.cu",
           "vefem_stability.cu", "vefem_frontal.cu", "vefem_tree.cu"]
# the exact-Jacobian, network, linear-solver and stability kernels are not held to bit-exactness:
# FMA contraction allowed
FMAD_ON = {"vefem_exact.cu", "vefem_mlp.cu", "vefem_frontal.cu", "vefem_tree.cu", "vefem_stability.cu"}
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _flags(src: str = ""):
    fmad = "-fmad=true" if src in FMAD_ON else "-fmad=false"
    return ARCH + ["-split-compile=0", "-O3", "-lineinfo", "-std=c++17", fmad, "-Xcompiler", "-fPIC",
                   "-Xcompiler", "-ffp-contract=off", "-I", INCLUDE, "-I", CSRC]


def _deps():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    files.append(os.path.join(INCLUDE, "vefem.h"))
    files.append(os.path.abspath(__file__))
    return files


def up_to_date() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(PROBE):
        return False
    t = os.path.getmtime(LIB)
    return all(os.path.getmtime(f) <= t for f in _deps())


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    os.makedirs(OUT, exist_ok=True)
    cc = nvcc()
    procs = []
    objs = []
    for src in SOURCES:
        obj = os.path.join(OUT, os.path.splitext(src)[0] + ".o")
        objs.append(obj)
        cmd = [cc] + _flags(src) + (["-Xptxas", "-v"] if verbose else []) + \
            ["-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT)))
    failed = False
    for cmd, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(out.decode(errors="replace"))
        if p.returncode != 0:
            sys.stderr.write("FAILED: " + " ".join(cmd) + "\n")
            failed = True
    if failed:
        raise RuntimeError("nvcc compilation failed")
    tmp = LIB + ".tmp"
    subprocess.check_call([cc] + ARCH + ["-shared", "-o", tmp] + objs)
    os.replace(tmp, LIB)
    # the FP64 peak probe used by the benchmark (not part of the assembly ABI)
    ptmp = PROBE + ".tmp"
    subprocess.check_call([cc] + _flags() + ["-shared", "-o", ptmp,
                                             os.path.join(CSRC, "vefem_probe.cu")])
    os.replace(ptmp, PROBE)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
