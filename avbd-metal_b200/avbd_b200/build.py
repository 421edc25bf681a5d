"""Build the CUDA solver library in-tree for sm_100a.

The library is a plain shared object with the C ABI of include/avbd.h; the
Python package loads it with ctypes.  Solver kernels are compiled with
-fmad=false (no multiply-add contraction) and IEEE division/sqrt, host code
with -ffp-contract=off, so results are reproducible bit for bit.
"""
import glob
import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(ROOT, "csrc")
LIBDIR = os.path.join(PKG, "_lib")
LIB = os.path.join(LIBDIR, "libavbd_b200.so")
NVCC = os.environ.get("NVCC", "nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cpp")))


def headers():
    return (glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh"))
            + [os.path.join(os.path.dirname(ROOT), "include", "avbd.h")])


def up_to_date() -> bool:
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    return all(os.path.getmtime(f) <= t for f in sources() + headers())


def compile_report(source: str) -> str:
    """What ptxas said of a source's kernels (registers, stack frames, spills)
    when it was last compiled."""
    path = os.path.join(LIBDIR, "obj", source + ".ptxas")
    if not os.path.exists(path) or not up_to_date():
        build(force=True)
    with open(path) as f:
        return f.read()


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    os.makedirs(LIBDIR, exist_ok=True)
    objdir = os.path.join(LIBDIR, "obj")
    os.makedirs(objdir, exist_ok=True)
    objs = []
    common = ["-O3", "-std=c++17", "-lineinfo", "-fmad=false", "-prec-div=true", "-prec-sqrt=true",
              "-Xcompiler", "-fPIC,-ffp-contract=off,-fno-fast-math", "-Xptxas", "-v", "-I", CSRC]
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src) + ".o")
        cmd = [NVCC] + ARCH + common + ["-c", src, "-o", obj]
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        done = subprocess.run(cmd, stderr=subprocess.PIPE, text=True)
        sys.stderr.writelines(line + "\n" for line in done.stderr.splitlines()
                              if done.returncode or "warning" in line)
        done.check_returncode()
        with open(os.path.join(objdir, os.path.basename(src) + ".ptxas"), "w") as f:
            f.write(done.stderr)
        objs.append(obj)
    cmd = [NVCC] + ARCH + ["-shared", "-cudart", "static", "-o", LIB] + objs
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
