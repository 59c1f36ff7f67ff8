"""Build libsoliton_b200.so in-tree for sm_100a.

    python -m soliton_solver_b200.build            # build if sources changed
    python -m soliton_solver_b200.build --force    # rebuild

The library is written to ``soliton_solver_b200/_lib/libsoliton_b200.so`` next to
the sources so that it travels with the checkout; nothing is installed elsewhere.
"""
from __future__ import annotations

import argparse
import concurrent.futures
import os
import shutil
import subprocess
import sys
import tempfile

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(ROOT, "include")
LIBDIR = os.path.join(PKG, "_lib")
LIB = os.path.join(LIBDIR, "libsoliton_b200.so")
SOURCES = ["abi.cu", "coop.cu", "batch.cu", "plain.cu"]
# --split-compile generates other code.  The FP32 step of plain rows gains by it (ten steps of 2000 x 1999,
# chiral magnet 2864 against 3215 us, Higgs 3378 against 3606); gradients and densities lose up to 14%
UNIT_FLAGS = {"plain.cu": ["--split-compile=0"]}
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA toolkit is required to build libsoliton_b200")


def _inputs():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))]
    files += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE) if f.endswith(".h")]
    files.append(os.path.abspath(__file__))
    return files


def up_to_date() -> bool:
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    return all(os.path.getmtime(f) <= t for f in _inputs())


def build(force: bool = False, verbose: bool = False, ptxas_verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    os.makedirs(LIBDIR, exist_ok=True)
    common = [_nvcc(), *ARCH, "-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC",
              "-cudart", "shared", "-I", INCLUDE, "-I", CSRC]
    if ptxas_verbose:
        common += ["-Xptxas", "-v"]
    with tempfile.TemporaryDirectory(dir=LIBDIR) as tmp:
        objects = [os.path.join(tmp, s + ".o") for s in SOURCES]
        cmds = [[*common, *UNIT_FLAGS.get(s, []), "-c", "-o", o, os.path.join(CSRC, s)] for s, o in zip(SOURCES, objects)]
        with concurrent.futures.ThreadPoolExecutor(len(cmds)) as pool:
            list(pool.map(lambda c: _run(c, verbose, ptxas_verbose), cmds))
        out = os.path.join(tmp, "lib.so")
        _run([*common, "-shared", "-Xlinker", "-rpath,/usr/local/cuda/lib64", "-o", out, *objects], verbose, ptxas_verbose)
        os.replace(out, LIB)
    return LIB


def _run(cmd, verbose, show):
    if verbose:
        print(" ".join(cmd), flush=True)
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError("nvcc failed building libsoliton_b200")
    if show or verbose:
        sys.stderr.write(res.stderr)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("-v", "--verbose", action="store_true")
    ap.add_argument("--ptxas", action="store_true", help="print register / shared-memory usage")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose, ptxas_verbose=a.ptxas))


if __name__ == "__main__":
    main()
