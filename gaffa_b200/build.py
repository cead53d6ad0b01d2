"""Builds libgaffa_b200.so in-tree from gaffa_b200/csrc with nvcc for sm_100a.

Usage: python -m gaffa_b200.build   (or gaffa_b200.build.build())
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
BUILD = PKG / "_build"
LIB = PKG / "libgaffa_b200.so"
SOURCES = ["host.cpp", "dedisperse.cu", "dedisperse_mma.cu", "preprocess.cu", "ffa.cu", "fold.cu", "synth.cu", "filterbank.cu", "proposal.cu", "candidates.cu", "harmonics.cu"]
# ffa_search.cu is compiled in parts, each an object (PARTS: macro, count).  No
# --split-compile: its output differs from run to run, and with it the speed of
# the dedispersion kernels, by up to 10 %.
PARTS = {"ffa_search.cu": ("GF_FFA_PART", 8)}
# gaffa's C++ API (include/gaffa/*.h) over the C ABI: plain C++20 host code
CXX_SOURCES = ["cxx_api.cpp"]
CXX_FLAGS = ["-std=c++20", "-O2", "-fPIC", "-ffp-contract=off", "-Wall", "-Wextra", f"-I{ROOT / 'include'}",
             "-I/usr/local/cuda/include"]

NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC,-O2,-ffp-contract=off",
    "--expt-relaxed-constexpr",
    f"-I{ROOT / 'include'}", f"-I{CSRC}",
]


def _nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found")


def _compile(src: Path, obj: Path, defines=()) -> None:
    if src.name in CXX_SOURCES:
        cmd = [shutil.which("g++") or "g++", *CXX_FLAGS, "-c", str(src), "-o", str(obj)]
    else:
        cmd = [_nvcc(), *NVCC_FLAGS, *defines, "-x", "cu", "-c", str(src), "-o", str(obj)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"compile failed for {src.name}:\n{r.stderr}")


def build(force: bool = False, verbose: bool = False) -> Path:
    BUILD.mkdir(exist_ok=True)
    units = [(CSRC / s, BUILD / (s + ".o"), ()) for s in SOURCES + CXX_SOURCES]
    # the longest first
    units = [(CSRC / s, BUILD / f"{s}.{k}.o", (f"-D{macro}={k}",))
             for s, (macro, n) in PARTS.items() for k in reversed(range(n))] + units
    headers = list(CSRC.glob("*.cuh")) + [ROOT / "include" / "gaffa_b200.h"] + list((ROOT / "include" / "gaffa").glob("*.h"))
    newest_header = max(h.stat().st_mtime for h in headers)
    objs = [obj for _, obj, _ in units]
    jobs = [u for u in units
            if force or not u[1].exists() or u[1].stat().st_mtime < max(u[0].stat().st_mtime, newest_header)]
    with cf.ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4) or 1) as ex:
        for f in [ex.submit(_compile, *u) for u in jobs]:
            f.result()
    if force or jobs or not LIB.exists():
        cmd = [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static",
               "-o", str(LIB), *map(str, objs)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stderr}")
    if verbose:
        print(f"built {LIB}")
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
