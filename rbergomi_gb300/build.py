"""Builds librbergomi_gb300.so in-tree with nvcc for sm_103a.

A small host program prints the fixed-point tables that one unit includes.  Each
translation unit compiles in parallel into rbergomi_gb300/_build/, then one nvcc
link produces rbergomi_gb300/librbergomi_gb300.so.  No cmake, no
torch extension machinery: the library is a plain C-ABI shared object.
"""
from __future__ import annotations

import os
import platform
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OUT_DIR = os.path.join(PKG, "_build")
LIB = os.path.join(PKG, "librbergomi_gb300.so")

ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC,
          "-I" + os.path.join(OUT_DIR, platform.machine())]
# by machine: the host's extended precision rounds the tables' last bit
TABLES = os.path.join(OUT_DIR, platform.machine(), "rbg_fixed_tables.inc")

SOURCES = ["rbg_plan.cpp", "rbg_api.cpp", "rbg_fp64.cu", "rbg_fp64x.cu", "rbg_mixed.cu", "rbg_fft.cu", "rbg_static.cu", "rbg_qmc.cu",
           "rbg_server.cpp", "rbg_cxx.cpp"]


def nvcc() -> str:
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(out: str, deps: list) -> bool:
    return not os.path.exists(out) or any(os.path.getmtime(out) < os.path.getmtime(d) for d in deps)


def _tables() -> None:
    """rbg_fixed_tables.inc, printed by rbg_tables_gen.cpp."""
    src, head = (os.path.join(CSRC, f) for f in ("rbg_tables_gen.cpp", "rbg_fixed.cuh"))
    if not _stale(TABLES, [src, head]):
        return
    os.makedirs(os.path.dirname(TABLES), exist_ok=True)
    exe = os.path.join(os.path.dirname(TABLES), "rbg_tables_gen")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + CSRC, src, "-o", exe], check=True)
    text = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    with open(TABLES + ".tmp", "w") as f:
        f.write(text)
    os.replace(TABLES + ".tmp", TABLES)


def _compile(src: str) -> str:
    obj = os.path.join(OUT_DIR, os.path.splitext(src)[0] + ".o")
    path = os.path.join(CSRC, src)
    deps = [path] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".hpp", ".cuh"))]
    deps += [os.path.join(ROOT, "include", h) for h in ("rbergomi_gb300.h", "rbergomi_gb300.hpp")]
    deps += [TABLES] if src == "rbg_fp64x.cu" else []
    if not _stale(obj, deps):
        return obj
    cmd = [nvcc()] + ARCH + COMMON + ["-c", path, "-o", obj]
    if src.endswith(".cu"):
        cmd += ["-Xptxas", "-v"] if os.environ.get("RBG_PTXAS_VERBOSE") else []
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f"nvcc failed on {src}")
    if r.stderr.strip():
        sys.stderr.write(r.stderr)
    return obj


def build(verbose: bool = False) -> str:
    os.makedirs(OUT_DIR, exist_ok=True)
    _tables()
    with ThreadPoolExecutor(max_workers=len(SOURCES)) as ex:
        objs = list(ex.map(_compile, SOURCES))
    if _stale(LIB, objs):
        cmd = [nvcc()] + ARCH + ["-shared", "-o", LIB] + objs + ["-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("nvcc link failed")
    if verbose:
        print("built", LIB)
    return LIB


if __name__ == "__main__":
    build(verbose=True)
