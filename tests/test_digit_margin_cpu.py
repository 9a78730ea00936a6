"""How far the digit convolution's accumulators stay from their limits, from the
plan's own Gamma, and the read-out chosen by it (host code of the library)."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_digit_margin(tmp_path):
    import rbergomi_gb300 as R
    from rbergomi_gb300 import build
    build.build()
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    exe, lib = str(tmp_path / "test_digit_margin"), os.path.dirname(R.LIB_PATH)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I", f"{cuda}/include", "-I",
                        os.path.join(ROOT, "rbergomi_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cxx", "test_digit_margin.cpp"), "-o", exe, "-L", lib,
                        "-lrbergomi_gb300", f"-Wl,-rpath,{lib}", f"-Wl,-rpath-link,{cuda}/lib64"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
