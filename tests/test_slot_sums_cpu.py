"""The fused variance pass's integer sums of 32 steps on the host: unbiased whatever
the number of live steps (the last sum of a path has N - 1 modulo 32)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_slot_sums(tmp_path):
    exe = str(tmp_path / "test_slot_sums")
    subprocess.run(["g++", "-O2", "-std=c++17", "-x", "c++", "-I", os.path.join(ROOT, "rbergomi_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cxx", "test_slot_sums.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
