"""The FP64 form's conditional calls far out of the money, on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_far_tails(tmp_path):
    exe = str(tmp_path / "test_far_tails")
    subprocess.run(["g++", "-O2", "-std=c++17", "-x", "c++", "-I", os.path.join(ROOT, "rbergomi_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cxx", "test_far_tails.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
