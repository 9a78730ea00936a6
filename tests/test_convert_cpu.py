"""double_to_float, the integer form of FP64 -> FP32 in the mixed form's
caller-normals producer, against the compiler's conversion."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_double_to_float(tmp_path):
    exe = str(tmp_path / "test_convert")
    subprocess.run(["g++", "-O2", "-std=c++17", "-x", "c++", "-I", os.path.join(ROOT, "rbergomi_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cxx", "test_convert.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[:2000]
