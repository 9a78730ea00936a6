"""The FP64 normals a caller asks for keep their significant bits however small."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_small_normals(tmp_path):
    exe = str(tmp_path / "test_small_normals")
    subprocess.run(["g++", "-O2", "-std=c++17", "-x", "c++", "-I", os.path.join(ROOT, "rbergomi_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cxx", "test_small_normals.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
