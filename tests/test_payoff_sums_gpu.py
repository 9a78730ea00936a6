"""Chunk sums of the FP64 payoffs against exact sums (tests/cxx/test_payoff_sums.cpp).

A thread adds up at most 8 paths in one FP64 sum and everything above the warps' sums
is compensated.  In units of 2^-53 a rounding is 0.41 of the sum it ends in, root
mean square.  Eight additions in a row come to 0.72 of a thread's sum, 0.05 once
averaged over 256 threads; the five levels of a warp's tree to 0.57, 0.20 over 8
warps; both less by the root of the rounds of 8 paths a chunk has.  One FP64 sum of
the warps' alone would leave 0.7 whatever the chunk; with one path a thread it is all
there is, as each 256 paths' sum of a longer chunk was before it was compensated."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_chunk_sums_keep_what_plain_sums_lose(tmp_path):
    import rbergomi_gb300 as R
    exe, lib, cuda = str(tmp_path / "test_payoff_sums"), os.path.dirname(R.LIB_PATH), "/usr/local/cuda"
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "include"), "-I", f"{cuda}/include", "-I",
                    os.path.join(ROOT, "rbergomi_gb300", "csrc"), os.path.join(ROOT, "tests", "cxx", "test_payoff_sums.cpp"),
                    "-o", exe, "-L", lib, "-lrbergomi_gb300", f"-Wl,-rpath,{lib}", "-L", f"{cuda}/lib64", "-lcudart",
                    f"-Wl,-rpath,{cuda}/lib64"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) == 8
    for mc, G, rms, most in rows:
        limit = 0.2 if int(G) > 9 else 0.35 if int(G) > 1 else 1.0
        assert float(rms) < limit, r.stdout
