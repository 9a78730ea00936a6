"""The FP64 form's 64-bit fixed-point functions on the host, and the digit
convolution's layout: a model of the digits, panels and MMA operands as the
kernels write and read them, against the direct sum."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fixed_point_functions(tmp_path):
    exe = str(tmp_path / "test_fixed")
    subprocess.run(["g++", "-O2", "-std=c++17", "-x", "c++", "-I", os.path.join(ROOT, "rbergomi_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cxx", "test_fixed.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


# k_normals_fixed / k_panels / k_volterra_exact: 64 paths, 16-step chunks, 8
# digits, panels of 240 rows, K-major SW32 rows of 32 bytes
P, PANEL_ROWS = 64, 240
PANEL_DIGIT, CHUNK = PANEL_ROWS * 32, 8 * P * 32
PANEL = 8 * PANEL_DIGIT


def digits(v):
    u = [(int(x) + 0x8080808080808080) % (1 << 64) for x in v.ravel()]
    return np.array([[((x >> (8 * (7 - d))) & 255) - 128 for d in range(8)] for x in u], np.int64).reshape(v.shape + (8,))


def read_rows(buf, start, n):
    """n rows of 16 values from a 256-byte aligned address: 16-byte halves swapped by address bit 7."""
    assert start % 256 == 0 and start + 32 * n <= 2 * buf.size
    a = start + 32 * np.arange(n)[:, None] + 16 * (np.arange(2)[None, :] ^ ((start + 32 * np.arange(n)[:, None]) >> 7 & 1))
    return buf[a[:, :, None] // 2 + np.arange(8)].reshape(n, 16)


@pytest.mark.parametrize("N,B", [(2, 3), (16, 64), (17, 65), (100, 20), (128, 9), (129, 9), (300, 5)])
def test_digit_convolution_layout(N, B):
    rng = np.random.default_rng(N)
    W, G = rng.integers(-2 ** 62, 2 ** 62, (B, N)), rng.integers(-2 ** 61, 2 ** 62, N)
    dW, dG = digits(W), digits(G)
    nb, nch, groups = -(-N // 128), -(-N // 16), -(-B // P)
    dig = np.full(groups * nch * CHUNK // 2, 999)
    for m in range(groups * P):
        for c in range(nch):
            for g in range(4):
                at = ((m // P) * nch + c) * CHUNK + (m % P) * 32 + ((((g >> 1) ^ (m >> 2)) & 1) << 4) + ((g & 1) << 3)
                for q in range(4):
                    j = 16 * c + 4 * g + q
                    dig[at // 2 + q + 16 * P * np.arange(8)] = dW[m, j] if m < B and j < N else 0
    pan = np.full(nb * PANEL // 2, 999)
    for L in range(nb):
        for r in range(PANEL_ROWS):
            for half in range(2):
                at = L * PANEL + r * 32 + ((half ^ (r >> 2)) & 1) * 16
                for i in range(8):
                    d = 128 * L + r - 112 - (8 * half + i)
                    pan[at // 2 + i + PANEL_DIGIT // 2 * np.arange(8)] = dG[d] if 0 <= d < N else 0
    assert not (dig == 999).any() and not (pan == 999).any()  # every byte the MMAs read is written
    for grp in range(groups):
        for b in range(nb):
            D = np.zeros((128, 512), np.int64)
            for kc in range(min(8 * (b + 1), nch)):
                st = (grp * nch + kc) * CHUNK
                for j in range(8):
                    A = read_rows(pan, (b - kc // 8) * PANEL + j * PANEL_DIGIT + (7 - kc % 8) * 512, 128)
                    n = 64 * (8 - j)
                    n1 = min(n, 256)
                    D[:, 64 * j:64 * j + n1] += A @ read_rows(dig, st, n1).T
                    if n > 256:
                        D[:, 64 * j + 256:64 * j + n] += A @ read_rows(dig, st + 8192, n - 256).T
            assert np.abs(D).max() < 2 ** 22
            for m in range(grp * P, min(B, grp * P + P)):
                for j in range(128 * b, min(N, 128 * b + 128)):
                    got = sum(int(D[j - 128 * b, 64 * d + m % P]) << (8 * (7 - d)) for d in range(8))
                    want = sum(int(W[m, k]) * int(G[j - k]) for k in range(j + 1))
                    # the products of digits with i + j >= 8, below 8 x 128^2 a term
                    assert abs(got - want / 2 ** 56) < 8 * 128 ** 2 * (j + 1)
