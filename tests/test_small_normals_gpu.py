"""generate_normals against Box-Muller on the same Philox words in extended precision:
12 units of 2^-53 relatively (9 for a radius next to 2^-6, three elsewhere:
tests/cxx/test_small_normals.cpp), for every normal, the smallest included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L = np.longdouble


def words(seed, m, groups, stream):
    """Philox4x32-10, counter (group, path low, path high, stream), key = seed."""
    low = np.uint64(0xFFFFFFFF)
    shape = (len(m), groups)
    c = [np.broadcast_to(np.arange(groups, dtype=np.uint64), shape), np.broadcast_to((m & low)[:, None], shape),
         np.broadcast_to((m >> np.uint64(32))[:, None], shape), np.full(shape, stream, np.uint64)]
    k = [np.uint64(seed & 0xFFFFFFFF), np.uint64(seed >> 32)]
    for _ in range(10):
        p, q = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(q >> np.uint64(32)) ^ c[1] ^ k[0], q & low, (p >> np.uint64(32)) ^ c[3] ^ k[1], p & low]
        k = [(k[0] + np.uint64(0x9E3779B9)) & low, (k[1] + np.uint64(0xBB67AE85)) & low]
    return np.stack(c, -1)


@pytest.mark.parametrize("N,M,streams", [(64, 20000, 2), (7, 1000, 3)])
def test_every_normal_keeps_its_bits(N, M, streams):
    import rbergomi_gb300 as R
    seed, pi = 77, L("3.14159265358979323846264338327950288")
    got = R.generate_normals(seed, M, N, streams=streams)
    for s in range(streams):
        w = words(seed, np.arange(M, dtype=np.uint64), (N + 3) // 4, s)
        q = (2 * w[..., 0::2] + np.uint64(1)).astype(np.int64)  # u0 = q 2^-33
        log = np.where(q >> 32, np.log1p((q - (1 << 33)).astype(L) / L(2 ** 33)), np.log(q.astype(L) / L(2 ** 33)))
        r, b = np.sqrt(-2 * log), w[..., 1::2]
        a = (2 * (b & np.uint64(0x3FFFFFFF)) + np.uint64(1)).astype(np.int64)  # angle a pi 2^-32 in its quadrant
        sn, cs = np.sin(pi * a.astype(L) / L(2 ** 32)), np.sin(pi * (2 ** 31 - a).astype(L) / L(2 ** 32))
        k = (b >> np.uint64(30)).astype(int)
        z = np.stack((r * np.choose(k, [cs, -sn, -cs, sn]), r * np.choose(k, [sn, cs, -sn, -cs])), -1).reshape(M, -1)[:, :N]
        off = np.abs(got[:, s].astype(L) / z - 1) * L(2 ** 53)
        assert off.max() < 12, float(off.max())
