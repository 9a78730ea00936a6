"""The mixed form's producers draw Philox from per-launch entries (rounds 0 to 2
shared by all paths of one upper counter word): prices on their normals against
the payoffs of the same normals drawn by the counter's plain form, around path
2^32 where the upper word changes, in every pass mode.  The payoffs are the same
FP32 numbers; their sums differ in the order of FP32 additions (chunks of up to
256 values: eight levels of 2^-24, 5e-7; 1e-6 taken)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ARGS = (0.055, [0.1, 0.3], [1.9, 1.2], [-0.9, -0.4], [1.0, 0.5], [0.95, 1.05])


@pytest.fixture(scope="module")
def R():
    import rbergomi_gb300 as R
    return R


@pytest.mark.parametrize("off", [0, 2 ** 32 - 1, 2 ** 32 - 150, 2 ** 32, 5 * 2 ** 32 - 129])
@pytest.mark.parametrize("N", [1, 33, 512, 513, 1100])
@pytest.mark.parametrize("mc", [False, True])
def test_entries_are_the_counter_stream(R, off, N, mc):
    M, seed = 300, 2 ** 40 + 11
    price, payoffs = (R.price_mc, R.payoffs_mc) if mc else (R.price_rt, R.payoffs_rt)
    p = price(*ARGS, N, M, seed=seed, path_offset=off, precision=R.MIXED)[0]
    Z = R.generate_normals(seed, M, N, path_offset=off, precision=R.MIXED, **({"streams": 3} if mc else {}))
    q = payoffs(*ARGS, Z, precision=R.MIXED).mean(0)
    assert np.all(np.abs(p - q) <= 1e-6 * np.abs(q)), (p, q)


def test_shared_launches(R):
    """The serving loop's shared launch over requests of several seeds and offsets,
    one across path 2^32: as alone, but for the order of FP64 additions."""
    one = (0.055, [0.1], [1.9], [-0.9], [1.0] * 2, [0.95, 1.05])
    opts = [(3, 0), (2 ** 50 + 1, 2 ** 32 - 100), (7, 3 * 2 ** 32), (9, 2 ** 33 - 1)]
    with R.Server() as srv:
        tickets = [srv.submit(*one, 100 + 40 * i, 700, seed=a, path_offset=b) for i, (a, b) in enumerate(opts)]
        got = [srv.wait(t)[0] for t in tickets]
    for i, (a, b) in enumerate(opts):
        want = R.price_rt(*one, 100 + 40 * i, 700, seed=a, path_offset=b, precision=R.MIXED)[0]
        np.testing.assert_allclose(got[i], want, rtol=1e-12, atol=0)
