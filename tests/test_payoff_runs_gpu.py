"""FP32 payoff sums where one block takes several runs of 8 outputs (large
output counts): each output's sums are those of a call that prices it alone,
bit for bit -- the same paths, chunks and order of additions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def R():
    import rbergomi_gb300 as R
    return R


@pytest.mark.parametrize("mc", [False, True])
@pytest.mark.parametrize("M", [131072, 131072 - 77])  # 512 chunks: blocks of up to four runs from 80 outputs on
@pytest.mark.parametrize("n", [1, 8, 9, 79, 81, 161, 330])  # partial runs, partial blocks
def test_outputs_do_not_depend_on_their_neighbours(R, n, M, mc):
    price = R.price_mc if mc else R.price_rt
    K = np.linspace(0.7, 1.3, n) if n > 1 else np.array([1.0])
    T = np.where(np.arange(n) % 3 == 0, 0.5, 1.25)  # variance groups alternate inside a run
    opts = dict(precision=R.MIXED, seed=5, compute_iv=False)
    p, s, _ = price(0.04, [0.1], [1.9], [-0.7], T, K, 32, M, **opts)
    for i in sorted({0, n // 2, n - 1, min(n - 1, 8), min(n - 1, 31), min(n - 1, 32)}):
        p1, s1, _ = price(0.04, [0.1], [1.9], [-0.7], T[i:i + 1], K[i:i + 1], 32, M, **opts)
        assert p[i] == p1[0] and s[i] == s1[0]
