"""The fused variance pass leaves no bias in the sums of sqrt(v) dW: prices at a strike
next to zero (the mean of the terminal price) against the FP64 kernels' on the same
normals, averaged over 40 draws of 20000 paths, to half a unit of 2^-53, the last
bit of a price below one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mc", [False, True])
@pytest.mark.parametrize("N", [33, 250, 1000])
def test_no_bias_in_the_sums(N, mc):
    import rbergomi_gb300 as R
    price = R.price_mc if mc else R.price_rt
    d = []
    for seed in range(40):
        args = (0.09, [0.1 + 0.005 * seed], [1.9], [-0.9], [1.0], [1e-3], N, 20000)
        p, q = price(*args, seed=seed)[0][0], price(*args, seed=seed, conv=R.CONV_DIRECT)[0][0]
        d.append((p / q - 1.0) * 2.0 ** 53 if p != q else 0.0)
    assert abs(np.mean(d)) < 0.5, np.mean(d)
