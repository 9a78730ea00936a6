"""The path pass that the profile names is the one that ran, with its launches: one
kernel each, or pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,groups,name,launches", [
    (dict(N=64), 1, "k_volterra_exact + k_slot_sums", 2), (dict(N=64), 4, "k_volterra_exact + k_variance_fixed", 2),
    (dict(N=300, conv=2), 1, "k_path_fp64_fft", 1), (dict(N=300, conv=3), 1, "k_path_fp64", 1),
    (dict(N=300, eta=1e5), 1, "k_path_fp64_fft", 1), (dict(N=5000), 1, "k_path_fp64", 1)])
def test_profile_names_the_path_pass(kw, groups, name, launches):
    import rbergomi_gb300 as R
    N, eta = kw["N"], kw.get("eta", 1.5)
    R.profile_reset()
    R.profile_enable(True)
    try:
        R.price_rt(0.04, [0.1], [eta], [-0.7], np.linspace(0.5, 2.0, groups), np.ones(groups), N, 300, conv=kw.get("conv", 0))
        assert R.profile_path() == name
        assert R.profile_read(R.STAGE_PATH_FP64)[1] == launches
    finally:
        R.profile_enable(False)
        R.profile_reset()
