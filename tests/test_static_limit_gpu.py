"""The largest jobs of the allocation-free entry: what its 16 MiB hold is the jobs'
own tables and buffers.  Numbers of distinct H that just fit at a step count (one
more is refused), against the regular entry."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n", [(256, 473), (320, 382), (800, 293), (832, 283), (2048, 118)])
def test_largest_jobs_fit(N, n):
    import rbergomi_gb300 as R
    L, dp = R.lib(), C.POINTER(C.c_double)
    L.rbg_price_rt_static.argtypes = [C.POINTER(R.RbgParams), C.POINTER(R.RbgOptions), dp, dp, dp]

    def price(k):
        args = (0.04, np.linspace(0.05, 0.45, k), np.full(k, 1.5), np.full(k, -0.7), [1.0], [1.0], N, 128)
        p, o = R._Params(*args), R.options(precision=R.MIXED, seed=1)
        out = [np.empty(k) for _ in range(3)]
        return L.rbg_price_rt_static(C.byref(p.s), C.byref(o), *[x.ctypes.data_as(dp) for x in out]), out[0], args

    rc, got, args = price(n)
    assert rc == 0
    # 512 < N <= 1024: another kernel there, 2e-6 (tests/test_zz_no_alloc.py)
    np.testing.assert_allclose(got, R.price_rt(*args, seed=1, precision=R.MIXED)[0], rtol=2e-6 if 512 < N <= 1024 else 1e-12)
    assert price(n + 1)[0] != 0
