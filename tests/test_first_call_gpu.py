"""The first call of a process on the allocation-free entry waits for its own
stream and no other: a host function that sleeps on another stream is still
running when the prices are back.  Modules load eagerly here, so that their
loading, which may wait for the device, is over before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = """
import ctypes as C
import numpy as np
import rbergomi_gb300 as R
L, dp = R.lib(), C.POINTER(C.c_double)
rt, usleep = C.CDLL("libcudart.so"), C.CDLL(None).usleep
L.rbg_price_rt_static.argtypes = [C.POINTER(R.RbgParams), C.POINTER(R.RbgOptions), dp, dp, dp]
p = R._Params(0.04, [0.1], [1.9], [-0.7], [1.0] * 3, [0.9, 1.0, 1.1], 64, 4096)
o = R.options(precision=R.MIXED, seed=1)
out = [np.empty(3) for _ in range(3)]
other = C.c_void_p()
assert rt.cudaStreamCreateWithFlags(C.byref(other), 1) == 0  # non-blocking
assert rt.cudaLaunchHostFunc(other, usleep, C.c_void_p(900000)) == 0
rc = L.rbg_price_rt_static(C.byref(p.s), C.byref(o), *[x.ctypes.data_as(dp) for x in out])
running = rt.cudaStreamQuery(other) == 600  # cudaErrorNotReady
rt.cudaDeviceSynchronize()
print("rc", rc, "other stream still running", running, "priced", bool(np.all(out[0] > 0)))
"""


def test_first_static_call_leaves_other_streams_alone():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=120,
                       env=dict(os.environ, CUDA_MODULE_LOADING="EAGER"))
    assert "rc 0 other stream still running True priced True" in r.stdout, r.stdout + r.stderr
