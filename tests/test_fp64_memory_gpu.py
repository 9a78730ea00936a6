"""Device memory of the FP64 form's digit convolution: calls whose other buffers fit
still run where its digits, sums or panels do not, on the FP64 kernels and with
their results bit for bit.  Every free byte but a stated number is held by the test
meanwhile."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture(scope="module")
def R():
    import rbergomi_gb300 as R
    R.lib()
    return R


def free_bytes():
    free, total = C.c_size_t(), C.c_size_t()
    assert C.CDLL("libcudart.so").cudaMemGetInfo(C.byref(free), C.byref(total)) == 0
    return free.value


class Leave:
    """All device memory but `mb` MB held from here on."""

    def __init__(self, R, mb):
        # a call of each form first: kernels and modules are loaded
        for conv in (R.CONV_AUTO, R.CONV_DIRECT):
            R.price_rt(0.04, [0.1], [1.5], [-0.7], [1.0], [1.0], 64, 500, conv=conv)
        R.release()
        self.rt, self.mb, self.p = C.CDLL("libcudart.so"), mb, C.c_void_p()

    def __enter__(self):
        n = free_bytes() - self.mb * MB
        if n > 0:
            assert self.rt.cudaMalloc(C.byref(self.p), C.c_size_t(n)) == 0
        return self

    def __exit__(self, *exc):
        self.rt.cudaFree(self.p)


def test_no_room_for_the_digits(R):
    args = (0.04, [0.1], [1.5], [-0.7], [1.0], [1.0], 128, 1 << 18)  # 512 MB normals, 512 MB digits
    with Leave(R, 800):
        got = R.price_rt(*args, seed=1)
    R.release()
    want = R.price_rt(*args, seed=1, conv=R.CONV_DIRECT)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_no_room_for_the_panels(R):
    n = 3000  # 184 MB of panels, 60 KB a pass
    args = (0.04, np.linspace(0.05, 0.45, n), np.full(n, 1.5), np.full(n, -0.7), [1.0], [1.0], 100, 256)
    with Leave(R, 170):
        got = R.price_rt(*args, seed=1)
    R.release()
    want = R.price_rt(*args, seed=1, conv=R.CONV_DIRECT)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_digits_leave_room_for_what_every_form_needs(R):
    K = np.linspace(0.8, 1.2, 20000)  # 64 MB normals, 320 MB and more of chunk sums; 80 MB digits and sums
    args = (0.04, [0.1], [1.5], [-0.7], np.full(20000, 1.0), K, 16, 1 << 18)
    with Leave(R, 2000):
        want = R.price_rt(*args, seed=1, conv=R.CONV_DIRECT)
        used = 2000 * MB - free_bytes()
    with Leave(R, used // MB + 40):
        got = R.price_rt(*args, seed=1)
    R.release()
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_an_earlier_calls_digits_make_room(R):
    args = (0.04, [0.1], [1.5], [-0.7], [1.0], [1.0], 128)
    with Leave(R, 1300):
        R.price_rt(*args, 1 << 18, seed=1)  # leaves 512 MB of normals and 512 MB of digits
        got = R.price_rt(*args, 1 << 19, seed=1, conv=R.CONV_DIRECT)  # 1 GB of normals
    R.release()
    want = R.price_rt(*args, 1 << 19, seed=1, conv=R.CONV_DIRECT)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_no_room_for_the_digits_of_callers_normals(R):
    Z = np.random.default_rng(3).standard_normal((1 << 17, 2, 128))  # 256 MB, as much of digits
    args = (0.04, [0.1], [1.5], [-0.7], [1.0], [1.0], Z)
    with Leave(R, 400):
        got = R.payoffs_rt(*args)
    R.release()
    assert np.array_equal(got, R.payoffs_rt(*args, conv=R.CONV_DIRECT))


@pytest.mark.parametrize("ext", [False, True])
def test_more_passes_than_kept_panels(R, ext):
    """Panels beyond 2 GB (34952 passes) are built a launch at a time: the FP64 form's
    parity bound against the direct sum."""
    n = 35000
    par = (0.04, np.linspace(0.05, 0.45, n), np.full(n, 1.5), np.full(n, -0.7), [1.0], [1.0])
    if ext:
        Z = np.random.default_rng(3).standard_normal((64, 2, 100))  # steps enough for the digits
        p, q = R.payoffs_rt(*par, Z), R.payoffs_rt(*par, Z, conv=R.CONV_DIRECT)
        assert np.all(np.abs(p - q) <= 2e-13 * np.maximum(np.abs(q), 1.0))
    else:
        p, q = R.price_rt(*par, 16, 256, seed=2)[0], R.price_rt(*par, 16, 256, seed=2, conv=R.CONV_DIRECT)[0]
        assert np.all(np.abs(p - q) <= 1e-12 * np.abs(q))
    assert not np.array_equal(p, q)
