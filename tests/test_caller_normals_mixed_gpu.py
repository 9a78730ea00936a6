"""The mixed form's caller-normals producer takes 16-byte loads where every row
starts on a 16-byte boundary and 8-byte loads otherwise: the same bits from
aligned and odd buffers, at the edges of its 4-step and 32-step shares and of the
passes, and the FP64 form's payoffs within the mixed form's 2e-4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ARGS = (0.04, [0.1, 0.4], [1.5, 1.0], [-0.7, 0.2], [0.5, 1.0], [0.9, 1.1])


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 31, 32, 33, 34, 66, 511, 512, 514, 1026])
@pytest.mark.parametrize("M", [1, 127, 300])
def test_aligned_and_odd_buffers(N, M):
    import rbergomi_gb300 as R
    torch = pytest.importorskip("torch")
    Z = np.random.default_rng(N).standard_normal((M, 2, N))
    want = R.payoffs_rt(*ARGS, Z)
    got = []
    for shift in (0, 1, 2):
        buf = torch.full((shift + Z.size + 64,), float("nan"), dtype=torch.float64, device="cuda")
        buf[shift:shift + Z.size] = torch.from_numpy(Z.ravel()).cuda()
        out = torch.empty(want.shape, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        R.payoffs_rt(*ARGS, buf.data_ptr() + 8 * shift, device_ptrs=True, M=M, N=N, out_ptr=out.data_ptr(),
                     precision=R.MIXED)
        got.append(out.cpu().numpy())
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    assert np.all(np.abs(got[0] - want) <= 2e-4 * np.maximum(np.abs(want), 1.0))


def test_plain_mc():
    import rbergomi_gb300 as R
    for N in (33, 34, 512):
        Z = np.random.default_rng(N).standard_normal((200, 3, N))
        p, q = R.payoffs_mc(*ARGS, Z, precision=R.MIXED), R.payoffs_mc(*ARGS, Z)
        assert np.all(np.abs(p - q) <= 2e-4 * np.maximum(np.abs(q), 1.0))
