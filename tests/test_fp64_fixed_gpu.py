"""The FP64 form's fixed-point / tensor-core path pass (Philox normals, no
backend asked for) against the FP64 kernels on the same normals: prices to
1e-12 relative, the FP64 form's parity bound, at the edges of its tiles (16-step
chunks, 128-step blocks, 64 paths), over several passes and variance groups,
and where its ranges end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
XI, K = 0.235 ** 2, [0.85, 1.0, 1.1]


@pytest.fixture(scope="module")
def R():
    import rbergomi_gb300 as R
    return R


def close(a, b, tol=1e-12):
    assert np.all(np.abs(a - b) <= tol * np.abs(b)), np.max(np.abs(a - b) / np.abs(b))


@pytest.mark.parametrize("N", [1, 2, 3, 15, 16, 17, 33, 127, 128, 129, 143, 145, 256, 257, 400, 1023, 1025])
@pytest.mark.parametrize("M", [1, 63, 65, 700])
def test_against_the_direct_sum(R, N, M):
    args = (XI, [0.07], [1.9], [-0.9], [1.0] * 3, K, N, M)
    p, s, _ = R.price_rt(*args, seed=3, path_offset=2 ** 32 - 50)
    q, t, _ = R.price_rt(*args, seed=3, path_offset=2 ** 32 - 50, conv=R.CONV_DIRECT)
    close(p, q)
    if M > 1:
        close(s, t, 1e-8)


@pytest.mark.parametrize("N", [2047, 2049, 4096])
def test_long_horizons(R, N):
    args = (XI, [0.1, 0.45], [1.9, 1.0], [-0.9, -0.5], [2.0] * 3, K, N, 300)
    close(R.price_rt(*args, seed=5)[0], R.price_rt(*args, seed=5, conv=R.CONV_DIRECT)[0])


@pytest.mark.parametrize("n_t", [1, 3, 4, 5, 9])  # variance groups per pass: one, short and full batches of four
@pytest.mark.parametrize("mc", [False, True])
def test_passes_and_groups(R, n_t, mc):
    price = R.price_mc if mc else R.price_rt
    H, eta, rho = [0.05, 0.3, 0.45], [1.5, 2.0, 1.0], [-0.7, -0.3, -0.9]
    T, Ks = np.repeat(np.linspace(0.1, 2.5, n_t), 2), np.tile([0.9, 1.05], n_t)
    args = (0.05, H, eta, rho, T, Ks, 150, 333)
    close(price(*args, seed=8)[0], price(*args, seed=8, conv=R.CONV_DIRECT)[0])


@pytest.mark.parametrize("H,eta,T", [(0.01, 3.0, 3.0), (0.5, 0.0, 1.0), (0.9, 0.5, 0.01), (0.3, -1.5, 1.0), (0.2, 40.0, 5.0),
                                     (0.1, 1e5, 1.0)])
def test_parameter_corners(R, H, eta, T):
    # the last ones' exponents do not fit the fixed-point range: the FP64 kernels take them
    args = (XI, [H], [eta], [-0.5], [T] * 3, K, 200, 500)
    p, q = R.price_rt(*args, seed=2)[0], R.price_rt(*args, seed=2, conv=R.CONV_DIRECT)[0]
    assert np.array_equal(np.isnan(p), np.isnan(q))
    close(p[~np.isnan(q)], q[~np.isnan(q)])


@pytest.mark.parametrize("xi", [0.0, -1.0, 1e-300, 1e6])
def test_forward_variance_corners(R, xi):
    args = (xi, [0.1], [1.0], [-0.5], [1.0], [1.2], 64, 100)
    p, q = R.price_rt(*args, seed=2)[0], R.price_rt(*args, seed=2, conv=R.CONV_DIRECT)[0]
    assert np.array_equal(np.isnan(p), np.isnan(q))
    ok = ~np.isnan(q)
    assert np.all(np.abs(p - q)[ok] <= 1e-12 * np.abs(q[ok]) + 1e-300)


def test_fp32_normals(R):
    args = (XI, [0.07], [1.9], [-0.9], [1.0] * 3, K, 130, 500)
    p = R.price_rt(*args, seed=4, normals=R.NORMALS_F32)[0]
    close(p, R.price_rt(*args, seed=4, normals=R.NORMALS_F32, conv=R.CONV_DIRECT)[0])


@pytest.mark.parametrize("M", [1, 255, 257, 5000])
def test_sums_are_the_payoffs_sums(R, M):
    """The exact merge of the chunk sums against fsum over the per-path payoffs
    of the same normals (another path pass: 1e-12), and shards against the whole
    (the same payoffs in other chunks: additions of up to 256 values, 1e-13)."""
    import math
    args = (XI, [0.07], [1.9], [-0.9], [1.0] * 3, [0.5, 1.0, 2.5], 60)
    s1, s2 = R.price_rt_sums(*args, M, seed=6)
    pay = R.payoffs_rt(*args[:6], R.generate_normals(6, M, 60))
    close(s1, np.array([math.fsum(pay[:, i]) for i in range(3)]))
    close(s2, np.array([math.fsum(pay[:, i] ** 2) for i in range(3)]))
    if M > 1:
        a, b = R.price_rt_sums(*args, M // 2, seed=6), R.price_rt_sums(*args, M - M // 2, seed=6, path_offset=M // 2)
        close(a[0] + b[0], s1, 1e-13)
        close(a[1] + b[1], s2, 1e-13)


@pytest.mark.parametrize("kind", ["normal", "constant", "extreme digits", "zero"])
@pytest.mark.parametrize("N,M", [(1, 5), (2, 64), (17, 65), (128, 63), (129, 70), (300, 130), (1030, 20)])
def test_caller_normals(R, N, M, kind):
    """Per-path payoffs of the caller's normals against the FP64 direct sum's:
    2e-13 of the larger of the payoff and 1 (FP64 roundoff of the exponent over
    N steps), for inputs whose digits add up as well as for normals."""
    g = np.random.default_rng(N + M)
    Z = {"normal": lambda: g.standard_normal((M, 2, N)), "zero": lambda: np.zeros((M, 2, N)),
         "constant": lambda: np.broadcast_to(g.uniform(-1, 1, (M, 2, 1)), (M, 2, N)).copy(),
         # every lower digit of W1 at an end of its range
         "extreme digits": lambda: np.where(g.random((M, 2, 1)) < 0.5, -1, 1) * np.full((M, 2, N), 0x7f7f7f7f7f7f7 / 2.0 ** 51)
         }[kind]()
    eta = 1.9 if kind in ("normal", "zero") else 1.9 / np.sqrt(N)
    args = (XI, [0.07, 0.4], [eta, eta], [-0.9, 0.3], [1.0, 0.5], [0.9, 1.1], Z)
    p, q = R.payoffs_rt(*args), R.payoffs_rt(*args, conv=R.CONV_DIRECT)
    assert np.all(np.abs(p - q) <= 2e-13 * np.maximum(np.abs(q), 1.0)), np.max(np.abs(p - q))


@pytest.mark.parametrize("bad", [15.5, -16.0, 1e3, np.inf, np.nan])
@pytest.mark.parametrize("stream", [0, 1])
def test_caller_normals_out_of_range_take_the_fp64_kernels(R, bad, stream):
    Z = np.random.default_rng(1).standard_normal((70, 2, 40))
    Z[66, stream, 21] = bad
    args = (XI, [0.1], [0.5], [-0.7], [1.0], [1.0], Z)
    p, q = R.payoffs_rt(*args), R.payoffs_rt(*args, conv=R.CONV_DIRECT)
    assert np.array_equal(p, q, equal_nan=True)  # the whole batch is the direct sum's
    Zm = np.concatenate([Z, np.random.default_rng(2).standard_normal((70, 1, 40))], 1)
    p, q = R.payoffs_mc(*args[:6], Zm), R.payoffs_mc(*args[:6], Zm, conv=R.CONV_DIRECT)
    assert np.array_equal(p, q, equal_nan=True)


# calls large enough for the digit convolution, at the edges of its tiles
LARGE = [(2, 12001), (17, 12002), (128, 3009), (129, 3007), (300, 1030), (1030, 641)]


def large_inputs(kind, N, M, ns):
    g = np.random.default_rng(N + M)
    if kind == "normal":
        return g.standard_normal((M, ns, N)), 1.9
    if kind == "constant":
        return np.broadcast_to(g.uniform(-1, 1, (M, ns, 1)), (M, ns, N)).copy(), 1.9 / np.sqrt(N)
    # every lower digit of W1 at an end of its range
    return np.where(g.random((M, ns, 1)) < 0.5, -1, 1) * np.full((M, ns, N), 0x7f7f7f7f7f7f7 / 2.0 ** 51), 1.9 / np.sqrt(N)


@pytest.mark.parametrize("kind", ["normal", "constant", "extreme digits"])
@pytest.mark.parametrize("mc", [False, True])
@pytest.mark.parametrize("N,M", LARGE)
def test_caller_normals_large_calls(R, N, M, mc, kind):
    """As test_caller_normals, where the call takes the digit convolution (its
    results are not the direct sum's bit for bit)."""
    Z, eta = large_inputs(kind, N, M, 3 if mc else 2)
    args = (XI, [0.07, 0.4], [eta, eta], [-0.9, 0.3], [1.0, 0.5], [0.9, 1.1], Z)
    pay = R.payoffs_mc if mc else R.payoffs_rt
    p, q = pay(*args), pay(*args, conv=R.CONV_DIRECT)
    assert np.all(np.abs(p - q) <= 2e-13 * np.maximum(np.abs(q), 1.0)), np.max(np.abs(p - q))
    assert kind != "normal" or not np.array_equal(p, q)


@pytest.mark.parametrize("bad", [15.5, -np.inf, np.nan])
@pytest.mark.parametrize("N,fft", [(16, False), (199, False), (200, True), (300, True), (2048, True), (2049, False)])
def test_caller_normals_out_of_range_take_the_backend_of_their_length(R, N, fft, bad):
    """Large calls with a normal past the digits' range: the FP64 kernels' own choice
    for N steps (FFT from 200 to 2048 steps, else the direct sum), bit for bit, and
    the call after it is in range again."""
    conv, M = R.CONV_FFT if fft else R.CONV_DIRECT, 12001 if N < 100 else 2003 if N < 1000 else 901
    Z = np.random.default_rng(1).standard_normal((M, 2, N))
    args = (XI, [0.1], [0.5], [-0.7], [1.0], [1.0])
    want = R.payoffs_rt(*args, Z)
    assert not np.array_equal(want, R.payoffs_rt(*args, Z, conv=conv))
    Zb = Z.copy()
    Zb[7, 1, N // 2] = bad
    assert np.array_equal(R.payoffs_rt(*args, Zb), R.payoffs_rt(*args, Zb, conv=conv), equal_nan=True)
    assert np.array_equal(R.payoffs_rt(*args, Z), want)


def test_small_quadrature_calls_take_the_fp64_kernels(R):
    """Few paths of few steps: the FP64 path kernel's one launch, its results bit for bit."""
    for N, M, conv in ((2, 500, R.CONV_DIRECT), (64, 1000, R.CONV_DIRECT), (199, 100, R.CONV_DIRECT),
                       (200, 400, R.CONV_FFT), (512, 130, R.CONV_FFT)):
        Z = np.random.default_rng(N).standard_normal((M, 2, N))
        args = (XI, [0.1], [1.5], [-0.7], [1.0], [1.0], Z)
        assert np.array_equal(R.payoffs_rt(*args), R.payoffs_rt(*args, conv=conv))
    # and not where a path alone takes long: one path of 4096 steps 0.5 ms by digits, 10.9 in FP64
    for N, M, conv in ((700, 1, R.CONV_FFT), (2048, 1, R.CONV_FFT), (2049, 1, R.CONV_DIRECT), (4096, 5, R.CONV_DIRECT)):
        Z = np.random.default_rng(N).standard_normal((M, 2, N))
        args = (XI, [0.1, 0.2], [1.5, 1.0], [-0.7, -0.5], [1.0, 1.0], [0.8, 1.0], Z)
        p, q = R.payoffs_rt(*args), R.payoffs_rt(*args, conv=conv)
        assert not np.array_equal(p, q) and np.all(np.abs(p - q) <= 1e-12)


def test_caller_normals_plain_mc(R):
    Z = np.random.default_rng(3).standard_normal((130, 3, 150))
    Z[5, 2, 7] = 1e3  # Wperp only meets FP64 sums: no range
    args = (XI, [0.1, 0.3], [1.5, 1.0], [-0.7, 0.2], [1.0, 0.5, 2.0], [1.0, 0.9, 1.1], Z)
    p, q = R.payoffs_mc(*args), R.payoffs_mc(*args, conv=R.CONV_DIRECT)
    assert np.all(np.abs(p - q) <= 2e-13 * np.maximum(np.abs(q), 1.0))


@pytest.mark.parametrize("M,n_out", [(1, 1), (255, 3), (257, 9), (3000, 40), (60000, 17)])
def test_plain_mc_payoffs_small_and_large_calls(R, M, n_out):
    """Calls whose payoff blocks read the exponential's table in place (a task a block)
    and calls whose blocks copy it: the payoff of one output does not depend on the
    others, nor on how many paths there are."""
    Z = np.random.default_rng(M).standard_normal((M, 3, 4))
    par = (XI, [0.1], [1.5], [-0.7])
    p = R.payoffs_mc(*par, [1.0] * n_out, np.linspace(0.6, 1.4, n_out), Z, conv=R.CONV_DIRECT)
    for i in (0, n_out - 1):
        q = R.payoffs_mc(*par, [1.0], [np.linspace(0.6, 1.4, n_out)[i]], Z[:1], conv=R.CONV_DIRECT)
        assert np.array_equal(p[:1, i], q[:, 0])


@pytest.mark.parametrize("mc,n_t", [(False, 2), (False, 3), (True, 6), (True, 7)])  # around the last fused group count
@pytest.mark.parametrize("N,M", [(2, 65), (31, 129), (33, 64), (161, 700), (1100, 130)])
def test_variance_in_the_read_out(R, mc, n_t, N, M):
    """Variance groups up to and past the count the convolution's read-out takes,
    at the edges of its 32-step sums, 128-step blocks and 16-path shares: the FP64
    form's parity bound against the direct sum."""
    price = R.price_mc if mc else R.price_rt
    T = np.linspace(0.1, 3.0, n_t)
    args = (XI, [0.08, 0.35], [2.2, -1.0], [-0.8, 0.4], T, [1.0] * n_t, N, M)
    close(price(*args, seed=9)[0], price(*args, seed=9, conv=R.CONV_DIRECT)[0])
