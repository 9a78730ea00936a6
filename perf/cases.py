"""The measured cases: the work a user of the pricer has it do, through its public entry points.

listed()  the named cases; draw(rng) one more of the same families
prepare() the inputs a program has in hand before the call, from a seed
run()     one call (or one burst of requests) and its results
work()    what one pass cannot do without
exact()   the same results in 64 bits, by plain torch and numpy
"""
import math

import numpy as np
import torch

import rbergomi_gb300 as R

# family -> (N range, path-steps range) of a drawn case.  A path-step is one
# path x one time step x one distinct H.
RANGES = {
    "dropin_rt": ((16, 400), (2 ** 18, 2 ** 24)),
    "dropin_mc": ((16, 600), (2 ** 18, 2 ** 24)),
    "price_fp64": ((16, 2048), (2 ** 18, 2 ** 25)),
    "grid_fp64": ((64, 512), (2 ** 20, 2 ** 24)),
    "quadrature": ((2, 600), (2 ** 16, 2 ** 22)),
    "price_mixed": ((16, 4096), (2 ** 18, 2 ** 29)),
    "grid_mixed": ((64, 1024), (2 ** 22, 2 ** 28)),
    "payoffs_mixed": ((16, 1024), (2 ** 18, 2 ** 25)),
    "serving": ((64, 1024), (2 ** 20, 2 ** 27)),
}


def listed():
    return [
        # the reference's own call: FP64 Romano-Touzi through the drop-in C entry, its 100-step CPU configuration
        dict(name="dropin_rt_n100", family="dropin_rt", N=100, M=65536, tuples=1, maturities=1, strikes=5),
        # the reference's plain Monte Carlo through the drop-in entry, ragged sizes, two parameter tuples
        dict(name="dropin_mc_n250", family="dropin_mc", N=250, M=30011, tuples=2, maturities=1, strikes=7),
        # the extended call's default precision (FP64) on the headline grid: one smile at 512 steps
        dict(name="price_fp64_n512", family="price_fp64", N=512, M=131072, tuples=1, maturities=1, strikes=21),
        # FP64 over a full ParamTot grid (4 H x 4 eta x 3 rho, 4 maturities x 11 strikes) sharing one draw
        dict(name="grid_fp64", family="grid_fp64", N=512, M=8192, H=4, eta=4, rho=3, maturities=4, strikes=11),
        # the drop-in quadrature entry: the caller's normals in host memory to per-path payoffs
        dict(name="quadrature_host_n252", family="quadrature", N=252, M=8190, tuples=1, maturities=2, strikes=3),
        # the inner call of a calibration: mixed precision, few paths, where latency and launches count
        dict(name="price_mixed_small", family="price_mixed", N=64, M=16384, tuples=1, maturities=1, strikes=8),
        # the headline workload: mixed precision, 512 steps, 2^22 paths, 21 strikes
        dict(name="price_mixed_n512", family="price_mixed", N=512, M=4194304, tuples=1, maturities=1, strikes=21),
        # long horizons of the step-count sweep: three H at 1024 steps
        dict(name="price_mixed_n1024", family="price_mixed", N=1024, M=524288, tuples=3, maturities=1, strikes=11),
        # a long, ragged horizon: step and path counts that are no multiples of the tiles
        dict(name="price_mixed_n2000", family="price_mixed", N=2000, M=262221, tuples=1, maturities=1, strikes=11),
        # the ParamTot grid in mixed precision: many variance paths and payoffs per draw
        dict(name="grid_mixed", family="grid_mixed", N=512, M=131072, H=4, eta=4, rho=3, maturities=4, strikes=11),
        # per-path payoffs of normals that already lie on the GPU, mixed precision
        dict(name="payoffs_mixed_n512", family="payoffs_mixed", N=512, M=65536, tuples=1, maturities=1, strikes=21),
        # calibration traffic: a burst of requests of different sizes through the serving loop
        dict(name="serving_burst", family="serving", requests=48, N_min=64, N_max=1024, M_min=16384, M_max=262144),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(sorted(RANGES))
    (n0, n1), (w0, w1) = RANGES[family]
    if family == "serving":
        top = _log_int(rng, 2 ** 15, 2 ** 18)
        return dict(family=family, requests=rng.randint(8, 48), N_min=n0, N_max=_log_int(rng, 100, n1), M_min=4096,
                    M_max=top)
    c = dict(family=family, N=_log_int(rng, n0, n1), M=0)
    if family.startswith("grid"):
        c.update(H=rng.randint(1, 4), eta=rng.randint(1, 4), rho=rng.randint(1, 3), maturities=rng.randint(1, 4),
                 strikes=rng.randint(3, 11))
    else:
        c.update(tuples=rng.choice((1, 1, 1, 2, 3)), maturities=rng.choice((1, 1, 2)), strikes=rng.randint(1, 21))
    # fewer path-steps where a step costs more: long horizons, grids
    if family == "price_mixed" and c["N"] > 1024:
        w1 //= 2
    n_h = c.get("H", c.get("tuples", 1))
    c["M"] = max(64, _log_int(rng, w0, w1) // (c["N"] * n_h))
    return c


# ------------------------------------------------------------------ inputs
def _shape(case):
    """(par_size, op_size, distinct H) of a case."""
    if "H" in case:
        return case["H"] * case["eta"] * case["rho"], case["maturities"] * case["strikes"], case["H"]
    return case["tuples"], case["maturities"] * case["strikes"], case["tuples"]


def _grid(case, rng):
    """xi, H, eta, rho, T, K of a case: a calibration's parameter ranges."""
    xi = float(rng.uniform(0.02, 0.08))
    if "H" in case:
        hs, es, rs = (np.sort(rng.uniform(a, b, n)) for a, b, n in
                      ((0.05, 0.35, case["H"]), (1.0, 2.2, case["eta"]), (-0.95, -0.4, case["rho"])))
        H, eta, rho = (a.ravel() for a in np.meshgrid(hs, es, rs, indexing="ij"))
    else:
        n = case["tuples"]
        H, eta, rho = rng.uniform(0.04, 0.4, n), rng.uniform(0.8, 2.2, n), rng.uniform(-0.95, -0.4, n)
    ts = np.sort(rng.uniform(0.25, 2.0, case["maturities"]))
    ks = np.linspace(0.75, 1.25, case["strikes"]) if case["strikes"] > 1 else np.array([1.0])
    T, K = np.repeat(ts, len(ks)), np.tile(ks + rng.uniform(-0.02, 0.02), len(ts))
    return xi, H, eta, rho, T, K


_SERVER = None


def _server():
    """A program's one serving loop."""
    global _SERVER
    if _SERVER is None:
        _SERVER = R.Server()
    return _SERVER


def _requests(case, seed):
    # the sizes belong to the case, the parameters to the seed
    sizes, rng = np.random.default_rng(case["requests"]), np.random.default_rng(seed)
    reqs = []
    for _ in range(case["requests"]):
        N = int(round(math.exp(sizes.uniform(math.log(case["N_min"]), math.log(case["N_max"])))))
        M = int(round(math.exp(sizes.uniform(math.log(case["M_min"]), math.log(case["M_max"])))))
        strikes = int(sizes.integers(1, 65))
        T = float(rng.uniform(0.2, 2.0))
        reqs.append(dict(xi=float(rng.uniform(0.02, 0.08)), H=[float(rng.uniform(0.04, 0.4))],
                         eta=[float(rng.uniform(0.8, 2.2))], rho=[float(rng.uniform(-0.95, -0.4))],
                         T=np.full(strikes, T), K=np.sort(rng.uniform(0.75, 1.25, strikes)), N=N, M=M,
                         seed=int(rng.integers(1 << 40))))
    return reqs


def _normals(case, seed):
    """The caller's normals [M, 2, N], on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn(case["M"], 2, case["N"], dtype=torch.float64, device="cuda", generator=g)


def prepare(case, seed):
    if case["family"] == "serving":
        return dict(case=case, server=_server(), requests=_requests(case, seed))
    rng = np.random.default_rng(seed)
    s = dict(case=case, grid=_grid(case, rng), seed=int(rng.integers(1 << 40)))
    if case["family"] == "quadrature":
        s["Z"] = _normals(case, seed).cpu().numpy()
    if case["family"] == "payoffs_mixed":
        s["Z"] = _normals(case, seed)
        par, op, _ = _shape(case)
        s["payoff"] = torch.empty(case["M"], par * op, dtype=torch.float64, device="cuda")
    return s


def run(state):
    case = state["case"]
    family = case["family"]
    if family == "serving":
        srv = state["server"]
        tickets = [srv.submit(**r) for r in state["requests"]]
        got = [srv.wait(t) for t in tickets]
        return dict(price=np.concatenate([g[0] for g in got]), stat=np.concatenate([g[1] for g in got]),
                    iv=np.concatenate([g[2] for g in got]))
    xi, H, eta, rho, T, K = state["grid"]
    N, M = case["N"], case["M"]
    if family == "dropin_rt":
        r = R.computeIVRT_tensor(xi, H, eta, rho, T, K, N, M, state["seed"])
        return dict(price=r.price, stat=r.stat, iv=r.iv, H=r.H, eta=r.eta, rho=r.rho, T=r.T, K=r.K)
    if family == "dropin_mc":
        r = R.computeIV_tensor(xi, H, eta, rho, T, K, N, M, state["seed"])
        return dict(price=r.price, stat=r.stat, iv=r.iv, H=r.H, eta=r.eta, rho=r.rho, T=r.T, K=r.K)
    if family == "quadrature":
        return dict(payoff=R.computeIVRT_tensor_quadrature(xi, H, eta, rho, T, K, state["Z"]))
    if family == "payoffs_mixed":
        R.payoffs_rt(xi, H, eta, rho, T, K, state["Z"].data_ptr(), device_ptrs=True, M=M, N=N,
                     out_ptr=state["payoff"].data_ptr(), precision=R.MIXED)
        return dict(payoff=state["payoff"])
    precision = R.MIXED if family.endswith("mixed") else R.FP64
    price, stat, iv = R.price_rt(xi, H, eta, rho, T, K, N, M, precision=precision, seed=state["seed"])
    return dict(price=price, stat=stat, iv=iv)


def _steps_flops(N, M, n_h, groups, out, streams):
    """Flops of M paths: normals (20 a pair), the causal convolution by the cheaper of the direct sum and two real
    FFTs of 2N points, the variance update (12 a group), one conditional Black-Scholes price (50) an output."""
    conv = min(N - 1, 10.0 * math.log2(2 * N + 2))
    return M * (N * (10.0 * streams + n_h * (conv + 4) + 12.0 * groups) + 50.0 * out)


def work(case):
    if case["family"] == "serving":
        reqs = _requests(case, 1)
        return dict(bytes=sum(8.0 * 5 * len(r["K"]) for r in reqs),
                    flops=sum(_steps_flops(r["N"], r["M"], 1, 1, len(r["K"]), 2) for r in reqs))
    par, op, n_h = _shape(case)
    N, M, out = case["N"], case["M"], par * op
    groups = (case["H"] * case["eta"] if "H" in case else case["tuples"]) * case["maturities"]
    streams = 3 if case["family"] == "dropin_mc" else 2
    ext = case["family"] in ("quadrature", "payoffs_mixed")
    moved = 8.0 * M * (2 * N + out) if ext else 8.0 * 5 * out
    return dict(bytes=moved, flops=_steps_flops(N, M, n_h, groups, out, 0 if ext else streams))


# ---------------------------------------------------- the same in 64 bits
_MASK = 0xFFFFFFFF


def _mulhilo(a, b):
    """32 x 32 -> 64-bit product of a constant and an int64 tensor of 32-bit values."""
    p = b * a  # wraps modulo 2^64
    return (p >> 32) & _MASK, p & _MASK


def _uniform_words(seed, m, groups, stream):
    """Philox4x32-10 words [paths, groups, 4], counter (group, path low, path high, stream), key = seed."""
    c0 = torch.arange(groups, device="cuda", dtype=torch.int64).expand(len(m), groups)
    c1 = (m & _MASK)[:, None].expand(len(m), groups)
    c2 = (m >> 32)[:, None].expand(len(m), groups)
    c3 = torch.full_like(c0, stream)
    k0, k1 = seed & _MASK, (seed >> 32) & _MASK
    for _ in range(10):
        h0, l0 = _mulhilo(0xD2511F53, c0)
        h1, l1 = _mulhilo(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & _MASK, (k1 + 0xBB67AE85) & _MASK
    return torch.stack((c0, c1, c2, c3), -1)


def _stream_normals(seed, m, N, stream):
    x = _uniform_words(seed, m, (N + 3) // 4, stream).double()
    u = (x + 0.5) * 2.0 ** -32
    r = torch.sqrt(-2.0 * torch.log(u[..., 0::2]))
    t = 2.0 * math.pi * u[..., 1::2]
    return torch.stack((r * torch.cos(t), r * torch.sin(t)), -1).reshape(len(m), -1)[:, :N]


def _cdf(x):
    return 0.5 * torch.special.erfc(x * -0.5 ** 0.5)


def _chunk_payoffs(grid, W, Wp, Wq=None):
    """Payoffs [out, paths] on the normals W1, W1perp (and, for plain Monte Carlo, Wperp) of one chunk of paths."""
    xi, H, eta, rho, T, K = grid
    N = W.shape[1]
    L = 1 << max(1, (2 * N - 1).bit_length())
    i = torch.arange(1, N, device="cuda", dtype=torch.float64)
    spec = torch.fft.rfft(W, L)
    conv, inte, rows = {}, {}, []
    for q in range(len(H)):
        h = float(H[q])
        if h not in conv:
            gamma = torch.zeros(N, device="cuda", dtype=torch.float64)
            gamma[1:] = ((i + 1) ** (h + 0.5) - i ** (h + 0.5)) / (h + 0.5)
            a1 = 1.0 / (h + 0.5)
            s2h = math.sqrt(2 * h)
            a2 = math.sqrt(max(0.0, 1.0 - (s2h * a1) ** 2)) / s2h
            conv[h] = torch.fft.irfft(spec * torch.fft.rfft(gamma, L), L)[:, :N] + a1 * W + a2 * Wp
        for o in range(len(T)):
            t, e = float(T[o]), float(eta[q])
            if (h, e, t) not in inte:
                dt = t / N
                scale = math.sqrt(2 * h) * (t / N) ** h
                j = torch.arange(0, N - 1, device="cuda", dtype=torch.float64)
                sv = torch.empty_like(W)
                sv[:, 0] = math.sqrt(xi)
                sv[:, 1:] = math.sqrt(xi) * torch.exp(0.5 * e * scale * conv[h][:, :-1]
                                                      - 0.25 * e * e * (j * dt) ** (2 * h))
                inte[h, e, t] = (dt * (sv * sv).sum(1), math.sqrt(dt) * (sv * W).sum(1),
                                 None if Wq is None else math.sqrt(dt) * (sv * Wq).sum(1))
            V, I, J = inte[h, e, t]
            r, k = float(rho[q]), float(K[o])
            if J is not None:
                rows.append(torch.clamp(torch.exp(r * I + math.sqrt(1 - r * r) * J - 0.5 * V) - k, min=0.0))
                continue
            vol, ln = torch.sqrt((1 - r * r) * V), r * I - 0.5 * r * r * V
            d1 = (ln - math.log(k)) / vol + 0.5 * vol
            rows.append(torch.exp(ln) * _cdf(d1) - k * _cdf(d1 - vol))
    return torch.stack(rows)


def _implied(price, K, T):
    """Black-Scholes volatility by bisection on the out-of-the-money price; NaN where none fits."""
    p, k, t = (torch.tensor(np.asarray(a, np.float64)) for a in (price, K, T))
    put = k < 1.0
    target = torch.where(put, p - 1.0 + k, p)
    ok = (target > 0) & (target < torch.where(put, k, torch.ones_like(k)))
    lo, hi, sq = torch.zeros_like(p), torch.full_like(p, 40.0), torch.sqrt(t)
    for _ in range(120):
        s = 0.5 * (lo + hi)
        d1 = -torch.log(k) / (s * sq) + 0.5 * s * sq
        d2 = d1 - s * sq
        v = torch.where(put, k * _cdf(-d2) - _cdf(-d1), _cdf(d1) - k * _cdf(d2))
        lo, hi = torch.where(v < target, s, lo), torch.where(v < target, hi, s)
    return torch.where(ok, 0.5 * (lo + hi), torch.full_like(p, float("nan"))).numpy()


def _price(grid, N, M, seed, streams=2):
    """(price, stat, iv) of a Philox call."""
    xi, H, eta, rho, T, K = grid
    n_out = len(H) * len(T)
    s1, s2 = (torch.zeros(n_out, device="cuda", dtype=torch.float64) for _ in range(2))
    step = max(64, (1 << 24) // N)
    for m0 in range(0, M, step):
        m = torch.arange(m0, min(M, m0 + step), device="cuda", dtype=torch.int64)
        x = _chunk_payoffs(grid, *(_stream_normals(seed, m, N, s) for s in range(streams)))
        s1 += x.sum(1)
        s2 += (x * x).sum(1)
    price = (s1 / M).cpu().numpy()
    stat = np.sqrt((s2 / M).cpu().numpy() - price ** 2) / math.sqrt(M)
    return price, stat, _implied(price, np.tile(K, len(H)), np.tile(T, len(H)))


def exact(case, seed):
    family = case["family"]
    if family == "serving":
        got = [_price(tuple(np.asarray(r[k], np.float64) if k != "xi" else r[k] for k in
                            ("xi", "H", "eta", "rho", "T", "K")), r["N"], r["M"], r["seed"])
               for r in _requests(case, seed)]
        return {k: np.concatenate([g[i] for g in got]) for i, k in enumerate(("price", "stat", "iv"))}
    rng = np.random.default_rng(seed)
    grid = _grid(case, rng)
    philox = int(rng.integers(1 << 40))
    if family in ("quadrature", "payoffs_mixed"):
        Z = _normals(case, seed)
        step = max(64, (1 << 24) // case["N"])
        return dict(payoff=torch.cat([_chunk_payoffs(grid, z[:, 0], z[:, 1]).T for z in Z.split(step)]))
    price, stat, iv = _price(grid, case["N"], case["M"], philox, 3 if family == "dropin_mc" else 2)
    out = dict(price=price, stat=stat, iv=iv)
    if family.startswith("dropin"):
        _, H, eta, rho, T, K = grid
        tot = {n: np.repeat(a, len(T)) for n, a in (("H", H), ("eta", eta), ("rho", rho))}
        if family == "dropin_mc":  # the plain Monte Carlo entry writes these two in swapped order
            tot["eta"], tot["rho"] = tot["rho"], tot["eta"]
        out.update(tot, T=np.tile(T, len(H)), K=np.tile(K, len(H)))
    return out
