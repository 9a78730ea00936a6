// rbg_fp64.cu -- the plain FP64 form of the RT pricer on the GPU: the path pass
// on normals of any source, payoffs and reductions (normals and the path pass
// on Philox normals: rbg_fp64x.cu).
//
// Kernels (one pass over a batch of paths):
//   k_path_fp64    per path: Volterra sum Y2 = (W1 * Gamma)[0..N) as a direct
//                  causal FP64 sum, X = Y2 + a1 W1 + a2 W1perp, then for every
//                  variance group v, Ivdt = dt sum v, IsvdW = sum sqrt(v) sdt W1
//                  (rBergLib/rBergomiMT.cpp:73-109, 163-167, 427-436)
//   k_path_fp64_fft  the same pass with Y2 as an FP64 FFT convolution, two
//                  paths per complex transform (from 200 steps; the direct
//                  sum's N^2 / 2 DFMA per path outgrow it there)
//   k_payoff_sums  conditional BS per (path, output) and per-chunk sums of x and
//                  x^2 (rBergomiMT.cpp:598-602, 404-409)
//   k_merge        exact merge of chunk sums (deterministic); after the last
//                  batch price, stat (reference formula), implied vol
//   k_payoff_store per-path payoffs for the quadrature entry point
// GB300's FP64 pipe (~2 DFMA/clk/SM) bounds the path kernels here, and the payoffs
// although their elementary functions are in fixed point (rbg_fixed.cuh).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>

#include "rbg_device.cuh"
#include "rbg_fixed.cuh"
#include "rbg_fp64x.hpp"
#include "rbg_internal.hpp"

namespace rbg {

// --------------------------------------------------------------- path pass
// One warp per path.  Shared memory: Gamma of the current pass (N doubles),
// then per warp W1 (N) and X (N).  NS = 3 (plain MC) also sums
// IsvdWp = sum sqrt(v) sdt Wperp into ivp.
// ANTI (control-variate form): also the antithetic path -W1, -W1perp.  The
// Volterra sum is linear, so its X is exactly -X; ivn[g][B] gets its
// (Ivdt, IsvdW).
template <int NS, bool ANTI>
__global__ void k_path_fp64(Fp64Tables t, const double* __restrict__ Z, int64_t B, double2* __restrict__ ivb,
                            double* __restrict__ ivp, double2* __restrict__ ivn)
{
    extern __shared__ double sm[];
    const int N = t.N;
    const int warps = blockDim.x >> 5;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* G = sm;
    double* W1s = sm + N + (size_t)w * 2 * N;
    double* X = W1s + N;
    const int64_t m = (int64_t)blockIdx.x * warps + w;
    const bool active = m < B;
    const double* W1 = Z + m * NS * (int64_t)N;
    const double* W1p = W1 + N;
    const double* Wperp = W1 + 2 * N;  // NS = 3 only
    if (active)
        for (int j = lane; j < N; j += 32) W1s[j] = W1[j];

    for (int v = 0; v < t.n_vol; ++v) {
        __syncthreads();
        for (int j = threadIdx.x; j < N; j += blockDim.x) G[j] = t.gamma[(size_t)v * N + j];
        __syncthreads();
        if (!active) continue;
        const VolDev vol = t.vols[v];
        // Y2[j] = sum_{k<j} W1[k] Gamma[j-k]   (Gamma[0] = 0)
        for (int j = lane; j < N; j += 32) {
            double acc = 0.0;
            for (int k = 0; k < j; ++k) acc = fma(W1s[k], G[j - k], acc);
            X[j] = acc + (vol.a1 * W1s[j] + vol.a2 * W1p[j]);
        }
        __syncwarp();
        for (int g = vol.vg_begin; g < vol.vg_end; ++g) {
            const VGDev vg = t.vgs[g];
            const double* comp = t.comp + (size_t)g * N;
            double sv = 0.0, sw = 0.0, sp = 0.0, nv = 0.0, nw = 0.0;
            // sqrt(v_j) = sqrt(xi) exp(a_j / 2) and v_j = sqrt(v_j)^2: one exp, no sqrt per step
            const double sxi = sqrt(vg.xi);
            for (int j = lane; j < vg.nsteps; j += 32) {
                const double su = (j == 0) ? sxi : sxi * exp(0.5 * (vg.eta * (vg.scale * X[j - 1]) - comp[j - 1]));
                const double vj = (j == 0) ? vg.xi : su * su;
                sv += vj;
                const double sq = su * vg.sdt;
                sw += sq * W1s[j];
                if (NS == 3) sp += sq * Wperp[j];
                if (ANTI) {
                    const double sa = (j == 0) ? sxi : sxi * exp(0.5 * (vg.eta * (vg.scale * -X[j - 1]) - comp[j - 1]));
                    nv += (j == 0) ? vg.xi : sa * sa;
                    nw += sa * vg.sdt * -W1s[j];
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sv += __shfl_xor_sync(0xffffffffu, sv, o);
                sw += __shfl_xor_sync(0xffffffffu, sw, o);
                if (NS == 3) sp += __shfl_xor_sync(0xffffffffu, sp, o);
                if (ANTI) {
                    nv += __shfl_xor_sync(0xffffffffu, nv, o);
                    nw += __shfl_xor_sync(0xffffffffu, nw, o);
                }
            }
            if (lane == 0) {
                ivb[(size_t)g * B + m] = make_double2(vg.dt * sv, sw);
                if (NS == 3) ivp[(size_t)g * B + m] = sp;
                if (ANTI) ivn[(size_t)g * B + m] = make_double2(vg.dt * nv, nw);
            }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------ path pass, FFT
// The same pass with the Volterra sum as an FP64 FFT convolution: O(N log N)
// FP64 operations per path instead of N^2 / 2, so from a few hundred steps it
// does the FP64 pipe a fraction of the work.  The reference convolves the
// same way (fftOMP over FFTW, rBergLib/rBergomiMT.cpp:83-109); the results
// differ from the direct sum by roundoff.
//
// One CTA of 256 threads per pair of paths (a, b): z = W1_a + i W1_b,
// zero-padded to L = 2^logL >= 2N - 1, so the circular convolution with the
// real Gamma holds both linear ones, y = conv(z, Gamma) = Y2_a + i Y2_b.
// y = IFFT(FFT(z) FFT(Gamma)) = conj(FFT(conj(FFT(z) spec))) with
// spec = FFT(Gamma) / L, so one forward Stockham transform serves both
// directions.  FFT(z) is kept for every distinct H (pass v).
//
// Stockham autosort, radix 4 (one radix-2 pass first when logL is odd), in
// place: each thread loads its butterflies' inputs, the block synchronises,
// then each thread writes its outputs (the formulation of Govindaraju et al.,
// "High performance discrete Fourier transforms on graphics processors",
// SC'08: pass (R, Ns) reads x[j + r L / R], twiddles by exp(-2 pi i r (j mod
// Ns) / (Ns R)) and writes x[(j - j mod Ns) R + j mod Ns + r Ns]).
constexpr int kFftThreads = 256;
constexpr int kFp64FftMinLogL = 8;  // shorter transforms run at L = 256 (any L >= 2N - 1 holds the sums)

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// MAXB: butterflies per thread, L / R / 256 rounded up
template <int R, int MAXB>
__device__ __forceinline__ void stockham_pass(double2* x, int L, int Ns, const double2* __restrict__ tw)
{
    const int nb = L / R;
    const int tstep = L / (Ns * R);
    double2 v[MAXB][R];
#pragma unroll
    for (int b = 0; b < MAXB; ++b) {
        const int j = threadIdx.x + b * kFftThreads;
        if (j < nb) {
            const int k = j & (Ns - 1);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const double2 a = x[j + r * nb];
                v[b][r] = (r == 0 || k == 0) ? a : cmul(a, __ldg(tw + r * k * tstep));
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < MAXB; ++b) {
        const int j = threadIdx.x + b * kFftThreads;
        if (j < nb) {
            const int k = j & (Ns - 1);
            const int d = (j - k) * R + k;
            if (R == 2) {
                const double2 a = v[b][0], c = v[b][1];
                x[d] = make_double2(a.x + c.x, a.y + c.y);
                x[d + Ns] = make_double2(a.x - c.x, a.y - c.y);
            } else {
                // X0 = a + b + c + e, X1 = a - i b - c + i e, X2 = a - b + c - e, X3 = a + i b - c - i e
                const double2 a = v[b][0], bb = v[b][1], c = v[b][2], e = v[b][3];
                const double2 s0 = make_double2(a.x + c.x, a.y + c.y), d0 = make_double2(a.x - c.x, a.y - c.y);
                const double2 s1 = make_double2(bb.x + e.x, bb.y + e.y), d1 = make_double2(bb.x - e.x, bb.y - e.y);
                x[d] = make_double2(s0.x + s1.x, s0.y + s1.y);
                x[d + Ns] = make_double2(d0.x + d1.y, d0.y - d1.x);       // d0 - i d1
                x[d + 2 * Ns] = make_double2(s0.x - s1.x, s0.y - s1.y);
                x[d + 3 * Ns] = make_double2(d0.x - d1.y, d0.y + d1.x);   // d0 + i d1
            }
        }
    }
    __syncthreads();
}

// forward DFT of x (L = 2^LOGL) in natural order
template <int LOGL>
__device__ __forceinline__ void fft_forward(double2* x, const double2* __restrict__ tw)
{
    constexpr int L = 1 << LOGL;
    constexpr int B2 = (L / 2 + kFftThreads - 1) / kFftThreads, B4 = (L / 4 + kFftThreads - 1) / kFftThreads;
    int Ns = 1;
    if (LOGL & 1) {
        stockham_pass<2, B2>(x, L, Ns, tw);
        Ns = 2;
    }
#pragma unroll 1
    for (; Ns < L; Ns *= 4) stockham_pass<4, B4>(x, L, Ns, tw);
}

// block sum over the 128 threads of one path half (threads 0..127 or 128..255)
__device__ __forceinline__ double half_sum(double s, double* red, int slot)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) red[slot * 8 + w] = s;
    __syncthreads();
    const int w0 = (threadIdx.x >> 7) * 4;
    const double r = (red[slot * 8 + w0] + red[slot * 8 + w0 + 1]) + (red[slot * 8 + w0 + 2] + red[slot * 8 + w0 + 3]);
    return r;
}

template <int LOGL, int NS, bool ANTI>
__global__ void __launch_bounds__(kFftThreads) k_path_fp64_fft(Fp64Tables t, const double* __restrict__ Z, int64_t B,
                                                              double2* __restrict__ ivb, double* __restrict__ ivp,
                                                              double2* __restrict__ ivn)
{
    extern __shared__ double2 fsm[];
    constexpr int L = 1 << LOGL;
    const int N = t.N;
    double2* zf = fsm;      // FFT(z), kept across passes v
    double2* y = fsm + L;   // work buffer
    double* red = (double*)(fsm + 2 * L);  // [5 sums][8 warps]
    const int64_t ma = 2 * (int64_t)blockIdx.x, mb = ma + 1;
    const bool has_b = mb < B;
    const double* Wa = Z + ma * NS * (int64_t)N;
    const double* Wb = Z + mb * NS * (int64_t)N;
    for (int k = threadIdx.x; k < L; k += kFftThreads)
        zf[k] = k < N ? make_double2(Wa[k], has_b ? Wb[k] : 0.0) : make_double2(0.0, 0.0);
    __syncthreads();
    fft_forward<LOGL>(zf, t.tw);
    // this thread's path and steps in the variance loops
    const int half = threadIdx.x >> 7, jt = threadIdx.x & 127;
    const int64_t m = half ? mb : ma;
    const bool active = half ? has_b : true;
    const double* W1 = Z + m * NS * (int64_t)N;  // valid only when active
    for (int v = 0; v < t.n_vol; ++v) {
        const double2* sp = t.spec + (size_t)v * L;
        for (int k = threadIdx.x; k < L; k += kFftThreads) {
            const double2 u = cmul(zf[k], __ldg(sp + k));
            y[k] = make_double2(u.x, -u.y);
        }
        __syncthreads();
        fft_forward<LOGL>(y, t.tw);
        // X = Y2 + a1 W1 + a2 W1perp: Y2_a = Re y = Re FFT(w), Y2_b = Im y = -Im FFT(w)
        const VolDev vol = t.vols[v];
        for (int j = threadIdx.x; j < N; j += kFftThreads) {
            const double2 q = y[j];
            const double xa = q.x + (vol.a1 * Wa[j] + vol.a2 * Wa[N + j]);
            const double xb = has_b ? -q.y + (vol.a1 * Wb[j] + vol.a2 * Wb[N + j]) : 0.0;
            y[j] = make_double2(xa, xb);
        }
        __syncthreads();
        for (int g = vol.vg_begin; g < vol.vg_end; ++g) {
            const VGDev vg = t.vgs[g];
            const double* comp = t.comp + (size_t)g * N;
            double sv = 0.0, sw = 0.0, sp2 = 0.0, nv = 0.0, nw = 0.0;
            if (active) {
                const double sxi = sqrt(vg.xi);
                for (int j = jt; j < vg.nsteps; j += 128) {
                    const double xp = (j == 0) ? 0.0 : (half ? y[j - 1].y : y[j - 1].x);
                    const double su = (j == 0) ? sxi : sxi * exp(0.5 * (vg.eta * (vg.scale * xp) - comp[j - 1]));
                    const double vj = (j == 0) ? vg.xi : su * su;
                    sv += vj;
                    const double sq = su * vg.sdt;
                    sw += sq * W1[j];
                    if (NS == 3) sp2 += sq * W1[2 * N + j];
                    if (ANTI) {
                        const double sa = (j == 0) ? sxi : sxi * exp(0.5 * (vg.eta * (vg.scale * -xp) - comp[j - 1]));
                        nv += (j == 0) ? vg.xi : sa * sa;
                        nw += sa * vg.sdt * -W1[j];
                    }
                }
            }
            sv = half_sum(sv, red, 0);
            sw = half_sum(sw, red, 1);
            if (NS == 3) sp2 = half_sum(sp2, red, 2);
            if (ANTI) {
                nv = half_sum(nv, red, 3);
                nw = half_sum(nw, red, 4);
            }
            if (jt == 0 && active) {
                ivb[(size_t)g * B + m] = make_double2(vg.dt * sv, sw);
                if (NS == 3) ivp[(size_t)g * B + m] = sp2;
                if (ANTI) ivn[(size_t)g * B + m] = make_double2(vg.dt * nv, nw);
            }
            __syncthreads();  // red is reused by the next group
        }
    }
}

size_t path_fp64_fft_smem(int logL) { return (size_t)2 * (16u << logL) + 5 * 8 * sizeof(double); }

int fp64_fft_log2_len(int N)
{
    int logL = kFp64FftMinLogL;
    while ((1 << logL) < 2 * N - 1) ++logL;
    return (N >= 2 && logL <= kFp64FftMaxLogL) ? logL : 0;
}

template <int LOGL>
static void launch_fp64_fft(const Fp64Tables& t, const double* Z, int64_t B, double* ivb, cudaStream_t st,
                            double* ivp, double* ivn)
{
    const size_t smem = path_fp64_fft_smem(LOGL);
    static bool configured = false;
    if (!configured) {
        cudaFuncSetAttribute(k_path_fp64_fft<LOGL, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(k_path_fp64_fft<LOGL, 3, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(k_path_fp64_fft<LOGL, 2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        configured = true;
    }
    const unsigned pairs = (unsigned)((B + 1) / 2);
    if (ivn)
        k_path_fp64_fft<LOGL, 2, true><<<pairs, kFftThreads, smem, st>>>(t, Z, B, (double2*)ivb, nullptr,
                                                                         (double2*)ivn);
    else if (ivp)
        k_path_fp64_fft<LOGL, 3, false><<<pairs, kFftThreads, smem, st>>>(t, Z, B, (double2*)ivb, ivp, nullptr);
    else
        k_path_fp64_fft<LOGL, 2, false><<<pairs, kFftThreads, smem, st>>>(t, Z, B, (double2*)ivb, nullptr, nullptr);
}

int path_fp64_warps(int N)
{
    const size_t budget = 200 * 1024;
    size_t per = 16 * (size_t)N;
    size_t w = (budget - 8 * (size_t)N) / per;
    if (w > 8) w = 8;
    if (w < 1) w = 1;
    return (int)w;
}

size_t path_fp64_smem(int N, int warps) { return 8 * (size_t)N + (size_t)warps * 16 * N; }

void launch_path_fp64(const Fp64Tables& t, const double* Z, int64_t B, double* ivb, void* stream, double* ivp,
                      double* ivn)
{
    const int warps = path_fp64_warps(t.N);
    const size_t smem = path_fp64_smem(t.N, warps);
    static size_t configured = 0;
    if (smem > configured) {
        cudaFuncSetAttribute(k_path_fp64<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(k_path_fp64<3, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(k_path_fp64<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        configured = smem;
    }
    cudaStream_t st = (cudaStream_t)stream;
    if (t.logL > 0) {
        switch (t.logL) {
        case 8: launch_fp64_fft<8>(t, Z, B, ivb, st, ivp, ivn); break;
        case 9: launch_fp64_fft<9>(t, Z, B, ivb, st, ivp, ivn); break;
        case 10: launch_fp64_fft<10>(t, Z, B, ivb, st, ivp, ivn); break;
        case 11: launch_fp64_fft<11>(t, Z, B, ivb, st, ivp, ivn); break;
        default: launch_fp64_fft<12>(t, Z, B, ivb, st, ivp, ivn); break;
        }
        count_launch();
        return;
    }
    const int64_t blocks = (B + warps - 1) / warps;
    if (ivn)
        k_path_fp64<2, true><<<(unsigned)blocks, warps * 32, smem, st>>>(t, Z, B, (double2*)ivb, nullptr,
                                                                         (double2*)ivn);
    else if (ivp)
        k_path_fp64<3, false><<<(unsigned)blocks, warps * 32, smem, st>>>(t, Z, B, (double2*)ivb, ivp, nullptr);
    else
        k_path_fp64<2, false><<<(unsigned)blocks, warps * 32, smem, st>>>(t, Z, B, (double2*)ivb, nullptr, nullptr);
    count_launch();
}

// ------------------------------------------------------------ payoff sums
// The conditional Black-Scholes call by Mills' ratio, the exponential and the
// square root in fixed point (rbg_fixed.cuh): 14 FP64 instructions an output and
// path with the sums (counted; the FP64 pipe is 82 % busy), the strike-independent
// parts shared, against about 250 for library
// log, exp, sqrt and two erfc each time (FP64 pipe: 64 cycles a warp
// operation).  Blocks keep both tables in shared memory (50 KB) and walk over
// (chunk, run of 8 outputs) tasks.  2^17 paths x 21 outputs: 1.17 -> 0.094
// ms; 8192 paths x 2112 outputs: 7.06 -> 0.49 ms.
constexpr int kOPB = 8;  // outputs per task
constexpr int kPayThreads = 256;
constexpr int kPlainPaths = 8;  // paths a thread adds up in one FP64 sum

struct OutF64 {
    double rho, K, lnK, om, hr;  // om = 1 - rho^2 (plain MC: its root), hr = -rho^2 / 2
    int vg;                      // -1 past the last output
    int ok;                      // K in the range of the fast form
};
template <int MC>
struct PayoffSmem {
    uint64_t E[kExpTable];
    MillsTable T;
    OutF64 out[kOPB];
    double red[kPayThreads / 32][2 * kOPB];
    double sum[2 * kOPB], comp[2 * kOPB];  // of a task's rounds so far
};

// Outputs o0 .. o0 + 7 of the task, by the first threads of the block.
template <int MC>
__device__ __forceinline__ void payoff_outs(PayoffSmem<MC>& sm, const Fp64Tables& t, int o0)
{
    if (threadIdx.x < kOPB) {
        const int i = o0 + (int)threadIdx.x;
        const OutDev od = (i < t.n_out) ? t.outs[i] : OutDev{0.0, 1.0, -1, 0};
        const bool ok = od.K > 1e-200 && od.K < 1e200;
        const double om = 1.0 - od.rho * od.rho;
        sm.out[threadIdx.x] = OutF64{od.rho, od.K, (ok && !MC) ? log(od.K) : 0.0, MC ? sqrt(om) : om,
                                     -0.5 * od.rho * od.rho, od.vg, ok};
    }
}

// The tables, and the first task's outputs while they are on their way.  With 8-byte
// loads a few at a time a block's first task waited 10 us longer: 2^16 paths x 5
// outputs 32.8 -> 22.5 us.
// DIRECT: the outputs alone, the tables stay where they are.
template <int MC, bool DIRECT = false>
__device__ __forceinline__ void payoff_start(PayoffSmem<MC>& sm, const Fp64Tables& t, int o0,
                                             const FixedTables* __restrict__ ft)
{
    if (DIRECT) {
        payoff_outs<MC>(sm, t, o0);
        __syncthreads();
        return;
    }
    const TableCopy<kPayThreads, kExpTable * 8> e(ft->exp2);
    const TableCopy<kPayThreads, MC ? 16 : (int)sizeof(MillsTable)> m(&ft->mills);
    payoff_outs<MC>(sm, t, o0);
    e.store(sm.E);
    if (!MC) m.store(&sm.T);
    __syncthreads();
}

// The strike-independent part of a path's conditional call, kept while
// consecutive outputs share variance group and rho.
struct RtState {
    double Iv = 0.0, Is = 0.0, rho = 0.0;
    SpotFixed s{};
    int vg = -1;
    bool ok = false;
};

__device__ __forceinline__ double payoff_rt(RtState& r, const OutF64& o, const double2* __restrict__ ivb, size_t at,
                                            const PayoffSmem<0>& sm)
{
    if (o.vg != r.vg || o.rho != r.rho) {
        const double2 iv = ivb[at];
        r.vg = o.vg;
        r.rho = o.rho;
        r.Iv = iv.x;
        r.Is = iv.y;
        r.ok = spot_fixed(o.om * iv.x, fma(o.hr, iv.x, o.rho * iv.y), sm.E, r.s);
    }
    // zero or undefined conditional variance, spots and strikes out of range: the plain formula
    if (!(r.ok && o.ok)) return rt_payoff(r.Iv, r.Is, o.rho, o.K);
    return call_fixed(r.s, o.K, o.lnK, sm.T, sm.E);
}

// Plain Monte Carlo payoff (rBergLib/rBergomiMT.cpp:134-136 updateZ, :129-132
// scaleZ, :111-116 updateS, aux.h:31-34 posPart): with Z = rho W1 + sqrt(1 - rho^2) Wperp,
// log S = sum sqrt(v) sdt Z - dt/2 sum v = rho IsvdW + sqrt(1 - rho^2) IsvdWp
// - Ivdt / 2, the same sum regrouped by normal stream; the exponential in fixed point.
__device__ __forceinline__ double payoff_mc(const OutF64& o, const double2* __restrict__ ivb,
                                            const double* __restrict__ ivp, size_t at, const uint64_t* E)
{
    const double2 iv = ivb[at];
    const double lnS = o.rho * iv.y + o.om * ivp[at] - 0.5 * iv.x;
    const double d = (fabs(lnS) < 60.0 ? exp2_fixed53(log2e_fixed53(lnS), E) : exp(lnS)) - o.K;
    return d > 0.0 ? d : 0.0;
}

// Warp sums of 16 doubles a lane in the order of the xor tree 16, 8, 4, 2, 1
// (16 additions a lane instead of 80): value lane >> 1 on every lane.
__device__ __forceinline__ double warp_sums16_f64(double (&v)[2 * kOPB])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 8, o = 16; n >= 1; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const double send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// s + e = a + b exactly, s the rounded sum (the larger of the two is found by integers).
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& e)
{
    const bool swap = (double_bits(a) << 1) < (double_bits(b) << 1);
    const double hi = swap ? b : a, lo = swap ? a : b;
    s = hi + lo;
    e = lo - (s - hi);
}

// One round's sums of the block's eight warps into the task's, by one warp: lanes 0-15
// take four warps' sums, lanes 16-31 the other four's; after the last round the
// chunk's (sum, comp, sum2, comp2) of n outputs go to p.
template <int MC>
__device__ __forceinline__ void merge_round(PayoffSmem<MC>& sm, bool first, bool last, double* __restrict__ p, int n)
{
    const int lane = threadIdx.x & 31, k = lane & 15;
    const double(*a)[2 * kOPB] = sm.red + 4 * (lane >> 4);
    double s01, s23, s, e01, e23, e03, e;
    two_sum(a[0][k], a[1][k], s01, e01);
    two_sum(a[2][k], a[3][k], s23, e23);
    two_sum(s01, s23, s, e03);
    e = e01 + e23 + e03;
    two_sum(s, __shfl_xor_sync(0xffffffffu, s, 16), s, e03);
    e += __shfl_xor_sync(0xffffffffu, e, 16) + e03;
    if (!first) {
        two_sum(sm.sum[k], s, s, e03);
        e += sm.comp[k] + e03;
    }
    if (!last) {
        __syncwarp();
        sm.sum[k] = s;
        sm.comp[k] = e;
    } else if (lane < 2 * kOPB && (lane & (kOPB - 1)) < n) {
        p += 4 * (lane & (kOPB - 1)) + 2 * (lane / kOPB);
        p[0] = s;
        p[1] = e;
    }
}

// chunk c covers paths [c G 256, (c+1) G 256) of the batch, G per thread;
// part[(c * n_out + i) * 4 + {0,1,2,3}] = (sum, comp, sum2, comp2).
// ONE: a path a thread, the warps' sums added up by 16 threads (no comp).  Else a
// thread adds up at most kPlainPaths paths in one FP64 sum, and from the warps' sums on
// every rounding error is kept in the compensation.  An FP64 warp instruction holds
// its pipe for 64 cycles: that merge is 16 of them by one warp, another one each
// task, where ONE's is 8 and 2 us faster a call (2^16 paths x 5 outputs 22.9 / 24.9 us).
// Three blocks an SM as the launcher asks for: left to itself the compiler takes 118
// registers and two blocks, 2.66 ms for the grid of 8192 paths x 2112 outputs instead
// of 2.48.
// MC = 1: plain Monte Carlo payoff from (Ivdt, IsvdW) and ivp = IsvdWp.
template <int MC, bool ONE>
__global__ void __launch_bounds__(kPayThreads, 3) k_payoff_sums(Fp64Tables t, const double2* __restrict__ ivb, int64_t B,
                                                     int64_t stride, int G, double* __restrict__ part, int nchunks,
                                                     const double* __restrict__ ivp, const FixedTables* __restrict__ ft)
{
    extern __shared__ __align__(16) uint64_t psm[];
    PayoffSmem<MC>& sm = *reinterpret_cast<PayoffSmem<MC>*>(psm);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t tasks = (int64_t)nchunks * ((t.n_out + kOPB - 1) / kOPB);
    payoff_start<MC>(sm, t, (int)(blockIdx.x / nchunks) * kOPB, ft);
    int sub0 = 0;  // the round of at most kPlainPaths paths a thread
    for (int64_t task = blockIdx.x; task < tasks;) {
        const int c = (int)(task % nchunks), o0 = (int)(task / nchunks) * kOPB;
        if (task != blockIdx.x || sub0) {
            __syncthreads();  // the previous round's readers
            if (!sub0) payoff_outs<MC>(sm, t, o0);
            __syncthreads();
        }
        double s[2 * kOPB];  // sums of x, then of x^2
#pragma unroll
        for (int q = 0; q < 2 * kOPB; ++q) s[q] = 0.0;
        const int sub1 = ONE ? 1 : min(sub0 + kPlainPaths, G);
        for (int sub = sub0; sub < sub1; ++sub) {
            const int64_t m = ((int64_t)c * (ONE ? 1 : G) + sub) * 256 + threadIdx.x;
            if (m >= B) break;
            RtState r;
#pragma unroll
            for (int q = 0; q < kOPB; ++q) {
                const OutF64 o = sm.out[q];
                if (o.vg < 0) continue;
                const size_t at = (size_t)o.vg * stride + m;
                double x;
                if constexpr (MC) x = payoff_mc(o, ivb, ivp, at, sm.E);
                else x = payoff_rt(r, o, ivb, at, sm);
                s[q] += x;
                s[kOPB + q] = fma(x, x, s[kOPB + q]);
            }
        }
        const double v = warp_sums16_f64(s);
        if (!(lane & 1)) sm.red[w][lane >> 1] = v;
        __syncthreads();
        if constexpr (ONE) {
            const int q = threadIdx.x & (kOPB - 1), z = threadIdx.x / kOPB;
            if (threadIdx.x < 2 * kOPB && o0 + q < t.n_out) {
                double S = 0;
                for (int k = 0; k < kPayThreads / 32; ++k) S += sm.red[k][threadIdx.x];
                double* p = part + ((size_t)c * t.n_out + o0 + q) * 4 + 2 * z;
                p[0] = S;
                p[1] = 0.0;
            }
        } else if (w == (int)(task & (kPayThreads / 32 - 1))) {
            merge_round<MC>(sm, sub0 == 0, sub1 == G, part + ((size_t)c * t.n_out + o0) * 4, t.n_out - o0);
        }
        if (!ONE && sub1 < G) {
            sub0 = sub1;
        } else {
            sub0 = 0;
            task += gridDim.x;
        }
    }
}

// Raises a payoff kernel's shared-memory limit, once per device.
template <class F>
static bool payoff_smem_ready(F* kern, size_t bytes, bool (&ready)[64])
{
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    std::lock_guard<std::mutex> lk(mu);
    if (!ready[dev] && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess)
        ready[dev] = true;
    return ready[dev];
}

int launch_payoff_sums(const Fp64Tables& t, const double* ivb, int64_t B, int64_t stride, int G, double* part,
                       int nchunks, void* stream, const double* ivp)
{
    static bool ready[4][64] = {};
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    const int64_t tasks = (int64_t)nchunks * ((t.n_out + kOPB - 1) / kOPB);
    const unsigned grid = (unsigned)std::min<int64_t>(tasks, 3 * (int64_t)device_sms());
    auto* kern = ivp ? (G == 1 ? k_payoff_sums<1, true> : k_payoff_sums<1, false>)
                     : (G == 1 ? k_payoff_sums<0, true> : k_payoff_sums<0, false>);
    const size_t smem = ivp ? sizeof(PayoffSmem<1>) : sizeof(PayoffSmem<0>);
    if (!payoff_smem_ready(kern, smem, ready[(ivp ? 2 : 0) + (G == 1)])) return -1;
    kern<<<grid, kPayThreads, smem, (cudaStream_t)stream>>>(t, (const double2*)ivb, B, stride, G, part, nchunks, ivp, ft);
    count_launch();
    return 0;
}

// ------------------------------------------------------------ chunk merge
// A call's chunk sums of one output, added exactly: the doubles become 128-bit
// integers in units of 2^-52 of the largest one's last bit, whose additions
// cost a few integer instructions and do not depend on their order.  (A
// compensated FP64 tree of 600 chunks took 14-17 us of serial warp operations
// on GB300's FP64 pipe.)
struct Fix128 {
    uint64_t lo;
    int64_t hi;
};

__device__ __forceinline__ void fix_add(Fix128& a, uint64_t lo, int64_t hi)
{
    const uint64_t s = a.lo + lo;
    a.hi += hi + (s < lo ? 1 : 0);
    a.lo = s;
}

__device__ __forceinline__ int double_exp(double x) { return (int)((double_bits(x) >> 52) & 2047u); }

// a += x, x's exponent field at most emax (< 2047); bits more than 52 places
// below emax's last one are dropped.
__device__ __forceinline__ void fix_add_double(Fix128& a, double x, int emax)
{
    const uint64_t b = double_bits(x);
    const int e = (int)(b >> 52) & 2047;
    uint64_t m = b & 0x000FFFFFFFFFFFFFull;
    if (e) m |= 0x0010000000000000ull;
    const int sh = 52 - (emax - (e ? e : 1));  // left shift of the significand in the 128-bit frame
    uint64_t lo = 0, hi = 0;
    if (sh > 0) {
        lo = m << sh;
        hi = m >> (64 - sh);
    } else if (sh > -64) {
        lo = m >> -sh;
    }
    if (b >> 63) {  // two's complement
        lo = ~lo + 1;
        hi = ~hi + (lo == 0 ? 1 : 0);
    }
    fix_add(a, lo, (int64_t)hi);
}

// a in the frame of emax as S + C, S its leading 53 bits.
__device__ void fix_split(const Fix128& a, int emax, double& S, double& C)
{
    uint64_t lo = a.lo, hi = (uint64_t)a.hi;
    const bool neg = a.hi < 0;
    if (neg) {
        lo = ~lo + 1;
        hi = ~hi + (lo == 0 ? 1 : 0);
    }
    S = C = 0.0;
    const int unit = emax - 1075 - 52;  // the frame's last bit is 2^unit
    double part[2] = {0.0, 0.0};
    for (int k = 0; k < 2 && (hi | lo); ++k) {
        const int top = hi ? 127 - __clzll((long long)hi) : 63 - __clzll((long long)lo);
        const int cut = top > 52 ? top - 52 : 0;  // the 53 bits from `top` down
        uint64_t m;
        if (cut >= 64) {
            m = hi >> (cut - 64);
            hi &= (1ull << (cut - 64)) - 1;
        } else {
            m = cut ? ((lo >> cut) | (hi << (64 - cut))) : lo;
            hi = 0;
            lo &= cut ? ((1ull << cut) - 1) : 0ull;
        }
        part[k] = ldexp((double)(long long)m, unit + cut);
    }
    S = neg ? -part[0] : part[0];
    C = neg ? -part[1] : part[1];
}

constexpr int kMergeThreads = 128;                  // that add up the chunks
constexpr int kMergeBlock = kMergeThreads + 32;     // and the warp of the implied volatility
struct MergeSmem {
    Fix128 s[kMergeThreads / 32][2];
    int emax[kMergeThreads / 32][2];
    double out[4];
};

// Output i: acc (S, C, S2, C2) plus every chunk's, or just these where `fresh`;
// stored to acc and sm.out.  By the first kMergeThreads threads of the block, which
// wait for one another only.  A sum with a NaN or infinity in
// it is added up in FP64 by one thread.
__device__ __forceinline__ void merge_add(const double* __restrict__ part, int nchunks, int n_out,
                                          double* __restrict__ acc, int i, bool fresh, MergeSmem& sm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    auto adders = [] { asm volatile("barrier.sync 1, %0;" ::"n"(kMergeThreads) : "memory"); };
    // the largest exponent of either sum
    int em[2] = {0, 0};
    for (int c = threadIdx.x; c < nchunks; c += kMergeThreads) {
        const double2* p = reinterpret_cast<const double2*>(part + ((size_t)c * n_out + i) * 4);
        const double2 x = p[0], y = p[1];
        em[0] = max(em[0], max(double_exp(x.x), double_exp(x.y)));
        em[1] = max(em[1], max(double_exp(y.x), double_exp(y.y)));
    }
    if (!fresh)
        for (int z = 0; z < 2; ++z) em[z] = max(em[z], max(double_exp(acc[i * 4 + 2 * z]), double_exp(acc[i * 4 + 2 * z + 1])));
#pragma unroll
    for (int z = 0; z < 2; ++z) {
        em[z] = __reduce_max_sync(0xffffffffu, em[z]);
        if (lane == 0) sm.emax[w][z] = em[z];
    }
    adders();
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int k = 0; k < kMergeThreads / 32; ++k) em[z] = max(em[z], sm.emax[k][z]);
    Fix128 s[2] = {{0, 0}, {0, 0}};
    for (int c = threadIdx.x; c < nchunks; c += kMergeThreads) {
        const double2* p = reinterpret_cast<const double2*>(part + ((size_t)c * n_out + i) * 4);
        const double2 x = p[0], y = p[1];
        fix_add_double(s[0], x.x, em[0]);
        fix_add_double(s[0], x.y, em[0]);
        fix_add_double(s[1], y.x, em[1]);
        fix_add_double(s[1], y.y, em[1]);
    }
    if (!fresh && threadIdx.x == 0) {
        for (int z = 0; z < 2; ++z) {
            fix_add_double(s[z], acc[i * 4 + 2 * z], em[z]);
            fix_add_double(s[z], acc[i * 4 + 2 * z + 1], em[z]);
        }
    }
#pragma unroll
    for (int z = 0; z < 2; ++z) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            fix_add(s[z], __shfl_xor_sync(0xffffffffu, s[z].lo, o), __shfl_xor_sync(0xffffffffu, s[z].hi, o));
        if (lane == 0) sm.s[w][z] = s[z];
    }
    adders();
    if (threadIdx.x < 2) {
        const int z = threadIdx.x;
        double S, C;
        if (em[z] < 2047) {
            Fix128 t = sm.s[0][z];
            for (int k = 1; k < kMergeThreads / 32; ++k) fix_add(t, sm.s[k][z].lo, sm.s[k][z].hi);
            fix_split(t, em[z], S, C);
        } else {
            S = fresh ? 0.0 : acc[i * 4 + 2 * z] + acc[i * 4 + 2 * z + 1];
            C = 0.0;
            for (int c = 0; c < nchunks; ++c) S += part[((size_t)c * n_out + i) * 4 + 2 * z];
        }
        acc[i * 4 + 2 * z] = sm.out[2 * z] = S;
        acc[i * 4 + 2 * z + 1] = sm.out[2 * z + 1] = C;
    }
}

// The same on every thread of the block, in v; the last warp only waits.
__device__ void merge_block(const double* __restrict__ part, int nchunks, int n_out, double* __restrict__ acc, int i,
                            bool fresh, MergeSmem& sm, double (&v)[4])
{
    if (threadIdx.x < kMergeThreads) merge_add(part, nchunks, n_out, acc, i, fresh, sm);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = sm.out[k];
}

// ------------------------------------------------------------- IV (FP64)
// The out-of-the-money Black-Scholes price (S0 = 1, r = 0; put for K < 1) at v =
// s sqrt(T) and what its derivatives need: f = phi(d1), vega = f sqrt(T).  lnK =
// ln K.
struct OtmPrice {
    double p, f;
    float d1d2;
};

// The price for |d1| above 37.6: below the doubles' normal range, which erfc still has.
// (Not inlined: four copies of two erfc made the merge kernel 2 us longer.)
__device__ __noinline__ double otm_far(double K, double d1, double v, bool put)
{
    return put ? fma(K, phi_cdf(v - d1), -phi_cdf(-d1)) : fma(-K, phi_cdf(d1 - v), phi_cdf(d1));
}

__device__ __forceinline__ OtmPrice otm_price(double K, double lnK, double v, bool put, const FixedTables* __restrict__ ft)
{
    const double d1 = fma(-lnK, 1.0 / v, 0.5 * v);
    const bool n1 = d1 < 0.0;
    const uint64_t x1 = tail_fixed(d1);
    const int64_t d2 = (n1 ? -(int64_t)x1 : (int64_t)x1) - (int64_t)tail_fixed(v);
    const bool n2 = !put || d2 < 0;  // out of the money a call's d2 is negative, if only just
    OtmPrice r;
    r.d1d2 = (float)d1 * ((float)d1 - (float)v);
    const uint64_t hs = half_square_log2(x1);
    constexpr uint64_t lim = density_limit(-kLog2Sqrt2Pi53);
    r.f = density_fixed(-kLog2Sqrt2Pi53, hs, lim, ft->exp2);
    const int64_t m1 = (int64_t)mills_fixed(x1, ft->mills), m2 = (int64_t)mills_fixed((uint64_t)(n2 ? -d2 : d2), ft->mills);
    // call: [d1 >= 0] - K [d2 >= 0] + f (-+ M1 +- M2); put: less 1 - K, which only leaves K [d2 < 0]
    const double base = put ? (n2 ? K : 0.0) : (n1 ? 0.0 : 1.0);
    r.p = fma(r.f, tail_to_double((n1 ? m1 : -m1) + (n2 ? -m2 : m2)), base);
    if (hs >= lim) r.p = otm_far(K, d1, v, put);
    return r;
}

// The same price in FP32: the bracketing rounds of implied_vol_warp.  lnK1 =
// ln(1 / K), sqT = sqrt(T).
__device__ __forceinline__ float bs_gen_f32(float lnK1, float sqT, float K, float s, int put)
{
    const float ssq = s * sqT;
    const float d1 = fmaf(0.5f, ssq, lnK1 * rcp_approx(ssq));
    const float d2 = d1 - ssq;
    return put ? fmaf(K, phi_f32(-d2), -phi_f32(-d1)) : fmaf(-K, phi_f32(d2), phi_f32(d1));
}

// log(p / target) for e = p / target - 1
__device__ __forceinline__ double log_ratio(double e)
{
    if (fabs(e) > 1e-3) return log1p(e);
    double s = fma(e, -1.0 / 6, 1.0 / 5);
    s = fma(e, s, -1.0 / 4);
    s = fma(e, s, 1.0 / 3);
    s = fma(e, s, -1.0 / 2);
    return fma(e * e, s, e);
}

// What implied_vol_warp needs of strike and maturity alone; p0: the lane's price
// on the geometric grid.
struct IvStart {
    double lnK, sqT;
    float lnK1, sqT32, p0;
};
__device__ __forceinline__ IvStart iv_start(double K, double T)
{
    IvStart r;
    r.lnK = log(K);
    r.sqT = sqrt(T);
    r.lnK1 = -log1pf((float)(K - 1.0));
    r.sqT32 = sqrtf((float)T);
    r.p0 = bs_gen_f32(r.lnK1, r.sqT32, (float)K, 1e-3f * exp2f(0.5f * (threadIdx.x & 31)), 1.0 > K);
    return r;
}

// Implied vol by a warp: inverts on the out-of-the-money side (put-call
// parity for K < 1, as rBergLib/BlackScholes.cpp:38-41 does).  The 32 lanes
// price 32 volatilities at once:
//   1. a geometric grid 1e-3 * 2^(l/2) brackets the root within a factor
//      sqrt(2), in FP32; where the FP32 grid brackets nothing, the same grid in
//      FP64 decides (no bracket there: no volatility fits, NaN);
//   2. three 33-section rounds in FP32 narrow the bracket ~36,000-fold (FP32
//      resolves it no further);
//   3. one FP64 step checks the narrowed bracket, widened by 1e-4 (near the
//      money FP32 prices cancel to a few 1e-6: a margin of 1e-6 sent those
//      outputs to step 4's search, 60 us longer): lanes 0 and 1 price its
//      ends, the others its middle; if the check fails -- FP32 cannot resolve
//      the price, e.g. far in a wing -- the FP64 grid and FP64 33-section
//      rounds (to 1e-6) take over;
//   4. from the checked bracket's middle one Halley step on the log price
//      (cubic: from 1e-5 the error left is 1e-15 near the money, below ~1e-12
//      in the wings), then safeguarded Newton on the log price where a step is
//      still larger than that.
// Prices are Mills' ratios (otm_price): the density they contain is the vega,
// so an FP64 step is one short chain.  All lanes
// return the same value; NaN when no volatility fits.
__device__ double implied_vol_warp(double price, double K, double T, const IvStart& st,
                                   const FixedTables* __restrict__ ft)
{
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int put = 1.0 > K;
    const double target = put ? price - 1.0 + K : price;
    const double upper = put ? K : 1.0;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    // (strikes and maturities that are NaN or infinite included)
    constexpr double most = 1.7976931348623157e308;
    if (!(target > 0.0) || !(target < upper) || !(T > 0.0) || !(T <= most) || !(K <= most)) return nan;
    const double lnK = st.lnK, sqT = st.sqT;
    const float lnK1 = st.lnK1, sqT32 = st.sqT32, K32 = (float)K, t32 = (float)target;
    double lo = 0.0, hi = 0.0, s = 0.0;
    bool narrowed = false;
    OtmPrice q{};
    {
        // FP32 grid and rounds, then the FP64 check
        const unsigned b32 = __ballot_sync(FULL, st.p0 >= t32);
        if (b32 != 0u) {
            const int f = __ffs(b32) - 1;
            float lo32 = (f > 0) ? 1e-3f * exp2f(0.5f * (f - 1)) : 0.f, hi32 = 1e-3f * exp2f(0.5f * f);
#pragma unroll 1
            for (int it = 0; it < 3; ++it) {
                const float sl = fmaf(hi32 - lo32, (float)(lane + 1) * (1.0f / 33.0f), lo32);
                const unsigned bb = __ballot_sync(FULL, bs_gen_f32(lnK1, sqT32, K32, sl, put) >= t32);
                const int ff = bb ? __ffs(bb) - 1 : 32;
                const float nlo = __shfl_sync(FULL, sl, ff > 0 ? ff - 1 : 0);
                const float nhi = __shfl_sync(FULL, sl, ff < 32 ? ff : 31);
                if (ff > 0) lo32 = nlo;
                if (ff < 32) hi32 = nhi;
            }
            const double mid = 0.5 * ((double)lo32 + (double)hi32);
            const double lo2 = fmax((double)lo32 - 1e-4 * mid, 1e-12), hi2 = (double)hi32 + 1e-4 * mid;
            const double sv = lane == 0 ? lo2 : (lane == 1 ? hi2 : mid);
            q = otm_price(K, lnK, sv * sqT, put, ft);
            const double plo = __shfl_sync(FULL, q.p, 0), phi_ = __shfl_sync(FULL, q.p, 1);
            if (plo < target && phi_ >= target) {
                narrowed = true;
                lo = lo2;
                hi = hi2;
                s = mid;
            }
        }
    }
    if (!narrowed) {
        // FP64 grid, then FP64 33-section rounds (one evaluation per lane)
        // until the bracket is within 1e-6 relative
        const double sig = 1e-3 * exp2(0.5 * lane);
        unsigned b = __ballot_sync(FULL, otm_price(K, lnK, sig * sqT, put, ft).p >= target);
        if (b == 0u) return nan;
        int f = __ffs(b) - 1;
        lo = (f > 0) ? 1e-3 * exp2(0.5 * (f - 1)) : 0.0;
        hi = 1e-3 * exp2(0.5 * f);
        for (int it = 0; it < 14 && hi - lo > 1e-6 * hi; ++it) {
            const double sl = lo + (hi - lo) * (double)(lane + 1) / 33.0;
            b = __ballot_sync(FULL, otm_price(K, lnK, sl * sqT, put, ft).p >= target);
            f = b ? __ffs(b) - 1 : 32;
            const double nlo = __shfl_sync(FULL, sl, f > 0 ? f - 1 : 0);
            const double nhi = __shfl_sync(FULL, sl, f < 32 ? f : 31);
            if (f > 0) lo = nlo;
            if (f < 32) hi = nhi;
        }
        s = 0.5 * (lo + hi);
    }
    if (narrowed) {
        // Halley on g(s) = log p(s) - log target: with r = g / g', g'' / g' = d1 d2 / s - vega / p,
        // the step is r / (1 - r g'' / (2 g')); the bracket's ends move to the middle's side.
        // (Lanes 0 and 1 hold the ends' prices: lane 2's values decide.)
        const double vega = q.f * sqT;
        const double r = log_ratio((q.p - target) / target) * (q.p / vega);
        const float h = 0.5f * (float)r * (q.d1d2 / (float)s - (float)vega / (float)q.p);
        const double step = r + r * (double)(h / (1.0f - h));
        double nt = __shfl_sync(FULL, s - step, 2);
        const bool above = __shfl_sync(FULL, q.p > target ? 1 : 0, 2) != 0;
        if (nt > lo && nt < hi) {
            if (fabs(nt - s) <= 1e-5 * s) return nt;  // cubic: the error left is below ~1e-12 relative
            if (above) hi = s;
            else lo = s;
            if (!(nt > lo && nt < hi)) nt = 0.5 * (lo + hi);
            s = nt;
        } else {
            if (above) hi = s;
            else lo = s;
            s = 0.5 * (lo + hi);
        }
    }
    // safeguarded Newton on the log price (every lane computes the same
    // iterate).  A Newton step below 1e-14 relative ends the search: the
    // convergence is quadratic, so the iterate it gives is at roundoff.  A
    // step that leaves the bracket, or a vanishing price, falls back to
    // bisection; 40 halvings take a 1e-6 bracket below 1e-15 on their own.
    for (int it = 0; it < 40; ++it) {
        q = otm_price(K, lnK, s * sqT, put, ft);
        if (q.p == target) break;
        if (q.p > target) hi = s;
        else lo = s;
        double sn = 0.5 * (lo + hi);
        if (q.p > 0.0) {
            const double nt = s - log_ratio((q.p - target) / target) * q.p / (q.f * sqT);
            if (fabs(nt - s) <= 1e-14 * s) {
                s = nt;
                break;
            }
            if (nt > lo && nt < hi) sn = nt;
        }
        s = sn;
        if (hi - lo <= 1e-15 * hi) break;
    }
    return s;
}

// Output i of a merge: its sums, price and stat by the first thread, its implied
// volatility by the last warp, which takes what depends on strike and maturity
// alone (logarithm, root, the FP32 grid) while the others add up the chunks.
// res: [0,n) price, [n,2n) stat, [2n,3n) iv, [3n,4n) sum, [4n,5n) sum2.
__device__ __forceinline__ void merge_finish(const double* __restrict__ part, int nchunks, int n_out,
                                             double* __restrict__ acc, int i, bool fresh, double invM, double isqM,
                                             const OutDev* __restrict__ outs, const double* __restrict__ Tv,
                                             int compute_iv, double* __restrict__ res,
                                             const FixedTables* __restrict__ ft, MergeSmem& sm)
{
    double v[4];
    const bool solve = threadIdx.x >= kMergeThreads && res;
    double K = 1.0, T = 1.0;
    IvStart start{};
    if (solve && compute_iv) {
        K = outs[i].K;
        T = Tv[i];
        start = iv_start(K, T);
    }
    merge_block(part, nchunks, n_out, acc, i, fresh, sm, v);
    if (!res) return;
    const double S = v[0] + v[1];
    const double price = S * invM;
    if (solve) {
        const double iv = compute_iv ? implied_vol_warp(price, K, T, start, ft) : 0.0;
        if (threadIdx.x == kMergeThreads) res[2 * n_out + i] = iv;
    } else if (threadIdx.x == 0) {
        // rBergLib/rBergomiMT.cpp:404-409
        const double S2 = v[2] + v[3];
        const double var = 1.0 * (S2 * invM) + -1.0 * (price * price);
        res[i] = price;
        res[n_out + i] = sqrt(var) * isqM;
        res[3 * n_out + i] = S;
        res[4 * n_out + i] = S2;
    }
}

// One block per output: its chunk sums into acc and, after the call's last
// batch (res non-null), the price, stat and implied vol.
__global__ void __launch_bounds__(kMergeBlock) k_merge(const double* __restrict__ part, int nchunks, int n_out,
                                                      double* __restrict__ acc, int fresh, double invM, double isqM,
                                                      const OutDev* __restrict__ outs, const double* __restrict__ Tv,
                                                      int compute_iv, double* __restrict__ res,
                                                      const FixedTables* __restrict__ ft)
{
    __shared__ MergeSmem sm;
    merge_finish(part, nchunks, n_out, acc, blockIdx.x, fresh != 0, invM, isqM, outs, Tv, compute_iv, res, ft, sm);
}

// Job-table form: block b is output b - jobs[k].block0 of job k (both tables).
__global__ void __launch_bounds__(kMergeBlock) k_merge_jobs(const AccJob* __restrict__ jobs,
                                                           const FinJob* __restrict__ fins, int n_jobs,
                                                           const FixedTables* __restrict__ ft)
{
    __shared__ MergeSmem sm;
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].block0 <= (int64_t)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const AccJob& J = jobs[lo];
    const FinJob& F = fins[lo];
    const int i = (int)((int64_t)blockIdx.x - J.block0);
    merge_finish(J.part, J.nchunks, J.n_out, J.acc, i, true, F.invM, F.isqM, F.outs, F.Tv, F.compute_iv, F.res, ft, sm);
}

int launch_merge_jobs(const AccJob* jobs, const FinJob* fins, int n_jobs, int64_t blocks, void* stream)
{
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    k_merge_jobs<<<(unsigned)blocks, kMergeBlock, 0, (cudaStream_t)stream>>>(jobs, fins, n_jobs, ft);
    count_launch();
    return 0;
}

// Loads the merge kernels and looks up their tables (a serving loop's first
// request must not meet either).
void reduce_preload()
{
    cudaFuncAttributes fa;
    cudaFuncGetAttributes(&fa, k_merge);
    cudaFuncGetAttributes(&fa, k_merge_jobs);
    fixed_tables();
    cudaGetLastError();
}

int launch_merge(const double* part, int nchunks, int n_out, double* acc, bool fresh, void* stream, const MergeFinal* fin)
{
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    const MergeFinal f = fin ? *fin : MergeFinal{};
    k_merge<<<n_out, kMergeBlock, 0, (cudaStream_t)stream>>>(
        part, nchunks, n_out, acc, fresh ? 1 : 0, fin ? 1.0 / (double)f.M : 0.0, fin ? 1.0 / std::sqrt((double)f.M) : 0.0,
        f.outs, f.Tv, f.compute_iv, f.res, ft);
    count_launch();
    return 0;
}

__global__ void k_implied_vol(int n, const double* price, const double* K, const double* T, double* iv,
                              const FixedTables* __restrict__ ft)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= n) return;
    const double v = implied_vol_warp(price[i], K[i], T[i], iv_start(K[i], T[i]), ft);
    if ((threadIdx.x & 31) == 0) iv[i] = v;
}

int launch_implied_vol(int n, const double* price, const double* K, const double* T, double* iv, void* stream)
{
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    k_implied_vol<<<n, 32, 0, (cudaStream_t)stream>>>(n, price, K, T, iv, ft);  // one warp (output) per block
    count_launch();
    return 0;
}

// ------------------------------------------------------------ quadrature
// payoff[m * n_out + i]: tasks of 256 paths x nq <= 8 outputs.
// DIRECT (plain Monte Carlo, a task a block): the exponential's table is read from
// device memory, one entry a payoff; copying it first took longer than the rest (a call
// of 64 paths of 16 steps x 5 outputs: 66 us with the table copied, 59 so).
template <int MC, bool DIRECT>
__global__ void __launch_bounds__(kPayThreads) k_payoff_store(Fp64Tables t, const double2* __restrict__ ivb, int64_t B,
                               int64_t stride, double* __restrict__ payoff, const double* __restrict__ ivp, int nq,
                               const FixedTables* __restrict__ ft)
{
    extern __shared__ __align__(16) uint64_t psm[];
    PayoffSmem<MC>& sm = *reinterpret_cast<PayoffSmem<MC>*>(psm);
    const int64_t tiles = (B + kPayThreads - 1) / kPayThreads, tasks = tiles * ((t.n_out + nq - 1) / nq);
    payoff_start<MC, DIRECT>(sm, t, (int)(blockIdx.x / tiles) * nq, ft);
    const uint64_t* E = DIRECT ? ft->exp2 : sm.E;
    for (int64_t task = blockIdx.x; task < tasks; task += gridDim.x) {
        const int o0 = (int)(task / tiles) * nq;
        const int64_t m = task % tiles * kPayThreads + threadIdx.x;
        if (task != blockIdx.x) {
            __syncthreads();  // the previous task's readers
            payoff_outs<MC>(sm, t, o0);
            __syncthreads();
        }
        if (m >= B) continue;
        RtState r;
        for (int q = 0; q < nq; ++q) {
            const OutF64 o = sm.out[q];
            if (o.vg < 0) continue;
            const size_t at = (size_t)o.vg * stride + m;
            double x;
            if constexpr (MC) x = payoff_mc(o, ivb, ivp, at, E);
            else x = payoff_rt(r, o, ivb, at, sm);
            payoff[m * t.n_out + o0 + q] = x;
        }
    }
}

int launch_payoff_store(const Fp64Tables& t, const double* ivb, int64_t B, int64_t stride, double* payoff,
                        void* stream, const double* ivp)
{
    static bool ready[3][64] = {};
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    // fewer outputs a task where 8 would leave SMs idle
    const int64_t tiles = (B + kPayThreads - 1) / kPayThreads, most = 3 * (int64_t)device_sms();
    int nq = kOPB;
    while (nq > 1 && tiles * ((t.n_out + nq - 1) / nq) < 2 * (int64_t)device_sms()) nq >>= 1;
    const int64_t tasks = tiles * ((t.n_out + nq - 1) / nq);
    const bool direct = ivp && tasks <= most;
    auto* kern = !ivp ? k_payoff_store<0, false> : direct ? k_payoff_store<1, true> : k_payoff_store<1, false>;
    const size_t smem = ivp ? sizeof(PayoffSmem<1>) : sizeof(PayoffSmem<0>);
    if (!payoff_smem_ready(kern, smem, ready[!ivp ? 0 : direct ? 2 : 1])) return -1;
    kern<<<(unsigned)std::min(tasks, most), kPayThreads, smem, (cudaStream_t)stream>>>(t, (const double2*)ivb, B, stride,
                                                                                     payoff, ivp, nq, ft);
    count_launch();
    return 0;
}

// ------------------------------------------------------- control variate
// The Romano-Touzi estimator with the control variate of McCrickerd and
// Pakkanen and antithetic paths, as ML_console_ST/RBergomi.cpp implements it
// (estimateControlVariate :493-540, ComputePriceRTVarRed :218-289,
// updatePayoffControlVariate :478-491).
//   X = BS(S, K, 1, sqrt((1 - rho^2) Ivdt)),  S = exp(-rho^2 Ivdt / 2 + rho IsvdW)
//   Y = BS(S, K, 1, sqrt(rho^2 (Q - Ivdt)))   (Qmax in place of Q where Q <= Ivdt)

// Fixed-shape block sum (256 threads): the same order on every run.
__device__ double block_sum_256(double x, double* red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    double t = 0.0;
    for (int k = 0; k < 8; ++k) t += red[k];
    return t;
}

// One block of 256 threads per output: Q = max_m 2 Ivdt_m; X_m, Y_m on the
// pilot paths (stored in xy); means; centred covariance sums (two passes, as
// aux.h:206-220 computes them); alpha = -cov(X, Y) / cov(Y, Y).
__global__ void __launch_bounds__(256) k_cv_pilot(Fp64Tables t, const double2* __restrict__ ivb, int64_t Mc,
                                                  double* __restrict__ xy, double* __restrict__ alpha,
                                                  double* __restrict__ Qout)
{
    __shared__ double red[8];
    const int i = blockIdx.x;
    const OutDev od = t.outs[i];
    const double2* iv = ivb + (size_t)od.vg * Mc;
    double* X = xy + (size_t)i * 2 * Mc;
    double* Y = X + Mc;
    double q = 0.0;
    for (int64_t m = threadIdx.x; m < Mc; m += 256) q = fmax(q, 2 * iv[m].x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q = fmax(q, __shfl_xor_sync(0xffffffffu, q, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = q;
    __syncthreads();
    q = 0.0;
    for (int k = 0; k < 8; ++k) q = fmax(q, red[k]);
    const double r = od.rho;
    double sx = 0.0, sy = 0.0;
    for (int64_t m = threadIdx.x; m < Mc; m += 256) {
        const double a = iv[m].x, b = iv[m].y;
        const double spot = exp(-0.5 * r * r * a + r * b);
        X[m] = bs_call_tau1(spot, od.K, sqrt((1.0 - r * r) * a));
        Y[m] = bs_call_tau1(spot, od.K, sqrt(r * r * (q - a)));
        sx += X[m];
        sy += Y[m];
    }
    const double mx = block_sum_256(sx, red) / (double)Mc;
    const double my = block_sum_256(sy, red) / (double)Mc;
    double cxy = 0.0, cyy = 0.0;
    for (int64_t m = threadIdx.x; m < Mc; m += 256) {
        const double dy = Y[m] - my;
        cxy += (X[m] - mx) * dy;
        cyy += dy * dy;
    }
    cxy = block_sum_256(cxy, red);
    cyy = block_sum_256(cyy, red);
    if (threadIdx.x == 0) {
        alpha[i] = -(cxy / (double)(Mc - 1)) / (cyy / (double)(Mc - 1));
        Qout[i] = q;
    }
}

void launch_cv_pilot(const Fp64Tables& t, const double* ivb, int64_t Mc, double* xy, double* alpha, double* Q,
                     void* stream)
{
    k_cv_pilot<<<t.n_out, 256, 0, (cudaStream_t)stream>>>(t, (const double2*)ivb, Mc, xy, alpha, Q);
    count_launch();
}

__device__ __forceinline__ double cv_half(double2 iv, double rho, double K, double alpha, double Q, double Qmax,
                                          unsigned& exc)
{
    const double spot = exp(-0.5 * rho * rho * iv.x + rho * iv.y);
    const double x = bs_call_tau1(spot, K, sqrt((1.0 - rho * rho) * iv.x));
    const bool inside = Q > iv.x;
    if (!inside) ++exc;
    const double y = bs_call_tau1(spot, K, inside ? sqrt(rho * rho * (Q - iv.x)) : sqrt(rho * rho * (Qmax - iv.x)));
    return x + alpha * y;
}

// grid (nchunks, ceil(n_out / kOPB)), as k_payoff_sums: per path the
// antithetic mean 0.5 (f(W) + f(-W)).
__global__ void __launch_bounds__(256) k_payoff_sums_cv(Fp64Tables t, const double2* __restrict__ ivb,
                                                        const double2* __restrict__ ivn, int64_t B,
                                                        const double* __restrict__ alpha,
                                                        const double* __restrict__ Q, double Qmax, int G,
                                                        double* __restrict__ part,
                                                        unsigned long long* __restrict__ count)
{
    __shared__ double red[8][kOPB][2];
    const int c = blockIdx.x;
    const int o0 = blockIdx.y * kOPB;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double S = 0, CS = 0, S2 = 0, CS2 = 0;
    OutDev od[kOPB];
    double al[kOPB], qq[kOPB];
    unsigned exc[kOPB];
#pragma unroll
    for (int q = 0; q < kOPB; ++q) {
        const int i = o0 + q;
        od[q] = (i < t.n_out) ? t.outs[i] : OutDev{0.0, 1.0, -1, 0};
        al[q] = (i < t.n_out) ? alpha[i] : 0.0;
        qq[q] = (i < t.n_out) ? Q[i] : 0.0;
        exc[q] = 0;
    }
    for (int sub = 0; sub < G; ++sub) {
        const int64_t m = ((int64_t)c * G + sub) * 256 + threadIdx.x;
#pragma unroll
        for (int q = 0; q < kOPB; ++q) {
            double x = 0.0;
            if (m < B && od[q].vg >= 0) {
                const size_t at = (size_t)od[q].vg * B + m;
                x = 0.5 * cv_half(ivb[at], od[q].rho, od[q].K, al[q], qq[q], Qmax, exc[q]);
                x += 0.5 * cv_half(ivn[at], od[q].rho, od[q].K, al[q], qq[q], Qmax, exc[q]);
            }
            double x2 = x * x;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                x += __shfl_xor_sync(0xffffffffu, x, o);
                x2 += __shfl_xor_sync(0xffffffffu, x2, o);
            }
            if (lane == 0) { red[w][q][0] = x; red[w][q][1] = x2; }
        }
        __syncthreads();
        if (threadIdx.x < kOPB) {
            const int q = threadIdx.x;
            double a = 0, a2 = 0;
            for (int k = 0; k < 8; ++k) { a += red[k][q][0]; a2 += red[k][q][1]; }
            neumaier_add(S, CS, a);
            neumaier_add(S2, CS2, a2);
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < kOPB; ++q) {
        unsigned e = exc[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
        if (lane == 0 && e && o0 + q < t.n_out) atomicAdd(count + o0 + q, (unsigned long long)e);
    }
    if (threadIdx.x < kOPB && o0 + (int)threadIdx.x < t.n_out) {
        double* p = part + ((size_t)c * t.n_out + o0 + threadIdx.x) * 4;
        p[0] = S; p[1] = CS; p[2] = S2; p[3] = CS2;
    }
}

void launch_payoff_sums_cv(const Fp64Tables& t, const double* ivb, const double* ivn, int64_t B, const double* alpha,
                           const double* Q, double Qmax, int G, double* part, unsigned long long* count, int nchunks,
                           void* stream)
{
    dim3 grid(nchunks, (t.n_out + kOPB - 1) / kOPB);
    k_payoff_sums_cv<<<grid, 256, 0, (cudaStream_t)stream>>>(t, (const double2*)ivb, (const double2*)ivn, B, alpha,
                                                             Q, Qmax, G, part, count);
    count_launch();
}

// price = mean - alpha ((1 - p) BS(1, K, 1, sqrt(rho^2 Q)) + p BS(1, K, 1, sqrt(rho^2 Qmax))),
// p = exceptions / M; stat from the unadjusted payoffs (RBergomi.cpp:266-284).
__global__ void k_finalize_cv(const double* __restrict__ acc, int n_out, int64_t M, const OutDev* __restrict__ outs,
                              const double* __restrict__ Tv, const double* __restrict__ alpha,
                              const double* __restrict__ Q, const unsigned long long* __restrict__ count,
                              double Qmax, int compute_iv, double* __restrict__ res,
                              const FixedTables* __restrict__ ft)
{
    const int i = blockIdx.x;
    if (i >= n_out) return;
    const double S = acc[i * 4 + 0] + acc[i * 4 + 1];
    const double S2 = acc[i * 4 + 2] + acc[i * 4 + 3];
    const double mean = S * (1.0 / (double)M);
    const double var = 1.0 * (S2 * (1.0 / (double)M)) + -1.0 * (mean * mean);
    const double stat = sqrt(var) * (1.0 / sqrt((double)M));
    const double p = (double)count[i] / (double)M, r = outs[i].rho, K = outs[i].K;
    const double adj = (1.0 - p) * bs_call_tau1(1.0, K, sqrt(r * r * Q[i])) + p * bs_call_tau1(1.0, K, sqrt(r * r * Qmax));
    const double price = mean - alpha[i] * adj;
    const double iv = compute_iv ? implied_vol_warp(price, K, Tv[i], iv_start(K, Tv[i]), ft) : 0.0;
    if ((threadIdx.x & 31) == 0) {
        res[i] = price;
        res[n_out + i] = stat;
        res[2 * n_out + i] = iv;
        res[3 * n_out + i] = S;
        res[4 * n_out + i] = S2;
    }
}

int launch_finalize_cv(const double* acc, int n_out, int64_t M, const OutDev* outs, const double* Tvals,
                        const double* alpha, const double* Q, const unsigned long long* count, double Qmax,
                        int compute_iv, double* res, void* stream)
{
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    k_finalize_cv<<<n_out, 32, 0, (cudaStream_t)stream>>>(acc, n_out, M, outs, Tvals, alpha, Q, count, Qmax,
                                                          compute_iv, res, ft);
    count_launch();
    return 0;
}

}  // namespace rbg
