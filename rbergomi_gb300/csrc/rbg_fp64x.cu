// rbg_fp64x.cu -- the FP64 form on Philox normals and on the caller's: exact
// convolution on the tensor cores, elementary functions in 64-bit fixed point.
//
// GB300's FP64 pipe (2 DFMA per clock and SM) bounds every kernel that does
// its arithmetic in FP64.  These do it elsewhere, with no less precision:
//   k_normals_fixed  Philox4x32-10 -> Box-Muller in 64-bit integers
//                    (rbg_fixed.cuh) -> normals, quadrature layout, FP64 or
//                    fixed point, and W1 as eight signed 8-bit digits in FP16
//                    for the next
//   k_digits         the digits of the caller's W1
//   k_volterra_exact X_j = sum_{k<=j} W1_k Gamma'_{j-k}, Gamma' = (a1, Gamma_1,
//                    ...), as digit products on tcgen05: both operands are
//                    64-bit fixed-point numbers cut into 8 signed digits, and
//                    the digit products of weight 2^(-8 d), d = i + j <= 7, are
//                    summed in one FP32 accumulator each
//   k_variance_fixed X + a2 W1perp, v = xi 2^t with t and 2^t in 64-bit fixed
//                    point, FP64 sums of v and sqrt(v) W1 (, Wperp); with few
//                    variance groups inside k_volterra_exact instead, k_slot_sums
//                    adding up its parts
//
// Exactness of the convolution.  A digit is an integer in [-128, 127], exact in
// FP16; a product has 14 bits, and an FP32 accumulator holds integers up to
// 2^24 exactly.  The digits of W1 below the first are uniform over [-128, 127] (mean
// -1/2, root mean square 73.9) and independent between steps; the first is round(8 W1), below
// 55 and of root mean square 8.  Gamma's digits are what they are: a diagonal's mean and
// standard deviation follow from the sums of them and of their squares, which
// digit_margin adds up for the plan's own Gamma.  The read-out by 1.5 2^23 is taken up
// to 1024 steps where every partial sum is 9 standard deviations or more from that one's
// limit of 2^22 (2e-19 a sum; x64_wide), else the conversion, and x64_prepare leaves to the FP64
// kernels a plan that comes closer than that to 2^24.  The least over H = 0.01 .. 0.99: 18.4 standard
// deviations from 2^22 at 256 steps, 13.0 at 512, 9.1 at 1024 (H = 0.6), and from 2^24 26 at
// 2048, 18 at 4096.  Left out are the products with d >= 8, below 2^-60 of the
// operands' product each: the sums are within about 2^-54 of the exact ones,
// against 2^-45 for an FP64 FFT of 1024 points and 2^-50 for the direct FP64
// sum of 100 steps.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <set>

#include "rbg_device.cuh"
#include "rbg_fixed.cuh"
#include "rbg_fp64x.hpp"
#include "rbg_tc.cuh"

namespace rbg {

// ------------------------------------------------------------------ tables
// Printed by rbg_tables_gen.cpp when the library is built.
__device__ const FixedTables g_fixed_tables = {
#include "rbg_fixed_tables.inc"
};

// The tables' address on the current device, looked up once; null where that fails.
const FixedTables* fixed_tables()
{
    static std::mutex mu;
    static const FixedTables* at[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(mu);
    if (!at[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_fixed_tables) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        at[dev] = static_cast<const FixedTables*>(p);
    }
    return at[dev];
}

// ----------------------------------------------------------------- normals
// Digits of W1, [group of 64 paths][16-step chunk][digit][64 paths][16 steps]
// FP16: one 16 KB block per chunk, the layout the MMA reads (K-major SW32 rows
// of 32 bytes, row = 64 digit + path, 16-byte halves swapped where row / 4 is
// odd).
constexpr int kXPaths = 64, kXSteps = 16, kXDigits = 8;
constexpr int kXChunkBytes = kXDigits * kXPaths * kXSteps * 2;  // 16 KB

// The signed bytes of four values, digit by digit (most significant first),
// as FP16: each value plus 0x80 in every byte has digit + 128 as its bytes,
// and FP16 0x6400 + byte is 1024 + byte.
__device__ __forceinline__ void store_digits(const int64_t (&v)[4], unsigned char* at)
{
    uint32_t w[2][4];  // high, low words
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint64_t u = (uint64_t)v[q] + 0x8080808080808080ull;
        w[0][q] = hi32(u);
        w[1][q] = lo32(u);
    }
    const __half2 off = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1152
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int b = 3; b >= 0; b -= 2) {  // bytes b and b - 1 of the word: digits 4 h + 3 - b and the next
            const uint32_t sel = (uint32_t)(b | ((4 + b) << 4) | ((b - 1) << 8) | ((3 + b) << 12));
            const uint32_t t01 = __byte_perm(w[h][0], w[h][1], sel), t23 = __byte_perm(w[h][2], w[h][3], sel);
#pragma unroll
            for (int z = 0; z < 2; ++z) {
                const uint32_t s2 = z ? 0x4342u : 0x4140u;
                uint32_t a = __byte_perm(t01, 0x64646464u, s2), c = __byte_perm(t23, 0x64646464u, s2);
                const __half2 ha = __hsub2(*reinterpret_cast<__half2*>(&a), off);
                const __half2 hc = __hsub2(*reinterpret_cast<__half2*>(&c), off);
                const int digit = 4 * h + 3 - b + z;
                *(uint2*)(at + digit * (kXPaths * 32)) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&ha), *reinterpret_cast<const uint32_t*>(&hc));
            }
        }
    }
}

// Z[m][s][j], s < ns: W1, W1perp and (plain MC) Wperp on Philox streams 0, 1,
// 2.  dig non-null (the fixed-point path pass follows): also the digits of W1,
// zero past N and past B.  Streams s with bit s of fix set are stored as 64-bit
// fixed point (unit 2^-59) in place of doubles.
// FORM 0: 64-bit integers; 1: FP32 Box-Muller; 2: doubles with all their bits significant
// however small (box_muller_double; a draw takes 1.8 times as long).
// A warp takes up to kSeg chunks of 16 steps (forms 1 and 2 one where that leaves fewer warps
// than the launch has: 1000 paths of 100 steps in FP32 39 -> 31 us a call) of 8 paths' stream, four lanes a path and four steps a lane, so a path's 16 values and each digit's 8 rows are
// contiguous.  Integer instructions bound it: 330 a warp and pair of normals, 57
// of them 32 x 32 -> 64 multiplies (four cycles each): the FMA-heavy pipe is 78 %
// busy.  2 x 512 steps, 2^17 paths, left in fixed point: 0.84 ms, against 5.40 ms
// for the same draw in FP64 (table-driven logarithm and sine, about 40 FP64
// operations a pair).
constexpr int kNormalThreads = 256, kSeg = 8;
template <int FORM>
__global__ void __launch_bounds__(kNormalThreads, FORM == 2 ? 3 : 4) k_normals_fixed(uint64_t seed, int64_t path0, int64_t B, int N, int ns,
                                                                    double* __restrict__ Z,
                                                                    unsigned char* __restrict__ dig, int fix, int short_seg,
                                                                    const FixedTables* __restrict__ ft)
{
    __shared__ NormalTables T;
    if (FORM != 1) {
        TableCopy<kNormalThreads, (int)sizeof(NormalTables)>(&ft->normals).store(&T);
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, g = lane & 3, pl = lane >> 2;
    const int seg = FORM == 0 ? kSeg : short_seg;
    const int nch = (N + kXSteps - 1) / kXSteps, segs = (nch + seg - 1) / seg;
    const int64_t tasks = (B + kXPaths - 1) / kXPaths * (kXPaths / 8) * ns * segs;
    const bool vec = (N & 1) == 0;
    const PhiloxKeys keys = philox_keys(seed);
    const int64_t warps = (int64_t)gridDim.x * (kNormalThreads / 32);
    for (int64_t t = blockIdx.x * (int64_t)(kNormalThreads / 32) + warp_index(); t < tasks; t += warps) {
        const int64_t r = t / segs;
        const int c0 = (int)(t - r * segs) * seg, c1 = min(nch, c0 + seg);
        const int s = (int)(r % ns);
        const int64_t m = r / ns * 8 + pl;
        const bool valid = m < B, digits = s == 0 && dig != nullptr;
        if (!valid && !digits) continue;
        double* zrow = Z + (m * ns + s) * (int64_t)N;
        const int p = (int)(m & (kXPaths - 1));
        unsigned char* drow = dig + (m / kXPaths) * nch * kXChunkBytes + p * 32 + ((((g >> 1) ^ (p >> 2)) & 1) << 4) +
                              ((g & 1) << 3);
#pragma unroll 1
        for (int c = c0; c < c1; ++c) {
            const int j0 = kXSteps * c + 4 * g;
            int64_t v[4] = {0, 0, 0, 0};
            if (valid && j0 < N) {
                const uint4 x = philox_group(keys, (uint64_t)(path0 + m), (uint32_t)(j0 >> 2), (uint32_t)s);
                double z[4];
                if constexpr (FORM == 2) {
                    box_muller_double(x.x, x.y, T, z[0], z[1]);
                    box_muller_double(x.z, x.w, T, z[2], z[3]);
                } else if constexpr (FORM == 1) {
                    float f0, f1, f2, f3;
                    box_muller_f32(x.x, x.y, f0, f1);
                    box_muller_f32(x.z, x.w, f2, f3);
                    z[0] = f0; z[1] = f1; z[2] = f2; z[3] = f3;
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = double_to_fixed(z[q]);
                } else {
                    box_muller_fixed(x.x, x.y, T, v[0], v[1]);
                    box_muller_fixed(x.z, x.w, T, v[2], v[3]);
                }
                if (FORM != 2 && ((fix >> s) & 1)) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) z[q] = __longlong_as_double(v[q]);
                } else if (FORM == 0) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) z[q] = fixed_to_double(v[q]);
                }
                double* o = zrow + j0;
                if (j0 + 4 <= N) {
                    if (vec) {
                        *(double2*)o = make_double2(z[0], z[1]);
                        *(double2*)(o + 2) = make_double2(z[2], z[3]);
                    } else {
                        o[0] = z[0]; o[1] = z[1]; o[2] = z[2]; o[3] = z[3];
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (j0 + q < N) o[q] = z[q];
                        else v[q] = 0;
                    }
                }
            }
            if (digits) store_digits(v, drow + (size_t)c * kXChunkBytes);
        }
    }
}

int launch_normals_fixed(uint64_t seed, int64_t path0, int64_t B, int N, int f32, double* Z, unsigned char* dig, int fix,
                         int ns, cudaStream_t st, bool exact)
{
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    const int nch = (N + kXSteps - 1) / kXSteps;
    const int64_t rows = (B + kXPaths - 1) / kXPaths * (kXPaths / 8) * ns, most = 8 * (int64_t)device_sms();
    int seg = kSeg;
    auto need = [&] { return (rows * ((nch + seg - 1) / seg) + kNormalThreads / 32 - 1) / (kNormalThreads / 32); };
    auto* kern = f32 ? k_normals_fixed<1> : exact ? k_normals_fixed<2> : k_normals_fixed<0>;
    if ((f32 || exact) && need() < most) seg = 1;
    kern<<<(unsigned)std::min<int64_t>(need(), most), kNormalThreads, 0, st>>>(seed, path0, B, N, ns, Z, dig, fix, seg, ft);
    count_launch();
    return 0;
}

// Digits of the caller's W1 (Z[m][s][j] as k_normals_fixed's), zero past N and
// past B.  W1 and W1perp below kExtMax in size, which finite normals are, fit the
// fixed-point ranges; *flag is set where one is not (or is NaN), and the FP64
// path kernels take the batch.
__global__ void __launch_bounds__(kNormalThreads) k_digits(const double* __restrict__ Z, int64_t B, int N, int ns,
                                                          unsigned char* __restrict__ dig, unsigned int* __restrict__ flag)
{
    const int lane = threadIdx.x & 31, g = lane & 3, pl = lane >> 2;
    const int nch = (N + kXSteps - 1) / kXSteps, segs = (nch + kSeg - 1) / kSeg;
    const int64_t tasks = (B + kXPaths - 1) / kXPaths * (kXPaths / 8) * segs;
    const int64_t warps = (int64_t)gridDim.x * (kNormalThreads / 32);
    bool bad = false;
    for (int64_t t = blockIdx.x * (int64_t)(kNormalThreads / 32) + warp_index(); t < tasks; t += warps) {
        const int64_t r = t / segs, m = r * 8 + pl;
        const int c0 = (int)(t - r * segs) * kSeg, c1 = min(nch, c0 + kSeg);
        const double* z0 = Z + m * ns * (int64_t)N;
        const int p = (int)(m & (kXPaths - 1));
        unsigned char* drow = dig + (m / kXPaths) * nch * kXChunkBytes + p * 32 + ((((g >> 1) ^ (p >> 2)) & 1) << 4) +
                              ((g & 1) << 3);
        for (int c = c0; c < c1; ++c) {
            const int j0 = kXSteps * c + 4 * g;
            double z[4] = {0.0, 0.0, 0.0, 0.0}, w[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (m < B && j0 + q < N) {
                    z[q] = z0[j0 + q];
                    w[q] = z0[N + j0 + q];
                }
            }
            int64_t v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                // a double's size as the integer of its bits; NaN compares above every number
                constexpr uint64_t lim = 0x402F000000000000ull;  // kExtMax
                bad |= (double_bits(z[q]) & ~(1ull << 63)) >= lim || (double_bits(w[q]) & ~(1ull << 63)) >= lim;
                v[q] = double_to_fixed(z[q]);
            }
            store_digits(v, drow + (size_t)c * kXChunkBytes);
        }
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(flag, 1u);
}

void launch_digits(const double* Z, int64_t B, int N, int ns, unsigned char* dig, unsigned int* flag, cudaStream_t st)
{
    const int nch = (N + kXSteps - 1) / kXSteps;
    const int64_t tasks = (B + kXPaths - 1) / kXPaths * (kXPaths / 8) * ((nch + kSeg - 1) / kSeg);
    const int64_t need = (tasks + kNormalThreads / 32 - 1) / (kNormalThreads / 32);
    k_digits<<<(unsigned)std::min<int64_t>(need, 8 * (int64_t)device_sms()), kNormalThreads, 0, st>>>(Z, B, N, ns, dig, flag);
    count_launch();
}

// ------------------------------------------------------------- convolution
// D[step][path] per diagonal d: the Toeplitz operand is MMA's A (128 output
// steps), the W1 digits its B, eight digits x 64 paths = 512 rows of a chunk,
// so one MMA of N = 256 covers four digit products of one Gamma digit and the
// accumulators of a block are [d][64 paths] = all 512 TMEM columns.  Gamma
// digit j multiplies W1 digits 0 .. 7 - j into columns 64 j .. 511.
//
// Gamma panels.  Output block b (steps 128 b ..) takes the 16-step chunks of
// blocks s = 0 .. b; with L = b - s the entries it needs are Gamma'[128 L + i -
// k], i, k < 128: panel L holds, per digit, rows r < 240 of 16 FP16, P[r][k''] =
// Gamma'[128 L + r - 112 - k''] (zero for negative indices), and chunk kk of the
// block reads rows 16 (7 - kk) .. + 127.  60 KB a panel, two in shared memory.
constexpr int kPanelRows = 240;
constexpr int kPanelDigit = kPanelRows * 32;           // 7680 B
constexpr int kPanelBytes = kXDigits * kPanelDigit;    // 61440 B
constexpr int kXBlock = 128;                           // output steps per block
constexpr int kXChunks = kXBlock / kXSteps;            // 8 chunks per block of steps
constexpr int kXStagesPlain = 5, kXStagesFused = 4;
constexpr int kXEpiWarps = 16;
constexpr int kXThreads = (kXEpiWarps + 3) * 32;
// SEG: steps a sum takes where the digits may be anything: 8 digit pairs x 128 x 2^14 = 2^24
constexpr int kAnyChunks = 128 / kXSteps;
constexpr int kXSmemPlain = 2 * kPanelBytes + kXStagesPlain * kXChunkBytes + 256 + 1024;
constexpr int kXSmemFused = 2 * kPanelBytes + kXStagesFused * kXChunkBytes + 256 + kExpTable * 8 + 1024;

int x64_blocks(int N) { return (N + kXBlock - 1) / kXBlock; }
size_t x64_panel_bytes(int N) { return (size_t)x64_blocks(N) * kPanelBytes; }
size_t x64_digit_bytes(int64_t B, int N)
{
    return (size_t)((B + kXPaths - 1) / kXPaths) * ((N + kXSteps - 1) / kXSteps) * kXChunkBytes;
}

// Panels of every pass from its fixed-point Gamma' (unit 2^(e - 62)): one
// thread per 16-byte half row of one digit.
__global__ void k_panels(const int64_t* __restrict__ gam, int nv, int N, int nb, unsigned char* __restrict__ panels)
{
    const int64_t total = (int64_t)nv * nb * kXDigits * kPanelRows * 2;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int half = (int)(t & 1);
        int64_t q = t >> 1;
        const int r = (int)(q % kPanelRows);
        q /= kPanelRows;
        const int digit = (int)(q % kXDigits);
        q /= kXDigits;
        const int L = (int)(q % nb), v = (int)(q / nb);
        uint32_t h[4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int d = kXBlock * L + r - 112 - (8 * half + i);
            const uint64_t u = (uint64_t)((d >= 0 && d < N) ? gam[(size_t)v * N + d] : 0) + 0x8080808080808080ull;
            const int x = (int)((u >> (8 * (7 - digit))) & 255u) - 128;
            const uint32_t f = __half_as_ushort(__int2half_rn(x));
            if (i & 1) h[i >> 1] |= f << 16;
            else h[i >> 1] = f;
        }
        unsigned char* at = panels + ((size_t)v * nb + L) * kPanelBytes + digit * kPanelDigit + r * 32 +
                            ((half ^ (r >> 2)) & 1) * 16;
        *(uint4*)at = make_uint4(h[0], h[1], h[2], h[3]);
    }
}

void launch_panels(const int64_t* gam, int nv, int N, unsigned char* panels, cudaStream_t st)
{
    const int nb = x64_blocks(N);
    const int64_t total = (int64_t)nv * nb * kXDigits * kPanelRows * 2;
    k_panels<<<(unsigned)std::min<int64_t>((total + 255) / 256, 4096), 256, 0, st>>>(gam, nv, N, nb, panels);
    count_launch();
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

// Warp sums of NV integers a lane (a power of two up to 32): each halving step
// hands half of the values to the partner lane.  Value lane / (32 / NV) of every
// lane's sum on return.
template <int NV>
__device__ __forceinline__ int64_t warp_sums_i64(int64_t (&v)[NV])
{
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int n = NV / 2; n >= 1; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const int64_t send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// What a fused variance pass needs beside the convolution's arguments; its sums
// go to part[group of the launch][4 block + warp quadrant][path][NS].
struct FuseArgs {
    const X64Group* grps;
    const uint64_t* comp;
    const uint64_t* Z;
    double* part;
    const FixedTables* ft;
    int slots;
};

// The variance pass of a read-out warp on X of its 16 paths (x, without the
// offset of 2^63), step j of the unit in lane order: per group and path the
// warp's sums of 2^(2 t) and 2^t W over its 32 steps, v = xi 2^(2 t) (k_variance_fixed).
// The sums are taken in integers: with 2^t = m 2^(e - 63), E the largest e of the
// 32 steps and m' = m >> (E - e + 3), 32 terms m'^2 and m' W / 2 fit 64 bits, and
// what truncation takes of the live terms on average goes back (slot_square,
// slot_product, slot_back).  The square's unit is 2^-54 of
// the largest term or less, the product's 2^-54 2^E; an FP64 sum rounds every product
// to 2^-53 of itself and every partial sum likewise.  The same in FP64 (two
// products, the lanes' additions) holds the FP64 pipe: 30011 paths of 250 steps, two
// passes, three sums, 313 us for the path pass against 254.  Instructions and their latencies
// bound it: four warps a scheduler issue one every second cycle.
// Loads past the last step or path are clamped to it, and m is zero there.
// ONE: the pass has one group; without the loop over groups the four quarters
// of the paths overlap (two sums, 100 steps, 2^16 paths 117 -> 111 us; 512 steps, 2^17
// 1.045 -> 1.03 ms; with three sums it is slower, 254 -> 266 us for the case above).
template <int NS, bool ONE>
__device__ __forceinline__ void fused_variance(uint64_t (&x)[2][8], const X64Vol& vol, int grp0, const FuseArgs& fa,
                                               const uint64_t* E, int N, int64_t B, int64_t m0, int j, int slot)
{
    const int lane = threadIdx.x & 31;
    const bool in = j + 1 < N;
    const int jc = min(j, N - 2), left = (int)min(B - m0, (int64_t)16);  // paths of the warp's 16
    const bool whole = left == 16 && __all_sync(0xffffffffu, in);
    if (left <= 0) return;
    // what the live steps lose goes back (28 of 32); counted where it is used, as a register
    // held over the loops costs spills, and with several groups or sums only where the slot is partial
    // (2 groups a pass, 16 steps, 3 passes 2.78 -> 2.73 ms; with one group it is 1.15 times slower)
    auto back = [&] { return !ONE && whole ? 28 : (int)slot_back(__popc(__ballot_sync(0xffffffffu, in))); };
    const uint64_t* z0 = fa.Z + m0 * NS * (int64_t)N + jc;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        uint64_t xs[4], w1[4], wq[NS == 3 ? 4 : 1];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint64_t* W1 = z0 + (size_t)(min(4 * h + p, left - 1) * NS) * N;
            // a signed w as 2^63 + w, and half of it
            w1[p] = (W1[1] ^ (1ull << 63)) >> 1;
            if (NS == 3) wq[p] = (W1[2 * N + 1] ^ (1ull << 63)) >> 1;
            xs[p] = x[h >> 1][(4 * h + p) & 7] + (1ull << 63) + mulhi64(W1[N] ^ (1ull << 63), vol.a2f) - vol.a2h;
        }
#pragma unroll 1
        for (int g = vol.vg_begin; g < (ONE ? vol.vg_begin + 1 : vol.vg_end); ++g) {
            const uint64_t cf = fa.grps[g].cf, flip = fa.grps[g].neg ? ~0ull : 0ull;  // -x less one unit
            const uint64_t cj = __ldg(fa.comp + (size_t)g * N + jc);
            int64_t s[8], sq[4];
            int top[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                int32_t e;
                uint64_t mt = exp2_mantissa53((int64_t)(mulhi64(xs[p] ^ flip, cf) - cj), E, e);
                if (!whole && !(in && 4 * h + p < left)) {
                    mt = 0ull;
                    e = -1000;
                }
                top[p] = __reduce_max_sync(0xffffffffu, e);
                mt >>= min(top[p] - e + 3, 63);
                s[2 * p] = slot_square(mt);
                s[2 * p + 1] = slot_product(mt, w1[p]);
                if (NS == 3) sq[p] = slot_product(mt, wq[p]);
            }
            const int64_t i0 = warp_sums_i64<8>(s) + back();  // value lane / 4 = 2 path + sum
            const int pa = lane >> 3, c = (lane >> 2) & 1;
            const int tp = pa & 2 ? (pa & 1 ? top[3] : top[2]) : (pa & 1 ? top[1] : top[0]);
            const double sc = bits_double((uint64_t)(uint32_t)(tp + 1023) << 52);
            double* out = fa.part + (((size_t)(g - grp0) * fa.slots + slot) * B + m0 + 4 * h + pa) * NS;
            const double r = (c ? (double)i0 * 0x1p-54 : (double)i0 * 0x1p-56 * sc) * sc;
            if (!(lane & 3) && 4 * h + pa < left) out[c] = r;
            if constexpr (NS == 3) {
                const int64_t i2 = warp_sums_i64<4>(sq) + back();
                if (!(lane & 7) && 4 * h + pa < left) out[2] = (double)i2 * 0x1p-54 * sc;
            }
        }
    }
}

// Which of the two panel buffers a panel goes to: the one that holds it, else
// the one not used last.  The loader and the MMA thread follow the same rule.
struct PanelSlots {
    int key0 = -1, key1 = -1, last = 1;
    __device__ __forceinline__ int use(int key, bool& load)
    {
        int b;
        load = false;
        if (key == key0) {
            b = 0;
        } else if (key == key1) {
            b = 1;
        } else {
            b = 1 - last;
            load = true;
            if (b) key1 = key;
            else key0 = key;
        }
        last = b;
        return b;
    }
};

// One (block b, pass v, group of 64 paths) at a time, the longest blocks
// first.  Warps 0-15 read the accumulators, warp 16 loads, warps 17 and 18 issue
// the MMAs.  WIDE: accumulators may pass 2^22 (above 1024 steps, and where
// x64_wide finds it of Gamma's digits, which it does not for H below 1): converted by F2I, else by adding 1.5 2^23.  SEG: the caller's normals, whose digits may add up: the
// accumulators are read out every 128 steps and X summed in integers, which is
// exact for any digits.
// What bounds it: 2304 columns x 128 steps x 16 per chunk, 1152 MMA cycles,
// against 16 KB of digits and 7.5 KB of panel from L2; the accumulators fill
// TMEM, so the next block's MMAs wait for the read-out of this one's.
// FUSE > 0 (sums per path: 2 or 3; 1: two, one group a pass): the read-out warps
// also do the variance pass on their X, in registers, while the next unit's MMAs
// run, and write the sums of their 32 steps per path and group instead of X:
// 512 steps, 2^17 paths, one group 1.03 ms
// with k_slot_sums, against 0.88 + 0.38 ms with X through memory and
// k_variance_fixed, and 13.2 ms for the FP64 FFT convolution and exponentials; 100
// steps, 2^16 paths 0.111 ms, against 0.133 and, for the direct FP64 sum, 1.46 ms.
template <bool WIDE, bool SEG, int FUSE>
__global__ void __launch_bounds__(kXThreads, 1) k_volterra_exact(const unsigned char* __restrict__ dig,
                                                                 const unsigned char* __restrict__ panels,
                                                                 const X64Vol* __restrict__ vols, int nv, int N,
                                                                 int64_t B, uint64_t* __restrict__ X,
                                                                 unsigned int* __restrict__ err, const FuseArgs fa)
{
    constexpr int kXStages = FUSE ? kXStagesFused : kXStagesPlain;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    unsigned char* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    unsigned char* stage = base + 2 * kPanelBytes;
    uint64_t* bars = (uint64_t*)(stage + kXStages * kXChunkBytes);
    uint64_t* E = bars + 32;  // FUSE: the exponential's table
    uint64_t* wfull = bars;                 // [kXStages]
    uint64_t* wempty = bars + kXStages;     // [kXStages]
    uint64_t* pfull = bars + 2 * kXStages;  // [2]
    uint64_t* accf = pfull + 2;
    uint64_t* acce = accf + 1;
    uint64_t* fin = accf + 2;
    uint32_t* holder = (uint32_t*)(accf + 3);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int nb = (N + kXBlock - 1) / kXBlock, nch = (N + kXSteps - 1) / kXSteps;
    const int64_t groups = (B + kXPaths - 1) / kXPaths, per = groups * nv, units = per * nb;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kXStages; ++s) {
            mbar_init(smem_u32(wfull + s), 1);
            mbar_init(smem_u32(wempty + s), 2);
        }
        for (int b = 0; b < 2; ++b) mbar_init(smem_u32(pfull + b), 1);
        mbar_init(smem_u32(accf), 2);
        mbar_init(smem_u32(fin), 2);
        mbar_init(smem_u32(acce), kXEpiWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (FUSE)
        TableCopy<kXThreads, kExpTable * 8>(fa.ft->exp2).store(E);
    if (warp == kXEpiWarps + 1) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *holder;

    if (warp == kXEpiWarps) {
        if (lane == 0) {
            // ------------------------------------------------------ loader
            PanelSlots ps;
            int64_t used[2] = {-1, -1};  // the last chunk (of this thread's count n) that reads each panel buffer
            int loads[2] = {0, 0};
            int s = 0;
            uint32_t ph = 0;
            int64_t n = 0;
            bool ok = true;
            for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
                const int b = nb - 1 - (int)(u / per), v = (int)(u % per / groups);
                const int64_t g = u % groups;
                const int ke = min(kXChunks * (b + 1), nch);
                int pb = 0;
                for (int kc = 0; kc < ke && ok; ++kc, s = (s + 1 == kXStages) ? 0 : s + 1, ph ^= (s == 0)) {
                    if (kc % kXChunks == 0) {
                        const int L = b - kc / kXChunks;
                        bool load;
                        pb = ps.use(v * nb + L, load);
                        if (load) {
                            // every MMA on the buffer's old panel has completed once its last chunk's stage
                            // is free; chunks before n - kXStages were waited for when their stage was refilled
                            const int64_t i = used[pb];
                            if (i >= 0 && i >= n - kXStages &&
                                !mbar_wait(smem_u32(wempty + (int)(i % kXStages)), (uint32_t)((i / kXStages) & 1), err, 21)) {
                                ok = false;
                                break;
                            }
                            const uint32_t bar = smem_u32(pfull + pb);
                            mbar_expect_tx(bar, kPanelBytes);
                            bulk_g2s(smem_u32(base) + pb * kPanelBytes, panels + ((size_t)v * nb + L) * kPanelBytes,
                                     kPanelBytes, bar);
                            ++loads[pb];
                        }
                    }
                    used[pb] = n;
                    if (!mbar_wait(smem_u32(wempty + s), ph ^ 1u, err, 22)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(wfull + s);
                    mbar_expect_tx(bar, kXChunkBytes);
                    bulk_g2s(smem_u32(stage) + s * kXChunkBytes, dig + ((size_t)g * nch + kc) * kXChunkBytes, kXChunkBytes,
                             bar);
                    ++n;
                }
            }
            // the copies in flight land before the CTA exits, whatever the error word says
            for (int64_t i = n > kXStages ? n - kXStages : 0; i < n; ++i)
                mbar_drain(smem_u32(wfull + (int)(i % kXStages)), (uint32_t)((i / kXStages) & 1));
            for (int b = 0; b < 2; ++b)
                if (loads[b]) mbar_drain(smem_u32(pfull + b), (uint32_t)((loads[b] - 1) & 1));
        }
    } else if (warp > kXEpiWarps) {
        if (lane == 0) {
            // ------------------------------------------------- MMA issuers
            // Thread 0 accumulates the diagonals 0 .. 3 (four MMAs a chunk), thread 1 the
            // diagonals 4 .. 7 (eight): one thread issuing all twelve held the tensor pipe.
            const int me = warp - kXEpiWarps - 1;
            PanelSlots ps;
            int loads[2] = {0, 0};
            int s = 0;
            uint32_t ph = 0;
            int64_t drains = 0;  // accumulator read-outs asked for
            bool ok = true;
            const uint64_t a_base = sdesc_sw32(smem_u32(base)), b_base = sdesc_sw32(smem_u32(stage));
            const uint32_t a_lo = (uint32_t)a_base, a_hi = (uint32_t)(a_base >> 32);
            const uint32_t b_lo = (uint32_t)b_base, b_hi = (uint32_t)(b_base >> 32);
            for (int64_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
                const int b = nb - 1 - (int)(u / per), v = (int)(u % per / groups);
                const int ke = min(kXChunks * (b + 1), nch);
                int pb = 0, sc = 0;  // SEG: chunks of the current sum so far
                // (kept out of the chunk loop where a unit is one sum: inside it they cost the convolution 10 %)
                if (!SEG && drains > 0 && !mbar_wait(smem_u32(acce), (uint32_t)((drains - 1) & 1), err, 23)) break;
                for (int kc = 0; kc < ke; ++kc, s = (s + 1 == kXStages) ? 0 : s + 1, ph ^= (s == 0)) {
                    if (SEG && sc == 0 && drains > 0 && !mbar_wait(smem_u32(acce), (uint32_t)((drains - 1) & 1), err, 23)) {
                        ok = false;
                        break;
                    }
                    if (kc % kXChunks == 0) {
                        bool load;
                        pb = ps.use(v * nb + b - kc / kXChunks, load);
                        if (load) {
                            if (!mbar_wait(smem_u32(pfull + pb), (uint32_t)(loads[pb] & 1), err, 24)) { ok = false; break; }
                            ++loads[pb];
                        }
                    }
                    if (!mbar_wait(smem_u32(wfull + s), ph, err, 25)) { ok = false; break; }
                    tc_fence_after();
                    // descriptors differ in the start-address field only (address / 16, no carry out of it)
                    const uint32_t arow = a_lo + (uint32_t)(pb * kPanelBytes + (kXChunks - 1 - kc % kXChunks) * 512) / 16;
                    const uint32_t brow = b_lo + (uint32_t)(s * kXChunkBytes) / 16;
                    const uint32_t first = (SEG ? sc : kc) == 0 ? 0u : 1u;
                    if (me == 0) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)  // W1 digits 0 .. 3 - j into diagonals j .. 3
                            umma_f16(tmem + kXPaths * j, ((uint64_t)a_hi << 32) | (arow + (uint32_t)(j * kPanelDigit) / 16),
                                     ((uint64_t)b_hi << 32) | brow, idesc_f16(kXPaths * (4 - j), 0), j ? 1u : first);
                    } else {
#pragma unroll
                        for (int j = 0; j < kXDigits; ++j) {  // W1 digits max(0, 4 - j) .. 7 - j into diagonals max(4, j) .. 7
                            const int i0 = j < 4 ? 4 - j : 0, n = j < 4 ? 4 : kXDigits - j;
                            umma_f16(tmem + kXPaths * (i0 + j),
                                     ((uint64_t)a_hi << 32) | (arow + (uint32_t)(j * kPanelDigit) / 16),
                                     ((uint64_t)b_hi << 32) | (brow + (uint32_t)(i0 * kXPaths * 32) / 16),
                                     idesc_f16(kXPaths * n, 0), j ? 1u : first);
                        }
                    }
                    umma_commit(smem_u32(wempty + s));
                    if (SEG && (++sc == kAnyChunks || kc == ke - 1)) {
                        umma_commit(smem_u32(accf));
                        ++drains;
                        sc = 0;
                    }
                }
                if (!SEG) {
                    if (ok) umma_commit(smem_u32(accf));
                    ++drains;
                }
            }
            // every issued MMA completes before TMEM is released
            umma_commit(smem_u32(fin));
            mbar_wait(smem_u32(fin), 0, err, 26);
        }
    } else {
        // -------------------------------------------------------- read-out
        const int quad = warp & 3, wg = warp >> 2;
        const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16);
        int64_t drains = 0;
        for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
            const int b = nb - 1 - (int)(u / per), v = (int)(u % per / groups);
            const int64_t g = u % groups;
            const int sh = vols[v].sh, ke = min(kXChunks * (b + 1), nch);
            const int j = kXBlock * b + quad * 32 + lane;
          for (int k0 = 0; k0 < (SEG ? ke : 1); k0 += kAnyChunks, ++drains) {
            if (!mbar_wait_warp(smem_u32(accf), (uint32_t)(drains & 1), err, 27)) goto done;
            tc_fence_after();
            const bool add = SEG && k0 > 0;  // a further segment of the same sums
            // X of 8 paths (from column p0), the unit's step j
            auto read8 = [&](int p0, uint64_t (&xv)[8], bool last) {
                uint32_t D[kXDigits][8];
#pragma unroll
                for (int d = 0; d < kXDigits; ++d) tmem_ld8(tl + (uint32_t)(kXPaths * d + p0), D[d]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (last) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(acce));
                }
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    // S_hi in units of 2^(e - 33), S_lo of 2^(e - 65); X = S_hi 2^sh + S_lo 2^(sh - 32)
                    int64_t hi, lo;
                    if (WIDE) {
                        int64_t D8[kXDigits];
#pragma unroll
                        for (int d = 0; d < kXDigits; ++d) D8[d] = __float2int_rn(__uint_as_float(D[d][p]));
                        hi = (D8[0] << 24) + (D8[1] << 16) + (D8[2] << 8) + D8[3];
                        lo = (D8[4] << 24) + (D8[5] << 16) + (D8[6] << 8) + D8[7];
                    } else {
                        // |D| < 2^22: f + 1.5 2^23 has D + 0x4B400000 as its bits, and two neighbours
                        // make one 32-bit number; the offsets come off modulo 2^32
                        uint32_t I[kXDigits];
#pragma unroll
                        for (int d = 0; d < kXDigits; ++d) I[d] = __float_as_uint(__uint_as_float(D[d][p]) + 12582912.f);
                        constexpr uint32_t off = 0x4B400000u * 257u;
                        const int32_t h1 = (int32_t)(I[0] * 256u + I[1] - off), h0 = (int32_t)(I[2] * 256u + I[3] - off);
                        const int32_t l1 = (int32_t)(I[4] * 256u + I[5] - off), l0 = (int32_t)(I[6] * 256u + I[7] - off);
                        hi = (int64_t)h1 * 65536 + h0;
                        lo = (int64_t)l1 * 65536 + l0;
                    }
                    xv[p] = shl((uint64_t)hi, sh) + (uint64_t)(lo >> (32 - sh));
                }
            };
            if constexpr (FUSE == 0) {
#pragma unroll 1
                for (int q = 0; q < kXPaths / 8 / (kXEpiWarps / 4); ++q) {
                    const int p0 = wg * (kXPaths * 4 / kXEpiWarps) + q * 8;
                    uint64_t xv[8];
                    read8(p0, xv, q == kXPaths / 8 / (kXEpiWarps / 4) - 1);
                    const int64_t m = g * kXPaths + p0;
                    uint64_t* Xm = X + ((size_t)v * B + m) * N + j;
#pragma unroll
                    for (int p = 0; p < 8; ++p) {
                        if (m + p < B && j < N) {
                            uint64_t* at = Xm + (size_t)p * N;
                            *at = xv[p] + (add ? *at : 1ull << 63);
                        }
                    }
                }
            } else {
                static_assert(kXPaths * 4 / kXEpiWarps == 16, "two read-outs of 8 paths a warp");
                const int p0 = wg * 16;
                uint64_t xs[2][8];
                read8(p0, xs[0], false);
                read8(p0 + 8, xs[1], true);
                fused_variance<FUSE == 1 ? 2 : FUSE, FUSE == 1>(xs, vols[v], vols[0].vg_begin, fa, E, N, B, g * kXPaths + p0, j, 4 * b + quad);
            }
          }
        }
    }
done:
    tc_fence_before();
    __syncthreads();
    if (warp == kXEpiWarps + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// (Ivdt, IsvdW (, IsvdWp)) per path and group from the fused pass's sums over
// its slots of 32 steps; groups grp0 .. grp0 + ng - 1.
template <int NS>
__global__ void __launch_bounds__(256) k_slot_sums(const X64Group* __restrict__ grps, const double* __restrict__ part,
                                                  const int64_t* __restrict__ Z, int grp0, int ng, int slots, int N,
                                                  int64_t B, double* __restrict__ ivb, double* __restrict__ ivp)
{
    for (int64_t t = blockIdx.x * (int64_t)256 + threadIdx.x; t < B * ng; t += (int64_t)gridDim.x * 256) {
        const int g = (int)(t / B);
        const int64_t m = t - (int64_t)g * B;
        const double* p = part + ((size_t)g * slots * B + m) * NS;
        double s[NS];
#pragma unroll
        for (int c = 0; c < NS; ++c) s[c] = 0.0;
        for (int k = 0; k < slots; ++k, p += (size_t)B * NS) {
#pragma unroll
            for (int c = 0; c < NS; ++c) s[c] += p[c];
        }
        const X64Group& G = grps[grp0 + g];
        const size_t at = (size_t)(grp0 + g) * B + m;
        const int64_t* W1 = Z + m * NS * (int64_t)N;
        // Ivdt = dt xi (1 + sum), IsvdW = sqrt(dt xi) (W1_0 + sum): v_0 = xi
        ivb[2 * at] = G.dtxi * (1.0 + s[0]);
        ivb[2 * at + 1] = G.sdtxi * (fixed_to_double(W1[0]) + s[1]);
        if (NS == 3) ivp[at] = G.sdtxi * (fixed_to_double(W1[2 * N]) + s[NS - 1]);
    }
}

size_t x64_slot_bytes(int64_t B, int N, int ns) { return (size_t)4 * x64_blocks(N) * (size_t)B * ns * sizeof(double); }

// Raises a kernel's shared-memory limit, once per (device, kernel).
static bool allow_smem(const void* kern, int bytes)
{
    static std::mutex mu;
    static std::set<std::pair<int, const void*>> done;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> lk(mu);
    if (done.count({dev, kern})) return true;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    done.insert({dev, kern});
    return true;
}

static int volterra_grid(int64_t B, int N, int nv)
{
    const int64_t units = (B + kXPaths - 1) / kXPaths * nv * x64_blocks(N);
    return (int)std::min<int64_t>(units, device_sms());
}

int launch_volterra_variance(const unsigned char* dig, const unsigned char* panels, const X64Vol* vols,
                             const X64Group* grps, const uint64_t* comp, const double* Z, int nv, int grp0, int ng, int ns,
                             bool wide, int N, int64_t B, double* part, double* ivb, double* ivp, unsigned int* err,
                             cudaStream_t st)
{
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    const bool one = ng == nv;  // every pass has at least one group
    auto* kern = ns == 3 ? (wide ? k_volterra_exact<true, false, 3> : k_volterra_exact<false, false, 3>)
                 : one   ? (wide ? k_volterra_exact<true, false, 1> : k_volterra_exact<false, false, 1>)
                         : (wide ? k_volterra_exact<true, false, 2> : k_volterra_exact<false, false, 2>);
    if (!allow_smem((const void*)kern, kXSmemFused)) return -1;
    const int slots = 4 * x64_blocks(N);
    kern<<<volterra_grid(B, N, nv), kXThreads, kXSmemFused, st>>>(
        dig, panels, vols, nv, N, B, nullptr, err, FuseArgs{grps, comp, (const uint64_t*)Z, part, ft, slots});
    const unsigned blocks = (unsigned)std::min<int64_t>((B * ng + 255) / 256, 8 * (int64_t)device_sms());
    auto* sums = ns == 3 ? k_slot_sums<3> : k_slot_sums<2>;
    sums<<<blocks, 256, 0, st>>>(grps, part, (const int64_t*)Z, grp0, ng, slots, N, B, ivb, ivp);
    count_launch(2);
    return 0;
}

int launch_volterra_exact(const unsigned char* dig, const unsigned char* panels, const X64Vol* vols, int nv, int N,
                          int64_t B, bool any, bool wide, uint64_t* X, unsigned int* err, cudaStream_t st)
{
    // any digits: sums of at most 128 steps, whose diagonals stay within 2^24 whatever the digits are
    auto* kern = any ? k_volterra_exact<true, true, 0>
                     : (wide ? k_volterra_exact<true, false, 0> : k_volterra_exact<false, false, 0>);
    if (!allow_smem((const void*)kern, kXSmemPlain)) return -1;
    kern<<<volterra_grid(B, N, nv), kXThreads, kXSmemPlain, st>>>(dig, panels, vols, nv, N, B, X, err, FuseArgs{});
    count_launch();
    return 0;
}

// ----------------------------------------------------------- variance path
// One warp per path, lanes over steps; GB variance groups of one pass at a
// time.  sqrt(v_j) = sqrt(xi) 2^t, t = C (X + a2 W1perp)_{j-1} - comp_{j-1} in
// units of 2^-ut, 2^t by table and polynomial in integers; FP64 only for the
// two (three) sums, which leaves the FP64 pipe 128 (192) cycles a warp step and
// the integer pipes about as much.  The lanes' sums of several paths are
// reduced together through shared memory: one FP64 addition a value and lane
// instead of five.
constexpr int kVarVals = 16, kVarGroups = 4;  // variance groups a batch of a pass with several
__host__ __device__ constexpr int var_threads(int gb) { return gb > 1 ? 256 : 512; }
__host__ __device__ constexpr int var_smem(int gb) { return kExpTable * 8 + (var_threads(gb) / 32) * kVarVals * 33 * 8; }

template <int NS, int GB, bool U53, bool EXT>
__global__ void __launch_bounds__(var_threads(GB), 2) k_variance_fixed(const X64Vol* __restrict__ vols,
                                                               const X64Group* __restrict__ grps,
                                                               const uint64_t* __restrict__ comp,
                                                               const double* __restrict__ Z,
                                                               const uint64_t* __restrict__ X, int nv, int N, int64_t B,
                                                               double* __restrict__ ivb, double* __restrict__ ivp,
                                                               const FixedTables* __restrict__ ft)
{
    constexpr int PB = kVarVals / (GB * NS);  // paths per reduction
    constexpr int kVarThreads = var_threads(GB);
    extern __shared__ uint64_t vsm[];
    uint64_t* E = vsm;
    const int lane = threadIdx.x & 31, w = warp_index();
    double* red = reinterpret_cast<double*>(vsm + kExpTable) + (size_t)w * kVarVals * 33;
    for (int i = threadIdx.x; i < kExpTable; i += kVarThreads) E[i] = ft->exp2[i];
    __syncthreads();
    const int64_t runs = (B + PB - 1) / PB, warps = (int64_t)gridDim.x * (kVarThreads / 32);
    for (int64_t run = blockIdx.x * (int64_t)(kVarThreads / 32) + w; run < runs; run += warps) {
        for (int v = 0; v < nv; ++v) {
            const X64Vol vol = vols[v];
            for (int g0 = vol.vg_begin; g0 < vol.vg_end; g0 += GB) {
                const int ng = min(GB, vol.vg_end - g0);
                uint64_t cf[GB];
                int ut[GB];
                bool neg[GB];
#pragma unroll
                for (int q = 0; q < GB; ++q) {
                    const X64Group& G = grps[g0 + (q < ng ? q : 0)];
                    cf[q] = G.cf;
                    ut[q] = G.ut;
                    neg[q] = G.neg != 0;
                }
#pragma unroll 1
                for (int pl = 0; pl < PB; ++pl) {
                    const int64_t m = run * PB + pl;
                    double acc[GB][NS];
#pragma unroll
                    for (int q = 0; q < GB; ++q)
#pragma unroll
                        for (int c = 0; c < NS; ++c) acc[q][c] = 0.0;
                    if (m < B) {
                        const double* W1 = Z + m * NS * (int64_t)N;
                        const uint64_t* Wp = reinterpret_cast<const uint64_t*>(W1 + N);  // fixed point, EXT: doubles
                        const uint64_t* Xm = X + ((size_t)v * B + m) * N;
                        // operands are loaded two steps ahead: a step's 24 bytes a lane, 24 warps an SM,
                        // have to cover the latency of device memory
                        struct Step {
                            double w1, wq;
                            uint64_t wp, x;
                        } s[3];
                        auto load = [&](int j) {
                            Step r{0.0, 0.0, 0ull, 0ull};
                            if (j < N) {
                                r.w1 = W1[j];
                                if (NS == 3) r.wq = W1[2 * N + j];
                                r.wp = Wp[j - 1];
                                r.x = Xm[j - 1];
                            }
                            return r;
                        };
                        const uint64_t* cg = comp + (size_t)g0 * N - 1;
                        uint64_t cn[GB];
#pragma unroll
                        for (int q = 0; q < GB; ++q) cn[q] = (q < ng && 1 + lane < N) ? __ldg(cg + (size_t)q * N + 1 + lane) : 0ull;
                        s[0] = load(1 + lane);
                        s[1] = load(33 + lane);
                        for (int j = 1 + lane; j < N; j += 32) {
                            s[2] = load(j + 64);
                            uint64_t cc[GB];
#pragma unroll
                            for (int q = 0; q < GB; ++q) {
                                cc[q] = cn[q];
                                cn[q] = (q < ng && j + 32 < N) ? __ldg(cg + (size_t)q * N + j + 32) : 0ull;
                            }
                            const uint64_t wp = EXT ? (uint64_t)double_to_fixed(bits_double(s[0].wp)) : s[0].wp;
                            const uint64_t x = s[0].x + mulhi64(wp ^ (1ull << 63), vol.a2f) - vol.a2h;
#pragma unroll
                            for (int q = 0; q < GB; ++q) {
                                if (q < ng) {
                                    const uint64_t t = mulhi64(neg[q] ? 0ull - x : x, cf[q]) - cc[q];
                                    const double su = U53 ? exp2_fixed53((int64_t)t, E) : exp2_fixed((int64_t)t, ut[q], E);
                                    acc[q][0] = fma(su, su, acc[q][0]);
                                    acc[q][1] = fma(su, s[0].w1, acc[q][1]);
                                    if (NS == 3) acc[q][2] = fma(su, s[0].wq, acc[q][2]);
                                }
                            }
                            s[0] = s[1];
                            s[1] = s[2];
                        }
                    }
#pragma unroll
                    for (int q = 0; q < GB; ++q)
#pragma unroll
                        for (int c = 0; c < NS; ++c) red[((pl * GB + q) * NS + c) * 33 + lane] = acc[q][c];
                }
                __syncwarp();
                // value lane % 16 over the 16 lanes of half lane / 16, then both halves
                const int val = lane & 15;
                double s = 0.0;
                if (val < PB * GB * NS) {
                    const double* row = red + val * 33 + (lane >> 4) * 16;
#pragma unroll
                    for (int i = 0; i < 16; ++i) s += row[i];
                }
                s += __shfl_xor_sync(0xffffffffu, s, 16);
                const int c = val % NS, q = val / NS % GB;
                const int64_t m = run * PB + val / (NS * GB);
                if (lane < 16 && val < PB * GB * NS && q < ng && m < B) {
                    const X64Group& G = grps[g0 + q];
                    const size_t at = (size_t)(g0 + q) * B + m;
                    const double* W1 = Z + m * NS * (int64_t)N;
                    // Ivdt = dt xi (1 + sum), IsvdW = sqrt(dt xi) (W1_0 + sum): v_0 = xi
                    if (c == 0) ivb[2 * at] = G.dtxi * (1.0 + s);
                    else if (c == 1) ivb[2 * at + 1] = G.sdtxi * (W1[0] + s);
                    else ivp[at] = G.sdtxi * (W1[2 * N] + s);
                }
                __syncwarp();
            }
        }
    }
}

template <bool EXT>
static auto* variance_kernel(int ns, bool many, bool u53)
{
    if (ns == 3)
        return many ? (u53 ? k_variance_fixed<3, kVarGroups, true, EXT> : k_variance_fixed<3, kVarGroups, false, EXT>)
                    : (u53 ? k_variance_fixed<3, 1, true, EXT> : k_variance_fixed<3, 1, false, EXT>);
    return many ? (u53 ? k_variance_fixed<2, kVarGroups, true, EXT> : k_variance_fixed<2, kVarGroups, false, EXT>)
                : (u53 ? k_variance_fixed<2, 1, true, EXT> : k_variance_fixed<2, 1, false, EXT>);
}

int launch_variance_fixed(const X64Vol* vols, const X64Group* grps, const uint64_t* comp, const double* Z,
                          const uint64_t* X, int nv, int max_groups, bool u53, bool ext, int ns, int N, int64_t B,
                          double* ivb, double* ivp, cudaStream_t st)
{
    const FixedTables* ft = fixed_tables();
    if (!ft) return -1;
    auto* kern = ext ? variance_kernel<true>(ns, max_groups > 1, u53) : variance_kernel<false>(ns, max_groups > 1, u53);
    if (!allow_smem((const void*)kern, var_smem(max_groups > 1 ? kVarGroups : 1))) return -1;
    const int gb = max_groups > 1 ? kVarGroups : 1, pb = kVarVals / (gb * ns), threads = var_threads(gb);
    const int64_t runs = (B + pb - 1) / pb;
    const int64_t blocks =
        std::min<int64_t>((runs + threads / 32 - 1) / (threads / 32), 2 * (int64_t)device_sms());
    kern<<<(unsigned)blocks, threads, var_smem(gb), st>>>(vols, grps, comp, Z, X, nv, N, B, ivb, ivp, ft);
    count_launch();
    return 0;
}

// -------------------------------------------------------------------- host
double digit_margin(const int64_t* gam, int N, double limit)
{
    // sums of every digit and of its square; the largest partial sum is found every 16 steps
    double most[8] = {}, square[8] = {}, total[8] = {};
    for (int k0 = 0; k0 < N; k0 += 16) {
        int s[8] = {}, q[8] = {};
        for (int k = k0; k < std::min(N, k0 + 16); ++k) {
            const uint64_t u = (uint64_t)gam[k] + 0x8080808080808080ull;
            unsigned char byte[8];
            std::memcpy(byte, &u, 8);
            for (int b = 0; b < 8; ++b) {
                const int x = byte[b] - 128;
                s[b] += x;
                q[b] += x * x;
            }
        }
        for (int b = 0; b < 8; ++b) {
            total[b] += s[b];
            square[b] += q[b];
            most[b] = std::max(most[b], std::fabs(total[b]));
        }
    }
    // the digits of W1: root mean square squared, size of the mean (FP32 normals: the
    // last bits of the fourth are zero, mean -4.5)
    const double sq[8] = {64.0, 5461.5, 5461.5, 5461.5, 5461.5, 5461.5, 5461.5, 5461.5};
    const double mean[8] = {0.0, 0.5, 0.5, 5.0, 0.5, 0.5, 0.5, 0.5};
    double margin = HUGE_VAL;
    for (int d = 0; d < kXDigits; ++d) {
        double v = 0.0, m = 0.0;
        for (int j = 0; j <= d; ++j) {
            v += square[7 - j] * sq[d - j];
            m += (most[7 - j] + 16.0 * 128.0) * mean[d - j];
        }
        if (v > 0.0) margin = std::min(margin, (limit - m) / std::sqrt(v));
    }
    return margin;
}

bool x64_wide(const X64Tables& t, int N)
{
    if (N > 1024) return true;
    if (N <= 256) return false;  // the margin is 9 whatever Gamma's digits are
    for (size_t v = 0; v < t.vols.size(); ++v)
        if (digit_margin(t.gam.data() + v * N, N, 0x1p22) < kXMargin) return true;
    return false;
}

bool x64_prepare(const Plan& plan, X64Tables& out, bool ext)
{
    const int N = plan.N, nv = (int)plan.vols.size(), ng = (int)plan.vgs.size();
    if (N < 2 || N > kX64MaxN) return false;
    out.vols.assign(nv, X64Vol{});
    out.grps.assign(ng, X64Group{});
    out.gam.assign((size_t)nv * N, 0);
    out.comp.assign((size_t)ng * N, 0);
    std::vector<int> ux(nv);
    std::vector<double> xbound(nv);  // |X + a2 W1perp| at most
    // |Box-Muller on 32-bit uniforms| <= sqrt(66 ln 2) = 6.77; the caller's normals below kExtMax
    const double wmax = ext ? kExtMax : 6.9;
    for (int v = 0; v < nv; ++v) {
        const VolGroup& V = plan.vols[v];
        const double* G = plan.gamma.data() + (size_t)v * N;
        double gmax = std::fabs(V.a1), gsum = std::fabs(V.a1);
        for (int d = 1; d < N; ++d) {
            gmax = std::max(gmax, std::fabs(G[d]));
            gsum += std::fabs(G[d]);
        }
        const double bound = wmax * (gsum + std::fabs(V.a2));
        if (!(gmax > 0.0) || !std::isfinite(bound) || !(V.a2 >= 0.0)) return false;
        xbound[v] = bound;
        int e = 0, cb = 0;
        while (std::ldexp(1.0, e) < gmax) ++e;
        while (std::ldexp(1.0, cb) < bound) ++cb;
        // X in units of 2^-ux with |X| 2^ux < 2^62; a2 2^(ux - 59) < 1 for its fixed-point factor
        int u = 62 - cb;
        while (std::ldexp(V.a2, u - kNormalBits) >= 1.0) --u;
        const int sh = e - 33 + u;
        if (sh < 1 || sh > 31) return false;
        ux[v] = u;
        out.vols[v].sh = sh;
        out.vols[v].vg_begin = V.vg_begin;
        out.vols[v].vg_end = V.vg_end;
        const uint64_t a2f = (uint64_t)std::ldexp(V.a2, u - kNormalBits + 64);
        out.vols[v].a2f = a2f;
        out.vols[v].a2h = (a2f >> 1) - 1;  // the bias's share, and the product's mean truncation
        // unit 2^(e - 62): |gam| <= 2^62
        int64_t* q = out.gam.data() + (size_t)v * N;
        const double unit = std::ldexp(1.0, 62 - e);
        q[0] = (int64_t)(V.a1 * unit);  // whole units from 2^(e - 10) up, truncated below
        for (int d = 1; d < N; ++d) q[d] = (int64_t)(G[d] * unit);
        out.max_groups = std::max(out.max_groups, V.vg_end - V.vg_begin);
        // (up to 2048 steps the margin is larger whatever Gamma's digits are; the caller's normals are summed
        // in parts that no digits can take past 2^24)
        if (!ext && N > 2048 && digit_margin(q, N, 0x1p24) < kXMargin) return false;
    }
    const double l2 = 1.4426950408889634074, l2lo = 2.0355273740931033e-17;  // log2 e
    for (int g = 0; g < ng; ++g) {
        const VGroup& G = plan.vgs[g];
        const double* c = plan.comp.data() + (size_t)g * N;
        const double C = 0.5 * G.eta * G.scale * l2, Ca = std::fabs(C);
        double cmax = 0.0;
        bool finite = true;
        for (int j = 0; j + 1 < N; ++j) {
            finite = finite && std::fabs(c[j]) <= 1e300;
            cmax = std::max(cmax, std::fabs(c[j]));
        }
        // t in units of 2^-ut: |t| < 2^(62 - ut), C 2^(ut - ux) < 1 for its factor
        const double bound = Ca * xbound[G.vol] + 0.5 * l2 * cmax + 1.0;
        if (!finite || !std::isfinite(bound)) return false;
        int ut = 53;
        while (ut > 0 && (std::ldexp(bound, ut) >= std::ldexp(1.0, 62) || std::ldexp(Ca, ut - ux[G.vol]) >= 1.0)) --ut;
        if (ut < kX64MinUt) return false;
        X64Group& o = out.grps[g];
        o.ut = ut;
        out.u53 = out.u53 && ut == 53;
        o.neg = C < 0.0;
        o.cf = (uint64_t)std::ldexp(Ca, ut - ux[G.vol] + 64);
        o.dtxi = G.dt * G.xi;
        o.sdtxi = G.sdt * std::sqrt(G.xi);
        uint64_t* q = out.comp.data() + (size_t)g * N;
        const double unit = std::ldexp(1.0, ut);
        const uint64_t bias = (o.cf >> 1) - 1;
        for (int j = 0; j + 1 < N; ++j) {
            // comp / 2 log2 e in two parts, so the fixed-point value is rounded once
            const double hc = 0.5 * c[j], p = hc * l2, lo = (std::fma(hc, l2, -p) + hc * l2lo) * unit;
            q[j] = (uint64_t)((int64_t)(p * unit) + (int64_t)(lo + (lo < 0.0 ? -0.5 : 0.5))) + bias;
        }
    }
    return true;
}

}  // namespace rbg
