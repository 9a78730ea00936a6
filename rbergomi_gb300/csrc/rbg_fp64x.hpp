// rbg_fp64x.hpp -- the FP64 form's fixed-point / tensor-core path pass
// (rbg_fp64x.cu): its tables and launchers.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "rbg_internal.hpp"

namespace rbg {

// Steps the digit convolution takes (its accumulators' exactness, rbg_fp64x.cu).
constexpr int kX64MaxN = 4096;
// Fewest fraction bits of the variance exponent: parameters whose worst-case
// exponent leaves fewer go through the FP64 kernels.
constexpr int kX64MinUt = 50;

struct X64Vol {
    int sh;             // X = S_hi 2^sh + S_lo 2^(sh - 32), unit 2^-ux
    int vg_begin, vg_end, pad;
    uint64_t a2f, a2h;  // a2 2^(ux - 59 + 64); its half, less the product's mean truncation
};
struct X64Group {
    uint64_t cf;  // |eta scale log2(e) / 2| 2^(ut - ux + 64)
    int ut, neg;  // fraction bits of the exponent; sign of the factor
    double dtxi, sdtxi;
};
struct X64Tables {
    std::vector<X64Vol> vols;
    std::vector<X64Group> grps;
    std::vector<int64_t> gam;    // [n_vol][N] (a1, Gamma_1, ...), unit 2^(e - 62)
    std::vector<uint64_t> comp;  // [n_vg][N] compensator in exponent units, plus cf / 2 - 1
    int max_groups = 0;          // most variance groups of one pass
    bool u53 = true;             // every group has 53 fraction bits
};
// Size that the caller's normals (ext) stay below: 15.5.
constexpr double kExtMax = 15.5;
// Standard deviations the convolution's accumulators keep from their limits.
constexpr double kXMargin = 9.0;
// How many standard deviations every partial sum of W1's digits times those of Gamma' (gam, N
// steps) stays from `limit`, at least.
double digit_margin(const int64_t* gam, int N, double limit);
// Whether the convolution's accumulators may pass 2^22 (4 us a pass of 512 steps on the
// host: callers ask while the normals are drawn).
bool x64_wide(const X64Tables& t, int N);
// False where the plan's numbers do not fit the fixed-point ranges; ext: for the
// caller's normals.
bool x64_prepare(const Plan& plan, X64Tables& out, bool ext = false);

int x64_blocks(int N);
size_t x64_panel_bytes(int N);  // per Volterra pass
size_t x64_digit_bytes(int64_t B, int N);

// The fixed-point and tail tables on the current device (rbg_fixed.cuh), part of
// the module; null where their address could not be had.
struct FixedTables;
const FixedTables* fixed_tables();

// The launchers return nonzero where the device refuses.
// Philox normals Z[m][s][j] of ns streams per path (W1, W1perp, plain MC: Wperp);
// f32: the mixed form's FP32 normals, widened; dig non-null (for the path passes
// below): the digits of W1 too; fix: streams (bit s: stream s) stored in 64-bit
// fixed point, unit 2^-59, in place of doubles: kFixAll for the fused pass, kFixW1perp
// for the separate one, whose FP64 sums take the doubles.
constexpr int kFixAll = 7, kFixW1perp = 2;
// exact: doubles with all their bits significant however small (f32 = 0, no digits), for
// normals that leave the library; a unit of 2^-59 is all the pricing sums need.
int launch_normals_fixed(uint64_t seed, int64_t path0, int64_t B, int N, int f32, double* Z, unsigned char* dig, int fix,
                         int ns, cudaStream_t st, bool exact = false);
void launch_panels(const int64_t* gam, int nv, int N, unsigned char* panels, cudaStream_t st);
// Digits of the caller's W1; *flag |= 1 where W1 or W1perp is kExtMax or more in
// size, or NaN.
void launch_digits(const double* Z, int64_t B, int N, int ns, unsigned char* dig, unsigned int* flag, cudaStream_t st);
// X[v][m][j] + 2^63; any: exact for any digits, not only for those of independent
// normals
int launch_volterra_exact(const unsigned char* dig, const unsigned char* panels, const X64Vol* vols, int nv, int N,
                          int64_t B, bool any, bool wide, uint64_t* X, unsigned int* err, cudaStream_t st);
// Both passes in one kernel, for groups with 53 fraction bits; the passes'
// groups are grp0 .. grp0 + ng - 1, part holds x64_slot_bytes per group.
// Worth it up to x64_fuse_groups groups a pass (path pass in microseconds, fused
// against separate; 512 steps, 2^16 paths): two sums 1 group 550 / 775, 3 groups 912 /
// 1001, 4 groups 1146 / 1117, 8 groups 1908 / 1773; three sums 1 group 606 / 967, 4
// groups 1496 / 1506, 6 groups 2052 / 2215, 8 groups 2582 / 2549.
constexpr int x64_fuse_groups(int ns) { return ns == 3 ? 6 : 3; }
size_t x64_slot_bytes(int64_t B, int N, int ns);
int launch_volterra_variance(const unsigned char* dig, const unsigned char* panels, const X64Vol* vols,
                             const X64Group* grps, const uint64_t* comp, const double* Z, int nv, int grp0, int ng, int ns,
                             bool wide, int N, int64_t B, double* part, double* ivb, double* ivp, unsigned int* err, cudaStream_t st);
// ivb[g][B] (Ivdt, IsvdW); ns = 3: ivp[g][B] IsvdWp too; ext: Z holds doubles
// throughout
int launch_variance_fixed(const X64Vol* vols, const X64Group* grps, const uint64_t* comp, const double* Z,
                          const uint64_t* X, int nv, int max_groups, bool u53, bool ext, int ns, int N, int64_t B,
                          double* ivb, double* ivp, cudaStream_t st);

}  // namespace rbg
