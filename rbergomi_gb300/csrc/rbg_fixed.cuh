// rbg_fixed.cuh -- 64-bit fixed-point arithmetic for the FP64 form.
//
// GB300 issues an FP64 warp instruction every 64 cycles per SM sub-partition
// (2 DFMA per clock and SM) and an integer one every cycle, so the FP64 form's
// elementary functions -- Box-Muller's logarithm, square root and sine /
// cosine, the variance path's exponential -- are evaluated on 64-bit integers.
// Each keeps more bits than FP64 evaluation does: a few 2^-58 (absolute for a
// normal, relative for the exponential) against roundings of 2^-53.
// Everything here also compiles for the host, where it is tested against
// quadruple precision.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define RBG_HD __host__ __device__ __forceinline__
#else
#define RBG_HD inline
#endif

namespace rbg {

RBG_HD uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
RBG_HD uint32_t lo32(uint64_t x) { return (uint32_t)x; }
RBG_HD uint64_t mul32(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
RBG_HD uint32_t mulhi32(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
// High half of a 64 x 64-bit product without the low x low term: three
// 32 x 32 -> 64 multiplies, 0 to 2 below the exact one.
RBG_HD uint64_t mulhi64(uint64_t a, uint64_t b)
{
    return mul32(hi32(a), hi32(b)) + (mul32(hi32(a), lo32(b)) >> 32) + (mul32(lo32(a), hi32(b)) >> 32);
}
RBG_HD double bits_double(uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double d;
    std::memcpy(&d, &b, 8);
    return d;
#endif
}
RBG_HD uint64_t double_bits(double d)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(d);
#else
    uint64_t b;
    std::memcpy(&b, &d, 8);
    return b;
#endif
}

RBG_HD float bits_float(uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float d;
    std::memcpy(&d, &b, 4);
    return d;
#endif
}

// ------------------------------------------------------------------ normals
// Normals in signed fixed point, unit 2^-59 (|z| < 16; Box-Muller on 32-bit
// uniforms stays below 6.77).
constexpr int kNormalBits = 59;

// v 2^-59 as a double, rounded to nearest, in two FP64 additions: the words
// become the low bits of doubles near 2^25 and 2^-7, whose sum less (2^25 + 2^4
// + 2^-7) is v 2^-59; only the last addition rounds.  (Where integer
// instructions are what bounds a kernel, the FP64 pipe is the one to take.)
RBG_HD double fixed_to_double(int64_t v)
{
    const double a = bits_double(0x4180000000000000ull | (hi32((uint64_t)v) ^ 0x80000000u));
    const double b = bits_double(0x3F80000000000000ull | lo32((uint64_t)v));
    return (a - (33554448.0 + 0x1p-7)) + b;
}

// x in units of 2^-59, exact for 2^-6 <= |x| < 16 and truncated below.
RBG_HD int64_t double_to_fixed(double x)
{
    const uint64_t b = double_bits(x);
    const int sh = ((int)(b >> 52) & 2047) - (1023 + 52 - kNormalBits);  // <= 11 for |x| < 16
    const uint64_t m = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
    const uint64_t a = sh >= 0 ? m << (sh & 63) : (sh > -64 ? m >> (-sh & 63) : 0ull);
    const uint64_t s = (uint64_t)((int64_t)b >> 63);
    return (int64_t)((a ^ s) - s);
}

// x as a float, rounded to nearest even: integers in place of the conversion,
// which holds the FP64 pipe 64 cycles a warp, wherever the result is a normal float.
RBG_HD float double_to_float(double x)
{
    const uint64_t b = double_bits(x);
    const uint32_t h = hi32(b), l = lo32(b), a = h & 0x7FFFFFFFu;
    if (a - 0x38100000u >= 0x47EFFFFFu - 0x38100000u) return (float)x;  // zero, below 2^-126, near 2^128 and above, NaN
    uint32_t f = ((a - 0x38000000u) << 3) | (l >> 29);
    f += ((l << 3) | (f & 1u)) > 0x80000000u ? 1u : 0u;
    return bits_float(f | (h & 0x80000000u));
}

// Tables of the transform (shared memory on the device).
//   ln[k], k < 512: x = 1 / c in units of 2^-32, c next to the centre 1 + (k +
//          1/2) / 512 of m in [1, 2); y = ln c in units of 2^-63
//   trig[k], k < 512: (cos, sin)(pi k / 1024) in units of 2^-63
//   ln2[n], n <= 33: n ln 2 in units of 2^-58
struct FixedPair {
    uint64_t x, y;
};
constexpr int kLnTable = 512, kTrigTable = 512, kLn2Table = 34;
struct alignas(16) NormalTables {  // copied 16 bytes at a time
    FixedPair ln[kLnTable];
    FixedPair trig[kTrigTable];
    uint64_t ln2[kLn2Table];
};

RBG_HD int clz32(uint32_t x)
{
#ifdef __CUDA_ARCH__
    return __clz((int)x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}
// 64-bit shifts by 0 .. 31
RBG_HD uint64_t shl(uint64_t x, int n)
{
#ifdef __CUDA_ARCH__
    return ((uint64_t)__funnelshift_l(lo32(x), hi32(x), n) << 32) | (lo32(x) << n);
#else
    return x << n;
#endif
}
RBG_HD uint64_t shr(uint64_t x, int n)
{
#ifdef __CUDA_ARCH__
    return ((uint64_t)(hi32(x) >> n) << 32) | __funnelshift_r(lo32(x), hi32(x), n);
#else
    return x >> n;
#endif
}

// 1 / sqrt(w 2^-64) from below: y 2^-31 within (1 - 2^-20.4, 1) of it, the low
// byte of y zero.  w in [2^62, 2^64).
RBG_HD uint32_t rsqrt_seed(uint64_t w)
{
#ifdef __CUDA_ARCH__
    float f;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(__uint2float_rz(hi32(w)) * 2.3283064365386963e-10f));
    const uint32_t b = __float_as_uint(f) - 0x3f800000u;
#else
    const float f = (float)(1.0 / std::sqrt((double)hi32(w) * 0x1p-32));
    uint32_t b;
    std::memcpy(&b, &f, 4);
    b -= 0x3f800000u;
#endif
    return ((b < 0x007fffffu ? b : 0x007fffffu) << 8) + 0x7ffffc00u;
}

// sqrt(w 2^-64) in units of 2^-63 for w in [2^62, 2^64), within a few units.
// With y just below 1 / sqrt(w): w y^2 = 1 - n, sqrt(w) = w y (1 - n)^(-1/2)
// = w y (1 + n / 2 + 3 n^2 / 8 + O(2^-62)).
RBG_HD uint64_t sqrt_fixed(uint64_t w)
{
    const uint32_t y = rsqrt_seed(w);
    const uint64_t wy = mul32(hi32(w), y) + (mul32(lo32(w), y) >> 32);                  // unit 2^-63
    const uint64_t n = (1ull << 62) - mul32(hi32(wy), y) - (mul32(lo32(wy), y) >> 32);  // unit 2^-62, below 2^43
    const uint32_t n51 = (uint32_t)(n >> 11);                             // unit 2^-51
    const uint64_t c = (n << 20) + mul32(mulhi32(n51, n51), 3072u);       // n / 2 + 3 n^2 / 8, unit 2^-83
    return wy + (mulhi64(c, wy) >> 19);
}

// The factors of a pair of normals.
struct BoxMullerFactors {
    uint64_t root;  // sqrt(-2 ln u0) 2^63 2^-e
    int e;
    uint64_t c, s;  // cosine and sine of 2 pi u1 less its quadrant, unit 2^-63
};

// Box-Muller of two 32-bit words, u0 = (a + 1/2) 2^-32, u1 = (b + 1/2) 2^-32:
// sqrt(-2 ln u0) (cos, sin)(2 pi u1) in units of 2^-59, within 12.1 units and
// 1.53 in root mean square (against quadruple precision; a double of that size
// is rounded by up to 256 units).  Seven 64-bit multiplies fewer than the form
// with the residual of w y^2, four rotation products and every series term to
// 2^-60 (1.40 units): 0.91 -> 0.84 ms for k_normals_fixed's stated draw.  A second
// table for the next nine bits of the angle saves four more and is slower (0.85).
// Their factors are left in f where it is given.
RBG_HD void box_muller_fixed(uint32_t a, uint32_t b, const NormalTables& T, int64_t& z0, int64_t& z1,
                             BoxMullerFactors* f = nullptr)
{
    // -2 ln u0 = w 2^-64 2^ex, w in [2^62, 2^64), ex even
    uint64_t w;
    int ex;
    if (a - 1u >= 0xFFEFFFFFu) {
        if (a == 0u) {
            w = 0xB6FDA8B7905DF579ull;  // 66 ln 2 / 64
            ex = 6;
        } else {
            // 1 - u0 = d 2^-33, d < 2^21: -2 ln u0 = d 2^-32 (1 + x / 2 + x^2 / 3 + x^3 / 4 + x^4 / 5), x = d 2^-33
            // (relative accuracy to the end of the range)
            const uint32_t d = 0u - (2u * a + 1u);
            const uint64_t x = (uint64_t)d << 31;   // unit 2^-64
            const uint32_t x44 = d << 11;           // unit 2^-44, below 2^32
            const uint32_t x2 = mulhi32(x44, x44);  // unit 2^-56
            const uint64_t f = (1ull << 63) + (x >> 2) + (mul32(x2, 0x55555555u + (mulhi32(x44, 0x40000000u) >> 12) +
                                                                (mulhi32(x2, 0x33333333u) >> 24)) >> 25);  // unit 2^-63
            const int n = clz32(d);
            const uint32_t dn = d << n;
            // d 2^-32 f = (w 2^-64) 2^(1 - n)
            w = mul32(dn, hi32(f)) + (mul32(dn, lo32(f)) >> 32);
            ex = 1 - n;
            if (!(w >> 63)) { w <<= 1; --ex; }
            if (ex & 1) { w >>= 1; ++ex; }
        }
    } else {
        // u0 = q 2^-33, q = 2 a + 1 = 2^(32 - n) m; ln m = ln c + log1p(t), t = m / c - 1, |t| < 2^-10
        const int n = clz32(a);
        const uint32_t mh = (a << n) | ((1u << n) >> 1);  // m, unit 2^-31 (n = 0: its 2^-32 is added below)
        const FixedPair lc = T.ln[(mh >> 22) & (kLnTable - 1)];
        // t = m / c - 1, exact but for half a unit (1 / c is a 32-bit number), unit 2^-63
        const int64_t t = (int64_t)(mul32(mh, lo32(lc.x)) + (n ? 0u : lo32(lc.x) >> 1) - (1ull << 63));
        const int32_t th = (int32_t)(t >> 22);                                             // unit 2^-41
        const int32_t tl = (int32_t)lo32((uint64_t)t) & 0x3FFFFF;
        const uint64_t t2 = (uint64_t)((int64_t)th * th + (((int64_t)th * tl) >> 21));     // unit 2^-82
        const int32_t t3 = (int32_t)(((int64_t)th * (int32_t)hi32(t2)) >> 30);             // unit 2^-61
        // 1/3 - t/4 + t^2/5, unit 2^-31
        const int32_t g = 0x2AAAAAAB - (th >> 12) + (int32_t)(mulhi32(hi32(t2), 0x33333333u) >> 19);
        // ln m = ln c + t - t^2 / 2 + t^3 g, unit 2^-63
        const int64_t lm = (int64_t)lc.y + t - (int64_t)(t2 >> 20) + (((int64_t)t3 * g) >> 29);
        // -ln u0 = (n + 1) ln 2 - ln m: unit 2^-63 for u0 > 1/2, where it is small, else 2^-58
        const uint64_t L = n ? T.ln2[n + 1] - (uint64_t)(lm >> 5) : 0x58B90BFBE8E7BCD6ull - (uint64_t)lm;
        const int c0 = n ? 7 : 2;  // 2 L = (L << k) 2^-64 2^(c0 - k); the high word is never zero here
        int k = clz32(hi32(L));
        k -= (c0 - k) & 1;
        w = shl(L, k);
        ex = c0 - k;
    }
    const uint64_t r = shr(sqrt_fixed(w), 3 - (ex >> 1));  // sqrt(-2 ln u0), unit 2^-60

    // 2 pi u1 = (quadrant) pi / 2 + pi k / 1024 + d, d = p pi 2^-32 with p = 2 (b mod 2^21) + 1
    const uint32_t p = 2u * (b & 0x1FFFFFu) + 1u;
    const FixedPair cs = T.trig[(b >> 21) & (kTrigTable - 1)];
    const uint64_t d = (mul32(p, 0xC90FDAA2u) << 10) + (mul32(p, 0x2168C235u) >> 22);  // unit 2^-72
    const uint32_t dh = hi32(d);                                                      // unit 2^-40
    const uint64_t d2 = mul32(dh, dh) + (mul32(dh, lo32(d)) >> 31);                   // unit 2^-80
    const uint32_t d2h = hi32(d2);                                                    // unit 2^-48
    // 1 - cos d = d^2 / 2 - d^4 (1/24 - d^2 / 720), unit 2^-81
    const uint64_t nc = d2 - ((uint64_t)mulhi32(mulhi32(d2h, d2h), 0xAAAAA809u) << 13);
    // sin d = d - d^3 (1/6 - d^2 / 120), unit 2^-72
    const uint32_t c6 = 0xAAAAAAABu - (mulhi32(d2h, 0x02222222u) >> 14);
    const uint64_t sd = d - ((mul32(mulhi32(dh, d2h), c6) + (c6 >> 1)) >> 18);
    // (cos, sin)(a + d) = (x - x nc - y sd, y - y nc + x sd) in three products: with p = (x + y)(sd - nc) the
    // sine is y + p + x nc - y sd
    const uint64_t xn = mulhi64(cs.x, nc) >> 17, ys = mulhi64(cs.y, sd) >> 8;
    const uint64_t c = cs.x - xn - ys;  // unit 2^-63
    const uint64_t sn = cs.y + (mulhi64((cs.x >> 1) + (cs.y >> 1), sd - (nc >> 9)) >> 7) + xn - ys;
    // quadrant q: (c, s), (-s, c), (-c, -s), (s, -c)
    const bool odd = (b & 0x40000000u) != 0u;
    const uint64_t m0 = mulhi64(r, odd ? sn : c), m1 = mulhi64(r, odd ? c : sn);  // unit 2^-59
    const uint64_t s0 = (uint64_t)(int64_t)((int32_t)(b ^ (b << 1)) >> 31);  // cosine negative in quadrants 1, 2
    const uint64_t s1 = (uint64_t)(int64_t)((int32_t)b >> 31);               // sine in 2, 3
    z0 = (int64_t)((m0 ^ s0) - s0);
    z1 = (int64_t)((m1 ^ s1) - s1);
    if (f) *f = BoxMullerFactors{sqrt_fixed(w), ex >> 1, c, sn};
}

// sin(q pi 2^-32), relative accuracy for any 0 < q < 2^31: fixed, unit 2^-63, is it to
// within 2^-59 (half a unit of 2^-53 of it from 2^-5 up).
RBG_HD double sine_double(uint32_t q, uint64_t fixed)
{
    if (fixed >= 1ull << 58) return (double)fixed * 0x1p-63;  // (one is 2^63)
    // pi in two parts, and one more rounding for d - d^3 (1/6 - d^2 / 120 + d^4 / 5040)
    const double p = (double)(int32_t)q, d = fma(p, 0x1.921fb54442d18p+1 * 0x1p-32, p * (0x1.1a62633145c07p-53 * 0x1p-32));
    const double d2 = d * d;
    return fma(d * d2, fma(d2, fma(d2, -1.0 / 5040, 1.0 / 120), -1.0 / 6), d);
}

// The same normals as doubles, within 3 2^-53 of them relatively however small (9 2^-53
// for 1 - u0 down to 2^-12, 3 again below): from the fixed-point ones down to 1/8,
// below by their factors' significant bits.
// (Normals that a caller asks for; a unit of 2^-59 is all the pricing sums need.)
RBG_HD void box_muller_double(uint32_t a, uint32_t b, const NormalTables& T, double& z0, double& z1)
{
    int64_t v0, v1;
    BoxMullerFactors f;
    box_muller_fixed(a, b, T, v0, v1, &f);
    z0 = fixed_to_double(v0);
    z1 = fixed_to_double(v1);
    constexpr int64_t lim = 1ll << (kNormalBits - 3);
    const bool s0 = v0 < lim && v0 > -lim, s1 = v1 < lim && v1 > -lim;
    if (!s0 && !s1) return;
    // the radius in two parts
    const int64_t root = (int64_t)f.root;
    const double unit = bits_double((uint64_t)(uint32_t)(1023 - 63 + f.e) << 52);
    const double rh = (double)(root & ~0x3FFll) * unit, rl = (double)(root & 0x3FFll) * unit;
    const uint32_t q = 2u * (b & 0x3FFFFFFFu) + 1u;
    const double cd = sine_double(0x80000000u - q, f.c), sd = sine_double(q, f.s);
    const double x = fma(rh, cd, rl * cd), y = fma(rh, sd, rl * sd);
    const bool odd = (b & 0x40000000u) != 0u;
    const double m0 = odd ? y : x, m1 = odd ? x : y;
    if (s0) z0 = (int32_t)(b ^ (b << 1)) < 0 ? -m0 : m0;
    if (s1) z1 = (int32_t)b < 0 ? -m1 : m1;
}

// --------------------------------------------------------------- 2^x
// exp2 table: E[k] = 2^(k / 4096) in units of 2^-63.
constexpr int kExpTable = 4096;

// 2^(x 2^-ut) for a signed fixed-point x, ut <= 53, as a double: infinity
// above the range of a double, zero below its normal range.
RBG_HD double exp2_fixed(int64_t x, int ut, const uint64_t* E)
{
    const int64_t e = x >> ut;
    const uint64_t f = (uint64_t)x << (64 - ut);  // fraction, unit 2^-64
    const uint64_t T = E[f >> 52];
    const uint64_t r = f & 0x000FFFFFFFFFFFFFull;  // below 2^-12
    // 2^r - 1 = c1 r + r^2 (c2 + c3 r + c4 r^2), unit 2^-64
    const uint32_t rh = (uint32_t)(r >> 20);         // unit 2^-44
    const uint32_t r2 = mulhi32(rh, rh);             // unit 2^-56
    const uint32_t c = 0xF5FDEFFDu + ((mulhi32(rh, 0x0E35846Bu) + (mulhi32(r2, 0x0276556Eu) >> 12)) >> 10);  // unit 2^-34
    const uint64_t p = mulhi64(r, 0xB17217F7D1CF79ACull) + (mul32(r2, c) >> 26);
    const uint64_t m = T + mulhi64(T, p);            // in [2^63, 2^64)
    const uint64_t b = ((uint64_t)(e + 1022) << 52) + (m >> 11) + ((m >> 10) & 1u);
    return bits_double(e > 1023 ? 0x7FF0000000000000ull : (e < -1022 ? 0ull : b));
}

// 2^(x 2^-53) = m 2^(e - 63), m in [2^63, 2^64).
RBG_HD uint64_t exp2_mantissa53(int64_t x, const uint64_t* E, int32_t& e)
{
    const uint32_t h = hi32((uint64_t)x), l = lo32((uint64_t)x);
    e = (int32_t)h >> 21;
    const uint64_t T = E[(h >> 9) & (kExpTable - 1)];
    const uint32_t rt = h & 511u;                             // remainder below 2^-12: 9 + 32 bits, unit 2^-53
    const uint32_t rh = (rt << 23) | (l >> 9);                // unit 2^-44
    const uint64_t r = ((uint64_t)((rt << 11) | (l >> 21)) << 32) | (l << 11);  // unit 2^-64
    const uint32_t r2 = mulhi32(rh, rh);                      // unit 2^-56
    const uint32_t c = 0xF5FDEFFDu + ((mulhi32(rh, 0x0E35846Bu) + (mulhi32(r2, 0x0276556Eu) >> 12)) >> 10);  // unit 2^-34
    const uint64_t p = mulhi64(r, 0xB17217F7D1CF79ACull) + (mul32(r2, c) >> 26);
    return T + mulhi64(T, p);
}

// exp2_fixed(x, 53, E), its shifts constants.
RBG_HD double exp2_fixed53(int64_t x, const uint64_t* E)
{
    int32_t e;
    const uint64_t m = exp2_mantissa53(x, E, e);
    const uint64_t b = ((uint64_t)((uint32_t)(e + 1022) << 20) << 32) + (m >> 11) + ((m >> 10) & 1u);
    return bits_double(e < -1022 ? 0ull : b);                 // e <= 1023: x 2^-53 < 1024
}

// ------------------------------------------------------- sums of 32 steps
// Terms of the sums of 2^(2 t) and 2^t W over the 32 steps of a warp (the variance
// pass in the convolution's read-out), m = 2^t in units of 2^-61 of the steps'
// largest power of two: m^2 2^-64, and m (w 2^-64) for half = (2^63 + w) >> 1, the
// normal w in units of 2^-59.
RBG_HD int64_t slot_square(uint64_t m)
{
    return (int64_t)(mul32(hi32(m), hi32(m)) + (mul32(hi32(m), lo32(m)) >> 31));
}
RBG_HD int64_t slot_product(uint64_t m, uint64_t half) { return (int64_t)(mulhi64(m, half) - (m >> 2)); }
// What a sum of `live` terms loses to truncation on average, shifting 2^t to m
// included: seven eighths of a unit a term (square 0.75 and m 2^-64, product
// 0.9); steps past the last one lose nothing.
RBG_HD int64_t slot_back(int live) { return (7 * live + 4) >> 3; }

// ---------------------------------------------------------- normal tail
// Mills' ratio M(x) = (1 - Phi(x)) / phi(x), x >= 0, on 64 intervals per octave
// of y = 1 + x, y < 64: with f the position inside the interval (0 .. 1),
//   M = b0 - f (b1 - f (b2 - f (b3 - f (b4 - f (b5 - f b6))))),
// the Taylor series about the interval's left end (all b positive: the
// derivatives of M alternate in sign) with its terms 7 to 9 economised by
// shifted Chebyshev polynomials, which leaves less than 2^-57 of M.
// Units 2^-61.
constexpr int kMillsIntervals = 6 * 64;
struct alignas(16) MillsRow {
    uint64_t b0, b1, b2, b3, b4;
    uint32_t b5, b6;
};
struct MillsTable {
    MillsRow r[kMillsIntervals];
};
constexpr int kTailBits = 57;  // x in units of 2^-57
constexpr uint64_t kTailMax = 62ull << kTailBits;

// M in units of 2^-61 for x 2^-57 (62 from there on, where phi is zero).
RBG_HD uint64_t mills_fixed(uint64_t x, const MillsTable& T)
{
    const uint64_t y = (x < kTailMax ? x : kTailMax) + (1ull << kTailBits);
    const int n = clz32(hi32(y));  // octave 6 - n
    const uint64_t z = shl(y, n);
    const MillsRow& r = T.r[(6 - n) * 64 + (int)((hi32(z) >> 25) & 63u)];
    const uint64_t f = z << 7;
    uint64_t q = r.b4 - mulhi32(r.b5 - mulhi32(r.b6, hi32(f)), hi32(f));
    q = r.b3 - mulhi64(q, f);
    q = r.b2 - mulhi64(q, f);
    q = r.b1 - mulhi64(q, f);
    return r.b0 - mulhi64(q, f);
}

// |x| in units of 2^-57, at most kTailMax (which NaN gives too).
RBG_HD uint64_t tail_fixed(double x)
{
    const uint64_t b = double_bits(x) & 0x7FFFFFFFFFFFFFFFull;
    const int sh = (int)(b >> 52) - (1023 + 52 - kTailBits);  // <= 10 below 64
    const uint64_t m = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
    const uint64_t a = sh >= 0 ? m << (sh & 63) : (sh > -64 ? m >> (-sh & 63) : 0ull);
    return hi32(b) >= 0x404F0000u ? kTailMax : a;
}

// A signed value below 4 in units of 2^-61 as a double (fixed_to_double's form).
RBG_HD double tail_to_double(int64_t v)
{
    const double a = bits_double(0x4160000000000000ull | (hi32((uint64_t)v) ^ 0x80000000u));
    const double b = bits_double(0x3F60000000000000ull | lo32((uint64_t)v));
    return (a - (8388612.0 + 0x1p-9)) + b;
}

// The integrals I_n(x) of s^n exp(-x s - s^2 / 2), s > 0: M = I_0 and M's n-th
// derivative is (-1)^n I_n.  I_{n+1} = n I_{n-1} - x I_n with I_1 = 1 - x I_0:
// forward from erfc for x < 1; above, where that cancels, backward (the I_n are
// the recurrence's minimal solution), normalised by I_1 + x I_0 = 1.
inline void mills_table(MillsTable& T)
{
    constexpr int terms = 10;
    for (int i = 0; i < kMillsIntervals; ++i) {
        const int o = i / 64;
        const long double h = std::ldexp(1.0L, o - 6), x = std::ldexp(1.0L + (i % 64) / 64.0L, o) - 1.0L;
        long double I[terms];
        if (x < 1.0L) {
            I[0] = std::exp(x * x / 2) * std::erfc(x * 0.707106781186547524400844362104849039L) *
                   1.25331413731550025120788264240552263L;
            I[1] = 1.0L - x * I[0];
            for (int n = 1; n + 1 < terms; ++n) I[n + 1] = n * I[n - 1] - x * I[n];
        } else {
            const int top = 30 + (int)(600.0L / (x * x));  // the start value's weight decays as exp(-2 x sqrt(top))
            long double a = 0.0L, c = 1.0L;                // I_{n+1}, I_n up to a factor
            for (int n = top; n >= 1; --n) {
                const long double d = (a + x * c) / n;  // I_{n-1}
                a = c;
                c = d;
                if (n - 1 < terms) I[n - 1] = c;
                if (c > 1e300L) {  // keep the unnormalised values in range
                    a *= 1e-300L;
                    c *= 1e-300L;
                    for (int k = n - 1; k < terms; ++k) I[k] *= 1e-300L;
                }
            }
            const long double f = 1.0L / (I[1] + x * I[0]);
            for (int n = 0; n < terms; ++n) I[n] *= f;
        }
        long double c[terms], hn = 1.0L, fact = 1.0L;
        for (int n = 0; n < terms; ++n, hn *= h) {
            if (n) fact *= -n;
            c[n] = I[n] / fact * hn;
        }
        // f^n less T*_n(f) / 2^(2n - 1), n = 9, 8, 7 in turn (T*_n the shifted Chebyshev polynomials)
        const long double t9[10] = {-1, 162, -4320, 44352, -228096, 658944, -1118208, 1105920, -589824, 131072};
        const long double t8[9] = {1, -128, 2688, -21504, 84480, -180224, 212992, -131072, 32768};
        const long double t7[8] = {-1, 98, -1568, 9408, -26880, 39424, -28672, 8192};
        const long double* t[3] = {t9, t8, t7};
        for (int k = 0; k < 3; ++k) {
            const int n = 9 - k;
            for (int j = 0; j < n; ++j) c[j] -= c[n] * t[k][j] / t[k][n];
        }
        MillsRow& r = T.r[i];
        auto fix = [](long double v) { return (uint64_t)(std::ldexp(v, 61) + 0.5L); };
        r.b0 = fix(c[0]);
        r.b1 = fix(-c[1]);
        r.b2 = fix(c[2]);
        r.b3 = fix(-c[3]);
        r.b4 = fix(c[4]);
        r.b5 = (uint32_t)fix(-c[5]);
        r.b6 = (uint32_t)fix(c[6]);
    }
}

// Every table above, one copy per device.
struct FixedTables {
    NormalTables normals;
    uint64_t exp2[kExpTable];
    MillsTable mills;
};

// Their values, in extended precision on the host.
inline void fill_fixed_tables(FixedTables& F)
{
    NormalTables& T = F.normals;
    for (int k = 0; k < kLnTable; ++k) {
        const long double c = 1.0L + (k + 0.5L) / kLnTable;
        const uint64_t x = (uint64_t)(std::ldexp(1.0L / c, 32) + 0.5L);
        T.ln[k] = FixedPair{x, (uint64_t)(std::ldexp(-std::log(std::ldexp((long double)x, -32)), 63) + 0.5L)};
    }
    const long double pi = 3.14159265358979323846264338327950288L, ln2 = 0.693147180559945309417232121458176568L;
    for (int k = 0; k < kTrigTable; ++k) {
        const long double a = pi * k / (2 * kTrigTable);
        T.trig[k] = FixedPair{(uint64_t)(std::ldexp(std::cos(a), 63) + 0.5L),
                              (uint64_t)(std::ldexp(std::sin(a), 63) + 0.5L)};
    }
    for (int n = 0; n < kLn2Table; ++n) T.ln2[n] = (uint64_t)(std::ldexp(ln2 * n, 58) + 0.5L);
    for (int k = 0; k < kExpTable; ++k)
        F.exp2[k] = (uint64_t)(std::ldexp(std::exp2(k / (long double)kExpTable), 63) + 0.5L);
    mills_table(F.mills);
}

// sqrt(v) and its reciprocal as doubles, for a normal positive v: the square
// root of the significand in fixed point, the exponent halved.
RBG_HD void sqrt_recip(double v, double& root, double& recip)
{
    const uint64_t b = double_bits(v);
    const int e = (int)(b >> 52) - 1023;  // v = 2^e m, m in [1, 2)
    // w 2^-64 = v 2^-(2 k), in [1/4, 1): k = (e + 2) >> 1
    const int k = (e + 2) >> 1;
    const uint64_t m = ((b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << 11;  // m, unit 2^-63
    const uint64_t w = (e & 1) ? m : m >> 1;
    const uint32_t y = rsqrt_seed(w);
    const uint64_t n = (1ull << 62) - mulhi64(w, mul32(y, y));
    const uint64_t wy = mul32(hi32(w), y) + (mul32(lo32(w), y) >> 32);
    const uint32_t n51 = (uint32_t)(n >> 11);
    const uint64_t c = (n << 20) + mul32(mulhi32(n51, n51), 3072u);  // (1 - n)^(-1/2) - 1, unit 2^-83
    const uint64_t r = wy + (mulhi64(c, wy) >> 19);                  // sqrt, unit 2^-63, in [2^62, 2^63)
    const uint64_t yy = (uint64_t)y << 31;                           // y, unit 2^-62, in [2^62, 2^63)
    const uint64_t q = yy + (mulhi64(c, yy) >> 19);                  // reciprocal, unit 2^-62
    // r 2^-63 2^k and q 2^-62 2^-k, 53 bits each (the leading one adds to the exponent field)
    root = bits_double(((uint64_t)(uint32_t)(1023 - 1 + k - 1) << 52) + (r >> 10) + ((r >> 9) & 1u));
    recip = bits_double(((uint64_t)(uint32_t)(1023 - k - 1) << 52) + (q >> 10) + ((q >> 9) & 1u));
}

// x log2(e) in units of 2^-53, |x| < 62.
RBG_HD int64_t log2e_fixed53(double x)
{
    const uint64_t q = (mulhi64(tail_fixed(x), 0xB8AA3B295C17F0BCull) + 5) >> 3;  // log2(e) / 2: 2^-56 before the shift
    return (int64_t)double_bits(x) < 0 ? -(int64_t)q : (int64_t)q;
}

// log2 of S phi(d) sqrt(2 pi) less log2 S, in units of 2^-53: -d^2 / 2 log2 e, d
// as tail_fixed gives it (finer units below 8, where it matters).
RBG_HD uint64_t half_square_log2(uint64_t d)
{
    const bool small = hi32(d) < (8u << (kTailBits - 32));
    const uint64_t x = small ? d << 3 : d;
    const uint64_t q = mulhi64(mulhi64(x, x), 0xB8AA3B295C17F0BCull);  // log2(e) / 2
    return small ? (q + 6) >> 3 : (q < (1023ull << 50) ? q << 3 : 1023ull << 53);  // at most 1023
}
constexpr int64_t kLog2Sqrt2Pi53 = 0x002A6C873498DDF7ll;  // log2(2 pi) / 2, unit 2^-53

// S phi(d) for e = log2(S / sqrt(2 pi)): zero from half_square_log2(d) = lim on, where
// it leaves the doubles' normal range (S phi below 2^-1022, or phi).
constexpr RBG_HD uint64_t density_limit(int64_t e)
{
    constexpr int64_t top = (int64_t)1022 << 53;
    return (uint64_t)(e < 0 ? top + e : top);
}
RBG_HD double density_fixed(int64_t e, uint64_t hs, uint64_t lim, const uint64_t* E)
{
    const bool in = hs < lim;
    const double f = exp2_fixed53(e - (int64_t)(in ? hs : 0ull), E);
    return in ? f : 0.0;
}

// The strike-independent parts of a conditional Black-Scholes call (tau = 1, r
// = 0): spot and its logarithm, volatility and its reciprocal, and in fixed
// point the volatility (2^-57) and log2(S / sqrt(2 pi)) (2^-53).
struct SpotFixed {
    double S, lnS, vol, rv;
    int64_t volf, e;
    uint64_t lim;  // density_limit(e)
};

// False where the numbers leave the ranges of the fixed-point form.
RBG_HD bool spot_fixed(double v2, double lnS, const uint64_t* E, SpotFixed& r)
{
    // 1e-200 < v2 < 3000 and |lnS| < 60
    const uint32_t hv = hi32(double_bits(v2)), hs = hi32(double_bits(lnS)) & 0x7FFFFFFFu;
    if (!(hv - 0x16700000u < 0x40A77000u - 0x16700000u && hs < 0x404E0000u)) return false;
    sqrt_recip(v2, r.vol, r.rv);
    r.lnS = lnS;
    r.volf = (int64_t)tail_fixed(r.vol);
    const int64_t l = log2e_fixed53(lnS);
    r.S = exp2_fixed53(l, E);
    r.e = l - kLog2Sqrt2Pi53;
    r.lim = density_limit(r.e);
    return true;
}

// The call at strike K.  With S phi(d1) = K phi(d2) and 1 - Phi(x) = phi(x) M(x)
// it is
//   [d1 >= 0] S - [d2 >= 0] K + S phi(d1) (-+ M(|d1|) +- M(|d2|)):
// one exponential, tails that keep their relative accuracy, and nine FP64
// operations with the caller's two sums.
RBG_HD double call_fixed(const SpotFixed& r, double K, double lnK, const MillsTable& T, const uint64_t* E)
{
    const double d1 = fma(r.lnS - lnK, r.rv, 0.5 * r.vol);
    const bool n1 = (int64_t)double_bits(d1) < 0;
    const uint64_t x1 = tail_fixed(d1);
    const int64_t d2 = (n1 ? -(int64_t)x1 : (int64_t)x1) - r.volf;
    const bool n2 = d2 < 0;
    const uint64_t x2 = (uint64_t)(n2 ? -d2 : d2);
    const double f = density_fixed(r.e, half_square_log2(x1), r.lim, E);
    const int64_t m1 = (int64_t)mills_fixed(x1, T), m2 = (int64_t)mills_fixed(x2, T);
    const double m = tail_to_double((n1 ? m1 : -m1) + (n2 ? -m2 : m2));
    return fma(f, m, (n1 ? 0.0 : r.S) - (n2 ? 0.0 : K));
}

}  // namespace rbg
