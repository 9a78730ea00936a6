// Host check of rbg_fixed.cuh against extended precision: Box-Muller normals
// to 2^-53 absolute (one FP64 rounding at 1), 2^x to 2^-52 relative, the
// double conversions to half an ulp.  Exits nonzero at the first miss.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "rbg_fixed.cuh"

using namespace rbg;

static FixedTables F;
static const NormalTables& T = F.normals;
static const uint64_t* E = F.exp2;

static void check_normal(uint32_t a, uint32_t b)
{
    const long double tau = 6.28318530717958647692528676655900577L;
    int64_t z[2];
    box_muller_fixed(a, b, T, z[0], z[1]);
    const long double u0 = (a + 0.5L) / 4294967296.0L, u1 = (b + 0.5L) / 4294967296.0L;
    const long double r = std::sqrt(-2.0L * (a >> 31 ? std::log1p(u0 - 1.0L) : std::log(u0)));
    // the angle from its quadrant, so that its sine and cosine keep their accuracy
    const long double q = (long double)(b >> 30), f = u1 - q / 4;
    const long double c = std::cos(tau * f), s = std::sin(tau * f);
    const long double want[2] = {r * (q == 0 ? c : q == 1 ? -s : q == 2 ? -c : s), r * (q == 0 ? s : q == 1 ? c : q == 2 ? -s : -c)};
    for (int i = 0; i < 2; ++i) {
        const long double got = std::ldexp((long double)z[i], -kNormalBits);
        const double d = fixed_to_double(z[i]);
        if (std::fabs(got - want[i]) > 0x1p-53L || std::fabs((long double)d - got) > std::fabs(got) * 0x1p-53L ||
            std::llabs(double_to_fixed(d) - z[i]) > std::fabs(got) * 128 + 1) {
            std::printf("normal %08x %08x: %.20Lg, want %.20Lg, double %.17g\n", a, b, got, want[i], d);
            std::exit(1);
        }
    }
}

static void check_exp2(int64_t x, int ut)
{
    const double d = exp2_fixed(x, ut, E);
    const long double want = std::exp2(std::ldexp((long double)x, -ut));
    if (std::fabs(d - want) > want * 0x1p-52L) {
        std::printf("exp2 %lld 2^-%d: %.17g, want %.20Lg\n", (long long)x, ut, d, want);
        std::exit(1);
    }
    if (ut == 53 && exp2_fixed53(x, E) != d) {
        std::printf("exp2_fixed53 %lld: %.17g, not %.17g\n", (long long)x, exp2_fixed53(x, E), d);
        std::exit(1);
    }
}

// Conditional calls against extended precision: 2^-50 of S + K absolute and, out
// of the money, 1e-12 relative down to 1e-30 (FP64 d1 leaves 2^-53 d1^2).
static void check_call(double v2, double lnS, double K)
{
    SpotFixed sp;
    if (!spot_fixed(v2, lnS, E, sp)) {
        std::printf("spot refused %.17g %.17g\n", v2, lnS);
        std::exit(1);
    }
    const long double v = std::sqrt((long double)v2), S = std::exp((long double)lnS);
    const long double d1 = ((long double)lnS - std::log((long double)K)) / v + v / 2, d2 = d1 - v, h = 0.7071067811865475244L;
    const bool itm = S > K;  // through the put: both wings from small tails
    const long double want = itm ? (S - K) + (K * std::erfc(d2 * h) - S * std::erfc(d1 * h)) / 2
                                 : (S * std::erfc(-d1 * h) - K * std::erfc(-d2 * h)) / 2;
    const double got = call_fixed(sp, K, std::log(K), F.mills, E);
    const long double err = std::fabs(got - want);
    if (err > (S + K) * 0x1p-50L || (!itm && want > 1e-30L && err > want * 1e-12L)) {
        std::printf("call v2=%.17g lnS=%.17g K=%.17g: %.17g, want %.20Lg\n", v2, lnS, K, got, want);
        std::exit(1);
    }
    if (std::fabs(sp.vol / v - 1.0L) > 0x1p-52L || std::fabs(sp.rv * v - 1.0L) > 0x1p-52L) std::exit(1);
}

int main()
{
    fill_fixed_tables(F);
    const uint32_t ea[] = {0, 1, 2, 0x7FFFFFFFu, 0x80000000u, 0xFFEFFFFFu, 0xFFF00000u, 0xFFFFFFFEu, 0xFFFFFFFFu};
    const uint32_t eb[] = {0, 1, 0x1FFFFFu, 0x200000u, 0x3FFFFFFFu, 0x40000000u, 0x7FFFFFFFu, 0x80000000u, 0xBFFFFFFFu,
                           0xC0000000u, 0xFFFFFFFFu};
    for (uint32_t a : ea)
        for (uint32_t b : eb) check_normal(a, b);
    std::mt19937_64 g(7);
    for (int i = 0; i < 400000; ++i) {
        const uint64_t x = g();
        uint32_t a = (uint32_t)x;
        if (i % 8 == 1) a >>= (x >> 59);            // small u0: large radii
        if (i % 8 == 2) a = ~(a >> ((x >> 59)));    // u0 near 1: small radii
        check_normal(a, (uint32_t)(x >> 32));
    }
    for (int ut = 50; ut <= 53; ++ut) {
        for (int k = -kExpTable; k <= kExpTable; ++k)  // both sides of every table entry
            for (int64_t d : {-1, 0, 1}) check_exp2(((int64_t)k << (ut - 12)) + d, ut);
        for (int i = 0; i < 100000; ++i) check_exp2((int64_t)g() >> (64 - ut - 1 - (int)(g() % 9)), ut);
        check_exp2((int64_t)-1022 << ut, ut);
        check_exp2(((int64_t)1023 << ut) + ((int64_t)1 << ut) - 2, ut);
    }
    if (!std::isinf(exp2_fixed((int64_t)1024 << 50, 50, E)) || exp2_fixed(((int64_t)-1022 << 50) - 1, 50, E) != 0.0) return 1;
    for (int i = 0; i < 200000; ++i) {
        auto u = [&] { return (double)(g() >> 11) * 0x1p-53; };
        const double vol = std::exp2(-9.0 + 12.0 * u());
        check_call(vol * vol, (u() - 0.5) * std::min(1.0, 12.0 * vol), 1.0 + (u() - 0.5) * std::min(0.9, 6.0 * vol));
    }
    check_call(2999.0, 0.0, 1.0);
    check_call(1e-199, 1e-100, 1.0);
    check_call(0.04, 59.0, 1e20);
    check_call(0.04, -59.0, 1e-20);
    SpotFixed refused;
    for (double v2 : {0.0, -1.0, 1e-201, 3001.0, (double)NAN, (double)INFINITY})
        if (spot_fixed(v2, 0.0, E, refused)) return 1;
    for (double l : {60.1, -60.1, (double)NAN, (double)INFINITY})
        if (spot_fixed(0.04, l, E, refused)) return 1;
    const double ex[] = {0.0, -0.0, 1.0, -1.0, 6.77, -15.5, 0x1p-6, 0x1p-59, -0x1.8p-59, 0x1p-60, 1e-300};
    for (double d : ex) {
        const long double v = std::ldexp((long double)d, kNormalBits);
        if (std::fabs((long double)double_to_fixed(d) - v) >= 1.0L) return 1;
    }
    if (fixed_to_double(0) != 0.0 || fixed_to_double(1) != 0x1p-59 || fixed_to_double(-1) != -0x1p-59) return 1;
    return 0;
}
