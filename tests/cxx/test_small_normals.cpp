// box_muller_double (rbg_fixed.cuh) against extended precision, relative error in units
// of 2^-53, the smallest normals included (an angle next to an axis, a radius next to
// zero).  Three roundings of a unit; for u0 above 1/2 the logarithm's 3 units of 2^-63
// on top, relative to 1 - u0 and halved by the square root, up to where a series in 1 -
// u0 takes over at 2^-12.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <random>

#include "rbg_fixed.cuh"

using namespace rbg;

// the kernels copy every table 16 bytes at a time, the normals' into shared memory of its type
static_assert(alignof(NormalTables) % 16 == 0 && sizeof(NormalTables) % 16 == 0, "normals");
static_assert(alignof(MillsTable) % 16 == 0 && offsetof(FixedTables, exp2) % 16 == 0 &&
                  offsetof(FixedTables, mills) % 16 == 0, "exponential, tails");

static FixedTables F;

static long double worst = 0;

static bool check(uint32_t a, uint32_t b)
{
    const long double pi = 3.14159265358979323846264338327950288L;
    double z[2];
    box_muller_double(a, b, F.normals, z[0], z[1]);
    const long double u0 = (a + 0.5L) / 4294967296.0L;
    const long double r = std::sqrt(-2.0L * (a >> 31 ? std::log1p(u0 - 1.0L) : std::log(u0)));
    // sine and cosine from the nearer axis, exactly reduced
    const long double q = 2.0L * (b & 0x3FFFFFFFu) + 1.0L, c = std::sin(pi * ((1ll << 31) - q) / 4294967296.0L),
                      s = std::sin(pi * q / 4294967296.0L);
    const int k = (int)(b >> 30);
    const long double want[2] = {r * (k == 0 ? c : k == 1 ? -s : k == 2 ? -c : s), r * (k == 0 ? s : k == 1 ? c : k == 2 ? -s : -c)};
    for (int i = 0; i < 2; ++i) {
        const long double e = std::fabs(z[i] / want[i] - 1.0L) * 0x1p53L;
        worst = std::max(worst, e);
        const long double lim = 3.0L + (a >> 31 && a <= 0xFFEFFFFFu ? 0x1.8p-10L / (1.0L - u0) : 0.0L);
        if (!(e < lim)) {
            std::printf("%08x %08x: %.17g, want %.20Lg, off %Lg\n", a, b, z[i], want[i], e);
            return false;
        }
    }
    return true;
}

int main()
{
    fill_fixed_tables(F);
    const uint32_t ea[] = {0, 1, 2, 0x7FFFFFFFu, 0x80000000u, 0xFFEFFFFFu, 0xFFF00000u, 0xFFFFFFFEu, 0xFFFFFFFFu};
    for (uint32_t a : ea)
        for (uint32_t k = 0; k < 4; ++k)
            for (uint32_t d : {0u, 1u, 77u, 0x1FFFFFu, 0x200000u, 0x28BE60u, 0x28BE61u, 0x400000u, 0x10000000u})
                if (!check(a, (k << 30) + d) || !check(a, (k << 30) + 0x3FFFFFFFu - d)) return 1;
    std::mt19937_64 g(11);
    for (int i = 0; i < 600000; ++i) {
        const uint64_t x = g();
        uint32_t a = (uint32_t)x, b = (uint32_t)(x >> 32);
        const int sh = (int)(g() % 31);
        if (i % 4 == 1) a = ~(a >> sh);                                          // radius next to zero
        if (i % 4 == 2) b = (b & 0xC0000000u) | ((b & 0x3FFFFFFFu) >> sh);          // angle next to an axis
        if (i % 4 == 3) b = (b & 0xC0000000u) | (0x3FFFFFFFu - ((b & 0x3FFFFFFFu) >> sh));
        if (!check(a, b)) return 1;
    }
    std::printf("worst %.3Lf\n", worst);
    return 0;
}
