// Conditional calls far out of the money (rbg_fixed.cuh: call_fixed) against extended
// precision on the same d1, down to the smallest normal double; below that range zero.
// The density is within 4 units of 2^-50 in its logarithm and one FP64 rounding, 2^-47
// of the price; either of the two Mills ratios, whose difference may be small, within 11
// units of 2^-61 (five products up to 2 units low, table and remainder half a unit each).
#include <cmath>
#include <cstdio>
#include <random>

#include "rbg_fixed.cuh"

using namespace rbg;

int main()
{
    static FixedTables F;
    fill_fixed_tables(F);
    std::mt19937_64 g(3);
    auto u = [&] { return (double)(g() >> 11) * 0x1p-53; };
    int small = 0, zero = 0;
    for (int i = 0; i < 200000; ++i) {
        const double vol = std::exp2(-8.0 + 6.0 * u()), lnS = (u() - 0.5) * 8.0, d = 20.0 + 20.0 * u();
        SpotFixed sp;
        if (!spot_fixed(vol * vol, lnS, F.exp2, sp)) return 1;
        const double K = std::exp(lnS + vol * (d + 0.5 * vol)), lnK = std::log(K);
        const double got = call_fixed(sp, K, lnK, F.mills, F.exp2);
        const long double d1 = (long double)std::fma(sp.lnS - lnK, sp.rv, 0.5 * sp.vol), h = 0.7071067811865475244L;
        const long double S = std::exp((long double)lnS), phi = 0.39894228040143267794L * S * std::exp(-0.5L * d1 * d1);
        auto mills = [&](long double x) { return std::erfc(x * h) * 0.5L / (0.39894228040143267794L * std::exp(-0.5L * x * x)); };
        const long double want = phi * (mills(-d1) - mills(-d1 + sp.vol));
        if (want > 0x1p-1021L && std::exp(-0.5L * d1 * d1) > 0x1p-1020L) {
            ++small;
            if (std::fabs(got - want) > want * 0x1p-47L + phi * 22.0L * 0x1p-61L) {
                std::printf("vol %.17g lnS %.17g K %.17g: %.17g, want %.20Lg\n", vol, lnS, K, got, want);
                return 2;
            }
        } else if (phi < 0x1p-1024L) {
            ++zero;
            if (got != 0.0) return 3;
        }
    }
    return small > 100000 && zero > 1000 ? 0 : 4;
}
