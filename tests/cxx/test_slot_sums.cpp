// The 32-step sums of the fused variance pass (rbg_fixed.cuh: slot_square,
// slot_product, slot_back) against exact arithmetic: per number of live steps the
// mean error of each sum, in units a term.
#include <cmath>
#include <cstdio>
#include <random>

#include "rbg_fixed.cuh"

using namespace rbg;

int main()
{
    std::mt19937_64 g(5);
    std::normal_distribution<double> z;
    for (int live : {0, 1, 2, 7, 31, 32}) {
        const int trials = 200000;
        long double mean[2] = {0, 0}, most[2] = {0, 0};
        for (int t = 0; t < trials; ++t) {
            uint64_t M[32];
            int e[32], top = -1000;
            int64_t w[32];
            for (int i = 0; i < live; ++i) {
                M[i] = g() | (1ull << 63);  // 2^t = M 2^(e - 63)
                e[i] = -(int)(g() % 3);
                top = e[i] > top ? e[i] : top;
                w[i] = (int64_t)std::ldexp(z(g), kNormalBits) + (int64_t)(g() & 127);
            }
            int64_t s[2] = {slot_back(live), slot_back(live)};
            long double want[2] = {0, 0};
            for (int i = 0; i < live; ++i) {
                const uint64_t m = M[i] >> (top - e[i] + 3);
                s[0] += slot_square(m);
                s[1] += slot_product(m, ((uint64_t)w[i] ^ (1ull << 63)) >> 1);
                // exact: m without the shift's truncation
                const long double x = std::ldexp((long double)M[i], -(top - e[i] + 3));
                want[0] += x * x * 0x1p-64L;
                want[1] += x * std::ldexp((long double)w[i], -65);
            }
            for (int k = 0; k < 2; ++k) {
                const long double d = (long double)s[k] - want[k];
                mean[k] += d / trials;
                most[k] = std::fabs(d) > most[k] ? std::fabs(d) : most[k];
            }
        }
        std::printf("%d %.3Lf %.3Lf %.2Lf %.2Lf\n", live, mean[0], mean[1], most[0], most[1]);
        // half a unit for slot_back's rounding, an eighth a term for its mean; at most two units a term
        for (int k = 0; k < 2; ++k)
            if (std::fabs(mean[k]) > 0.5L + 0.125L * live || most[k] > 1.0L + 2.0L * live) return 1;
    }
    return 0;
}
