// digit_margin and the read-out that x64_prepare chooses by it, on the host: the margin
// against a direct count, over H and N, and for a Gamma whose digits are all extreme.
#include <cmath>
#include <cstdio>
#include <vector>

#include "rbg_fp64x.hpp"

using namespace rbg;

static Plan plan_of(int N, double a1, const std::vector<double>& gamma)
{
    Plan p;
    p.N = N;
    p.xi = 0.04;
    p.vols = {VolGroup{0.3, 1.0, a1, 0.1, 0, 1}};
    VGroup g{};
    g.scale = 0.1;
    g.eta = 1.0;
    g.dt = 1.0 / N;
    g.sdt = std::sqrt(g.dt);
    g.xi = 0.04;
    g.nsteps = N;
    p.vgs = {g};
    p.gamma = gamma;
    p.comp.assign(N, 0.1);
    return p;
}

int main()
{
    for (int N : {257, 512, 1000, 1024, 1025, 4096})
        for (double H : {0.01, 0.1, 0.49, 0.6, 0.99}) {
            std::vector<double> G(N, 0.0);
            for (int i = 1; i < N; ++i) G[i] = (std::pow(i + 1.0, H + 0.5) - std::pow(i, H + 0.5)) / (H + 0.5);
            X64Tables t;
            if (!x64_prepare(plan_of(N, 1.0 / (H + 0.5), G), t)) {  // a large H's sums leave the fixed-point range
                if (H < 0.5) return 1;
                continue;
            }
            if (x64_wide(t, N) != (N > 1024)) return 2;
            // every prefix, digit by digit
            const double limit = N > 1024 ? 0x1p24 : 0x1p22;
            double least = HUGE_VAL;
            for (int d = 0; d < 8; ++d) {
                double var = 0, mean = 0;
                for (int j = 0; j <= d; ++j) {
                    const double rms = d == j ? 8.0 : 73.9;
                    double s = 0, most = 0, q = 0;
                    for (int k = 0; k < N; ++k) {
                        const uint64_t u = (uint64_t)t.gam[k] + 0x8080808080808080ull;
                        const int x = (int)((u >> (8 * (7 - j))) & 255) - 128;
                        s += x;
                        q += x * x;
                        most = std::max(most, std::fabs(s));
                    }
                    var += q * rms * rms;
                    mean += most * (d == j ? 0.0 : d - j == 3 ? 5.0 : 0.5);
                }
                least = std::min(least, (limit - mean) / std::sqrt(var));
            }
            const double got = digit_margin(t.gam.data(), N, limit);
            std::printf("%d %.2f %.2f %.2f\n", N, H, got, least);
            if (!(got >= kXMargin && std::fabs(got - least) < 0.02 * least + 0.3)) return 3;
        }
    // Gamma' near 127/128 of its unit in every digit: 0x7f7f7f... 2^-62
    for (int N : {512, 1000, 1024, 4096}) {
        const double v = std::ldexp((double)0x3f7f7f7f7f7f7fll, -54);
        X64Tables t;
        const bool ok = x64_prepare(plan_of(N, v, std::vector<double>(N, v)), t);
        const double m = digit_margin(t.gam.data(), N, 0x1p22);
        std::printf("extreme %d %.2f wide %d ok %d\n", N, m, (int)x64_wide(t, N), (int)ok);
        if ((m < kXMargin || N > 1024) != x64_wide(t, N)) return 4;
        if (N == 1024 && m >= kXMargin) return 5;  // a case the rule is for
    }
    return 0;
}
