// The FP64 chunk sums of the payoffs (launch_payoff_sums) against exact sums of
// the per-path payoffs of the same path sums (launch_payoff_store): prints, per
// paths per thread G, the root mean square over chunks and outputs of the relative
// error of sum + compensation, in units of 2^-53, and the largest.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "rbg_internal.hpp"

using namespace rbg;

// s + c += x, a double-double sum: about 100 bits.
static void add(double& s, double& c, double x)
{
    const double t = s + x, z = t - s, e = (s - (t - z)) + (x - z);
    const double u = c + e;
    s = t + u;
    c = u - (s - t);
}

template <class T>
static T* upload(const std::vector<T>& v)
{
    void* p = nullptr;
    if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess ||
        cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess)
        std::exit(2);
    return static_cast<T*>(p);
}

int main()
{
    const int n_out = 9, n_vg = 2;
    for (int mc = 0; mc < 2; ++mc) {
        for (int G : {1, 8, 9, 54}) {
            const int nchunks = 40;
            const int64_t B = (int64_t)256 * G * (nchunks - 1) + 77;
            std::mt19937_64 g(G + mc);
            std::normal_distribution<double> z;
            std::vector<double> ivb((size_t)n_vg * B * 2), ivp((size_t)n_vg * B);
            for (size_t i = 0; i < (size_t)n_vg * B; ++i) {
                const double v = 0.05 * std::exp(0.5 * z(g));
                ivb[2 * i] = v;
                ivb[2 * i + 1] = std::sqrt(v) * z(g);
                ivp[i] = std::sqrt(v) * z(g);
            }
            std::vector<OutDev> outs;
            for (int i = 0; i < n_out; ++i) outs.push_back(OutDev{-0.8 + 0.1 * (i / 3), 0.8 + 0.1 * (i % 3), i / 5, 0});
            Fp64Tables t{};
            OutDev* douts = upload(outs);
            double *divb = upload(ivb), *divp = mc ? upload(ivp) : nullptr;
            std::vector<double> pay((size_t)B * n_out), part((size_t)nchunks * n_out * 4, NAN);
            double *dpay = upload(pay), *dpart = upload(part);
            t.outs = douts;
            t.n_out = n_out;
            if (launch_payoff_store(t, divb, B, B, dpay, nullptr, divp) ||
                launch_payoff_sums(t, divb, B, B, G, dpart, nchunks, nullptr, divp))
                return 3;
            if (cudaMemcpy(pay.data(), dpay, pay.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
                cudaMemcpy(part.data(), dpart, part.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess)
                return 4;
            double sq = 0.0, most = 0.0;
            for (int c = 0; c < nchunks; ++c)
                for (int i = 0; i < n_out; ++i) {
                    double s[2] = {0, 0}, e[2] = {0, 0};
                    for (int64_t m = (int64_t)c * G * 256; m < std::min(B, (int64_t)(c + 1) * G * 256); ++m) {
                        const double x = pay[(size_t)m * n_out + i], xx = x * x;
                        add(s[0], e[0], x);
                        add(s[1], e[1], xx);
                        add(s[1], e[1], std::fma(x, x, -xx));
                    }
                    for (int k = 0; k < 2; ++k) {
                        const double* p = &part[((size_t)c * n_out + i) * 4 + 2 * k];
                        const double r = std::fabs(((p[0] - s[k]) + (p[1] - e[k])) / s[k]) * 0x1p53;
                        sq += r * r;
                        most = std::max(most, r);
                    }
                }
            std::printf("%d %d %.4f %.4f\n", mc, G, std::sqrt(sq / (2 * nchunks * n_out)), most);
            for (void* p : {(void*)douts, (void*)divb, (void*)divp, (void*)dpay, (void*)dpart}) cudaFree(p);
        }
    }
    return 0;
}
