// double_to_float (rbg_fixed.cuh) against the conversion: the same bits for
// every exponent, at ties and one unit beside them, and at the ends of the range.
#include <cmath>
#include <cstdio>
#include <random>

#include "rbg_fixed.cuh"

using namespace rbg;

static int bad(uint64_t b)
{
    const double x = bits_double(b);
    const float f = double_to_float(x), g = (float)x;
    uint32_t u, v;
    std::memcpy(&u, &f, 4);
    std::memcpy(&v, &g, 4);
    if (u == v || (std::isnan(f) && std::isnan(g))) return 0;
    std::printf("%a: %a, not %a\n", x, f, g);
    return 1;
}

int main()
{
    std::mt19937_64 g(5);
    int n = 0;
    for (uint64_t sign = 0; sign < 2; ++sign) {
        for (uint64_t e = 0; e < 2048; ++e) {
            const uint64_t base = sign << 63 | e << 52;
            for (int i = 0; i < 200; ++i) {
                const uint64_t m = g() & 0xFFFFFFFFFFFFFull, top = m & ~0x1FFFFFFFull;
                for (uint64_t low : {m & 0x1FFFFFFFull, 0x0ull, 0x1ull, 0x0FFFFFFFull, 0x10000000ull, 0x10000001ull, 0x1FFFFFFFull})
                    n += bad(base | top | low);
            }
            for (uint64_t low : {0x0ull, 0x1ull, 0xFFFFFFFFFFFFFull, 0xFFFFFEFFFFFFFull, 0xFFFFFF0000000ull, 0xFFFFFE0000000ull})
                n += bad(base | low);
        }
    }
    return n != 0;
}
