// Holds sqrt_pos, rcp_pos, div_pos and pow_m43 of dgcom_gb300/csrc/fixed64.hpp to
// 0.75 ulp of the long double value, over their whole argument ranges:
// random mantissas, mantissas at both ends, every exponent (parity and
// remainder by three). Compiled with several DGSWE_SEED_ERROR, which stand
// for the device's special-function seeds (each within 2^-21).
#include <cmath>
#include <cstdio>
#include <random>

#include "fixed64.hpp"

using namespace dgswe;

static double ulps(double got, long double want) {
    const double w = std::fabs((double)want);
    return (double)(fabsl((long double)got - want) / (std::nextafter(w, INFINITY) - w));
}

int main() {
    std::mt19937_64 rng(1);
    double worst[4] = {0.0, 0.0, 0.0, 0.0};
    long checks = 0;
    for (int e = 1023 - 124; e < 1023 + 124; ++e)
        for (int i = 0; i < 3000; ++i) {
            uint64_t m = rng() & fx::kMantissa;
            if (i % 7 == 0) m = rng() % 64;
            if (i % 7 == 1) m = fx::kMantissa - rng() % 64;
            const double x = fp::from_bits((int64_t)(((uint64_t)e << 52) | m));
            const long double c = cbrtl((long double)x);
            const double y = fp::from_bits((int64_t)(((uint64_t)(1023 - 200 + rng() % 400) << 52) |
                                                     (i % 5 ? rng() & fx::kMantissa : m)));
            const double n = i % 2 ? x : -x;
            const double off[4] = {ulps(fx::sqrt_pos(x), sqrtl((long double)x)),
                                   ulps(fx::rcp_pos(x), 1.0L / (long double)x),
                                   ulps(fx::pow_m43(x), 1.0L / (c * c * c * c)),
                                   ulps(fx::div_pos(n, y), (long double)n / (long double)y)};
            for (int k = 0; k < 4; ++k) {
                if (!(off[k] <= 0.75)) {
                    std::printf("function %d at %a: %g ulp\n", k, x, off[k]);
                    return 1;
                }
                worst[k] = std::fmax(worst[k], off[k]);
                ++checks;
            }
        }
    std::printf("ok %ld checks; worst %.4f %.4f %.4f %.4f ulp\n", checks, worst[0],
                worst[1], worst[2], worst[3]);
}
