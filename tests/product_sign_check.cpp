// Holds fp::product_le0 (dgcom_gb300/csrc/fp64_bits.hpp) to a·b <= 0 over
// special values, random bit patterns and pairs whose product underflows.
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>
#include <vector>

#include "fp64_bits.hpp"

using namespace dgswe;

int main() {
    const double inf = std::numeric_limits<double>::infinity();
    std::vector<double> x{0.0, -0.0, 1.0, -1.0, 5e-324, -5e-324, 2.2250738585072014e-308, 1e-162,
                          -1e-162, 1.6e-162, 2.3e-162, 1.5e-154, 1.4e-154, 1e308, -1e308, inf, -inf,
                          std::nan("")};
    std::mt19937_64 rng(17);
    for (int i = 0; i < 400; ++i) x.push_back(fp::from_bits((int64_t)rng()));
    for (int e = -540; e <= -500; ++e)  // products from 2^-1080 to 2^-1000
        for (int s = -1; s <= 1; s += 2) {
            x.push_back(s * std::ldexp(1.0 + 1e-16 * (double)(rng() % 4503599627370496ull), e));
            x.push_back(s * std::ldexp(1.0, e));
        }
    long n = 0;
    for (double a : x)
        for (double b : x) {
            const volatile double p = a * b;
            if (fp::product_le0(a, b) != (p <= 0.0)) {
                std::printf("%a times %a\n", a, b);
                return 1;
            }
            ++n;
        }
    std::printf("ok %ld\n", n);
}
