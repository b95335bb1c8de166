// A fresh StepCtl is one that a dt pass may start from: the smallest step and
// the bound of it both +∞, nothing else set.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "device.hpp"

using namespace dgswe;

int main() {
    StepCtl c;
    std::memset((void*)&c, 0xFF, sizeof c);
    c = StepCtl{};
    double step;
    float bound;
    std::memcpy(&step, &c.dt_bits, sizeof step);
    std::memcpy(&bound, &c.dt_up, sizeof bound);
    if (!std::isinf(step) || step < 0.0 || !std::isinf(bound) || bound < 0.0f) {
        std::printf("smallest step %g, bound %g\n", step, bound);
        return 1;
    }
    if (c.t != 0.0 || c.steps != 0 || c.clips != 0 || c.active != 0 || c.failure != 0 ||
        c.stage[0].a != StageArgs{}.a || c.st_beta[0] != 0.0) {
        std::printf("not cleared\n");
        return 1;
    }
    std::printf("ok\n");
}
