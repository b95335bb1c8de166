// Holds the fixed-point flux between two sides (fx::face_flux of
// dgcom_gb300/csrc/fixed64.hpp) to long double side by side: the shallower side's
// momentum flux over that side's own pressure and momentum, the mass flux over
// the larger of the reconstructed sides' and the wave between them, beside the
// same formulas in FP64, for depths in the
// ratio 1 to 2^20: one surface over a step of the bed, one bed under a jump of
// the surface, films on a step above the water, steps and jumps at once, equal
// depths; surfaces at the datum and off it, currents from 1e-16 to 1 of the
// wave's speed, the shallow side's bed and the normal turned any way.
//
// The check asks, in each octave of the depths' ratio, that the root mean square
// error is no larger than FP64's and the largest no larger than twice FP64's
// largest, or below 2^-51 of the side's own where FP64 happens to be exact.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "host_common.hpp"

using namespace dgswe;
typedef long double Q;

struct Side {
    double h, u, v, b;
};

template <class T>
struct Five {
    T h, xa, ya, xb, yb;
};

constexpr double kHMin = 1e-9;

// hydro_hll with a reconstructed side above h_min
template <class T>
static Five<T> hll(const Side& a, const Side& b, T nx, T ny, T g, T sg, T hg) {
    const T top = std::max(a.b, b.b), zero = 0;
    const T sa = std::max((T)a.h + a.b - top, zero), sb = std::max((T)b.h + b.b - top, zero);
    const bool wet_a = sa > kHMin, wet_b = sb > kHMin;
    auto rotate = [&](const Side& q, T& n, T& t) {
        const T u = q.h > kHMin ? q.u : 0.0, v = q.h > kHMin ? q.v : 0.0;
        n = u * nx + v * ny;
        t = -u * ny + v * nx;
    };
    T ra, ta, rb, tb;
    rotate(a, ra, ta);
    rotate(b, rb, tb);
    const T na = wet_a ? ra : zero, nb = wet_b ? rb : zero;
    const T ca = sg * std::sqrt(sa), cb = sg * std::sqrt(sb);
    const T um = (std::sqrt(sa) * na + std::sqrt(sb) * nb) / (std::sqrt(sa) + std::sqrt(sb));
    const T cm = std::sqrt(g * (T)0.5 * (sa + sb));
    const T sl = wet_a ? std::min(na - ca, um - cm) : nb - 2 * cb;
    const T sr = wet_b ? std::max(nb + cb, um + cm) : na + 2 * ca;
    const T l[3] = {sa * na, sa * na * na + hg * sa * sa, sa * na * ta};
    const T r[3] = {sb * nb, sb * nb * nb + hg * sb * sb, sb * nb * tb};
    const T jump[3] = {sb - sa, sb * rb - sa * ra, sb * tb - sa * ta};
    T f[3];
    for (int k = 0; k < 3; ++k)
        f[k] = sl >= 0 ? l[k]
                       : (sr <= 0 ? r[k] : (sr * l[k] - sl * r[k] + sl * sr * jump[k]) / (sr - sl));
    const T da = hg * ((T)a.h * a.h - sa * sa), db = hg * ((T)b.h * b.h - sb * sb);
    const T x = f[1] * nx - f[2] * ny, y = f[1] * ny + f[2] * nx;
    return {f[0], x + da * nx, y + da * ny, x + db * nx, y + db * ny};
}

struct Score {
    double fixed = 0.0, fp64 = 0.0, worst = 0.0, worst64 = 0.0;
    long n = 0;
    void add(Q got, Q other, Q want, Q own) {
        const double f = (double)(fabsl(got - want) / own), d = (double)(fabsl(other - want) / own);
        fixed += f * f;
        fp64 += d * d;
        worst = std::max(worst, f);
        worst64 = std::max(worst64, d);
        ++n;
    }
    bool ok() const {
        return n < 200 || (worst <= std::max(2.0 * worst64, 0x1p-51) &&
                           (fixed <= fp64 || std::sqrt(fixed / n) <= 0x1p-53));
    }
};

int main() {
    std::uniform_real_distribution<double> U(0.0, 1.0);
    Physics P{};
    P.g = 9.81;
    P.sqrt_g = std::sqrt(P.g);
    P.half_g = 0.5 * P.g;
    P.two_g = 2.0 * P.g;
    Operators ops(1);
    DevTables T{};
    std::vector<FxLimb> coef;
    fixed_constants(PairSchedule(ops), P, T, coef);
    const char* names[7] = {"one surface at the datum, a step", "one surface off it, a step",
                            "a jump, one bed",                  "films on a step",
                            "steps and jumps",                  "slow currents, equal depths",
                            "one surface near the datum, a step"};
    bool good = true;
    for (int kind = 0; kind < 7; ++kind) {
        std::mt19937_64 rng(3 + kind);
        std::vector<Score> mass(24), momentum(24);
        long done = 0;
        for (int i = 0; i < 500000; ++i) {
            const double H = std::pow(10.0, -2.0 + 4.0 * U(rng)), turn = 6.283185307179586 * U(rng);
            const double r = std::exp2(-20.0 * U(rng));
            const double off = H * (U(rng) - 0.5) * (kind == 6 ? std::exp2(-14.0 * U(rng)) : 1.0);
            double nx = std::cos(turn), ny = std::sin(turn);
            if (i % 2) nx = 1.0, ny = 0.0;
            Side a, b;
            a.h = H;
            b.h = H * r;
            a.b = kind == 0 ? -H : -H + off;
            if (kind < 2 || kind == 6) b.b = a.h + a.b + 1e-3 * b.h * (U(rng) - 0.5) - b.h;
            if (kind == 2) b.b = a.b;
            if (kind == 3) b.b = a.h + a.b + H * U(rng);
            if (kind == 4) b.b = a.b + H * (1.0 - r) * U(rng);
            if (kind == 5) b.b = a.b, b.h = H * (i % 3 ? 1.0 : 1.0 + 1e-3 * (U(rng) - 0.5));
            const double froude = std::pow(10.0, kind == 5 ? -16.0 + 16.0 * U(rng) : -4.0 + 4.0 * U(rng));
            for (Side* s : {&a, &b}) {
                s->u = froude * std::sqrt(P.g * s->h) * (U(rng) - 0.5);
                s->v = froude * std::sqrt(P.g * s->h) * (U(rng) - 0.5);
            }
            if (i % 5 == 0) std::swap(a, b);
            const double geo[5] = {nx, ny, 1.0, nx, ny};
            fx::FaceFlux f;
            if (fx::face_flux(a, b, geo, T.fx_face, kHMin, f) != fx::kDone) continue;
            ++done;
            const Five<Q> q = hll<Q>(a, b, nx, ny, P.g, P.sqrt_g, P.half_g);
            const Five<double> d = hll<double>(a, b, nx, ny, P.g, P.sqrt_g, P.half_g);
            const int bin = std::min(23, (int)std::fabs(std::log2(a.h / b.h)));
            const Side& s = a.h < b.h ? a : b;
            const Q own = (Q)s.h * ((Q)P.half_g * s.h + (Q)s.u * s.u + (Q)s.v * s.v);
            Score& m = momentum[bin];
            m.add(a.h < b.h ? f.hu_a : f.hu_b, a.h < b.h ? d.xa : d.xb, a.h < b.h ? q.xa : q.xb, own);
            m.add(a.h < b.h ? f.hv_a : f.hv_b, a.h < b.h ? d.ya : d.yb, a.h < b.h ? q.ya : q.yb, own);
            const Q top = std::max(a.b, b.b);
            const Q sa = std::max((Q)a.h + a.b - top, 0.0L), sb = std::max((Q)b.h + b.b - top, 0.0L);
            mass[bin].add(f.h, d.h, q.h,
                          std::max({sa * hypotl(a.u, a.v), sb * hypotl(b.u, b.v),
                                    sqrtl((Q)P.g * std::max(sa, sb)) * fabsl(sa - sb)}));
        }
        bool ok = done > 100000;
        double most[2] = {0.0, 0.0};
        for (int k = 0; k < 24; ++k) {
            ok = ok && mass[k].ok() && momentum[k].ok();
            if (mass[k].n >= 200) most[0] = std::max(most[0], std::sqrt(mass[k].fixed / mass[k].fp64));
            if (mass[k].n >= 200)
                most[1] = std::max(most[1], std::sqrt(momentum[k].fixed / momentum[k].fp64));
        }
        good = good && ok;
        std::printf("%s %s: %ld, rms of FP64's up to %.2f (mass) %.2f (momentum)\n",
                    ok ? "ok" : "FAILED", names[kind], done, most[0], most[1]);
    }
    return good ? 0 : 1;
}
