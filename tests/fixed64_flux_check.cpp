// Holds the fixed-point face flux and wet element sums of
// dgcom_gb300/csrc/fixed64.hpp to long double beside the same formulas in
// FP64, over depths of 1 mm to 1 km, speeds from none to twice the wave's,
// surface jumps from none to a third of the depth, beds equal, stepped and
// above the datum, dry sides, normals along the axes and turned, and orders 1 to 4
// with element scales spread over 2^6.
//
// Both round: FP64 at 2^-53 of each operation's result, fixed point at 2^-57
// of an element's largest term or better. The check asks that fixed point's
// root mean square error is no larger than FP64's, that its largest stays
// below 2^-51 of the terms' size (FP64's own bound for some ten roundings),
// and that a face at rest has no mass flux.
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

constexpr double kHMin = 1e-6;

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
    double worst = 0.0, sq_fixed = 0.0, sq_fp64 = 0.0;
    void add(Q fixed, Q fp64, Q want, Q scale) {
        const double f = (double)(fabsl(fixed - want) / scale);
        const double d = (double)(fabsl(fp64 - want) / scale);
        worst = std::max(worst, f);
        sq_fixed += f * f;
        sq_fp64 += d * d;
    }
    bool ok() const { return sq_fixed <= sq_fp64 && worst <= 0x1p-51; }
};

static long faces(std::mt19937_64& rng, Score& mass, Score& momentum) {
    std::uniform_real_distribution<double> U(0.0, 1.0);
    Physics P{};
    P.g = 9.81;
    P.sqrt_g = std::sqrt(P.g);
    P.half_g = 0.5 * P.g;
    P.two_g = 2.0 * P.g;
    P.h_min = kHMin;
    Operators ops(1);
    DevTables T{};
    std::vector<FxLimb> coef;
    fixed_constants(PairSchedule(ops), P, T, coef);
    long done = 0;
    for (int i = 0; i < 400000; ++i) {
        const double H = std::pow(10.0, -3.0 + 6.0 * U(rng)), turn = 6.283185307179586 * U(rng);
        double nx = std::cos(turn), ny = std::sin(turn);
        if (i % 5 == 0) nx = 1.0, ny = 0.0;
        if (i % 5 == 1) nx = 0.0, ny = -1.0;
        const double speed =
            i % 17 == 0 ? 0.0 : std::pow(10.0, -12.0 + 12.0 * U(rng)) * 4.0 * std::sqrt(P.g * H);
        const double jump = i % 4 == 0 ? 0.0 : std::pow(10.0, -10.0 + 10.0 * U(rng)) * 0.3 * H;
        Side a, b;
        a.b = i % 3 == 0 ? -H + 0.1 * H * U(rng) : (i % 3 == 1 ? 5.0 * U(rng) : -H);
        b.b = i % 2 ? a.b : a.b + 0.2 * H * (U(rng) - 0.5);
        a.h = H;
        b.h = a.b + H + jump - b.b;
        if (i % 11 == 0) {  // a side dry, or dry over a higher bed
            b.b = a.b + H * (0.5 + U(rng));
            b.h = i % 2 ? 0.0 : 1e-4 * H * U(rng);
            if (i % 3 == 0) std::swap(a, b);
        }
        for (double* x : {&a.u, &a.v, &b.u, &b.v}) *x = speed * (U(rng) - 0.5);
        const double geo[5] = {nx, ny, 1.0, nx, ny};
        fx::FaceFlux f;
        if (fx::face_flux(a, b, geo, T.fx_face, kHMin, f) != fx::kDone) continue;
        ++done;
        const Five<Q> q = hll<Q>(a, b, nx, ny, P.g, P.sqrt_g, P.half_g);
        const Five<double> d = hll<double>(a, b, nx, ny, P.g, P.sqrt_g, P.half_g);
        const Q wave = sqrtl((Q)P.g * H) * fabsl(((Q)b.h + b.b) - ((Q)a.h + a.b));
        const Q scale = std::max({(Q)a.h * hypotl(a.u, a.v), (Q)b.h * hypotl(b.u, b.v), wave,
                                  i % 11 == 0 ? sqrtl((Q)P.g * H) * H : 0.0L});
        if (scale > 0.0L) {
            // the surfaces' sums h + B round in FP64, not in fixed point
            mass.sq_fixed += (double)powl((f.h - q.h) / scale, 2);
            mass.sq_fp64 += (double)powl((d.h - q.h) / scale, 2);
        } else if (f.h != 0.0) {
            std::printf("a face at rest: mass flux %g\n", f.h);
            return -1;
        }
        const Q u2 = std::max((Q)a.u * a.u + (Q)a.v * a.v, (Q)b.u * b.u + (Q)b.v * b.v);
        // the pressure of the surface sums h + B, and the momentum carried
        const Q sum = std::max(a.h + std::fabs(a.b), b.h + std::fabs(b.b));
        const Q p = std::max(a.h, b.h) * ((Q)P.half_g * sum + u2);
        momentum.add(f.hu_a, d.xa, q.xa, p);
        momentum.add(f.hv_a, d.ya, q.ya, p);
        momentum.add(f.hu_b, d.xb, q.xb, p);
        momentum.add(f.hv_b, d.yb, q.yb, p);
    }
    return done;
}

// One element of order N: the kernel's sums against the same in T
template <class T>
static void element_sums(const PairSchedule& s, const std::vector<double>& h,
                         const std::vector<double>& hu, const std::vector<double>& hv,
                         const std::vector<double>& u, const std::vector<double>& v,
                         const std::vector<double>& hm, const std::vector<double>& slope,
                         const std::vector<double>& lift, const std::vector<double>& flux,
                         const std::vector<double>& jinv, double two_g, std::vector<T>& out,
                         std::vector<T>& size) {
    const int np = s.n1 - 1, na = 2 * np;
    std::vector<T> f(s.owned.size() * 3);
    for (size_t q = 0; q < s.owned.size(); ++q) {
        const int a = s.owned[q].a, c = s.owned[q].c;
        const T m0 = hm[2 * q], m1 = hm[2 * q + 1];
        const T mass = ((T)hu[a] + hu[c]) * m0 + ((T)hv[a] + hv[c]) * m1;
        const T gp = (T)two_g * h[a] * h[c];
        f[3 * q] = mass;
        f[3 * q + 1] = mass * ((T)u[a] + u[c]) + gp * m0;
        f[3 * q + 2] = mass * ((T)v[a] + v[c]) + gp * m1;
    }
    out.assign(s.nn * 3, 0);
    size.assign(s.nn * 3, 0);
    for (int i = 0; i < s.nn; ++i)
        for (int k = 0; k < 3; ++k) {
            T sum = 0, abs = 0;
            auto take = [&](T x) {
                sum -= x;
                abs = std::max(abs, x < 0 ? -x : x);
            };
            for (int q = 0; q < na; ++q)
                take((k ? (T)0.5 : (T)1) * (T)s.accum_coef[i * na + q] *
                     f[3 * s.accum_slot[i * na + q] + k]);
            if (k) take((T)h[i] * slope[2 * i + k - 1]);
            take((T)lift[i] * flux[3 * i + k]);
            out[3 * i + k] = sum * (T)jinv[i];
            size[3 * i + k] = abs * (T)jinv[i];
        }
}

static long elements(std::mt19937_64& rng, int order, Score& score) {
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const Operators ops(order);
    const PairSchedule s(ops);
    Physics P{};
    P.g = 9.81;
    P.sqrt_g = std::sqrt(P.g);
    P.half_g = 0.5 * P.g;
    P.two_g = 2.0 * P.g;
    DevTables T{};
    std::vector<FxLimb> coef;
    fixed_constants(s, P, T, coef);
    const int nn = s.nn, np = order, na = 2 * np;
    long done = 0;
    for (int round = 0; round < 3000; ++round) {
        const double H = std::pow(10.0, -2.0 + 5.0 * U(rng)), size = std::pow(10.0, 4.0 * U(rng));
        const double speed = round % 7 == 0 ? 0.0 : std::pow(10.0, -8.0 + 8.0 * U(rng)) * 3.0 * std::sqrt(H);
        std::vector<double> h(nn), hu(nn), hv(nn), u(nn), v(nn), slope(2 * nn), lift(nn), flux(3 * nn),
            jinv(nn), hm(s.owned.size() * 2);
        for (int i = 0; i < nn; ++i) {
            h[i] = H * std::exp2(-6.0 * U(rng) * (round % 3 == 0));
            u[i] = speed * (U(rng) - 0.5);
            v[i] = speed * (U(rng) - 0.5);
            hu[i] = h[i] * u[i];
            hv[i] = h[i] * v[i];
            for (int k = 0; k < 2; ++k)
                slope[2 * i + k] = round % 5 == 0 ? 0.0 : P.g * H * size * (U(rng) - 0.5);
            jinv[i] = (0.5 + U(rng)) / (size * size);
            const bool on = i % (order + 1) == 0 || i % (order + 1) == order || i <= order;
            lift[i] = on ? size * order * (order + 1) / 2.0 * (0.5 + U(rng)) : 0.0;
            flux[3 * i] = H * (speed + 0.01 * U(rng)) * (U(rng) - 0.5);
            flux[3 * i + 1] = P.half_g * H * H * (U(rng) - 0.5);
            flux[3 * i + 2] = P.half_g * H * H * (U(rng) - 0.5);
        }
        for (double& m : hm) m = 0.25 * size * (U(rng) - 0.5) * (U(rng) < 0.1 ? 1e-6 : 1.0);
        // as fixed_tables_kernel and stage_kernel take them
        int et = 0, eg = 0, el = 0;
        for (double m : hm) et = std::max(et, fx::expo(m));
        for (double m : slope) eg = std::max(eg, fx::expo(m));
        for (double m : lift) el = std::max(el, fx::expo(m));
        eg = std::max(eg, fx::kExpLo - 400);
        fx::Exps x{0, 4095, 0, 0, 0, 0};
        for (int i = 0; i < nn; ++i) {
            x.h_max = std::max(x.h_max, fx::expo(h[i]));
            x.h_min = std::min(x.h_min, fx::expo(h[i]));
            x.m = std::max({x.m, fx::expo(hu[i]), fx::expo(hv[i])});
            x.v = std::max({x.v, fx::expo(u[i]), fx::expo(v[i])});
            if (lift[i] == 0.0) continue;
            x.fh = std::max(x.fh, fx::expo(flux[3 * i]));
            x.fm = std::max({x.fm, fx::expo(flux[3 * i + 1]), fx::expo(flux[3 * i + 2])});
        }
        const fx::Scale sc =
            fx::scales(x, FxExp{et - 1022, eg - 1022, el - 1022, 1}, T.fx_ec, T.fx_e2g);
        if (!sc.ok) {
            std::printf("order %d, round %d: no scale\n", order, round);
            return -1;
        }
        std::vector<fx::Flux> f(s.owned.size());
        for (int i = 0; i < nn; ++i)
            for (int q = 0; q < np; ++q) {
                const int sl = i * np + q, o = s.owned[sl].a + s.owned[sl].c - i;
                auto sum = [&](const std::vector<double>& y, int K) {
                    return fx::to_fixed(y[i], K) + fx::to_fixed(y[o], K);
                };
                const FxLimb hi = fx::split(fx::to_fixed(h[i], sc.kh));
                f[sl] = fx::pair_flux(fx::two_g_h(hi, T.fx_two_g, sc),
                                      fx::split(fx::to_fixed(h[o], sc.kh)), sum(hu, sc.km),
                                      sum(hv, sc.km), sum(u, sc.ku), sum(v, sc.ku),
                                      fx::split(fx::to_fixed(hm[2 * sl], et + 1)),
                                      fx::split(fx::to_fixed(hm[2 * sl + 1], et + 1)));
            }
        std::vector<Q> want, size_q, unused_q;
        std::vector<double> fp64, unused;
        element_sums<Q>(s, h, hu, hv, u, v, hm, slope, lift, flux, jinv, P.two_g, want, size_q);
        element_sums<double>(s, h, hu, hv, u, v, hm, slope, lift, flux, jinv, P.two_g, fp64, unused);
        Q big[3] = {0, 0, 0};  // the element's largest term of each sum
        for (int i = 0; i < nn; ++i)
            for (int k = 0; k < 3; ++k) big[k] = std::max(big[k], size_q[3 * i + k]);
        for (int i = 0; i < nn; ++i) {
            const FxLimb H1 = fx::split(fx::to_fixed(h[i], sc.kh));
            for (int k = 0; k < 3; ++k) {
                fx::PairSum a = fx::pair_sum();
                for (int q = 0; q < na; ++q) {
                    const fx::Flux& p = f[s.accum_slot[i * na + q]];
                    fx::mac(a, coef[i * na + q], k == 0 ? p.h : (k == 1 ? p.hu : p.hv));
                }
                int64_t sum = -fx::fold(a);
                if (k)
                    sum -= fx::bed_term(H1, fx::split(fx::to_fixed(slope[2 * i + k - 1], eg + 1)), sc);
                fx::Acc l{fx::half<0>(), 0};
                if (lift[i] != 0.0)
                    fx::mac(l, fx::split(fx::to_fixed(lift[i], el + 2)),
                            fx::split(fx::to_fixed(flux[3 * i + k], k ? sc.kfm : sc.kfh)));
                const double got =
                    fx::over_jacobian(sum - fx::fold<0>(l), k ? sc.sm : sc.sh, jinv[i]);
                if (big[k] > 0.0L) score.add(got, fp64[3 * i + k], want[3 * i + k], big[k]);
                else if (got != 0.0) return -1;
            }
        }
        ++done;
    }
    return done;
}

int main() {
    std::mt19937_64 rng(3);
    Score mass, momentum;
    long checks = faces(rng, mass, momentum);
    std::printf("%sfaces %ld: mass rms %.3g of FP64's, momentum %.3g, worst %.3g\n",
                checks > 100000 && mass.ok() && momentum.ok() ? "ok " : "FAILED ", checks,
                std::sqrt(mass.sq_fixed / mass.sq_fp64),
                std::sqrt(momentum.sq_fixed / momentum.sq_fp64), momentum.worst);
    if (checks <= 100000 || !mass.ok() || !momentum.ok()) return 1;
    for (int order = 1; order <= 4; ++order) {
        Score s;
        const long n = elements(rng, order, s);
        std::printf("order %d, %ld elements: rms %.3g of FP64's, worst %.3g\n", order, n,
                    std::sqrt(s.sq_fixed / s.sq_fp64), s.worst);
        if (n <= 0 || !s.ok()) return 1;
    }
    return 0;
}
