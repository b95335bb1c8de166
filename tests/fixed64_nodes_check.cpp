// Holds the wet elements' fixed-point sums (dgcom_gb300/csrc/fixed64.hpp) to
// long double node by node: each node's error over the node's own largest term,
// beside the same formulas in FP64, for the elements that the rules there
// (scales, thin_depth, thin, slow_node, own_mass_small) leave to fixed point.
// Rectangles of orders 1 to 4 at any angle, sides in the ratio 1 to 32, depths
// in the ratio 1 to 512, one deep corner among them, still water, currents of
// Froude numbers from 1e-6 to 2, sheared ones and ones with nodes at rest, and
// the face fluxes and bed slopes that belong to them.
//
// The check asks that at every position of a node the root mean square error
// is no larger than FP64's; that for terms below 2^53 places, next to the lines,
// it is no larger than 1.1 of it; that no error exceeds 2^-50 of the term; and
// that elements of even depth and sides are all left to fixed point.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "host_common.hpp"

using namespace dgswe;
typedef long double Q;

struct Score {
    double fixed = 0.0, fp64 = 0.0, worst = 0.0;
    long n = 0;
    void add(Q got, Q other, Q want, Q own) {
        const double f = (double)(fabsl(got - want) / own), d = (double)(fabsl(other - want) / own);
        fixed += f * f;
        fp64 += d * d;
        worst = std::max(worst, f);
        ++n;
    }
    double ratio() const { return std::sqrt(fixed / fp64); }
};

struct Element {
    std::vector<double> h, hu, hv, u, v, slope, lift, flux, jinv, hm;
};

// The sums in T, and each node's largest term
template <class T>
static void sums(const PairSchedule& s, const Element& x, double two_g, std::vector<T>& out,
                 std::vector<T>& own) {
    const int na = 2 * (s.n1 - 1);
    std::vector<T> f(s.owned.size() * 3);
    for (size_t q = 0; q < s.owned.size(); ++q) {
        const int a = s.owned[q].a, c = s.owned[q].c;
        const T m0 = x.hm[2 * q], m1 = x.hm[2 * q + 1];
        const T mass = ((T)x.hu[a] + x.hu[c]) * m0 + ((T)x.hv[a] + x.hv[c]) * m1;
        const T gp = (T)two_g * x.h[a] * x.h[c];
        f[3 * q] = mass;
        f[3 * q + 1] = mass * ((T)x.u[a] + x.u[c]) + gp * m0;
        f[3 * q + 2] = mass * ((T)x.v[a] + x.v[c]) + gp * m1;
    }
    out.assign(s.nn * 3, 0);
    own.assign(s.nn * 3, 0);
    for (int i = 0; i < s.nn; ++i)
        for (int k = 0; k < 3; ++k) {
            T sum = 0, most = 0;
            auto take = [&](T y) {
                sum -= y;
                most = std::max(most, y < 0 ? -y : y);
            };
            for (int q = 0; q < na; ++q)
                take((k ? (T)0.5 : (T)1) * (T)s.accum_coef[i * na + q] *
                     f[3 * s.accum_slot[i * na + q] + k]);
            if (k) take((T)x.h[i] * x.slope[2 * i + k - 1]);
            take((T)x.lift[i] * x.flux[3 * i + k]);
            out[3 * i + k] = sum * (T)x.jinv[i];
            own[3 * i + k] = most * (T)x.jinv[i];
        }
}

struct Group {
    std::vector<Score> node;  // [position][mass, momentum]
    Score edge[2];            // the last half bit before each line
    long made = 0, taken = 0;
};

static void run(int order, int kind, int rounds, std::mt19937_64& rng, Group& g) {
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
    const int two_g_64ths = (T.fx_two_g.hi >> 24) + 1, two_g_key = fx::key(P.two_g);
    const int n1 = order + 1, nn = s.nn, na = 2 * order;
    g.node.resize((size_t)nn * 2);
    for (int round = 0; round < rounds; ++round) {
        const bool even = kind == 0;
        const double H = std::pow(10.0, -2.0 + 5.0 * U(rng));
        const double depths = std::exp2(even ? 0.26 * U(rng) : 9.0 * U(rng) * U(rng) * U(rng));
        const double sides = std::exp2(even ? 0.0 : 5.0 * U(rng) * U(rng));
        const double dx = std::pow(10.0, 4.0 * U(rng)), dy = dx / sides;
        const double turn = round % 3 ? 6.283185307179586 * U(rng) : 0.0;
        const double c = std::cos(turn), si = std::sin(turn), gx = U(rng), gy = U(rng);
        const double froude = round % 11 == 0 ? 0.0 : std::pow(10.0, -6.0 + (even ? 5.4 : 6.3) * U(rng));
        const double dir = 6.283185307179586 * U(rng), shear = std::exp2(-9.0 * U(rng));
        Element x;
        for (auto* a : {&x.h, &x.hu, &x.hv, &x.u, &x.v, &x.jinv, &x.lift}) a->assign(nn, 0.0);
        x.slope.assign(2 * nn, 0.0);
        x.flux.assign(3 * nn, 0.0);
        std::vector<double> bed(nn);
        const double m[2][2] = {{0.5 * dy * c, 0.5 * dy * si}, {-0.5 * dx * si, 0.5 * dx * c}};
        for (int i = 0; i < nn; ++i) {
            const double r = 0.5 * (ops.x[i % n1] + 1.0), q = 0.5 * (ops.x[i / n1] + 1.0);
            const double w = kind == 2 ? (i == 0 ? 0.0 : 1.0)  // one deep corner
                                       : (gx * r + gy * q) / (gx + gy);
            x.h[i] = H * (1.0 - (1.0 - 1.0 / depths) * w) * (1.0 + 1e-3 * U(rng));
            bed[i] = -x.h[i] + 0.01 * H * U(rng);
            double speed = froude * std::sqrt(P.g * H) * (1.0 + 0.1 * (U(rng) - 0.5));
            double a = dir;
            if (kind == 3) {  // sheared along the rows, nothing across
                speed *= shear + (1.0 - shear) * q;
                a = turn;
            }
            if (kind == 4) speed *= U(rng) < 0.3 ? 0.0 : std::exp2(-8.0 * U(rng));
            x.u[i] = speed * std::cos(a);
            x.v[i] = speed * std::sin(a);
            x.hu[i] = x.h[i] * x.u[i];
            x.hv[i] = x.h[i] * x.v[i];
        }
        for (const PairSlot& p : s.owned)
            for (int k = 0; k < 2; ++k) x.hm.push_back(0.5 * m[(int)p.dir][k]);
        for (int i = 0; i < nn; ++i) {
            const int a = i % n1, j = i / n1;
            for (int k = 0; k < n1; ++k) {
                const double br = ops.d[a * n1 + k] * bed[j * n1 + k];
                const double bs = ops.d[j * n1 + k] * bed[k * n1 + a];
                x.slope[2 * i] += P.g * (br * m[0][0] + bs * m[1][0]);
                x.slope[2 * i + 1] += P.g * (br * m[0][1] + bs * m[1][1]);
            }
            x.jinv[i] = 4.0 / (dx * dy);
            const bool s_face = j == 0 || j == order, on = s_face || a == 0 || a == order;
            if (!on) continue;
            const double out = s_face ? (j ? 1.0 : -1.0) : (a ? 1.0 : -1.0);
            const double length = s_face ? dx : dy;
            const double nx = out * 2.0 * m[s_face][0] / length, ny = out * 2.0 * m[s_face][1] / length;
            x.lift[i] = 0.5 * length * order * (order + 1) / 2.0;
            const double jump = 1e-4 * (U(rng) - 0.5), un = x.u[i] * nx + x.v[i] * ny;
            const double p = P.half_g * x.h[i] * x.h[i] * (1.0 + jump);
            x.flux[3 * i] = x.h[i] * un + (froude > 0.0 ? jump * froude * x.h[i] * std::sqrt(P.g * x.h[i]) : 0.0);
            x.flux[3 * i + 1] = x.h[i] * un * x.u[i] + p * nx;
            x.flux[3 * i + 2] = x.h[i] * un * x.v[i] + p * ny;
        }
        // as fixed_tables_kernel and stage_kernel take them
        int et = 0, eg = 0, el = 0;
        fx::OwnMetric own{0x7FFF, 0x7FFF};
        for (double y : x.hm) et = std::max(et, fx::expo(y));
        for (double y : x.slope) eg = std::max(eg, fx::expo(y));
        for (double y : x.lift) el = std::max(el, fx::expo(y));
        eg = std::max(eg, fx::kExpLo - 400);
        for (int i = 0; i < nn; ++i) {
            const fx::OwnMetric o =
                fx::own_metric(x.hm.data(), &s.accum_slot[i * na], &s.accum_coef[i * na], na);
            own = {std::min(own.w, o.w), std::min(own.v, o.v)};
        }
        const FxExp t{et - 1022, eg - 1022, el - 1022, fx::own_deficits(own, et - 1022, T.fx_ec)};
        fx::Exps e{};
        int deepest = 0;
        e.h_key = e.m_key = 0x7FFF;
        for (int i = 0; i < nn; ++i) {
            deepest = std::max(deepest, fx::key(x.h[i]));
            e.h_key = std::min(e.h_key, fx::key(x.h[i]));
            const double q = std::max(std::fabs(x.hu[i]), std::fabs(x.hv[i]));
            e.m = std::max(e.m, fx::expo(q));
            e.m_key = std::min(e.m_key, fx::key(q));
            e.v = std::max({e.v, fx::expo(x.u[i]), fx::expo(x.v[i])});
            e.fh = std::max(e.fh, fx::expo(x.flux[3 * i]));
            e.fm = std::max({e.fm, fx::expo(x.flux[3 * i + 1]), fx::expo(x.flux[3 * i + 2])});
        }
        e.h_max = deepest >> 4;
        e.h_top = deepest & 15;
        e.h_min = e.h_key >> 4;
        const fx::Scale sc = fx::scales(e, t, T.fx_ec, T.fx_e2g, two_g_64ths);
        ++g.made;
        if (!sc.ok || fx::thin(e, sc, t, two_g_key)) continue;
        std::vector<fx::Flux> f(s.owned.size());
        for (int i = 0; i < nn; ++i)
            for (int q = 0; q < order; ++q) {
                const int sl = i * order + q, o = s.owned[sl].a + s.owned[sl].c - i;
                auto both = [&](const std::vector<double>& y, int K) {
                    return fx::to_fixed(y[i], K) + fx::to_fixed(y[o], K);
                };
                const FxLimb hi = fx::split(fx::to_fixed(x.h[i], sc.kh));
                f[sl] = fx::pair_flux(fx::two_g_h(hi, T.fx_two_g, sc),
                                      fx::split(fx::to_fixed(x.h[o], sc.kh)), both(x.hu, sc.km),
                                      both(x.hv, sc.km), both(x.u, sc.ku), both(x.v, sc.ku),
                                      fx::split(fx::to_fixed(x.hm[2 * sl], et + 1)),
                                      fx::split(fx::to_fixed(x.hm[2 * sl + 1], et + 1)));
            }
        std::vector<int64_t> lifted(3 * nn, 0);
        for (int i = 0; i < 3 * nn; ++i) {
            if (x.lift[i / 3] == 0.0) continue;
            lifted[i] = fx::mul<0>(fx::split(fx::to_fixed(x.lift[i / 3], el + 2)),
                                   fx::split(fx::to_fixed(x.flux[i], i % 3 ? sc.kfm : sc.kfh)));
        }
        const bool slow = fx::slow_node(e, sc, t, T.fx_e2g);
        ++g.taken;
        std::vector<Q> want, own_q;
        std::vector<double> fp64, own_d;
        sums<Q>(s, x, P.two_g, want, own_q);
        sums<double>(s, x, P.two_g, fp64, own_d);
        for (int i = 0; i < nn; ++i) {
            const FxLimb H1 = fx::split(fx::to_fixed(x.h[i], sc.kh));
            bool small = false;  // the node's mass in FP64
            if (slow) {
                int64_t own = 0;
                for (int q = 0; q < na; ++q)
                    fx::own_mass(own, coef[i * na + q], f[s.accum_slot[i * na + q]].h);
                fx::own_mass(own, lifted[3 * i]);
                small = fx::own_mass_small(own);
            }
            for (int k = small ? 1 : 0; k < 3; ++k) {
                fx::PairSum a = fx::pair_sum();
                for (int q = 0; q < na; ++q) {
                    const fx::Flux& p = f[s.accum_slot[i * na + q]];
                    fx::mac(a, coef[i * na + q], k == 0 ? p.h : (k == 1 ? p.hu : p.hv));
                }
                int64_t sum = -fx::fold(a);
                if (k)
                    sum -= fx::bed_term(H1, fx::split(fx::to_fixed(x.slope[2 * i + k - 1], eg + 1)), sc);
                const double got =
                    fx::over_jacobian(sum - lifted[3 * i + k], k ? sc.sm : sc.sh, x.jinv[i]);
                const Q own = own_q[3 * i + k];
                if (own == 0.0L) {
                    if (got != 0.0) g.node[0].worst = 1.0;  // nothing gave something
                    continue;
                }
                g.node[2 * i + (k > 0)].add(got, fp64[3 * i + k], want[3 * i + k], own);
                const double bits = std::log2((double)(own / (Q)x.jinv[i])) + (k ? sc.sm : sc.sh);
                if (bits < 53.0) g.edge[k > 0].add(got, fp64[3 * i + k], want[3 * i + k], own);
            }
        }
    }
}

int main() {
    const char* names[5] = {"even", "sloping", "one deep corner", "sheared", "nodes at rest"};
    bool good = true;
    for (int order = 1; order <= 4; ++order)
        for (int kind = 0; kind < 5; ++kind) {
            std::mt19937_64 rng(100 * order + kind);
            Group g;
            run(order, kind, 8000, rng, g);
            double most[2] = {0.0, 0.0}, worst = 0.0;
            for (size_t q = 0; q < g.node.size(); ++q) {
                most[q % 2] = std::max(most[q % 2], g.node[q].ratio());
                worst = std::max(worst, g.node[q].worst);
            }
            const bool ok = most[0] <= 1.0 && most[1] <= 1.0 && worst <= 0x1p-50 &&
                            (g.edge[0].n < 200 || g.edge[0].ratio() <= 1.1) &&
                            (g.edge[1].n < 200 || g.edge[1].ratio() <= 1.1) &&
                            (kind ? g.taken > 500 : g.taken == g.made);
            good = good && ok;
            std::printf("%s order %d, %s: %ld of %ld, rms of FP64's at a position up to %.2f (mass) "
                        "%.2f (momentum), before the line %.2f (%ld) %.2f (%ld), worst %.2g\n",
                        ok ? "ok" : "FAILED", order, names[kind], g.taken, g.made, most[0], most[1],
                        g.edge[0].ratio(), g.edge[0].n, g.edge[1].ratio(), g.edge[1].n, worst);
        }
    return good ? 0 : 1;
}
