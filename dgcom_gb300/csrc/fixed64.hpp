// 64-bit fixed-point arithmetic on doubles: square roots, reciprocals and
// h^(-4/3), and the sums and products of the flux-differencing volume term.
//
// GB300 takes one FP64 instruction of a warp in 64 cycles of an SM
// sub-partition, one 32×32+64-bit integer multiply-add in 2 (measured: 67.6
// and 2.3 cycles, in parallel on their two pipes), so a product of 62-bit
// integers costs a tenth of an FP64 one and a sum a sixteenth.
//
// The roots: each function takes a
// single-precision seed from the special-function unit, refines it on the
// mantissa as an integer to a relative error below 2^-55 and rounds once to
// the nearest double: at most 0.5 + 2^-2 ulp, where the FP64 sequences these
// replace had up to 1 (sqrt, reciprocal: 5 and 4 FP64 operations) and about
// 3 (h^(-4/3): 8).
//
// Host and device both compile this header; the host (the unit test) takes
// its seeds from the C library's single-precision functions, off by the
// relative error DGSWE_SEED_ERROR.
#pragma once

#include <math.h>
#include <stdint.h>

#include "device.hpp"
#include "fp64_bits.hpp"

#ifndef DGSWE_SEED_ERROR
#define DGSWE_SEED_ERROR 0.0f
#endif

namespace dgswe {
namespace fx {

// ---- seeds: relative error below 2^-21 for arguments in [1, 8) -------------

DG_HD float seed_rcp(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x * (1.0f + DGSWE_SEED_ERROR);
#endif
}

DG_HD float seed_rsqrt(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / sqrtf(x) * (1.0f + DGSWE_SEED_ERROR);
#endif
}

// x^(-1/3)
DG_HD float seed_rcbrt(float x) {
#if defined(__CUDA_ARCH__)
    float l, r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(l * (-1.0f / 3.0f)));
    return r;
#else
    return 1.0f / cbrtf(x) * (1.0f + DGSWE_SEED_ERROR);
#endif
}

DG_HD float as_float(uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float f;
    memcpy(&f, &b, sizeof f);
    return f;
#endif
}

// ---- integers --------------------------------------------------------------

// a·b and a·b + c of 32-bit factors: one multiply-add instruction
DG_HD int64_t mads(int32_t a, int32_t b, int64_t c) { return (int64_t)a * b + c; }
DG_HD uint64_t madu(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }
DG_HD uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
DG_HD uint32_t lo32(uint64_t x) { return (uint32_t)x; }
DG_HD uint64_t umulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
DG_HD int64_t smulhi(int64_t a, int64_t b) {
#if defined(__CUDA_ARCH__)
    return __mul64hi(a, b);
#else
    return (int64_t)(((__int128)a * b) >> 64);
#endif
}

// Leading zeros; 64 for 0
DG_HD int clz64(uint64_t x) {
#if defined(__CUDA_ARCH__)
    return __clzll((long long)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}

constexpr uint64_t kMantissa = 0x000FFFFFFFFFFFFFull, kImplicit = 0x0010000000000000ull;

// Biased exponent field and the mantissa with its implicit bit (2^52..2^53)
DG_HD int expo(double x) { return (int)((uint64_t)fp::bits(x) >> 52) & 0x7FF; }
DG_HD uint64_t mant(double x) { return ((uint64_t)fp::bits(x) & kMantissa) | kImplicit; }
// 2^62·√X from 2^60·X, X in [1, 4): s0 = X·rsqrt(X) to 2^-21 in 31 bits, one
// Newton step to 2^-42 in 47, a second from the exact residual X − s1² (its
// high bits cancel, so arithmetic modulo 2^64 holds it whole) to 2^-60
DG_HD uint64_t root62(uint64_t X) {
    // the float of X, truncated: 24 bits below the leading one
    const uint32_t two = (uint32_t)(X >> 61);  // 1 where X ≥ 2
    const float xf = as_float((uint32_t)((X >> two) >> 37) + 0x3F000000u + (two << 23));
    const uint32_t r = (uint32_t)(seed_rsqrt(xf) * 2147483648.0f);  // 2^31/√X, in [2^30, 2^31]
    // X·2^28 times 2^31/√X → √X·2^59, to 2^30·√X < 2^31
    uint32_t s0 = (uint32_t)(madu(hi32(X), r, 0) >> 29);
    s0 = s0 > 0x7FFFFFFFu ? 0x7FFFFFFFu : s0;
    const int64_t d0 = mads((int32_t)s0, -(int32_t)s0, (int64_t)X);  // 2^60·(X − s0²)
    const int32_t c1 = (int32_t)(mads((int32_t)(d0 >> 12), (int32_t)(r >> 1), 0) >> 33);
    // d0·2^-12 (2^48) · r/2 (2^30) = 2^78; half of it at 2^46 is >> 33
    const uint64_t s1 = ((uint64_t)s0 << 16) + (int64_t)c1;  // 2^46·√X
    const uint32_t l = lo32(s1), h = hi32(s1);
    const uint64_t sq = madu(l, l, 0) + ((uint64_t)(2u * h * l) << 32);  // s1² mod 2^64
    const int64_t d1 = (int64_t)((X << 32) - sq);  // 2^92·(X − s1²), below 2^54 in size
    const int64_t c2 = mads((int32_t)(d1 >> 25), (int32_t)(r >> 1), 0) >> 36;
    // d1·2^-25 (2^67) · r/2 (2^30) = 2^97; half of it at 2^62 is >> 36
    return (s1 << 16) + (uint64_t)c2;
}

// √x for x in [2^-126, 2^127) (the caller's guard)
DG_HD double sqrt_pos(double x) {
    const int e = expo(x);
    const int odd = (e & 1) ^ 1;  // 1023 is odd: an even field is an odd power of two
    const uint64_t s = root62(mant(x) << (8 + odd));
    const uint64_t q = (s + 512u) >> 10;  // rounded to 53 bits (2^52..2^53)
    // exponent field of √x: 1023 + k, k = (e − 1023 − odd)/2
    return fp::from_bits((int64_t)(q + ((uint64_t)((e - 1023 - odd) / 2 + 1022) << 52)));
}

// 2^61/Y in (2^60, 2^61] from 2^63·Y, Y in [1, 2): r0 to 2^-22, then
// r0·(1 + e + e²) with e = 1 − Y·r0 (relative error e³ = 2^-63)
DG_HD uint64_t reciprocal61(uint64_t Y) {
    const float yf = as_float((uint32_t)((Y >> 40) & 0x7FFFFFu) | 0x3F800000u);
    const uint32_t r = (uint32_t)(seed_rcp(yf) * 2147483648.0f);  // [2^30, 2^31]
    // 2^62·Y·r0
    const uint64_t p = madu(hi32(Y), r, hi32(madu(lo32(Y), r, 0)));
    const int64_t e1 = (int64_t)((1ull << 62) - p);  // 2^62·e, |e| < 2^-20
    const int32_t es = (int32_t)(e1 >> 12);          // 2^50·e
    const int64_t e2 = e1 + (mads(es, es, 0) >> 38);  // 2^62·(e + e²), below 2^42 in size
    // r0·(e + e²): 2^62 · 2^31 / 2^32; the high word times r in a signed
    // product of r's half, twice, and its odd bit
    const int32_t eh = (int32_t)(e2 >> 32);
    const int64_t c = mads(eh, (int32_t)(r >> 1), 0) * 2 + ((r & 1) ? eh : 0) +
                      (int64_t)hi32(madu(lo32((uint64_t)e2), r, 0));
    return ((uint64_t)r << 30) + (uint64_t)c;
}

// 1/y for y in [2^-125, 2^125) (the caller's guard)
DG_HD double rcp_pos(double y) {
    const uint64_t q = reciprocal61(mant(y) << 11);
    const uint64_t rounded = (q + 128u) >> 8;  // (2^52, 2^53]
    // 1/y = (1/Y)·2^(1023 − e), 1/Y in (½, 1]
    return fp::from_bits((int64_t)(rounded + ((uint64_t)(2044 - expo(y)) << 52)));
}

// h^(-4/3) for h in [2^-125, 2^125) (the caller's guard): with m = h·8^-k
// in [1, 8) and z = m^(-1/3) to 2^-21, e = 1 − m·z³ and
// m^(-4/3) = z⁴·(1 − e)^(-4/3) = z⁴·(1 + 4/3·(e + 7/6·e²) + …), the next
// term 140/81·e³ below 2^-58
DG_HD double pow_m43(double h) {
    const uint64_t mm = mant(h);
    const int e = expo(h);
    // e − 1023 = 3k + j, j = 0..2; e + 1 = 3·(k + 341) + 1 + j + …: shifted to
    // a positive number, e − 1023 + 1026 = e + 3
    const uint32_t k3 = (uint32_t)(e + 3) / 3u;  // k + 342
    const uint32_t j = (uint32_t)(e + 3) - 3u * k3;
    const uint64_t m = mm << (8 + j);  // 2^60·m, m in [1, 8)
    const float mf = as_float((uint32_t)(mm >> 29) + 0x3F000000u + (j << 23));
    const float zf = seed_rcbrt(mf);
    uint32_t z = (uint32_t)(zf * 2147483648.0f);  // 2^31·z, z in [½, 1]
    const uint64_t z2 = madu(z, z, 0);            // 2^62·z²
    const uint64_t z3 = madu(hi32(z2), z, hi32(madu(lo32(z2), z, 0)));  // 2^61·z³
    // 2^58·m·z³: 2^61 · (2^61·m) / 2^64
    const int64_t ee = (int64_t)((1ull << 58) - umulhi(z3, m << 1));  // 2^58·e, |e| < 2^-18
    const int32_t es = (int32_t)(ee >> 10);                           // 2^48·e, < 2^30
    const int32_t e2 = (int32_t)(mads(es, es, 0) >> 38);              // 2^58·e², < 2^22
    const int64_t q = ee + (mads(e2, 1252698795, 0) >> 30);           // e + 7/6·e²
    const int64_t p = q + q / 3;                                      // 4/3 of it
    const uint64_t z4 = umulhi(z2, z2) << 2;                          // 2^62·z⁴
    const uint64_t w = z4 + (uint64_t)(smulhi((int64_t)z4, p << 22) >> 16);
    // z⁴ (2^62) · p·2^22 (2^80) / 2^64 = 2^78; >> 16 for 2^62
    // w in (2^58, 2^62]: normalise (0..4 bits) and round to 53
    const int c = clz64(w);
    const uint64_t n = w << c;  // top bit 63
    const uint64_t rounded = (n >> 11) + ((n >> 10) & 1);
    // n·2^-63 in [1, 2): w·2^-62 = n·2^(-62 − c), so the exponent of
    // m^(-4/3) is 1 − c, of the result 1 − c − 4k, k = k3 − 342
    const int field = 1023 + 1 - c - 4 * ((int)k3 - 342);
    return fp::from_bits((int64_t)(rounded + ((uint64_t)(field - 1) << 52)));
}

// Right shifts, everything out from 64 on (the instruction's own rule)
DG_HD uint64_t shr_u(uint64_t v, int n) {
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
#else
    return n > 63 ? 0 : v >> n;
#endif
}
DG_HD int64_t shr(int64_t v, int n) {
#if defined(__CUDA_ARCH__)
    int64_t r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
#else
    return v >> (n > 63 ? 63 : n);
#endif
}

// ---- fixed-point numbers ----------------------------------------------------
//
// A number is an int64 whose scale (the power of two it is multiplied by) is
// known from the quantities' largest exponents; a double is cut to it
// exactly where its last bit fits, else towards zero. Products take the two
// 32-bit limbs, the low one signed, so that three multiply-adds give the
// high 64 of the 128 bits: the low × low part, at most a quarter of the last
// place, is left out.

using Lim = FxLimb;  // hi·2^32 + lo

DG_HD Lim split(int64_t v) {
    const uint32_t lo = (uint32_t)v;
    return {(int32_t)lo, (int32_t)((uint32_t)((uint64_t)v >> 32) + (lo >> 31))};
}

// A sum of products: r counts 2^64, t 2^32
struct Acc {
    int64_t t, r;
};

DG_HD void mac(Acc& s, const Lim& a, const Lim& b) {
    s.t = mads(a.hi, b.lo, s.t);
    s.t = mads(a.lo, b.hi, s.t);
    s.r = mads(a.hi, b.hi, s.r);
}

// The sum divided by 2^(64 − K), rounded: an accumulator starts at
// {half<K>(), 0}
template <int K>
DG_HD constexpr int64_t half() {
    return 1ll << (31 - K);
}
template <int K>
DG_HD int64_t fold(const Acc& s) {
    return (int64_t)((uint64_t)s.r << K) + (s.t >> (32 - K));
}

// A node's sum over its pairs, whose terms lie well below the accumulator's
// range: with the low × low parts, a quarter of each (l counts 4)
struct PairSum {
    Acc s;
    int64_t l;
};
DG_HD PairSum pair_sum() { return {{half<4>(), 0}, 0}; }
DG_HD void mac(PairSum& p, const Lim& coef, const Lim& f) {
    mac(p.s, coef, f);
    p.l = mads(coef.lo >> 2, f.lo, p.l);
}
DG_HD int64_t fold(const PairSum& p) {
    return fold<4>(Acc{p.s.t + (p.l >> 30), p.s.r});
}

// x·2^(1085 − K), towards zero: |x| < 2^(K − 1023), so the result is below
// 2^62. Subnormal x count as zero (K is far above their exponent).
DG_HD int64_t to_fixed_nn(double x, int K) {  // x ≥ +0
    return (int64_t)shr_u(mant(x) << 10, K - expo(x));
}
DG_HD int64_t to_fixed(double x, int K) {
    const int64_t v = to_fixed_nn(x, K);
    const int64_t sign = fp::bits(x) >> 63;
    return (v ^ sign) - sign;
}

// v·2^-s rounded to the nearest double, for results in the normal range
DG_HD double from_fixed(int64_t v, int s) {
    const int64_t sign = v >> 63;
    const uint64_t a = (uint64_t)((v ^ sign) - sign);
    if (a == 0) return 0.0;
    const int c = clz64(a);
    const uint64_t m = a << c;
    const uint64_t q = (m >> 11) + ((m >> 10) & 1);
    const uint64_t bits = q + ((uint64_t)(1085 - c - s) << 52);
    return fp::from_bits((int64_t)(bits | ((uint64_t)sign & 0x8000000000000000ull)));
}

// Products of two numbers
template <int K>
DG_HD int64_t mul(const Lim& a, const Lim& b) {
    Acc s{half<K>(), 0};
    mac(s, a, b);
    return fold<K>(s);
}

// x/y for normal x and y > 0 whose exponents lie within 2^±400 (the caller's
// guard): x's mantissa times 1/y to 2^-59, rounded once
DG_HD double div_pos(double x, double y) {
    const uint64_t r = reciprocal61(mant(y) << 11);
    const int64_t q = mul<3>(split((int64_t)(mant(x) << 9)), split((int64_t)r));  // 2^61·
    const double v = from_fixed(q, 61 - expo(x) + expo(y));
    return fp::bits(x) < 0 ? fp::neg(v) : v;
}

// from_fixed by the conversion instruction, which runs on the FP64 pipe
DG_HD double convert(int64_t v, int s) {
#if defined(__CUDA_ARCH__)
    const double x = __ll2double_rn(v);
    return v ? fp::from_bits(fp::bits(x) - ((int64_t)s << 52)) : 0.0;
#else
    return from_fixed(v, s);
#endif
}

// ---- the wet element's right-hand side --------------------------------------
//
// Volume pairs, bed slope, surface lift and 1/J of a wet element, the FP64
// sums' terms in fixed point with one scale per element and quantity. Where
// the exponents go (E of a quantity: |x| < 2^E over the element):
//   h          2^(62 − eh)       exact: the element's depths lie within 2^9
//   hu, hv     2^(60 − em)       (u, v at 2^(61 − ev)); exact down to 2^-8
//   pair metric 2^(62 − et), bed slope 2^(62 − eg), lift 2^(61 − el)
//   mass flux of a pair 2^(58 − em − et), its momentum flux 2^(59 − eP − et),
//   eP covering 2g·h² and the advected momentum, whichever is larger
// Every sum stays below 2^63. Its last place is one for all of an element's
// nodes, where FP64 rounds each node's operations at 2^-53 of their own
// results: where a node's own terms are so small beside the element's that FP64
// would be closer (thin_depth, thin and own_mass_small below), it is FP64 that
// takes them.

struct Exps {  // biased exponent fields over an element; 0: all zero
    int h_max, h_min, m, v, fh, fm;  // depth, momentum, velocity, face fluxes
    int h_top = 15;                  // the deepest node's four bits after the leading one
    int h_key = 0, m_key = 0;        // the smallest node's depth and momentum as key() has them
};

struct Scale {
    bool ok;
    int eP, em;
    int kh, km, ku;   // to_fixed's K of h, of hu and hv, of u and v
    int g_shift;      // of 2g·h, and of the bed slope's products
    int b_shift;
    int kfh, kfm;     // K of the face fluxes
    int sh, sm;       // the sums are values times 2^sh (mass), 2^sm (momentum)
};

// exponent fields within 2^±120 (beyond it the element takes FP64)
constexpr int kExpLo = 1023 - 120, kExpHi = 1023 + 120;

// The sign, the exponent field and four bits of the mantissa: for x > 0 a
// lower bound of 16·(log2 x + 1023), at most 2.4 below it
DG_HD int key(double x) { return (int)((uint64_t)fp::bits(x) >> 48); }
constexpr int kKeyOne = 16 * 1023;

// The least e with 2g·h² < 2^e by the deepest node's leading bits (top of the
// 64ths above 2g·2^-e2g): e2g + 2·eh, or up to two less
DG_HD int pressure_exponent(int h_max, int h_top, int e2g, int two_g_64ths) {
    const unsigned x = 17u + (unsigned)h_top;  // h < x·2^(eh − 5)
    const unsigned p = x * x * (unsigned)two_g_64ths;  // 2g·h² < p·2^(e2g + 2·eh − 16)
    return e2g + 2 * (h_max - 1022) + (int)(p > 16384u) + (int)(p > 32768u) +
           (int)(p > 65536u) - 2;
}

DG_HD Scale scales(const Exps& x, const FxExp& t, int ec, int e2g, int two_g_64ths = 64) {
    Scale s;
    s.ok = t.ok && x.h_max <= kExpHi && x.h_max >= kExpLo && x.h_min >= x.h_max - 9 &&
           x.m <= kExpHi && (x.m == 0 || x.m >= kExpLo) && x.v <= kExpHi && x.fh <= kExpHi &&
           x.fm <= kExpHi;
    const int eh = x.h_max - 1022;
    const int lift = t.el - t.et - ec - 1022;
    int em = (x.m > kExpLo ? x.m : kExpLo) - 1022;
    if (x.fh && em < x.fh + lift + 1) em = x.fh + lift + 1;
    int eP = pressure_exponent(x.h_max, x.h_top, e2g, two_g_64ths);
    if (x.v && eP < em + x.v - 1022 + 3) eP = em + x.v - 1022 + 3;
    if (x.fm && eP < x.fm + lift + 3) eP = x.fm + lift + 3;
    const int steep = t.eg + eh + 1 - t.et - ec;
    if (eP < steep) eP = steep;
    s.eP = eP;
    s.em = em;
    s.kh = 1023 + eh;
    s.km = 1025 + em;
    s.ku = 1021 + eP - em;
    s.g_shift = eP - e2g - 2 * eh;
    s.b_shift = eP - steep;
    s.sh = 60 - em - t.et - ec;
    s.sm = 62 - eP - t.et - ec;
    s.kfh = 1082 - s.sh - t.el;
    s.kfm = 1082 - s.sm - t.el;
    return s;
}

// Whether FP64 is closer to an element's nodes than these sums. Fixed point
// rounds a node's sum at its last place, FP64 at 2^-53 of the node's largest
// term, so the line is drawn at how many of these places that term has: over
// elements of orders 1 to 4 with depths in the ratio 1 to 512, sides in the
// ratio 1 to 32, sheared and still currents (tests/fixed64_nodes_check.cpp) the
// root mean square error against extended precision passes FP64's at 2^52 to
// 2^52.3 places and halves with each further bit. A lower bound of the term
// stands for it, in sixteenths of its log2, and metrics that are made with the
// tables (FxExp::ok):
//  - momentum: the pressure of the shallowest node with itself, 2g·h_min²·W, W
//    the smallest over the nodes and both components of the largest
//    ½|coefficient·metric|;
//  - mass: twice the slowest node's momentum across its lines, 4·m_min·V, V the
//    least over the nodes and the directions of a current. The bound is far
//    below the term where a few nodes are at rest among moving ones, so where it
//    fails each node looks at its fluxes themselves (own_mass_small).
// An element whose momentum is too close takes FP64 whole, a node whose mass is
// takes that alone.
// Elements of even depth have 53.3 bits or more on the meshes here, so that
// depths in the ratio 1.3 (order 4, the least favourable scale) to 2 still stay.
constexpr int kMomentumBits = 16 * 52 + 4, kMassBits = 16 * 52 + 8;

// How much smaller than 2^(et + ec) W and V are, a half word each: FxExp::ok of
// a usable element (not 0)
struct OwnMetric {
    int w, v;  // the keys of a node's, then of an element's
};
DG_HD OwnMetric own_metric(const double* hm, const int32_t* slots, const double* coefs, int na) {
    double w0 = 0.0, w1 = 0.0, a0 = 0.0, a1 = 0.0, size = 0.0;  // a: the largest
    for (int q = 0; q < na; ++q) {
        const double c = 0.5 * fabs(coefs[q]);
        const double x = c * hm[2 * slots[q]], y = c * hm[2 * slots[q] + 1];
        w0 = fmax(w0, fabs(x));
        w1 = fmax(w1, fabs(y));
        if (fabs(x) + fabs(y) > size) {
            size = fabs(x) + fabs(y);
            a0 = x;
            a1 = y;
        }
    }
    // a current lies along at most one of two lines: with the pair that is most
    // across the largest, |a × b|/(|a| + |b|) of it is across one or the other
    double across = 0.0, both = 1.0;
    for (int q = 0; q < na; ++q) {
        const double c = 0.5 * fabs(coefs[q]);
        const double x = c * hm[2 * slots[q]], y = c * hm[2 * slots[q] + 1];
        const double cross = fabs(a0 * y - a1 * x);
        if (cross > across) {
            across = cross;
            both = size + fabs(x) + fabs(y);
        }
    }
    return {key(fmin(w0, w1)), key(across / both)};
}
DG_HD int own_deficits(const OwnMetric& m, int et, int ec) {
    int w = 16 * (et + ec) - (m.w - kKeyOne), v = 16 * (et + ec) - (m.v - kKeyOne);
    w = w < 0 ? 0 : (w > 0x7FFE ? 0x7FFE : w);
    v = v < 0 ? 0 : (v > 0x7FFF ? 0x7FFF : v);
    return (v << 16) | (w + 1);
}

DG_HD bool thin_at(int eP, int h_key, const FxExp& t, int two_g_key) {
    return 16 * (62 - eP) + (two_g_key - kKeyOne) + 2 * (h_key - kKeyOne) -
               ((t.ok & 0x7FFF) - 1) < kMomentumBits;
}

// By the depths alone, which are known before the face fluxes
DG_HD bool thin_depth(const Exps& x, const FxExp& t, int e2g, int two_g_64ths, int two_g_key) {
    return thin_at(pressure_exponent(x.h_max, x.h_top, e2g, two_g_64ths), x.h_key, t, two_g_key);
}

// By all that goes into the scale
DG_HD bool thin(const Exps& x, const Scale& s, const FxExp& t, int two_g_key) {
    return thin_at(s.eP, x.h_key, t, two_g_key);
}

// Whether the mass fluxes have to be looked at. Not in water at rest, where the
// element's momentum and face fluxes stay below 2^-48·h·√(gh): the momentum is
// what the pressure's rounding left there (2^-53 of it a stage), and the sums'
// last place is 2^-55 of the depth's in a step. (A 1 M-quad box's first steps
// from rest took 7.33 ms each with every such element looked at, 6.03 without.)
DG_HD bool slow_node(const Exps& x, const Scale& s, const FxExp& t, int e2g) {
    return (x.m | x.fh) != 0 && 2 * s.em > 3 * (x.h_max - 1022) + e2g - 97 &&
           16 * (62 - s.em) + (x.m_key - kKeyOne) - (t.ok >> 16) < kMassBits;
}

// A node's largest mass term so far (in 2^4 places of its sum), from a pair's
// coefficient and flux, and from a lifted face flux
DG_HD void own_mass(int64_t& own, const Lim& coef, const Lim& f) {
    const int64_t p = mads(coef.hi, f.hi, 0);
    const int64_t a = (p < 0 ? -p : p) | ((f.lo | f.hi) != 0);
    own = own > a ? own : a;
}
DG_HD void own_mass(int64_t& own, int64_t lifted) {
    const int64_t v = lifted < 0 ? -lifted : lifted;
    const int64_t a = (v >> 4) | (v != 0);
    own = own > a ? own : a;
}
// too small, unless the node has no flux at all
DG_HD bool own_mass_small(int64_t own) {
    return own != 0 && own < 398000000000000ll;  // 2^48.5
}

// 2g·h at 2^(62 − eP + eh), below 2^63, from h and 2g (two_g: at 2^(62 − e2g))
DG_HD Lim two_g_h(const Lim& H, const Lim& two_g, const Scale& s) {
    Acc a{half<2>(), 0};
    mac(a, H, two_g);
    const int64_t v = fold<2>(a);
    const int up = s.g_shift < 0 ? -s.g_shift : 0;
    return split(shr((int64_t)((uint64_t)v << up), s.g_shift + up));
}

struct Flux {
    Lim h, hu, hv;
};

// The two-point flux of a pair along its half metric (m0, m1), twice for the
// momentum: mass = Σhu·m0 + Σhv·m1, mass·Σu + 2g·h_a·h_c·m0, …; the sums of
// momentum and velocity over the two nodes
DG_HD Flux pair_flux(const Lim& G, const Lim& H, int64_t M0, int64_t M1, int64_t U0, int64_t U1,
                     const Lim& m0, const Lim& m1) {
    Flux f;
    Acc a{half<0>(), 0};
    mac(a, split(M0), m0);
    mac(a, split(M1), m1);
    f.h = split(fold<0>(a));
    Acc p{half<0>(), 0};
    mac(p, G, H);
    const Lim gp = split(fold<0>(p));
    Acc b{half<1>(), 0};
    mac(b, f.h, split(U0));
    mac(b, gp, m0);
    f.hu = split(fold<1>(b));
    Acc c{half<1>(), 0};
    mac(c, f.h, split(U1));
    mac(c, gp, m1);
    f.hv = split(fold<1>(c));
    return f;
}

// h times the bed slope at the momentum sums' scale
DG_HD int64_t bed_term(const Lim& H, const Lim& slope, const Scale& s) {
    Acc a{half<1>(), 0};
    mac(a, H, slope);
    return shr(fold<1>(a), s.b_shift);
}

// V·2^-s/J as a double
DG_HD double over_jacobian(int64_t V, int s, double jinv) {
    Acc a{half<1>(), 0};
    mac(a, split(V), split((int64_t)(mant(jinv) << 9)));
    return convert(fold<1>(a), s + 1021 - expo(jinv));
}

// ---- the flux between two sides ----------------------------------------------
//
// hydro_hll (point.cuh) with at least one reconstructed side wet, each
// quantity at a scale of the face node's own exponents (E: |x| < 2^E):
//   surface sums 2^(62 − eL) (eL: depths and beds), reconstructed depths
//   2^(62 − es), velocities 2^(60 − ev) and 2^(62 − ev), speeds of waves
//   2^(60 − eS), momenta 2^(60 − es − ev), mass flux 2^(58 − eM), momentum flux
//   2^(59 − eQ), weights 2^62.
// With S_L and S_R the wave speeds held to S_L ≤ 0 ≤ S_R, α = S_R/(S_R − S_L),
// β = 1 − α and w = −α·S_L, the flux is
//   α·F_l + β·F_r − w·(q_r − q_l),
// the star flux in sub-critical flow and one side's (α or β = 1, w = 0)
// otherwise. The differences of depths in it are exact, so that a face at
// rest has no mass flux; eM follows the depths' difference, not their size.
// The integer pipe that shifts and selects is the bound, so the scales are
// such that most products end at theirs (fold<0>, one shift), and the results
// become doubles on the idle FP64 pipe.

using FaceConstants = FxFaceConstants;

struct FaceFlux {
    double h, hu_a, hv_a, hu_b, hv_b;  // seen along the normal from both sides
};

DG_HD int64_t min64(int64_t a, int64_t b) { return a < b ? a : b; }
DG_HD int64_t max64(int64_t a, int64_t b) { return a > b ? a : b; }
DG_HD int imax(int a, int b) { return a > b ? a : b; }
DG_HD int imin(int a, int b) { return a < b ? a : b; }
DG_HD int64_t shl(int64_t v, int n) { return (int64_t)((uint64_t)v << n); }
DG_HD int64_t abs64(int64_t v) { return v < 0 ? -v : v; }

// √(g·x) at 2^(58 − eC) for 0 ≤ x at 2^s (below 2^62), √(g·x) < 2^eC
DG_HD int64_t celerity(int64_t x, int s, const FaceConstants& c, int eC) {
    int up = clz64((uint64_t)x) - 2;     // x·2^up in [2^61, 2^62)
    up -= (60 - up - s) & 1;             // one less where that makes the exponent even
    const uint64_t X = up >= 0 ? (uint64_t)x << up : (uint64_t)x >> 1;
    const int p = 60 - up - s;           // x's value is X·2^(p − 60)
    const int64_t v = mul<0>(split((int64_t)(root62(x ? X : 1ull << 60) >> 1)), c.sqrt_g);
    return x ? shr(v, 1 - c.e_sqrt_g - p / 2 + eC) : 0;
}

// a/(a + b) at 2^62 for 0 ≤ a, b < 2^61, not both 0
DG_HD int64_t share(int64_t a, int64_t b) {
    const uint64_t d = (uint64_t)(a + b);
    const int up = clz64(d) - 2;  // (a + b)·2^up in [2^61, 2^62)
    const uint64_t q = reciprocal61(d << (up + 2));
    return mul<4>(split(shl(a, up)), split((int64_t)q));
}

// The flux along the vector m = |m|·n (geo: m, |m|, n) as seen from both
// sides. The rotations into the normal and back, 17 operations, and the
// conversions of the results run on the FP64 pipe, which is idle here.
// Nothing is written where both reconstructed sides are dry (kBothDry, but
// for two sides without any water) or the exponents are out of range
// (kNoScale).
enum FaceCase { kNoScale = 0, kDone = 1, kBothDry = 2 };

template <class Side>
DG_HD FaceCase face_flux(const Side& qa, const Side& qb, const double* geo,
                         const FaceConstants& c, double h_min, FaceFlux& out) {
    const int xa = (int)((uint64_t)fp::bits(qa.h) >> 52), xb = (int)((uint64_t)fp::bits(qb.h) >> 52);
    const int xh = imax(xa, xb);
    if (xh == 0) {  // depths of +0 or subnormal
        out = {0.0, 0.0, 0.0, 0.0, 0.0};
        return fp::bits(qa.h) == 0 && fp::bits(qb.h) == 0 ? kDone : kNoScale;
    }
    const int xl = imax(xh, imax(expo(qa.b), expo(qb.b)));
    auto rotate = [&](const Side& q, double& normal, double& along) {
        const bool moves = fp::gt(q.h, h_min);
        const double u = moves ? q.u : 0.0, v = moves ? q.v : 0.0;
        normal = fma(u, geo[3], v * geo[4]);
        along = fma(v, geo[3], fp::neg(u) * geo[4]);
    };
    double na, ta, nb, tb;
    rotate(qa, na, ta);
    rotate(qb, nb, tb);
    const int xv = imax(imax(expo(na), expo(ta)), imax(expo(nb), expo(tb)));
    // within 2^±120 (a negative depth's sign field is above), h_min not above
    // everything
    if (imax(xv, xl) > kExpHi || xh < kExpLo || expo(h_min) > xl) return kNoScale;
    const int eL = xl - 1022;
    // hydrostatic reconstruction: the depths less the step up to the higher bed
    const int64_t la = to_fixed_nn(qa.h, xl + 1), lb = to_fixed_nn(qb.h, xl + 1);
    const int64_t ba = to_fixed(qa.b, xl + 1), bb = to_fixed(qb.b, xl + 1);
    const int64_t top = max64(ba, bb);
    const int64_t ra = max64(la + (ba - top), 0), rb = max64(lb + (bb - top), 0);
    const int64_t dry = to_fixed_nn(h_min, xl + 1);
    const bool wet_a = ra > dry, wet_b = rb > dry;
    if (!wet_a && !wet_b) return kBothDry;
    const int es = 2 + eL - clz64((uint64_t)(ra | rb));
    const int eC = (es + c.e_g + 1) >> 1;
    const int ev = imax(xv - 1022, -120);
    if (es < -60 || ev > eC + 30) return kNoScale;
    // films left of much deeper water by a step, their surface within 2^-9 of the
    // datum: FP64's sums h + B round at the surface, these at 2^-62 of the deep
    // side (at 2^-6 instead of 2^-8 and 2^-9, some lane of most shore elements
    // took FP64: a 90,000-quad box's stage at N = 1 44 us, not 40)
    if (ba != bb && es < eL - 8 && (max64(abs64(la + ba), abs64(lb + bb)) >> 53) == 0)
        return kNoScale;
    const int64_t sa = shl(ra, eL - es), sb = shl(rb, eL - es);
    const int kv = 1025 + ev;
    const int64_t un_a = to_fixed(na, kv), ut_a = to_fixed(ta, kv);  // 2^(60 − ev)
    const int64_t un_b = to_fixed(nb, kv), ut_b = to_fixed(tb, kv);
    // wave speeds (Einfeldt; beside a dry side, the front's)
    const int64_t c_a = celerity(sa, 62 - es, c, eC), c_b = celerity(sb, 62 - es, c, eC);
    const int64_t c_m = celerity((sa >> 1) + (sb >> 1), 62 - es, c, eC);
    const int64_t va = wet_a ? un_a : 0, vb = wet_b ? un_b : 0;
    const int64_t u_m = vb + mul<2>(split(share(c_a, c_b)), split(va - vb));
    const int eS = imax(ev, eC) + 2;
    const int dv = eS - ev, dc = eS - eC - 2;  // dc at most 30
    const int64_t wa = c_a >> dc, wb = c_b >> dc, wm = c_m >> dc;
    const int64_t xl_ = shr(va, dv), xr_ = shr(vb, dv), xm = shr(u_m, dv);
    const int64_t s_l = min64(wet_a ? min64(xl_ - wa, xm - wm) : xr_ - 2 * wb, 0);
    const int64_t s_r = max64(wet_b ? max64(xr_ + wb, xm + wm) : xl_ + 2 * wa, 0);
    if (s_l == s_r) return kNoScale;
    const int64_t alpha = share(s_r, -s_l);
    const Lim al = split(alpha), be = split((1ll << 62) - alpha);
    const Lim w = split(mul<4>(al, split(-s_l)));  // 2^(62 − eS), below 2^61
    // momenta hs·un, hs·ut; a dry side carries none in its own flux
    const Lim da = split(sa), db = split(sb);
    const Lim ul = split(shl(un_a, 2)), ur = split(shl(un_b, 2));  // 2^(62 − ev)
    const int64_t m_a = mul<0>(da, ul), m_b = mul<0>(db, ur);
    const Lim tl = split(shl(ut_a, 2)), tr = split(shl(ut_b, 2));
    const int64_t t_a = mul<0>(da, tl), t_b = mul<0>(db, tr);
    const Lim ml = split(wet_a ? m_a : 0), mr = split(wet_b ? m_b : 0);
    // mass
    const int64_t dh = sb - sa;
    const int grow = clz64((uint64_t)abs64(dh)) - 2;  // dh·2^grow below 2^62
    const int eD = dh ? es - grow : es - 300;
    const int eM = imax(es + ev + 1, eS + eD);
    Acc f{half<0>(), 0};
    mac(f, al, ml);
    mac(f, be, mr);
    const int64_t f_h = shr(fold<0>(f), eM - es - ev) -
                        shr(mul<0>(w, split(shl(dh, grow))), 2 + eM - eS - eD);
    out.h = geo[2] * convert(f_h, 58 - eM);
    // momentum
    const int eQ = imax(imax(2 * es + c.e_half_g + 1, es + 2 * ev + 1), eS + es + ev);
    const int dp = eQ - 2 * es - c.e_half_g, dm = eQ - es - 2 * ev, dw = eQ - eS - es - ev;
    auto pressure = [&](int64_t x) {  // ½g·x² of a depth at 2^(62 − es)
        const Lim l = split(x);
        return shr(mul<1>(split(mul<0>(l, l)), c.half_g), dp);
    };
    Acc g{half<2>(), 0};
    mac(g, al, split(pressure(sa) + shr(mul<1>(ml, ul), dm)));
    mac(g, be, split(pressure(sb) + shr(mul<1>(mr, ur), dm)));
    const double f_n = convert(fold<2>(g) - shr(mul<1>(w, split(m_b - m_a)), dw), 59 - eQ);
    Acc t{half<2>(), 0};
    mac(t, al, split(shr(mul<1>(ml, tl), dm)));
    mac(t, be, split(shr(mul<1>(mr, tr), dm)));
    const double f_t = convert(fold<2>(t) - shr(mul<1>(w, split(t_b - t_a)), dw), 59 - eQ);
    const double along_x = f_t * geo[1], along_y = f_t * geo[0];
    out.hu_a = out.hu_b = fma(f_n, geo[0], fp::neg(along_x));
    out.hv_a = out.hv_b = fma(f_n, geo[1], along_y);
    // Each side's own pressure over the reconstructed one, ½g(h − hs)(h + hs):
    // none over one bed, where the depth reaches its last place in the surface
    // sums; else at the side's own scale, which a step of the bed sets far from
    // the other's, and added in FP64.
    if (ba == bb && imin(xa, xb) >= xl - 9) return kDone;
    auto own = [&](const Side& q, int x, int64_t s) {
        const int e = x - 1022;
        const int64_t hq = x ? (int64_t)(mant(q.h) << 9) : 0;  // at 2^(62 − e)
        const int64_t gq = shl(s, imin(eL - e, 63)), d = hq - gq;
        const int up = clz64((uint64_t)d) - 2;
        const int64_t p = mul<2>(split(mul<2>(split(shl(d, up)), split((hq >> 1) + (gq >> 1)))),
                                 c.half_g);
        return convert(p, 61 - 2 * e + up - c.e_half_g);
    };
    const double f_a = f_n + own(qa, xa, ra), f_b = f_n + own(qb, xb, rb);
    out.hu_a = fma(f_a, geo[0], fp::neg(along_x));
    out.hv_a = fma(f_a, geo[1], along_y);
    out.hu_b = fma(f_b, geo[0], fp::neg(along_x));
    out.hv_b = fma(f_b, geo[1], along_y);
    return kDone;
}

}  // namespace fx
}  // namespace dgswe
