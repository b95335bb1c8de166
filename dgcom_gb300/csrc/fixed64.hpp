// Square roots, reciprocals and h^(-4/3) of doubles in 64-bit fixed point.
//
// GB300 takes one FP64 instruction of a warp in 64 cycles of an SM
// sub-partition, one 32×32+64-bit integer multiply-add in 2 (measured: 67.6
// and 2.3 cycles, in parallel on their two pipes), so a Newton step of
// 64-bit integers costs a tenth of one in FP64. Each function takes a
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

constexpr uint64_t kMantissa = 0x000FFFFFFFFFFFFFull, kImplicit = 0x0010000000000000ull;

// Biased exponent field and the mantissa with its implicit bit (2^52..2^53)
DG_HD int expo(double x) { return (int)((uint64_t)fp::bits(x) >> 52) & 0x7FF; }
DG_HD uint64_t mant(double x) { return ((uint64_t)fp::bits(x) & kMantissa) | kImplicit; }
// The float in [1, 2) of a mantissa, truncated
DG_HD float mant_f32(uint64_t m) { return as_float((uint32_t)(m >> 29) + 0x3F000000u); }

// √x for x in [2^-126, 2^127) (the caller's guard). With X = x·4^-k in
// [1, 4): s0 = X·rsqrt(X) to 2^-21 in 31 bits, one Newton step to 2^-42 in
// 47, a second from the exact residual X − s1² (its high bits cancel, so
// arithmetic modulo 2^64 holds it whole) to 2^-60.
DG_HD double sqrt_pos(double x) {
    const uint64_t m = mant(x);
    const int e = expo(x);            // x = m·2^(e − 1075)
    const int odd = (e & 1) ^ 1;      // 1023 is odd: an even field is an odd power of two
    const uint64_t X = m << (8 + odd);                  // 2^60·X
    const float xf = as_float((uint32_t)(m >> 29) + 0x3F000000u + ((uint32_t)odd << 23));
    const uint32_t r = (uint32_t)(seed_rsqrt(xf) * 2147483648.0f);  // 2^31/√X, in [2^30, 2^31]
    // X·2^60 / 2^32 (29–31 bits) times 2^31/√X → √X·2^59, to 2^30·√X < 2^31
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
    const uint64_t s = (s1 << 16) + (uint64_t)c2;  // 2^62·√X in [2^62, 2^63)
    const uint64_t q = (s + 512u) >> 10;           // rounded to 53 bits (2^52..2^53)
    // exponent field of √x: 1023 + k, k = (e − 1023 − odd)/2
    return fp::from_bits((int64_t)(q + ((uint64_t)((e - 1023 - odd) / 2 + 1022) << 52)));
}

// 1/y for y in [2^-125, 2^125) (the caller's guard): r0 to 2^-22, then
// r0·(1 + e + e²) with e = 1 − Y·r0 (relative error e³ = 2^-63)
DG_HD double rcp_pos(double y) {
    const uint64_t m = mant(y);
    const int e = expo(y);
    const uint64_t Y = m << 11;  // 2^63·Y, Y in [1, 2)
    const uint32_t r = (uint32_t)(seed_rcp(mant_f32(m)) * 2147483648.0f);  // [2^30, 2^31]
    // 2^62·Y·r0
    const uint64_t p = madu(hi32(Y), r, hi32(madu(lo32(Y), r, 0)));
    const int64_t e1 = (int64_t)((1ull << 62) - p);  // 2^62·e, |e| < 2^-20
    const int32_t es = (int32_t)(e1 >> 12);          // 2^50·e
    const int64_t e2 = e1 + (mads(es, es, 0) >> 38);  // 2^62·(e + e²)
    // r0·(e + e²): 2^62 · 2^31 / 2^32
    const int64_t c = mads((int32_t)(e2 >> 32), (int32_t)(r >> 1), 0) * 2 +
                      (int64_t)hi32(madu(lo32((uint64_t)e2), r, 0)) +
                      ((r & 1) ? (e2 >> 32) : 0);
    const uint64_t q = ((uint64_t)r << 30) + (uint64_t)c;  // 2^61/Y in (2^60, 2^61]
    const uint64_t rounded = (q + 128u) >> 8;              // (2^52, 2^53]
    // 1/y = (1/Y)·2^(1023 − e), 1/Y in (½, 1]
    return fp::from_bits((int64_t)(rounded + ((uint64_t)(2044 - e) << 52)));
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
#if defined(__CUDA_ARCH__)
    const int c = __clz((int)hi32(w));
#else
    const int c = __builtin_clzll(w);
#endif
    const uint64_t n = w << c;  // top bit 63
    const uint64_t rounded = (n >> 11) + ((n >> 10) & 1);
    // n·2^-63 in [1, 2): w·2^-62 = n·2^(-62 − c), so the exponent of
    // m^(-4/3) is 1 − c, of the result 1 − c − 4k, k = k3 − 342
    const int field = 1023 + 1 - c - 4 * ((int)k3 - 342);
    return fp::from_bits((int64_t)(rounded + ((uint64_t)(field - 1) << 52)));
}

}  // namespace fx
}  // namespace dgswe
