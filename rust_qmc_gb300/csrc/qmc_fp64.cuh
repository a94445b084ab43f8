// qmc_fp64.cuh -- FP64 elementary functions with few FP64 instructions.
//
// Every FP64 instruction of a warp (add, multiply, fma, compare, conversion)
// holds its SM sub-partition for 64 cycles here, whether one lane is active or
// 32 (four sub-partitions together issue one per 19 cycles), so the cost of a
// function is its number of FP64 instructions and the integer and FP32 work
// around them is close to free.  Hence: conversions, comparisons and scalings
// by powers of two run on the bits of the value, arguments are reduced with
// tables, and reciprocals and square roots start from FP32 seeds.
// Measured cycles per call, one warp (these functions / CUDA's, the latter
// compiled with the library's flags): exp 709 / 1062, log 907 / 2035,
// sqrt 476 / 623, 1/x 225 / 383 and 1/sqrt 291 / 511 (both sides one Newton
// step), 1/x to the last bits 289 / 378; a Box-Muller pair 2466.  Errors against
// 64 bits: exp 0.55 ulp, log 0.9 ulp, sqrt and the full reciprocal 0.5 ulp, sine
// and cosine 1.7e-16 absolute (tests/test_fp64_functions.py and
// tests/test_fp64_domains.py have the bounds).
// Argument reduction of exp after Tang, ACM TOMS 15 (1989), of log after Tang,
// ACM TOMS 16 (1990).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "qmc_fp64_tables.cuh"

namespace qmc {

__device__ __forceinline__ int d_hi(double x) { return __double2hiint(x); }
__device__ __forceinline__ int d_lo(double x) { return __double2loint(x); }

// Double of a float: exact for normal floats and zero (subnormals excluded).
__device__ __forceinline__ double d_of_float(float f) {
    const int u = __float_as_int(f);
    const int mag = u & 0x7fffffff;
    const int hi = mag ? (mag >> 3) + 0x38000000 : 0;
    return __hiloint2double(hi | (u & 0x80000000), u << 29);
}
// Nearest float of a positive double inside the normal FP32 range.
__device__ __forceinline__ float float_of_pos(double x) {
    const uint64_t b = (uint64_t)__double_as_longlong(x) + 0x10000000ull;
    return __int_as_float(__funnelshift_l((unsigned)b, (unsigned)(b >> 32) - 0x38000000u, 3));
}
// x 2^k for normal x and result (zero stays zero only for k = 0).
__device__ __forceinline__ double d_scale(double x, int k) { return __hiloint2double(d_hi(x) + (k << 20), d_lo(x)); }
// x < c for non-negative x (NaN: false), on the high words: c is compared with
// 20 bits of mantissa, which is all a threshold needs.
__device__ __forceinline__ bool d_below(double x, double c) { return d_hi(x) < d_hi(c); }
__device__ __forceinline__ bool d_positive(double x) { return d_hi(x) > 0; }

// 1/x for normal x of either sign below 2^1022 (zero, subnormal and larger x, inf and
// NaN give NaN): FP32 seed on the mantissa and one Newton step, relative error ~1e-14.
// Sign and exponent are put back on the bits, which costs no FP64 instruction.
__device__ __forceinline__ double d_rcp(double x) {
    const int hi = d_hi(x), ex = (hi >> 20) & 0x7ff;
    const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, d_lo(x));
    const double y = d_of_float(__fdividef(1.0f, float_of_pos(m)));
    const double e = fma(-m, y, 1.0);
    const double r = fma(e, y, y);
    const int rh = (d_hi(r) - ((ex - 1023) << 20)) ^ (hi & 0x80000000);
    return __hiloint2double((unsigned)(ex - 1) < 2044u ? rh : 0x7ff80000, d_lo(r));
}
// 1/sqrt(x) for positive normal x, the same way on x 4^-k in [1/2, 2): y + (y/2)(1 - x y^2).
__device__ __forceinline__ double d_rsqrt(double x) {
    const int hi = d_hi(x), k = (hi >> 21) - 511;
    const double m = __hiloint2double(hi - (k << 21), d_lo(x));
    const double y = d_of_float(rsqrtf(float_of_pos(m)));
    const double e = fma(-m * y, y, 1.0);
    const double r = fma(d_scale(y, -1), e, y);
    return __hiloint2double((unsigned)(hi - 0x00100000) < 0x7fe00000u ? d_hi(r) - (k << 20) : 0x7ff80000, d_lo(r));
}

// 1/x to the last bit or two: seed on the mantissa, two Newton steps in one
// (y (1 + e + e^2)); arguments whose reciprocal is not a normal number, or that are
// none themselves, are divided.
__device__ __forceinline__ double d_rcp_full(double x) {
    const int hi = d_hi(x), ex = ((hi >> 20) & 0x7ff) - 1023;
    if ((unsigned)(ex + 1022) >= 2044u) return 1.0 / x;               // zero, subnormal, from 2^1022 on, inf, NaN
    const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, d_lo(x));
    double y = d_of_float(__fdividef(1.0f, float_of_pos(m)));
    const double e = fma(-m, y, 1.0);
    y = fma(y, fma(e, e, e), y);
    return __hiloint2double((d_hi(y) - (ex << 20)) ^ (hi & 0x80000000), d_lo(y));
}

// sqrt(x): coupled Newton iteration for g = sqrt(m) and h = 1/(2 sqrt(m)) on
// m = x 4^-k, then one residual correction.
__device__ __forceinline__ double d_sqrt(double x) {
    const int hi = d_hi(x);
    if ((unsigned)(hi - 0x00100000) >= 0x7fe00000u) return sqrt(x);   // zero, subnormal, negative, inf, NaN
    const int k = (hi >> 21) - 511;                                   // m in [1/2, 2)
    const double m = __hiloint2double(hi - (k << 21), d_lo(x));
    const double y = d_of_float(rsqrtf(float_of_pos(m)));
    double g = m * y, h = d_scale(y, -1);
    const double r = fma(-g, h, 0.5);
    g = fma(g, r, g);
    h = fma(h, r, h);
    g = fma(fma(-g, g, m), h, g);
    return d_scale(g, k);
}

// e^x: x = (256 k + j) ln2/256 + r, |r| < 1.4e-3; e^x = 2^k 2^(j/256) e^r with
// e^r through r^4 and the r^3 coefficient raised by 0.87 max|r|^2 / 120, which
// leaves an eighth of the r^5 term (5e-18).  From |x| = 708 on the result is scaled in
// two steps, so that it may be subnormal, 0 or inf.
__device__ __forceinline__ double d_exp(double x) {
    const int hi = d_hi(x), mag = hi & 0x7fffffff;
    const bool out = mag >= 0x40862000;                               // |x| >= 708, inf, NaN
    // x as a truncated float (|x| < 2^-38: 0)
    const float xf = mag < 0x3d900000 ? 0.0f
                                      : __int_as_float((hi & 0x80000000) | __funnelshift_l(d_lo(x), mag - 0x38000000, 3));
    const float kf = rintf(xf * 369.32994f);
    const int n = (int)kf;
    const double kd = d_of_float(kf);
    double r = fma(kd, -0x1.62e42fee00000p-9, x);
    r = fma(kd, -0x1.a39ef35793c76p-41, r);
    const double2 t = kExp2T[n & 255];
    double p = fma(r, 1.0 / 24.0, 1.0 / 6.0 + 1.3288e-8);
    p = fma(r, p, 0.5);
    const double s = fma(r * r, p, r);
    const double v = t.x + fma(t.x, s, t.y);
    if (!out) return d_scale(v, n >> 8);
    if (mag < 0x40880000)                                             // |x| < 768
        return d_scale(v, (n >> 8) + (hi < 0 ? 128 : -128)) * __hiloint2double(hi < 0 ? (1023 - 128) << 20 : (1023 + 128) << 20, 0);
    return mag > 0x7ff00000 ? x : (hi < 0 ? 0.0 : __hiloint2double(0x7ff00000, 0));
}

// log x: x = 2^k z with z in [0.6875, 1.375), log x = k ln2 + log c + log(1 + r)
// with r = z (1/c) - 1, |r| <= 2^-7 next to 1 (where c = 1 keeps the result
// relatively exact) and below 4e-3 elsewhere.  k ln2 + log c is exact in its leading
// parts (multiples of 2^-42); what these leave goes with the polynomial.  The interval
// bounds (z from 0x3fe60000 of the high word, seven more bits) are those of the
// logarithm in ARM's optimized-routines.
__device__ __forceinline__ double d_log(double x) {
    const int hi = d_hi(x);
    if ((unsigned)(hi - 0x00100000) >= 0x7fe00000u) return log(x);    // zero, subnormal, negative, inf, NaN
    const int tmp = hi - 0x3fe60000, k = tmp >> 20;
    const double z = __hiloint2double(hi - (tmp & 0xfff00000), d_lo(x));
    const int i = (tmp >> 13) & 127;
    const double2 c = kLogT[i];
    const double r = fma(z, c.x, -1.0);
    double p = fma(r, -1.0 / 8.0, 1.0 / 7.0);
    p = fma(r, p, -1.0 / 6.0);
    p = fma(r, p, 1.0 / 5.0);
    p = fma(r, p, -1.0 / 4.0);
    p = fma(r, p, 1.0 / 3.0);
    p = fma(r, p, -0.5);
    const double kd = d_of_float((float)k);
    return fma(kd, kLn2Hi, c.y) + (r + fma(r * r, p, fma(kd, kLn2Lo, kLogLo[i])));
}

// (sin, cos) of 2 pi (j + rem scale) with integer j / 256 of a turn and the odd
// remainder rem: |2 pi rem scale| <= pi/256.
__device__ __forceinline__ void d_sincos_turn(unsigned j, int rem, double scale, double& s, double& c) {
    const double2 t = kSinCosT[j & 63];
    const double d = d_of_float((float)rem) * scale;
    const double d2 = d * d;
    const double sd = fma(d * d2, fma(d2, 1.0 / 120.0, -1.0 / 6.0), d);
    const double cm = d2 * fma(d2, fma(d2, -1.0 / 720.0, 1.0 / 24.0), -0.5);   // cos d - 1
    const double sn = fma(t.x, sd, fma(t.y, cm, t.y)), cn = fma(-t.y, sd, fma(t.x, cm, t.x));
    const bool odd = (j & 64) != 0;
    const unsigned ns = (j & 128) << 24, nc = ((j + 64) & 128) << 24;          // sign bits of the quadrant
    const double a = odd ? cn : sn, b = odd ? sn : cn;
    s = __hiloint2double(d_hi(a) ^ ns, d_lo(a));
    c = __hiloint2double(d_hi(b) ^ nc, d_lo(b));
}

// (k + 1/2) 2^-24 and (x + 1/2) 2^-32 exactly, from their bits.
__device__ __forceinline__ double d_u24(uint32_t k) {
    const uint32_t v = 2u * k + 1u;                                   // value v 2^-25
    const int lz = __clz(v);
    const uint32_t m = lz == 31 ? 0u : v << (lz + 1);                 // mantissa below the leading one
    return __hiloint2double(((1023 + 6 - lz) << 20) | (m >> 12), m << 20);
}
__device__ __forceinline__ double d_u32(uint32_t x) {
    const int lz = __clz(x);                                          // 32 for x = 0
    const uint64_t m = (((uint64_t)x << 1) | 1u) << (31 + lz);        // leading one at bit 63
    const uint64_t f = (m << 1) >> 12;
    return __hiloint2double(((1022 - lz) << 20) | (int)(f >> 32), (int)f);
}

// Box-Muller pair of the uniforms (a + 1/2) 2^-24, (b + 1/2) 2^-24.
__device__ __forceinline__ void d_normals24(uint32_t a, uint32_t b, double& n0, double& n1) {
    const double l = d_log(d_u24(a));
    const double r = d_sqrt(__hiloint2double((d_hi(l) + 0x00100000) ^ 0x80000000, d_lo(l)));   // -2 log u
    const uint32_t v = 2u * b + 1u, j = (v + 0x10000u) >> 17;         // u = v 2^-25
    double s, c;
    d_sincos_turn(j, (int)(v - (j << 17)), 6.283185307179586 / 33554432.0, s, c);
    n0 = r * c;
    n1 = r * s;
}
// The same from the 32-bit uniforms (a + 1/2) 2^-32, (b + 1/2) 2^-32.
__device__ __forceinline__ void d_normals32(uint32_t a, uint32_t b, double& n0, double& n1) {
    const double l = d_log(d_u32(a));
    const double r = d_sqrt(__hiloint2double((d_hi(l) + 0x00100000) ^ 0x80000000, d_lo(l)));
    const uint32_t j = (uint32_t)(((uint64_t)b + 0x800000u) >> 24);
    const int rem = 2 * (int)(b - (j << 24)) + 1;                     // u = j/256 + rem 2^-33
    double s, c;
    d_sincos_turn(j, rem, 6.283185307179586 / 8589934592.0, s, c);
    n0 = r * c;
    n1 = r * s;
}

}  // namespace qmc
