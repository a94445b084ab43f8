// qmc_ewald.cuh -- real-space Ewald terms of the electron gas: erfc in float-float
// arithmetic for the minimum image, and the FP32 sum over the other images.
// tests/test_ewald_functions.py compiles this header for the host and holds the bounds
// stated here.
#pragma once
#include <cmath>
#include "qmc_ff.cuh"

namespace qmc {

// Intervals of the erfc table: width 1/32 on [0, 6].
constexpr int HERFC_N = 192;

// Taylor coefficients of erfc at the interval centres: orders 0..3 as float-float
// pairs, 4..7 as floats.
inline void fill_erfc_table(float4 (*tab)[3]) {
    for (int j = 0; j < HERFC_N; ++j) {
        // derivatives of erfc: f' = g = -2/sqrt(pi) e^{-x^2}, f^(n+1) = -2 x f^(n) - 2 (n-1) f^(n-1)
        const double x = (j + 0.5) / 32.0;
        double d[8];
        d[0] = std::erfc(x);
        d[1] = -2.0 / std::sqrt(M_PI) * std::exp(-x * x);
        d[2] = -2.0 * x * d[1];
        for (int n = 2; n < 7; ++n) d[n + 1] = -2.0 * x * d[n] - 2.0 * (n - 1) * d[n - 1];
        double f = 1.0;
        float c[12];
        for (int n = 0; n < 8; ++n) {
            if (n) f *= n;
            const double v = d[n] / f;
            if (n < 4) {
                c[2 * n] = (float)v;
                c[2 * n + 1] = (float)(v - (double)c[2 * n]);
            } else {
                c[4 + n] = (float)v;
            }
        }
        for (int q = 0; q < 3; ++q) tab[j][q] = make_float4(c[4 * q], c[4 * q + 1], c[4 * q + 2], c[4 * q + 3]);
    }
}

// erfc on [0, 6] in float-float arithmetic (0 beyond): Taylor series about the
// centre of the argument's interval of width 1/32 (|d| <= 1/64: the truncated
// order 8 is below 4e-17), orders 4..7 in FP32 (|d|^4 = 6e-8), the lower ones
// in float-float.  Absolute error below 2e-14 on [0, 6].  A Chebyshev series
// over the whole range took 23 float-float steps (about 720 instructions
// against 75 and three 16-byte loads).
__device__ __forceinline__ ff erfc_ff(const float4 (*__restrict__ tab)[3], ff x) {
    if (!(x.hi < 6.0f)) return ff(0.0f);
    const int j = max(0, min((int)(x.hi * 32.0f), HERFC_N - 1));   // set_params takes any splitting: x may be negative
    const ff d = x + ff(-((float)j + 0.5f) * 0.03125f);
    const float4 a = tab[j][0], b = tab[j][1], c = tab[j][2];
    const float t = __fmaf_rn(d.hi, __fmaf_rn(d.hi, __fmaf_rn(d.hi, c.w, c.z), c.y), c.x);
    const ff p = ff_two_prod(d.hi, t);
    ff s = ff_fast_two_sum(b.z, __fadd_rn(b.w, p.hi));
    s = d * s + ff(b.x, b.y);
    s = d * s + ff(a.z, a.w);
    return d * s + ff(a.x, a.y);
}

// 2^-(q c) for FP32 q >= 0 with its rounding error qe and the constant c as a
// float pair: the product in two parts, a degree-6 polynomial for the fraction (fitted at
// Chebyshev nodes of |f| <= 1/2; within one ulp with its rounding), the integer in the exponent.
__device__ __forceinline__ float exp2_neg(float q, float qe, ff c) {
    const float p = __fmul_rn(q, c.hi);
    float pe = __fmaf_rn(q, c.hi, -p);
    pe = __fmaf_rn(q, c.lo, pe);
    pe = __fmaf_rn(qe, c.hi, pe);
    const float n = fminf(rintf(p), 125.0f);
    const float f = fmaxf(__fsub_rn(__fsub_rn(n, p), pe), -200.0f);   // clamped with n: the result underflows to 0
    float r = __fmaf_rn(f, 0.00015461445f, 0.0013400428f);
    r = __fmaf_rn(f, r, 0.009618057f);
    r = __fmaf_rn(f, r, 0.05550327f);
    r = __fmaf_rn(f, r, 0.2402265f);
    r = __fmaf_rn(f, r, 0.6931472f);
    r = __fmaf_rn(f, r, 1.0f);
    return p > 125.0f ? 0.0f : __fmul_rn(r, __int_as_float((127 - (int)n) << 23));
}

// Sum over the 26 images n != 0 of erfc(aL |s + n|) / |s + n| inside the cutoff,
// s the minimum-image separation in box units, in FP32.  erfc(x) = e^{-x^2}
// Q(1/x^2) / x with Q a degree-8 polynomial fitted at Chebyshev nodes of 1/x^2 in
// [1/36, 1/1.86^2] (7e-8 with its FP32 rounding), and e^{-x^2} is a product over
// the axes, so 9 exponentials serve the 26 terms and no square root is left:
// erfc(x) / d = e^{-x^2} Q(1/x^2) / (aL d^2).  Images with two axes shifted away
// (d^2 > 2) are skipped when the cutoff excludes them for every pair.
__device__ __forceinline__ float image_erfc(float sx, float sy, float sz, float aL, float rc2u, ff a2l2) {
    float qx[3], qy[3], qz[3], ex[3], ey[3], ez[3];
    // axis values ordered: no shift, shift towards the image (|s| - 1), shift away (|s| + 1)
    auto axis = [&](float s, float (&q)[3], float (&e)[3]) {
        const float a = fabsf(s);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float t = k == 0 ? a : (k == 1 ? __fsub_rn(a, 1.0f) : __fadd_rn(a, 1.0f));
            q[k] = __fmul_rn(t, t);
            e[k] = exp2_neg(q[k], __fmaf_rn(t, t, -q[k]), a2l2);
        }
    };
    axis(sx, qx, ex);
    axis(sy, qy, ey);
    axis(sz, qz, ez);
    const float ia = __fdividef(1.0f, aL), ia2 = ia * ia;
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            if ((i == 2) + (j == 2) == 2 && rc2u <= 2.0f) continue;
            const float qij = qx[i] + qy[j], eij = __fmul_rn(ex[i], ey[j]);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (i + j + k == 0) continue;
                if ((i == 2) + (j == 2) + (k == 2) >= 2 && rc2u <= 2.0f) continue;
                const float d2 = qij + qz[k];
                float id = __fdividef(1.0f, d2);
                id = __fmaf_rn(__fmaf_rn(-d2, id, 1.0f), id, id);
                const float w = id * ia2;
                float g = __fmaf_rn(w, 12.996532f, -21.552807f);
                g = __fmaf_rn(w, g, 16.388454f);
                g = __fmaf_rn(w, g, -7.8752494f);
                g = __fmaf_rn(w, g, 2.9005704f);
                g = __fmaf_rn(w, g, -1.0063616f);
                g = __fmaf_rn(w, g, 0.42103583f);
                g = __fmaf_rn(w, g, -0.28204688f);
                g = __fmaf_rn(w, g, 0.56418914f);
                const float v = __fmul_rn(__fmul_rn(eij, ez[k]), __fmul_rn(g, id));
                acc += d2 < rc2u ? v : 0.0f;
            }
        }
    return __fmul_rn(acc, ia);
}

}  // namespace qmc
