"""csrc/qmc_ewald.cuh compiled for the host, its device intrinsics written out and the
approximate reciprocal perturbed by the hardware's error bound, against long double
arithmetic: erfc of the minimum image, 2^-x of the images' factors and the sum over the
26 images at shifted coordinates that are FP32 numbers, as the walkers' are.

Bounds: erfc 2e-14 and 2^-x one ulp (1.2e-7) as the header states.  A term of the image sum is a
product of three such factors, of the polynomial (7e-8), of 1/d^2 (one Newton step, a few
roundings) and of 1/(alpha L)^3 from one reciprocal of 2^-23: 3 * 1.2e-7 + 7e-8 +
3 * 1.2e-7 and five roundings of 6e-8 make 1.1e-6, all terms positive.  Over many separations
roundings go either way: the mean stays below 2e-7, where the reciprocal is exact."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rust_qmc_gb300", "csrc")

SOURCE = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __host__
#define __forceinline__ inline
#define __restrict__
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
static float4 make_float4(float a, float b, float c, float d) { return {a, b, c, d}; }
static float2 make_float2(float a, float b) { return {a, b}; }
static double seed_err = 0;
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static float __frcp_rn(float a) { return 1.0f / a; }
static float __fdividef(float a, float b) { return (float)(a / (double)b * (1.0 + seed_err)); }
static float rsqrtf(float a) { return (float)(1.0 / std::sqrt((double)a)); }
static int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
static float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
using std::max;
using std::min;
#include "qmc_ewald.cuh"
using namespace qmc;
typedef long double ld;
static float4 room[3 * HERFC_N][3];                  // the table between rows of NaN
static float4 (*tab)[3] = room + HERFC_N;
int main() {
    for (auto& row : room)
        for (auto& v : row) v = {NAN, NAN, NAN, NAN};
    std::mt19937_64 g(5);
    auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    auto mx = [](double& m, double v) { if (!(v <= m)) m = v; };
    fill_erfc_table(tab);
    double e_erfc = 0, e_exp = 0, e_img = 0, bias = 0;
    auto one = [&](double v) {
        const ff x(v);
        mx(e_erfc, std::fabs((double)((ld)erfc_ff(tab, x).hi + (ld)erfc_ff(tab, x).lo - erfcl((ld)x.hi + (ld)x.lo))));
    };
    for (int i = 0; i < 200000; ++i) one(U(0, 6));
    for (int j = 0; j <= HERFC_N; ++j)
        for (double d : {-1e-7, 0.0, 1e-7}) one(std::fmax(0.0, j / 32.0 + d));
    for (double v : {0.0, 1e-30, 5.9999999, 6.0, 7.0, 100.0}) one(v);
    for (int i = 0; i < 200000; ++i) {
        const double aL = U(3.74, 30), t = U(0, 1.5);
        const float q = (float)t * (float)t, qe = std::fmaf((float)t, (float)t, -q);
        const ff c(aL * aL * 1.4426950408889634);
        const ld want = exp2l(-((ld)q + qe) * ((ld)c.hi + c.lo));
        const double got = exp2_neg(q, qe, c);
        if (want > 1e-36L) mx(e_exp, std::fabs((double)(got / want - 1)));
        else mx(e_exp, got > 2e-36 ? 1.0 : 0.0);
    }
    int n = 0;
    for (int i = 0; i < 60000; ++i) {
        const bool exact = i % 2;
        seed_err = exact ? 0.0 : U(-1, 1) * 0x1p-23;
        const float aL = (float)(i % 5 == 0 ? 3.74 : (i % 5 == 1 ? 4.0 : U(3.74, 8.0))), rc2 = (float)(5.6 / aL * (5.6 / aL));
        float s[3];
        for (float& v : s) v = (float)(i % 7 == 0 ? (U(-1, 1) < 0 ? -0.5 : 0.5) : U(-0.5, 0.5));
        const double got = image_erfc(s[0], s[1], s[2], aL, rc2, ff((double)aL * aL * 1.4426950408889634));
        ld want = 0;
        for (int a = -1; a <= 1; ++a)
            for (int b = -1; b <= 1; ++b)
                for (int c = -1; c <= 1; ++c) {
                    if (!a && !b && !c) continue;
                    // the shifted coordinates are FP32 numbers
                    auto at = [](float v, int k) { return k ? std::fabs(v) + (float)k : std::fabs(v); };
                    const ld x = at(s[0], a), y = at(s[1], b), z = at(s[2], c), d = sqrtl(x * x + y * y + z * z);
                    want += erfcl((ld)aL * d) / d;
                }
        // left out beyond alpha r = 5.6: up to 26 erfc(5.6) / d, 1e-13
        const double e = (double)(got / want - 1);
        mx(e_img, std::fmax(0.0, (double)(fabsl(got - want) - 1e-13L)) / (double)want);
        if (exact) { bias += e * (want > 1e-6L); n += want > 1e-6L; }
    }
    bool inside = true;                              // every argument reads the table's own rows
    for (double v : {-1e-6, -0.02, -3.0, -5.99, -6.0, -11.0, 6.0, 1e30}) inside = inside && std::isfinite(erfc_ff(tab, ff(v)).hi);
    std::printf("%g %g %g %g %d\n", e_erfc, e_exp, e_img, std::fabs(bias / n), (int)inside);
}
"""


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    d = tmp_path_factory.mktemp("ewald")
    (d / "cuda_runtime.h").write_text("")
    (d / "t.cpp").write_text(SOURCE)
    exe = str(d / "t")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-I", str(d), "-I", CSRC, str(d / "t.cpp"), "-o", exe],
                   check=True)
    return [float(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()]


@pytest.mark.parametrize("k, name, bound", [(0, "erfc (absolute)", 2e-14), (1, "2^-x (relative)", 1.2e-7),
                                            (2, "image sum (relative)", 1.1e-6), (3, "image sum, mean", 2e-7)])
def test_error_bound(errors, k, name, bound):
    assert errors[k] <= bound, (name, errors[k])


def test_no_argument_reads_past_the_table(errors):
    assert errors[4] == 1
