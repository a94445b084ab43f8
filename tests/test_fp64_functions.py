"""The FP64 elementary functions of csrc/qmc_fp64.cuh against 80-bit (or wider)
long double arithmetic: the header is compiled for the host with its device
intrinsics written out, FP32 seeds perturbed by the hardware's error bound.

Bounds, from the algorithms: exp, log and sqrt end in one or two roundings of
a result whose corrections are small (2 ulp), sine and cosine in two roundings
of values below 1 (3e-16 absolute), one Newton step squares a seed error of
2^-22 plus the rounding of its argument to FP32 (3/2 (1.5 2^-22)^2 < 2e-13),
the full reciprocal cubes it (2 ulp).  The uniforms are exact."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rust_qmc_gb300", "csrc")

SHIM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__ static
#define __forceinline__ inline
struct double2 { double x, y; };
static double seed_err = 0;
static uint64_t bits(double x) { uint64_t b; memcpy(&b, &x, 8); return b; }
static int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static int __double2loint(double x) { return (int)bits(x); }
static double __hiloint2double(int h, int l) {
    uint64_t b = ((uint64_t)(uint32_t)h << 32) | (uint32_t)l; double x; memcpy(&x, &b, 8); return x;
}
static long long __double_as_longlong(double x) { return (long long)bits(x); }
static int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }
static float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
static unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) { return (hi << s) | (lo >> (32 - s)); }
static int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
static float __fdividef(float a, float b) { return (float)(a / (double)b * (1.0 + seed_err)); }
static float rsqrtf(float a) { return (float)(1.0 / std::sqrt((double)a) * (1.0 + seed_err)); }
using std::fma; using std::sqrt; using std::exp; using std::log;
#include "qmc_fp64.cuh"
using namespace qmc;
typedef long double ld;
static double ulp(double v) { return std::ldexp(1.0, std::ilogb(v) - 52); }
int main() {
    std::mt19937_64 g(7);
    auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    double e_exp = 0, e_log = 0, e_sqrt = 0, e_rcp = 0, e_rsq = 0, e_full = 0, e_sc = 0, e_u = 0, e_n = 0;
    auto mx = [](double& m, double v) { if (!(v <= m)) m = v; };
    for (int i = 0; i < 400000; ++i) {
        seed_err = U(-1, 1) * 0x1p-22;
        double x = i % 4 == 0 ? U(-707.9, 707.9) : (i % 4 == 1 ? U(-1, 1) : (i % 4 == 2 ? U(-40, 5) : std::ldexp(U(-1, 1), -(i % 60))));
        mx(e_exp, std::fabs((double)((ld)d_exp(x) - expl((ld)x))) / ulp((double)expl((ld)x)));
        double y = i % 3 == 0 ? U(0.5, 1.5) : (i % 3 == 1 ? std::ldexp(U(1, 2), (int)U(-1000, 1000)) : 1.0 + std::ldexp(U(-1, 1), -(i % 50) - 1));
        double l = (double)logl((ld)y);
        mx(e_log, l == 0 ? std::fabs(d_log(y)) * 1e300 : std::fabs((double)((ld)d_log(y) - logl((ld)y))) / ulp(l));
        mx(e_sqrt, std::fabs((double)((ld)d_sqrt(y) - sqrtl((ld)y))) / ulp(std::sqrt(y)));
        mx(e_full, std::fabs((double)((ld)d_rcp_full(-y) + 1 / (ld)y)) / ulp(1 / y));
        double z = std::ldexp(U(1, 2), (int)U(-100, 100));
        mx(e_rcp, std::fabs((double)((ld)d_rcp(z) * (ld)z - 1)));
        mx(e_rsq, std::fabs((double)((ld)d_rsqrt(z) * sqrtl((ld)z) - 1)));
        uint32_t a = (uint32_t)g(), b = i < 8 ? (uint32_t)(i < 4 ? i : -i) : (uint32_t)g();
        if (i < 40) a >>= (i & 31);
        uint32_t a24 = a & 0xffffffu, b24 = b & 0xffffffu;
        mx(e_u, std::fabs(d_u24(a24) - ((double)a24 + 0.5) / 16777216.0) + std::fabs(d_u32(a) - ((double)a + 0.5) / 4294967296.0));
        const ld tau = 6.283185307179586476925286766559L;
        double s, c, n0, n1;
        uint32_t v = 2u * b24 + 1u, j = (v + 0x10000u) >> 17;
        d_sincos_turn(j, (int)(v - (j << 17)), 6.283185307179586 / 33554432.0, s, c);
        ld t = tau * ((ld)b24 + 0.5L) / 16777216.0L;
        mx(e_sc, std::fabs((double)((ld)s - sinl(t))));
        mx(e_sc, std::fabs((double)((ld)c - cosl(t))));
        d_normals32(a, b, n0, n1);
        t = tau * ((ld)b + 0.5L) / 4294967296.0L;
        ld r = sqrtl(-2 * logl(((ld)a + 0.5L) / 4294967296.0L));
        mx(e_n, std::fabs((double)((ld)n0 - r * cosl(t))));
        mx(e_n, std::fabs((double)((ld)n1 - r * sinl(t))));
    }
    double inf = INFINITY, nan = NAN;
    bool edge = d_exp(0.0) == 1.0 && d_exp(-0.0) == 1.0 && d_exp(-inf) == 0 && d_exp(-800.0) == 0 && d_exp(inf) == inf &&
                std::isnan(d_exp(nan)) && std::isnan(d_exp(-nan)) && d_log(1.0) == 0 && d_log(0.0) == -inf &&
                std::isnan(d_log(-1.0)) && d_log(inf) == inf && d_sqrt(0.0) == 0 && d_sqrt(inf) == inf &&
                std::isnan(d_sqrt(-1.0)) && std::isnan(d_sqrt(nan)) && d_sqrt(4.0) == 2.0 && d_sqrt(1e-310) > 0 &&
                std::isnan(d_rcp(nan)) && std::isnan(d_rsqrt(nan)) && d_exp(1e-300) == 1.0 && d_exp(-3e-20) == 1.0;
    std::printf("%g %g %g %g %g %g %g %g %g %d\n", e_exp, e_log, e_sqrt, e_full, e_rcp, e_rsq, e_sc, e_u, e_n, (int)edge);
    return 0;
}
"""


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64")
    (d / "cuda_runtime.h").write_text("")
    (d / "t.cpp").write_text(SHIM)
    exe = str(d / "t")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-I", str(d), "-I", CSRC, str(d / "t.cpp"), "-o", exe],
                   check=True)
    return [float(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()]


@pytest.mark.parametrize("k, name, bound", [
    (0, "exp (ulp)", 2.0), (1, "log (ulp)", 2.0), (2, "sqrt (ulp)", 2.0), (3, "full reciprocal (ulp)", 2.0),
    (4, "reciprocal (relative)", 2e-13), (5, "reciprocal square root (relative)", 2e-13),
    (6, "sine and cosine (absolute)", 3e-16), (7, "uniforms", 0.0), (8, "normals (absolute)", 3e-15)])
def test_error_bound(errors, k, name, bound):
    assert errors[k] <= bound, (name, errors[k])


def test_special_values(errors):
    assert errors[9] == 1
