"""The FP64 elementary functions of csrc/qmc_fp64.cuh outside the arguments of
test_fp64_functions.py: negative numbers, the whole exponent range, zero,
infinities and NaN.  The header is compiled for the host with that test's
device intrinsics.  Bounds as there: one Newton step on a seed of relative error
2^-22 leaves less than 2e-13."""
import subprocess

import pytest

from tests.test_fp64_functions import CSRC, SHIM

MAIN = r"""
static bool isn(double x) { return x != x; }
int main() {
    std::mt19937_64 g(11);
    auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    auto mx = [](double& m, double v) { if (!(v <= m)) m = v; };
    const double inf = INFINITY, nan = NAN;
    double e_rcp = 0, e_rsq = 0;
    for (int i = 0; i < 400000; ++i) {
        seed_err = U(-1, 1) * 0x1p-22;
        const double x = (i & 1 ? -1 : 1) * std::ldexp(U(1, 2), (int)U(i % 3 ? -8 : -1021, i % 3 ? 8 : 1022));
        mx(e_rcp, std::fabs((double)((ld)d_rcp(x) * (ld)x - 1)));
        const double y = std::ldexp(U(1, 2), (int)U(-1021, 1023));
        mx(e_rsq, std::fabs((double)((ld)d_rsqrt(y) * sqrtl((ld)y) - 1)));
    }
    seed_err = 0;
    const bool special = isn(d_rcp(0.0)) && isn(d_rcp(-0.0)) && isn(d_rcp(inf)) && isn(d_rcp(-inf)) && isn(d_rcp(nan)) &&
                         isn(d_rcp(1e-310)) && isn(d_rsqrt(0.0)) && isn(d_rsqrt(-2.0)) && isn(d_rsqrt(inf)) &&
                         isn(d_rsqrt(nan)) && isn(d_rsqrt(1e-310)) && d_rcp(-2.0) == -0.5 && d_rsqrt(0x1p-400) == 0x1p200;
    std::printf("%g %g %d\n", e_rcp, e_rsq, (int)special);
    return 0;
}
"""


def run_host(tmp, main):
    """Output of `main` compiled with the functions under test."""
    (tmp / "cuda_runtime.h").write_text("")
    (tmp / "t.cpp").write_text(SHIM.split("int main")[0] + main)
    exe = str(tmp / "t")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-I", str(tmp), "-I", CSRC, str(tmp / "t.cpp"), "-o", exe],
                   check=True)
    return [float(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()]


@pytest.fixture(scope="module")
def one_step(tmp_path_factory):
    return run_host(tmp_path_factory.mktemp("domains"), MAIN)


@pytest.mark.parametrize("k, name", [(0, "reciprocal"), (1, "reciprocal square root")])
def test_one_newton_step_over_all_exponents(one_step, k, name):
    assert one_step[k] <= 2e-13, (name, one_step[k])


def test_one_newton_step_special_values(one_step):
    assert one_step[2] == 1


FULL = r"""
int main() {
    std::mt19937_64 g(13);
    auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    double worst = 0;
    const double inf = INFINITY, nan = NAN;
    const double xs[] = {0.0, -0.0, inf, -inf, 5e-324, -1e-310, 0x1.8p1022, -0x1p1023, 0x1.fffffffffffffp1023, 0x1p-1022, 0x1p1021};
    bool special = d_rcp_full(nan) != d_rcp_full(nan);
    for (double x : xs) special = special && (std::isinf(1 / x) ? d_rcp_full(x) == 1 / x : std::fabs(d_rcp_full(x) - 1 / x) <= 2 * ulp(1 / x) || d_rcp_full(x) == 1 / x);
    for (int i = 0; i < 200000; ++i) {
        seed_err = U(-1, 1) * 0x1p-22;
        const double x = (i & 1 ? -1 : 1) * std::ldexp(U(1, 2), (int)U(-1022, 1022));
        const double e = std::fabs((double)((ld)d_rcp_full(x) - 1 / (ld)x)) / ulp(1 / x);
        if (!(e <= worst)) worst = e;
    }
    std::printf("%g %d\n", worst, (int)special);
    return 0;
}
"""


@pytest.fixture(scope="module")
def full(tmp_path_factory):
    return run_host(tmp_path_factory.mktemp("full"), FULL)


def test_full_reciprocal_over_all_exponents(full):
    assert full[0] <= 2.0


def test_full_reciprocal_special_values(full):
    """Zero, subnormal numbers, the largest exponents, infinities and NaN as a division gives them."""
    assert full[1] == 1


EXP = r"""
int main() {
    std::mt19937_64 g(17);
    auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    double hi = 0, lo = 0;
    auto mx = [](double& m, double v) { if (!(v <= m)) m = v; };
    for (int i = 0; i < 100000; ++i) {
        const double x = U(700.0, 709.78), y = U(-745.13, -700.0);
        mx(hi, std::fabs((double)((ld)d_exp(x) - expl((ld)x))) / ulp(std::exp(x)));
        const double want = std::exp(y);
        mx(lo, std::fabs((double)((ld)d_exp(y) - expl((ld)y))) / std::fmax(want >= 0x1p-1022 ? ulp(want) : 0, 0x1p-1074));
    }
    const bool ends = std::isinf(d_exp(709.79)) && std::isinf(d_exp(767.9)) && std::isinf(d_exp(768.0)) && std::isinf(d_exp(1e300)) &&
                      d_exp(-745.2) == 0 && d_exp(-767.9) == 0 && d_exp(-768.0) == 0 && d_exp(-1e300) == 0;
    std::printf("%g %g %d\n", hi, lo, (int)ends);
    return 0;
}
"""


@pytest.fixture(scope="module")
def ends_of_exp(tmp_path_factory):
    return run_host(tmp_path_factory.mktemp("exp"), EXP)


def test_exp_at_the_ends_of_its_range(ends_of_exp):
    """Up to the largest double and down to the smallest subnormal one (2 ulp; a
    subnormal result is rounded once more, in units of 2^-1074)."""
    assert ends_of_exp[0] <= 2.0 and ends_of_exp[1] <= 2.0
    assert ends_of_exp[2] == 1


LOG = r"""
int main() {
    std::mt19937_64 g(19);
    auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    double worst = 0;
    for (int i = 0; i < 1000000; ++i) {
        const double y = i % 4 == 0 ? U(0.6, 1.5) : (i % 4 == 1 ? std::ldexp(U(1, 2), (int)U(-1000, 1000)) : (i % 4 == 2 ? U(0.0, 1.0) : 1.0 + U(-1, 1) * 0x1p-6));
        const ld l = logl((ld)y);
        const double e = std::fabs((double)((ld)d_log(y) - l)) / ulp((double)l);
        if (!(e <= worst)) worst = e;
    }
    std::printf("%g\n", worst);
    return 0;
}
"""


def test_logarithm_is_as_exact_as_the_librarys(tmp_path):
    """1 ulp, the documented bound of CUDA's log."""
    err, = run_host(tmp_path, LOG)
    assert err <= 1.0, err
