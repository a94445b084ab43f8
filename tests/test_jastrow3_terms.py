"""jastrow3_pair and jastrow3_term of csrc/qmc_jastrow3_logderiv.h -- the pair order and
the terms that the device kernel k_jastrow3_logderiv deals to its lanes -- compiled
unchanged for the host: every pair comes once, 32 in a row (an N above 32) join distinct
electrons, and the terms add up to the header's plain sums (64-bit sums of up to 1400
terms in another order: 1e-12 of the largest sum's magnitude)."""
import shutil
import subprocess

import pytest

from tests.test_jastrow3_logderiv_header import HEADER_DIR

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include <set>
#include <utility>
#include <vector>
#include "qmc_jastrow3_logderiv.h"
using namespace qmc;
int main() {
    std::mt19937_64 g(3);
    auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    int bad = 0;
    double worst = 0;
    for (int N : {1, 2, 3, 4, 7, 10, 11, 31, 32, 33, 42, 54, 63, 64}) {
        std::set<std::pair<int, int>> seen;
        const int n_pair = N * (N - 1) / 2;
        std::vector<int> pi(n_pair), pj(n_pair);
        for (int t = 0; t < n_pair; ++t) {
            int i, j;
            jastrow3_pair(t, N, i, j);
            if (i < 0 || j < 0 || i >= N || j >= N || i == j || !seen.insert({i < j ? i : j, i < j ? j : i}).second) ++bad;
            pi[t] = i; pj[t] = j;
        }
        if ((int)seen.size() != n_pair) ++bad;
        for (int t0 = 0; N > 32 && t0 < n_pair; t0 += 32) {
            std::set<int> a, b;
            for (int t = t0; t < t0 + 32 && t < n_pair; ++t)
                if (!a.insert(pi[t]).second || !b.insert(pj[t]).second) ++bad;
        }
        for (int n_nuc : {0, 1, 12}) {
            const int n_up = (N + 1) / 2;
            std::vector<double> pos(3 * N), gr(3 * N), nuc(5 * n_nuc + 5);
            for (auto& v : pos) v = U(-3, 3);
            for (auto& v : gr) v = U(-2, 2);
            for (int I = 0; I < n_nuc; ++I) {
                for (int c = 0; c < 3; ++c) nuc[5 * I + c] = U(-3, 3);
                nuc[5 * I + 3] = 1 + I % 6;
                nuc[5 * I + 4] = I % 2;
            }
            if (n_nuc && N > 1)
                for (int c = 0; c < 3; ++c) { pos[3 + c] = pos[c]; nuc[c] = pos[c]; }   // coincident electrons and nucleus
            const double p[8] = {1.3, 1.7, 0.45, 0.3, 1.9, 2.4, 0.8, 1.1};
            auto at = [&](int i, int c) { return pos[3 * i + c]; };
            auto gd = [&](int i, int c) { return gr[3 * i + c]; };
            double want[16], got[16] = {0}, size = 1, only[16] = {0};
            jastrow3_log_derivatives(N, n_up, n_nuc, nuc.data(), p, at, want);
            jastrow3_el_derivatives(N, n_up, n_nuc, nuc.data(), p, at, gd, want + 8);
            auto root = [](double x) { return std::sqrt(x); };
            auto rcp = [](double x) { return 1.0 / x; };
            for (int t = 0; t < jastrow3_terms(N, n_nuc); ++t) {
                jastrow3_term(t, N, n_up, nuc.data(), p, at, gd, true, root, rcp, [&](int k, double v) { got[k] += v; });
                jastrow3_term(t, N, n_up, nuc.data(), p, at, gd, false, root, rcp, [&](int k, double v) { only[k] += v; });
            }
            for (int k = 0; k < 16; ++k) size = std::fmax(size, std::fabs(want[k]));
            for (int k = 0; k < 16; ++k) worst = std::fmax(worst, std::fabs(got[k] - want[k]) / size);
            for (int k = 0; k < 16; ++k) bad += only[k] != (k < 8 ? got[k] : 0.0);
        }
    }
    std::printf("%d %g\n", bad, worst);
}
"""


def test_terms_are_the_plain_sums(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    (tmp_path / "t.cpp").write_text(SOURCE)
    exe = str(tmp_path / "t")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", HEADER_DIR, str(tmp_path / "t.cpp"), "-o", exe], check=True)
    bad, worst = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert int(bad) == 0 and float(worst) <= 1e-12, (bad, worst)
