// qmc_team_kernels.cuh -- FP64 evaluation of the small shapes (H2, Li, CH4) by
// a team of G lanes per walker.
//
// An FP64 warp instruction costs the same whether 1 or 32 of its lanes work
// (qmc_fp64.cuh), so a thread per walker leaves an ensemble of a few thousand
// walkers on a few dozen warps, each with a whole walker's serial chain.  Here
// lane t of a team is electron t mod NE with every PARTS-th AO (PARTS = G / NE):
// AOs, orbitals, pair terms and the columns of the Slater matrices are spread
// over the lanes, sums over parts and electrons go through shuffles, and the
// matrices turn from rows to columns in the team's shared memory.  Derivatives
// contract the inverse's column into the MO coefficients first (c'_a = sum_k
// C[a][k] D^-1[k][q]), so an AO costs 5 + 4 multiply-adds instead of 5 per MO.
// G: 4 for H2, 8 for Li, 32 for CH4 (30 lanes busy).
#pragma once
#include <algorithm>
#include <atomic>
#include <cstring>
#include <vector>
#include "qmc_internal.h"
#include "qmc_device.cuh"

namespace qmc {

// System table of the team kernels (staged in shared memory).
template <class SH>
struct TeamTab {
    static constexpr int NPT = 3 * SH::NPRIM;
    static constexpr int NPAIR = SH::NE * (SH::NE - 1) / 2;
    static constexpr int NTERM = NPAIR + (SH::JAS == JAS_PADE_EEN ? SH::NE * SH::NNUC : 0);
    double nuc[SH::NNUC][3];
    double Z[SH::NNUC], enA[SH::NNUC], enB[SH::NNUC];
    double fnn[SH::NNUC][3];               // nuclear part of the Hellmann-Feynman force
    double F, invF, b_ee[2], a_ee[2], qa, v_nn;
    double C[2][SH::NAO][SH::NMAX];        // [sector][AO][column], AOs by falling primitive count
    double dC[SH::NROT][SH::NAO];
    double2 prim[NPT];                     // (exponent, coefficient)
    double pown[NPT];                      // Slater-type powers
    int powi[NPT];
    int ao[SH::NAO];                       // nucleus | type << 4 | primitives << 8 | first primitive << 16
    int ord[SH::NAO];                      // position here of the AOs in shell order
    int term[NTERM > 0 ? NTERM : 1];       // Jastrow value terms: i | partner << 8 | class << 16 | nucleus flag << 24
    int species[SH::NNUC];
    int rot_col[SH::NROT][2];
    int quirk_lap, n_ao, n_rot, pad;
};

template <class SH>
static bool fill_team(const HostSys& hs, TeamTab<SH>& S) {
    std::memset(&S, 0, sizeof(S));
    if (hs.N != SH::NE || hs.n_up != SH::NUP || hs.n_nuc != SH::NNUC) return false;
    if (hs.n_ao > SH::NAO || (int)hs.rot_occ.size() > SH::NROT) return false;
    // the limits of the other kernels' table (this one has room for more primitives)
    size_t prims = 0;
    for (const HostShell& sh : hs.shells) prims += sh.exps.size();
    if (hs.shells.size() > SH::NSH || prims > SH::NPRIM) return false;
    for (int I = 0; I < SH::NNUC; ++I) {
        const int sp = hs.species[I];
        for (int c = 0; c < 3; ++c) S.nuc[I][c] = hs.R[3 * I + c];
        S.Z[I] = hs.Z[I];
        S.species[I] = sp;
        S.enA[I] = hs.jas[6 + sp] * hs.Z[I];
        S.enB[I] = hs.jas[4 + sp];
        for (int J = 0; J < SH::NNUC; ++J) {
            if (J == I) continue;
            double x[3], r2 = 0.0;
            for (int c = 0; c < 3; ++c) { x[c] = hs.R[3 * I + c] - hs.R[3 * J + c]; r2 += x[c] * x[c]; }
            const double d = std::sqrt(r2);
            if (d > 1e-10)
                for (int c = 0; c < 3; ++c) S.fnn[I][c] -= hs.Z[I] * hs.Z[J] / (d * d * d) * x[c];
        }
    }
    S.F = hs.F;
    S.invF = 1.0 / hs.F;
    for (int c = 0; c < 2; ++c) { S.b_ee[c] = hs.jas[c]; S.a_ee[c] = hs.jas[2 + c]; }
    S.qa = (hs.quirks & 1) ? hs.F : 1.0;
    S.quirk_lap = (hs.quirks & 2) ? 1 : 0;
    S.v_nn = hs.v_nn;
    S.n_ao = hs.n_ao;
    S.n_rot = (int)hs.rot_occ.size();
    // AOs with their primitives (a p triplet shares one list), longest lists first
    struct Ao { int caller, packed, np; };
    std::vector<Ao> aos;
    int np = 0;
    for (const HostShell& sh : hs.shells) {
        const int n = (int)sh.exps.size();
        auto put = [&](const std::vector<double>& coef) -> int {
            const int p0 = np;
            if (np + n > TeamTab<SH>::NPT || n > 255) return -1;
            for (int p = 0; p < n; ++p, ++np) {
                S.prim[np].x = sh.exps[p];
                S.prim[np].y = coef[p];
                S.powi[np] = sh.pows.empty() ? 0 : sh.pows[p];
                S.pown[np] = S.powi[np];
            }
            return p0;
        };
        for (int k = 0; k < 2; ++k) {
            if (sh.s_ao[k] < 0) continue;
            const int p0 = put(sh.s_coef[k]);
            if (p0 < 0) return false;
            aos.push_back({sh.s_ao[k], sh.nuc | (n << 8) | (p0 << 16), n});
        }
        if (sh.p_ao[0] >= 0) {
            const int p0 = put(sh.p_coef);
            if (p0 < 0) return false;
            for (int m = 0; m < 3; ++m) aos.push_back({sh.p_ao[m], sh.nuc | ((1 + m) << 4) | (n << 8) | (p0 << 16), n});
        }
    }
    if ((int)aos.size() != hs.n_ao) return false;
    std::stable_sort(aos.begin(), aos.end(), [](const Ao& a, const Ao& b) { return a.np > b.np; });
    const std::vector<double> Ce = hs.effective_mo(), dC = hs.rotation_derivative_rows();
    for (int a = 0; a < hs.n_ao; ++a) {
        S.ao[a] = aos[a].packed;
        S.ord[hs.ao_int[aos[a].caller]] = a;
        int col[2] = {0, 0};
        for (int ei = 0; ei < hs.N; ++ei) {
            const int e = hs.perm[ei], sig = hs.spins[e] > 0 ? 0 : 1;
            S.C[sig][a][col[sig]++] = Ce[(size_t)hs.occ[e] * hs.n_ao + aos[a].caller];
        }
        for (int q = 0; q < S.n_rot; ++q) S.dC[q][a] = dC[(size_t)q * hs.n_ao + aos[a].caller];
    }
    for (int q = 0; q < S.n_rot; ++q) {
        int col[2] = {0, 0};
        S.rot_col[q][0] = S.rot_col[q][1] = -1;
        for (int ei = 0; ei < hs.N; ++ei) {
            const int e = hs.perm[ei], sig = hs.spins[e] > 0 ? 0 : 1;
            if (hs.occ[e] == hs.rot_occ[q]) S.rot_col[q][sig] = col[sig];
            ++col[sig];
        }
    }
    int n = 0;
    for (int i = 0; i < SH::NE; ++i)
        for (int j = i + 1; j < SH::NE; ++j)
            S.term[n++] = i | (j << 8) | ((((i < SH::NUP) == (j < SH::NUP)) ? 1 : 0) << 16);
    if (SH::JAS == JAS_PADE_EEN)
        for (int i = 0; i < SH::NE; ++i)
            for (int I = 0; I < SH::NNUC; ++I) S.term[n++] = i | (I << 8) | (1 << 24);
    return true;
}

// AO a at (x, y, z): value and, with MODE >= 1 / 2, gradient / Laplacian; zero
// unless ok.  LIB: the CUDA library's exponential (see team_evaluate).
template <class SH, int MODE, bool LIB = false>
__device__ __forceinline__ void team_ao(const TeamTab<SH>& S, int a, bool ok, double x, double y, double z, double& v,
                                        double& gx, double& gy, double& gz, double& l) {
    const int d = S.ao[ok ? a : 0];
    const int I = d & 15, type = (d >> 4) & 15, np = (d >> 8) & 255, p0 = d >> 16;
    const double dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    double s0 = 0, s1 = 0, s2 = 0;
    if constexpr (SH::BASIS == BASIS_GTO) {
        for (int p = p0; p < p0 + np; ++p) {
            const double2 pr = S.prim[p];
            const double f = pr.y * (LIB ? exp(-pr.x * r2) : d_exp(-pr.x * r2));
            s0 += f;
            if (MODE >= 1) {
                const double fa = pr.x * f;
                s1 += fa;
                if (MODE >= 2) s2 += pr.x * fa;
            }
        }
        // s: chi = R0, grad = -2 R1 dr, lap = -6 R1 + 4 r^2 R2; p_m: chi = x_m R0,
        // grad = x_m (-2 R1 dr) + e_m R0, lap = x_m (-10 R1 + 4 r^2 R2)
        const double ang = type == 0 ? 1.0 : (type == 1 ? dx : (type == 2 ? dy : dz));
        v = ang * s0;
        if (MODE >= 1) {
            const double g = -2.0 * s1 * ang;
            gx = g * dx + (type == 1 ? s0 : 0.0);
            gy = g * dy + (type == 2 ? s0 : 0.0);
            gz = g * dz + (type == 3 ? s0 : 0.0);
        }
        if (MODE >= 2) l = ang * ((type == 0 ? -6.0 : -10.0) * s1 + 4.0 * r2 * s2);
    } else {
        // R(r) = sum c r^n e^{-zeta r}: with t = n/r - zeta a term's derivatives
        // are f t and f (t^2 - n/r^2)
        const double r = d_sqrt(r2);
        const double id = d_positive(r) ? d_rcp(r) : 0.0;
        for (int p = p0; p < p0 + np; ++p) {
            const double2 pr = S.prim[p];
            double f = pr.y * d_exp(-pr.x * r);
            for (int m = S.powi[p]; m > 0; --m) f *= r;
            s0 += f;
            if (MODE >= 1) {
                const double nr = S.pown[p] * id, u = nr - pr.x, fu = f * u;
                s1 += fu;
                if (MODE >= 2) s2 += f * (u * u - nr * id);
            }
        }
        v = s0;
        if (MODE >= 1) {
            const double g = s1 * id;
            gx = g * dx; gy = g * dy; gz = g * dz;
            if (MODE >= 2) l = d_positive(r) ? s2 + 2.0 * g : 0.0;
        }
    }
    if (!ok) {
        v = 0;
        if (MODE >= 1) { gx = 0; gy = 0; gz = 0; }
        if (MODE >= 2) l = 0;
    }
}

// |psi| = pm 2^pe exp(u): a step compares these without a logarithm.
struct PsiAbs {
    double pm, u;
    int pe;
    __device__ __forceinline__ double log_abs() const { return d_log(pm) + (double)pe * 0.6931471805599453 + u; }
    // From log|psi| (pm = 1).
    static __device__ __forceinline__ PsiAbs of_log(double l) {
        const int pe = __float2int_rn(fminf(fmaxf((float)l * 1.44269504f, -1e6f), 1e6f));
        return {1.0, fma(-(double)pe, 0.6931471805599453, l), pe};
    }
};
// Whether uniform ua is below |a|^2 / |b|^2 (bm2 = b.pm^2).  A power of two or an
// exponential out of range by itself (a kept |psi| has its Jastrow exponent in pe, a new
// one in u) is joined with the other factor first.
__device__ __forceinline__ bool below_ratio2(double ua, const PsiAbs& a, const PsiAbs& b, double bm2) {
    const double t = 2.0 * (a.u - b.u);
    const int k = 2 * (a.pe - b.pe);
    // (two calls: one with joined arguments took 6.48 ms for 20-walker CH4 sampling, 6.34 so)
    if ((unsigned)(k + 900) <= 1800u && (d_hi(t) & 0x7fffffff) < 0x40860000)         // |t| < 704
        return ua * bm2 < a.pm * a.pm * __hiloint2double((1023 + k) << 20, 0) * d_exp(t);
    return ua * bm2 < a.pm * a.pm * d_exp(fma((double)k, 0.6931471805599453, t));
}

// Lanes of a walker (team) and the pieces of an evaluation.
template <class SH, int G>
struct Team {
    static constexpr int NE = SH::NE, NM = SH::NMAX, NUP = SH::NUP, NDN = SH::NDN, NNUC = SH::NNUC;
    static constexpr int PARTS = G / NE, SLOTS = (SH::NAO + PARTS - 1) / PARTS;
    static constexpr int ROUNDS = (NE + NNUC + PARTS - 1) / PARTS;
    static constexpr int ROWS = NE * NM;               // shared doubles of a team
    using Tab = TeamTab<SH>;
    static_assert(PARTS >= 1 && G <= 32 && (G & (G - 1)) == 0, "a team is a power of two of lanes, one or more per electron");

    int base, t, e, part, sig, q;
    bool on;                                            // spare lanes copy an electron and add nothing

    __device__ __forceinline__ Team() {
        const int lane = threadIdx.x & 31;
        base = lane & ~(G - 1);
        t = lane - base;
        on = t < NE * PARTS;
        e = t % NE;
        part = on ? t / NE : 0;
        sig = e < NUP ? 0 : 1;
        q = e - sig * NUP;
    }
    static __device__ __forceinline__ double shfl(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
    static __device__ __forceinline__ int shfl(int v, int src) { return __shfl_sync(0xffffffffu, v, src); }
    // Sum over the team (the same bits on every lane).
    static __device__ __forceinline__ double sum(double v) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }
    // Sum over the parts of the lane's electron.
    __device__ __forceinline__ double part_sum(double v) const {
        double r = v;
#pragma unroll
        for (int d = 1; d < PARTS; ++d) {
            int p = part + d;
            p = p >= PARTS ? p - PARTS : p;
            r += shfl(v, base + e + NE * p);
        }
        return r;
    }

    // AO of this lane's slot at (x, y, z) (zero past the basis).
    template <bool DER, bool LIB = false>
    __device__ __forceinline__ void ao(const Tab& S, int slot, double x, double y, double z, double& v, double& gx,
                                       double& gy, double& gz, double& l) const {
        const int a = slot * PARTS + part;
        team_ao<SH, DER ? 2 : 0, LIB>(S, a, on && a < S.n_ao, x, y, z, v, gx, gy, gz, l);
    }

    // Determinants of both sectors from the electrons' orbital rows v (part 0's),
    // by elimination with partial pivoting on lane-columns; with INV in place, so
    // that w[k] = D^-1[k][q] of the lane's electron.  |det| = pm 2^pe.  READY: the rows
    // are in sh already (and pivots are inverted by a division).
    template <bool INV, bool READY = false>
    __device__ __forceinline__ void det(const double (&v)[NM], double* sh, double (&w)[NM], double& pm, int& pe,
                                        int& sg, bool& ok) const {
        if (!READY && on && part == 0) {
#pragma unroll
            for (int k = 0; k < NM; ++k) sh[e * NM + k] = v[k];
        }
        __syncwarp();
        const int NS = sig == 0 ? NUP : NDN, s0 = base + sig * NUP;
#pragma unroll
        for (int i = 0; i < NM; ++i) w[i] = i < NS ? sh[(sig * NUP + (i < NS ? i : 0)) * NM + q] : 0.0;
        __syncwarp();
        double m = 1.0;
        int ex = 0, s = 0, src = q;
        bool good = true;
#pragma unroll
        for (int k = 0; k < NM; ++k) {
            const bool step = NUP == NDN || k < NS;
            const int from = s0 + (step ? k : 0);
            int p = k, best = pivot_mag(w[k]);
#pragma unroll
            for (int i = k + 1; i < NM; ++i) {
                const int a = pivot_mag(w[i]);
                if ((NUP == NDN || i < NS) && a > best) { best = a; p = i; }
            }
            p = shfl(p, from);
            if (!step) p = k;
#pragma unroll
            for (int i = k + 1; i < NM; ++i) {
                const bool sw = i == p;
                const double a = w[k], b = w[i];
                w[k] = sw ? b : a;
                w[i] = sw ? a : b;
            }
            s ^= p != k;
            src = src == k ? p : (src == p ? k : src);
            double piv = shfl(w[k], from);
            if (step && ((d_hi(piv) & 0x7fffffff) | d_lo(piv)) == 0) { good = false; piv = 1.0; }
            if (!step) piv = 1.0;
            s ^= d_hi(piv) < 0;
            m *= fabs(piv);
            const int be = (d_hi(m) >> 20) & 0x7ff;
            if (be != 0 && be != 0x7ff) {
                ex += be - 1023;
                m = d_scale(m, 1023 - be);
            }
            if (INV || k + 1 < NM) {
                const double ip = READY ? 1.0 / piv : d_rcp_full(piv);
                if (INV) {
                    const bool own = q == k;
                    const double x = own ? ip : w[k] * ip;
#pragma unroll
                    for (int i = 0; i < NM; ++i) {
                        if (i == k) continue;
                        const double f = shfl(w[i], from);
                        const double r = fma(-f, x, own ? 0.0 : w[i]);
                        w[i] = step ? r : w[i];
                    }
                    w[k] = step ? x : w[k];
                } else {
#pragma unroll
                    for (int i = k + 1; i < NM; ++i) {
                        const double f = shfl(w[i], from) * ip;
                        w[i] = step ? fma(-f, w[k], w[i]) : w[i];
                    }
                }
            }
        }
        if (INV) {
#pragma unroll
            for (int k = 0; k < NM; ++k) w[k] = shfl(w[k], s0 + src);
        }
        pm = shfl(m, base) * (NDN > 0 ? shfl(m, base + NUP) : 1.0);
        pe = shfl(ex, base) + (NDN > 0 ? shfl(ex, base + NUP) : 0);
        s = shfl(s, base) ^ (NDN > 0 ? shfl(s, base + NUP) : 0);
        // every lane takes both shuffles: a team with a singular matrix that skipped the second
        // would leave the warp's other teams waiting in it
        const int g = good, g0 = shfl(g, base), g1 = NDN > 0 ? shfl(g, base + NUP) : 1;
        ok = g0 != 0 && g1 != 0;
        sg = s ? -1 : 1;
    }
    // Jastrow u alone: the pairs and electron-nucleus terms spread over the lanes.
    __device__ __forceinline__ double jastrow_value(const Tab& S, double x, double y, double z) const {
        double u = 0;
#pragma unroll
        for (int r = 0; r < (Tab::NTERM + G - 1) / G; ++r) {
            const int p = t + G * r;
            const bool ok = p < Tab::NTERM;
            const int d = S.term[ok ? p : 0];
            const int i = d & 255, b = (d >> 8) & 255, c = (d >> 16) & 255;
            const bool en = (d >> 24) != 0;
            const int j = base + (en ? 0 : b), I = en ? b : 0;
            double xj = shfl(x, j), yj = shfl(y, j), zj = shfl(z, j);
            if (en) { xj = S.nuc[I][0]; yj = S.nuc[I][1]; zj = S.nuc[I][2]; }
            const double dx = shfl(x, base + i) - xj, dy = shfl(y, base + i) - yj, dz = shfl(z, base + i) - zj;
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double ri = d_positive(r2) ? d_rsqrt(r2) : 0.0;
            double uu;
            if (SH::JAS == JAS_PADE_F) {
                uu = -0.5 * S.F * d_rcp(1.0 + r2 * ri * S.invF);
            } else {
                const double pa = en ? -S.enA[I] : S.a_ee[c], pb = en ? S.enB[I] : S.b_ee[c];
                uu = d_positive(r2) ? pa * d_rcp(pb + ri) : 0.0;
            }
            u += ok ? uu : 0.0;
        }
        return sum(u);
    }

    // Partner m of the lane's electron in round r of the full pair pass: electrons,
    // then nuclei.  Returns whether the term counts.
    __device__ __forceinline__ bool partner(const Tab& S, int r, double x, double y, double z, bool& el, int& m,
                                            int& I, double& dx, double& dy, double& dz, double& r2) const {
        m = part + PARTS * r;
        el = m < NE;
        I = m >= NE && m < NE + NNUC ? m - NE : 0;
        const int j = base + (el ? m : 0);
        double xj = shfl(x, j), yj = shfl(y, j), zj = shfl(z, j);
        if (!el) { xj = S.nuc[I][0]; yj = S.nuc[I][1]; zj = S.nuc[I][2]; }
        dx = x - xj; dy = y - yj; dz = z - zj;
        const bool ok = on && m < NE + NNUC && m != e;
        r2 = dx * dx + dy * dy + dz * dz;
        r2 = ok ? r2 : 1.0;
        return ok;
    }

    // The electron's Jastrow gradient g, Laplacian lu and squared-gradient sum gsq
    // (all parts), this lane's share of u and V; term(...) sees every partner.
    template <class Term>
    __device__ __forceinline__ void jastrow_full(const Tab& S, double x, double y, double z, double (&g)[3], double& lu,
                                                 double& gsq, double& u, double& V, Term term) const {
        g[0] = g[1] = g[2] = 0; lu = 0; gsq = 0; u = 0; V = 0;
#pragma unroll 1
        for (int r = 0; r < ROUNDS; ++r) {
            bool el;
            int m, I;
            double dx, dy, dz, r2;
            const bool ok = partner(S, r, x, y, z, el, m, I, dx, dy, dz, r2);
            double d, ri;
            dist(r2, d, ri);
            V += ok ? (el ? 0.5 : -S.Z[I]) * ri : 0.0;
            // nuclei alone in a round, and no electron-nucleus Jastrow terms
            if (SH::JAS == JAS_PADE_F && PARTS * r >= NE) continue;
            double inv = 0, f = 0, l = 0, uu = 0, up = 0;
            const int c = (m < NUP) == (e < NUP) ? 1 : 0;
            if (SH::JAS == JAS_PADE_EEN) {
                const double a = el ? S.a_ee[c] : -S.enA[I], b = el ? S.b_ee[c] : S.enB[I];
                inv = d_rcp(1.0 + b * d);
                uu = a * d * inv;
                up = a * inv * inv;
                f = up * ri;
                l = 2.0 * (f - up * b * inv);
                u += ok ? (el ? 0.5 : 1.0) * uu : 0.0;
            } else {
                inv = d_rcp(1.0 + d * S.invF);
                up = 0.5 * inv * inv;
                f = up * ri;
                l = inv * inv * inv * ri;
                uu = -0.25 * S.F * inv;                 // half of the pair, seen from both ends
                u += ok && el ? uu : 0.0;
            }
            const bool near = SH::JAS == JAS_PADE_EEN ? d_below(d, 1e-10) : !d_positive(d);
            const bool use = ok && !near && (SH::JAS == JAS_PADE_EEN || el);
            f = use ? f : 0.0;
            g[0] += f * dx; g[1] += f * dy; g[2] += f * dz;
            lu += use ? l : 0.0;
            if (S.quirk_lap) gsq += use ? up * up : 0.0;
            term(ok, near, el, m, I, c, dx, dy, dz, d, ri, inv);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) g[c] = part_sum(g[c]);
        lu = part_sum(lu);
        if (S.quirk_lap) gsq = part_sum(gsq);
    }
};

// Whole-block copy of a table into shared memory (ends with a block barrier).
template <class TAB>
__device__ __forceinline__ void stage_team(TAB* dst, const TAB* __restrict__ src) {
    static_assert(sizeof(TAB) % 8 == 0, "tables are whole doubles");
    const double* s = reinterpret_cast<const double*>(src);
    double* d = reinterpret_cast<double*>(dst);
    for (int i = threadIdx.x; i < (int)(sizeof(TAB) / 8); i += blockDim.x) d[i] = s[i];
    __syncthreads();
}

// |psi| and sign at the team's positions; ok false for a singular matrix.
template <class SH, int G>
__device__ __forceinline__ PsiAbs team_psi(const Team<SH, G>& T, const TeamTab<SH>& S, double* sh, double x, double y,
                                           double z, int& sg, bool& ok) {
    using TM = Team<SH, G>;
    double v[TM::NM], w[TM::NM], u0, u1, u2, u3;
#pragma unroll
    for (int k = 0; k < TM::NM; ++k) v[k] = 0;
#pragma unroll 1
    for (int s = 0; s < TM::SLOTS; ++s) {
        double chi;
        T.template ao<false>(S, s, x, y, z, chi, u0, u1, u2, u3);
        const int a = min(s * TM::PARTS + T.part, SH::NAO - 1);
#pragma unroll
        for (int k = 0; k < TM::NM; ++k) v[k] += S.C[T.sig][a][k] * chi;
    }
#pragma unroll
    for (int k = 0; k < TM::NM; ++k) v[k] = T.part_sum(v[k]);
    PsiAbs a;
    T.template det<false>(v, sh, w, a.pm, a.pe, sg, ok);
    a.u = T.jastrow_value(S, x, y, z);
    return a;
}

// a[q] of a register array.
template <int N>
__device__ __forceinline__ double pick(const double (&a)[N], int q) {
    double r = a[0];
#pragma unroll
    for (int i = 1; i < N; ++i) r = i == q ? a[i] : r;
    return r;
}

// Full evaluation.  NR: MO-rotation rows, DEL: with dE_L/dp, FORCE: with forces;
// `red` is the team's [32][RED] reduction scratch of those.  LIB (Gaussian bases; `chi`
// is the team's [NE][NAO] scratch): the orbital matrix with the CUDA library's
// exponential and every element's sum in AO order by one lane, and pivots inverted by
// a division -- the rounding of a thread per walker.  Configurations next to a node
// amplify the matrix's rounding: over 60 sets of 5000 CH4 configurations another order
// moved SR rows by 7e-12 of their norm in the median and 6.5e-9 at worst.
struct TeamOut {
    double* grad;                          // [N][3] of this walker, or null
    double* lap;
    double* O;                             // [P]
    double* dEL;                           // [P]
    double* fhf;                           // [n_nuc][3]
    double* omega;
};

template <class SH, int G, int NR, bool DEL, bool FORCE, bool LIB, class Store>
__device__ __forceinline__ double team_evaluate(const Team<SH, G>& T, const TeamTab<SH>& S, double* sh, double* red, double* chis,
                                                double x, double y, double z, PsiAbs& psi, int& sg, bool& ok,
                                                const TeamOut& out, bool act, Store store) {
    using TM = Team<SH, G>;
    constexpr int NM = TM::NM, NNUC = TM::NNUC, SLOTS = TM::SLOTS;
    constexpr int NRa = NR > 0 ? NR : 1;
    constexpr int NQ = NR > 0 ? 8 + NR : 1, NF = FORCE ? 3 * NNUC : 1;
    static_assert(!(NR > 0 && FORCE), "one kind of extra output at a time");
    constexpr bool EXTRA = NR > 0 || FORCE;
    constexpr int RED = FORCE ? NF : NQ;
    double* mine = red + (EXTRA ? T.t * RED : 0);
    if (EXTRA) {
#pragma unroll
        for (int i = 0; i < RED; ++i) mine[i] = 0.0;
    }
    double v[NM], w[NM], dv[NRa];
    double ax[SLOTS], ay[SLOTS], az[SLOTS], al[SLOTS];
#pragma unroll
    for (int k = 0; k < NM; ++k) v[k] = 0;
#pragma unroll
    for (int q = 0; q < NRa; ++q) dv[q] = 0;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
        double chi;
        T.template ao<true, LIB>(S, s, x, y, z, chi, ax[s], ay[s], az[s], al[s]);
        const int a = min(s * TM::PARTS + T.part, SH::NAO - 1);
        if constexpr (LIB) {
            if (T.on && s * TM::PARTS + T.part < S.n_ao) chis[T.e * SH::NAO + a] = chi;
        } else {
#pragma unroll
            for (int k = 0; k < NM; ++k) v[k] += S.C[T.sig][a][k] * chi;
        }
        if (NR > 0) {
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (q < S.n_rot) dv[q] += S.dC[q][a] * chi;
        }
    }
    if constexpr (LIB) {
        __syncwarp();
        constexpr int KP = (NM + TM::PARTS - 1) / TM::PARTS;        // columns part, part + PARTS, ... of the row
        double vk[KP];
#pragma unroll
        for (int i = 0; i < KP; ++i) vk[i] = 0;
#pragma unroll 1
        for (int i = 0; i < S.n_ao; ++i) {
            const int a = S.ord[i];
            const double chi = chis[T.e * SH::NAO + a];
#pragma unroll
            for (int c = 0; c < KP; ++c) vk[c] += S.C[T.sig][a][min(T.part + TM::PARTS * c, NM - 1)] * chi;
        }
#pragma unroll
        for (int c = 0; c < KP; ++c)
            if (T.on && T.part + TM::PARTS * c < NM) sh[T.e * NM + T.part + TM::PARTS * c] = vk[c];
    } else {
#pragma unroll
        for (int k = 0; k < NM; ++k) v[k] = T.part_sum(v[k]);
    }
    T.template det<true, LIB>(v, sh, w, psi.pm, psi.pe, sg, ok);
    store(w);
    // grad ln D and lap D / D of the electron from c'_a
    double gx = 0, gy = 0, gz = 0, ld = 0;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
        const int a = min(s * TM::PARTS + T.part, SH::NAO - 1);
        double c = 0;
#pragma unroll
        for (int k = 0; k < NM; ++k) c += S.C[T.sig][a][k] * w[k];
        if (FORCE) {
            const int I = S.ao[a] & 15;
            const double tx = c * ax[s], ty = c * ay[s], tz = c * az[s];
            gx += tx; gy += ty; gz += tz;
            mine[3 * I] -= tx; mine[3 * I + 1] -= ty; mine[3 * I + 2] -= tz;
        } else {
            gx += c * ax[s]; gy += c * ay[s]; gz += c * az[s];
        }
        ld += c * al[s];
    }
    gx = T.part_sum(gx); gy = T.part_sum(gy); gz = T.part_sum(gz); ld = T.part_sum(ld);
    double g[3], lu, gsq, u, V;
    T.jastrow_full(S, x, y, z, g, lu, gsq, u, V,
                   [&](bool use, bool near, bool el, int m, int I, int c, double dx, double dy, double dz, double d,
                       double ri, double inv) {
        if (NR > 0) {
            // du/db = -a (r/(1+br))^2, du/da = r/(1+br) per pair (half from each
            // end), du/dB = A Z (...)^2, du/dA = -Z ... per nucleus
            const double full = fma(fma(-(1.0 + (el ? S.b_ee[c] : S.enB[I]) * d), inv, 1.0), inv, inv);
            const double s1 = d * full;
            const int k = el ? c : 4 + S.species[I];
            const double fb = el ? -0.5 * S.a_ee[c] : S.enA[I], fa = el ? 0.5 : -S.Z[I];
            if (use) {
                mine[k] += fb * s1 * s1;
                mine[k + 2] += fa * s1;
            }
        }
        if (FORCE) {
            // Jastrow part of d ln|psi| / dR_I
            if (use && !near && !el && SH::JAS == JAS_PADE_EEN) {
                // (full precision: ri and inv are one Newton step, 1e-14 each)
                const double r = d_sqrt(dx * dx + dy * dy + dz * dz), den = 1.0 + S.enB[I] * r;
                const double f = S.enA[I] * d_rcp_full(r * den * den);
                mine[3 * I] += f * dx; mine[3 * I + 1] += f * dy; mine[3 * I + 2] += f * dz;
            }
        }
    });
    if (NR > 0) {
        // rotation rows: d ln|D| / d theta = sum_q psi(r_q) D^-1[c][q]
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            if (q >= S.n_rot) break;
            dv[q] = T.part_sum(dv[q]);
            if (T.on && T.part == 0) {
                const int c = S.rot_col[q][T.sig];
                double b = 0;
#pragma unroll
                for (int k = 0; k < NM; ++k) b = k == c ? w[k] : b;
                mine[8 + q] += b * dv[q];
            }
        }
    }
    const double qx = S.qa * g[0], qy = S.qa * g[1], qz = S.qa * g[2];
    const double lj = S.quirk_lap ? lu + gsq : lu + g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
    const double lp = ld + 2.0 * (gx * qx + gy * qy + gz * qz) + lj;
    const bool first = T.on && T.part == 0;
    if (act && first) {
        if (out.grad) {
            out.grad[3 * T.e] = gx + qx; out.grad[3 * T.e + 1] = gy + qy; out.grad[3 * T.e + 2] = gz + qz;
        }
        if (out.lap) out.lap[T.e] = lp;
    }
    const double e_l = TM::sum(V - (first ? 0.5 * lp : 0.0)) + S.v_nn;
    psi.u = TM::sum(u);
    // sums over the lanes' rows of red, column by column (a whole warp: half of
    // the rows by lane p and half by lane p + 16)
    auto reduce = [&](int n, double* to, auto map) {
        __syncwarp();
        if constexpr (G == 32) {
            const int p = T.t & 15, h = T.t & 16;
            double s = 0;
            if (p < n) {
#pragma unroll 4
                for (int i = 0; i < 16; ++i) s += red[(h + i) * RED + p];
            }
            s += __shfl_xor_sync(0xffffffffu, s, 16);
            if (act && to && p < n && T.t < 16) to[p] = map(s, p);
        } else {
            for (int p = T.t; p < n; p += G) {
                double s = 0;
#pragma unroll
                for (int i = 0; i < G; ++i) s += red[i * RED + p];
                if (act && to) to[p] = map(s, p);
            }
        }
        __syncwarp();
    };
    if constexpr (NR > 0) {
        static_assert(NQ <= 16 || G < 32, "a half-warp holds the parameters");
        reduce(8 + S.n_rot, out.O, [](double s, int) { return s; });
        if constexpr (DEL) {
            // Jastrow columns: -1/2 sum over both ends of [ l + 2 f G_i . dr ] with the
            // parameter derivatives f of u'/r and l of u'' + 2u'/r (EEN forms)
#pragma unroll
            for (int i = 0; i < RED; ++i) mine[i] = 0.0;
            const double Gx = gx + qx, Gy = gy + qy, Gz = gz + qz;
#pragma unroll 1
            for (int r = 0; r < TM::ROUNDS; ++r) {
                bool el;
                int m, I;
                double dx, dy, dz, r2, d, ri;
                const bool use = T.partner(S, r, x, y, z, el, m, I, dx, dy, dz, r2);
                dist(r2, d, ri);
                const int c = (m < TM::NUP) == (T.e < TM::NUP) ? 1 : 0;
                const double b = el ? S.b_ee[c] : S.enB[I], a = el ? S.a_ee[c] : -S.enA[I];
                const double i1 = recip_full(1.0 + b * d), i2 = i1 * i1, i3 = i2 * i1;
                // f = -2 a i3, l = 3 f i1 for b; f = s i2 / r, l = 2 f - 2 s b i3 for a
                const double ms = el ? -1.0 : S.Z[I];
                const double h = Gx * dx + Gy * dy + Gz * dz;
                const int k = el ? c : 4 + S.species[I];
                if (use && !d_below(d, 1e-10)) {
                    mine[k] += a * i3 * fma(3.0, i1, 2.0 * h);
                    mine[k + 2] += ms * fma(i2 * ri, 1.0 + h, -b * i3);
                }
            }
            // rotation columns: with beta = D^-1 psi (over the sector's rows) and
            // d_a = sum_k C[a][k] beta_k - dC[a], sum_a d_a X_a = sum_k X_k beta_k - X_psi
#pragma unroll 1
            for (int q = 0; q < NR; ++q) {
                if (q >= S.n_rot) break;
                const int c = S.rot_col[q][T.sig];
                if (first) {
#pragma unroll
                    for (int k = 0; k < NM; ++k) sh[T.e * NM + k] = w[k] * pick(dv, q);
                }
                __syncwarp();
                double beta = 0, bc = 0, tx = 0, ty = 0, tz = 0, tl = 0, bk[NM];
                const int NS = T.sig == 0 ? TM::NUP : TM::NDN;
#pragma unroll
                for (int i = 0; i < NM; ++i)
                    if (i < NS) beta += sh[(T.sig * TM::NUP + i) * NM + T.q];
#pragma unroll
                for (int k = 0; k < NM; ++k) {
                    bk[k] = TM::shfl(beta, T.base + T.sig * TM::NUP + (k < NS ? k : 0));
                    bk[k] = k < NS ? bk[k] : 0.0;
                    bc = k == c ? w[k] : bc;
                }
#pragma unroll
                for (int s = 0; s < SLOTS; ++s) {
                    const int a = min(s * TM::PARTS + T.part, SH::NAO - 1);
                    double da = -S.dC[q][a];
#pragma unroll
                    for (int k = 0; k < NM; ++k) da += S.C[T.sig][a][k] * bk[k];
                    tx += da * ax[s]; ty += da * ay[s]; tz += da * az[s]; tl += da * al[s];
                }
                // linear in the AO sums: the reduction adds the parts
                if (T.on && c >= 0) mine[8 + q] += 0.5 * bc * (tl + 2.0 * (tx * g[0] + ty * g[1] + tz * g[2]));
                __syncwarp();
            }
            reduce(8 + S.n_rot, out.dEL, [](double s, int) { return s; });
        }
    }
    if constexpr (FORCE) {
        static_assert(NF <= 16 || G < 32, "a half-warp holds the components");
        reduce(NF, out.omega, [](double s, int) { return s; });
        // Hellmann-Feynman: Z (r - R) / |r - R|^3 of every electron and nucleus
#pragma unroll
        for (int i = 0; i < RED; ++i) mine[i] = 0.0;
#pragma unroll 1
        for (int I = T.part; I < NNUC; I += TM::PARTS) {
            const double dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
            const double r2 = dx * dx + dy * dy + dz * dz;
            const double r = d_sqrt(r2);
            if (T.on && !d_below(r, 1e-10)) {
                const double f = S.Z[I] * d_rcp_full(r2 * r);
                mine[3 * I] += f * dx; mine[3 * I + 1] += f * dy; mine[3 * I + 2] += f * dz;
            }
        }
        reduce(NF, out.fhf, [&](double s, int p) { return s + S.fnn[p / 3][p % 3]; });
    }
    return e_l;
}


// Compensated sum of v over the block's teams (v on every lane of a team) into
// partial[2 slot], partial[2 slot + 1]; ends with a block barrier.
template <int G, int TPB>
__device__ __forceinline__ void team_block_partial(double v, double* partial, int slot) {
    constexpr int N = TPB / G;
    __shared__ double ps[N];
    if (threadIdx.x % G == 0) ps[threadIdx.x / G] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        Comp c{(int)threadIdx.x < N ? ps[threadIdx.x] : 0.0, 0.0};
#pragma unroll
        for (int o = N / 2; o > 0; o >>= 1)
            c = comp_add(c, Comp{__shfl_down_sync(0xffffffffu, c.s, o), __shfl_down_sync(0xffffffffu, c.c, o)});
        if (threadIdx.x == 0) { partial[2 * slot] = c.s; partial[2 * slot + 1] = c.c; }
    }
    __syncthreads();
}

// All-electron Metropolis steps of FP64 walkers (src/sampling/vmc.rs:95-119),
// a team per walker.  A step needs log|psi| alone; with REC the E_L of every
// step is recorded (per-block compensated sums in partial[step][block]),
// otherwise E_L is evaluated once, at the final configuration.
constexpr int TEAM_REC = 32;               // steps between reductions of the recorded energies

template <class SH, int G, int MOVE, bool REC, int TPB>
__global__ void __launch_bounds__(TPB) k_team_steps(const TeamTab<SH>* __restrict__ tab, double* __restrict__ gpos,
                                                    double* __restrict__ glog, int* __restrict__ gsign,
                                                    double* __restrict__ gel, int W, int Wcap, int n_steps,
                                                    uint64_t step0, double step, uint64_t seed,
                                                    unsigned long long* acc_out, double* partial, int nblk, int* flags) {
    using TM = Team<SH, G>;
    constexpr int NT = TPB / G;
    __shared__ TeamTab<SH> S;
    __shared__ double rows[NT][TM::ROWS];
    __shared__ double rec[REC ? TEAM_REC : 1][REC ? NT : 1];
    stage_team(&S, tab);
    const TM T;
    const int tm = threadIdx.x / G, w = blockIdx.x * NT + tm;
    const bool act = w < W;
    double* sh = rows[tm];
    double x, y, z;
    {
        const size_t i = (size_t)(3 * T.e) * Wcap + w;
        x = act ? gpos[i] : (T.e + 1) * 0.37;
        y = act ? gpos[i + Wcap] : (T.e + 1) * 1.37;
        z = act ? gpos[i + 2 * (size_t)Wcap] : (T.e + 1) * 2.37;
    }
    PsiAbs cur = PsiAbs::of_log(act ? glog[w] : 0.0);
    double pm2 = 1.0;                          // cur.pm^2
    int sg = act ? gsign[w] : 1;
    double el = act ? gel[w] : 0.0;
    unsigned acc = 0;
    int flg = 0;
    const TeamOut none{};
    auto nostore = [](const double (&)[TM::NM]) {};
    for (int it = 0; it < n_steps; ++it) {
        const uint64_t st = step0 + (uint64_t)it;
        const U4 r = rng_draw(seed, (uint32_t)w, st, (uint32_t)T.e, TAG_PROPOSE);
        double nx, ny, nz;
        if (MOVE == MOVE_ALL_GAUSS) {
            // (x, y) from the first Box-Muller pair, z from the second: one pair
            // per lane where an electron has two parts
            double n0, n1, n2, n3;
            if constexpr (TM::PARTS >= 2) {
                bm(T.part == 0 ? r.x : r.z, T.part == 0 ? r.y : r.w, n0, n1);
                n2 = TM::shfl(n0, T.base + T.e + TM::NE);
                n0 = TM::shfl(n0, T.base + T.e);
                n1 = TM::shfl(n1, T.base + T.e);
            } else {
                bm(r.x, r.y, n0, n1);
                bm(r.z, r.w, n2, n3);
            }
            nx = x + step * n0; ny = y + step * n1; nz = z + step * n2;
        } else {
            nx = x + step * (d_u32(r.x) - 0.5);
            ny = y + step * (d_u32(r.y) - 0.5);
            nz = z + step * (d_u32(r.z) - 0.5);
        }
        PsiAbs next;
        double en = 0;
        int sn;
        bool ok;
        if constexpr (REC)
            en = team_evaluate<SH, G, 0, false, false, false>(T, S, sh, nullptr, nullptr, nx, ny, nz, next, sn, ok, none, false, nostore);
        else
            next = team_psi(T, S, sh, nx, ny, nz, sn, ok);
        const U4 a = rng_draw(seed, (uint32_t)w, st, 0, TAG_ACCEPT);
        const int take = act && ok && below_ratio2(d_u32(a.x), next, cur, pm2);
        if (TM::shfl(take, T.base)) {
            x = nx; y = ny; z = nz;
            cur = next;
            pm2 = next.pm * next.pm;
            sg = sn;
            ++acc;
            if (REC) {
                el = en;
                if (!isfinite(el)) flg |= FLAG_NONFINITE;
            }
        }
        if constexpr (REC) {
            const int row = it % TEAM_REC;
            if (T.t == 0) rec[row][tm] = act ? el : 0.0;
            if (row == TEAM_REC - 1 || it == n_steps - 1) {
                __syncthreads();
                if ((int)threadIdx.x <= row) {
                    Comp c{0.0, 0.0};
                    for (int i = 0; i < NT; ++i) c = comp_add(c, Comp{rec[threadIdx.x][i], 0.0});
                    double* o = partial + 2 * ((size_t)(it - row + (int)threadIdx.x) * nblk + blockIdx.x);
                    o[0] = c.s;
                    o[1] = c.c;
                }
                __syncthreads();
            }
        }
    }
    if (!REC && __any_sync(0xffffffffu, acc > 0)) {
        PsiAbs again;
        int sn;
        bool ok;
        const double en = team_evaluate<SH, G, 0, false, false, false>(T, S, sh, nullptr, nullptr, x, y, z, again, sn, ok, none, false, nostore);
        if (acc) {
            el = en;
            if (!isfinite(el)) flg |= FLAG_NONFINITE;
        }
    }
    if (act) {
        if (T.on && T.part == 0) {
            const size_t i = (size_t)(3 * T.e) * Wcap + w;
            gpos[i] = x;
            gpos[i + Wcap] = y;
            gpos[i + 2 * (size_t)Wcap] = z;
        }
        if (T.t == 0) {
            if (acc) glog[w] = cur.log_abs();
            gsign[w] = sg;
            gel[w] = el;
            if (acc) atomicAdd(acc_out, (unsigned long long)acc);
            if (flg) atomicOr(flags, flg);
        }
    }
}

// Shared doubles of a team's reduction rows.
template <class SH, int G, int NR, bool FORCE>
__host__ __device__ constexpr int team_red() { return NR > 0 ? G * (8 + NR) : (FORCE ? G * 3 * SH::NNUC : 1); }

// Whether an evaluation keeps a thread per walker's rounding (team_evaluate): SR rows,
// whose derivatives amplify it most (5000 configurations 461 us through the host call,
// 440 us without).  Forces would pay more (531 and 434 us) for less: 60 sets moved by
// 3e-12 in the median and 4e-10 at worst.
template <class SH, int NR>
__host__ __device__ constexpr bool team_lib() { return SH::BASIS == BASIS_GTO && NR > 0; }
template <class SH, int NR>
__host__ __device__ constexpr int team_chi() { return team_lib<SH, NR>() ? SH::NE * SH::NAO : 1; }

// Refresh or evaluation of walker w by its team; E_L (0 for an idle team).
template <class SH, int G, int NR, bool DEL, bool FORCE>
__device__ __forceinline__ double team_measure(const Team<SH, G>& T, const TeamTab<SH>& S, double* sh, double* red, double* chis,
                                               const double* __restrict__ pos, double* __restrict__ dinv,
                                               double* __restrict__ logabs, int* __restrict__ sign,
                                               double* __restrict__ el, int w, bool act, int Wcap, int write_state,
                                               const MeasureOut& mo, int P, int* flags) {
    using TM = Team<SH, G>;
    const size_t i = (size_t)(3 * T.e) * Wcap + w;
    const double x = act ? pos[i] : (T.e + 1) * 0.37, y = act ? pos[i + Wcap] : (T.e + 1) * 1.37,
                 z = act ? pos[i + 2 * (size_t)Wcap] : (T.e + 1) * 2.37;
    TeamOut out{};
    if (mo.grad) out.grad = mo.grad + (size_t)w * 3 * SH::NE;
    if (mo.lap) out.lap = mo.lap + (size_t)w * SH::NE;
    if (NR > 0 && mo.O) out.O = mo.O + (size_t)w * P;
    if (DEL && mo.dEL) out.dEL = mo.dEL + (size_t)w * P;
    if (FORCE && mo.fhf) out.fhf = mo.fhf + (size_t)w * 3 * SH::NNUC;
    if (FORCE && mo.omega) out.omega = mo.omega + (size_t)w * 3 * SH::NNUC;
    const bool first = T.on && T.part == 0;
    auto store = [&](const double (&d)[TM::NM]) {
        if (!act || !write_state || !first) return;
        const int NS = T.sig == 0 ? TM::NUP : TM::NDN;
#pragma unroll
        for (int k = 0; k < TM::NM; ++k)
            if (k < NS) dinv[((size_t)(T.sig * TM::NM * TM::NM + k * TM::NM + T.q)) * Wcap + w] = d[k];
    };
    PsiAbs psi;
    int sg;
    bool ok;
    const double e = team_evaluate<SH, G, NR, DEL, FORCE, team_lib<SH, NR>()>(T, S, sh, red, chis, x, y, z, psi, sg, ok, out, act, store);
    if (act && T.t == 0) {
        int fl = 0;
        if (!ok) fl |= FLAG_SINGULAR;
        if (!isfinite(e)) fl |= FLAG_NONFINITE;
        if (fl) atomicOr(flags, fl);
        if (write_state) { logabs[w] = psi.log_abs(); sign[w] = sg; el[w] = e; }
    }
    return act ? e : 0.0;
}

template <class SH, int G, int NR, bool DEL, bool FORCE, int TPB>
__global__ void __launch_bounds__(TPB) k_team_measure(const TeamTab<SH>* __restrict__ tab,
                                                      const double* __restrict__ pos, double* __restrict__ dinv,
                                                      double* __restrict__ logabs, int* __restrict__ sign,
                                                      double* __restrict__ el, int W, int Wcap, int write_state,
                                                      MeasureOut out, int P, double* partial, int* flags) {
    using TM = Team<SH, G>;
    constexpr int NT = TPB / G;
    __shared__ TeamTab<SH> S;
    __shared__ double rows[NT][TM::ROWS];
    __shared__ double red[NT][team_red<SH, G, NR, FORCE>()];
    __shared__ double chis[NT][team_chi<SH, NR>()];
    stage_team(&S, tab);
    const TM T;
    const int tm = threadIdx.x / G, w = blockIdx.x * NT + tm;
    const double e = team_measure<SH, G, NR, DEL, FORCE>(T, S, rows[tm], red[tm], chis[tm], pos, dinv, logabs, sign, el, w, w < W,
                                                         Wcap, write_state, out, P, flags);
    if (partial) team_block_partial<G, TPB>(e, partial, blockIdx.x);
}

// Batched refresh: a block of TPB threads takes a tile of TW walkers, TPB / G at
// a time; the tile's energies are summed in the order of its walkers.
template <class SH, int G, int TPB, int TW>
__global__ void __launch_bounds__(TPB) kb_team_measure(const BatchTile* __restrict__ tiles, int ntiles,
                                                       const BatchRec* __restrict__ recs, double* tile_partial) {
    using TM = Team<SH, G>;
    constexpr int NT = TPB / G;
    static_assert(TW % NT == 0, "a tile is whole rounds");
    __shared__ TeamTab<SH> S;
    __shared__ double rows[NT][TM::ROWS];
    __shared__ double es[TW];
    if ((int)blockIdx.x >= ntiles) return;
    const BatchTile tl = tiles[blockIdx.x];
    const BatchRec& R = recs[tl.rec];
    stage_team(&S, static_cast<const TeamTab<SH>*>(R.tab_d));
    const TM T;
    const int tm = threadIdx.x / G;
    const MeasureOut none{};
    for (int i = tm; i < TW; i += NT) {
        const int w = tl.w0 + i;
        const double e = team_measure<SH, G, 0, false, false>(T, S, rows[tm], nullptr, nullptr, (const double*)R.pos,
                                                              (double*)R.dinv, R.logabs, R.sign, R.el, w, w < R.W,
                                                              R.Wcap, 1, none, 0, R.flags);
        if (T.t == 0) es[i] = e;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        Comp c{0.0, 0.0};
        for (int i = threadIdx.x; i < TW; i += 32) c = comp_add(c, Comp{es[i], 0.0});
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            c = comp_add(c, Comp{__shfl_down_sync(0xffffffffu, c.s, o), __shfl_down_sync(0xffffffffu, c.c, o)});
        if (threadIdx.x == 0) { tile_partial[2 * blockIdx.x] = c.s; tile_partial[2 * blockIdx.x + 1] = c.c; }
    }
}

// ---------------------------------------------------------------------------
// Single-electron sweeps of FP64 walkers, a team per walker: lane t takes the AOs
// and the partners (electrons, then nuclei) t, t + G, ... of the moving electron
// and column t of its sector's inverse; the walker is in shared memory.  Every
// pair's u (and for drift moves its gradient, and every electron's AO gradients)
// at the current positions is kept there, so a proposal evaluates only the new
// position; c'_a = sum_k C[a][k] D^-1[k][q] turns grad ln D into one
// multiply-add per AO and component.
// ---------------------------------------------------------------------------
template <class SH, int MOVE>
struct SweepState {
    static constexpr bool DRIFT = MOVE == MOVE_ONE_DRIFT;
    static constexpr int NE = SH::NE, NM = SH::NMAX, NP = SH::NE + SH::NNUC;
    double pos[NE][3];
    double dinv[2][NM][NM];
    double pu[NE][NP];                                  // u of (electron, partner), nuclei negative
    double draw[NE][4];                                 // the sweep's normals and acceptance uniforms
    double pf[DRIFT ? NE : 1][DRIFT ? NP : 1][3];       // grad_e u of (electron, partner)
    double ga[DRIFT ? NE : 1][DRIFT ? SH::NAO : 1][3];  // AO gradients at the electron's position
};

template <class SH, int G, int MOVE>
struct SweepTeam {
    using St = SweepState<SH, MOVE>;
    using Tab = TeamTab<SH>;
    static constexpr bool DRIFT = St::DRIFT;
    static constexpr int NE = SH::NE, NM = SH::NMAX, NNUC = SH::NNUC, NP = St::NP;
    static constexpr int AS = (SH::NAO + G - 1) / G, PS = (NP + G - 1) / G;
    static_assert(G >= NM, "a lane per column of the inverse");

    static __device__ __forceinline__ double sum(double v) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    }

    // u of electron e at (x, y, z) with partner m (nuclei: -u) and, for drift
    // moves, its gradient; zero for e itself.
    static __device__ __forceinline__ void pair(const Tab& S, const St& W, int e, int m, double x, double y, double z,
                                                double& u, double (&f)[3]) {
        u = 0;
        f[0] = f[1] = f[2] = 0;
        if (m >= NP || m == e) return;
        const bool el = m < NE;
        const int I = el ? 0 : m - NE;
        if (SH::JAS != JAS_PADE_EEN && !el) return;
        const double dx = x - (el ? W.pos[el ? m : 0][0] : S.nuc[I][0]), dy = y - (el ? W.pos[el ? m : 0][1] : S.nuc[I][1]),
                     dz = z - (el ? W.pos[el ? m : 0][2] : S.nuc[I][2]);
        double d, ri, g;
        dist(dx * dx + dy * dy + dz * dz, d, ri);
        if (SH::JAS == JAS_PADE_EEN) {
            const int c = (m < SH::NUP) == (e < SH::NUP) ? 1 : 0;
            const double a = el ? S.a_ee[c] : -S.enA[I], b = el ? S.b_ee[c] : S.enB[I];
            const double inv = d_rcp(1.0 + b * d);
            u = a * d * inv;
            g = a * inv * inv * ri;
        } else {
            const double inv = d_rcp(1.0 + d * S.invF);
            u = -0.5 * S.F * inv;
            g = 0.5 * inv * inv * ri;
        }
        if (DRIFT) { f[0] = g * dx; f[1] = g * dy; f[2] = g * dz; }
    }

    // tau F capped at maxd.
    static __device__ __forceinline__ void cap(double& x, double& y, double& z, double maxd) {
        const double m = d_sqrt(x * x + y * y + z * z);
        if (m > maxd) {
            const double s = maxd * recip_full(m);
            x *= s; y *= s; z *= s;
        }
    }

    // n_sweeps sweeps of walker w; every lane of the warp calls it (idle teams,
    // act false, run on a dummy configuration and store nothing).
    static __device__ __forceinline__ void run(const Tab& S, St& W, int w, bool act, double* __restrict__ gpos,
                                               double* __restrict__ gdinv, int* __restrict__ gsign, int Wcap,
                                               int n_sweeps, uint64_t step0, double step, double tau, double maxd,
                                               uint64_t seed, int fixed_node, unsigned long long* acc_out, int* flags) {
        const int lane = threadIdx.x & 31, base = lane & ~(G - 1), t = lane - base;
        for (int i = t; i < 3 * NE; i += G)
            W.pos[i / 3][i % 3] = act ? gpos[(size_t)i * Wcap + w] : (i / 3 + 1) * (0.37 + i % 3);
        for (int i = t; i < 2 * NM * NM; i += G) (&W.dinv[0][0][0])[i] = act ? gdinv[(size_t)i * Wcap + w] : 0.0;
        __syncwarp();
        double g0, g1, g2, gl;
        for (int e = 0; e < NE; ++e) {
            const double x = W.pos[e][0], y = W.pos[e][1], z = W.pos[e][2];
            for (int m = t; m < NP; m += G) {
                double u, f[3];
                pair(S, W, e, m, x, y, z, u, f);
                W.pu[e][m] = u;
                if (DRIFT) { W.pf[e][m][0] = f[0]; W.pf[e][m][1] = f[1]; W.pf[e][m][2] = f[2]; }
            }
            if (DRIFT)
                for (int a = t; a < SH::NAO; a += G) {
                    double v;
                    team_ao<SH, 1>(S, a, a < S.n_ao, x, y, z, v, g0, g1, g2, gl);
                    W.ga[e][a][0] = g0; W.ga[e][a][1] = g1; W.ga[e][a][2] = g2;
                }
        }
        int sgn = act ? gsign[w] : 1;
        unsigned acc = 0;
        int flg = 0;
        const double sd2 = DRIFT ? d_sqrt(2.0 * tau) : step, i4t = DRIFT ? recip_full(4.0 * tau) : 0.0;
        for (int it = 0; it < n_sweeps; ++it) {
            __syncwarp();
            // an electron's two Box-Muller pairs are two items of the lanes
            for (int i = t; i < 2 * NE; i += G) {
                const int e = i >> 1;
                const U4 x = rng_draw(seed, (uint32_t)w, step0 + (uint64_t)it, (uint32_t)e, TAG_PROPOSE);
                double n0, n1;
                if (i & 1) {
                    bm24(x.z & 0xFFFFFFu, x.w & 0xFFFFFFu, n0, n1);
                    W.draw[e][2] = n0;
                    W.draw[e][3] = u24((x.x >> 24) | ((x.y >> 24) << 8) | ((x.z >> 24) << 16), 0.0);
                } else {
                    bm24(x.x & 0xFFFFFFu, x.y & 0xFFFFFFu, n0, n1);
                    W.draw[e][0] = n0;
                    W.draw[e][1] = n1;
                }
            }
            __syncwarp();
            for (int e = 0; e < NE; ++e) {
                const int sig = e < SH::NUP ? 0 : 1, q = e - sig * SH::NUP;
                const int NS = sig == 0 ? SH::NUP : SH::NDN;
                const double rx = W.pos[e][0], ry = W.pos[e][1], rz = W.pos[e][2];
                double wq[NM];
#pragma unroll
                for (int k = 0; k < NM; ++k) wq[k] = k < NS ? W.dinv[sig][k][q] : 0.0;
                double cw[AS], dlx = 0, dly = 0, dlz = 0;
                if (DRIFT) {
                    double gx = 0, gy = 0, gz = 0, jx = 0, jy = 0, jz = 0;
#pragma unroll
                    for (int s = 0; s < AS; ++s) {
                        const int a = min(t + G * s, SH::NAO - 1);
                        double c = 0;
#pragma unroll
                        for (int k = 0; k < NM; ++k) c += S.C[sig][a][k] * wq[k];
                        cw[s] = t + G * s < S.n_ao ? c : 0.0;
                        gx += cw[s] * W.ga[e][a][0]; gy += cw[s] * W.ga[e][a][1]; gz += cw[s] * W.ga[e][a][2];
                    }
#pragma unroll
                    for (int r = 0; r < PS; ++r) {
                        const int m = t + G * r;
                        if (m < NP) { jx += W.pf[e][m][0]; jy += W.pf[e][m][1]; jz += W.pf[e][m][2]; }
                    }
                    gx = sum(gx + S.qa * jx); gy = sum(gy + S.qa * jy); gz = sum(gz + S.qa * jz);
                    dlx = tau * (2.0 * gx); dly = tau * (2.0 * gy); dlz = tau * (2.0 * gz);
                    cap(dlx, dly, dlz, maxd);
                }
                const double nx = rx + dlx + sd2 * W.draw[e][0], ny = ry + dly + sd2 * W.draw[e][1],
                             nz = rz + dlz + sd2 * W.draw[e][2];
                // AOs at r': orbital values on every lane, then t_j = sum_k phi_k D^-1[k][j]
                double na[DRIFT ? AS : 1][3], phi[NM];
#pragma unroll
                for (int k = 0; k < NM; ++k) phi[k] = 0;
#pragma unroll
                for (int s = 0; s < AS; ++s) {
                    const int a = t + G * s, ac = min(a, SH::NAO - 1);
                    double v;
                    team_ao<SH, DRIFT ? 1 : 0>(S, a, a < S.n_ao, nx, ny, nz, v, g0, g1, g2, gl);
                    if (DRIFT) { na[s][0] = g0; na[s][1] = g1; na[s][2] = g2; }
#pragma unroll
                    for (int k = 0; k < NM; ++k) phi[k] += S.C[sig][ac][k] * v;
                }
                double tj = 0;
                const int col = t < NS ? t : 0;
#pragma unroll
                for (int k = 0; k < NM; ++k) {
                    phi[k] = sum(phi[k]);
                    if (k < NS) tj += phi[k] * W.dinv[sig][k][col];
                }
                const double R = __shfl_sync(0xffffffffu, tj, base + q);
                // Jastrow at r' against the kept terms at r
                double un[PS], fn[PS][3], du = 0;
#pragma unroll
                for (int r = 0; r < PS; ++r) {
                    const int m = t + G * r;
                    pair(S, W, e, m, nx, ny, nz, un[r], fn[r]);
                    du += m < NP ? un[r] - W.pu[e][m] : 0.0;
                }
                du = sum(du);
                const bool zero = ((d_hi(R) & 0x7fffffff) | d_lo(R)) == 0;
                const double iR = zero ? 0.0 : recip_full(R);
                double lg = 2.0 * du;
                if (DRIFT) {
                    double bx = 0, by = 0, bz = 0, jx = 0, jy = 0, jz = 0;
#pragma unroll
                    for (int s = 0; s < AS; ++s) { bx += cw[s] * na[s][0]; by += cw[s] * na[s][1]; bz += cw[s] * na[s][2]; }
#pragma unroll
                    for (int r = 0; r < PS; ++r) { jx += fn[r][0]; jy += fn[r][1]; jz += fn[r][2]; }
                    bx = sum(bx * iR + S.qa * jx); by = sum(by * iR + S.qa * jy); bz = sum(bz * iR + S.qa * jz);
                    bx *= tau * 2.0; by *= tau * 2.0; bz *= tau * 2.0;
                    cap(bx, by, bz, maxd);
                    const double fx = nx - rx - dlx, fy = ny - ry - dly, fz = nz - rz - dlz;
                    const double qx = rx - nx - bx, qy = ry - ny - by, qz = rz - nz - bz;
                    lg += ((fx * fx + fy * fy + fz * fz) - (qx * qx + qy * qy + qz * qz)) * i4t;
                }
                const double prob = R * R * d_exp(lg);
                if (prob != prob) flg |= FLAG_NONFINITE;
                const int take = W.draw[e][3] < prob && !zero && !(fixed_node && d_hi(R) < 0);
                if (__shfl_sync(0xffffffffu, take, base)) {
                    if (t < NS) {
#pragma unroll
                        for (int k = 0; k < NM; ++k) {
                            if (k >= NS) break;
                            const double c = wq[k] * iR;
                            W.dinv[sig][k][t] = t == q ? c : W.dinv[sig][k][t] - c * tj;
                        }
                    }
#pragma unroll
                    for (int r = 0; r < PS; ++r) {
                        const int m = t + G * r;
                        if (m >= NP) break;
                        W.pu[e][m] = un[r];
                        if (m < NE) W.pu[m][e] = un[r];
                        if (DRIFT) {
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                W.pf[e][m][c] = fn[r][c];
                                if (m < NE && m != e) W.pf[m][e][c] = -fn[r][c];
                            }
                        }
                    }
                    if (DRIFT) {
#pragma unroll
                        for (int s = 0; s < AS; ++s) {
                            const int a = t + G * s;
                            if (a >= SH::NAO) break;
                            W.ga[e][a][0] = na[s][0]; W.ga[e][a][1] = na[s][1]; W.ga[e][a][2] = na[s][2];
                        }
                    }
                    if (t == 0) { W.pos[e][0] = nx; W.pos[e][1] = ny; W.pos[e][2] = nz; }
                    if (d_hi(R) < 0) sgn = -sgn;
                    ++acc;
                }
                __syncwarp();
            }
        }
        if (!act) return;
        for (int i = t; i < 3 * NE; i += G) gpos[(size_t)i * Wcap + w] = W.pos[i / 3][i % 3];
        for (int i = t; i < 2 * NM * NM; i += G) gdinv[(size_t)i * Wcap + w] = (&W.dinv[0][0][0])[i];
        if (t == 0) {
            gsign[w] = sgn;
            if (acc) atomicAdd(acc_out, (unsigned long long)acc);
        }
        if (flg) atomicOr(flags, flg);
    }
};

// A warp per block: the walkers' state is most of a block's shared memory.
template <class SH, int G, int MOVE>
__global__ void __launch_bounds__(32) k_team_sweep(const TeamTab<SH>* __restrict__ tab, double* __restrict__ gpos,
                                                   double* __restrict__ gdinv, int* __restrict__ gsign, int W, int Wcap,
                                                   int n_sweeps, uint64_t step0, double step, double tau, double maxd,
                                                   uint64_t seed, unsigned long long* acc_out, int* flags,
                                                   int fixed_node) {
    constexpr int NT = 32 / G;
    __shared__ TeamTab<SH> S;
    __shared__ SweepState<SH, MOVE> st[NT];
    stage_team(&S, tab);
    const int tm = threadIdx.x / G, w = blockIdx.x * NT + tm;
    SweepTeam<SH, G, MOVE>::run(S, st[tm], w, w < W, gpos, gdinv, gsign, Wcap, n_sweeps, step0, step, tau, maxd, seed,
                                fixed_node, acc_out, flags);
}

// Batched form: TW / NT blocks per (system, TW-walker tile).
template <class SH, int G, int MOVE, int TW>
__global__ void __launch_bounds__(32) kb_team_sweep(const BatchTile* __restrict__ tiles, int ntiles,
                                                    const BatchRec* __restrict__ recs,
                                                    const BatchCtl* __restrict__ ctl) {
    constexpr int NT = 32 / G, BPT = TW / NT;
    static_assert(TW % NT == 0, "a tile splits into whole blocks");
    __shared__ TeamTab<SH> S;
    __shared__ SweepState<SH, MOVE> st[NT];
    if ((int)blockIdx.x >= ntiles * BPT) return;
    const BatchTile tl = tiles[blockIdx.x / BPT];
    const BatchRec& R = recs[tl.rec];
    const int tm = threadIdx.x / G, w0 = tl.w0 + (int)(blockIdx.x % BPT) * NT, w = w0 + tm;
    if (w0 >= R.W) return;                              // the whole block
    stage_team(&S, static_cast<const TeamTab<SH>*>(R.tab_d));
    SweepTeam<SH, G, MOVE>::run(S, st[tm], w, w < R.W, (double*)R.pos, (double*)R.dinv, R.sign, R.Wcap, ctl->n_sweeps,
                                ctl->step, ctl->step_size, ctl->tau, ctl->max_drift,
                                batch_system_seed(ctl->seed, R.index), R.fixed_node, R.acc, R.flags);
}

// SMs of the current device, asked for once per device.
inline int device_sms() {
    constexpr int N = 64;
    static std::atomic<int> known[N];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= N) dev = 0;
    n = known[dev].load(std::memory_order_relaxed);
    if (!n && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
        known[dev].store(n, std::memory_order_relaxed);
    return n > 0 ? n : 1;
}

// Launchers of a shape with teams of G lanes.
template <class SH, int G>
struct TeamOps {
    static int table(const HostSys& hs, const TeamTab<SH>** out) {
        constexpr int slot = 3;
        if (!hs.dev_table[slot] || hs.dev_table_version[slot] != hs.version) {
            TeamTab<SH> h;
            if (!fill_team(hs, h)) return 7;
            if (!hs.dev_table[slot] && cudaMalloc(&hs.dev_table[slot], sizeof(h)) != cudaSuccess) return 8;
            if (cudaMemcpy(hs.dev_table[slot], &h, sizeof(h), cudaMemcpyHostToDevice) != cudaSuccess) return 2;
            hs.dev_table_version[slot] = hs.version;
        }
        *out = static_cast<const TeamTab<SH>*>(hs.dev_table[slot]);
        return 0;
    }

    // One warp per block while every warp can have a sub-partition of its own
    // (four an SM), so that the block scheduler spreads them over the SMs;
    // four beyond that, which share one copy of the table.
    static bool spread(int W) { return (long long)W * G <= 32LL * 4 * device_sms(); }

    static int step_blocks(int W) {
        const int nt = (spread(W) ? 32 : 128) / G;
        return (W + nt - 1) / nt;
    }

    template <int MOVE, bool REC, int TPB>
    static int steps_t(const TeamTab<SH>* tab, DevWalkers& dw, int n, uint64_t s0, double step, uint64_t seed,
                       double* partial, cudaStream_t st) {
        const int nb = step_blocks(dw.W);
        k_team_steps<SH, G, MOVE, REC, TPB><<<nb, TPB, 0, st>>>(tab, (double*)dw.pos, dw.logabs, dw.sign, dw.el, dw.W,
                                                                dw.Wcap, n, s0, step, seed, dw.acc, partial, nb, dw.flags);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }
    template <int MOVE>
    static int steps(const HostSys& hs, DevWalkers& dw, int n, uint64_t s0, double step, uint64_t seed, double* partial,
                     cudaStream_t st) {
        const TeamTab<SH>* tab;
        const int rc = table(hs, &tab);
        if (rc) return rc;
        if (spread(dw.W))
            return partial ? steps_t<MOVE, true, 32>(tab, dw, n, s0, step, seed, partial, st)
                           : steps_t<MOVE, false, 32>(tab, dw, n, s0, step, seed, partial, st);
        return partial ? steps_t<MOVE, true, 128>(tab, dw, n, s0, step, seed, partial, st)
                       : steps_t<MOVE, false, 128>(tab, dw, n, s0, step, seed, partial, st);
    }

    template <int NR, bool DEL, bool FORCE>
    static int measure_t(const HostSys& hs, DevWalkers& dw, bool ws, const MeasureOut& out, cudaStream_t st) {
        constexpr int TPB = 128, NT = TPB / G;
        const TeamTab<SH>* tab;
        int rc = table(hs, &tab);
        if (rc) return rc;
        if (dw.W == 0) return 0;
        const int nb = (dw.W + NT - 1) / NT;
        // the sums of the sampled rows include E_L's: no partials beside them
        double* partial = ws && NR == 0 && !FORCE && dw.partial && dw.partial_cap >= 2 * nb + 1 ? dw.partial : nullptr;
        k_team_measure<SH, G, NR, DEL, FORCE, TPB><<<nb, TPB, 0, st>>>(
            tab, (const double*)dw.pos, (double*)dw.dinv, dw.logabs, dw.sign, dw.el, dw.W, dw.Wcap, ws ? 1 : 0, out,
            hs.n_params(), partial, dw.flags);
        ++g_launch_count;
        if (cudaGetLastError() != cudaSuccess) return 2;
        return partial ? launch_sum_partials(partial, nb, 1, dw.partial + dw.partial_cap - 1, st) : 0;
    }
    static int measure(const HostSys& hs, DevWalkers& dw, bool ws, const MeasureOut& out, cudaStream_t st) {
        if (out.O) {
            if constexpr (SH::JAS == JAS_PADE_EEN)
                return out.dEL ? measure_t<SH::NROT, true, false>(hs, dw, ws, out, st)
                               : measure_t<SH::NROT, false, false>(hs, dw, ws, out, st);
            else
                return 7;
        }
        if (out.fhf || out.omega) return measure_t<0, false, true>(hs, dw, ws, out, st);
        return measure_t<0, false, false>(hs, dw, ws, out, st);
    }

    // Lanes per walker of the sweeps.
    static constexpr int GS = SH::NE <= 3 ? 4 : 8;
    template <int MOVE>
    static int sweep(const HostSys& hs, DevWalkers& dw, int n, uint64_t s0, double step, double tau, double maxd,
                     uint64_t seed, cudaStream_t st) {
        constexpr int NT = 32 / GS;
        const TeamTab<SH>* tab;
        const int rc = table(hs, &tab);
        if (rc) return rc;
        k_team_sweep<SH, GS, MOVE><<<(dw.W + NT - 1) / NT, 32, 0, st>>>(
            tab, (double*)dw.pos, (double*)dw.dinv, dw.sign, dw.W, dw.Wcap, n, s0, step, tau, maxd, seed, dw.acc,
            dw.flags, dw.fixed_node);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }
    template <int MOVE, int TW>
    static int batch_sweep(const BatchClass& bc, const BatchCtl* ctl, cudaStream_t st, int* occ) {
        auto kern = kb_team_sweep<SH, GS, MOVE, TW>;
        if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, 32, 0) == cudaSuccess ? 0 : 2;
        if (bc.ntiles == 0) return 0;
        kern<<<bc.ntiles * (TW * GS / 32), 32, 0, st>>>(bc.tiles, bc.ntiles, bc.recs, ctl);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    template <int TW>
    static int batch_measure(const BatchClass& bc, cudaStream_t st, int* occ) {
        constexpr int TPB = 128;
        auto kern = kb_team_measure<SH, G, TPB, TW>;
        if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, TPB, 0) == cudaSuccess ? 0 : 2;
        if (bc.ntiles == 0) return 0;
        kern<<<bc.ntiles, TPB, 0, st>>>(bc.tiles, bc.ntiles, bc.recs, bc.tile_partial);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }
};

}  // namespace qmc
