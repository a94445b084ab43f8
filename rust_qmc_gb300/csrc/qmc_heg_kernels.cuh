// qmc_heg_kernels.cuh -- warp-per-walker kernels of the periodic homogeneous
// electron gas (src/systems/heg.rs): complex plane-wave determinants
// phi_k(r) = e^{i k.r}, a spin-dependent Jastrow with minimum image and a
// cutoff at L/2, and the Ewald Coulomb energy.
//
// Lane j holds column j of each complex inverse Slater matrix; lane k
// evaluates its own orbital e^{i k.r} (no AO contraction is needed).  The
// FP64 measurement rebuilds the inverses by complex Gauss-Jordan elimination
// and evaluates the Ewald sum: real-space pairs with images inside the erfc
// cutoff, the reciprocal sum by octants of k vectors (a lane per octant vector,
// per-electron phases in shared memory), and FP64 constants from the host.
#pragma once
#include <cstdio>
#include <cmath>
#include <cstring>
#include <vector>
#include "qmc_internal.h"
#include "qmc_device.cuh"
#include "qmc_ewald.cuh"

namespace qmc {

// A pair of scalars as one vector: complex inverse columns, phases.
template <class T> struct HComplex;
template <> struct HComplex<float> { using type = float2; };
template <> struct HComplex<double> { using type = double2; };

constexpr int HMAX_K = 1800;      // reciprocal half-space vectors (|n_i| <= 7 cube: 1687)
constexpr int HMAX_KMAX = 9;      // largest component they leave room for (|n| <= 10: 2084)

template <class T>
struct SysH {
    T L, invL, halfL;
    T F, pb, pc;                   // Jastrow: F, RPA b = 1/F, c = 0.2/F^2
    int form;                      // 0 Pade, 1 RPA, 2 Yukawa
    T a_ee[2];                     // [0] antiparallel, [1] parallel
    int quirk_cross;               // reference cross term without the orbital factor
    int real_images;               // 1: images inside the erfc cutoff; 0: minimum image only
    T alpha, rcut;
    double e_const;                // FP64 constant part of the Ewald energy
    double ksum_const;             // added per walker with the reciprocal sum
    T k2sum;                       // (1/2) sum over occupied |k|^2 of both sectors
    T kvec[2][32][3];              // [sector][column][xyz]
    T k2[2][32];                   // |k|^2 of each
    // columns by opposite wave vectors: column rep[sig][i] and, unless 255, column
    // mate[sig][i] with the negated vector
    int n_rep[2];
    unsigned char rep[2][32], mate[2][32];
    int nt;                        // octant vectors of the reciprocal sum
    int kmax;                      // their largest component
    float aL, rc2u;                // alpha L and the squared real-space cutoff, in box units
    ff a2l2;                       // (alpha L)^2 log2(e)
    int perm[64];                  // internal -> caller electron index
};

// Ewald tables (global memory).
struct KTable {
    // Octant vectors (a, b, c) >= 0 packed a | b << 8 | c << 16, and the Ewald
    // weight times the number of half-space vectors (+-a, +-b, +-c) they stand for.
    int tri[HMAX_K];
    double kw[HMAX_K];
    float2 kwf[HMAX_K];            // kw as a float-float pair (hi, lo)
    float4 erfc_tab[HERFC_N][3];   // fill_erfc_table
};

template <class T>
static bool fill_sysh(const HostSys& hs, int NE, int NUP, SysH<T>& S, KTable& KT) {
    std::memset(&S, 0, sizeof(S));
    std::memset(&KT, 0, sizeof(KT));
    for (int ei = 0; ei < hs.N && ei < 64; ++ei) S.perm[ei] = hs.perm[ei];
    if (hs.N != NE || hs.n_up != NUP || !(hs.box_L > 0)) return false;
    const double L = hs.box_L, V = L * L * L;
    S.L = (T)L; S.invL = (T)(1.0 / L); S.halfL = (T)(0.5 * L);
    S.F = (T)hs.F; S.pb = (T)(1.0 / hs.F); S.pc = (T)(0.2 / (hs.F * hs.F));
    S.form = (int)hs.jas[0];
    S.a_ee[0] = (T)hs.jas[2]; S.a_ee[1] = (T)hs.jas[3];
    S.quirk_cross = (hs.quirks & 8) ? 1 : 0;
    const bool qe = (hs.quirks & 4) != 0;
    const double alpha = qe ? 5.0 / L : hs.jas[4] / L;
    const int K = reciprocal_kmax(hs);
    if (K > HMAX_KMAX) return false;
    S.alpha = (T)alpha;
    S.real_images = qe ? 0 : 1;
    S.rcut = (T)(5.6 / alpha);
    // the device sums the 27 nearest images: the cutoff must stay below 1.5 L (which
    // also keeps alpha L above 3.73, the range of image_erfc's polynomial)
    if (!qe && 5.6 / alpha >= 1.5 * L) return false;
    // reciprocal half space, by octants; weight (4 pi / V) e^{-k^2 / 4 alpha^2} / k^2
    int nk = 0, nt = 0;
    double wsum = 0.0;
    const double dk = 2.0 * M_PI / L;
    for (int nx = 0; nx <= K; ++nx)
        for (int ny = 0; ny <= K; ++ny)
            for (int nz = 0; nz <= K; ++nz) {
                if (nx == 0 && ny == 0 && nz == 0) continue;
                if (!qe && nx * nx + ny * ny + nz * nz > K * K) continue;
                const int signs = (nx ? 2 : 1) * (ny ? 2 : 1) * (nz ? 2 : 1);
                nk += signs / 2;
                if (nk > HMAX_K) return false;
                const double k2 = dk * dk * (nx * nx + ny * ny + nz * nz);
                const double w = 4.0 * M_PI / V * std::exp(-k2 / (4.0 * alpha * alpha)) / k2;
                KT.tri[nt] = nx | (ny << 8) | (nz << 16);
                KT.kw[nt] = w * (signs / 2);
                KT.kwf[nt].x = (float)KT.kw[nt];
                KT.kwf[nt].y = (float)(KT.kw[nt] - (double)KT.kwf[nt].x);
                wsum += KT.kw[nt];
                ++nt;
            }
    fill_erfc_table(KT.erfc_tab);
    S.nt = nt;
    S.kmax = K;
    S.aL = (float)(alpha * L);
    S.a2l2 = ff(alpha * L * alpha * L * 1.4426950408889634);
    S.rc2u = (float)(5.6 / (alpha * L) * (5.6 / (alpha * L)));
    const int N = hs.N;
    if (qe) {
        // heg.rs:526-581: (1/2) sum_k f_k (|rho_k|^2 - N) and -0.448 N / r_s
        const double rs = L / std::cbrt(4.0 * M_PI * N / 3.0);
        S.ksum_const = -N * wsum;
        S.e_const = -N * 0.448 / rs;
    } else {
        // one-component plasma: N [ (1/2) sum_{n!=0} erfc(alpha nL)/(nL) - alpha/sqrt(pi) - pi N/(2 V alpha^2) ]
        double img = 0.0;
        for (int a = -3; a <= 3; ++a)
            for (int b = -3; b <= 3; ++b)
                for (int c = -3; c <= 3; ++c) {
                    if (!a && !b && !c) continue;
                    double d = L * std::sqrt((double)(a * a + b * b + c * c));
                    img += std::erfc(alpha * d) / d;
                }
        S.ksum_const = 0.0;
        S.e_const = N * (0.5 * img - alpha / std::sqrt(M_PI) - M_PI * N / (2.0 * V * alpha * alpha));
    }
    double k2s = 0.0;
    for (int sig = 0; sig < 2; ++sig) {
        int col = 0, of[32];                       // orbital of each column
        for (int ei = 0; ei < hs.N; ++ei) {
            int e = hs.perm[ei];
            if ((hs.spins[e] > 0) != (sig == 0)) continue;
            int k = hs.occ[e];
            if (col >= 32) return false;
            of[col] = k;
            for (int c = 0; c < 3; ++c) S.kvec[sig][col][c] = (T)hs.kvec[3 * k + c];
            const double k2 = hs.kvec[3 * k] * hs.kvec[3 * k] + hs.kvec[3 * k + 1] * hs.kvec[3 * k + 1] +
                              hs.kvec[3 * k + 2] * hs.kvec[3 * k + 2];
            S.k2[sig][col] = (T)k2;
            k2s += k2;
            ++col;
        }
        bool taken[32] = {};
        for (int j = 0; j < col; ++j) {
            if (taken[j]) continue;
            const double* k = &hs.kvec[3 * of[j]];
            int m = j + 1;
            while (m < col && (taken[m] || hs.kvec[3 * of[m]] != -k[0] || hs.kvec[3 * of[m] + 1] != -k[1] ||
                               hs.kvec[3 * of[m] + 2] != -k[2]))
                ++m;
            S.rep[sig][S.n_rep[sig]] = (unsigned char)j;
            S.mate[sig][S.n_rep[sig]++] = (unsigned char)(m < col ? m : 255);
            if (m < col) taken[m] = true;
        }
    }
    S.k2sum = (T)(0.5 * k2s);
    return true;
}

template <class T>
__device__ __forceinline__ void load_sysh(SysH<T>* dst, const SysH<T>* __restrict__ src, int bytes) {
    const int4* s = reinterpret_cast<const int4*>(src);
    int4* d = reinterpret_cast<int4*>(dst);
    const int n16 = bytes / (int)sizeof(int4);
    for (int i = threadIdx.x; i < n16; i += blockDim.x) d[i] = s[i];
    // tail words when the size is not a multiple of 16 bytes
    for (int i = n16 * 4 + threadIdx.x; i < bytes / 4; i += blockDim.x)
        reinterpret_cast<int*>(dst)[i] = reinterpret_cast<const int*>(src)[i];
    __syncthreads();
}

__device__ __forceinline__ void fsincos(double x, double* s, double* c) { sincos(x, s, c); }
__device__ __forceinline__ void fsincos(float x, float* s, float* c) { __sincosf(x, s, c); }
// float-float sine and cosine without FP64: Cody-Waite reduction
// r = x - n pi/2 with pi/2 in three FP32 parts (the leading difference is
// exact by Sterbenz's lemma, the n multiples by TwoProd), then the Taylor
// series on |r| <= pi/4 -- terms through r^7 (sine) and r^8 (cosine) in
// float-float, the rest (below 3.1e-7) in FP32 -- and the quadrant n mod 4.
// Absolute error below 1e-13 for |x| <= 60.
__device__ __forceinline__ void fsincos(ff x, ff* s, ff* c) {
    const float n = rintf(__fmul_rn(x.hi, 0.63661975f));
    const ff p = ff_two_prod(1.5707964f, n), q = ff_two_prod(-4.371139e-08f, n);
    ff r = ff(__fsub_rn(x.hi, p.hi)) + ff(x.lo);
    r = r + ff(-p.lo);
    r = r - q;
    r = r + ff(-__fmul_rn(-1.7151245e-15f, n));
    const ff r2 = r * r;
    const float h2 = r2.hi;
    // sin r = r + r^3 (-1/3! + r^2 (1/5! + r^2 (-1/7! + r^2 (1/9! - r^2/11! + r^4/13!))))
    const float qs = __fmul_rn(h2, __fmaf_rn(h2, __fmaf_rn(h2, 1.6059044e-10f, -2.5052108e-08f), 2.7557319e-06f));
    ff cs = ff(-1.0 / 5040.0) + ff(qs);
    cs = cs * r2 + ff(1.0 / 120.0);
    cs = cs * r2 + ff(-1.0 / 6.0);
    const ff sn = r + cs * r2 * r;
    // cos r = 1 + r^2 (-1/2 + r^2 (1/4! + r^2 (-1/6! + r^2 (1/8! + r^2 (-1/10! + r^2/12! - ...)))))
    const float qc = __fmaf_rn(h2, __fmaf_rn(h2, __fmaf_rn(h2, 4.7794773e-14f, -1.1470746e-11f), 2.0876757e-09f),
                               -2.7557319e-07f);
    ff cc = ff(1.0 / 40320.0) + ff(__fmul_rn(qc, h2));
    cc = cc * r2 + ff(-1.0 / 720.0);
    cc = cc * r2 + ff(1.0 / 24.0);
    cc = cc * r2 + ff(-0.5);
    const ff cn = ff(1.0f) + cc * r2;
    switch ((int)n & 3) {
        case 0: *s = sn; *c = cn; break;
        case 1: *s = cn; *c = -sn; break;
        case 2: *s = -sn; *c = -cn; break;
        default: *s = -cn; *c = sn; break;
    }
}

// Nearest integer of a float-float value (ties resolved by the leading part).
using ::rint;
__device__ __forceinline__ ff rint(ff x) {
    float r = rintf(x.hi);
    const float d = __fadd_rn(__fsub_rn(x.hi, r), x.lo);   // x.hi - r is exact
    if (d > 0.5f) r += 1.0f;
    else if (d < -0.5f) r -= 1.0f;
    return ff(r);
}

template <class T>
__device__ __forceinline__ T min_img(T d, const SysH<T>& S) { return d - S.L * rint(d * S.invL); }

// Warp shuffles for every compute type of the electron-gas kernels.
__device__ __forceinline__ float hshfl(float v, int s) { return __shfl_sync(0xffffffffu, v, s); }
__device__ __forceinline__ double hshfl(double v, int s) { return __shfl_sync(0xffffffffu, v, s); }
__device__ __forceinline__ ff hshfl(ff v, int s) { return wshfl(v, s); }

// Two consecutive values of shared memory as one load.
template <class T>
__device__ __forceinline__ void load_pair(const T* p, T& a, T& b) {
    const auto v = *reinterpret_cast<const typename HComplex<T>::type*>(p);
    a = v.x; b = v.y;
}
__device__ __forceinline__ void load_pair(const ff* p, ff& a, ff& b) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = ff(v.x, v.y); b = ff(v.z, v.w);
}

template <class T>
__device__ __forceinline__ void store_pair(T* p, T a, T b) {
    *reinterpret_cast<typename HComplex<T>::type*>(p) = {a, b};
}
__device__ __forceinline__ void store_pair(ff* p, ff a, ff b) {
    *reinterpret_cast<float4*>(p) = make_float4(a.hi, a.lo, b.hi, b.lo);
}

// Exchange registers 0 and p (0 < p < N, the same on every lane): one case runs.
template <int N, class T>
__device__ __forceinline__ void swap_rows(int p, T (&a)[N], T (&b)[N]) {
#pragma unroll
    for (int r = 1; r < N; ++r)
        if (p == r) {
            T t = a[0]; a[0] = a[r]; a[r] = t;
            t = b[0]; b[0] = b[r]; b[r] = t;
        }
}

// |z|^2 of a pivot candidate on the leading parts (pivot choice only).
__device__ __forceinline__ float pivot_mag(float r, float i) { return r * r + i * i; }
__device__ __forceinline__ float pivot_mag(double r, double i) { return (float)(r * r + i * i); }
__device__ __forceinline__ float pivot_mag(ff r, ff i) { return r.hi * r.hi + i.hi * i.hi; }
__device__ __forceinline__ float hshfl_xor(float v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ double hshfl_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ ff hshfl_xor(ff v, int m) { return shfl_xor(v, m); }

// Jastrow pair (src/systems/heg.rs:352-444): u, u'(r) and u'' + 2u'/r;
// zero outside (1e-10, L/2).
template <class T>
__device__ __forceinline__ void heg_u(const SysH<T>& S, T r, T a, T& u, T& du, T& lu) {
    u = 0; du = 0; lu = 0;
    if (!(r < S.halfL && r > T(1e-10))) return;
    if (S.form == 0) {
        T fr = S.F + r;
        u = a * r / (1 + r / S.F);
        du = a * S.F * S.F / (fr * fr);
        lu = 2 * a * S.F * S.F * S.F / (r * fr * fr * fr);
    } else if (S.form == 1) {
        T den = 1 + S.pb * r + S.pc * r * r;
        u = a * r / den;
        du = a * (1 - S.pc * r * r) / (den * den);
        T d2 = -a * 2 * (S.pc * r * den + (1 - S.pc * r * r) * (S.pb + 2 * S.pc * r)) / (den * den * den);
        lu = d2 + 2 / r * du;
    } else {
        T x = r / S.F, ex = fexp(-x), op = 1 + x;
        u = a * r * ex / op;
        du = a * ex * (1 - x - x * x) / (op * op);
        T d2 = a * ex / (S.F * S.F * op * op * op) * (-3 - 3 * x + x * x + x * x * x);
        lu = d2 + 2 / r * du;
    }
}

// Refresh pair geometry: minimum image of xi - xj.  FP32 walkers' positions are
// floats (the low parts are zero), so the difference is one exact TwoSum.  Positions
// need not lie in the box: n L is a two-product for any n.
template <class T>
__device__ __forceinline__ T pair_image(T a, T b, const SysH<T>& S) { return min_img(a - b, S); }
__device__ __forceinline__ ff pair_image(ff a, ff b, const SysH<ff>& S) {
    const ff d = ff_two_sum(a.hi, -b.hi);
    const float n = rintf(__fmul_rn(d.hi, S.invL.hi));
    const float p = __fmul_rn(-n, S.L.hi);
    return d + ff_fast_two_sum(p, __fmaf_rn(-n, S.L.lo, __fmaf_rn(-n, S.L.hi, -p)));
}

// Squared length; the float-float form sums the exact squares lazily.
template <class T>
__device__ __forceinline__ T length2(T x, T y, T z) { return x * x + y * y + z * z; }
__device__ __forceinline__ ff length2(ff x, ff y, ff z) {
    ff r = ff_two_prod(x.hi, x.hi);
    r.lo = __fmaf_rn(2.0f * x.hi, x.lo, r.lo);
    ff_fma_lazy(r, y, y);
    ff_fma_lazy(r, z, z);
    return ff_norm(r);
}

// Reciprocal of a pair term: to the last bits in FP64 (one Newton step is 1e-14 off, the
// same way in each of the 1431 pairs: log|psi| was 1.3e-12 off in the median, 5e-14 now).
__device__ __forceinline__ float pair_rcp(float a) { return frcp(a); }
__device__ __forceinline__ ff pair_rcp(ff a) { return frcp(a); }
__device__ __forceinline__ double pair_rcp(double a) { return d_rcp_full(a); }

// Pair function of the refresh: u, u'(r)/r and u'' + 2u'/r of heg_u inside its
// cutoff, from r, r^2 and 1/r, with one reciprocal for the RPA form.
template <class T>
__device__ __forceinline__ void heg_pair(const SysH<T>& S, T r, T r2, T ri, T a, T& u, T& f, T& lu) {
    if (S.form != 1) {
        T du;
        heg_u(S, r, a, u, du, lu);
        f = du * ri;
        return;
    }
    const T cr = S.pc * r, cr2 = S.pc * r2, q = T(1) - cr2;
    const T inv = pair_rcp(T(1) + S.pb * r + cr2);
    const T ai = a * inv, ai2 = ai * inv;
    u = ai * r;
    f = ai2 * q * ri;
    // u'' + 2u'/r = 2 a inv^2 ( q / r - c r - q (b + 2 c r) inv )
    lu = T(2) * ai2 * (q * ri - cr - q * (S.pb + T(2) * cr) * inv);
    const bool in = r < S.halfL && r > T(1e-10);
    u = in ? u : T(0);
    f = in ? f : T(0);
    lu = in ? lu : T(0);
}

// Phase of the reciprocal sum at coordinate x: (cos, sin)(2 pi x / L).
template <class T>
__device__ __forceinline__ void unit_phase(T x, const SysH<T>& S, T& c, T& s) {
    double sd, cd;
    sincos(2.0 * M_PI / (double)S.L * (double)x, &sd, &cd);
    c = (T)cd;
    s = (T)sd;
}
__device__ __forceinline__ void unit_phase(ff x, const SysH<ff>& S, ff& c, ff& s) {
    ff t = x * S.invL;
    t = t - rint(t);
    fsincos(ff(6.283185307179586) * t, &s, &c);
}

// Product that is only multiplied or summed further (float-float: not renormalised).
template <class T>
__device__ __forceinline__ T mul_lazy(T a, T b) { return a * b; }
__device__ __forceinline__ ff mul_lazy(ff a, ff b) {
    const ff p = ff_two_prod(a.hi, b.hi);
    return ff(p.hi, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, p.lo)));
}

// acc += x without renormalising (closed with macc_norm).
template <class T>
__device__ __forceinline__ T add_lazy(T acc, T x) { return acc + x; }
__device__ __forceinline__ ff add_lazy(ff acc, ff x) {
    const ff t = ff_two_sum(acc.hi, x.hi);
    return ff(t.hi, __fadd_rn(acc.lo, __fadd_rn(t.lo, x.lo)));
}

template <class T, int NE>
struct HLanePos {
    T x[2], y[2], z[2];
    __device__ __forceinline__ void get(int e, T& ex, T& ey, T& ez) const {
        T a = e < 32 ? x[0] : x[1], b = e < 32 ? y[0] : y[1], c = e < 32 ? z[0] : z[1];
        ex = hshfl(a, e & 31);
        ey = hshfl(b, e & 31);
        ez = hshfl(c, e & 31);
    }
    // Same, for an index that differs between lanes: the source lane cannot know which
    // half the reading lane wants, so both halves travel and the reader selects.
    __device__ __forceinline__ void get_own(int e, T& ex, T& ey, T& ez) const {
        const int s = e & 31;
        T x0 = hshfl(x[0], s), x1 = hshfl(x[1], s);
        T y0 = hshfl(y[0], s), y1 = hshfl(y[1], s);
        T z0 = hshfl(z[0], s), z1 = hshfl(z[1], s);
        ex = e < 32 ? x0 : x1; ey = e < 32 ? y0 : y1; ez = e < 32 ? z0 : z1;
    }
};

// Ewald weight of table entry t in the compute type.
template <class T>
__device__ __forceinline__ T kweight(const KTable* __restrict__ KT, int t) { return (T)KT->kw[t]; }
template <>
__device__ __forceinline__ ff kweight<ff>(const KTable* __restrict__ KT, int t) {
    const float2 w = KT->kwf[t];
    return ff(w.x, w.y);
}

template <class T>
__device__ __forceinline__ T hsum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += hshfl_xor(v, o);
    return v;
}

// u(r) alone, heg_u's expression for it, evaluated on every lane and masked
// (no divergent branch; out-of-range lanes may compute non-finite values).
template <class T>
__device__ __forceinline__ T heg_u_value(const SysH<T>& S, T r, T a) {
    T u;
    if (S.form == 0) {
        u = a * r / (1 + r / S.F);
    } else if (S.form == 1) {
        const T den = 1 + S.pb * r + S.pc * r * r;
        u = a * r / den;
    } else {
        const T x = r / S.F, ex = fexp(-x), op = 1 + x;
        u = a * r * ex / op;
    }
    return (r < S.halfL && r > T(1e-10)) ? u : T(0);
}

// Jastrow change (and gradients) for electron e moving o -> n.
template <int NE, int NUP, class T, bool GRAD>
__device__ __forceinline__ T hjastrow_delta(const SysH<T>& S, const HLanePos<T, NE>& P, int lane, int e, T ox, T oy,
                                            T oz, T nx, T ny, T nz, T (&go)[3], T (&gn)[3]) {
    T du = 0, g[6] = {0, 0, 0, 0, 0, 0};
    if constexpr (!GRAD) {
        // value only: every lane evaluates its partners and masks the unused ones
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int j = lane + 32 * r;
            const T a = S.a_ee[((j < NUP) == (e < NUP)) ? 1 : 0];
            T ax = min_img(ox - P.x[r], S), ay = min_img(oy - P.y[r], S), az = min_img(oz - P.z[r], S);
            T bx = min_img(nx - P.x[r], S), by = min_img(ny - P.y[r], S), bz = min_img(nz - P.z[r], S);
            T ra = fsqrt(ax * ax + ay * ay + az * az), rb = fsqrt(bx * bx + by * by + bz * bz);
            const T d = heg_u_value(S, rb, a) - heg_u_value(S, ra, a);
            du += (j < NE && j != e) ? d : T(0);
        }
        return hsum(du);
    } else {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int j = lane + 32 * r;
            if (j < NE && j != e) {
                const T a = S.a_ee[((j < NUP) == (e < NUP)) ? 1 : 0];
                T ax = min_img(ox - P.x[r], S), ay = min_img(oy - P.y[r], S), az = min_img(oz - P.z[r], S);
                T bx = min_img(nx - P.x[r], S), by = min_img(ny - P.y[r], S), bz = min_img(nz - P.z[r], S);
                T ra = fsqrt(ax * ax + ay * ay + az * az), rb = fsqrt(bx * bx + by * by + bz * bz);
                T ua, dua, lua, ub, dub, lub;
                heg_u(S, ra, a, ua, dua, lua);
                heg_u(S, rb, a, ub, dub, lub);
                du += ub - ua;
                if (GRAD) {
                    T fa = ra > 0 ? dua / ra : T(0), fb = rb > 0 ? dub / rb : T(0);
                    g[0] += fa * ax; g[1] += fa * ay; g[2] += fa * az;
                    g[3] += fb * bx; g[4] += fb * by; g[5] += fb * bz;
                }
            }
        }
        du = hsum(du);
        if (GRAD) {
            go[0] = hsum(g[0]); go[1] = hsum(g[1]); go[2] = hsum(g[2]);
            gn[0] = hsum(g[3]); gn[1] = hsum(g[4]); gn[2] = hsum(g[5]);
        }
        return du;
    }
}

template <class TS>
__global__ void khw_init(const SysH<double>* __restrict__ S, TS* __restrict__ pos, int NE, int W, int Wcap,
                         uint64_t seed) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NE * W) return;
    int e = i / W, w = i - e * W;
    U4 x = rng_draw(seed, (uint32_t)w, 0, (uint32_t)S->perm[e], TAG_INIT);
    double L = S->L;
    pos[(3 * e + 0) * (size_t)Wcap + w] = (TS)(L * to_u01(x.x, 0.0));
    pos[(3 * e + 1) * (size_t)Wcap + w] = (TS)(L * to_u01(x.y, 0.0));
    pos[(3 * e + 2) * (size_t)Wcap + w] = (TS)(L * to_u01(x.z, 0.0));
}

// Single-electron sweeps, one warp per walker.
// Shared bytes per warp of the generic sweep's inverse columns (both sectors).
template <int NM, class T>
__host__ __device__ constexpr size_t hsweep_warp_bytes() { return sizeof(T) * 2 * 2 * NM * 32; }

// The FP32 Gaussian sweep's shared rows: both sectors' inverses in row pairs, a
// column per electron of the sector, then two columns for each of two proposals'
// phases.
template <int NM>
__host__ __device__ constexpr int hgauss_rows() { return (NM + 1) / 2; }
template <int NM>
__host__ __device__ constexpr int hgauss_cols() { return NM + 4; }
template <int NM>
__host__ __device__ constexpr size_t hgauss_warp_bytes() { return 16 * 2 * hgauss_rows<NM>() * hgauss_cols<NM>(); }

// Jastrow change of the RPA form for electron e moving o -> n, both partner rounds
// of a lane in packed instructions: hjastrow_delta<..., false>'s operations in its
// order (rint by adding and subtracting 1.5 2^23, which rounds the same way).
template <int NE, int NUP>
__device__ __forceinline__ float hjastrow_delta_rpa(const SysH<float>& S, const HLanePos<float, NE>& P, int lane, int e,
                                                    float ox, float oy, float oz, float nx, float ny, float nz) {
    const F2 a(S.a_ee[((lane < NUP) == (e < NUP)) ? 1 : 0], S.a_ee[((lane + 32 < NUP) == (e < NUP)) ? 1 : 0]);
    const F2 px(P.x[0], P.x[1]), py(P.y[0], P.y[1]), pz(P.z[0], P.z[1]);
    const F2 one(1.0f), neg(-1.0f), iL(S.invL), nL(-S.L), big(12582912.0f), nbig(-12582912.0f), pb(S.pb), pc(S.pc);
    auto image = [&](float o, F2 q) -> F2 {
        const F2 d = fma2(q, neg, F2(o));
        return fma2(nL, add2(add2(mul2(d, iL), big), nbig), d);
    };
    auto value = [&](float x, float y, float z, float (&u)[2]) {
        const F2 dx = image(x, px), dy = image(y, py), dz = image(z, pz);
        float r2[2], r[2], n[2], den[2];
        fma2(dz, dz, fma2(dx, dx, mul2(dy, dy))).get(r2[0], r2[1]);
        r[0] = fsqrt(r2[0]);
        r[1] = fsqrt(r2[1]);
        const F2 rr(r[0], r[1]);
        fma2(mul2(pc, rr), rr, fma2(pb, rr, one)).get(den[0], den[1]);
        mul2(a, rr).get(n[0], n[1]);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float v = n[k] / den[k];
            u[k] = (r[k] < S.halfL && r[k] > 1e-10f) ? v : 0.0f;
        }
    };
    float uo[2], un[2];
    value(ox, oy, oz, uo);
    value(nx, ny, nz, un);
    float du = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int j = lane + 32 * k;
        const float d = un[k] - uo[k];
        du += (j < NE && j != e) ? d : 0.0f;
    }
    return hsum(du);
}

// FP32 Gaussian sweeps.  The generic form below does the same arithmetic in the
// same order; here a lane's inverse column lies in row pairs (re, re', im, im'), so
// that a ratio and an update take two rows per packed FP32 instruction, and the
// proposal's phases and the moving electron's column are read from shared memory as
// broadcasts instead of two shuffles a row.  The next proposal's phases (its electron
// has not moved yet) are written while this one is decided.  A sector's columns stay
// in registers during its turn (with them in shared memory that pipe was 90 % busy,
// now 62 %); each electron's column is written back before its own proposal.  8 sweeps
// of 8192 walkers: 2.06 ms, 2.19 ms with the columns in shared memory, 2.35 ms in the
// generic form; issue 59 % busy at 415 instructions a proposal.
template <int NE, int NUP, class A>
__device__ __forceinline__ void khw_gauss_walker(const SysH<float>& S, A& a, float4* Dsh, int w) {
    constexpr int NDN = NE - NUP;
    constexpr int NM = NUP > NDN ? NUP : NDN, NR = hgauss_rows<NM>(), NC = hgauss_cols<NM>();
    static_assert(NUP <= 32 && NDN <= 32 && NC <= 32, "one lane per sector electron");
    const int lane = threadIdx.x & 31;
    const int col = min(lane, NC - 1);                    // spare lanes read along and store nothing
    HLanePos<float, NE> P;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = lane + 32 * r;
        const bool ok = j < NE;
        P.x[r] = ok ? a.pos[(3 * j + 0) * (size_t)a.Wcap + w] : 0.0f;
        P.y[r] = ok ? a.pos[(3 * j + 1) * (size_t)a.Wcap + w] : 0.0f;
        P.z[r] = ok ? a.pos[(3 * j + 2) * (size_t)a.Wcap + w] : 0.0f;
    }
    auto row = [&](int sig, int k, bool im) -> size_t {
        return (((size_t)(sig * NM * NM + k * NM + lane)) * 2 + (im ? 1 : 0)) * a.Wcap + w;
    };
#pragma unroll
    for (int sig = 0; sig < 2; ++sig) {
        const bool own = lane < (sig == 0 ? NUP : NDN);
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const bool two = 2 * r + 1 < NM;
            float4 d;
            d.x = own ? a.dinv[row(sig, 2 * r, false)] : 0.0f;
            d.y = own && two ? a.dinv[row(sig, two ? 2 * r + 1 : 0, false)] : 0.0f;
            d.z = own ? a.dinv[row(sig, 2 * r, true)] : 0.0f;
            d.w = own && two ? a.dinv[row(sig, two ? 2 * r + 1 : 0, true)] : 0.0f;
            if (lane < NM) Dsh[(sig * NR + r) * NC + lane] = d;
        }
    }
    unsigned acc = 0;
    int flg = 0;
    for (int it = 0; it < a.n_sweeps; ++it) {
        const uint64_t st = a.step0 + (uint64_t)it;
#pragma unroll 1
        for (int sig = 0; sig < 2; ++sig) {
            float4* D = Dsh + sig * NR * NC;
            const int NS = sig == 0 ? NUP : NDN;
            const float kx = S.kvec[sig][lane][0], ky = S.kvec[sig][lane][1], kz = S.kvec[sig][lane][2];
            const MoveDraw<float> draws = sector_draws<float>(a.seed, (uint32_t)w, st, sig * NUP, NS, lane);
            float csr = 1, csi = 0;                        // pending complex scale of this lane's column
            // proposal q: old and new position, and the phase of row `lane` (zero past
            // the sector) into columns NM + 2 (q mod 2), (cos, cos', sin, sin') of a row
            // pair, and the one after, (-sin, -sin')
            float rx, ry, rz, nx, ny, nz, uacc;
            auto propose = [&](int q) {
                P.get(sig * NUP + q, rx, ry, rz);
                const MoveDraw<float> md = draw_of(draws, q);
                const float step = a.step;
                nx = rx + step * md.n0; ny = ry + step * md.n1; nz = rz + step * md.n2;
                uacc = md.uacc;
                float ps, pc;
                fsincos(kx * nx + ky * ny + kz * nz, &ps, &pc);
                if (lane < 2 * NR) {
                    const bool own = lane < NS;
                    float* f = reinterpret_cast<float*>(D + (lane >> 1) * NC + NM + 2 * (q & 1)) + (lane & 1);
                    f[0] = own ? pc : 0.0f;
                    f[2] = own ? ps : 0.0f;
                    f[4] = own ? -ps : 0.0f;
                }
            };
            propose(0);
            __syncwarp();
            // the lane's column for the sector's turn: rows 2r, 2r + 1 (re, re') and (im, im')
            F2 dre[NR], dim[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                load2x2(D + r * NC + col, dre[r], dim[r]);
            }
            for (int q = 0; q < NS; ++q) {
                const int e = sig * NUP + q;
                const float4* ph = D + NM + 2 * (q & 1);
                const float cx = rx, cy = ry, cz = rz, mx = nx, my = ny, mz = nz, ua = uacc;
                if (q + 1 < NS) propose(q + 1);
                // t_l = sum_j phi_j Dinv[j][l]; R = t_q
                float tr = 0, ti = 0;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    F2 pr, pi, np;
                    load2x2(ph + r * NC, pr, pi);
                    np.v = *reinterpret_cast<const unsigned long long*>(ph + r * NC + 1);
                    float a0, a1, b0, b1;
                    fma2(pr, dre[r], mul2(np, dim[r])).get(a0, a1);
                    fma2(pr, dim[r], mul2(pi, dre[r])).get(b0, b1);
                    tr += a0; ti += b0;
                    if (2 * r + 1 < NM) { tr += a1; ti += b1; }
                }
                const float Rr = __shfl_sync(0xffffffffu, tr, q), Ri = __shfl_sync(0xffffffffu, ti, q);
                const float R2 = Rr * Rr + Ri * Ri;
                float du, g0[3], gn[3];
                if (S.form == 1) du = hjastrow_delta_rpa<NE, NUP>(S, P, lane, e, cx, cy, cz, mx, my, mz);
                else du = hjastrow_delta<NE, NUP, float, false>(S, P, lane, e, cx, cy, cz, mx, my, mz, g0, gn);
                const float prob = R2 * fexp(2 * du);
                if (prob != prob) flg |= FLAG_NONFINITE;
                if (ua < prob && R2 > 0.0f) {
                    // wrap the new position into the box
                    const float wx = mx - S.L * floor(mx * S.invL), wy = my - S.L * floor(my * S.invL),
                                wz = mz - S.L * floor(mz * S.invL);
                    if ((e & 31) == lane) {
                        if (e < 32) { P.x[0] = wx; P.y[0] = wy; P.z[0] = wz; }
                        else { P.x[1] = wx; P.y[1] = wy; P.z[1] = wz; }
                    }
                    // complex Sherman-Morrison: D'[k][l] = D[k][l] - D[k][q] t_l / R; column q
                    // keeps its values and takes the factor 1/R when the sector ends (a
                    // column's scale is 1 until its own electron moves, so t_q and R are
                    // read unscaled), so it is not written while the others read it
                    const float iR2 = 1.0f / R2;
                    const float iRr = Rr * iR2, iRi = -Ri * iR2;              // 1/R
                    const float fr = tr * iRr - ti * iRi, fi = tr * iRi + ti * iRr;   // t_l / R
                    if (lane == q) { csr = iRr; csi = iRi; }
                    if (lane != q) {
                        const F2 f(fi), nfr(-fr), nfi(-fi);
#pragma unroll
                        for (int r = 0; r < NR; ++r) {
                            F2 qr, qi;
                            load2x2(D + r * NC + q, qr, qi);
                            // d - (qr fr - qi fi) and d - (qr fi + qi fr)
                            dre[r] = add2(dre[r], fma2(qr, nfr, mul2(qi, f)));
                            dim[r] = add2(dim[r], fma2(qr, nfi, mul2(qi, nfr)));
                        }
                    }
                    ++acc;
                }
                // the next moving electron's column, for the others to read
                if (lane == q + 1 && lane < NS) {
#pragma unroll
                    for (int r = 0; r < NR; ++r) store2x2(D + r * NC + lane, dre[r], dim[r]);
                }
                __syncwarp();                          // this proposal's reads before the next one's writes
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                float4 d, n;
                dre[r].get(d.x, d.y);
                dim[r].get(d.z, d.w);
                n.x = d.x * csr - d.z * csi; n.z = d.x * csi + d.z * csr;
                n.y = d.y * csr - d.w * csi; n.w = d.y * csi + d.w * csr;
                if (lane < NM) D[r * NC + lane] = n;
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = lane + 32 * r;
        if (j < NE) {
            a.pos[(3 * j + 0) * (size_t)a.Wcap + w] = P.x[r];
            a.pos[(3 * j + 1) * (size_t)a.Wcap + w] = P.y[r];
            a.pos[(3 * j + 2) * (size_t)a.Wcap + w] = P.z[r];
        }
    }
#pragma unroll
    for (int sig = 0; sig < 2; ++sig) {
        if (lane >= (sig == 0 ? NUP : NDN)) continue;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const float4 d = Dsh[(sig * NR + r) * NC + lane];
            a.dinv[row(sig, 2 * r, false)] = d.x;
            a.dinv[row(sig, 2 * r, true)] = d.z;
            if (2 * r + 1 < NM) {
                a.dinv[row(sig, 2 * r + 1, false)] = d.y;
                a.dinv[row(sig, 2 * r + 1, true)] = d.w;
            }
        }
    }
    if (lane == 0) {
        if (acc) atomicAdd(a.acc, (unsigned long long)acc);
        if (flg) atomicOr(a.flags, flg);
    }
}

// A is const volatile SweepArgs<T> (block-shared; see SweepArgs).
template <int NE, int NUP, class T, int MOVE, class A>
__device__ __forceinline__ void khw_sweep_walker(const SysH<T>& S, A& a, typename HComplex<T>::type* Dsh, int w) {
    constexpr int NDN = NE - NUP;
    constexpr int NM = NUP > NDN ? NUP : NDN;
    const int lane = threadIdx.x & 31;
    HLanePos<T, NE> P;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = lane + 32 * r;
        const bool ok = j < NE;
        P.x[r] = ok ? a.pos[(3 * j + 0) * (size_t)a.Wcap + w] : T(0);
        P.y[r] = ok ? a.pos[(3 * j + 1) * (size_t)a.Wcap + w] : T(0);
        P.z[r] = ok ? a.pos[(3 * j + 2) * (size_t)a.Wcap + w] : T(0);
    }
    // complex inverse columns in the warp's shared rows: Dsh[(sig NM + k) 32 + lane]
    // = D^-1[k][lane] (re, im) of sector sig; each lane touches only its own
    // column (HBM storage [2][NM*NM][2][Wcap])
    using C2 = typename HComplex<T>::type;
#pragma unroll
    for (int k = 0; k < NM; ++k) {
        size_t b0 = ((size_t)(0 * NM * NM + k * NM + lane)) * 2 * a.Wcap, b1 = ((size_t)(1 * NM * NM + k * NM + lane)) * 2 * a.Wcap;
        C2 d0, d1;
        d0.x = lane < NUP ? a.dinv[b0 + w] : T(0);
        d0.y = lane < NUP ? a.dinv[b0 + a.Wcap + w] : T(0);
        d1.x = lane < NDN ? a.dinv[b1 + w] : T(0);
        d1.y = lane < NDN ? a.dinv[b1 + a.Wcap + w] : T(0);
        Dsh[(0 * NM + k) * 32 + lane] = d0;
        Dsh[(1 * NM + k) * 32 + lane] = d1;
    }
    unsigned acc = 0;
    int flg = 0;
    for (int it = 0; it < a.n_sweeps; ++it) {
        const uint64_t st = a.step0 + (uint64_t)it;
#pragma unroll
        for (int sig = 0; sig < 2; ++sig) {
            C2* Dc = Dsh + sig * NM * 32 + lane;      // Dc[k * 32] = D^-1[k][lane]
            const int NS = sig == 0 ? NUP : NDN;
            const T kx = S.kvec[sig][lane][0], ky = S.kvec[sig][lane][1], kz = S.kvec[sig][lane][2];
            static_assert(NUP <= 32 && NE - NUP <= 32, "one lane per sector electron");
            const MoveDraw<T> draws = sector_draws<T>(a.seed, (uint32_t)w, st, sig * NUP, NS, lane);
            T csr = 1, csi = 0;                        // pending complex scale of this lane's column (Gaussian moves)
            for (int q = 0; q < NS; ++q) {
                const int e = sig * NUP + q;
                T rx, ry, rz;
                P.get(e, rx, ry, rz);
                const MoveDraw<T> md = draw_of(draws, q);
                T nx, ny, nz, logG = 0, dlx = 0, dly = 0, dlz = 0;
                if (MOVE == MOVE_ONE_DRIFT) {
                    // Re(grad ln D) at the current position: lane l sums (i k_j phi_j) Dinv[j][l]
                    T s, c;
                    fsincos(kx * rx + ky * ry + kz * rz, &s, &c);
                    T ax = 0, ay = 0, az = 0;
#pragma unroll 9
                    for (int j = 0; j < NM; ++j) {
                        T pr = __shfl_sync(0xffffffffu, c, j), pi = __shfl_sync(0xffffffffu, s, j);
                        T kjx = S.kvec[sig][j][0], kjy = S.kvec[sig][j][1], kjz = S.kvec[sig][j][2];
                        // Re(i k phi D) = -k Im(phi D)
                        const C2 d = Dc[j * 32];
                        T im = pr * d.y + pi * d.x;
                        ax -= kjx * im; ay -= kjy * im; az -= kjz * im;
                    }
                    ax = __shfl_sync(0xffffffffu, ax, q); ay = __shfl_sync(0xffffffffu, ay, q); az = __shfl_sync(0xffffffffu, az, q);
                    T g0[3], g1[3];
                    hjastrow_delta<NE, NUP, T, true>(S, P, lane, e, rx, ry, rz, rx, ry, rz, g0, g1);
                    const T tau = a.tau, maxd = a.maxd;
                    dlx = tau * 2 * (ax + g0[0]); dly = tau * 2 * (ay + g0[1]); dlz = tau * 2 * (az + g0[2]);
                    T m = fsqrt(dlx * dlx + dly * dly + dlz * dlz);
                    if (m > maxd) { T sc = maxd / m; dlx *= sc; dly *= sc; dlz *= sc; }
                    T sd2 = fsqrt(2 * tau);
                    nx = rx + dlx + sd2 * md.n0; ny = ry + dly + sd2 * md.n1; nz = rz + dlz + sd2 * md.n2;
                } else {
                    const T step = a.step;
                    nx = rx + step * md.n0; ny = ry + step * md.n1; nz = rz + step * md.n2;
                }
                T ps, pc;
                fsincos(kx * nx + ky * ny + kz * nz, &ps, &pc);
                // t_l = sum_j phi_j Dinv[j][l]; R = t_q
                T tr = 0, ti = 0;
#pragma unroll 9
                for (int j = 0; j < NM; ++j) {
                    T pr = __shfl_sync(0xffffffffu, pc, j), pi = __shfl_sync(0xffffffffu, ps, j);
                    const C2 d = Dc[j * 32];
                    tr += pr * d.x - pi * d.y;
                    ti += pr * d.y + pi * d.x;
                }
                const T Rr = __shfl_sync(0xffffffffu, tr, q), Ri = __shfl_sync(0xffffffffu, ti, q);
                const T R2 = Rr * Rr + Ri * Ri;
                T g0[3], gn[3];
                T du = hjastrow_delta<NE, NUP, T, MOVE == MOVE_ONE_DRIFT>(S, P, lane, e, rx, ry, rz, nx, ny, nz, g0, gn);
                if (MOVE == MOVE_ONE_DRIFT) {
                    // Re(grad ln D') = Re(G / R) with G = sum_j i k_j phi_j(r') Dinv[j][q]
                    T Gx_r = 0, Gy_r = 0, Gz_r = 0, Gx_i = 0, Gy_i = 0, Gz_i = 0;
#pragma unroll 9
                    for (int j = 0; j < NM; ++j) {
                        T pr = __shfl_sync(0xffffffffu, pc, j), pi = __shfl_sync(0xffffffffu, ps, j);
                        const C2 d = Dc[j * 32];
                        T re = pr * d.x - pi * d.y, im = pr * d.y + pi * d.x;
                        T kjx = S.kvec[sig][j][0], kjy = S.kvec[sig][j][1], kjz = S.kvec[sig][j][2];
                        Gx_r -= kjx * im; Gy_r -= kjy * im; Gz_r -= kjz * im;
                        Gx_i += kjx * re; Gy_i += kjy * re; Gz_i += kjz * re;
                    }
                    Gx_r = __shfl_sync(0xffffffffu, Gx_r, q); Gy_r = __shfl_sync(0xffffffffu, Gy_r, q); Gz_r = __shfl_sync(0xffffffffu, Gz_r, q);
                    Gx_i = __shfl_sync(0xffffffffu, Gx_i, q); Gy_i = __shfl_sync(0xffffffffu, Gy_i, q); Gz_i = __shfl_sync(0xffffffffu, Gz_i, q);
                    const T tau = a.tau, maxd = a.maxd;
                    T iR2 = R2 > 0 ? T(1) / R2 : T(0);
                    // Re(G / R) = (G_r R_r + G_i R_i) / |R|^2
                    T cx = (Gx_r * Rr + Gx_i * Ri) * iR2 + gn[0];
                    T cy = (Gy_r * Rr + Gy_i * Ri) * iR2 + gn[1];
                    T cz = (Gz_r * Rr + Gz_i * Ri) * iR2 + gn[2];
                    cx *= 2 * tau; cy *= 2 * tau; cz *= 2 * tau;
                    T m = fsqrt(cx * cx + cy * cy + cz * cz);
                    if (m > maxd) { T sc = maxd / m; cx *= sc; cy *= sc; cz *= sc; }
                    T fx = nx - rx - dlx, fy = ny - ry - dly, fz = nz - rz - dlz;
                    T qx = rx - nx - cx, qy = ry - ny - cy, qz = rz - nz - cz;
                    logG = ((fx * fx + fy * fy + fz * fz) - (qx * qx + qy * qy + qz * qz)) / (4 * tau);
                }
                T prob = R2 * fexp(2 * du);
                if (MOVE == MOVE_ONE_DRIFT) prob *= fexp(logG);
                if (prob != prob) flg |= FLAG_NONFINITE;
                if (md.uacc < prob && R2 > T(0)) {
                    // wrap the new position into the box
                    T wx = nx - S.L * floor(nx * S.invL), wy = ny - S.L * floor(ny * S.invL), wz = nz - S.L * floor(nz * S.invL);
                    if ((e & 31) == lane) {
                        if (e < 32) { P.x[0] = wx; P.y[0] = wy; P.z[0] = wz; }
                        else { P.x[1] = wx; P.y[1] = wy; P.z[1] = wz; }
                    }
                    // complex Sherman-Morrison: D'[k][l] = D[k][l] - D[k][q] t_l / R, D'[k][q] = D[k][q] / R
                    const T iR2 = T(1) / R2;
                    const T iRr = Rr * iR2, iRi = -Ri * iR2;              // 1/R
                    T fr = tr * iRr - ti * iRi, fi = tr * iRi + ti * iRr;   // t_l / R
                    if constexpr (MOVE == MOVE_ONE_GAUSS) {
                        // column q keeps its values and takes the factor 1/R when the
                        // sector ends (a column's scale is 1 until its own electron
                        // moves, so t_q and R are read unscaled)
                        if (lane == q) { fr = 0; fi = 0; csr = iRr; csi = iRi; }
#pragma unroll 9
                        for (int k = 0; k < NM; ++k) {
                            const C2 d = Dc[k * 32];
                            T qr = __shfl_sync(0xffffffffu, d.x, q), qi = __shfl_sync(0xffffffffu, d.y, q);
                            C2 n;
                            n.x = d.x - (qr * fr - qi * fi); n.y = d.y - (qr * fi + qi * fr);
                            Dc[k * 32] = n;
                        }
                    } else {
#pragma unroll 9
                        for (int k = 0; k < NM; ++k) {
                            const C2 d = Dc[k * 32];
                            T qr = __shfl_sync(0xffffffffu, d.x, q), qi = __shfl_sync(0xffffffffu, d.y, q);
                            C2 n;
                            if (lane == q) { n.x = qr * iRr - qi * iRi; n.y = qr * iRi + qi * iRr; }
                            else { n.x = d.x - (qr * fr - qi * fi); n.y = d.y - (qr * fi + qi * fr); }
                            Dc[k * 32] = n;
                        }
                    }
                    ++acc;
                }
            }
            if constexpr (MOVE == MOVE_ONE_GAUSS) {
#pragma unroll 9
                for (int k = 0; k < NM; ++k) {
                    const C2 d = Dc[k * 32];
                    C2 n;
                    n.x = d.x * csr - d.y * csi; n.y = d.x * csi + d.y * csr;
                    Dc[k * 32] = n;
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = lane + 32 * r;
        if (j < NE) {
            a.pos[(3 * j + 0) * (size_t)a.Wcap + w] = P.x[r];
            a.pos[(3 * j + 1) * (size_t)a.Wcap + w] = P.y[r];
            a.pos[(3 * j + 2) * (size_t)a.Wcap + w] = P.z[r];
        }
    }
#pragma unroll
    for (int k = 0; k < NM; ++k) {
        size_t b0 = ((size_t)(0 * NM * NM + k * NM + lane)) * 2 * a.Wcap, b1 = ((size_t)(1 * NM * NM + k * NM + lane)) * 2 * a.Wcap;
        const C2 d0 = Dsh[(0 * NM + k) * 32 + lane], d1 = Dsh[(1 * NM + k) * 32 + lane];
        if (lane < NUP) { a.dinv[b0 + w] = d0.x; a.dinv[b0 + a.Wcap + w] = d0.y; }
        if (lane < NDN) { a.dinv[b1 + w] = d1.x; a.dinv[b1 + a.Wcap + w] = d1.y; }
    }
    if (lane == 0) {
        if (acc) atomicAdd(a.acc, (unsigned long long)acc);
        if (flg) atomicOr(a.flags, flg);
    }
}

// Sweeps of walker w by its warp, with the block's dynamic shared memory.
template <int NM, class T, int MOVE>
__host__ __device__ constexpr size_t hsweep_bytes() {
    return std::is_same<T, float>::value && MOVE == MOVE_ONE_GAUSS ? hgauss_warp_bytes<NM>() : hsweep_warp_bytes<NM, T>();
}
template <int NE, int NUP, class T, int MOVE>
__device__ __forceinline__ void hsweep_walker(const SysH<T>& S, const volatile SweepArgs<T>& a, unsigned char* sm, int w) {
    constexpr int NM = NUP > NE - NUP ? NUP : NE - NUP;
    unsigned char* mine = sm + (size_t)(threadIdx.x >> 5) * hsweep_bytes<NM, T, MOVE>();
    if constexpr (std::is_same<T, float>::value && MOVE == MOVE_ONE_GAUSS)
        khw_gauss_walker<NE, NUP>(S, a, reinterpret_cast<float4*>(mine), w);
    else
        khw_sweep_walker<NE, NUP, T, MOVE>(S, a, reinterpret_cast<typename HComplex<T>::type*>(mine), w);
}

template <int NE, int NUP, class T, int MOVE, int WPB>
// 16 warps per SM for FP32 walkers (four blocks of four: 56 KB of shared
// memory each, at most 128 registers), 8 for FP64 walkers.
__global__ void __launch_bounds__(32 * WPB, (sizeof(T) == 4 ? 16 : 8) / WPB) khw_sweep(const SysH<T>* __restrict__ Sg, T* __restrict__ gpos,
                                                      T* __restrict__ gdinv, int W, int Wcap, int n_sweeps,
                                                      uint64_t step0, T step, T tau, T maxd, uint64_t seed,
                                                      unsigned long long* acc_out, int* flags) {
    __shared__ SysH<T> S;
    __shared__ SweepArgs<T> args;
    extern __shared__ __align__(16) unsigned char hsm[];
    if (threadIdx.x == 0)
        args = SweepArgs<T>{gpos, gdinv, nullptr, acc_out, flags, step0, seed, step, tau, maxd, W, Wcap, n_sweeps, 0};
    load_sysh(&S, Sg, (int)sizeof(SysH<T>));   // ends with a block barrier
    const int w = blockIdx.x * WPB + (threadIdx.x >> 5);
    if (w >= W) return;
    hsweep_walker<NE, NUP, T, MOVE>(S, args, hsm, w);
}

// Batched form: one block per (system, WPB-walker tile); the hardware block
// scheduler balances uneven systems and classes that run side by side.
template <int NE, int NUP, class T, int MOVE, int WPB>
__global__ void __launch_bounds__(32 * WPB, (sizeof(T) == 4 ? 16 : 8) / WPB) khwb_sweep(const BatchTile* __restrict__ tiles, int ntiles,
                                                       const BatchRec* __restrict__ recs,
                                                       const BatchCtl* __restrict__ ctl) {
    __shared__ SysH<T> S;
    __shared__ SweepArgs<T> args;
    extern __shared__ __align__(16) unsigned char hsm[];
    if ((int)blockIdx.x >= ntiles) return;
    const BatchTile tl = tiles[blockIdx.x];
    if (threadIdx.x == 0) args = sweep_args<T>(recs[tl.rec], *ctl);
    load_sysh(&S, static_cast<const SysH<T>*>(recs[tl.rec].tab_s), (int)sizeof(SysH<T>));   // ends with a barrier
    const int w = tl.w0 + (int)(threadIdx.x >> 5);
    if (w >= args.W) return;
    hsweep_walker<NE, NUP, T, MOVE>(S, args, hsm, w);
}

// Row stride of the refresh's matrix scratch (odd: rows and columns read without
// bank conflicts).
constexpr int HRS = 33;

// Inverse of one sector's complex orbital matrix (rows in Mr, Mi) by the warp: lane j
// ends with column j.  |det| goes into (pmag, pexp) (float-float: |det|^2) or logdet.
template <int NM, class TC>
__device__ __forceinline__ void invert_sector(const TC* Mr, const TC* Mi, TC* bc, int NS, int lane, TC (&Ar)[NM],
                                              TC (&Ai)[NM], ff& pmag, int& pexp, double& logdet, bool& ok) {
                #pragma unroll
                for (int i = 0; i < NM; ++i) {
                    bool in = i < NS && lane < NS;
                    Ar[i] = in ? Mr[i * HRS + lane] : TC(i == lane ? 1 : 0);
                    Ai[i] = in ? Mi[i * HRS + lane] : TC(0);
                }
                int src = lane;
#pragma unroll 1
                for (int k = 0; k < NS; ++k) {
                    // column k, row by row, to the warp's broadcast buffer
                    if (lane == k) {
#pragma unroll
                        for (int i = 0; i < NM; ++i) store_pair(bc + 2 * i, Ar[i], Ai[i]);
                    }
                    __syncwarp();
                    // pivot: the largest |D[i][k]| over the rows not yet pivoted, a row
                    // per lane (leading parts, whose bits order as integers; the first
                    // of equal ones)
                    unsigned key = 0;
                    if (lane < NS - k) {
                        TC r, m;
                        load_pair(bc + 2 * lane, r, m);
                        key = __float_as_uint(pivot_mag(r, m));
                    }
                    const unsigned top = __reduce_max_sync(0xffffffffu, key);
                    const int p = __ffs(__ballot_sync(0xffffffffu, lane < NS - k && key == top)) - 1;
                    if (p != 0) {
                        swap_rows<NM>(p, Ar, Ai);             // p is the same on every lane
                        if (lane == 0) {
                            TC r0, i0, rp, ip;
                            load_pair(bc, r0, i0);
                            load_pair(bc + 2 * p, rp, ip);
                            store_pair(bc, rp, ip);
                            store_pair(bc + 2 * p, r0, i0);
                        }
                        __syncwarp();
                    }
                    const int pk = k + p;
                    src = (src == k) ? pk : ((src == pk) ? k : src);
                    TC pr, pi;
                    load_pair(bc, pr, pi);
                    TC pa = pr * pr + pi * pi;
                    if (!(pa > TC(0))) { ok = false; pr = 1; pi = 0; pa = 1; }
                    if constexpr (std::is_same<TC, ff>::value) {
                        pmag = pmag * pa;                  // |det|^2 as a rescaled product
                        ff_rescale(pmag, pexp);
                    } else {
                        logdet += 0.5 * d_log((double)pa);
                    }
                    const TC ipr = pr / pa, ipi = -pi / pa;           // 1/a
                    TC tr, ti;
                    if (lane == k) {
                        tr = TC(1) + ipr; ti = ipi;
                        Ar[0] = ipr; Ai[0] = ipi;
                    } else {
                        tr = Ar[0] * ipr - Ai[0] * ipi; ti = Ar[0] * ipi + Ai[0] * ipr;
                        Ar[0] = tr; Ai[0] = ti;
                    }
#pragma unroll
                    for (int i = 1; i < NM; ++i) {
                        if (i >= NS) continue;
                        TC fr, fi;
                        load_pair(bc + 2 * i, fr, fi);
                        Ar[i] -= fr * tr - fi * ti; Ai[i] -= fr * ti + fi * tr;
                    }
                    __syncwarp();                             // bc is read
                    // rotate registers 0..NS-1 by one: the pivoted row goes last
                    const TC r0 = Ar[0], i0 = Ai[0];
#pragma unroll
                    for (int i = 0; i + 1 < NM; ++i) {
                        if (i + 1 < NS) { Ar[i] = Ar[i + 1]; Ai[i] = Ai[i + 1]; }
                        else if (i + 1 == NS) { Ar[i] = r0; Ai[i] = i0; }
                    }
                    if (NS == NM) { Ar[NM - 1] = r0; Ai[NM - 1] = i0; }
                }
                // unscramble: lane j takes column src(j)
#pragma unroll
                for (int i = 0; i < NM; ++i) {
                    if (i >= NS) break;
                    Ar[i] = hshfl(Ar[i], src);
                    Ai[i] = hshfl(Ai[i], src);
                }
}

// The float-float form: a row's real and imaginary parts share packed instructions,
// in the operations and the order of the generic form (a product's low part and a
// subtraction's operand are carried negated, which rounds the same way).  Half the
// instructions also keep the pivot loop's body inside the instruction cache, whose
// misses were 45 % of the generic form's stalls.
struct C2 { F2 hi, lo; };                             // complex float-float: (re, im) of both parts
// a + b as operator+(ff, ff)
__device__ __forceinline__ C2 add_c2(C2 a, C2 b) {
    const F2 s = add2(a.hi, b.hi), bb = sub2(s, a.hi);
    const F2 e = add2(sub2(a.hi, sub2(s, bb)), sub2(b.hi, bb));
    const F2 t = add2(e, add2(a.lo, b.lo));
    const F2 h = add2(s, t);
    return {h, sub2(t, sub2(h, s))};
}
// -(f t) for a splatted factor -f (nfh, nfl) and -t (nth, ntl), t.hi = th; low part negated
__device__ __forceinline__ C2 mul_neg(F2 nfh, F2 nfl, F2 th, F2 nth, F2 ntl) {
    const F2 q = mul2(nfh, th);
    F2 ne = fma2(nfh, nth, q);
    ne = fma2(nfh, ntl, ne);
    ne = fma2(nfl, nth, ne);
    const F2 h = sub2(q, ne);
    return {h, add2(ne, sub2(h, q))};
}
template <int NM>
__device__ __forceinline__ void invert_sector(const ff* Mr, const ff* Mi, ff* bc, int NS, int lane, ff (&Ar)[NM],
                                              ff (&Ai)[NM], ff& pmag, int& pexp, double&, bool& ok) {
    C2 A[NM];
#pragma unroll
    for (int i = 0; i < NM; ++i) {
        const bool in = i < NS && lane < NS;
        const ff r = in ? Mr[i * HRS + lane] : ff(i == lane ? 1 : 0), m = in ? Mi[i * HRS + lane] : ff(0);
        A[i] = {F2(r.hi, m.hi), F2(r.lo, m.lo)};
    }
    float4* b4 = reinterpret_cast<float4*>(bc);        // [row](re.hi, im.hi, re.lo, im.lo), negated
    int src = lane;
#pragma unroll 1
    for (int k = 0; k < NS; ++k) {
        if (lane == k) {
#pragma unroll
            for (int i = 0; i < NM; ++i) {
                float4 v;
                A[i].hi.get(v.x, v.y);
                A[i].lo.get(v.z, v.w);
                b4[i] = make_float4(-v.x, -v.y, -v.z, -v.w);
            }
        }
        __syncwarp();
        unsigned key = 0;
        if (lane < NS - k) {
            const float4 v = b4[lane];
            key = __float_as_uint(pivot_mag(ff(v.x, v.z), ff(v.y, v.w)));
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, key);
        const int p = __ffs(__ballot_sync(0xffffffffu, lane < NS - k && key == top)) - 1;
        if (p != 0) {
#pragma unroll
            for (int r = 1; r < NM; ++r)
                if (p == r) { const C2 t = A[0]; A[0] = A[r]; A[r] = t; }   // the same row on every lane
            if (lane == 0) {
                const float4 u = b4[0], v = b4[p];
                b4[0] = v;
                b4[p] = u;
            }
            __syncwarp();
        }
        const int pk = k + p;
        src = (src == k) ? pk : ((src == pk) ? k : src);
        const float4 pv = b4[0];
        ff pr(-pv.x, -pv.z), pi(-pv.y, -pv.w);
        ff pa = pr * pr + pi * pi;
        if (!(pa > ff(0))) { ok = false; pr = 1; pi = 0; pa = 1; }
        pmag = pmag * pa;                              // |det|^2 as a rescaled product
        ff_rescale(pmag, pexp);
        const ff ipr = pr / pa, ipi = -pi / pa;        // 1/a
        ff ar, ai, tr, ti;
        A[0].hi.get(ar.hi, ai.hi);
        A[0].lo.get(ar.lo, ai.lo);
        if (lane == k) {
            tr = ff(1) + ipr; ti = ipi;
            ar = ipr; ai = ipi;
        } else {
            tr = ar * ipr - ai * ipi; ti = ar * ipi + ai * ipr;
            ar = tr; ai = ti;
        }
        // -(f t) = (-fr)(tr, ti) + (-fi)(-ti, tr)
        const F2 th(tr.hi, ti.hi), nth(-tr.hi, -ti.hi), ntl(-tr.lo, -ti.lo);
        const F2 uh(-ti.hi, tr.hi), nuh(ti.hi, -tr.hi), nul(ti.lo, -tr.lo);
        const C2 first{F2(ar.hi, ai.hi), F2(ar.lo, ai.lo)};
        // rows 1..NS-1 lose f x row k and move one register down; row k goes last
#pragma unroll
        for (int i = 1; i < NM; ++i) {
            if (i == NS) A[i - 1] = first;
            if (i >= NS) continue;
            const float4 f = b4[i];
            const C2 x = mul_neg(F2(f.x), F2(f.z), th, nth, ntl), y = mul_neg(F2(f.y), F2(f.w), uh, nuh, nul);
            // x + y with both low parts negated: e - (x.lo + y.lo)
            const F2 s = add2(x.hi, y.hi), bb = sub2(s, x.hi);
            const F2 e = add2(sub2(x.hi, sub2(s, bb)), sub2(y.hi, bb));
            const F2 t = sub2(e, add2(x.lo, y.lo)), h = add2(s, t);
            A[i - 1] = add_c2(A[i], C2{h, sub2(t, sub2(h, s))});
        }
        if (NS == NM) A[NM - 1] = first;
        __syncwarp();                                  // bc is read
    }
    // unscramble: lane j takes column src(j)
#pragma unroll
    for (int i = 0; i < NM; ++i) {
        float a0, a1, b0, b1;
        A[i].hi.get(a0, a1);
        A[i].lo.get(b0, b1);
        Ar[i] = ff(a0, b0);
        Ai[i] = ff(a1, b1);
        if (i >= NS) continue;
        Ar[i] = hshfl(Ar[i], src);
        Ai[i] = hshfl(Ai[i], src);
    }
}

// FP64 (or FP32) full evaluation: complex Gauss-Jordan, kinetic terms, Ewald.
// PART 0: the whole refresh.  The float-float refresh of FP32 walkers can
// also run as two launches over per-walker scratch drows [7][NE][Wcap]:
// PART 1, the determinant half (orbital matrix, inverse, log|D| into glog,
// grad ln D and lap D / D per electron into drows), and PART 2, the energy
// half (Jastrow, Ewald sums, E_L), which reads them back.  Each launch
// carries half the code and PART 2 none of the inversion's registers.
template <int NE, int NUP, class TC, class TS, int PART, class A>
__device__ __forceinline__ double khw_measure_walker(const SysH<TC>& S, A& a, TC* Mr, int w, bool act) {
    static_assert(PART == 0 || std::is_same<TC, ff>::value, "the two-part refresh is float-float only");
    constexpr int NDN = NE - NUP;
    constexpr int NM = NUP > NDN ? NUP : NDN;
    const int lane = threadIdx.x & 31;
    TC* Mi = Mr + NM * HRS;                           // Mr: [re|im][row][lane]
    TC* bc = Mr + 2 * NM * HRS;                       // [row][re|im] of the pivot column
    double e_l = 0.0;
    if (act) {
        HLanePos<TC, NE> P;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int j = lane + 32 * r;
            const bool ok = j < NE;
            P.x[r] = ok ? (TC)a.pos[(3 * j + 0) * (size_t)a.Wcap + w] : TC(0);
            P.y[r] = ok ? (TC)a.pos[(3 * j + 1) * (size_t)a.Wcap + w] : TC(0);
            P.z[r] = ok ? (TC)a.pos[(3 * j + 2) * (size_t)a.Wcap + w] : TC(0);
        }
        double logdet = 0.0;
        ff pmag = ff(1.0f);                       // float-float form: |det|^2 = pmag 2^pexp
        int pexp = 0;
        bool ok = true;
        TC gdx[2] = {0, 0}, gdy[2] = {0, 0}, gdz[2] = {0, 0}, gqx[2] = {0, 0}, gqy[2] = {0, 0}, gqz[2] = {0, 0};
        TC ldet[2] = {0, 0};
        if constexpr (PART != 2) {
        // one copy of the sector's code, for the instruction cache
#pragma unroll 1
        for (int sig = 0; sig < 2; ++sig) {
            const int NS = NUP == NDN || sig == 0 ? NUP : NDN;
            if constexpr (std::is_same<TC, ff>::value) {
                // opposite wave vectors share a sine and cosine (every step of fsincos
                // is odd or even in its argument, to the bit): (pair of columns,
                // electron) tasks over the lanes, 378 of them for an untwisted cell's 27
                // columns where a lane per column took 27 rounds
                float* pos = reinterpret_cast<float*>(bc);
                if (lane < NS) {
                    const int e = sig * NUP + lane;
#pragma unroll
                    for (int c = 0; c < 3; ++c) pos[3 * lane + c] = a.pos[(3 * e + c) * (size_t)a.Wcap + w];
                }
                __syncwarp();
                const int nr = S.n_rep[sig];
#pragma unroll 1
                for (int t = lane; t < nr * NS; t += 32) {
                    const int q = t / nr, i = t - q * nr, col = S.rep[sig][i], mate = S.mate[sig][i];
                    const TC kx = S.kvec[sig][col][0], ky = S.kvec[sig][col][1], kz = S.kvec[sig][col][2];
                    const TC rx = TC(pos[3 * q]), ry = TC(pos[3 * q + 1]), rz = TC(pos[3 * q + 2]);
                    TC s, c;
                    fsincos(kx * rx + ky * ry + kz * rz, &s, &c);
                    Mr[q * HRS + col] = c;
                    Mi[q * HRS + col] = s;
                    if (mate != 255) {
                        Mr[q * HRS + mate] = c;
                        Mi[q * HRS + mate] = -s;
                    }
                }
            } else {
                const TC kx = S.kvec[sig][lane][0], ky = S.kvec[sig][lane][1], kz = S.kvec[sig][lane][2];
                for (int q = 0; q < NS; ++q) {
                    TC rx, ry, rz;
                    P.get(sig * NUP + q, rx, ry, rz);
                    TC s, c;
                    fsincos(kx * rx + ky * ry + kz * rz, &s, &c);
                    Mr[q * HRS + lane] = c;
                    Mi[q * HRS + lane] = s;
                }
            }
            __syncwarp();
            // complex Gauss-Jordan in place: lane j carries column j of D and
            // ends with column j of D^-1.  Step k: pivot row p by |D[i][k]|,
            // rows k and p interchanged; with a = D[k][k], row k is divided by
            // a, column k becomes -D[i][k]/a (and 1/a on the diagonal), the rest
            // loses D[i][k] x row k.  Lane k's own update is the same form with
            // t = 1 + 1/a.  The row interchanges are undone at the end as column
            // interchanges in reverse order: lane j gathers column src(j),
            // src = tau_{n-1}( ... tau_0(j)), tau_k the swap of k and p_k.
            // The pivot loop is rolled (one copy of the step's code, which an
            // unrolled loop would repeat NS times): the registers hold the rows
            // rotated so that row k sits in register 0 at step k -- the rows not
            // yet pivoted in registers 0..NS-1-k, in the unrolled form's order,
            // the pivoted ones after them -- and each step ends by moving
            // register 0 to the back.  After NS steps the order is row k in
            // register k again.
            TC Ar[NM], Ai[NM];
            invert_sector<NM>(Mr, Mi, bc, NS, lane, Ar, Ai, pmag, pexp, logdet, ok);
            TC (&Ir)[NM] = Ar;
            TC (&Ii)[NM] = Ai;
            if (a.write_state && lane < NS) {
#pragma unroll
                for (int k = 0; k < NM; ++k) {
                    if (k >= NS) break;
                    size_t b = ((size_t)(sig * NM * NM + k * NM + lane)) * 2 * a.Wcap;
                    a.dinv[b + w] = (TS)Ir[k];
                    a.dinv[b + a.Wcap + w] = (TS)Ii[k];
                }
            }
            // lane = electron row q: grad ln D = sum_j Dinv[j][q] i k_j phi_j(r_q); lap D / D = -sum_j Dinv phi k^2
            // (a rolled loop over a thread-local copy of the column: unrolled it is
            // longer than the instruction cache)
            if (lane < NS) {
                TC Dr[NM], Dm[NM];
#pragma unroll
                for (int j = 0; j < NM; ++j) { Dr[j] = Ir[j]; Dm[j] = Ii[j]; }
                TC ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0, lr = 0;
#pragma unroll 1
                for (int j = 0; j < NS; ++j) {
                    const TC pr = Mr[lane * HRS + j], pi = Mi[lane * HRS + j], dr = Dr[j], di = Dm[j];
                    TC re = mul_lazy(pr, dr), im = mul_lazy(pr, di);
                    macc(re, -pi, di);
                    macc(im, pi, dr);
                    re = macc_norm(re);
                    im = macc_norm(im);
                    const TC kjx = -S.kvec[sig][j][0], kjy = -S.kvec[sig][j][1], kjz = -S.kvec[sig][j][2];
                    macc(ax, kjx, im); macc(ay, kjy, im); macc(az, kjz, im);        // Re(i k w phi)
                    if (S.quirk_cross) { macc(bx, kjx, di); macc(by, kjy, di); macc(bz, kjz, di); }   // Re(i k w), reference form
                    macc(lr, -S.k2[sig][j], re);
                }
                ax = macc_norm(ax); ay = macc_norm(ay); az = macc_norm(az);
                bx = macc_norm(bx); by = macc_norm(by); bz = macc_norm(bz); lr = macc_norm(lr);
                gdx[sig] = ax; gdy[sig] = ay; gdz[sig] = az;
                gqx[sig] = bx; gqy[sig] = by; gqz[sig] = bz;
                ldet[sig] = lr;
            }
            __syncwarp();
        }
        if constexpr (std::is_same<TC, ff>::value)
            logdet = 0.5 * (d_log((double)pmag) + (double)pexp * 0.6931471805599453);
        }
        if constexpr (PART == 1) {
#pragma unroll
            for (int sig = 0; sig < 2; ++sig) {
                const int NS = sig == 0 ? NUP : NDN;
                if (lane < NS) {
                    const int i = sig * NUP + lane;
                    const TC v[7] = {gdx[sig], gdy[sig], gdz[sig], gqx[sig], gqy[sig], gqz[sig], ldet[sig]};
#pragma unroll
                    for (int c = 0; c < 7; ++c) ff_store(a.rows + (size_t)(c * NE + i) * a.Wcap + w, v[c]);
                }
            }
            if (lane == 0) {
                if (!ok) atomicOr(a.flags, FLAG_SINGULAR);
                a.log[w] = logdet;
            }
            return 0.0;
        }
        if constexpr (PART == 2) {
#pragma unroll
            for (int sig = 0; sig < 2; ++sig) {
                const int NS = sig == 0 ? NUP : NDN;
                if (lane < NS) {
                    const int i = sig * NUP + lane;
                    TC v[7];
#pragma unroll
                    for (int c = 0; c < 7; ++c) v[c] = ff_load(a.rows + (size_t)(c * NE + i) * a.Wcap + w);
                    gdx[sig] = v[0]; gdy[sig] = v[1]; gdz[sig] = v[2];
                    gqx[sig] = v[3]; gqy[sig] = v[4]; gqz[sig] = v[5]; ldet[sig] = v[6];
                }
            }
            logdet = a.log[w];
        }
        // Jastrow and real-space Ewald, each unordered pair once, spread evenly
        // over the lanes: pair p < NE (NE-1)/2 pairs electron i = p mod NE with
        // j = i + p / NE + 1 (mod NE) for the first NE floor((NE-1)/2) pairs and
        // i = p - that with i + NE/2 for the rest (even NE).  Consecutive pairs
        // have distinct i and distinct j, so the lanes add the gradient and
        // Laplacian terms of their i, and then of their j, to shared sums
        // without conflicts.  Per-electron sums over all partners from both
        // ends took 108 pair evaluations on 27 of 32 lanes against 45 here.
        // The minimum image term is in the compute type (FP64 for FP32 compute);
        // the other 26 images lie beyond L/2, where each term is below
        // erfc(alpha L/2)/(L/2), and are summed in FP32.
        TC u = 0, kin = 0;
        double vreal = 0.0;
        ff vreal_ff = ff(0.0f);
        {
            TC* ps = Mr;                                  // [3][NE] positions, then [4][NE] sums
            TC* sums = Mr + 3 * NE;
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int j = lane + 32 * r;
                if (j < NE) {
                    ps[j] = P.x[r]; ps[NE + j] = P.y[r]; ps[2 * NE + j] = P.z[r];
#pragma unroll
                    for (int c = 0; c < 4; ++c) sums[c * NE + j] = TC(0);
                }
            }
            __syncwarp();
            static_assert(NE > 32, "the lanes of one round hold distinct electrons");
            constexpr int NPAIR = NE * (NE - 1) / 2, HALF = (NE - 1) / 2, FULL = NE * HALF;
            for (int p0 = 0; p0 < NPAIR; p0 += 32) {
                const bool on = p0 + lane < NPAIR;
                const int p = on ? p0 + lane : NPAIR - 1;
                int i, j;
                if (p < FULL) {
                    i = p % NE;
                    j = i + p / NE + 1;
                } else {
                    i = p - FULL;
                    j = i + NE / 2;
                }
                if (j >= NE) j -= NE;
                const TC dx = pair_image(ps[i], ps[j], S), dy = pair_image(ps[NE + i], ps[NE + j], S),
                         dz = pair_image(ps[2 * NE + i], ps[2 * NE + j], S);
                const TC r2 = length2(dx, dy, dz);
                const TC r = fsqrt(r2);
                const bool apart = on && r > TC(1e-10);
                const TC ri = apart ? pair_rcp(r) : TC(0);
                TC uu, f, l;
                heg_pair(S, r, r2, ri, S.a_ee[((j < NUP) == (i < NUP)) ? 1 : 0], uu, f, l);
                if (on) u += uu;
                const TC g[4] = {f * dx, f * dy, f * dz, l};
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (on) sums[c * NE + i] = add_lazy(sums[c * NE + i], g[c]);
                __syncwarp();
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (on) sums[c * NE + j] = add_lazy(sums[c * NE + j], c < 3 ? -g[c] : g[c]);
                __syncwarp();
                if constexpr (std::is_same<TC, ff>::value) {
                    if (apart) vreal_ff += erfc_ff(static_cast<const KTable*>(a.kt)->erfc_tab, S.alpha * r) * ri;
                } else {
                    if (apart) vreal += erfc((double)S.alpha * (double)r) / (double)r;
                }
                if (S.real_images) {
                    // box units: the image shifts are exact integers; the sum is
                    // scaled by 1/L in the compute type
                    const float acc = image_erfc(lead(dx * S.invL), lead(dy * S.invL), lead(dz * S.invL), S.aL, S.rc2u,
                                                 S.a2l2);
                    if (on) {
                        if constexpr (std::is_same<TC, ff>::value) vreal_ff += ff(acc) * S.invL;
                        else vreal += (double)acc * (double)S.invL;
                    }
                }
            }
#pragma unroll
            for (int sig = 0; sig < 2; ++sig) {
                const int NS = sig == 0 ? NUP : NDN;
                const int i = sig * NUP + lane;
                if (lane < NS) {
                    const TC gx = macc_norm(sums[i]), gy = macc_norm(sums[NE + i]), gz = macc_norm(sums[2 * NE + i]),
                             lu = macc_norm(sums[3 * NE + i]);
                    TC cx = S.quirk_cross ? gqx[sig] : gdx[sig], cy = S.quirk_cross ? gqy[sig] : gdy[sig],
                       cz = S.quirk_cross ? gqz[sig] : gdz[sig];
                    TC lp = ldet[sig] + lu + gx * gx + gy * gy + gz * gz + TC(2) * (cx * gx + cy * gy + cz * gz);
                    kin += lp;
                    if (a.grad) {
                        a.grad[((size_t)w * NE + i) * 3 + 0] = (double)(gdx[sig] + gx);
                        a.grad[((size_t)w * NE + i) * 3 + 1] = (double)(gdy[sig] + gy);
                        a.grad[((size_t)w * NE + i) * 3 + 2] = (double)(gdz[sig] + gz);
                    }
                    if (a.lap) a.lap[(size_t)w * NE + i] = (double)lp;
                }
            }
            __syncwarp();
        }
        // Reciprocal Ewald: sum over the half space of integer vectors n of
        // w_n |rho_n|^2, rho_n = sum_i e^{2 pi i n.r_i / L}.  With c, s the cosines
        // and sines of an electron's phases (a x, b y, c z), the sums over the sign
        // combinations of an octant vector (a, b, c) collapse: the cross terms of
        // the eight sums T = sum_i {c,s}_x {c,s}_y {c,s}_z cancel and
        // sum_{signs} |rho|^2 = (number of distinct signs) sum T^2.  A lane takes
        // an octant vector and runs over the electrons, whose phases (powers
        // 0..K of e^{2 pi i x / L} per axis) are in the warp's shared memory:
        // 4 products and 8 multiply-adds per octant vector and electron for up
        // to 4 half-space vectors, and no reduction between lanes.  A lane per
        // electron, with a running phase and a warp reduction per vector, took
        // about 275 000 sub-partition cycles per walker against 45 000 here.
        TC vkt = TC(0);
        {
            const int K1 = S.kmax + 1;
            TC* ph = Mr;                                  // [3 (K+1)][NE] pairs (cos, sin)
            for (int it = lane; it < 3 * NE; it += 32) {
                const int ax = it / NE, i = it - ax * NE;
                TC c1, s1;
                unit_phase((TC)a.pos[(3 * i + ax) * (size_t)a.Wcap + w], S, c1, s1);
                TC c = TC(1), sn = TC(0);
                TC* out = ph + 2 * ((size_t)ax * K1 * NE + i);
                for (int n = 0; n < K1; ++n) {
                    out[0] = c;
                    out[1] = sn;
                    out += 2 * NE;
                    const TC t = c * c1 - sn * s1;
                    sn = c * s1 + sn * c1;
                    c = t;
                }
            }
            __syncwarp();
            const KTable* KT = static_cast<const KTable*>(a.kt);
            for (int t = lane; t < S.nt; t += 32) {
                const int v = KT->tri[t];
                const TC* px = ph + 2 * NE * (v & 255);
                const TC* py = ph + 2 * NE * (K1 + ((v >> 8) & 255));
                const TC* pz = ph + 2 * NE * (2 * K1 + (v >> 16));
                TC T[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) T[q] = TC(0);
#pragma unroll 2
                for (int i = 0; i < NE; ++i) {
                    TC xc, xs, yc, ys, zc, zs;
                    load_pair(px + 2 * i, xc, xs);
                    load_pair(py + 2 * i, yc, ys);
                    load_pair(pz + 2 * i, zc, zs);
                    const TC cc = mul_lazy(xc, yc), cs = mul_lazy(xc, ys), sc = mul_lazy(xs, yc), ss = mul_lazy(xs, ys);
                    macc(T[0], cc, zc); macc(T[1], cc, zs);
                    macc(T[2], cs, zc); macc(T[3], cs, zs);
                    macc(T[4], sc, zc); macc(T[5], sc, zs);
                    macc(T[6], ss, zc); macc(T[7], ss, zs);
                }
                TC q = TC(0);
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    const TC x = macc_norm(T[m]);
                    q += x * x;
                }
                vkt += kweight<TC>(KT, t) * q;
            }
        }
        const double vk = (double)hsum(vkt);
        u = hsum(u);
        kin = hsum(kin);
        if constexpr (std::is_same<TC, ff>::value) vreal = (double)hsum(vreal_ff);
        else vreal = hsum(vreal);
        double V = vreal + vk + S.ksum_const + S.e_const;
        e_l = -0.5 * (double)kin + V;
        if (lane == 0) {
            int fl = 0;
            if (!ok) fl |= FLAG_SINGULAR;
            if (!isfinite(e_l)) fl |= FLAG_NONFINITE;
            if (fl) atomicOr(a.flags, fl);
            if (a.write_state) { a.log[w] = logdet + (double)u; a.sign[w] = 1; a.el[w] = e_l; }
        }
    }
    return act ? e_l : 0.0;
}

template <int WPB>
__device__ __forceinline__ void hwarp_block_partial(double v, double* partial, int slot) {
    __shared__ double ps[WPB];
    if ((threadIdx.x & 31) == 0) ps[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        Comp c{0.0, 0.0};
        for (int i = 0; i < WPB; ++i) c = comp_add(c, Comp{ps[i], 0.0});
        partial[2 * slot] = c.s;
        partial[2 * slot + 1] = c.c;
    }
    __syncthreads();
}

// Shared words per warp of a refresh launch: the orbital matrix rows of the
// determinant half, and for the energy half the pair sums (positions and four
// sums per electron), then the phase table of a reciprocal cutoff kmax.
template <int NE, int NUP, int PART>
__host__ __device__ constexpr int hmeasure_warp_words(int kmax) {
    const int det = PART == 2 ? 0 : 2 * (NUP > NE - NUP ? NUP : NE - NUP) * (HRS + 1);
    const int pair = PART == 1 ? 0 : 7 * NE, ph = PART == 1 ? 0 : 6 * (kmax + 1) * NE;
    const int e = pair > ph ? pair : ph;
    return det > e ? det : e;
}
// Energy-half blocks per SM: 12 warps at up to 168 registers (the phase table
// takes 73 KB a block at kmax = 6).

template <int NE, int NUP, class TC, class TS, int WPB, int PART = 0>
__global__ void __launch_bounds__(32 * WPB, PART == 0 ? 2 : 3) khw_measure(
    const SysH<TC>* __restrict__ Sg, const KTable* __restrict__ KT, const TS* __restrict__ gpos,
    TS* __restrict__ gdinv, double* __restrict__ glog, int* __restrict__ gsign, double* __restrict__ gel, int W,
    int Wcap, int write_state, double* __restrict__ out_grad, double* __restrict__ out_lap, double* partial,
    int* flags, float2* __restrict__ drows) {
    extern __shared__ __align__(16) unsigned char hsm[];
    __shared__ MeasureArgs<TS> args;
    SysH<TC>& S = *reinterpret_cast<SysH<TC>*>(hsm);
    TC* rows = reinterpret_cast<TC*>(hsm + ((sizeof(SysH<TC>) + 15) / 16) * 16);
    if (threadIdx.x == 0)
        args = MeasureArgs<TS>{gpos, gdinv, glog, gsign, gel, out_grad, out_lap, flags, drows, KT, W, Wcap,
                               write_state};
    load_sysh(&S, Sg, (int)sizeof(SysH<TC>));   // ends with a block barrier
    const volatile MeasureArgs<TS>& a = args;
    const int wib = threadIdx.x >> 5;
    const int w = blockIdx.x * WPB + wib;
    double e_l = khw_measure_walker<NE, NUP, TC, TS, PART>(
        S, a, rows + (size_t)wib * hmeasure_warp_words<NE, NUP, PART>(S.kmax), w, w < W);
    if (PART != 1 && partial) hwarp_block_partial<WPB>(e_l, partial, blockIdx.x);
}

// Batched form (compute type TC, state written, per-tile E_L partials), one
// block per tile.
template <int NE, int NUP, class TC, class TS, int WPB, int PART = 0>
__global__ void __launch_bounds__(32 * WPB, PART == 0 ? 2 : 3) khwb_measure(const BatchTile* __restrict__ tiles,
                                                                         int ntiles, const BatchRec* __restrict__ recs,
                                                                         double* tile_partial) {
    extern __shared__ __align__(16) unsigned char hsm[];
    __shared__ MeasureArgs<TS> args;
    SysH<TC>& S = *reinterpret_cast<SysH<TC>*>(hsm);
    TC* rows = reinterpret_cast<TC*>(hsm + ((sizeof(SysH<TC>) + 15) / 16) * 16);
    if ((int)blockIdx.x >= ntiles) return;
    const int wib = threadIdx.x >> 5;
    const BatchTile tl = tiles[blockIdx.x];
    if (threadIdx.x == 0) args = measure_args<TS>(recs[tl.rec]);
    load_sysh(&S, static_cast<const SysH<TC>*>(recs[tl.rec].tab_d), (int)sizeof(SysH<TC>));   // ends with a barrier
    const volatile MeasureArgs<TS>& a = args;
    const int w = tl.w0 + wib;
    double e_l = khw_measure_walker<NE, NUP, TC, TS, PART>(
        S, a, rows + (size_t)wib * hmeasure_warp_words<NE, NUP, PART>(S.kmax), w, w < a.W);
    if (PART != 1) hwarp_block_partial<WPB>(e_l, tile_partial, blockIdx.x);
}

int launch_sum_partials(const double* partial, int nblk, int nrows, double* out, cudaStream_t st);

template <int NE, int NUP>
struct HegShapeOps {
    static constexpr int NM = NUP > NE - NUP ? NUP : NE - NUP;
    static constexpr int WPB = 4;

    // Device copies: [SysH<T> | pad | KTable], cached per system and rebuilt
    // when the parameters change (HostSys::version).
    template <class T>
    static int table(const HostSys& hs, const SysH<T>** out, const KTable** kt = nullptr) {
        const int slot = std::is_same<T, double>::value ? 0 : (std::is_same<T, float>::value ? 1 : 2);
        const size_t off = ((sizeof(SysH<T>) + 255) / 256) * 256;
        if (!hs.dev_table[slot] || hs.dev_table_version[slot] != hs.version) {
            std::vector<unsigned char> buf(off + sizeof(KTable));
            SysH<T>* h = reinterpret_cast<SysH<T>*>(buf.data());
            KTable* k = reinterpret_cast<KTable*>(buf.data() + off);
            if (!fill_sysh<T>(hs, NE, NUP, *h, *k)) return 7;
            if (!hs.dev_table[slot] && cudaMalloc(&hs.dev_table[slot], buf.size()) != cudaSuccess) return 8;
            if (cudaMemcpy(hs.dev_table[slot], buf.data(), buf.size(), cudaMemcpyHostToDevice) != cudaSuccess) return 2;
            hs.dev_table_version[slot] = hs.version;
        }
        *out = static_cast<const SysH<T>*>(hs.dev_table[slot]);
        if (kt) *kt = reinterpret_cast<const KTable*>(static_cast<const unsigned char*>(hs.dev_table[slot]) + off);
        return 0;
    }

    // ---- batched launches ---------------------------------------------------
    // tab_s: the sweep table (walker precision); tab_d: the refresh table
    // (FP64 for FP64 walkers, float-float for FP32 walkers).
    static int batch_tables(const HostSys& hs, int prec, BatchRec& r) {
        const KTable* kt;
        if (prec == 0) {
            const SysH<double>* d;
            int rc = table<double>(hs, &d, &kt);
            if (rc) return rc;
            r.tab_d = r.tab_s = d;
            r.ktab = kt;
            return 0;
        }
        const SysH<ff>* m;
        const SysH<float>* f;
        int rc = table<ff>(hs, &m, &kt);
        if (!rc) rc = table<float>(hs, &f);
        if (rc) return rc;
        r.tab_d = m;
        r.tab_s = f;
        r.ktab = kt;
        return 0;
    }

    template <class T, int MOVE>
    static int batch_sweep_t(const BatchClass& bc, const BatchCtl* ctl, cudaStream_t st, int* occ) {
        auto kern = khwb_sweep<NE, NUP, T, MOVE, WPB>;
        const size_t smem = WPB * hsweep_bytes<NM, T, MOVE>();
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
                return 2;
            cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
            attr = true;
        }
        if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, 32 * WPB, smem) == cudaSuccess ? 0 : 2;
        if (bc.ntiles == 0) return 0;
        kern<<<bc.ntiles, 32 * WPB, smem, st>>>(bc.tiles, bc.ntiles, bc.recs, ctl);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    // The electron-gas sweep has no fixed-node form: batches of it run VMC only.
    static int batch_sweep(const BatchClass& bc, int mk, const BatchCtl* ctl, cudaStream_t st, int* occ = nullptr) {
        if (mk == MOVE_ONE_GAUSS)
            return bc.prec == 0 ? batch_sweep_t<double, MOVE_ONE_GAUSS>(bc, ctl, st, occ)
                                : batch_sweep_t<float, MOVE_ONE_GAUSS>(bc, ctl, st, occ);
        if (mk == MOVE_ONE_DRIFT)
            return bc.prec == 0 ? batch_sweep_t<double, MOVE_ONE_DRIFT>(bc, ctl, st, occ)
                                : batch_sweep_t<float, MOVE_ONE_DRIFT>(bc, ctl, st, occ);
        return 7;
    }

    template <class TC, class TS, int PART>
    static size_t measure_smem(int kmax) {
        return ((sizeof(SysH<TC>) + 15) / 16) * 16 + sizeof(TC) * WPB * hmeasure_warp_words<NE, NUP, PART>(kmax);
    }

    template <class TC, class TS, int PART>
    static int batch_measure_t(const BatchClass& bc, cudaStream_t st, int* occ) {
        const size_t smem = measure_smem<TC, TS, PART>(bc.kmax);
        auto kern = khwb_measure<NE, NUP, TC, TS, WPB, PART>;
        // the largest cutoff's, whatever this one: a limit that depends on the call could be
        // lowered again by another thread's
        static bool attr = false;
        if (!attr) {
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)measure_smem<TC, TS, PART>(HMAX_KMAX));
            attr = true;
        }
        if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, 32 * WPB, smem) == cudaSuccess ? 0 : 2;
        if (bc.ntiles == 0) return 0;
        kern<<<bc.ntiles, 32 * WPB, smem, st>>>(bc.tiles, bc.ntiles, bc.recs, bc.tile_partial);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    // FP32 walker sets (which carry the refresh scratch) refresh in two
    // launches, FP64 ones in one; the occupancy reported is the lower of the
    // two halves'.
    static int batch_measure(const BatchClass& bc, cudaStream_t st, int* occ = nullptr) {
        if (bc.prec == 0) return batch_measure_t<double, double, 0>(bc, st, occ);
        if (occ) {
            int o1 = 0, o2 = 0;
            int rc = batch_measure_t<ff, float, 1>(bc, st, &o1);
            if (!rc) rc = batch_measure_t<ff, float, 2>(bc, st, &o2);
            *occ = o1 < o2 ? o1 : o2;
            return rc;
        }
        int rc = batch_measure_t<ff, float, 1>(bc, st, nullptr);
        return rc ? rc : batch_measure_t<ff, float, 2>(bc, st, nullptr);
    }

    static int init(const HostSys& hs, DevWalkers& dw, uint64_t seed, cudaStream_t st) {
        const SysH<double>* S;
        int rc = table<double>(hs, &S);
        if (rc) return rc;
        int n = NE * dw.W, tpb = 256;
        if (dw.prec == 0) khw_init<double><<<(n + tpb - 1) / tpb, tpb, 0, st>>>(S, (double*)dw.pos, NE, dw.W, dw.Wcap, seed);
        else khw_init<float><<<(n + tpb - 1) / tpb, tpb, 0, st>>>(S, (float*)dw.pos, NE, dw.W, dw.Wcap, seed);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    template <class TC, class TS, int PART>
    static int launch_measure_part(int kmax, const SysH<TC>* S, const KTable* KT, DevWalkers& dw, bool ws,
                                   const MeasureOut& out, double* partial, int nb, cudaStream_t st) {
        const size_t smem = measure_smem<TC, TS, PART>(kmax);
        auto kern = khw_measure<NE, NUP, TC, TS, WPB, PART>;
        // the largest cutoff's, whatever this one: a limit that depends on the call could be
        // lowered again by another thread's
        static bool attr = false;
        if (!attr) {
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)measure_smem<TC, TS, PART>(HMAX_KMAX));
            attr = true;
        }
        kern<<<nb, 32 * WPB, smem, st>>>(S, KT, (const TS*)dw.pos, (TS*)dw.dinv, dw.logabs, dw.sign, dw.el, dw.W,
                                         dw.Wcap, ws ? 1 : 0, out.grad, out.lap, partial, dw.flags, dw.rows);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    template <class TC, class TS>
    static int measure2(const HostSys& hs, DevWalkers& dw, bool ws, const MeasureOut& out, cudaStream_t st) {
        const SysH<TC>* S;
        const KTable* KT;
        int rc = table<TC>(hs, &S, &KT);
        if (rc) return rc;
        int nb = (dw.W + WPB - 1) / WPB;
        double* partial = (ws && dw.partial && dw.partial_cap >= 2 * nb + 1) ? dw.partial : nullptr;
        bool two = false;
        if constexpr (std::is_same<TC, ff>::value) two = ws && dw.rows && !out.grad && !out.lap;
        if (two) {
            if constexpr (std::is_same<TC, ff>::value) {
                rc = launch_measure_part<TC, TS, 1>(reciprocal_kmax(hs), S, KT, dw, ws, out, nullptr, nb, st);
                if (!rc) rc = launch_measure_part<TC, TS, 2>(reciprocal_kmax(hs), S, KT, dw, ws, out, partial, nb, st);
            }
        } else {
            rc = launch_measure_part<TC, TS, 0>(reciprocal_kmax(hs), S, KT, dw, ws, out, partial, nb, st);
        }
        if (rc) return rc;
        if (!partial) return 0;
        return launch_sum_partials(partial, nb, 1, dw.partial + dw.partial_cap - 1, st);
    }

    static int measure(const HostSys& hs, DevWalkers& dw, int cp, bool ws, const MeasureOut& out, cudaStream_t st) {
        if (out.O || out.fhf || out.omega) return 7;
        // FP32 walkers refresh in float-float arithmetic on the FP32 pipe
        if (cp == 0) return dw.prec == 0 ? measure2<double, double>(hs, dw, ws, out, st)
                                         : measure2<ff, float>(hs, dw, ws, out, st);
        if (dw.prec == 1) return measure2<float, float>(hs, dw, ws, out, st);
        return 7;
    }

    template <class T, int MOVE>
    static int sweep_t(const HostSys& hs, DevWalkers& dw, int n, uint64_t s0, double step, double tau, double maxd,
                       uint64_t seed, cudaStream_t st) {
        const SysH<T>* S;
        int rc = table<T>(hs, &S);
        if (rc) return rc;
        int nb = (dw.W + WPB - 1) / WPB;
        auto kern = khw_sweep<NE, NUP, T, MOVE, WPB>;
        const size_t smem = WPB * hsweep_bytes<NM, T, MOVE>();
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
                return 2;
            cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
            attr = true;
        }
        kern<<<nb, 32 * WPB, smem, st>>>(S, (T*)dw.pos, (T*)dw.dinv, dw.W, dw.Wcap, n, s0, (T)step, (T)tau, (T)maxd,
                                         seed, dw.acc, dw.flags);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    static int sweep(const HostSys& hs, DevWalkers& dw, int mk, int n, uint64_t s0, double step, double tau,
                     double maxd, uint64_t seed, cudaStream_t st) {
        if (dw.fixed_node) return 7;     // complex determinants have no nodal surface to fix
        if (mk == MOVE_ONE_GAUSS)
            return dw.prec == 0 ? sweep_t<double, MOVE_ONE_GAUSS>(hs, dw, n, s0, step, tau, maxd, seed, st)
                                : sweep_t<float, MOVE_ONE_GAUSS>(hs, dw, n, s0, step, tau, maxd, seed, st);
        if (mk == MOVE_ONE_DRIFT)
            return dw.prec == 0 ? sweep_t<double, MOVE_ONE_DRIFT>(hs, dw, n, s0, step, tau, maxd, seed, st)
                                : sweep_t<float, MOVE_ONE_DRIFT>(hs, dw, n, s0, step, tau, maxd, seed, st);
        return 7;
    }
};

}  // namespace qmc
