// qmc_warp_kernels.cuh -- warp-per-walker kernels for systems with large spin
// sectors (benzene: 21x21 determinants, 42 electrons, 36 Gaussian AOs).
//
// One warp owns one walker.  Lane j holds column j of each inverse Slater
// matrix in registers (Dinv[k][j], k = 0..n-1) and the positions of
// electrons j and j+32.  The kernels:
//   kw_gauss    FP32 Gaussian sweeps (packed FP32 instructions)
//   kw_sweep    drift-diffusion sweeps, and FP64 Gaussian sweeps
//   kw_refresh  float-float refresh of FP32 walkers (packed, both sectors)
//   kw_eval     FP64 evaluation and refresh
//   kw_measure  FP32 refresh of FP32 walkers
// and kwb_* their batched forms.  Tables lie in shared memory; what all lanes need of
// one lane or of one proposal (inverse column, orbital values) is broadcast from
// there or by shuffles, so every register index stays static.  Inverses come from a
// warp-cooperative Gauss-Jordan elimination in which lane j ends holding column j of
// D^-1 -- exactly the sweep kernels' layout.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <vector>
#include "qmc_internal.h"
#include "qmc_device.cuh"

namespace qmc {

constexpr int WMAX_AO = 96;       // up to three rounds of 32 AOs (BenzeneGTO's 6-31G basis has 66)
constexpr int WAO_ROUNDS = WMAX_AO / 32;
constexpr int WNCOL = 24;         // Slater columns held per sector (lanes >= WNCOL read no coefficients)
constexpr int AO_REP = 16;        // ao_type flag: radial part equal to the previous AO's
constexpr int WMAX_PRIM = 256;
constexpr int WMAX_NUC = 16;

// Radial-group descriptor: nucleus (bits 0-3), kind (bit 4: 0 s, 1 p triplet),
// primitive count (bits 5-8), first primitive (bits 9-16), first AO (bits 17-23).
__host__ __device__ constexpr int grp_pack(int nuc, int kind, int np, int p0, int a0) {
    return nuc | (kind << 4) | (np << 5) | (p0 << 9) | (a0 << 17);
}
__host__ __device__ constexpr int grp_a0(int g) { return (g >> 17) & 127; }
static_assert(WMAX_NUC <= 16 && WMAX_PRIM <= 256 && WMAX_AO <= 128, "group descriptor fields");

// Shared-memory system table of the warp kernels (one copy per block).
template <class T>
struct SysW {
    int n_ao;
    int quirk_lap;
    T F, invF, qa, v_nn;
    T b_ee[2], a_ee[2];
    T nuc[WMAX_NUC][3];
    T Z[WMAX_NUC], enA[WMAX_NUC], enB[WMAX_NUC];
    // ao_type: bits 0-3 the kind (0 s, 1..3 p_x..p_z); AO_REP set when the AO has the
    // centre and primitives of the previous AO (p_y and p_z after p_x share its radial part)
    int ao_nuc[WMAX_AO], ao_type[WMAX_AO], ao_p0[WMAX_AO], ao_np[WMAX_AO];
    // radial groups in AO order: an s AO alone, or a p triplet sharing one
    // radial part; packed by grp_pack (nucleus, kind, primitives, first AO)
    int n_grp;
    int grp[WMAX_AO];
    alignas(16) T prim[WMAX_PRIM][2];   // (exponent, coefficient) of every primitive
    alignas(16) T C[2][WMAX_AO][WNCOL];     // [sector][AO][column]; 16-byte rows of 4 columns read as vectors
    T init_sigma;
    int init_nuc[64];           // internal electron order
    int perm[64];
};

template <class T>
static bool fill_sysw(const HostSys& hs, int NE, int NUP, int NNUC, SysW<T>& S) {
    std::memset(&S, 0, sizeof(S));
    if (hs.N != NE || hs.n_up != NUP || hs.n_nuc != NNUC || hs.n_ao > WMAX_AO || NNUC > WMAX_NUC) return false;
    if (NUP > WNCOL || NE - NUP > WNCOL) return false;
    if (hs.basis != BASIS_GTO) return false;
    S.n_ao = hs.n_ao;
    S.quirk_lap = (hs.quirks & 2) ? 1 : 0;
    S.F = (T)hs.F;
    S.invF = (T)(1.0 / hs.F);
    S.qa = (hs.quirks & 1) ? (T)hs.F : (T)1;
    S.v_nn = (T)hs.v_nn;
    S.b_ee[0] = (T)hs.jas[0]; S.b_ee[1] = (T)hs.jas[1];
    S.a_ee[0] = (T)hs.jas[2]; S.a_ee[1] = (T)hs.jas[3];
    for (int I = 0; I < NNUC; ++I) {
        for (int c = 0; c < 3; ++c) S.nuc[I][c] = (T)hs.R[3 * I + c];
        S.Z[I] = (T)hs.Z[I];
        int sp = hs.species[I];
        S.enA[I] = (T)(hs.jas[6 + sp] * hs.Z[I]);
        S.enB[I] = (T)hs.jas[4 + sp];
    }
    // AOs in internal (shell) order; each AO keeps its own primitive list
    int np = 0;
    for (const HostShell& sh : hs.shells) {
        auto put = [&](int caller_ao, int type, const std::vector<double>& coef) -> bool {
            int a = hs.ao_int[caller_ao];
            if ((int)(np + sh.exps.size()) > WMAX_PRIM || sh.exps.size() > 15) return false;
            S.ao_nuc[a] = sh.nuc;
            S.ao_type[a] = type;
            S.ao_p0[a] = np;
            S.ao_np[a] = (int)sh.exps.size();
            for (size_t p = 0; p < sh.exps.size(); ++p) { S.prim[np][0] = (T)sh.exps[p]; S.prim[np][1] = (T)coef[p]; ++np; }
            return true;
        };
        for (int k = 0; k < 2; ++k) {
            if (sh.s_ao[k] < 0) continue;
            const int p0 = np;
            if (!put(sh.s_ao[k], 0, sh.s_coef[k])) return false;
            S.grp[S.n_grp++] = grp_pack(sh.nuc, 0, (int)sh.exps.size(), p0, hs.ao_int[sh.s_ao[k]]);
        }
        // the p triplet's members are consecutive in the internal order and share
        // one radial part: p_y and p_z reuse p_x's
        if (sh.p_ao[0] >= 0) {
            const int p0 = np, a0 = hs.ao_int[sh.p_ao[0]];
            for (int m = 0; m < 3; ++m) {
                if (hs.ao_int[sh.p_ao[m]] != a0 + m) return false;
                if (!put(sh.p_ao[m], (1 + m) | (m > 0 ? AO_REP : 0), sh.p_coef)) return false;
            }
            S.grp[S.n_grp++] = grp_pack(sh.nuc, 1, (int)sh.exps.size(), p0, a0);
        }
    }
    std::vector<double> Ce = hs.effective_mo();
    for (int sig = 0; sig < 2; ++sig) {
        int col = 0;
        for (int ei = 0; ei < hs.N; ++ei) {
            int e = hs.perm[ei];
            if ((hs.spins[e] > 0) != (sig == 0)) continue;
            int k = hs.occ[e];
            for (int a = 0; a < hs.n_ao; ++a) S.C[sig][hs.ao_int[a]][col] = (T)Ce[(size_t)k * hs.n_ao + a];
            ++col;
        }
    }
    S.init_sigma = (T)hs.init_sigma;
    for (int ei = 0; ei < hs.N; ++ei) {
        S.perm[ei] = hs.perm[ei];
        S.init_nuc[ei] = hs.init_nuc[hs.perm[ei]];
    }
    return true;
}

// Shells of a table's basis: consecutive radial groups as they stand, but an s group
// and the p triplet after it on the same nucleus with the same exponents (the sp
// shells of Pople's sets) as one, whose exponentials are evaluated once.
// Descriptor: nucleus (bits 0-3), s (bit 4), p triplet (bit 5), primitive count (bits
// 6-9), first primitive (bits 10-17), first AO (bits 18-24).
constexpr int SHELL_S = 16, SHELL_P = 32;
__host__ __device__ constexpr int shell_pack(int nuc, int kind, int np, int p0, int a0) {
    return nuc | kind | (np << 6) | (p0 << 10) | (a0 << 18);
}
__host__ __device__ constexpr int shell_nuc(int d) { return d & 15; }
__host__ __device__ constexpr int shell_np(int d) { return (d >> 6) & 15; }
__host__ __device__ constexpr int shell_p0(int d) { return (d >> 10) & 255; }
__host__ __device__ constexpr int shell_a0(int d) { return d >> 18; }

template <class T>
struct ShellList {
    std::vector<int> desc;                     // in AO order
    std::vector<T> al, c, cp;                  // exponent; the s or lone p coefficient; an sp shell's p coefficient
    explicit ShellList(const SysW<T>& S) {
        for (int g = 0; g < S.n_grp; ++g) {
            const int d = S.grp[g], I = d & 15, np = (d >> 5) & 15, q0 = (d >> 9) & 255, a0 = grp_a0(d);
            const bool p = (d >> 4) & 1;
            int q1 = -1;
            if (!p && g + 1 < S.n_grp) {
                const int n = S.grp[g + 1];
                bool same = (n & 15) == I && ((n >> 4) & 1) && ((n >> 5) & 15) == np && grp_a0(n) == a0 + 1;
                for (int i = 0; same && i < np; ++i)
                    same = (double)S.prim[q0 + i][0] == (double)S.prim[((n >> 9) & 255) + i][0];
                if (same) { q1 = (n >> 9) & 255; ++g; }
            }
            desc.push_back(shell_pack(I, p ? SHELL_P : (q1 >= 0 ? SHELL_S | SHELL_P : SHELL_S), np, (int)al.size(), a0));
            for (int i = 0; i < np; ++i) {
                al.push_back(S.prim[q0 + i][0]);
                c.push_back(S.prim[q0 + i][1]);
                cp.push_back(S.prim[(q1 >= 0 ? q1 : q0) + i][1]);
            }
        }
    }
};

// Shells dealt into three lists of equal kinds, by primitive count: out[3 i + t] is
// third t's shell i, rows filled up with shells without primitives; returns the rows.
constexpr int WMAX_THIRD = WMAX_AO + 12;
static int deal_thirds(const std::vector<int>& shells, int (&out)[WMAX_THIRD]) {
    std::vector<int> by[3];
    for (int d : shells) by[(d & SHELL_S) ? ((d & SHELL_P) ? 2 : 0) : 1].push_back(d);
    int n = 0;
    for (auto& v : by) {
        std::stable_sort(v.begin(), v.end(), [](int a, int b) { return shell_np(a) < shell_np(b); });
        for (size_t i = 0; i < (v.size() + 2) / 3 * 3; ++i)
            out[n++] = i < v.size() ? v[i] : shell_pack(0, v[0] & (SHELL_S | SHELL_P), 0, 0, 0);
    }
    return n / 3;
}

// Copy the table from global to shared memory (whole block).
template <class T>
__device__ __forceinline__ void load_sysw(SysW<T>* dst, const SysW<T>* __restrict__ src) {
    static_assert(sizeof(SysW<T>) % 4 == 0, "table size must be a multiple of 4 bytes");
    const int4* s = reinterpret_cast<const int4*>(src);
    int4* d = reinterpret_cast<int4*>(dst);
    constexpr int n16 = (int)(sizeof(SysW<T>) / sizeof(int4));
    for (int i = threadIdx.x; i < n16; i += blockDim.x) d[i] = s[i];
    // tail words when the size is not a multiple of 16 bytes
    for (int i = n16 * 4 + threadIdx.x; i < (int)(sizeof(SysW<T>) / 4); i += blockDim.x)
        reinterpret_cast<int*>(dst)[i] = reinterpret_cast<const int*>(src)[i];
    __syncthreads();
}

// Used part of a table (a whole number of 16-byte words) into the block's shared
// memory; ends with a block barrier.
template <class TAB>
__device__ __forceinline__ void load_tab(TAB* dst, const TAB* __restrict__ src) {
    const int n = (int)(TAB::used(src) / sizeof(float4));
    const float4* s = reinterpret_cast<const float4*>(src);
    float4* d = reinterpret_cast<float4*>(dst);
    for (int i = threadIdx.x; i < n; i += blockDim.x) d[i] = s[i];
    __syncthreads();
}

// (exponent, coefficient) pair of a primitive: one 8- or 16-byte shared load.
template <class T>
__device__ __forceinline__ void load2(const T (&p)[2], T& a, T& b) { a = p[0]; b = p[1]; }
__device__ __forceinline__ void load2(const float (&p)[2], float& a, float& b) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    a = v.x; b = v.y;
}
__device__ __forceinline__ void load2(const double (&p)[2], double& a, double& b) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    a = v.x; b = v.y;
}

// ---------------------------------------------------------------------------
// Lane-parallel AO evaluation: lane l evaluates AO l + 32 r in round r at
// point (x,y,z): value, gradient, Laplacian (MODE >= 1 / 2).  Rounds past the
// basis are skipped (a warp-uniform branch).
// ---------------------------------------------------------------------------
template <class T, int MODE>
struct AOLane {
    T v[WAO_ROUNDS], gx[WAO_ROUNDS], gy[WAO_ROUNDS], gz[WAO_ROUNDS], l[WAO_ROUNDS];
};

template <class T, int MODE>
__device__ __forceinline__ void ao_lane(const SysW<T>& S, T x, T y, T z, int lane, AOLane<T, MODE>& o) {
#pragma unroll
    for (int r = 0; r < WAO_ROUNDS; ++r) {
        const int a = lane + 32 * r;
        T v = 0, gxx = 0, gyy = 0, gzz = 0, lp = 0;
        if (32 * r < S.n_ao && a < S.n_ao) {
            const int I = S.ao_nuc[a], type = S.ao_type[a] & 15, p0 = S.ao_p0[a], np = S.ao_np[a];
            T dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
            T r2 = dx * dx + dy * dy + dz * dz;
            T s0 = 0, s1 = 0, s2 = 0;
            for (int p = p0; p < p0 + np; ++p) {
                T al, cp;
                load2(S.prim[p], al, cp);
                T e = cp * fexp(-al * r2);
                s0 += e;
                if (MODE >= 1) s1 += al * e;
                if (MODE >= 2) s2 += al * al * e;
            }
            // s: chi = R; grad = -2 R1 dr; lap = -6 R1 + 4 r^2 R2
            // p_m: chi = x_m R; grad = x_m(-2 R1 dr) + e_m R; lap = x_m(-10 R1 + 4 r^2 R2)
            T ang = type == 0 ? T(1) : (type == 1 ? dx : (type == 2 ? dy : dz));
            v = ang * s0;
            if (MODE >= 1) {
                T g = -2 * s1 * ang;
                gxx = g * dx + (type == 1 ? s0 : T(0));
                gyy = g * dy + (type == 2 ? s0 : T(0));
                gzz = g * dz + (type == 3 ? s0 : T(0));
            }
            if (MODE >= 2) lp = ang * ((type == 0 ? T(-6) : T(-10)) * s1 + 4 * r2 * s2);
        }
        o.v[r] = v;
        if (MODE >= 1) { o.gx[r] = gxx; o.gy[r] = gyy; o.gz[r] = gzz; }
        if (MODE >= 2) o.l[r] = lp;
    }
}

__device__ __forceinline__ float wshfl(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ double wshfl(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ int wshfl(int v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float wshfl_xor(float v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ double wshfl_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ ff wshfl_xor(ff v, int m) { return shfl_xor(v, m); }
template <class T>
__device__ __forceinline__ T wsum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += wshfl_xor(v, o);
    return v;
}

// v[i] = wsum(v[i]) for N <= 8 values at once.  The two halves of a warp hold the same
// partial sums after a butterfly step, so each step that is left over folds two values
// into one: 9 shuffles and additions and 8 broadcasts for 8 values instead of 40 of
// each.  The same additions, hence the same bits.
template <int N, class T>
__device__ __forceinline__ void wsum_n(T (&v)[N], int lane) {
    static_assert(N <= 8, "three folds");
    T a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (2 * i >= N) break;
        const T x = v[2 * i], y = 2 * i + 1 < N ? v[2 * i + 1 < N ? 2 * i + 1 : 0] : T(0);
        a[i] = (lane & 16 ? y : x) + wshfl_xor(lane & 16 ? x : y, 16);
    }
    constexpr int NA = (N + 1) / 2, NB = (NA + 1) / 2;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const T x = a[2 * i], y = 2 * i + 1 < NA ? a[2 * i + 1 < NA ? 2 * i + 1 : 0] : T(0);
        b[i] = (lane & 8 ? y : x) + wshfl_xor(lane & 8 ? x : y, 8);
    }
    T c;
    if constexpr (NB > 1) c = (lane & 4 ? b[1] : b[0]) + wshfl_xor(lane & 4 ? b[0] : b[1], 4);
    else c = b[0] + wshfl_xor(b[0], 4);
    c += wshfl_xor(c, 2);
    c += wshfl_xor(c, 1);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = wshfl(c, (i & 1) << 4 | (i >> 1 & 1) << 3 | (i >> 2) << 2);
}

// Four consecutive elements of 16-byte-aligned shared memory as one vector
// access (two for double).
__device__ __forceinline__ void load4(const float* p, float& a, float& b, float& c, float& d) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a = v.x; b = v.y; c = v.z; d = v.w;
}
__device__ __forceinline__ void load4(const double* p, double& a, double& b, double& c, double& d) {
    const double2 u = reinterpret_cast<const double2*>(p)[0], v = reinterpret_cast<const double2*>(p)[1];
    a = u.x; b = u.y; c = v.x; d = v.y;
}
__device__ __forceinline__ void store4(float* p, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void store4(double* p, double a, double b, double c, double d) {
    reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
    reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}

// Jastrow cache of the Gaussian sweep: u(r_ij) of every electron pair i < j
// at slot j (j - 1) / 2 + i, then the one-body sum U1_i = sum_I A_I Z_I r/(1 + B_I r)
// of every electron, rounded up to 4 elements.
template <int NE>
__host__ __device__ constexpr int jcache_elems() { return (NE * (NE - 1) / 2 + NE + 3) / 4 * 4; }
__device__ __forceinline__ int pair_slot(int i, int j) {
    const int a = i < j ? i : j, b = i < j ? j : i;
    return b * (b - 1) / 2 + a;
}

// Elements of the per-warp scratch of the single-electron sweep.  Gaussian moves: one
// row of WNCOL orbital values per proposal of a sector, then the Jastrow cache.
// Drift-diffusion moves: a column of the inverse, the proposal's orbital values and
// its AO values, then the sector's draws.
template <int NE, int NUP, int MOVE>
__host__ __device__ constexpr int sweep_scratch_elems() {
    constexpr int NM = NUP > NE - NUP ? NUP : NE - NUP;
    return MOVE == MOVE_ONE_GAUSS ? NM * WNCOL + jcache_elems<NE>() : 2 * WNCOL + WMAX_AO + 4 * NM;
}
// The FP32 Gaussian sweep's (kw_gauss_walker): per sector and proposal a row of
// WNCOL orbital values, then the proposed position and the acceptance draw (a stride
// of 7 16-byte words: row stores of neighbouring lanes fall on different banks); two
// columns of the inverse; the Jastrow cache.
constexpr int GRS = WNCOL + 4;
template <int NE, int NUP>
__host__ __device__ constexpr int gauss_scratch_elems() {
    return 2 * (NUP > NE - NUP ? NUP : NE - NUP) * GRS + 2 * WNCOL + jcache_elems<NE>();
}

// MO contraction: lane k < WNCOL receives phi_k = sum_a C[sig][a][k] chi_a, chi in
// shared memory (16-byte aligned); lanes past the table's columns repeat column 0.
template <class T>
__device__ __forceinline__ T mo_lane(const SysW<T>& S, int sig, int lane, const T* chi) {
    T v = 0;
    const T* c = S.C[sig][0] + (lane < WNCOL ? lane : 0);
    const int n4 = S.n_ao / 4 * 4;
#pragma unroll 3
    for (int t = 0; t < n4; t += 4) {
        T x0, x1, x2, x3;
        load4(chi + t, x0, x1, x2, x3);
        v += c[t * WNCOL] * x0;
        v += c[(t + 1) * WNCOL] * x1;
        v += c[(t + 2) * WNCOL] * x2;
        v += c[(t + 3) * WNCOL] * x3;
    }
    for (int t = n4; t < S.n_ao; ++t) v += c[t * WNCOL] * chi[t];
    return v;
}

// c'_a = sum_k C[sig][a][k] Dinv[k][q] for the lane's AOs a = lane + 32 r, column q of
// the inverse in shared memory (col), the lane's coefficient rows read as 16-byte
// vectors.  Lanes past the basis get 0.
template <class T, int NM>
__device__ __forceinline__ void inverse_column_coefficients(const SysW<T>& S, int sig, int lane, const T* col,
                                                            T (&cw)[WAO_ROUNDS]) {
#pragma unroll
    for (int r = 0; r < WAO_ROUNDS; ++r) cw[r] = 0;
#pragma unroll
    for (int k0 = 0; k0 < NM; k0 += 4) {
        T dq[4];
        load4(col + k0, dq[0], dq[1], dq[2], dq[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) dq[i] = k0 + i < NM ? dq[i] : T(0);
#pragma unroll
        for (int r = 0; r < WAO_ROUNDS; ++r) {
            if (32 * r >= S.n_ao) break;
            const int a = lane + 32 * r;
            T c0, c1, c2, c3;
            load4(&S.C[sig][a < S.n_ao ? a : 0][k0], c0, c1, c2, c3);
            T t = c0 * dq[0] + c1 * dq[1] + c2 * dq[2] + c3 * dq[3];
            cw[r] += a < S.n_ao ? t : T(0);
        }
    }
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
template <class TS>
__global__ void kw_init(const SysW<double>* __restrict__ Sg, TS* __restrict__ pos, int NE, int W, int Wcap,
                        uint64_t seed) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NE * W) return;
    int e = i / W, w = i - e * W;
    const SysW<double>& S = *Sg;
    U4 x = rng_draw(seed, (uint32_t)w, 0, (uint32_t)S.perm[e], TAG_INIT);
    double n0, n1, n2, n3;
    bm(x.x, x.y, n0, n1);
    bm(x.z, x.w, n2, n3);
    int c = S.init_nuc[e];
    double cx = c >= 0 ? S.nuc[c][0] : 0.0, cy = c >= 0 ? S.nuc[c][1] : 0.0, cz = c >= 0 ? S.nuc[c][2] : 0.0;
    pos[(3 * e + 0) * (size_t)Wcap + w] = (TS)(cx + S.init_sigma * n0);
    pos[(3 * e + 1) * (size_t)Wcap + w] = (TS)(cy + S.init_sigma * n1);
    pos[(3 * e + 2) * (size_t)Wcap + w] = (TS)(cz + S.init_sigma * n2);
}

// Positions of electrons `lane` and `lane + 32` live in this lane.
template <class T, int NE>
struct LanePos {
    T x[2], y[2], z[2];
    __device__ __forceinline__ void get(int e, T& ex, T& ey, T& ez) const {
        T a = e < 32 ? x[0] : x[1], b = e < 32 ? y[0] : y[1], c = e < 32 ? z[0] : z[1];
        ex = wshfl(a, e & 31); ey = wshfl(b, e & 31); ez = wshfl(c, e & 31);
    }
    // Same, for an index that differs between lanes: the source lane cannot know which
    // half the reading lane wants, so both halves travel and the reader selects.
    __device__ __forceinline__ void get_own(int e, T& ex, T& ey, T& ez) const {
        const int s = e & 31;
        T x0 = wshfl(x[0], s), x1 = wshfl(x[1], s), y0 = wshfl(y[0], s), y1 = wshfl(y[1], s);
        T z0 = wshfl(z[0], s), z1 = wshfl(z[1], s);
        ex = e < 32 ? x0 : x1; ey = e < 32 ? y0 : y1; ez = e < 32 ? z0 : z1;
    }
};

// This lane's share of the Jastrow terms of electron e at (x, y, z): u =
// sum_j u_ee(r_ej) - sum_I u_en(r_eI) and its gradient with respect to the
// electron, over partner electron `lane` (first round) and partner electron
// 32 + lane (lanes < NE1) or nucleus lane - NE1 (the next NNUC lanes; second
// round).  Every lane evaluates and the unused terms are masked by selects.
template <int NE, int NUP, int NNUC, class T>
__device__ __forceinline__ void wjastrow_lane_terms(const SysW<T>& S, const LanePos<T, NE>& P, int lane, int e,
                                                    T x, T y, T z, T& u, T (&g)[3]) {
    constexpr int NE1 = NE > 32 ? NE - 32 : 0;
    static_assert(NE <= 64 && NE1 + NNUC <= 32, "second round: electrons 32.. and the nuclei share the lanes");
    const bool e_up = e < NUP;
    {
        const int j = lane < NE ? lane : NE - 1;
        const bool ok = lane < NE && lane != e;
        const int c = ((j < NUP) == e_up) ? 1 : 0;
        const T dx = x - P.x[0], dy = y - P.y[0], dz = z - P.z[0];
        T d, ri, uu, upr, lt;
        dist(dx * dx + dy * dy + dz * dz, d, ri);
        pade_ab(S.a_ee[c], S.b_ee[c], d, ri, uu, upr, lt);
        u = ok ? uu : T(0);
        const T f = ok ? upr : T(0);
        g[0] = f * dx; g[1] = f * dy; g[2] = f * dz;
    }
    {
        const bool is_el = lane < NE1, is_nuc = !is_el && lane - NE1 < NNUC;
        const int j = is_el ? 32 + lane : 0, I = is_nuc ? lane - NE1 : 0;
        const bool el_ok = is_el && j != e;
        const T ox = is_el ? P.x[1] : S.nuc[I][0], oy = is_el ? P.y[1] : S.nuc[I][1];
        const T oz = is_el ? P.z[1] : S.nuc[I][2];
        const int c = ((j < NUP) == e_up) ? 1 : 0;
        const T pa = is_el ? S.a_ee[c] : S.enA[I], pb = is_el ? S.b_ee[c] : S.enB[I];
        const T dx = x - ox, dy = y - oy, dz = z - oz;
        T d, ri, uu, upr, lt;
        dist(dx * dx + dy * dy + dz * dz, d, ri);
        pade_ab(pa, pb, d, ri, uu, upr, lt);
        u += el_ok ? uu : (is_nuc ? -uu : T(0));
        const T f = el_ok ? upr : (is_nuc ? -upr : T(0));
        g[0] += f * dx; g[1] += f * dy; g[2] += f * dz;
    }
}

// Row stride of the per-warp proposal-orbital scratch (a multiple of 4
// elements, so that rows start 16-byte aligned and read as vectors).
constexpr int PHS = WNCOL;

// acc[k] += c[k] chi for k < NM: coefficient rows are read as 16-byte vectors
// (NM / 4 of them) and NM % 4 scalars, so no padding column is multiplied.
template <class T, int NM>
__device__ __forceinline__ void row_axpy(const T* c, T chi, T (&acc)[NM]) {
#pragma unroll
    for (int v = 0; v < NM / 4; ++v) {
        T c0, c1, c2, c3;
        load4(c + 4 * v, c0, c1, c2, c3);
        acc[4 * v + 0] += c0 * chi; acc[4 * v + 1] += c1 * chi;
        acc[4 * v + 2] += c2 * chi; acc[4 * v + 3] += c3 * chi;
    }
#pragma unroll
    for (int k = 4 * (NM / 4); k < NM; ++k) acc[k] += c[k] * chi;
}

// Orbital values phi_k(x, y, z), k < NM, of sector sig by one lane: one pass
// over the radial groups (an s AO, or a p triplet sharing its radial part),
// each contracted into the table's columns (broadcast reads: every lane reads
// the same coefficients); written to out[k].
template <class T, int NM>
__device__ __forceinline__ void proposal_orbitals(const SysW<T>& S, int sig, T x, T y, T z, T* out) {
    T acc[NM];
#pragma unroll
    for (int k = 0; k < NM; ++k) acc[k] = 0;
    for (int g = 0; g < S.n_grp; ++g) {
        const int d = S.grp[g];
        const int I = d & 15, kind = (d >> 4) & 1, np = (d >> 5) & 15, p0 = (d >> 9) & 255, a0 = grp_a0(d);
        const T dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
        const T r2 = dx * dx + dy * dy + dz * dz;
        T s0 = 0;
        for (int p = p0; p < p0 + np; ++p) {
            T al, cp;
            load2(S.prim[p], al, cp);
            s0 += cp * fexp(-al * r2);
        }
        const T* c = S.C[sig][a0];
        if (kind == 0) {
            row_axpy<T, NM>(c, s0, acc);
        } else {
            row_axpy<T, NM>(c, dx * s0, acc);
            row_axpy<T, NM>(c + WNCOL, dy * s0, acc);
            row_axpy<T, NM>(c + 2 * WNCOL, dz * s0, acc);
        }
    }
#pragma unroll
    for (int v = 0; v < NM / 4; ++v) store4(out + 4 * v, acc[4 * v], acc[4 * v + 1], acc[4 * v + 2], acc[4 * v + 3]);
#pragma unroll
    for (int k = 4 * (NM / 4); k < NM; ++k) out[k] = acc[k];
}

// Single-electron sweeps, one warp per walker, WPB walkers per block.  A is
// const SweepArgs<T> or const volatile SweepArgs<T>.  Gaussian moves take a
// sector's proposals together: an electron of the sector keeps its position
// until its own proposal, so all NS proposed positions are known when the
// sector's turn starts; lane i evaluates the orbitals at proposal i into the
// warp's scratch ph (proposal_orbitals), and each proposal then reads its row
// as a broadcast instead of contracting AO values broadcast lane to lane.
// Drift-diffusion proposals depend on the current drift and stay one at a
// time.
template <int NE, int NUP, int NNUC, class T, int MOVE, class A>
__device__ __forceinline__ void kw_sweep_walker(const SysW<T>& S, A& a, int w, T* ph) {
    constexpr int NDN = NE - NUP;
    constexpr int NM = NUP > NDN ? NUP : NDN;
    constexpr int NE1 = NE > 32 ? NE - 32 : 0;   // partner electrons of the second round
    static_assert(NE <= 64 && NE1 + NNUC <= 32, "second round: electrons 32.. and the nuclei share the lanes");
    const int lane = threadIdx.x & 31;
    LanePos<T, NE> P;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = lane + 32 * r;
        const bool ok = j < NE;
        P.x[r] = ok ? a.pos[(3 * j + 0) * (size_t)a.Wcap + w] : T(0);
        P.y[r] = ok ? a.pos[(3 * j + 1) * (size_t)a.Wcap + w] : T(0);
        P.z[r] = ok ? a.pos[(3 * j + 2) * (size_t)a.Wcap + w] : T(0);
    }
    T D0[NM], D1[NM];
#pragma unroll
    for (int k = 0; k < NM; ++k) {
        D0[k] = lane < NUP ? a.dinv[((size_t)(0 * NM * NM + k * NM + lane)) * a.Wcap + w] : T(0);
        D1[k] = lane < NDN ? a.dinv[((size_t)(1 * NM * NM + k * NM + lane)) * a.Wcap + w] : T(0);
    }
    int sgn = a.sign[w];
    unsigned acc = 0;
    int flg = 0;
    // Gaussian moves keep every pair term and every one-body sum in the
    // warp's cache (jc), so a proposal evaluates only the moving electron's
    // new terms; a cached term is the same expression on the same squared
    // distance as a recomputation, hence the same value.
    constexpr int NPAIR = NE * (NE - 1) / 2;
    T* jc = ph + NM * PHS;
    // drift moves: column q of the inverse, the proposal's orbital and AO values, draws
    T *colq = ph, *phs = ph + WNCOL, *aos = ph + 2 * WNCOL, *drw = aos + WMAX_AO;
    if constexpr (MOVE == MOVE_ONE_GAUSS) {
        for (int i = 0; i < NE; ++i) {
            T xi, yi, zi;
            P.get(i, xi, yi, zi);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int j = lane + 32 * r;
                if (j < NE && j > i) {
                    T dx = xi - (r ? P.x[1] : P.x[0]), dy = yi - (r ? P.y[1] : P.y[0]), dz = zi - (r ? P.z[1] : P.z[0]);
                    T d, ri, uu, upr, lt;
                    dist(dx * dx + dy * dy + dz * dz, d, ri);
                    const int c = ((j < NUP) == (i < NUP)) ? 1 : 0;
                    pade_ab(S.a_ee[c], S.b_ee[c], d, ri, uu, upr, lt);
                    jc[pair_slot(i, j)] = uu;
                }
            }
            T en = 0;
            if (lane < NNUC) {
                T dx = xi - S.nuc[lane][0], dy = yi - S.nuc[lane][1], dz = zi - S.nuc[lane][2];
                T d, ri, uu, upr, lt;
                dist(dx * dx + dy * dy + dz * dz, d, ri);
                pade_ab(S.enA[lane], S.enB[lane], d, ri, uu, upr, lt);
                en = uu;
            }
            en = wsum(en);
            if (lane == 0) jc[NPAIR + i] = en;
        }
        __syncwarp();
    }
    for (int it = 0; it < a.n_sweeps; ++it) {
        const uint64_t st = a.step0 + (uint64_t)it;
#pragma unroll
        for (int sig = 0; sig < 2; ++sig) {
            T (&D)[NM] = sig == 0 ? D0 : D1;
            const int NS = sig == 0 ? NUP : NDN;
            static_assert(NUP <= 32 && NE - NUP <= 32, "one lane per sector electron");
            const MoveDraw<T> draws = sector_draws<T>(a.seed, (uint32_t)w, st, sig * NUP, NS, lane);
            T pnx = 0, pny = 0, pnz = 0;              // this lane's proposal (Gaussian moves)
            if constexpr (MOVE == MOVE_ONE_GAUSS) {
                T ex, ey, ez;
                P.get_own(min(sig * NUP + lane, NE - 1), ex, ey, ez);
                const T step = a.step;
                pnx = ex + step * draws.n0; pny = ey + step * draws.n1; pnz = ez + step * draws.n2;
                __syncwarp();                          // the previous sector's rows are read
                if (lane < NS) proposal_orbitals<T, NM>(S, sig, pnx, pny, pnz, ph + lane * PHS);
                __syncwarp();
            }
            if constexpr (MOVE == MOVE_ONE_DRIFT) {
                if (lane < NS) store4(drw + 4 * lane, draws.n0, draws.n1, draws.n2, draws.uacc);
                __syncwarp();
            }
            T csc = 1;                                 // pending scale of this lane's column (Gaussian moves)
            for (int q = 0; q < NS; ++q) {
                const int e = sig * NUP + q;
                T rx, ry, rz;
                P.get(e, rx, ry, rz);
                MoveDraw<T> md;
                if constexpr (MOVE == MOVE_ONE_DRIFT) load4(drw + 4 * q, md.n0, md.n1, md.n2, md.uacc);
                else md = draw_of(draws, q);
                T nx, ny, nz, logG = 0, dlx = 0, dly = 0, dlz = 0;
                // drift: c'_a = sum_k C[sig][a][k] Dinv[k][q] on the lanes of AO a, so that
                // grad ln D at r and at r' are sums over the AOs (warp sums)
                T cw[WAO_ROUNDS];
                T u_old = 0;                           // drift: this lane's Jastrow terms at r
                if constexpr (MOVE == MOVE_ONE_DRIFT) {
                    if (lane == q) {
#pragma unroll
                        for (int k = 0; k < NM; k += 4)
                            store4(colq + k, D[k], D[k + 1 < NM ? k + 1 : k], D[k + 2 < NM ? k + 2 : k], D[k + 3 < NM ? k + 3 : k]);
                    }
                    __syncwarp();
                    inverse_column_coefficients<T, NM>(S, sig, lane, colq, cw);
                    AOLane<T, 1> ao;
                    ao_lane<T, 1>(S, rx, ry, rz, lane, ao);
                    T ax = 0, ay = 0, az = 0;
#pragma unroll
                    for (int r = 0; r < WAO_ROUNDS; ++r) { ax += cw[r] * ao.gx[r]; ay += cw[r] * ao.gy[r]; az += cw[r] * ao.gz[r]; }
                    T gl[3];
                    wjastrow_lane_terms<NE, NUP, NNUC, T>(S, P, lane, e, rx, ry, rz, u_old, gl);
                    T sm[6] = {ax, ay, az, gl[0], gl[1], gl[2]};
                    wsum_n(sm, lane);
                    ax = sm[0]; ay = sm[1]; az = sm[2];
                    T g0[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) g0[c] = sm[3 + c] * S.qa;
                    const T tau = a.tau, maxd = a.maxd;
                    dlx = tau * 2 * (ax + g0[0]); dly = tau * 2 * (ay + g0[1]); dlz = tau * 2 * (az + g0[2]);
                    T m = fsqrt(dlx * dlx + dly * dly + dlz * dlz);
                    if (m > maxd) { T s = maxd / m; dlx *= s; dly *= s; dlz *= s; }
                    T sd2 = fsqrt(2 * tau);
                    nx = rx + dlx + sd2 * md.n0; ny = ry + dly + sd2 * md.n1; nz = rz + dlz + sd2 * md.n2;
                } else {
                    nx = wshfl(pnx, q); ny = wshfl(pny, q); nz = wshfl(pnz, q);
                }
                // t_j = sum_k phi_k Dinv[k][j]; R = t_q
                T tj = 0, bx = 0, by = 0, bz = 0;
                if constexpr (MOVE == MOVE_ONE_DRIFT) {
                    AOLane<T, 1> ao;
                    ao_lane<T, 1>(S, nx, ny, nz, lane, ao);
                    // orbital values at r' (every t_j is needed for the update), the
                    // gradient term of column q from c'
#pragma unroll
                    for (int r = 0; r < WAO_ROUNDS; ++r)
                        if (lane + 32 * r < S.n_ao) aos[lane + 32 * r] = ao.v[r];
                    __syncwarp();
                    const T phi = mo_lane(S, sig, lane, aos);
                    if (lane < NM) phs[lane] = phi;
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < NM; k += 4) {
                        T f0, f1, f2, f3;
                        load4(phs + k, f0, f1, f2, f3);
                        tj += f0 * D[k];
                        if (k + 1 < NM) tj += f1 * D[k + 1 < NM ? k + 1 : 0];
                        if (k + 2 < NM) tj += f2 * D[k + 2 < NM ? k + 2 : 0];
                        if (k + 3 < NM) tj += f3 * D[k + 3 < NM ? k + 3 : 0];
                    }
#pragma unroll
                    for (int r = 0; r < WAO_ROUNDS; ++r) { bx += cw[r] * ao.gx[r]; by += cw[r] * ao.gy[r]; bz += cw[r] * ao.gz[r]; }
                } else {
                    const T* row = ph + q * PHS;
                    T t0 = 0, t1 = 0;
#pragma unroll
                    for (int v = 0; v < (NM + 3) / 4; ++v) {
                        T f0, f1, f2, f3;
                        load4(row + 4 * v, f0, f1, f2, f3);
                        if (4 * v + 0 < NM) t0 += f0 * D[4 * v + 0];
                        if (4 * v + 1 < NM) t1 += f1 * D[4 * v + 1];
                        if (4 * v + 2 < NM) t0 += f2 * D[4 * v + 2];
                        if (4 * v + 3 < NM) t1 += f3 * D[4 * v + 3];
                    }
                    tj = t0 + t1;
                }
                const T R = wshfl(tj, q);
                T gn[3];
                T du, unew[2] = {T(0), T(0)}, enn = 0;
                if constexpr (MOVE == MOVE_ONE_GAUSS) {
                    // new terms of the moving electron against the cached old
                    // ones: partner electron `lane` in the first round; in the
                    // second, partner electron 32 + lane on lanes < NE1 and
                    // nucleus lane - NE1 on the next NNUC lanes
                    // Every lane evaluates its terms and the unused ones are
                    // masked out (no divergent branch; the masked lanes read a
                    // valid cache slot and may compute non-finite values).
                    T ds;
                    {
                        const int j = lane < NE ? lane : NE - 1;
                        T dx = nx - P.x[0], dy = ny - P.y[0], dz = nz - P.z[0];
                        T d, ri, uu, upr, lt;
                        dist(dx * dx + dy * dy + dz * dz, d, ri);
                        const int c = ((j < NUP) == (e < NUP)) ? 1 : 0;
                        pade_ab(S.a_ee[c], S.b_ee[c], d, ri, uu, upr, lt);
                        unew[0] = uu;
                        const T old = jc[pair_slot(e, j)];
                        ds = (lane < NE && lane != e) ? uu - old : T(0);
                    }
                    {
                        const bool is_el = lane < NE1, is_nuc = !is_el && lane - NE1 < NNUC;
                        const int j = is_el ? 32 + lane : 0, I = is_nuc ? lane - NE1 : 0;
                        const T ox = is_el ? P.x[1] : S.nuc[I][0], oy = is_el ? P.y[1] : S.nuc[I][1];
                        const T oz = is_el ? P.z[1] : S.nuc[I][2];
                        const int c = ((j < NUP) == (e < NUP)) ? 1 : 0;
                        const T pa = is_el ? S.a_ee[c] : S.enA[I], pb = is_el ? S.b_ee[c] : S.enB[I];
                        T dx = nx - ox, dy = ny - oy, dz = nz - oz;
                        T d, ri, uu, upr, lt;
                        dist(dx * dx + dy * dy + dz * dz, d, ri);
                        pade_ab(pa, pb, d, ri, uu, upr, lt);
                        unew[1] = uu;
                        const T old = jc[pair_slot(e, j)];
                        ds += (is_el && j != e) ? uu - old : T(0);
                        enn = is_nuc ? uu : T(0);
                        ds -= enn;
                    }
                    du = wsum(ds) + jc[NPAIR + e];
                } else {
                    // new position's terms against the old position's (kept from the drift)
                    T un, gl[3];
                    wjastrow_lane_terms<NE, NUP, NNUC, T>(S, P, lane, e, nx, ny, nz, un, gl);
                    T sm[7] = {bx, by, bz, gl[0], gl[1], gl[2], un - u_old};
                    wsum_n(sm, lane);
                    bx = sm[0]; by = sm[1]; bz = sm[2];
                    du = sm[6];
#pragma unroll
                    for (int c = 0; c < 3; ++c) gn[c] = sm[3 + c] * S.qa;
                }
                if constexpr (MOVE == MOVE_ONE_DRIFT) {
                    const T tau = a.tau, maxd = a.maxd;
                    T iR = R != T(0) ? T(1) / R : T(0);
                    T cx = tau * 2 * (bx * iR + gn[0]), cy = tau * 2 * (by * iR + gn[1]), cz = tau * 2 * (bz * iR + gn[2]);
                    T m = fsqrt(cx * cx + cy * cy + cz * cz);
                    if (m > maxd) { T s = maxd / m; cx *= s; cy *= s; cz *= s; }
                    T fx = nx - rx - dlx, fy = ny - ry - dly, fz = nz - rz - dlz;
                    T qx = rx - nx - cx, qy = ry - ny - cy, qz = rz - nz - cz;
                    logG = ((fx * fx + fy * fy + fz * fz) - (qx * qx + qy * qy + qz * qz)) / (4 * tau);
                }
                T ratio = R * fexp(du);
                T prob = ratio * ratio;
                if (MOVE == MOVE_ONE_DRIFT) prob *= fexp(logG);
                if (prob != prob) flg |= FLAG_NONFINITE;
                if (md.uacc < prob && R != T(0) && !(a.fixed_node && R < T(0))) {
                    // positions: the owner lane of e stores the new coordinates
                    if ((e & 31) == lane) {
                        if (e < 32) { P.x[0] = nx; P.y[0] = ny; P.z[0] = nz; }
                        else { P.x[1] = nx; P.y[1] = ny; P.z[1] = nz; }
                    }
                    const T iR = T(1) / R;
                    if constexpr (MOVE == MOVE_ONE_GAUSS) {
                        // column q keeps its values and takes the factor 1/R,
                        // applied when the sector ends (every column's scale is
                        // 1 until its own electron moves, so t_q and R are read
                        // unscaled); the others take t_j / R times column q
                        const T f = lane == q ? T(0) : tj * iR;
                        if (lane == q) csc = iR;
#pragma unroll
                        for (int k = 0; k < NM; ++k) D[k] -= wshfl(D[k], q) * f;
                    } else {
                        const T f = tj * iR;
#pragma unroll
                        for (int k = 0; k < NM; k += 4) {
                            T dq[4];
                            load4(colq + k, dq[0], dq[1], dq[2], dq[3]);
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (k + i < NM) {
                                    T& d = D[k + i < NM ? k + i : 0];
                                    d = (lane == q) ? dq[i] * iR : d - dq[i] * f;
                                }
                        }
                    }
                    if (R < 0) sgn = -sgn;
                    ++acc;
                    if constexpr (MOVE == MOVE_ONE_GAUSS) {
                        if (lane < NE && lane != e) jc[pair_slot(e, lane)] = unew[0];
                        if (lane < NE1 && 32 + lane != e) jc[pair_slot(e, 32 + lane)] = unew[1];
                        const T u1 = wsum(enn);
                        if (lane == 0) jc[NPAIR + e] = u1;
                    }
                }
                __syncwarp();                      // cache writes before the next proposal's reads
            }
            if constexpr (MOVE == MOVE_ONE_GAUSS) {
#pragma unroll
                for (int k = 0; k < NM; ++k) D[k] *= csc;
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
        if (lane < NUP) a.dinv[((size_t)(0 * NM * NM + k * NM + lane)) * a.Wcap + w] = D0[k];
        if (lane < NDN) a.dinv[((size_t)(1 * NM * NM + k * NM + lane)) * a.Wcap + w] = D1[k];
    }
    if (lane == 0) {
        a.sign[w] = sgn;
        if (acc) atomicAdd(a.acc, (unsigned long long)acc);
        if (flg) atomicOr(a.flags, flg);
    }
}

// An inverse column in registers: rows 2v and 2v + 1 in p[v], the last row of an odd
// sector in t.
template <int NM>
struct ColF2 {
    F2 p[NM / 2 > 0 ? NM / 2 : 1];
    float t;
};

// Table of the FP32 Gaussian sweep, values of both halves of a packed instruction
// doubled: shells as (-x, -x, -y, -y), (-z, -z, descriptor bits, 0) of the nucleus,
// primitives (-exponent, -exponent, c, c) and (p coefficient of an sp shell twice),
// coefficients of both sectors side by side, the columns padded to pairs.
template <int NNUC, int NM>
struct GaussTab {
    static constexpr int NC = (NM + 1) / 2 * 2;
    int n_ao, n_sh;
    float a_ee[2], b_ee[2];
    float pad[2];
    float nuc[NNUC][4];                       // x, y, z, unused
    float en[NNUC][2];                        // A, B
    alignas(16) float4 sh[WMAX_AO][2];
    float4 prim[WMAX_PRIM];
    float2 prim_p[WMAX_PRIM];
    float2 C[WMAX_AO][NC];
    __host__ __device__ static size_t bytes(int n_ao) { return offsetof(GaussTab, C) + sizeof(float2) * NC * (size_t)n_ao; }
    __device__ static size_t used(const GaussTab* t) { return bytes(t->n_ao); }
};

template <int NNUC, int NM>
static void fill_gausstab(const SysW<float>& w, GaussTab<NNUC, NM>& S) {
    std::memset(static_cast<void*>(&S), 0, sizeof(S));
    const ShellList<float> L(w);
    S.n_ao = w.n_ao;
    S.n_sh = (int)L.desc.size();
    for (int c = 0; c < 2; ++c) { S.a_ee[c] = w.a_ee[c]; S.b_ee[c] = w.b_ee[c]; }
    for (int I = 0; I < NNUC; ++I) {
        for (int c = 0; c < 3; ++c) S.nuc[I][c] = w.nuc[I][c];
        S.en[I][0] = w.enA[I];
        S.en[I][1] = w.enB[I];
    }
    for (int g = 0; g < S.n_sh; ++g) {
        const int I = shell_nuc(L.desc[g]);
        float bits;
        std::memcpy(&bits, &L.desc[g], sizeof bits);
        S.sh[g][0] = make_float4(-w.nuc[I][0], -w.nuc[I][0], -w.nuc[I][1], -w.nuc[I][1]);
        S.sh[g][1] = make_float4(-w.nuc[I][2], -w.nuc[I][2], bits, 0.0f);
    }
    for (size_t p = 0; p < L.al.size(); ++p) {
        S.prim[p] = make_float4(-L.al[p], -L.al[p], L.c[p], L.c[p]);
        S.prim_p[p] = make_float2(L.cp[p], L.cp[p]);
    }
    for (int a = 0; a < w.n_ao; ++a)
        for (int k = 0; k < NM; ++k) S.C[a][k] = make_float2(w.C[0][a][k], w.C[1][a][k]);
}

// Orbital values of one proposal of each sector (x, y, z: the up sector's coordinate,
// the down sector's) in packed instructions: proposal_orbitals' operations in the same
// order on each, an sp shell's exponentials once.  Written to out0[k] and out1[k].
template <int NNUC, int NM>
__device__ __forceinline__ void proposal_orbitals2(const GaussTab<NNUC, NM>& S, F2 x, F2 y, F2 z, float* out0, float* out1) {
    F2 acc[NM];
#pragma unroll
    for (int k = 0; k < NM; ++k) acc[k] = F2(0.0f);
    auto axpy = [&](const float2* c, F2 chi) {
#pragma unroll
        for (int k = 0; k < NM; k += 2) {
            const float4 v = *reinterpret_cast<const float4*>(c + k);
            acc[k] = fma2(F2(v.x, v.y), chi, acc[k]);
            if (k + 1 < NM) acc[k + 1 < NM ? k + 1 : 0] = fma2(F2(v.z, v.w), chi, acc[k + 1 < NM ? k + 1 : 0]);
        }
    };
#pragma unroll 1
    for (int g = 0; g < S.n_sh; ++g) {
        const float4 G = S.sh[g][0], H = S.sh[g][1];
        const int d = __float_as_int(H.z);
        const int np = shell_np(d);
        const float4* prim = S.prim + shell_p0(d);
        const float2* prim_p = S.prim_p + shell_p0(d);
        const float2* c = S.C[shell_a0(d)];
        const F2 dx = add2(x, F2(G.x, G.y)), dy = add2(y, F2(G.z, G.w)), dz = add2(z, F2(H.x, H.y));
        const F2 r2 = fma2(dz, dz, fma2(dx, dx, mul2(dy, dy)));
        // s0: the s (or lone p) radial part, s1: an sp shell's p part
        F2 s0(0.0f), s1(0.0f);
#pragma unroll 3
        for (int p = 0; p < np; ++p) {
            const float4 t = prim[p];
            const float2 u = prim_p[p];
            float e0, e1;
            mul2(F2(t.x, t.y), r2).get(e0, e1);
            const F2 e(fexp(e0), fexp(e1));
            s0 = fma2(F2(t.z, t.w), e, s0);
            s1 = fma2(F2(u.x, u.y), e, s1);
        }
        if (d & SHELL_S) {
            axpy(c, s0);
            c += S.NC;
        }
        if (d & SHELL_P) {
            axpy(c, mul2(dx, s1));
            axpy(c + S.NC, mul2(dy, s1));
            axpy(c + 2 * S.NC, mul2(dz, s1));
        }
    }
#pragma unroll
    for (int k = 0; k < NM; k += 4) {
        float4 u, v;
        acc[k].get(u.x, v.x);
        acc[k + 1 < NM ? k + 1 : k].get(u.y, v.y);
        acc[k + 2 < NM ? k + 2 : k].get(u.z, v.z);
        acc[k + 3 < NM ? k + 3 : k].get(u.w, v.w);
        *reinterpret_cast<float4*>(out0 + k) = u;
        *reinterpret_cast<float4*>(out1 + k) = v;
    }
}

// v[0] + ... + v[N - 1] in the order of wsum with v[i] on lane L0 + i (N <= 32 - L0) and
// zeros elsewhere, which are left out.
template <int L0, int N>
__device__ __forceinline__ float wsum_order(const float* v) {
    float s[32];
    bool on[32];
#pragma unroll
    for (int l = 0; l < 32; ++l) {
        on[l] = l >= L0 && l < L0 + N;
        s[l] = on[l] ? v[on[l] ? l - L0 : 0] : 0.0f;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1)
#pragma unroll
        for (int l = 0; l < o; ++l) {
            s[l] = on[l] && on[l + o] ? s[l] + s[l + o] : (on[l] ? s[l] : s[l + o]);
            on[l] = on[l] || on[l + o];
        }
    return s[0];
}

// FP32 Gaussian sweeps.  Issue slots and the latency of the proposal chain bound them:
// at 16 warps per SM (128 registers) 272 warp instructions a proposal, issue 62 % busy,
// shared-memory pipe 68 %, where the shuffle form had 315; 8 sweeps of 16 384 benzene
// walkers take 1.93 ms after 2.39 ms.  kw_sweep_walker's operations in its order on every value;
// here a lane's inverse columns lie in row pairs, so that ratio, update, orbital
// contraction and the two rounds of Jastrow partners take packed FP32 instructions,
// and a proposal's position and draw and the moving electron's column are read from
// shared memory as broadcasts instead of a shuffle per value.
template <int NE, int NUP, int NNUC, class TAB, class A>
__device__ __forceinline__ void kw_gauss_walker(const TAB& S, A& a, int w, float* ph) {
    constexpr int NDN = NE - NUP;
    constexpr int NM = NUP > NDN ? NUP : NDN;
    constexpr int NE1 = NE > 32 ? NE - 32 : 0;   // partner electrons of the second round
    constexpr int NPAIR = NE * (NE - 1) / 2;
    static_assert(NE <= 64 && NE1 + NNUC <= 32, "second round: electrons 32.. and the nuclei share the lanes");
    static_assert(NUP <= 32 && NDN <= 32, "one lane per sector electron");
    static_assert(NNUC <= WNCOL, "a row takes the nuclei's terms");
    const int lane = threadIdx.x & 31;
    float* cols = ph + 2 * NM * GRS;              // column q of the inverse, at (q mod 2) WNCOL
    float* jc = cols + 2 * WNCOL;
    const bool is_el = lane < NE1, is_nuc = !is_el && lane - NE1 < NNUC;
    // partner positions: electron `lane`; electron 32 + lane or nucleus lane - NE1
    // (the lanes past both repeat a partner and are masked)
    const int j0 = lane < NE ? lane : NE - 1, j1 = is_el ? 32 + lane : 0, I1 = is_nuc ? lane - NE1 : 0;
    auto load = [&](int j, int c) -> float { return a.pos[(3 * j + c) * (size_t)a.Wcap + w]; };
    // p1 = (x, y'), p2 = (y, x'), pz = (z, z'), the second partner primed: its squared
    // distance sums in the order y, x, z and the first one's in the order x, y, z
    F2 p1(lane < NE ? load(j0, 0) : 0.0f, is_el ? load(j1, 1) : S.nuc[I1][1]),
       p2(lane < NE ? load(j0, 1) : 0.0f, is_el ? load(j1, 0) : S.nuc[I1][0]),
       pz(lane < NE ? load(j0, 2) : 0.0f, is_el ? load(j1, 2) : S.nuc[I1][2]);
    ColF2<NM> D0, D1;
    {
        auto row = [&](int sig, int k) -> float {
            return lane < (sig == 0 ? NUP : NDN) ? a.dinv[((size_t)(sig * NM * NM + k * NM + lane)) * a.Wcap + w] : 0.0f;
        };
#pragma unroll
        for (int v = 0; v < NM / 2; ++v) {
            D0.p[v] = F2(row(0, 2 * v), row(0, 2 * v + 1));
            D1.p[v] = F2(row(1, 2 * v), row(1, 2 * v + 1));
        }
        if constexpr (NM % 2) { D0.t = row(0, NM - 1); D1.t = row(1, NM - 1); }
    }
    int sgn = a.sign[w];
    unsigned acc = 0;
    int flg = 0;
    const bool fixed = a.fixed_node;
    // position of electron e (any lane's own choice) from the lane that holds it
    auto get = [&](int e, float& x, float& y, float& z) {
        float a0, a1, b0, b1, c0, c1;
        p1.get(a0, b1);
        p2.get(b0, a1);
        pz.get(c0, c1);
        const int s = e & 31;
        a0 = wshfl(a0, s); a1 = wshfl(a1, s); b0 = wshfl(b0, s); b1 = wshfl(b1, s); c0 = wshfl(c0, s); c1 = wshfl(c1, s);
        x = e < 32 ? a0 : a1; y = e < 32 ? b0 : b1; z = e < 32 ? c0 : c1;
    };
    // the Jastrow cache (see kw_sweep_walker)
    for (int i = 0; i < NE; ++i) {
        float xi, yi, zi;
        get(i, xi, yi, zi);
        auto value = [&](float x, float y, float z, float A, float B) -> float {
            const float dx = xi - x, dy = yi - y, dz = zi - z;
            float d, ri, uu, upr, lt;
            dist(dx * dx + dy * dy + dz * dz, d, ri);
            pade_ab(A, B, d, ri, uu, upr, lt);
            return uu;
        };
        float x[2], y[2], z[2];
        p1.get(x[0], y[1]);
        p2.get(y[0], x[1]);
        pz.get(z[0], z[1]);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int j = lane + 32 * r, c = ((j < NUP) == (i < NUP)) ? 1 : 0;
            if (j < NE && j > i) jc[pair_slot(i, j)] = value(x[r], y[r], z[r], S.a_ee[c], S.b_ee[c]);
        }
        float en = 0;
        if (lane < NNUC) en = value(S.nuc[lane][0], S.nuc[lane][1], S.nuc[lane][2], S.en[lane][0], S.en[lane][1]);
        en = wsum(en);
        if (lane == 0) jc[NPAIR + i] = en;
    }
    for (int it = 0; it < a.n_sweeps; ++it) {
        const uint64_t st = a.step0 + (uint64_t)it;
        // Proposals of both sectors: an electron keeps its position until its own
        // proposal, so all of them are known when the sweep starts.  Lane i evaluates the
        // orbitals at proposal i of either sector.
        __syncwarp();                                  // the previous sweep's rows are read
        {
            const float step = a.step;
            const MoveDraw<float> du = sector_draws<float>(a.seed, (uint32_t)w, st, 0, NUP, lane),
                                  dd = sector_draws<float>(a.seed, (uint32_t)w, st, NUP, NDN, lane);
            const int eu = min(lane, NE - 1), ed = min(NUP + lane, NE - 1);
            float ux, uy, uz, vx, vy, vz;
            get(eu, ux, uy, uz);
            get(ed, vx, vy, vz);
            ux += step * du.n0; uy += step * du.n1; uz += step * du.n2;
            vx += step * dd.n0; vy += step * dd.n1; vz += step * dd.n2;
            if (lane < NM) {
                float *r0 = ph + lane * GRS, *r1 = r0 + NM * GRS;
                *reinterpret_cast<float4*>(r0 + WNCOL) = make_float4(ux, uy, uz, du.uacc);
                *reinterpret_cast<float4*>(r1 + WNCOL) = make_float4(vx, vy, vz, dd.uacc);
                proposal_orbitals2(S, F2(ux, vx), F2(uy, vy), F2(uz, vz), r0, r1);
            }
        }
#pragma unroll
        for (int sig = 0; sig < 2; ++sig) {
            ColF2<NM>& D = sig == 0 ? D0 : D1;
            const int NS = sig == 0 ? NUP : NDN;
            // Padé parameters of the lane's two partners
            const int c0 = ((j0 < NUP) == (sig == 0)) ? 1 : 0, c1 = ((j1 < NUP) == (sig == 0)) ? 1 : 0;
            const F2 pa(S.a_ee[c0], is_el ? S.a_ee[c1] : S.en[I1][0]), pb(S.b_ee[c0], is_el ? S.b_ee[c1] : S.en[I1][1]);
            float csc = 1;                             // pending scale of this lane's column
            float* row = ph + sig * NM * GRS;
            unsigned moved = 0;                        // accepted proposals of the sector
            // the cache slots of e and the two partners: pair_slot, which grows by 1 while
            // e < j and by e from there on
            float *s0 = jc + pair_slot(sig * NUP, j0), *s1 = jc + pair_slot(sig * NUP, j1);
            for (int q = 0; q < NS; ++q) {
                const int e = sig * NUP + q;
                float* colq = cols + (q & 1) * WNCOL;
                if (lane == q) {
#pragma unroll
                    for (int v = 0; v < NM / 4; ++v) {
                        float4 c;
                        D.p[2 * v].get(c.x, c.y);
                        D.p[2 * v + 1].get(c.z, c.w);
                        reinterpret_cast<float4*>(colq)[v] = c;
                    }
                    if constexpr (NM % 4 >= 2) {
                        float2 c;
                        D.p[NM / 2 - 1].get(c.x, c.y);
                        *reinterpret_cast<float2*>(colq + NM / 4 * 4) = c;
                    }
                    if constexpr (NM % 2) colq[NM - 1] = D.t;
                }
                __syncwarp();                          // column and rows before their reads
                const float4 np = *reinterpret_cast<const float4*>(row + WNCOL);
                // t_j = sum_k phi_k Dinv[k][j], even and odd rows apart; R = t_q
                F2 t2(0.0f);
                float ta, tb;
#pragma unroll
                for (int v = 0; v < NM / 4; ++v) {
                    const float4 f = reinterpret_cast<const float4*>(row)[v];
                    t2 = fma2(F2(f.x, f.y), D.p[2 * v], t2);
                    t2 = fma2(F2(f.z, f.w), D.p[2 * v + 1], t2);
                }
                if constexpr (NM % 4 >= 2) {
                    const float2 f = *reinterpret_cast<const float2*>(row + NM / 4 * 4);
                    t2 = fma2(F2(f.x, f.y), D.p[NM / 2 - 1], t2);
                }
                t2.get(ta, tb);
                if constexpr (NM % 2) ta += row[NM - 1] * D.t;
                const float tj = ta + tb;
                const float R = wshfl(tj, q);
                // the moving electron's new Jastrow terms against the cached old ones
                // (unused terms are masked out; their lanes read a valid cache slot and may
                // compute non-finite values)
                float u0, u1;
                {
                    const F2 neg(-1.0f);
                    const F2 d1 = fma2(p1, neg, F2(np.x, np.y)), d2 = fma2(p2, neg, F2(np.y, np.x)), dz = fma2(pz, neg, F2(np.z));
                    float ra, rb, da, db;
                    fma2(dz, dz, fma2(d1, d1, mul2(d2, d2))).get(ra, rb);
                    float ia, ib;
                    dist(ra, da, ia);
                    dist(rb, db, ib);
                    const F2 d(da, db);
                    float na, nb;
                    fma2(pb, d, F2(1.0f)).get(na, nb);
                    const F2 ad = mul2(pa, d), inv(frcp(na), frcp(nb));
                    mul2(ad, inv).get(u0, u1);
                }
                const bool on0 = lane < NE && lane != e, on1 = is_el && j1 != e;
                const float enn = is_nuc ? u1 : 0.0f;
                float ds = on0 ? u0 - *s0 : 0.0f;
                ds += on1 ? u1 - *s1 : 0.0f;
                ds -= enn;
                const float du = wsum(ds) + jc[NPAIR + e];
                const float ratio = R * fexp(du);
                const float prob = ratio * ratio;
                if (prob != prob) flg |= FLAG_NONFINITE;
                if (np.w < prob && R != 0.0f && !(fixed && R < 0.0f)) {
                    // the lane that holds e takes the new position
                    {
                        float a0, a1, b0, b1, c0, c1;
                        p1.get(a0, b1);
                        p2.get(b0, a1);
                        pz.get(c0, c1);
                        const bool h0 = lane == e, h1 = lane + 32 == e;
                        a0 = h0 ? np.x : a0; b0 = h0 ? np.y : b0; c0 = h0 ? np.z : c0;
                        a1 = h1 ? np.x : a1; b1 = h1 ? np.y : b1; c1 = h1 ? np.z : c1;
                        p1 = F2(a0, b1); p2 = F2(b0, a1); pz = F2(c0, c1);
                    }
                    const float iR = 1.0f / R;
                    // column q keeps its values and takes the factor 1/R when the sector
                    // ends; the others take t_j / R times column q
                    const float f = lane == q ? 0.0f : tj * iR;
                    if (lane == q) csc = iR;
                    const F2 nf(-f);
#pragma unroll
                    for (int v = 0; v < NM / 4; ++v) {
                        const float4 c = reinterpret_cast<const float4*>(colq)[v];
                        D.p[2 * v] = fma2(F2(c.x, c.y), nf, D.p[2 * v]);
                        D.p[2 * v + 1] = fma2(F2(c.z, c.w), nf, D.p[2 * v + 1]);
                    }
                    if constexpr (NM % 4 >= 2) {
                        const float2 c = *reinterpret_cast<const float2*>(colq + NM / 4 * 4);
                        D.p[NM / 2 - 1] = fma2(F2(c.x, c.y), nf, D.p[NM / 2 - 1]);
                    }
                    if constexpr (NM % 2) D.t -= colq[NM - 1] * f;
                    if (R < 0) sgn = -sgn;
                    ++acc;
                    if (on0) *s0 = u0;
                    if (on1) *s1 = u1;
                    // the one-body terms wait in the proposal's row, which has been read
                    if (is_nuc) row[lane - NE1] = enn;
                    moved |= 1u << q;
                }
                s0 += e < j0 ? 1 : e;
                s1 += e < j1 ? 1 : e;
                row += GRS;
            }
            __syncwarp();
            // one-body sums of the moved electrons, by their lanes, as the warp sum over the
            // nuclei's lanes adds them
            if (moved >> lane & 1) jc[NPAIR + sig * NUP + lane] = wsum_order<NE1, NNUC>(ph + (sig * NM + lane) * GRS);
            __syncwarp();
            const F2 sc(csc);
#pragma unroll
            for (int v = 0; v < NM / 2; ++v) D.p[v] = mul2(D.p[v], sc);
            if constexpr (NM % 2) D.t *= csc;
        }
    }
    {
        float x[2], y[2], z[2];
        p1.get(x[0], y[1]);
        p2.get(y[0], x[1]);
        pz.get(z[0], z[1]);
#pragma unroll
        for (int r = 0; r < 2; ++r)
            if (r == 0 ? lane < NE : is_el) {
                const int j = lane + 32 * r;
                a.pos[(3 * j + 0) * (size_t)a.Wcap + w] = x[r];
                a.pos[(3 * j + 1) * (size_t)a.Wcap + w] = y[r];
                a.pos[(3 * j + 2) * (size_t)a.Wcap + w] = z[r];
            }
    }
#pragma unroll
    for (int sig = 0; sig < 2; ++sig) {
        const ColF2<NM>& D = sig == 0 ? D0 : D1;
        if (lane >= (sig == 0 ? NUP : NDN)) continue;
        float* out = a.dinv + ((size_t)sig * NM * NM + lane) * a.Wcap + w;
        const size_t rs = (size_t)NM * a.Wcap;
#pragma unroll
        for (int v = 0; v < NM / 2; ++v) {
            float lo, hi;
            D.p[v].get(lo, hi);
            out[2 * v * rs] = lo;
            out[(2 * v + 1) * rs] = hi;
        }
        if constexpr (NM % 2) out[(NM - 1) * rs] = D.t;
    }
    if (lane == 0) {
        a.sign[w] = sgn;
        if (acc) atomicAdd(a.acc, (unsigned long long)acc);
        if (flg) atomicOr(a.flags, flg);
    }
}

// Block size of the FP32 Gaussian sweep in dynamic shared memory.
template <int NE, int NUP, int NNUC, int WPB>
static size_t gauss_smem(int n_ao) {
    return GaussTab<NNUC, (NUP > NE - NUP ? NUP : NE - NUP)>::bytes(n_ao) + sizeof(float) * WPB * gauss_scratch_elems<NE, NUP>();
}
// Dynamic shared memory: the table's used part, then the warps' scratch.
template <int NE, int NUP, int NNUC, class TAB>
__device__ __forceinline__ void gauss_block(const TAB* __restrict__ Sg, const volatile SweepArgs<float>& a, unsigned char* sm,
                                            int w) {
    TAB& S = *reinterpret_cast<TAB*>(sm);
    load_tab(&S, Sg);                      // ends with a block barrier
    if (w >= a.W) return;                      // whole warps only; no block barrier below
    kw_gauss_walker<NE, NUP, NNUC>(S, a, w, reinterpret_cast<float*>(sm + TAB::bytes(S.n_ao)) +
                                                (size_t)(threadIdx.x >> 5) * gauss_scratch_elems<NE, NUP>());
}
template <int NE, int NUP, int NNUC, int WPB, class TAB>
__global__ void __launch_bounds__(32 * WPB, 16 / WPB) kw_gauss(const TAB* __restrict__ Sg, const __grid_constant__ SweepArgs<float> args0) {
    __shared__ SweepArgs<float> args;
    extern __shared__ __align__(16) unsigned char wsm[];
    if (threadIdx.x == 0) args = args0;
    gauss_block<NE, NUP, NNUC>(Sg, args, wsm, (int)blockIdx.x * WPB + (int)(threadIdx.x >> 5));
}
template <int NE, int NUP, int NNUC, int WPB, int TW, class TAB>
__global__ void __launch_bounds__(32 * WPB, 16 / WPB) kwb_gauss(const BatchTile* __restrict__ tiles, int ntiles,
                                                                const BatchRec* __restrict__ recs, const BatchCtl* __restrict__ ctl) {
    static_assert(TW % WPB == 0, "a tile splits into whole blocks");
    constexpr int BPT = TW / WPB;
    __shared__ SweepArgs<float> args;
    extern __shared__ __align__(16) unsigned char wsm[];
    if ((int)blockIdx.x >= ntiles * BPT) return;
    const BatchTile tl = tiles[blockIdx.x / BPT];
    if (threadIdx.x == 0) args = sweep_args<float>(recs[tl.rec], *ctl);
    gauss_block<NE, NUP, NNUC>(static_cast<const TAB*>(recs[tl.rec].tab_g), args, wsm,
                               tl.w0 + (int)(blockIdx.x % BPT) * WPB + (int)(threadIdx.x >> 5));
}

// FP32: four 4-walker blocks per SM (<= 128 registers)
template <int NE, int NUP, int NNUC, class T, int MOVE, int WPB>
__global__ void __launch_bounds__(32 * WPB, sizeof(T) == 4 ? 16 / WPB : 1) kw_sweep(const SysW<T>* __restrict__ Sg, T* __restrict__ gpos,
                                                     T* __restrict__ gdinv, int* __restrict__ gsign, int W, int Wcap,
                                                     int n_sweeps, uint64_t step0, T step, T tau, T maxd,
                                                     uint64_t seed, unsigned long long* acc_out, int* flags,
                                                     int fixed_node) {
    __shared__ SysW<T> S;
    __shared__ SweepArgs<T> args;
    if (threadIdx.x == 0)
        args = SweepArgs<T>{gpos, gdinv, gsign, acc_out, flags, step0, seed, step, tau, maxd, W, Wcap, n_sweeps,
                            fixed_node};
    extern __shared__ __align__(16) unsigned char wsm[];
    load_sysw(&S, Sg);                         // ends with a block barrier
    const int w = blockIdx.x * WPB + (threadIdx.x >> 5);
    if (w >= W) return;                        // whole warps only; no block barrier below
    const volatile SweepArgs<T>& a = args;
    T* ph = reinterpret_cast<T*>(wsm) + (size_t)(threadIdx.x >> 5) * sweep_scratch_elems<NE, NUP, MOVE>();
    kw_sweep_walker<NE, NUP, NNUC, T, MOVE>(S, a, w, ph);
}

// Batched form: TW / WPB blocks per (system, TW-walker tile), each sweeping
// WPB walkers of it.  The hardware block scheduler balances uneven systems
// and classes that run side by side, and the kernel carries no tile-loop
// state into the walker's registers.
template <int NE, int NUP, int NNUC, class T, int MOVE, int WPB, int TW>
__global__ void __launch_bounds__(32 * WPB, sizeof(T) == 4 ? 16 / WPB : 1) kwb_sweep(const BatchTile* __restrict__ tiles, int ntiles,
                                                      const BatchRec* __restrict__ recs,
                                                      const BatchCtl* __restrict__ ctl) {
    static_assert(TW % WPB == 0, "a tile splits into whole blocks");
    constexpr int BPT = TW / WPB;
    __shared__ SysW<T> S;
    __shared__ SweepArgs<T> args;
    if ((int)blockIdx.x >= ntiles * BPT) return;
    const BatchTile tl = tiles[blockIdx.x / BPT];
    if (threadIdx.x == 0) args = sweep_args<T>(recs[tl.rec], *ctl);
    extern __shared__ __align__(16) unsigned char wsm[];
    load_sysw(&S, static_cast<const SysW<T>*>(recs[tl.rec].tab_s));   // ends with a block barrier
    const volatile SweepArgs<T>& a = args;
    const int w = tl.w0 + (int)(blockIdx.x % BPT) * WPB + (int)(threadIdx.x >> 5);
    if (w >= a.W) return;                      // whole warps only; no block barrier below
    T* ph = reinterpret_cast<T*>(wsm) + (size_t)(threadIdx.x >> 5) * sweep_scratch_elems<NE, NUP, MOVE>();
    kw_sweep_walker<NE, NUP, NNUC, T, MOVE>(S, a, w, ph);
}

// Full evaluation from positions (refresh + E_L) in FP32, one warp per walker.
// Per-warp shared scratch holds the sector's D rows, then the rows of its
// inverse; orbital derivatives are evaluated in a second pass.
// Row stride of the refresh's per-warp matrix scratch: lane q writes row q
// (element (q, k) at q MRS + k) and lane j reads column j; an odd stride keeps
// both conflict-free.
constexpr int MRS = 33;

// Orbital values phi_k(x, y, z), k < NM, of sector sig by one lane: one pass
// over the radial groups, lazily accumulated in the compute type.
template <class TC, int NM>
__device__ __forceinline__ void orbital_values(const SysW<TC>& S, int sig, TC x, TC y, TC z, TC (&v)[NM]) {
#pragma unroll
    for (int k = 0; k < NM; ++k) v[k] = 0;
    for (int g = 0; g < S.n_grp; ++g) {
        const int d = S.grp[g];
        const int I = d & 15, kind = (d >> 4) & 1, np = (d >> 5) & 15, p0 = (d >> 9) & 255, a0 = grp_a0(d);
        const TC dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
        const TC r2 = dx * dx + dy * dy + dz * dz;
        TC s0 = 0;
        for (int p = p0; p < p0 + np; ++p) {
            TC al_p, cp;
            load2(S.prim[p], al_p, cp);
            s0 += cp * fexp(-al_p * r2);
        }
        for (int m = 0; m < (kind ? 3 : 1); ++m) {
            const TC chi = kind ? (m == 0 ? dx : (m == 1 ? dy : dz)) * s0 : s0;
            const TC* c = S.C[sig][a0 + m];
#pragma unroll
            for (int k = 0; k < NM; ++k) macc(v[k], c[k], chi);
        }
    }
#pragma unroll
    for (int k = 0; k < NM; ++k) v[k] = macc_norm(v[k]);
}

// sum_a c'_a (grad chi_a, lap chi_a) at (x, y, z) with c'_a = sum_k C[sig][a][k] dcol[k]:
// one pass over the radial groups (s AO, or p triplet sharing its radial part;
// s: grad = -2 R1 dr, lap = -6 R1 + 4 r^2 R2; p_m: grad = x_m (-2 R1 dr) + e_m R0,
// lap = x_m (-10 R1 + 4 r^2 R2), with R0, R1, R2 the radial sums weighted by
// 1, alpha, alpha^2).
template <class TC, int NM>
__device__ __forceinline__ void inverse_weighted_derivatives(const SysW<TC>& S, int sig, TC x, TC y, TC z,
                                                             const TC (&dcol)[NM], TC& gx, TC& gy, TC& gz, TC& lp) {
    TC ax = 0, ay = 0, az = 0, al = 0;
    for (int g = 0; g < S.n_grp; ++g) {
        const int d = S.grp[g];
        const int I = d & 15, kind = (d >> 4) & 1, np = (d >> 5) & 15, p0 = (d >> 9) & 255, a0 = grp_a0(d);
        const TC dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
        const TC r2 = dx * dx + dy * dy + dz * dz;
        TC s0 = 0, s1 = 0, s2 = 0;
        for (int p = p0; p < p0 + np; ++p) {
            TC al_p, cp;
            load2(S.prim[p], al_p, cp);
            const TC e = cp * fexp(-al_p * r2), ea = al_p * e;
            s0 += e; s1 += ea; s2 += al_p * ea;
        }
        const TC l0 = TC(4) * r2 * s2;
        for (int m = 0; m < (kind ? 3 : 1); ++m) {
            const TC* c = S.C[sig][a0 + m];
            TC cw = 0;
#pragma unroll
            for (int k = 0; k < NM; ++k) macc(cw, c[k], dcol[k]);
            cw = macc_norm(cw);
            TC gxa, gya, gza, la;
            if (kind == 0) {
                const TC t = TC(-2) * s1;
                gxa = t * dx; gya = t * dy; gza = t * dz;
                la = TC(-6) * s1 + l0;
            } else {
                const TC xm = m == 0 ? dx : (m == 1 ? dy : dz);
                const TC t = TC(-2) * s1 * xm;
                gxa = t * dx + (m == 0 ? s0 : TC(0));
                gya = t * dy + (m == 1 ? s0 : TC(0));
                gza = t * dz + (m == 2 ? s0 : TC(0));
                la = xm * (TC(-10) * s1 + l0);
            }
            macc(ax, cw, gxa); macc(ay, cw, gya); macc(az, cw, gza); macc(al, cw, la);
        }
    }
    gx = macc_norm(ax); gy = macc_norm(ay); gz = macc_norm(az); lp = macc_norm(al);
}

template <int NE, int NUP, int NNUC, class TC, class TS>
__device__ __forceinline__ double kw_measure_walker(const SysW<TC>& S, TC* Mrow, const TS* __restrict__ gpos,
                                                    TS* __restrict__ gdinv, double* __restrict__ glog,
                                                    int* __restrict__ gsign, double* __restrict__ gel, int w,
                                                    bool act, int Wcap, int write_state,
                                                    double* __restrict__ out_grad, double* __restrict__ out_lap,
                                                    int* flags) {
    constexpr int NDN = NE - NUP;
    constexpr int NM = NUP > NDN ? NUP : NDN;
    const int lane = threadIdx.x & 31;
    double e_l = 0.0;
    if (act) {
        LanePos<TC, NE> P;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int j = lane + 32 * r;
            const bool ok = j < NE;
            P.x[r] = ok ? (TC)gpos[(3 * j + 0) * (size_t)Wcap + w] : TC(0);
            P.y[r] = ok ? (TC)gpos[(3 * j + 1) * (size_t)Wcap + w] : TC(0);
            P.z[r] = ok ? (TC)gpos[(3 * j + 2) * (size_t)Wcap + w] : TC(0);
        }
        double logdet = 0.0;
        int sg = 1;
        bool ok = true;
        // per-lane electron results: lane owns electron (sig*NUP + lane) of each sector
        TC gdx[2] = {0, 0}, gdy[2] = {0, 0}, gdz[2] = {0, 0}, ld[2] = {0, 0};
#pragma unroll
        for (int sig = 0; sig < 2; ++sig) {
            const int NS = sig == 0 ? NUP : NDN;
            // pass 1, lane q = electron q of the sector: its orbital values,
            // written as row q of D
            TC xq, yq, zq;
            P.get_own(min(sig * NUP + lane, NE - 1), xq, yq, zq);
            if (lane < NS) {
                TC v[NM];
                orbital_values<TC, NM>(S, sig, xq, yq, zq, v);
#pragma unroll
                for (int k = 0; k < NM; ++k)
                    if (k < NS) Mrow[lane * MRS + k] = v[k];
            }
            __syncwarp();
            // Gauss-Jordan in place with partial pivoting: lane j carries
            // column j of D and ends with column j of the inverse of the
            // row-permuted matrix.  Step k: rows k and p = argmax |D[i][k]|
            // interchanged; row k divided by a = D[k][k], column k becomes
            // -D[i][k]/a (1/a on the diagonal), the rest loses D[i][k] x row k
            // -- lane k's update takes the same form with t = 1 + 1/a.  The row
            // interchanges are undone as column interchanges: lane j gathers
            // column src(j), src = tau_{n-1}( ... tau_0(j)).  The pivot loop is
            // rolled, one copy of the step's code for all NS steps: the
            // registers hold the rows rotated so that row k sits in register 0
            // at step k (rows not yet pivoted first, in the order an unrolled
            // loop would have them), and each step moves register 0 to the back.
            TC A[NM];
#pragma unroll
            for (int i = 0; i < NM; ++i) A[i] = (i < NS && lane < NS) ? Mrow[i * MRS + lane] : TC(i == lane ? 1 : 0);
            int src = lane;
#pragma unroll 1
            for (int k = 0; k < NS; ++k) {
                int p = 0;
                float best = fabsf(lead(A[0]));
#pragma unroll
                for (int r = 1; r < NM; ++r) {
                    const float m = fabsf(lead(A[r]));
                    if (r < NS - k && m > best) { best = m; p = r; }
                }
                p = wshfl(p, k);
#pragma unroll
                for (int r = 1; r < NM; ++r) {
                    bool sw = (r == p);
                    TC a = A[0], b = A[r];
                    A[0] = sw ? b : a; A[r] = sw ? a : b;
                }
                if (p != 0) sg = -sg;
                const int pk = k + p;
                src = (src == k) ? pk : ((src == pk) ? k : src);
                TC piv = wshfl(A[0], k);
                if (!(piv != TC(0))) { ok = false; piv = TC(1); }
                if (piv < 0) sg = -sg;
                logdet += log(fabs((double)piv));
                const TC ip = TC(1) / piv;
                const TC t = (lane == k) ? TC(1) + ip : A[0] * ip;
                A[0] = (lane == k) ? ip : t;
#pragma unroll
                for (int i = 1; i < NM; ++i) {
                    if (i >= NS) continue;
                    const TC f = wshfl(A[i], k);
                    A[i] -= f * t;
                }
                // rotate registers 0..NS-1 by one: the pivoted row goes last
                const TC r0 = A[0];
#pragma unroll
                for (int i = 0; i + 1 < NM; ++i) {
                    if (i + 1 < NS) A[i] = A[i + 1];
                    else if (i + 1 == NS) A[i] = r0;
                }
                if (NS == NM) A[NM - 1] = r0;
            }
            // unscramble: lane j takes column src(j); then A[k] = D^-1[k][lane]
#pragma unroll
            for (int i = 0; i < NM; ++i) {
                if (i >= NS) break;
                A[i] = wshfl(A[i], src);
            }
            if (write_state && lane < NS) {
#pragma unroll
                for (int k = 0; k < NM; ++k)
                    if (k < NS) gdinv[((size_t)(sig * NM * NM + k * NM + lane)) * Wcap + w] = (TS)A[k];
            }
            __syncwarp();
            // pass 2, lane q = electron q of the sector, holding column q of
            // D^-1: grad ln D = sum_k grad phi_k(r_q) D^-1[k][q] = sum_a c'_a
            // grad chi_a(r_q) with c'_a = sum_k C[a][k] D^-1[k][q] (the inverse
            // column contracted into the coefficients first), and the same for
            // lap D / D, over the radial groups at the lane's own electron
            if (lane < NS)
                inverse_weighted_derivatives<TC, NM>(S, sig, xq, yq, zq, A, gdx[sig], gdy[sig], gdz[sig], ld[sig]);
            __syncwarp();
        }
        // Jastrow + Coulomb for this lane's electrons (pairs counted from both ends)
        TC u = 0, V = 0, kin = 0;
#pragma unroll
        for (int sig = 0; sig < 2; ++sig) {
            const int NS = sig == 0 ? NUP : NDN;
            const int i = sig * NUP + lane;
            const bool own = lane < NS;
            TC xi, yi, zi;
            P.get_own(min(i, NE - 1), xi, yi, zi);
            TC gx = 0, gy = 0, gz = 0, lu = 0, gsq = 0;
            for (int j = 0; j < NE; ++j) {
                TC xj, yj, zj;
                P.get(j, xj, yj, zj);
                if (!own || j == i) continue;
                const bool para = ((j < NUP) == (i < NUP));
                TC dx = xi - xj, dy = yi - yj, dz = zi - zj;
                TC d, ri;
                dist(dx * dx + dy * dy + dz * dz, d, ri);
                V += TC(0.5) * ri;
                TC uu, upr, lt;
                const int c = para ? 1 : 0;
                pade_ab(S.a_ee[c], S.b_ee[c], d, ri, uu, upr, lt);
                u += TC(0.5) * uu;
                if (!(d < TC(1e-10))) {
                    gx += upr * dx; gy += upr * dy; gz += upr * dz;
                    lu += lt;
                    TC up = upr * d;
                    gsq += up * up;
                }
            }
            if (own) {
                for (int I = 0; I < NNUC; ++I) {
                    TC dx = xi - S.nuc[I][0], dy = yi - S.nuc[I][1], dz = zi - S.nuc[I][2];
                    TC d, ri;
                    dist(dx * dx + dy * dy + dz * dz, d, ri);
                    V -= S.Z[I] * ri;
                    TC uu, upr, lt;
                    pade_ab(S.enA[I], S.enB[I], d, ri, uu, upr, lt);
                    u -= uu;
                    if (!(d < TC(1e-10))) {
                        gx -= upr * dx; gy -= upr * dy; gz -= upr * dz;
                        lu -= lt;
                    }
                }
                TC ax = S.qa * gx, ay = S.qa * gy, az = S.qa * gz;
                TC lj = S.quirk_lap ? (lu + gsq) : (lu + gx * gx + gy * gy + gz * gz);
                TC lp = ld[sig] + 2 * (gdx[sig] * ax + gdy[sig] * ay + gdz[sig] * az) + lj;
                kin += lp;
                const int ecall = i;   // internal index; host permutes to caller order
                if (out_grad) {
                    out_grad[((size_t)w * NE + ecall) * 3 + 0] = (double)(gdx[sig] + ax);
                    out_grad[((size_t)w * NE + ecall) * 3 + 1] = (double)(gdy[sig] + ay);
                    out_grad[((size_t)w * NE + ecall) * 3 + 2] = (double)(gdz[sig] + az);
                }
                if (out_lap) out_lap[(size_t)w * NE + ecall] = (double)lp;
            }
        }
        u = wsum(u);
        V = wsum(V);
        kin = wsum(kin);
        e_l = (double)(TC(-0.5) * kin + V + S.v_nn);
        if (lane == 0) {
            int fl = 0;
            if (!ok) fl |= FLAG_SINGULAR;
            if (!isfinite(e_l)) fl |= FLAG_NONFINITE;
            if (fl) atomicOr(flags, fl);
            if (write_state) { glog[w] = logdet + (double)u; gsign[w] = sg; gel[w] = e_l; }
        }
    }
    return act ? e_l : 0.0;
}

// ---------------------------------------------------------------------------
// FP64 evaluation and refresh, one warp per walker.  An FP64 instruction holds its
// sub-partition for 64 cycles however many of its lanes are active, so the work is
// laid out to fill lanes, where one lane per electron of a sector left 11 of 32 idle:
// radial parts are (electron, shell) tasks, orbital values (electron, third of the
// columns), derivative sums (electron, third of the shells); pairs and nucleus terms
// are evaluated once each and added to per-electron sums; pivots are compared, and
// |det| is kept, on the bits, with one logarithm a walker.  Orbital matrices and
// inverses keep the rounding of a lane per electron with the CUDA library's
// exponential, so that configurations next to a node, which amplify it, keep their
// values (largest change over 30 000 configurations 4e-13).  500 configurations
// through the host call: 797 us before, 521 us now (484 us with d_exp and the values
// summed in thirds, which moved such configurations by up to 1e-8).
// ---------------------------------------------------------------------------
template <int NNUC, int NM>
struct EvalTab {
    int n_ao, n_sh, n_third, quirk_lap;
    double qa, v_nn, a_ee[2], b_ee[2];
    double nuc[NNUC][6];                      // x, y, z, Z, enA, enB
    int sh[WMAX_AO], third[WMAX_THIRD];       // shells in AO order; the same in thirds
    // exponent; c, c a, c a^2 of the s or lone p part; the same of an sp shell's p part
    alignas(16) double prim[WMAX_PRIM][8];
    double C[WMAX_AO][2][NM + 1];             // [AO][sector][column], rows of whole 16-byte words
    __host__ __device__ static size_t bytes(int n_ao) {
        return offsetof(EvalTab, C) + sizeof(double) * 2 * (NM + 1) * (size_t)n_ao;
    }
    __device__ static size_t used(const EvalTab* t) { return bytes(t->n_ao); }
};

template <int NNUC, int NM>
static void fill_evaltab(const SysW<double>& w, EvalTab<NNUC, NM>& S) {
    static_assert(NM % 2 == 1, "padded rows are 16-byte words");
    std::memset(static_cast<void*>(&S), 0, sizeof(S));
    const ShellList<double> L(w);
    S.n_ao = w.n_ao;
    S.n_sh = (int)L.desc.size();
    for (int g = 0; g < S.n_sh; ++g) S.sh[g] = L.desc[g];
    S.n_third = deal_thirds(L.desc, S.third);
    S.quirk_lap = w.quirk_lap;
    S.qa = w.qa;
    S.v_nn = w.v_nn;
    for (int c = 0; c < 2; ++c) { S.a_ee[c] = w.a_ee[c]; S.b_ee[c] = w.b_ee[c]; }
    for (int I = 0; I < NNUC; ++I) {
        const double v[6] = {w.nuc[I][0], w.nuc[I][1], w.nuc[I][2], w.Z[I], w.enA[I], w.enB[I]};
        for (int c = 0; c < 6; ++c) S.nuc[I][c] = v[c];
    }
    for (size_t p = 0; p < L.al.size(); ++p) {
        const double a = L.al[p], v[7] = {a, L.c[p], L.c[p] * a, L.c[p] * a * a, L.cp[p], L.cp[p] * a, L.cp[p] * a * a};
        for (int c = 0; c < 7; ++c) S.prim[p][c] = v[c];
    }
    for (int a = 0; a < w.n_ao; ++a)
        for (int sig = 0; sig < 2; ++sig)
            for (int k = 0; k < NM; ++k) S.C[a][sig][k] = w.C[sig][a][k];
}

// Shared doubles of a warp: row e of the electron's orbital values, then of its column
// of the inverse, later positions [3][NE] and sums [5][NE] over the same storage; then
// the derivative sums [4][NE]; then radial parts [EVAL_SH][2][NM] of a sector's
// electrons (six shells: 126 tasks, four rounds of lanes).
constexpr int EVAL_SH = 6;
template <int NE, int NM>
__host__ __device__ constexpr int eval_rows() { return (NE * NM > 8 * NE ? NE * NM : 8 * NE) + (NE * NM) % 2; }
template <int NE, int NM>
__host__ __device__ constexpr int eval_scratch() { return eval_rows<NE, NM>() + 4 * NE + 2 * NM * EVAL_SH; }

template <int NE, int NUP, int NNUC, class TAB>
__device__ __forceinline__ double kw_eval_walker(const TAB& S, double* scr, const double* __restrict__ gpos,
                                                 double* __restrict__ gdinv, double* __restrict__ glog,
                                                 int* __restrict__ gsign, double* __restrict__ gel, int w, int Wcap,
                                                 int write_state, double* __restrict__ out_grad,
                                                 double* __restrict__ out_lap, int* flags) {
    static_assert(NE == 2 * NUP && NUP <= 32 && NE >= 32, "equal sectors; a round's tasks are of distinct electrons");
    constexpr int NM = NUP, ROUNDS = (3 * NE + 31) / 32;
    const int lane = threadIdx.x & 31;
    double* der = scr + eval_rows<NE, NM>();
    // task of this lane in a round (the spare lanes of the last round repeat the last task)
    auto task_of = [&](int round, int& e, int& t3) {
        const int task = min(32 * round + lane, 3 * NE - 1);
        t3 = task / NE;
        e = task - t3 * NE;
        return 32 * round + lane < 3 * NE;
    };
    auto coord = [&](int e, int c) { return gpos[(size_t)(3 * e + c) * Wcap + w]; };
    // Orbital values, row e of the electron's matrix, in the plain order of operations
    // (the sum over a shell's primitives, then the sum over the AOs as they come):
    // next to a node their rounding is what the inverse amplifies, so another order
    // would be another, equally good, value there.  The radial parts are (electron,
    // shell) tasks, the contraction (electron, third of the columns) tasks.
    static_assert(NM % 3 == 0 && 3 * NM <= 64, "columns in thirds, two tasks a lane");
    constexpr int NC = NM / 3;
    double* rad = der + 4 * NE;
#pragma unroll 1
    for (int sig = 0; sig < 2; ++sig) {
        double v[2][NC];                       // the lane's tasks `lane` and `lane + 32`
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < NC; ++k) v[h][k] = 0;
#pragma unroll 1
        for (int g0 = 0; g0 < S.n_sh; g0 += EVAL_SH) {
            const int ng = min(EVAL_SH, S.n_sh - g0);
#pragma unroll 1
            for (int t = lane; t < NM * ng; t += 32) {
                const int g = t / NM, q = t - g * NM, e = sig * NUP + q, d = S.sh[g0 + g];
                const int I = shell_nuc(d), np = shell_np(d), p0 = shell_p0(d);
                const bool sp = (d & SHELL_S) && (d & SHELL_P);
                const double dx = coord(e, 0) - S.nuc[I][0], dy = coord(e, 1) - S.nuc[I][1], dz = coord(e, 2) - S.nuc[I][2];
                const double r2 = dx * dx + dy * dy + dz * dz;
                double s0 = 0, s1 = 0;
                for (int p = p0; p < p0 + np; ++p) {
                    const double ex = exp(-S.prim[p][0] * r2);
                    s0 += S.prim[p][1] * ex;
                    if (sp) s1 += S.prim[p][4] * ex;
                }
                rad[2 * g * NM + q] = s0;
                rad[(2 * g + 1) * NM + q] = sp ? s1 : s0;
            }
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = min(lane + 32 * h, 3 * NM - 1), third = t / NM, q = t - third * NM, e = sig * NUP + q;
                const double x = coord(e, 0), y = coord(e, 1), z = coord(e, 2);
#pragma unroll 1
                for (int g = 0; g < ng; ++g) {
                    const int d = S.sh[g0 + g], I = shell_nuc(d);
                    const double s0 = rad[2 * g * NM + q], s1 = rad[(2 * g + 1) * NM + q];
                    const double* c = &S.C[shell_a0(d)][sig][third * NC];
                    constexpr int row = 2 * (NM + 1);
                    if (d & SHELL_S) {
#pragma unroll
                        for (int k = 0; k < NC; ++k) v[h][k] += c[k] * s0;
                        c += row;
                    }
                    if (d & SHELL_P) {
                        const double cx = (x - S.nuc[I][0]) * s1, cy = (y - S.nuc[I][1]) * s1, cz = (z - S.nuc[I][2]) * s1;
#pragma unroll
                        for (int k = 0; k < NC; ++k) v[h][k] += c[k] * cx;
#pragma unroll
                        for (int k = 0; k < NC; ++k) v[h][k] += c[row + k] * cy;
#pragma unroll
                        for (int k = 0; k < NC; ++k) v[h][k] += c[2 * row + k] * cz;
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = lane + 32 * h, third = t / NM, q = t - third * NM;
            if (t < 3 * NM) {
#pragma unroll
                for (int k = 0; k < NC; ++k) scr[(sig * NUP + q) * NM + third * NC + k] = v[h][k];
            }
        }
    }
    __syncwarp();
    // Gauss-Jordan of each sector (kw_measure_walker's steps), lane j with column j
    double det = 1.0, logdet = 0.0;            // |det| = det 2^ex exp(logdet)
    int ex = 0, sg = 1;
    bool ok = true;
#pragma unroll 1
    for (int sig = 0; sig < 2; ++sig) {
        double* M = scr + sig * NM * NM;
        double A[NM];
#pragma unroll
        for (int i = 0; i < NM; ++i) A[i] = lane < NM ? M[i * NM + lane] : 0.0;
        __syncwarp();
        int src = lane;
#pragma unroll 1
        for (int k = 0; k < NM; ++k) {
            // magnitudes to 24 bits, on the bits (a conversion is an FP64 instruction)
            auto mag = [](double a) {
                return (((unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffull) + 0x10000000ull) >> 29;
            };
            int p = 0;
            unsigned long long best = mag(A[0]);
#pragma unroll
            for (int r = 1; r < NM; ++r) {
                const unsigned long long m = mag(A[r]);
                if (r < NM - k && m > best) { best = m; p = r; }
            }
            p = wshfl(p, k);
#pragma unroll
            for (int r = 1; r < NM; ++r) {
                const bool sw = r == p;
                const double a = A[0], b = A[r];
                A[0] = sw ? b : a;
                A[r] = sw ? a : b;
            }
            if (p != 0) sg = -sg;
            const int pk = k + p;
            src = src == k ? pk : (src == pk ? k : src);
            double piv = wshfl(A[0], k);
            if (((d_hi(piv) & 0x7fffffff) | d_lo(piv)) == 0) { ok = false; piv = 1.0; }
            const int h = d_hi(piv), f = (h >> 20) & 0x7ff;
            if (h < 0) sg = -sg;
            if (f == 0 || f == 0x7ff) {
                logdet += log(fabs(piv));
            } else {
                det *= __hiloint2double((h & 0x000fffff) | 0x3ff00000, d_lo(piv));
                ex += f - 1023;
            }
            const double ip = 1.0 / piv;
            const double t = lane == k ? 1.0 + ip : A[0] * ip, first = lane == k ? ip : t;
#pragma unroll
            for (int i = 1; i < NM; ++i) A[i - 1] = A[i] - wshfl(A[i], k) * t;
            A[NM - 1] = first;
        }
#pragma unroll
        for (int i = 0; i < NM; ++i) A[i] = wshfl(A[i], src);
        if (lane < NM) {
#pragma unroll
            for (int k = 0; k < NM; ++k) {
                M[lane * NM + k] = A[k];
                if (write_state) gdinv[((size_t)(sig * NM * NM + k * NM + lane)) * Wcap + w] = A[k];
            }
        }
    }
    logdet += d_log(det) + (double)ex * 0.6931471805599453;
    __syncwarp();
    // grad ln D and lap D / D of each electron: sum_a c'_a (grad, lap) chi_a with
    // c'_a = sum_k C[a][k] D^-1[k][q] (kw_refresh_walker has the formulas)
#pragma unroll 1
    for (int round = 0; round < ROUNDS; ++round) {
        int e, t3;
        const bool on = task_of(round, e, t3);
        const int sig = e >= NUP;
        const double x = coord(e, 0), y = coord(e, 1), z = coord(e, 2);
        double A[NM];
#pragma unroll
        for (int k = 0; k < NM; ++k) A[k] = scr[e * NM + k];
        double gx = 0, gy = 0, gz = 0, ld = 0;
#pragma unroll 1
        for (int g = 0; g < S.n_third; ++g) {
            const int d = S.third[3 * g + t3];
            const int I = shell_nuc(d), np = shell_np(d), p0 = shell_p0(d), a0 = shell_a0(d);
            const int ns = (d & SHELL_S) ? 1 : 0, na = ns + ((d & SHELL_P) ? 3 : 0);
            const bool sp = na == 4;
            const double dx = x - S.nuc[I][0], dy = y - S.nuc[I][1], dz = z - S.nuc[I][2];
            const double r2 = dx * dx + dy * dy + dz * dz, r4 = 4.0 * r2;
            double s0 = 0, s1 = 0, s2 = 0, q0 = 0, q1 = 0, q2 = 0;
            for (int p = p0; p < p0 + np; ++p) {
                const double* t = S.prim[p];
                const double E = d_exp(-t[0] * r2);
                s0 += t[1] * E;
                s1 += t[2] * E;
                s2 += t[3] * E;
                if (sp) {
                    q0 += t[4] * E;
                    q1 += t[5] * E;
                    q2 += t[6] * E;
                }
            }
            double cd = 0;
#pragma unroll 1
            for (int m = 0; m < na; ++m) {
                const double* c = S.C[a0 + m][sig];
                // two sums, for the latency of the chain
                double c0 = 0, c1 = 0;
#pragma unroll
                for (int k = 0; k + 1 < NM; k += 2) { c0 += c[k] * A[k]; c1 += c[k + 1] * A[k + 1]; }
                if (NM % 2) c0 += c[NM - 1] * A[NM - 1];
                const double cw = c0 + c1;
                const int c3 = m - ns;
                if (c3 < 0) {
                    cd = cw;
                } else {
                    if (c3 == 0 && sp) { s0 = q0; s1 = q1; s2 = q2; cd = 0; }
                    cd += cw * (c3 == 0 ? dx : (c3 == 1 ? dy : dz));
                    const double o = s0 * cw;
                    if (c3 == 0) gx += o;
                    else if (c3 == 1) gy += o;
                    else gz += o;
                }
                if (c3 < 0 || c3 == 2) {
                    const double t = -2.0 * s1 * cd;
                    gx += t * dx; gy += t * dy; gz += t * dz;
                    ld += cd * (r4 * s2 - (c3 < 0 ? 6.0 : 10.0) * s1);
                }
            }
        }
        if (on) {
            const double v[4] = {gx, gy, gz, ld};
#pragma unroll
            for (int c = 0; c < 4; ++c) der[c * NE + e] = t3 == 0 ? v[c] : der[c * NE + e] + v[c];
        }
        __syncwarp();
    }
    // Jastrow and Coulomb terms: pair p joins electron i = p mod NE with i + p / NE + 1
    // (mod NE), the last NE / 2 pairs i with i + NE / 2; 32 consecutive pairs have
    // distinct i and distinct j, so the sums need no atomics
    double *pos = scr, *sums = scr + 3 * NE;
    for (int e = lane; e < NE; e += 32) {
#pragma unroll
        for (int c = 0; c < 3; ++c) pos[c * NE + e] = coord(e, c);
#pragma unroll
        for (int c = 0; c < 5; ++c) sums[c * NE + e] = 0.0;
    }
    __syncwarp();
    double u = 0, V = 0;
    // terms at separation r2: u, u'/r, u'' + 2u'/r, 1/r (0 at r = 0) and r
    auto pade = [](double a, double b, double r2, double& uu, double& f, double& l, double& ri, double& r) {
        dist(r2, r, ri);
        const double inv = frcp(1.0 + b * r), ai = a * inv, up = ai * inv;
        uu = ai * r;
        f = up * ri;
        l = 2.0 * (f - up * (b * inv));
    };
    constexpr int NPAIR = NE * (NE - 1) / 2, FULL = NE * ((NE - 1) / 2);
    static_assert(NE % 2 == 0, "the last NE / 2 pairs join opposite electrons");
#pragma unroll 1
    for (int r0 = 0; r0 < NPAIR; r0 += 32) {
        const bool on = r0 + lane < NPAIR;
        const int p = on ? r0 + lane : NPAIR - 1;
        const int i = p < FULL ? p % NE : p - FULL;
        int j = p < FULL ? i + p / NE + 1 : i + NE / 2;
        if (j >= NE) j -= NE;
        const double dx = pos[i] - pos[j], dy = pos[NE + i] - pos[NE + j], dz = pos[2 * NE + i] - pos[2 * NE + j];
        const int c = (j < NUP) == (i < NUP) ? 1 : 0;
        double uu, f, l, ri, r;
        pade(S.a_ee[c], S.b_ee[c], dx * dx + dy * dy + dz * dz, uu, f, l, ri, r);
        if (on) { u += uu; V += ri; }
        const bool use = on && !closer(r, 1e-10);
        const double fx = f * dx, fy = f * dy, fz = f * dz;
        if (use) {
            sums[i] += fx; sums[NE + i] += fy; sums[2 * NE + i] += fz; sums[3 * NE + i] += l;
        }
        __syncwarp();
        if (use) {
            sums[j] -= fx; sums[NE + j] -= fy; sums[2 * NE + j] -= fz; sums[3 * NE + j] += l;
        }
        if (S.quirk_lap) {
            const double up = f * r, sq = up * up;
            if (use) sums[4 * NE + i] += sq;
            __syncwarp();
            if (use) sums[4 * NE + j] += sq;
        }
        __syncwarp();
    }
#pragma unroll 1
    for (int r0 = 0; r0 < NE * NNUC; r0 += 32) {
        const bool on = r0 + lane < NE * NNUC;
        const int p = on ? r0 + lane : NE * NNUC - 1, I = p / NE, e = p - I * NE;
        const double dx = pos[e] - S.nuc[I][0], dy = pos[NE + e] - S.nuc[I][1], dz = pos[2 * NE + e] - S.nuc[I][2];
        double uu, f, l, ri, r;
        pade(S.nuc[I][4], S.nuc[I][5], dx * dx + dy * dy + dz * dz, uu, f, l, ri, r);
        if (on) {
            u -= uu;
            V -= S.nuc[I][3] * ri;
            if (!closer(r, 1e-10)) {
                sums[e] -= f * dx; sums[NE + e] -= f * dy; sums[2 * NE + e] -= f * dz; sums[3 * NE + e] -= l;
            }
        }
        __syncwarp();
    }
    double kin = 0;
#pragma unroll 1
    for (int e = lane; e < NE; e += 32) {
        const double jx = sums[e], jy = sums[NE + e], jz = sums[2 * NE + e], lu = sums[3 * NE + e];
        const double gx = der[e], gy = der[NE + e], gz = der[2 * NE + e];
        const double ax = S.qa * jx, ay = S.qa * jy, az = S.qa * jz;
        const double lj = S.quirk_lap ? lu + sums[4 * NE + e] : lu + jx * jx + jy * jy + jz * jz;
        const double lp = der[3 * NE + e] + 2.0 * (gx * ax + gy * ay + gz * az) + lj;
        kin += lp;
        if (out_grad) {                         // internal order; the host permutes to the caller's
            double* o = out_grad + ((size_t)w * NE + e) * 3;
            o[0] = gx + ax;
            o[1] = gy + ay;
            o[2] = gz + az;
        }
        if (out_lap) out_lap[(size_t)w * NE + e] = lp;
    }
    V += -0.5 * kin;
    u = wsum(u);
    V = wsum(V);
    const double e_l = V + S.v_nn;
    if (lane == 0) {
        int fl = 0;
        if (!ok) fl |= FLAG_SINGULAR;
        if (!isfinite(e_l)) fl |= FLAG_NONFINITE;
        if (fl) atomicOr(flags, fl);
        if (write_state) { glog[w] = logdet + u; gsign[w] = sg; gel[w] = e_l; }
    }
    return e_l;
}

// ---------------------------------------------------------------------------
// Float-float refresh of FP32 walkers, both spin sectors at once: the sectors have
// the same size and the same walk over the basis, so sector 0 and sector 1 are the
// two components of packed instructions (ff2), lane q holding electrons q and
// NUP + q.  Orbital values and the inversion keep the rounding of the one-sector
// form, component by component, so the inverses the sweeps start from are its bits;
// pairs are evaluated once, two per lane and instruction.  The kernel is an
// instruction stream of several loops, each longer than the instruction cache likes
// to hold beside the others: the block's warps (one block per SM) walk the phases
// together, so that one loop is in use at a time (16 384 walkers: 2.16 ms, 2.69 ms in
// four-warp blocks that do not wait for each other, 3.15 ms for one sector at a time).
// The FP32 pipe bounds it, 74 % busy; of the cycles 30 % are orbital values, 25 % the
// inversion, 29 % derivatives, 16 % pairs and nuclei.  1.98 ms with the derivatives as
// (electron pair, third) tasks.
// ---------------------------------------------------------------------------
struct PairTabHead {                // sizes and scalars; the arrays follow in the block's shared memory
    int n_ao, n_sh, n_third, quirk_lap;
    ff qa, v_nn;
    ff b_ee[2], a_ee[2];
};
// Device table: head, nuclei [NNUC] (x, y, z, Z, enA, enB as ff), shells in AO order,
// the same in thirds (deal_thirds), primitives (exponent, coefficient) and (c a,
// c a^2) of each, an sp shell's p coefficients beside them, then the
// coefficients [n_ao][NM] of both sectors as (hi, hi', lo, lo').
template <int NNUC, int NM>
struct PairTab {
    PairTabHead head;
    ff nuc[NNUC][6];
    int sh[WMAX_AO], third[WMAX_THIRD];
    float4 prim[WMAX_PRIM], primd[WMAX_PRIM];      // s or lone p
    float4 prim_p[WMAX_PRIM], primd_p[WMAX_PRIM];  // p of an sp shell
    float4 C[WMAX_AO][NM];
    __host__ __device__ static size_t bytes(int n_ao) { return offsetof(PairTab, C) + sizeof(float4) * NM * (size_t)n_ao; }
    __device__ static size_t used(const PairTab* t) { return bytes(t->head.n_ao); }
};

template <int NNUC, int NM>
static void fill_pairtab(const SysW<ff>& w, PairTab<NNUC, NM>& S) {
    std::memset(static_cast<void*>(&S), 0, sizeof(S));
    S.head.n_ao = w.n_ao;
    const ShellList<ff> L(w);
    S.head.n_sh = (int)L.desc.size();
    S.head.n_third = deal_thirds(L.desc, S.third);
    S.head.quirk_lap = w.quirk_lap;
    S.head.qa = w.qa;
    S.head.v_nn = w.v_nn;
    for (int c = 0; c < 2; ++c) { S.head.b_ee[c] = w.b_ee[c]; S.head.a_ee[c] = w.a_ee[c]; }
    for (int I = 0; I < NNUC; ++I) {
        const ff v[6] = {w.nuc[I][0], w.nuc[I][1], w.nuc[I][2], w.Z[I], w.enA[I], w.enB[I]};
        for (int c = 0; c < 6; ++c) S.nuc[I][c] = v[c];
    }
    for (int g = 0; g < S.head.n_sh; ++g) S.sh[g] = L.desc[g];
    auto two = [](ff a, ff b) { return make_float4(a.hi, a.lo, b.hi, b.lo); };
    for (size_t p = 0; p < L.al.size(); ++p) {
        const double al = (double)L.al[p];
        for (int k = 0; k < 2; ++k) {
            const ff c = k ? L.cp[p] : L.c[p];
            (k ? S.prim_p : S.prim)[p] = two(L.al[p], c);
            (k ? S.primd_p : S.primd)[p] = two(ff((double)c * al), ff((double)c * al * al));
        }
    }
    for (int a = 0; a < w.n_ao; ++a)
        for (int k = 0; k < NM; ++k) {
            const ff c0 = w.C[0][a][k], c1 = w.C[1][a][k];
            S.C[a][k] = make_float4(c0.hi, c1.hi, c0.lo, c1.lo);
        }
}

__device__ __forceinline__ ff2 load_ff2(const float4* p) {
    const float4 v = *p;
    return ff2(F2(v.x, v.y), F2(v.z, v.w));
}
__device__ __forceinline__ void store_ff2(float4* p, ff2 v) {
    float4 t;
    v.hi.get(t.x, t.y);
    v.lo.get(t.z, t.w);
    *p = t;
}

// Shared float4 of a warp: the sectors' rows (row q at q NM), then, over the same
// storage, the inverse's columns, then positions [3][NE] and sums [5][NE] of the pair
// pass as ff; after it the derivative sums [round][4][lane].
template <int NE, int NM>
__host__ __device__ constexpr int pair_rows() { return NM * NM > (8 * NE + 1) / 2 ? NM * NM : (8 * NE + 1) / 2; }
template <int NE, int NM>
__host__ __device__ constexpr int pair_scratch() {
    return pair_rows<NE, NM>() + 2 * 4 * 32;
}

// Pade pair terms of two pairs at separations (dx, dy, dz): u = a r / (1 + b r),
// u'/r, u'' + 2u'/r, 1/r (0 at r = 0) and the distances' leading parts.
__device__ __forceinline__ void pair_terms(ff2 dx, ff2 dy, ff2 dz, ff2 a, ff2 b, ff2& u, ff2& f, ff2& l, ff2& ri,
                                           float (&d)[2]) {
    const ff2 r2 = dx * dx + dy * dy + dz * dz;
    float h0, h1;
    r2.hi.get(h0, h1);
    if (!(h0 > 0.0f && h1 > 0.0f)) {
        // 1/r = 0 at a vanishing distance (and NaN stays NaN through r^2)
        const ff2 s = ff2_frsqrt(ff2(F2(h0 > 0.0f ? h0 : 1.0f, h1 > 0.0f ? h1 : 1.0f), r2.lo));
        const F2 m(h0 > 0.0f ? 1.0f : 0.0f, h1 > 0.0f ? 1.0f : 0.0f);
        ri = ff2(mul2(s.hi, m), mul2(s.lo, m));
    } else {
        ri = ff2_frsqrt(r2);
    }
    const ff2 r = r2 * ri;
    const ff2 inv = ff2_frcp(ff2(1.0f) + b * r), ai = a * inv, up = ai * inv;
    u = ai * r;
    f = up * ri;
    // 2 (u'/r - a b inv^3)
    l = f - up * (b * inv);
    l = ff2(add2(l.hi, l.hi), add2(l.lo, l.lo));
    r.hi.get(d[0], d[1]);
}

template <int NE, int NUP, int NNUC>
__device__ __forceinline__ double kw_refresh_walker(const PairTab<NNUC, NUP>& S, float4* scr,
                                                    const float* __restrict__ gpos, float* __restrict__ gdinv,
                                                    double* __restrict__ glog, int* __restrict__ gsign,
                                                    double* __restrict__ gel, int w, bool act, int Wcap,
                                                    int write_state, int* flags) {
    static_assert(NE == 2 * NUP && NUP <= 32, "equal sectors, an electron of each per lane");
    constexpr int NM = NUP;
    const int lane = threadIdx.x & 31;
    const int q = min(lane, NM - 1);                        // spare lanes repeat the last electron
    // coordinate c of electron pair e
    auto coord = [&](int e, int c) {
        return ff2(F2(gpos[(size_t)(3 * e + c) * Wcap + w], gpos[(size_t)(3 * (NUP + e) + c) * Wcap + w]), F2(0.0f));
    };
    // orbital values of the lane's electrons, row q of both matrices
    __syncthreads();
    {
        const ff2 x = coord(q, 0), y = coord(q, 1), z = coord(q, 2);
        ff2 v[NM];
#pragma unroll
        for (int k = 0; k < NM; ++k) v[k] = ff2(0.0f);
        for (int g = 0; g < S.head.n_sh; ++g) {
            const int d = S.sh[g];
            const int I = shell_nuc(d), np = shell_np(d), p0 = shell_p0(d), a0 = shell_a0(d);
            const int ns = (d & SHELL_S) ? 1 : 0, na = ns + ((d & SHELL_P) ? 3 : 0);
            const bool sp = na == 4;
            const ff2 dx = x - ff2(S.nuc[I][0]), dy = y - ff2(S.nuc[I][1]), dz = z - ff2(S.nuc[I][2]);
            const ff2 r2 = dx * dx + dy * dy + dz * dz;
            ff2 s0(0.0f), s1(0.0f);
            for (int p = p0; p < p0 + np; ++p) {
                const float4 t = S.prim[p];
                const ff2 e = ff2_fexp(ff2(ff(-t.x, -t.y)) * r2);
                s0 += ff2(ff(t.z, t.w)) * e;
                if (sp) {
                    const float4 u = S.prim_p[p];
                    s1 += ff2(ff(u.z, u.w)) * e;
                }
            }
            if (!sp) s1 = s0;
#pragma unroll 1
            for (int m = 0; m < na; ++m) {
                const int c3 = m - ns;
                const ff2 chi = c3 < 0 ? s0 : (c3 == 0 ? dx : (c3 == 1 ? dy : dz)) * s1;
                const F2 nh = neg2(chi.hi), nl = neg2(chi.lo);
                const float4* c = S.C[a0 + m];
                // ff_fma_lazy(v[k], c[k], chi) with the error term carried negated
#pragma unroll
                for (int k = 0; k < NM; ++k) {
                    const ff2 ck = load_ff2(c + k);
                    const F2 t = mul2(ck.hi, chi.hi);
                    F2 ne = fma2(ck.hi, nh, t);
                    ne = fma2(ck.hi, nl, ne);
                    ne = fma2(ck.lo, nh, ne);
                    const ff2 u = ff2_two_sum(v[k].hi, t);
                    v[k] = ff2(u.hi, add2(v[k].lo, sub2(u.lo, ne)));
                }
            }
        }
        if (lane < NM) {
#pragma unroll
            for (int k = 0; k < NM; ++k) store_ff2(scr + lane * NM + k, ff2_norm(v[k]));
        }
    }
    __syncwarp();
    // Gauss-Jordan of both matrices in place (kw_measure_walker's steps): the pivot
    // column goes through the warp's shared memory, negated, which also lets a lane
    // per row search the pivots
    __syncthreads();
    ff2 A[NM];
#pragma unroll
    for (int i = 0; i < NM; ++i) {
        A[i] = load_ff2(scr + i * NM + q);
        if (lane >= NM) A[i] = ff2(0.0f);
    }
    __syncwarp();
    ff pm0 = ff(1.0f), pm1 = ff(1.0f);
    int pe = 0, sg = 1, src0 = lane, src1 = lane;
    bool ok = true;
#pragma unroll 1
    for (int k = 0; k < NM; ++k) {
        if (lane == k) {
#pragma unroll
            for (int i = 0; i < NM; ++i) {
                float4 t;
                A[i].hi.get(t.x, t.y);
                A[i].lo.get(t.z, t.w);
                scr[i] = make_float4(-t.x, -t.y, -t.z, -t.w);
            }
        }
        __syncwarp();
        // the largest |D[i][k]| over the rows not yet pivoted; the first of equal ones
        unsigned k0 = 0, k1 = 0;
        const bool cand = lane < NM - k;
        if (cand) {
            const float4 t = scr[lane];
            k0 = __float_as_uint(t.x) & 0x7fffffffu;
            k1 = __float_as_uint(t.y) & 0x7fffffffu;
        }
        const unsigned m0 = __reduce_max_sync(0xffffffffu, k0), m1 = __reduce_max_sync(0xffffffffu, k1);
        const int p0 = __ffs(__ballot_sync(0xffffffffu, cand && k0 == m0)) - 1;
        const int p1 = __ffs(__ballot_sync(0xffffffffu, cand && k1 == m1)) - 1;
        if (p0 != 0 || p1 != 0) {
            // the same rows on every lane
#pragma unroll
            for (int r = 1; r < NM; ++r)
                if (p0 == r || p1 == r) {
                    float a0, a1, b0, b1, c0, c1, d0, d1;
                    A[0].hi.get(a0, a1); A[0].lo.get(b0, b1);
                    A[r].hi.get(c0, c1); A[r].lo.get(d0, d1);
                    if (p0 == r) { float t = a0; a0 = c0; c0 = t; t = b0; b0 = d0; d0 = t; }
                    if (p1 == r) { float t = a1; a1 = c1; c1 = t; t = b1; b1 = d1; d1 = t; }
                    A[0] = ff2(F2(a0, a1), F2(b0, b1));
                    A[r] = ff2(F2(c0, c1), F2(d0, d1));
                }
            if (lane == 0) {
                float4 t = scr[0], u = scr[p0];
                scr[p0] = make_float4(t.x, u.y, t.z, u.w);
                t.x = u.x; t.z = u.z;
                scr[0] = t;
                t = scr[0]; u = scr[p1];
                scr[p1] = make_float4(u.x, t.y, u.z, t.w);
                t = scr[0];
                if (p1 != 0) { t.y = u.y; t.w = u.w; }
                scr[0] = t;
            }
            __syncwarp();
        }
        if (p0 != 0) sg = -sg;
        if (p1 != 0) sg = -sg;
        const int q0 = k + p0, q1 = k + p1;
        src0 = src0 == k ? q0 : (src0 == q0 ? k : src0);
        src1 = src1 == k ? q1 : (src1 == q1 ? k : src1);
        const float4 pv = scr[0];
        ff v0(-pv.x, -pv.z), v1(-pv.y, -pv.w);
        if (!(v0 != ff(0))) { ok = false; v0 = ff(1); }
        if (!(v1 != ff(0))) { ok = false; v1 = ff(1); }
        if (v0.hi < 0.0f) sg = -sg;
        if (v1.hi < 0.0f) sg = -sg;
        pm0 = pm0 * fabs(v0);                              // |det| as rescaled products
        pm1 = pm1 * fabs(v1);
        ff_rescale(pm0, pe);
        ff_rescale(pm1, pe);
        const ff2 ip(ff(1) / v0, ff(1) / v1);
        const ff2 scaled = A[0] * ip, own = ff2(1.0f) + ip;
        const bool me = lane == k;
        const ff2 t = me ? own : scaled, first = me ? ip : scaled;
        const F2 nth = neg2(t.hi), ntl = neg2(t.lo);
        // rows 1.. lose f x row k and move one register down; row k goes last
#pragma unroll
        for (int i = 1; i < NM; ++i) {
            const ff2 f = load_ff2(scr + i);               // -f
            const F2 m = mul2(f.hi, t.hi);
            F2 ne = fma2(f.hi, nth, m);
            ne = fma2(f.hi, ntl, ne);
            ne = fma2(f.lo, nth, ne);
            const F2 h = sub2(m, ne), nl = add2(ne, sub2(h, m));   // -(f t), low part negated
            const ff2 s = ff2_two_sum(A[i].hi, h);
            A[i - 1] = ff2_fast_two_sum(s.hi, add2(s.lo, sub2(A[i].lo, nl)));
        }
        A[NM - 1] = first;
        __syncwarp();                                      // the column is read
    }
    // unscramble: lane j takes columns src(j); then A[k] = D^-1[k][lane]
#pragma unroll
    for (int i = 0; i < NM; ++i) {
        ff a, b;
        A[i].get(a, b);
        a = wshfl(a, src0);
        b = wshfl(b, src1);
        A[i] = ff2(a, b);
        if (act && write_state && lane < NM) {
            gdinv[((size_t)(i * NM + lane)) * Wcap + w] = (float)a;
            gdinv[((size_t)(NM * NM + i * NM + lane)) * Wcap + w] = (float)b;
        }
    }
    // grad ln D and lap D / D of the lane's electrons: sum_a c'_a (grad, lap) chi_a with
    // c'_a = sum_k C[a][k] D^-1[k][q].  s: grad = -2 R1 dr, lap = -6 R1 + 4 r^2 R2; a p
    // triplet takes its three c' as a vector c: grad = -2 R1 (c.dr) dr + R0 c,
    // lap = (c.dr)(-10 R1 + 4 r^2 R2).  The work is 3 NM (electron pair, third of the
    // shells) tasks in two rounds of 32 lanes, two thirds of the time of one round of NM
    // lanes over all shells: round 0 takes third 0 of every pair and third 1 of the first
    // R1, round 1 the rest.  The inverse's columns go through the warp's shared memory.
    __syncthreads();
    static_assert(3 * NM <= 64 && NM <= 32, "three tasks per electron pair in two rounds");
    constexpr int R1 = 32 - NM;
    if (lane < NM) {
#pragma unroll
        for (int k = 0; k < NM; ++k) store_ff2(scr + k * NM + lane, A[k]);
    }
    __syncwarp();
    float4* part = scr + pair_rows<NE, NM>();
#pragma unroll 1
    for (int round = 0; round < 2; ++round) {
        const int t3 = round == 0 ? (lane < NM ? 0 : 1) : (lane < NM - R1 ? 1 : 2);
        const int tq = min(round == 0 ? (lane < NM ? lane : lane - NM) : (lane < NM - R1 ? R1 + lane : lane - (NM - R1)), NM - 1);
        const ff2 x = coord(tq, 0), y = coord(tq, 1), z = coord(tq, 2);
#pragma unroll
        for (int k = 0; k < NM; ++k) A[k] = load_ff2(scr + k * NM + tq);
        ff2 gx(0.0f), gy(0.0f), gz(0.0f), ld(0.0f);
        for (int g = 0; g < S.head.n_third; ++g) {
            const int d = S.third[3 * g + t3];
            const int I = shell_nuc(d), np = shell_np(d), p0 = shell_p0(d), a0 = shell_a0(d);
            const int ns = (d & SHELL_S) ? 1 : 0, na = ns + ((d & SHELL_P) ? 3 : 0);
            const bool sp = na == 4;
            const ff2 dx = x - ff2(S.nuc[I][0]), dy = y - ff2(S.nuc[I][1]), dz = z - ff2(S.nuc[I][2]);
            const ff2 r2 = dx * dx + dy * dy + dz * dz;
            ff2 s0(0.0f), s1(0.0f), s2(0.0f), p_0(0.0f), p_1(0.0f), p_2(0.0f);
            for (int p = p0; p < p0 + np; ++p) {
                const float4 t = S.prim[p], u = S.primd[p];
                const ff2 e = ff2_fexp(ff2(ff(-t.x, -t.y)) * r2);
                ff2_fma_lazy(s0, ff2(ff(t.z, t.w)), e);
                ff2_fma_lazy(s1, ff2(ff(u.x, u.y)), e);
                ff2_fma_lazy(s2, ff2(ff(u.z, u.w)), e);
                if (sp) {
                    const float4 tp = S.prim_p[p], up = S.primd_p[p];
                    ff2_fma_lazy(p_0, ff2(ff(tp.z, tp.w)), e);
                    ff2_fma_lazy(p_1, ff2(ff(up.x, up.y)), e);
                    ff2_fma_lazy(p_2, ff2(ff(up.z, up.w)), e);
                }
            }
            const ff2 two(F2(-2.0f), F2(0.0f)), r4 = ff2(F2(4.0f), F2(0.0f)) * r2;
            s0 = ff2_norm(s0); s1 = ff2_norm(s1); s2 = ff2_norm(s2);
            // cd: c' of an s AO, then (c'.dr) of a p triplet; a triplet's radial parts
            // replace the s AO's once that is added
            ff2 cd(0.0f);
#pragma unroll 1
            for (int m = 0; m < na; ++m) {
                const float4* c = S.C[a0 + m];
                ff2 cw(0.0f);
#pragma unroll
                for (int k = 0; k < NM; ++k) ff2_fma_lazy(cw, load_ff2(c + k), A[k]);
                cw = ff2_norm(cw);
                const int c3 = m - ns;
                if (c3 < 0) {
                    cd = cw;
                } else {
                    if (c3 == 0 && sp) { s0 = ff2_norm(p_0); s1 = ff2_norm(p_1); s2 = ff2_norm(p_2); cd = ff2(0.0f); }
                    ff2_fma_lazy(cd, cw, c3 == 0 ? dx : (c3 == 1 ? dy : dz));
                    ff2 o = c3 == 0 ? gx : (c3 == 1 ? gy : gz);
                    ff2_fma_lazy(o, s0, cw);
                    if (c3 == 0) gx = o;
                    else if (c3 == 1) gy = o;
                    else gz = o;
                }
                if (c3 < 0 || c3 == 2) {
                    cd = ff2_norm(cd);
                    const ff2 t = two * s1 * cd;
                    ff2_fma_lazy(gx, t, dx); ff2_fma_lazy(gy, t, dy); ff2_fma_lazy(gz, t, dz);
                    ff2_fma_lazy(ld, cd, r4 * s2 - ff2(F2(c3 < 0 ? 6.0f : 10.0f), F2(0.0f)) * s1);
                }
            }
        }
        store_ff2(part + (4 * round + 0) * 32 + lane, ff2_norm(gx));
        store_ff2(part + (4 * round + 1) * 32 + lane, ff2_norm(gy));
        store_ff2(part + (4 * round + 2) * 32 + lane, ff2_norm(gz));
        store_ff2(part + (4 * round + 3) * 32 + lane, ff2_norm(ld));
    }
    // electron pairs, each once, two per lane: pair p joins electron i = p mod NE with
    // i + p / NE + 1 (mod NE), the last NE / 2 pairs i with i + NE / 2; 32 consecutive
    // pairs have distinct i and distinct j, so their sums need no atomics
    ff* pos = reinterpret_cast<ff*>(scr);
    ff* sums = pos + 3 * NE;
    __syncthreads();
    if (lane < NM) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int e = s * NUP + lane;
#pragma unroll
            for (int c = 0; c < 3; ++c) pos[c * NE + e] = ff(gpos[(size_t)(3 * e + c) * Wcap + w]);
#pragma unroll
            for (int c = 0; c < 5; ++c) sums[c * NE + e] = ff(0.0f);
        }
    }
    __syncwarp();
    ff2 u(0.0f), V(0.0f);
    constexpr int NPAIR = NE * (NE - 1) / 2, FULL = NE * ((NE - 1) / 2);
    static_assert(NE > 32 && NE % 2 == 0, "the pairs of one round hold distinct electrons");
    for (int r0 = 0; r0 < NPAIR; r0 += 64) {
        int i[2], j[2];
        bool on[2];
        float d0[2], d1[2], d2[2];
        ff pa[2], pb[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            on[s] = r0 + 32 * s + lane < NPAIR;
            const int p = on[s] ? r0 + 32 * s + lane : NPAIR - 1;
            i[s] = p < FULL ? p % NE : p - FULL;
            j[s] = p < FULL ? i[s] + p / NE + 1 : i[s] + NE / 2;
            if (j[s] >= NE) j[s] -= NE;
            d0[s] = pos[i[s]].hi; d1[s] = pos[NE + i[s]].hi; d2[s] = pos[2 * NE + i[s]].hi;
            const int c = (j[s] < NUP) == (i[s] < NUP) ? 1 : 0;
            pa[s] = S.head.a_ee[c]; pb[s] = S.head.b_ee[c];
        }
        // positions are floats: the differences are exact pairs
        const ff2 dx = ff2_two_sum(F2(d0[0], d0[1]), F2(-pos[j[0]].hi, -pos[j[1]].hi));
        const ff2 dy = ff2_two_sum(F2(d1[0], d1[1]), F2(-pos[NE + j[0]].hi, -pos[NE + j[1]].hi));
        const ff2 dz = ff2_two_sum(F2(d2[0], d2[1]), F2(-pos[2 * NE + j[0]].hi, -pos[2 * NE + j[1]].hi));
        ff2 uu, f, l, ri;
        float dd[2];
        pair_terms(dx, dy, dz, ff2(pa[0], pa[1]), ff2(pb[0], pb[1]), uu, f, l, ri, dd);
        const ff2 fx = f * dx, fy = f * dy, fz = f * dz;
        ff2 sq(0.0f);
        if (S.head.quirk_lap) {
            const ff2 up2 = f * f;
            sq = up2 * (dx * dx + dy * dy + dz * dz);
        }
        ff t[7][2];
        uu.get(t[0][0], t[0][1]); ri.get(t[1][0], t[1][1]);
        fx.get(t[2][0], t[2][1]); fy.get(t[3][0], t[3][1]); fz.get(t[4][0], t[4][1]);
        l.get(t[5][0], t[5][1]); sq.get(t[6][0], t[6][1]);
        u += ff2(on[0] ? t[0][0] : ff(0.0f), on[1] ? t[0][1] : ff(0.0f));
        V += ff2(on[0] ? t[1][0] : ff(0.0f), on[1] ? t[1][1] : ff(0.0f));
        const int nq = S.head.quirk_lap ? 5 : 4;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const bool use = on[s] && !(dd[s] < 1e-10f);
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int e = side ? j[s] : i[s];
                if (use) {
#pragma unroll
                    for (int c = 0; c < 5; ++c) {
                        if (c >= nq) break;
                        const ff v = t[2 + c][s];
                        const ff o = sums[c * NE + e], n = ff_two_sum(o.hi, side && c < 3 ? -v.hi : v.hi);
                        sums[c * NE + e] = ff(n.hi, __fadd_rn(o.lo, __fadd_rn(n.lo, side && c < 3 ? -v.lo : v.lo)));
                    }
                }
                __syncwarp();
            }
        }
    }
    // the lane's electrons: sums over electrons, then the nuclei
    auto both = [&](int c) {
        return ff2(ff_norm(sums[c * NE + q]), ff_norm(sums[c * NE + NUP + q]));
    };
    ff2 jx = both(0), jy = both(1), jz = both(2), lu = both(3);
    const ff2 gsq = both(4);
    const ff2 x = coord(q, 0), y = coord(q, 1), z = coord(q, 2);
    ff2 un(0.0f), Vn(0.0f);
    for (int I = 0; I < NNUC; ++I) {
        const ff2 dx = x - ff2(S.nuc[I][0]), dy = y - ff2(S.nuc[I][1]), dz = z - ff2(S.nuc[I][2]);
        ff2 uu, f, l, ri;
        float dd[2];
        pair_terms(dx, dy, dz, ff2(S.nuc[I][4]), ff2(S.nuc[I][5]), uu, f, l, ri, dd);
        un -= uu;
        Vn -= ff2(S.nuc[I][3]) * ri;
        if (dd[0] < 1e-10f || dd[1] < 1e-10f) {            // a coincident nucleus: no gradient terms
            ff a, b;
            f.get(a, b);
            f = ff2(dd[0] < 1e-10f ? ff(0.0f) : a, dd[1] < 1e-10f ? ff(0.0f) : b);
            l.get(a, b);
            l = ff2(dd[0] < 1e-10f ? ff(0.0f) : a, dd[1] < 1e-10f ? ff(0.0f) : b);
        }
        jx -= f * dx; jy -= f * dy; jz -= f * dz;
        lu -= l;
    }
    // the pair's thirds: its own lane's, and the lanes that took the other two
    ff2 dsum[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
        dsum[c] = load_ff2(part + c * 32 + q) + load_ff2(part + (q < R1 ? c * 32 + NM + q : (4 + c) * 32 + q - R1)) +
                  load_ff2(part + (4 + c) * 32 + NM - R1 + q);
    const ff2 gx = dsum[0], gy = dsum[1], gz = dsum[2], ld = dsum[3];
    const ff2 qa(S.head.qa);
    const ff2 lj = S.head.quirk_lap ? lu + gsq : lu + jx * jx + jy * jy + jz * jz;
    const ff2 lp = ld + ff2(2.0f) * (qa * (gx * jx + gy * jy + gz * jz)) + lj;
    const bool mine = lane < NM;
    ff a, b;
    u.get(a, b);
    ff us = a + b;
    un.get(a, b);
    us = mine ? us + (a + b) : us;
    V.get(a, b);
    ff Vs = a + b;
    Vn.get(a, b);
    Vs = mine ? Vs + (a + b) : Vs;
    lp.get(a, b);
    if (mine) Vs = Vs - ff(0.5f) * (a + b);
    us = wsum(us);
    Vs = wsum(Vs);
    const double e_l = (double)(Vs + S.head.v_nn);
    if (act && lane == 0) {
        int fl = 0;
        if (!ok) fl |= FLAG_SINGULAR;
        if (!isfinite(e_l)) fl |= FLAG_NONFINITE;
        if (fl) atomicOr(flags, fl);
        if (write_state) {
            glog[w] = d_log((double)(pm0 * pm1)) + (double)pe * 0.6931471805599453 + (double)us;
            gsign[w] = sg;
            gel[w] = e_l;
        }
    }
    return act ? e_l : 0.0;
}

// Compensated sum of the block's per-warp values (lane 0 of each warp) into
// partial[2 slot], partial[2 slot + 1]; ends with a block barrier.
template <int WPB>
__device__ __forceinline__ void warp_block_partial(double v, double* partial, int slot) {
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

template <int NE, int NUP, int NNUC, class TC, class TS, int WPB>
__global__ void __launch_bounds__(32 * WPB) kw_measure(const SysW<TC>* __restrict__ Sg, const TS* __restrict__ gpos,
                                                       TS* __restrict__ gdinv, double* __restrict__ glog,
                                                       int* __restrict__ gsign, double* __restrict__ gel, int W,
                                                       int Wcap, int write_state, double* __restrict__ out_grad,
                                                       double* __restrict__ out_lap, double* partial, int* flags) {
    constexpr int NM = NUP > NE - NUP ? NUP : NE - NUP;
    __shared__ SysW<TC> S;
    extern __shared__ __align__(16) unsigned char wsm[];
    load_sysw(&S, Sg);
    const int wib = threadIdx.x >> 5;
    const int w = blockIdx.x * WPB + wib;
    TC* Mrow = reinterpret_cast<TC*>(wsm) + (size_t)wib * NM * MRS;   // [NM rows][MRS]
    double e_l = kw_measure_walker<NE, NUP, NNUC, TC, TS>(S, Mrow, gpos, gdinv, glog, gsign, gel, w, w < W, Wcap,
                                                          write_state, out_grad, out_lap, flags);
    if (partial) warp_block_partial<WPB>(e_l, partial, blockIdx.x);
}

// FP64 evaluation, standalone and batched (state written, per-tile E_L partials; one
// block of WPB warps per WPB-walker tile).  Dynamic shared memory: the table's used
// part, then the warps' scratch.
template <int NE, int NUP, int NNUC, int WPB>
static size_t eval_smem(int n_ao) {
    return EvalTab<NNUC, NUP>::bytes(n_ao) + sizeof(double) * WPB * eval_scratch<NE, NUP>();
}
template <int NE, int NUP, int NNUC, int WPB>
__global__ void __launch_bounds__(32 * WPB) kw_eval(const EvalTab<NNUC, NUP>* __restrict__ Sg, const double* __restrict__ gpos,
                                                    double* __restrict__ gdinv, double* __restrict__ glog,
                                                    int* __restrict__ gsign, double* __restrict__ gel, int W, int Wcap,
                                                    int write_state, double* __restrict__ out_grad,
                                                    double* __restrict__ out_lap, double* partial, int* flags) {
    using TAB = EvalTab<NNUC, NUP>;
    extern __shared__ __align__(16) unsigned char wsm[];
    TAB& S = *reinterpret_cast<TAB*>(wsm);
    load_tab(&S, Sg);
    const int wib = threadIdx.x >> 5, w = blockIdx.x * WPB + wib;
    double* scr = reinterpret_cast<double*>(wsm + TAB::bytes(S.n_ao)) + (size_t)wib * eval_scratch<NE, NUP>();
    double e_l = 0.0;
    if (w < W)
        e_l = kw_eval_walker<NE, NUP, NNUC>(S, scr, gpos, gdinv, glog, gsign, gel, w, Wcap, write_state, out_grad, out_lap,
                                            flags);
    if (partial) warp_block_partial<WPB>(e_l, partial, blockIdx.x);
}
template <int NE, int NUP, int NNUC, int WPB>
__global__ void __launch_bounds__(32 * WPB) kwb_eval(const BatchTile* __restrict__ tiles, int ntiles,
                                                     const BatchRec* __restrict__ recs, double* tile_partial) {
    using TAB = EvalTab<NNUC, NUP>;
    extern __shared__ __align__(16) unsigned char wsm[];
    if ((int)blockIdx.x >= ntiles) return;
    const BatchTile tl = tiles[blockIdx.x];
    const BatchRec& R = recs[tl.rec];
    TAB& S = *reinterpret_cast<TAB*>(wsm);
    load_tab(&S, static_cast<const TAB*>(R.tab_d));
    const int wib = threadIdx.x >> 5, w = tl.w0 + wib;
    double* scr = reinterpret_cast<double*>(wsm + TAB::bytes(S.n_ao)) + (size_t)wib * eval_scratch<NE, NUP>();
    double e_l = 0.0;
    if (w < R.W)
        e_l = kw_eval_walker<NE, NUP, NNUC>(S, scr, (const double*)R.pos, (double*)R.dinv, R.logabs, R.sign, R.el, w, R.Wcap,
                                            1, nullptr, nullptr, R.flags);
    warp_block_partial<WPB>(e_l, tile_partial, blockIdx.x);
}

// Float-float refresh of FP32 walkers: standalone and batched.
template <int NE, int NUP, int NNUC, int WPB>
__global__ void __launch_bounds__(32 * WPB, 12 / WPB) kw_refresh(const PairTab<NNUC, NUP>* __restrict__ Sg,
                                                                const float* __restrict__ gpos,
                                                                float* __restrict__ gdinv, double* __restrict__ glog,
                                                                int* __restrict__ gsign, double* __restrict__ gel, int W,
                                                                int Wcap, int write_state, double* partial, int* flags) {
    extern __shared__ __align__(16) unsigned char wsm[];
    const int wib = threadIdx.x >> 5, w = blockIdx.x * WPB + wib;
    float4* scr = reinterpret_cast<float4*>(wsm) + (size_t)wib * pair_scratch<NE, NUP>();
    auto& S = *reinterpret_cast<PairTab<NNUC, NUP>*>(wsm + sizeof(float4) * WPB * pair_scratch<NE, NUP>());
    load_tab(&S, Sg);
    // warps past the last walker repeat it and store nothing
    const double e_l = kw_refresh_walker<NE, NUP, NNUC>(S, scr, gpos, gdinv, glog, gsign, gel, min(w, W - 1), w < W,
                                                        Wcap, write_state, flags);
    if (partial) warp_block_partial<WPB>(e_l, partial, blockIdx.x);
}
template <int NE, int NUP, int NNUC, int WPB>
__global__ void __launch_bounds__(32 * WPB, 12 / WPB) kwb_refresh(const BatchTile* __restrict__ tiles, int ntiles,
                                                                 const BatchRec* __restrict__ recs,
                                                                 double* tile_partial) {
    extern __shared__ __align__(16) unsigned char wsm[];
    if ((int)blockIdx.x >= ntiles) return;
    const int wib = threadIdx.x >> 5;
    float4* scr = reinterpret_cast<float4*>(wsm) + (size_t)wib * pair_scratch<NE, NUP>();
    auto& S = *reinterpret_cast<PairTab<NNUC, NUP>*>(wsm + sizeof(float4) * WPB * pair_scratch<NE, NUP>());
    const BatchTile tl = tiles[blockIdx.x];
    const BatchRec& R = recs[tl.rec];
    load_tab(&S, static_cast<const PairTab<NNUC, NUP>*>(R.tab_d));
    const int w = tl.w0 + wib;
    const double e_l = kw_refresh_walker<NE, NUP, NNUC>(S, scr, (const float*)R.pos, (float*)R.dinv, R.logabs, R.sign,
                                                        R.el, min(w, R.W - 1), w < R.W, R.Wcap, 1, R.flags);
    warp_block_partial<WPB>(e_l, tile_partial, blockIdx.x);
}

int launch_sum_partials(const double* partial, int nblk, int nrows, double* out, cudaStream_t st);

// Per-shape launchers for the warp kernels.
template <int NE, int NUP, int NNUC>
struct WarpShapeOps {
    static constexpr int NM = NUP > NE - NUP ? NUP : NE - NUP;
    static constexpr int WPB = 4;
    // Warps of a float-float refresh block, one block per SM (168 registers).
    static constexpr int RWPB = 12;
    // Batch tiles hold BTW walkers: BTW / WPB sweep blocks each, and one
    // refresh block of BTW warps.
    static constexpr int BTW = RWPB;
    // dynamic shared memory of a sweep block: the WPB warps' proposal rows
    template <class T, int MOVE>
    static constexpr size_t sweep_smem() { return sizeof(T) * WPB * (size_t)sweep_scratch_elems<NE, NUP, MOVE>(); }

    template <class T>
    static int table(const HostSys& hs, const SysW<T>** out) {
        // device copies of the table, cached per system and rebuilt when the
        // parameters or nuclei change (HostSys::version)
        const int slot = std::is_same<T, double>::value ? 0 : 1;
        if (!hs.dev_table[slot] || hs.dev_table_version[slot] != hs.version) {
            SysW<T>* h = new SysW<T>;
            if (!fill_sysw<T>(hs, NE, NUP, NNUC, *h)) { delete h; return 7; }
            if (!hs.dev_table[slot]) {
                if (cudaMalloc(&hs.dev_table[slot], sizeof(SysW<T>)) != cudaSuccess) { delete h; return 8; }
            }
            cudaError_t e = cudaMemcpy(hs.dev_table[slot], h, sizeof(SysW<T>), cudaMemcpyHostToDevice);
            delete h;
            if (e != cudaSuccess) return 2;
            hs.dev_table_version[slot] = hs.version;
        }
        *out = static_cast<const SysW<T>*>(hs.dev_table[slot]);
        return 0;
    }

    static int init(const HostSys& hs, DevWalkers& dw, uint64_t seed, cudaStream_t st) {
        const SysW<double>* S;
        int rc = table<double>(hs, &S);
        if (rc) return rc;
        int n = NE * dw.W, tpb = 256;
        if (dw.prec == 0) kw_init<double><<<(n + tpb - 1) / tpb, tpb, 0, st>>>(S, (double*)dw.pos, NE, dw.W, dw.Wcap, seed);
        else kw_init<float><<<(n + tpb - 1) / tpb, tpb, 0, st>>>(S, (float*)dw.pos, NE, dw.W, dw.Wcap, seed);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    template <class TC, class TS>
    static int measure_w(const HostSys& hs, DevWalkers& dw, bool ws, const MeasureOut& out, cudaStream_t st) {
        const SysW<TC>* S;
        int rc = table<TC>(hs, &S);
        if (rc) return rc;
        int nb = (dw.W + WPB - 1) / WPB;
        size_t smem = sizeof(TC) * WPB * NM * MRS;
        auto kern = kw_measure<NE, NUP, NNUC, TC, TS, WPB>;
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
                return 2;
            attr = true;
        }
        double* partial = (ws && dw.partial && dw.partial_cap >= 2 * nb + 1) ? dw.partial : nullptr;
        kern<<<nb, 32 * WPB, smem, st>>>(S, (const TS*)dw.pos, (TS*)dw.dinv, dw.logabs, dw.sign, dw.el, dw.W, dw.Wcap,
                                        ws ? 1 : 0, out.grad, out.lap, partial, dw.flags);
        ++g_launch_count;
        if (cudaGetLastError() != cudaSuccess) return 2;
        if (!partial) return 0;
        return launch_sum_partials(partial, nb, 1, dw.partial + dw.partial_cap - 1, st);
    }

    // The kernels' own tables, filled from a SysW of their precision: device copies
    // cached like the others.
    using PT = PairTab<NNUC, NUP>;
    using GT = GaussTab<NNUC, NM>;
    using ET = EvalTab<NNUC, NUP>;
    template <class T, class TAB>
    static int own_table(const HostSys& hs, int slot, void (*fill)(const SysW<T>&, TAB&), const TAB** out) {
        if (!hs.dev_table[slot] || hs.dev_table_version[slot] != hs.version) {
            SysW<T>* w = new SysW<T>;
            TAB* h = new TAB;
            const bool good = fill_sysw<T>(hs, NE, NUP, NNUC, *w);
            if (good) fill(*w, *h);
            int rc = good ? 0 : 7;
            if (!rc && !hs.dev_table[slot] && cudaMalloc(&hs.dev_table[slot], sizeof(TAB)) != cudaSuccess) rc = 8;
            if (!rc && cudaMemcpy(hs.dev_table[slot], h, sizeof(TAB), cudaMemcpyHostToDevice) != cudaSuccess) rc = 2;
            delete w;
            delete h;
            if (rc) return rc;
            hs.dev_table_version[slot] = hs.version;
        }
        *out = static_cast<const TAB*>(hs.dev_table[slot]);
        return 0;
    }
    static int pair_table(const HostSys& hs, const PT** out) { return own_table<ff, PT>(hs, 2, fill_pairtab<NNUC, NUP>, out); }
    static int gauss_table(const HostSys& hs, const GT** out) { return own_table<float, GT>(hs, 4, fill_gausstab<NNUC, NM>, out); }
    static int eval_table(const HostSys& hs, const ET** out) { return own_table<double, ET>(hs, 5, fill_evaltab<NNUC, NUP>, out); }

    // FP64 evaluation.
    static int eval(const HostSys& hs, DevWalkers& dw, bool ws, const MeasureOut& out, cudaStream_t st) {
        const ET* S;
        const int rc = eval_table(hs, &S);
        if (rc) return rc;
        const int nb = (dw.W + WPB - 1) / WPB;
        auto kern = kw_eval<NE, NUP, NNUC, WPB>;
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)eval_smem<NE, NUP, NNUC, WPB>(WMAX_AO)) != cudaSuccess)
                return 2;
            attr = true;
        }
        double* partial = (ws && dw.partial && dw.partial_cap >= 2 * nb + 1) ? dw.partial : nullptr;
        kern<<<nb, 32 * WPB, eval_smem<NE, NUP, NNUC, WPB>(hs.n_ao), st>>>(
            S, (const double*)dw.pos, (double*)dw.dinv, dw.logabs, dw.sign, dw.el, dw.W, dw.Wcap, ws ? 1 : 0, out.grad, out.lap,
            partial, dw.flags);
        ++g_launch_count;
        if (cudaGetLastError() != cudaSuccess) return 2;
        if (!partial) return 0;
        return launch_sum_partials(partial, nb, 1, dw.partial + dw.partial_cap - 1, st);
    }

    // FP32 Gaussian sweeps.
    static int gauss(const HostSys& hs, DevWalkers& dw, int n, uint64_t s0, double step, uint64_t seed, cudaStream_t st) {
        const GT* S;
        const int rc = gauss_table(hs, &S);
        if (rc) return rc;
        auto kern = kw_gauss<NE, NUP, NNUC, WPB, GT>;
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)gauss_smem<NE, NUP, NNUC, WPB>(WMAX_AO)) != cudaSuccess)
                return 2;
            attr = true;
        }
        const SweepArgs<float> a{(float*)dw.pos, (float*)dw.dinv, dw.sign, dw.acc, dw.flags, s0, seed,
                                 (float)step, 0.0f, 0.0f, dw.W, dw.Wcap, n, dw.fixed_node};
        kern<<<(dw.W + WPB - 1) / WPB, 32 * WPB, gauss_smem<NE, NUP, NNUC, WPB>(hs.n_ao), st>>>(S, a);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }
    static int batch_gauss(const BatchClass& bc, const BatchCtl* ctl, cudaStream_t st, int* occ) {
        auto kern = kwb_gauss<NE, NUP, NNUC, WPB, BTW, GT>;
        const size_t smem = gauss_smem<NE, NUP, NNUC, WPB>(bc.n_ao);
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)gauss_smem<NE, NUP, NNUC, WPB>(WMAX_AO)) != cudaSuccess)
                return 2;
            attr = true;
        }
        if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, 32 * WPB, smem) == cudaSuccess ? 0 : 2;
        if (bc.ntiles == 0) return 0;
        kern<<<bc.ntiles * (BTW / WPB), 32 * WPB, smem, st>>>(bc.tiles, bc.ntiles, bc.recs, ctl);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    static size_t refresh_smem(int n_ao) { return sizeof(float4) * RWPB * pair_scratch<NE, NUP>() + PT::bytes(n_ao); }

    static int refresh(const HostSys& hs, DevWalkers& dw, bool ws, cudaStream_t st) {
        const PT* S;
        const int rc = pair_table(hs, &S);
        if (rc) return rc;
        const int nb = (dw.W + RWPB - 1) / RWPB;
        auto kern = kw_refresh<NE, NUP, NNUC, RWPB>;
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)refresh_smem(WMAX_AO)) != cudaSuccess)
                return 2;
            attr = true;
        }
        double* partial = (ws && dw.partial && dw.partial_cap >= 2 * nb + 1) ? dw.partial : nullptr;
        kern<<<nb, 32 * RWPB, refresh_smem(hs.n_ao), st>>>(S, (const float*)dw.pos, (float*)dw.dinv, dw.logabs, dw.sign, dw.el,
                                                          dw.W, dw.Wcap, ws ? 1 : 0, partial, dw.flags);
        ++g_launch_count;
        if (cudaGetLastError() != cudaSuccess) return 2;
        if (!partial) return 0;
        return launch_sum_partials(partial, nb, 1, dw.partial + dw.partial_cap - 1, st);
    }

    static int measure(const HostSys& hs, DevWalkers& dw, int cp, bool ws, const MeasureOut& out, cudaStream_t st) {
        if (out.O || out.fhf || out.omega) return 7;
        // FP32 walkers refresh in float-float arithmetic on the FP32 pipe
        if (cp == 0 && dw.prec == 0) return eval(hs, dw, ws, out, st);
        if (cp == 0) return out.grad || out.lap ? 7 : refresh(hs, dw, ws, st);
        if (dw.prec == 1) return measure_w<float, float>(hs, dw, ws, out, st);
        return 7;
    }

    template <class T, int MOVE>
    static int sweep_t(const HostSys& hs, DevWalkers& dw, int n, uint64_t s0, double step, double tau, double maxd,
                       uint64_t seed, cudaStream_t st) {
        const SysW<T>* S;
        int rc = table<T>(hs, &S);
        if (rc) return rc;
        int nb = (dw.W + WPB - 1) / WPB;
        auto kern = kw_sweep<NE, NUP, NNUC, T, MOVE, WPB>;
        const size_t smem = sweep_smem<T, MOVE>();
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
                return 2;
            attr = true;
        }
        kern<<<nb, 32 * WPB, smem, st>>>(S, (T*)dw.pos, (T*)dw.dinv, dw.sign, dw.W, dw.Wcap, n, s0, (T)step, (T)tau,
                                         (T)maxd, seed, dw.acc, dw.flags, dw.fixed_node);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    // ---- batched launches ---------------------------------------------------
    // tab_s: the sweep table (walker precision); tab_d: the refresh table
    // (FP64 for FP64 walkers, float-float for FP32 walkers).
    static int batch_tables(const HostSys& hs, int prec, BatchRec& r) {
        r.ktab = nullptr;
        if (prec == 0) {
            const SysW<double>* d;
            const ET* e;
            int rc = table<double>(hs, &d);
            if (!rc) rc = eval_table(hs, &e);
            if (rc) return rc;
            r.tab_d = e;
            r.tab_s = d;
            return 0;
        }
        const PT* m;
        const SysW<float>* f;
        int rc = pair_table(hs, &m);
        const GT* g;
        if (!rc) rc = table<float>(hs, &f);
        if (!rc) rc = gauss_table(hs, &g);
        if (rc) return rc;
        r.tab_d = m;
        r.tab_s = f;
        r.tab_g = g;
        return 0;
    }

    template <class T, int MOVE>
    static int batch_sweep_t(const BatchClass& bc, const BatchCtl* ctl, cudaStream_t st, int* occ) {
        auto kern = kwb_sweep<NE, NUP, NNUC, T, MOVE, WPB, BTW>;
        const size_t smem = sweep_smem<T, MOVE>();
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
                return 2;
            attr = true;
        }
        if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, 32 * WPB, smem) == cudaSuccess ? 0 : 2;
        if (bc.ntiles == 0) return 0;
        kern<<<bc.ntiles * (BTW / WPB), 32 * WPB, smem, st>>>(bc.tiles, bc.ntiles, bc.recs, ctl);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    static int batch_sweep(const BatchClass& bc, int mk, const BatchCtl* ctl, cudaStream_t st, int* occ = nullptr) {
        if (mk == MOVE_ONE_GAUSS)
            return bc.prec == 0 ? batch_sweep_t<double, MOVE_ONE_GAUSS>(bc, ctl, st, occ)
                                : batch_gauss(bc, ctl, st, occ);
        if (mk == MOVE_ONE_DRIFT)
            return bc.prec == 0 ? batch_sweep_t<double, MOVE_ONE_DRIFT>(bc, ctl, st, occ)
                                : batch_sweep_t<float, MOVE_ONE_DRIFT>(bc, ctl, st, occ);
        return 7;
    }

    static int batch_eval(const BatchClass& bc, cudaStream_t st, int* occ) {
        auto kern = kwb_eval<NE, NUP, NNUC, BTW>;
        const size_t smem = eval_smem<NE, NUP, NNUC, BTW>(bc.n_ao);
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)eval_smem<NE, NUP, NNUC, BTW>(WMAX_AO)) != cudaSuccess)
                return 2;
            attr = true;
        }
        if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, 32 * BTW, smem) == cudaSuccess ? 0 : 2;
        if (bc.ntiles == 0) return 0;
        kern<<<bc.ntiles, 32 * BTW, smem, st>>>(bc.tiles, bc.ntiles, bc.recs, bc.tile_partial);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    static int batch_measure(const BatchClass& bc, cudaStream_t st, int* occ = nullptr) {
        if (bc.prec == 0) return batch_eval(bc, st, occ);
        auto kern = kwb_refresh<NE, NUP, NNUC, RWPB>;
        const size_t smem = refresh_smem(WMAX_AO);
        static bool attr = false;
        if (!attr) {
            if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 2;
            attr = true;
        }
        if (occ) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, 32 * RWPB, smem) == cudaSuccess ? 0 : 2;
        if (bc.ntiles == 0) return 0;
        kern<<<bc.ntiles, 32 * RWPB, refresh_smem(bc.n_ao), st>>>(bc.tiles, bc.ntiles, bc.recs, bc.tile_partial);
        ++g_launch_count;
        return cudaGetLastError() == cudaSuccess ? 0 : 2;
    }

    static int sweep(const HostSys& hs, DevWalkers& dw, int mk, int n, uint64_t s0, double step, double tau,
                     double maxd, uint64_t seed, cudaStream_t st) {
        if (mk == MOVE_ONE_GAUSS)
            return dw.prec == 0 ? sweep_t<double, MOVE_ONE_GAUSS>(hs, dw, n, s0, step, tau, maxd, seed, st)
                                : gauss(hs, dw, n, s0, step, seed, st);
        if (mk == MOVE_ONE_DRIFT)
            return dw.prec == 0 ? sweep_t<double, MOVE_ONE_DRIFT>(hs, dw, n, s0, step, tau, maxd, seed, st)
                                : sweep_t<float, MOVE_ONE_DRIFT>(hs, dw, n, s0, step, tau, maxd, seed, st);
        return 7;   // all-electron moves are not compiled for this shape
    }
};

}  // namespace qmc
