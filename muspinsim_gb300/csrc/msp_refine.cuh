// Device code shared by the per-snapshot kernels (msp_snap.cu, msp_snap64.cu):
// shared-memory layout, Hamiltonian assembly, the FP32 eigenvectors of the
// first stage and their double-word refinement.
#pragma once

#include "msp_internal.cuh"
#include "msp_cluster.cuh"
#include "msp_dw.cuh"
#include "msp_jacobi.cuh"
#include "msp_rho.cuh"

#include <math_constants.h>

namespace msp {

static_assert(sizeof(JRot<float>) == 16 && sizeof(JRot<double>) == 32, "JRot layout");

// ------------------------------------------------------------------ smem layout

struct SnapLayout {
    size_t H, U, rot, dia, red, tab, diag;     // Jacobi work
    size_t lam, acc, rank;                     // eigenvalues, reductions, sort
    size_t Hh, Hl, Yl, SR, corr, rd, lamf, rk, ord, cst, scal, rn, cn, yn;  // refinement (MIXED)
    size_t fac, facf, B2;                      // general path
    size_t total;
};

__host__ __device__ inline size_t lay_take(size_t &off, size_t bytes) {
    off = (off + 15) & ~size_t(15);
    const size_t o = off;
    off += bytes;
    return o;
}

// Byte offsets of every shared-memory buffer of a snapshot kernel.  The
// same function sizes the launch (host) and carves the buffers (device).
__host__ __device__ inline SnapLayout snap_layout(int n, int esize, bool refine, bool rho,
                                                  int fac_len, int nwarps) {
    SnapLayout L;
    const size_t m = (size_t)(n + (n & 1));
    const size_t mm = m * (m + 1);  // leading dimension m + 1 (odd): no bank conflicts
    // the two Jacobi buffers hold either a matrix with row stride m + 1 or
    // the eigenvector planes with column stride jacobi_ldu(m)
    const size_t mj = (size_t)jacobi_buffer((int)m);
    size_t off = 0;
    L.H = lay_take(off, mj * 2 * esize);
    L.U = lay_take(off, mj * 2 * esize);
    L.rot = lay_take(off, 2 * (m / 2) * (esize == 4 ? 16 : 32));  // sizeof(JRot<T>)
    L.dia = lay_take(off, 2 * m * esize);
    L.red = lay_take(off, 2 * (size_t)nwarps * esize);
    L.tab = lay_take(off, (m / 2) * (m / 2 + 1) / 2 * 8);
    L.diag = lay_take(off, m * esize);
    L.lam = lay_take(off, m * 8);
    L.acc = lay_take(off, 2 * 8);
    L.rank = lay_take(off, m * 4);
    L.Hh = L.Hl = L.Yl = L.SR = L.corr = L.rd = L.lamf = 0;
    L.rk = L.ord = L.cst = L.scal = L.rn = L.cn = L.yn = 0;
    if (refine) {
        L.Hh = lay_take(off, mm * 8);
        L.Hl = lay_take(off, mm * 8);
        L.Yl = lay_take(off, mm * 8);
        L.SR = lay_take(off, mm * 8);
        L.corr = lay_take(off, m * 4);
        L.rd = lay_take(off, m * 8);
        L.lamf = lay_take(off, m * 4);
        L.rk = lay_take(off, m * 4);
        L.ord = lay_take(off, m * 4);
        L.cst = lay_take(off, m * 4);
        L.scal = lay_take(off, 4 * 4);
        L.rn = lay_take(off, m * 4);
        L.cn = lay_take(off, m * 4);
        L.yn = lay_take(off, m * 4);
    }
    L.fac = L.facf = L.B2 = 0;
    if (rho) {
        L.fac = lay_take(off, (size_t)fac_len * 16);
        if (refine) L.facf = lay_take(off, (size_t)fac_len * 8);
        // MIXED: the second basis buffer reuses Hh (free after refinement)
        L.B2 = refine ? L.Hh : lay_take(off, mm * 2 * esize);
    }
    L.total = (off + 15) & ~size_t(15);
    return L;
}

static inline int jacobi_threads(int m) {
    if (m <= 8) return 32;
    if (m <= 16) return 64;
    if (m <= 32) return 128;
    return 256;
}

template <typename T>
struct SnapSmem {
    JacobiWork<T> w;
    double *lam, *acc;  // FP64 path: eigenvalues
    float2 *lw;         // MIXED: eigenvalues as double-words (msp_dw.cuh), over lam
    int *rank;
    cx<float> *Hh, *Hl, *Yl, *SR;
    float2 *gd;         // MIXED: x_i^H x_i - 1 of the refinement step (double-word)
    float *corr, *lamf;
    int *rk, *ord, *cst, *scal;  // refinement clusters
    float *rn, *cn, *yn;         // norms: rows of H, columns of X and of Y
    cx<double> *fac;
    cx<float> *facf;    // MIXED: FP32 copy of fac
    cx<T> *B2;
    float4 *H4, *part;  // refinement by rows: H as double-words, a slot per thread
};

template <typename T, bool REFINE>
__device__ __forceinline__ SnapSmem<T> snap_carve(char *base, int n, bool rho, int fac_len) {
    const SnapLayout L =
        snap_layout(n, sizeof(T), REFINE, rho, fac_len, (blockDim.x + 31) >> 5);
    SnapSmem<T> s;
    s.w.H = reinterpret_cast<cx<T> *>(base + L.H);
    s.w.U = reinterpret_cast<cx<T> *>(base + L.U);
    s.w.rot = reinterpret_cast<JRot<T> *>(base + L.rot);
    s.w.dia = reinterpret_cast<T *>(base + L.dia);
    s.w.red = reinterpret_cast<T *>(base + L.red);
    s.w.tab = reinterpret_cast<uint2 *>(base + L.tab);
    s.w.diag = reinterpret_cast<T *>(base + L.diag);
    s.lam = reinterpret_cast<double *>(base + L.lam);
    s.lw = REFINE ? reinterpret_cast<float2 *>(base + L.lam) : nullptr;
    s.acc = reinterpret_cast<double *>(base + L.acc);
    s.rank = reinterpret_cast<int *>(base + L.rank);
    s.Hh = REFINE ? reinterpret_cast<cx<float> *>(base + L.Hh) : nullptr;
    s.Hl = REFINE ? reinterpret_cast<cx<float> *>(base + L.Hl) : nullptr;
    s.Yl = REFINE ? reinterpret_cast<cx<float> *>(base + L.Yl) : nullptr;
    s.SR = REFINE ? reinterpret_cast<cx<float> *>(base + L.SR) : nullptr;
    s.corr = REFINE ? reinterpret_cast<float *>(base + L.corr) : nullptr;
    s.gd = REFINE ? reinterpret_cast<float2 *>(base + L.rd) : nullptr;
    s.lamf = REFINE ? reinterpret_cast<float *>(base + L.lamf) : nullptr;
    s.rk = REFINE ? reinterpret_cast<int *>(base + L.rk) : nullptr;
    s.ord = REFINE ? reinterpret_cast<int *>(base + L.ord) : nullptr;
    s.cst = REFINE ? reinterpret_cast<int *>(base + L.cst) : nullptr;
    s.scal = REFINE ? reinterpret_cast<int *>(base + L.scal) : nullptr;
    s.rn = REFINE ? reinterpret_cast<float *>(base + L.rn) : nullptr;
    s.cn = REFINE ? reinterpret_cast<float *>(base + L.cn) : nullptr;
    s.yn = REFINE ? reinterpret_cast<float *>(base + L.yn) : nullptr;
    s.fac = rho ? reinterpret_cast<cx<double> *>(base + L.fac) : nullptr;
    s.facf = rho && REFINE ? reinterpret_cast<cx<float> *>(base + L.facf) : nullptr;
    s.B2 = rho ? reinterpret_cast<cx<T> *>(base + L.B2) : nullptr;
    return s;
}

// ------------------------------------------------------------------ helpers

__device__ __forceinline__ void tri_index(int e, int &j, int &k) {
    // e -> (j, k) with j >= k, e = j (j + 1) / 2 + k
    j = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
    while ((j + 1) * (j + 2) / 2 <= e) ++j;
    while (j * (j + 1) / 2 > e) --j;
    k = e - j * (j + 1) / 2;
}

__device__ __forceinline__ int pair_index(int j, int k) { return j * (j - 1) / 2 + k; }

// Frequency record of pair o (FP64 snapshot kernels): the FP64 angular
// frequency w, or -- on a uniform grid in mixed precision -- the phases
// w dt and w t0 reduced modulo 2 pi in FP64 and stored as double-word
// floats.  The mixed kernels use store_frequency_dw instead.
__device__ __forceinline__ void store_frequency(const SnapArgs &a, size_t o, double w) {
    if (a.pair_phase) {
        const double psi = reduce_2pi(w * a.dt);
        const double ph0 = a.t0 == 0.0 ? 0.0 : reduce_2pi(w * a.t0);
        const float psh = (float)psi, p0h = (float)ph0;
        a.pair_phase[o] = make_float4(psh, (float)(psi - (double)psh), p0h,
                                      (float)(ph0 - (double)p0h));
    } else {
        a.pair_omega[o] = w;
    }
}

// Frequency record of pair o on the mixed path from its level gap d
// (double-word): the phases d (2 pi dt) and d (2 pi t0) reduced modulo 2 pi,
// or the FP64 angular frequency for arbitrary grids.  No FP64 arithmetic on
// a uniform grid.
__device__ __forceinline__ void store_frequency_dw(const SnapArgs &a, size_t o, float2 d) {
    if (a.pair_phase) {
        const float2 psi = dw_phase_mod2pi(d, a.c_dt);
        const float2 ph0 = a.t0_zero ? make_float2(0.f, 0.f) : dw_phase_mod2pi(d, a.c_t0);
        a.pair_phase[o] = make_float4(psi.x, psi.y, ph0.x, ph0.y);
    } else {
        a.pair_omega[o] = 6.283185307179586476925 * dw_to_double(d);
    }
}

// Row norms of H's hi part (bounds of the refinement's anchored sums).
template <typename T>
__device__ void hamiltonian_row_norms(SnapSmem<T> &s, int n, int m) {
    const int ld = m + 1;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        float acc = 0.f;
        for (int k = 0; k < n; ++k) {
            const cx<float> h = s.Hh[i * ld + k];
            acc = fmaf(h.re, h.re, fmaf(h.im, h.im, acc));
        }
        s.rn[i] = sqrtf(acc);
    }
    __syncthreads();
}

// (s, c) += b z for a double-word b and z = zh + zl: the product's high
// part summed with its rounding error (TwoSum) and every low-order term
// into c.
__device__ __forceinline__ void dw_acc_prod(float &s, float &c, float2 b, float zh, float zl) {
    const float p = __fmul_rn(b.x, zh);
    const float e = fmaf(b.x, zh, -p);
    const float t = __fadd_rn(s, p);
    const float bb = __fsub_rn(t, s);
    const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bb)), __fsub_rn(p, bb));
    s = t;
    c = __fadd_rn(c, __fadd_rn(err, __fadd_rn(e, fmaf(b.x, zl, b.y * zh))));
}

// v[0..3) in precision T; FP32: converted by lanes 0..2 and shared across
// the warp (one FP64 conversion per warp instead of one per thread).
template <typename T>
__device__ __forceinline__ void load_vec3(const double *v, T &x, T &y, T &z) {
    if constexpr (sizeof(T) == 8) {
        x = v[0];
        y = v[1];
        z = v[2];
    } else {
        const int lane = threadIdx.x & 31;
        const float f = lane < 3 ? (float)v[lane] : 0.f;
        x = __shfl_sync(0xffffffffu, f, 0);
        y = __shfl_sync(0xffffffffu, f, 1);
        z = __shfl_sync(0xffffffffu, f, 2);
    }
}

// b[0..3) as double-words, computed by lanes 0..2 of the warp and shared.
__device__ __forceinline__ void field_dw(const double *b, float2 &bx, float2 &by, float2 &bz) {
    const int lane = threadIdx.x & 31;
    const float2 v = lane < 3 ? dw_of(b[lane]) : make_float2(0.f, 0.f);
    bx = make_float2(__shfl_sync(0xffffffffu, v.x, 0), __shfl_sync(0xffffffffu, v.y, 0));
    by = make_float2(__shfl_sync(0xffffffffu, v.x, 1), __shfl_sync(0xffffffffu, v.y, 1));
    bz = make_float2(__shfl_sync(0xffffffffu, v.x, 2), __shfl_sync(0xffffffffu, v.y, 2));
}

// H = Hsys + b . Z into the Jacobi buffer (FP32, padded to m) unless PRE, and its split
// H = Hh + Hl into two FP32 matrices.
// With Hdw / Zdw (Hsys and Z pre-split into double-words, (re_hi, im_hi,
// re_lo, im_lo) per entry) assembles in double-word FP32 (~2^-47 relative),
// otherwise in FP64 (split exactly).  blockDim.x is a multiple of 32.
template <bool PRE>
__device__ void load_hamiltonian(const cx<double> *Hsys, const cx<double> *Z, const float4 *Hdw,
                                 const float4 *Zdw, const double *b, int n, int m,
                                 SnapSmem<float> &s) {
    const int tid = threadIdx.x, nt = blockDim.x, ld = m + 1, ldh = jacobi_ldh(m);
    const size_t nn = (size_t)n * n;
    if (Hdw != nullptr) {
        float2 bx, by, bz;
        field_dw(b, bx, by, bz);
        for (int e = tid; e < m * m; e += nt) {
            const int i = FastDiv(m).div(e), j = e - i * m;
            float2 hr = make_float2(0.f, 0.f), hi = hr;
            if (i < n && j < n) {
                const size_t o = (size_t)i * n + j;
                const float4 hs = Hdw[o], z0 = Zdw[o], z1 = Zdw[nn + o], z2 = Zdw[2 * nn + o];
                float sr = hs.x, cr = hs.z, si = hs.y, ci = hs.w;
                dw_acc_prod(sr, cr, bx, z0.x, z0.z);
                dw_acc_prod(si, ci, bx, z0.y, z0.w);
                dw_acc_prod(sr, cr, by, z1.x, z1.z);
                dw_acc_prod(si, ci, by, z1.y, z1.w);
                dw_acc_prod(sr, cr, bz, z2.x, z2.z);
                dw_acc_prod(si, ci, bz, z2.y, z2.w);
                hr = dw_two_sum(sr, cr);
                hi = dw_two_sum(si, ci);
            }
            if (!PRE) s.w.H[i * ldh + j] = mk<float>(hr.x, hi.x);
            s.Hh[i * ld + j] = mk<float>(hr.x, hi.x);
            s.Hl[i * ld + j] = mk<float>(hr.y, hi.y);
        }
    } else {
        const double bx = b[0], by = b[1], bz = b[2];
        for (int e = tid; e < m * m; e += nt) {
            const int i = FastDiv(m).div(e), j = e - i * m;
            cx<double> h = mk<double>(0.0, 0.0);
            if (i < n && j < n) {
                const size_t o = (size_t)i * n + j;
                const cx<double> hs = Hsys[o], z0 = Z[o], z1 = Z[nn + o], z2 = Z[2 * nn + o];
                h.re = hs.re + bx * z0.re + by * z1.re + bz * z2.re;
                h.im = hs.im + bx * z0.im + by * z1.im + bz * z2.im;
            }
            const float hr = (float)h.re, hi = (float)h.im;
            if (!PRE) s.w.H[i * ldh + j] = mk<float>(hr, hi);
            s.Hh[i * ld + j] = mk<float>(hr, hi);
            s.Hl[i * ld + j] = mk<float>((float)(h.re - (double)hr), (float)(h.im - (double)hi));
        }
    }
    __syncthreads();
    hamiltonian_row_norms(s, n, m);
}

// The FP32 eigensolve of a snapshot: Jacobi in this CTA, or (PRE)
// the FP32 eigenvectors the warp Jacobi stage left in a.evec, with the
// status it wrote.  Leaves the eigenvectors in s.w.U (row stride ld; m + 1 after Jacobi).
template <bool PRE>
__device__ __forceinline__ int snap_eigvecs(const SnapArgs &a, int sn, int g, int n, int m, int ld,
                                            SnapSmem<float> &s) {
    if (!PRE) return jacobi_sweeps<float>(s.w, m, a.max_sweeps);
    const float2 *X = reinterpret_cast<const float2 *>(a.evec) + (size_t)sn * n * n;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = FastDiv(n).div(e), j = e - i * n;
        const float2 x = X[e];
        s.w.U[i * ld + j] = mk<float>(x.x, x.y);
    }
    const int st = a.status[g];
    __syncthreads();
    return st;
}

// One Ogita-Aishima refinement step of the FP32 eigenvector matrix X
// (columns) against H = Hh + Hl (Ogita & Aishima, Japan J. Indust. Appl.
// Math. 35 (2018) 1007, Algorithm 1, Hermitian form):
//   R = I - X^H X,  S = X^H H X,  l_i = S_ii / (1 - R_ii),
//   E_ij = (S_ij + l_j R_ij) / (l_j - l_i)  (i != j),
//   E_ii = R_ii / 2,   X <- X + X E,
// with eigenvalues l_i plus the second-order term
// sum_j |S_ij + l_i R_ij|^2 / (l_i - l_j).  H X, X^H H X and X^H X use
// double-word FP32 accumulation and l_i is a double-word (S_ii over
// 1 - R_ii = 1 + g_i as S_ii - S_ii g_i / (1 + g_i)); E, the second-order
// terms and X E are FP32 (they are small corrections).  No FP64.
// Levels too close for the first-order E (near-degenerate clusters, e.g.
// at level anticrossings, and exactly degenerate multiplets) are resolved
// as clusters (msp_cluster.cuh).  Returns this step's largest correction.
// NN > 0: n = NN at compile time (the product loops unroll with constant
// shared-memory offsets); NN = 0: n from the argument.
// LO: also keeps what the FP32 rounding of the corrected vectors drops, in Xl
// (zero in columns that a cluster's rotations, which act on the rounded
// vectors, have changed).
template <int NN, bool LO = false>
__device__ float oa_refine(SnapSmem<float> &s, int n_rt, int m_rt, cx<float> *Xl = nullptr) {
    const int n = NN > 0 ? NN : n_rt, m = NN > 0 ? NN + (NN & 1) : m_rt;
    const int tid = threadIdx.x, nt = blockDim.x, ld = m + 1;
    cx<float> *X = s.w.U;
    cx<float> *Yh = s.w.H;  // Jacobi work matrix is free now
    if (tid < 4) s.scal[tid] = 0;  // [0]: amax, [1]: max|l|, [2]: step (float bits)
    // anchored double-word products (msp_dw.cuh): column norms of X bound
    // every partial sum
    for (int j = tid; j < n; j += nt) {
        float acc = 0.f;
        #pragma unroll

        for (int k = 0; k < n; ++k) acc = fmaf(X[k * ld + j].re, X[k * ld + j].re,
                                               fmaf(X[k * ld + j].im, X[k * ld + j].im, acc));
        s.cn[j] = sqrtf(acc);
    }
    __syncthreads();
    // Y = H X (H as hi + lo)
    for (int e = tid; e < n * n; e += nt) {
        const int i = FastDiv(n).div(e), j = e - i * n;
        const u64 K = lm_anchor(s.rn[i] * s.cn[j]);
        u64 s1 = K, s2 = K, c1 = 0ull, c2 = 0ull;
        const u64 *hh = reinterpret_cast<const u64 *>(s.Hh + i * ld);
        const u64 *hl = reinterpret_cast<const u64 *>(s.Hl + i * ld);
        #pragma unroll

        for (int k = 0; k < n; ++k) {
            const cx<float> x = X[k * ld + j];
            lm_step<true, false>(s1, c1, s2, c2, hh[k], hl[k], f32x2(x.re, x.re),
                                 f32x2(x.im, x.im), 0ull, 0ull);
        }
        const float4 r = lm_dw<false>(s1, c1, s2, c2, K);
        Yh[i * ld + j] = mk<float>(r.x, r.y);
        s.Yl[i * ld + j] = mk<float>(r.z, r.w);
    }
    __syncthreads();
    for (int j = tid; j < n; j += nt) {
        float acc = 0.f;
        #pragma unroll

        for (int k = 0; k < n; ++k) acc = fmaf(Yh[k * ld + j].re, Yh[k * ld + j].re,
                                               fmaf(Yh[k * ld + j].im, Yh[k * ld + j].im, acc));
        s.yn[j] = sqrtf(acc);
    }
    __syncthreads();
    // S_ij = X_i^H Y_j (i <= j) into SR upper triangle / sd; R_ij = -X_i^H X_j
    // (i < j) into SR lower triangle at (j, i); R_ii into rd
    const int ntri = n * (n + 1) / 2;
    for (int e = tid; e < ntri; e += nt) {
        int j, i;
        tri_index(e, j, i);  // j >= i
        const u64 KS = lm_anchor(s.cn[i] * s.yn[j]), KG = lm_anchor(s.cn[i] * s.cn[j]);
        u64 a1 = KS, a2 = KS, ac1 = 0ull, ac2 = 0ull;
        u64 g1 = KG, g2 = KG, gc1 = 0ull, gc2 = 0ull;
        #pragma unroll

        for (int k = 0; k < n; ++k) {
            const u64 xi = *reinterpret_cast<const u64 *>(X + k * ld + i);
            const cx<float> y = Yh[k * ld + j], yl = s.Yl[k * ld + j], xj = X[k * ld + j];
            lm_step<false, true>(a1, ac1, a2, ac2, xi, 0ull, f32x2(y.re, y.re), f32x2(y.im, y.im),
                                 f32x2(yl.re, yl.re), f32x2(yl.im, yl.im));
            lm_step<false, false>(g1, gc1, g2, gc2, xi, 0ull, f32x2(xj.re, xj.re),
                                  f32x2(xj.im, xj.im), 0ull, 0ull);
        }
        const float4 S = lm_dw<true>(a1, ac1, a2, ac2, KS);
        const float4 G = lm_dw<true>(g1, gc1, g2, gc2, KG);
        if (i == j) {
            s.gd[i] = make_float2(G.x - 1.0f, G.z);  // G_ii - 1 (G.x - 1 exact)
            s.lw[i] = make_float2(S.x, S.z);         // S_ii until l_i replaces it
        } else {
            s.SR[i * ld + j] = mk<float>(S.x + S.z, S.y + S.w);
            s.SR[j * ld + i] = mk<float>(-(G.x + G.z), -(G.y + G.w));  // R_ij = -G_ij
        }
    }
    __syncthreads();
    float lmax = 0.f;
    for (int i = tid; i < n; i += nt) {
        const float2 lw = dw_rayleigh(s.lw[i], s.gd[i]);
        const float l = lw.x;
        s.lw[i] = lw;
        s.lamf[i] = l;
        lmax = fmaxf(lmax, fabsf(l));
    }
    atomicMax(&s.scal[1], __float_as_int(lmax));  // non-negative: int order = float order
    __syncthreads();
    // clusters; T in Yl (free now)
    OaCluster cl;
    cl.rank = s.rk;
    cl.order = s.ord;
    cl.cstart = s.cst;
    cl.scal = s.scal;
    cl.T = s.Yl;
    cl.ldt = ld;
    oa_clusters(s.SR, ld, s.lw, s.lamf, n, cl);
    float emax = 0.f;
    const int nup = n * (n - 1) / 2;
    for (int e = tid; e < nup; e += nt) {
        int i, j;
        oa_pair_of(e, i, j);
        oa_pair_correction(s.SR, ld, s.lw, s.lamf, cl, i, j, emax);
    }
    __syncthreads();
    oa_second_order(s.SR, ld, s.lw, n, cl, s.corr);
    __syncthreads();
    oa_cluster_diagonal(s.lw, s.corr, n, cl);
    // X' = X + X E  (into Yh), E_ii = R_ii / 2
    for (int e = tid; e < n * n; e += nt) {
        const int k = FastDiv(n).div(e), j = e - k * n;
        const cx<float> xkj = X[k * ld + j];
        const float hr = -0.5f * (s.gd[j].x + s.gd[j].y);  // R_jj / 2
        float ar = LO ? hr * xkj.re : xkj.re + hr * xkj.re;
        float ai = LO ? hr * xkj.im : xkj.im + hr * xkj.im;
        #pragma unroll

        for (int i = 0; i < n; ++i) {
            if (i == j) continue;
            const cx<float> x = X[k * ld + i], E = s.SR[i * ld + j];
            ar = fmaf(x.re, E.re, fmaf(-x.im, E.im, ar));
            ai = fmaf(x.re, E.im, fmaf(x.im, E.re, ai));
        }
        if constexpr (LO) {
            const float2 xr = dw_two_sum(xkj.re, ar), xi = dw_two_sum(xkj.im, ai);
            Yh[k * ld + j] = mk<float>(xr.x, xi.x);
            Xl[k * ld + j] = mk<float>(xr.y, xi.y);
        } else {
            Yh[k * ld + j] = mk<float>(ar, ai);
        }
    }
    __syncthreads();
    for (int e = tid; e < n * n; e += nt) {
        const int k = FastDiv(n).div(e), j = e - k * n;
        X[k * ld + j] = Yh[k * ld + j];
    }
    __syncthreads();
    emax = fmaxf(emax, oa_resolve_clusters(X, ld, n, s.lw, s.corr, n, cl,
                                           __int_as_float(s.scal[1]), LO ? Xl : nullptr));
    atomicMax(&s.scal[2], __float_as_int(emax));  // non-negative: int order = float order
    __syncthreads();
    const float step = __int_as_float(s.scal[2]);
    __syncthreads();
    return step;
}

// Applies the single-spin matrix F (dim x dim, complex FP64 or FP32) on
// digit `stride` of the row index of X (n x n, row stride ld) into Y:
// Y = (1 (x) F (x) 1) X.
template <typename T, typename TF>
__device__ void apply_digit(const cx<TF> *F, int dim, int stride, const cx<T> *X, cx<T> *Y, int n,
                            int ld) {
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = FastDiv(n).div(e), k = e - i * n;
        const int di = (i / stride) % dim;
        const int base = i - di * stride;
        T yr = 0, yi = 0;
        for (int l = 0; l < dim; ++l) {
            const cx<TF> f = F[di * dim + l];
            const cx<T> x = X[(base + l * stride) * ld + k];
            yr += (T)f.re * x.re - (T)f.im * x.im;
            yi += (T)f.re * x.im + (T)f.im * x.re;
        }
        Y[i * ld + k] = mk<T>(yr, yi);
    }
    __syncthreads();
}

// Y[j][k] = sum_i conj(U_ij) X_ik for j >= k (row stride ld = n + (n & 1) + 1).
template <typename T>
__device__ __forceinline__ void tri_conj_products(const cx<T> *U, const cx<T> *X, cx<T> *Y, int n) {
    const int ld = n + (n & 1) + 1, ntri = n * (n + 1) / 2;
    for (int e = threadIdx.x; e < ntri; e += blockDim.x) {
        int j, k;
        tri_index(e, j, k);
        T gr = 0, gi = 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const cx<T> u = U[i * ld + j], x = X[i * ld + k];
            gr += u.re * x.re + u.im * x.im;
            gi += u.re * x.im - u.im * x.re;
        }
        Y[j * ld + k] = mk<T>(gr, gi);
    }
}

// Refined eigenpairs: eigenvalues as double-words into s.lw[0..n), the
// eigenvectors in place.  One refinement step leaves an error of order E^2; a
// step whose largest correction exceeds 2e-4 (clusters resolved by large
// rotations, levels within ~1e3 FP32 resolutions) is followed by another, at
// most max_refine in all; a last step still above 2e-4 sets
// MSP_ITEM_REFINE_LIMIT.
static __device__ int eigenpairs(SnapSmem<float> &s, int n, int m, int max_refine) {
    if (max_refine <= 0) max_refine = 4;
    for (int it = 0; it < max_refine; ++it) {
        const float step = n == 24   ? oa_refine<24>(s, n, m)
                           : n == 32 ? oa_refine<32>(s, n, m)
                                     : oa_refine<0>(s, n, m);
        if (step <= 2e-4f) return MSP_ITEM_OK;
    }
    return MSP_ITEM_REFINE_LIMIT;
}

// ------------------------------------------------------------------ refinement by rows

// The refinement of the two-stage kernels (n <= 32), in residual form:
//   l_j = x_j^H H x_j / x_j^H x_j,  r_j = H x_j - l_j x_j,  B = X^H R,
//   E_ij = B_ij / (l_j - l_i),  E_jj = (1 - x_j^H x_j) / 2,  X <- X + X E
// (B_ij is the S_ij + l_j R_ij of oa_refine).  r_j is small, so only H X and the
// Rayleigh quotients need double-words, where oa_refine forms X^H H X and X^H X
// in them too.  A thread owns a column j and four rows of every product: H X's
// stay in its registers until the residuals are formed, B's until they have
// become E, and an element of the row operand is a broadcast that serves four
// elements (oa_refine loads three operands for each).  n = 32: FP32 pipe 10
// + 2 + 2 packed FMAs per complex product against 22, 42 KB of shared memory
// against 59.  Scan of n = 32: 19.4 ms against 28.6; powder of n =
// 24: 0.41 ms against 0.47.

// Groups of rows, rows per group and rows the matrices are padded to.
constexpr int ROW_MAX = 4;  // largest number of rows per thread

struct RowShape {
    int groups, rows, padded;
};

__host__ __device__ inline RowShape row_shape(int n, int threads) {
    RowShape s;
    s.groups = threads / n < n ? threads / n : n;
    s.rows = (n + s.groups - 1) / s.groups;
    s.rows += s.rows & 1;  // pairs of rows start on 16 bytes
    s.groups = (n + s.rows - 1) / s.rows;
    s.padded = (s.groups - 1) * s.rows + ROW_MAX;
    if (s.padded < n) s.padded = n;
    return s;
}

// At most four rows per thread.  (Eight, in half the threads, spill at 96
// registers and leave too few warps at 128: scan of n = 32, 27 ms against 22.)
// Four rows per thread of n = 20 need 100 threads: 160 leave room for fewer CTAs (2,000
// snapshots in three rounds of six per SM, 88 us; 75 in two of eight).
inline int row_threads(int n) { return n <= 8 ? 32 : n <= 16 ? 64 : n <= 20 ? 128 : n <= 24 ? 160 : 256; }

// Row stride of the FP32 matrices: even, so that two elements of a row operand are
// one 16-byte load (the plain products are bound by shared-memory loads: scan of n = 32
// 29.9 -> 29.5 ms in all, powder of n = 24 1.17 -> 1.15).
__host__ __device__ constexpr int row_ld(int n) { return n + (n & 1) + 2; }

// Row stride of H4: odd, for the transposed stores
__host__ __device__ inline int row_ldh(int n) { return n | 1; }

struct RowLayout {
    size_t H4, U, R, SR, part, red, lw, corr, rk, ord, cst, scal, rn, fac, facf, total;
};

__host__ __device__ inline RowLayout row_layout(int n, bool rho, int fac_len, int threads) {
    RowLayout L;
    const size_t m = (size_t)(n + (n & 1)), mm = (size_t)row_shape(n, threads).padded * row_ld(n) * 8;
    size_t off = 0;
    L.H4 = lay_take(off, (size_t)row_shape(n, threads).padded * row_ldh(n) * 16);
    L.U = lay_take(off, mm);
    L.R = lay_take(off, mm);
    L.SR = lay_take(off, mm);
    L.part = lay_take(off, (size_t)threads * 16);
    L.red = lay_take(off, (size_t)(threads / 32) * 8);
    L.lw = lay_take(off, m * 8);
    L.corr = lay_take(off, m * 4);
    L.rk = lay_take(off, m * 4);
    L.ord = lay_take(off, m * 4);
    L.cst = lay_take(off, m * 4);
    L.scal = lay_take(off, 4 * 4);
    L.rn = lay_take(off, (size_t)row_shape(n, threads).padded * 4);
    L.fac = L.facf = 0;
    if (rho) {
        L.fac = lay_take(off, (size_t)fac_len * 16);
        L.facf = lay_take(off, (size_t)fac_len * 8);
    }
    L.total = (off + 15) & ~size_t(15);
    return L;
}

__device__ __forceinline__ SnapSmem<float> row_carve(char *base, int n, bool rho, int fac_len) {
    const RowLayout L = row_layout(n, rho, fac_len, blockDim.x);
    SnapSmem<float> s = {};
    s.H4 = reinterpret_cast<float4 *>(base + L.H4);
    s.w.U = reinterpret_cast<cx<float> *>(base + L.U);
    s.w.H = reinterpret_cast<cx<float> *>(base + L.R);
    s.SR = s.B2 = reinterpret_cast<cx<float> *>(base + L.SR);
    s.part = reinterpret_cast<float4 *>(base + L.part);
    s.w.red = reinterpret_cast<float *>(base + L.red);
    s.lw = reinterpret_cast<float2 *>(base + L.lw);
    s.corr = reinterpret_cast<float *>(base + L.corr);
    s.rk = reinterpret_cast<int *>(base + L.rk);
    s.ord = reinterpret_cast<int *>(base + L.ord);
    s.cst = reinterpret_cast<int *>(base + L.cst);
    s.scal = reinterpret_cast<int *>(base + L.scal);
    s.rn = reinterpret_cast<float *>(base + L.rn);
    if (rho) {
        s.fac = reinterpret_cast<cx<double> *>(base + L.fac);
        s.facf = reinterpret_cast<cx<float> *>(base + L.facf);
    }
    return s;
}

// H = Hsys + b . Z as double-words into s.H4 (row stride n, the upper triangle
// mirrored), in double-word FP32 from pre-split matrices or in FP64, and the
// row norms of its high words.
__device__ __forceinline__ void load_hamiltonian_rows(const SnapSource &src, const double *b, int n,
                                                      SnapSmem<float> &s) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, ldh = row_ldh(n);
    const size_t nn = (size_t)n * n;
    float2 bx, by, bz;
    field_dw(b, bx, by, bz);
#pragma unroll 3
    for (int e = tid; e < n * (n + 1) / 2; e += nt) {
        int i, j;
        tri_index(e, j, i);  // i <= j
        const size_t o = (size_t)i * n + j;
        float4 h;
        if (src.Hdw != nullptr) {
            const float4 hs = src.Hdw[o], z0 = src.Zdw[o], z1 = src.Zdw[nn + o], z2 = src.Zdw[2 * nn + o];
            float sr = hs.x, cr = hs.z, si = hs.y, ci = hs.w;
            dw_acc_prod(sr, cr, bx, z0.x, z0.z);
            dw_acc_prod(si, ci, bx, z0.y, z0.w);
            dw_acc_prod(sr, cr, by, z1.x, z1.z);
            dw_acc_prod(si, ci, by, z1.y, z1.w);
            dw_acc_prod(sr, cr, bz, z2.x, z2.z);
            dw_acc_prod(si, ci, bz, z2.y, z2.w);
            const float2 hr = dw_two_sum(sr, cr), hi = dw_two_sum(si, ci);
            h = make_float4(hr.x, hi.x, hr.y, hi.y);
        } else {
            const cx<double> hs = src.Hsys[o], z0 = src.Z[o], z1 = src.Z[nn + o], z2 = src.Z[2 * nn + o];
            h = dw_split(make_double2(hs.re + b[0] * z0.re + b[1] * z1.re + b[2] * z2.re,
                                      hs.im + b[0] * z0.im + b[1] * z1.im + b[2] * z2.im));
        }
        if (i == j) h.y = h.w = 0.f;
        s.H4[i * ldh + j] = h;
        if (i != j) s.H4[j * ldh + i] = make_float4(h.x, -h.y, h.z, -h.w);
    }
    __syncthreads();
    for (int i = tid >> 5; i < n; i += nt >> 5) {
        const float4 h = lane < n ? s.H4[i * ldh + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
        float acc = fmaf(h.x, h.x, h.y * h.y);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) s.rn[i] = sqrtf(acc);
    }
    __syncthreads();
}

// (X^H X)_ij, i != j, to FP32 rounding of its terms' sum
__device__ __forceinline__ cx<float> row_gram(const cx<float> *X, int n, int ld, int i, int j, u64 K) {
    u64 s1 = K, c1 = 0ull, s2 = K, c2 = 0ull;
    for (int k = 0; k < n; ++k) {
        const cx<float> y = X[k * ld + j];
        lm_step<false, false>(s1, c1, s2, c2, *reinterpret_cast<const u64 *>(X + k * ld + i), 0ull,
                              f32x2(y.re, y.re), f32x2(y.im, y.im), 0ull, 0ull);
    }
    const float4 r = lm_dw<true>(s1, c1, s2, c2, K);
    return mk<float>(r.x + r.z, r.y + r.w);
}

// This thread's rows of column j of X^H W: b[r] = sum_k conj(X_k,i1+r) W_kj
template <int NN, int RB>
__device__ __forceinline__ void row_products(const cx<float> *X, const cx<float> *W, int n_rt, int i1,
                                             int j, cx<float> (&b)[RB]) {
    static_assert(RB % 2 == 0, "pairs of rows");
    const int n = NN > 0 ? NN : n_rt, ld = row_ld(n);
    u64 s1[RB], s2[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) s1[r] = s2[r] = 0ull;
#pragma unroll 8
    for (int k = 0; k < n; ++k) {
        const cx<float> q = W[k * ld + j];
        const u64 bx = f32x2(q.re, q.re), by = f32x2(q.im, q.im);
        u64 x[RB];
#pragma unroll
        for (int r = 0; r < RB; r += 2) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(X + k * ld + i1 + r);
            x[r] = v.x;
            x[r + 1] = v.y;
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            s1[r] = fma_f32x2(x[r], bx, s1[r]);
            s2[r] = fma_f32x2(x[r], by, s2[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) b[r] = lm_plain<true>(s1[r], s2[r]);
}

// s1, s2 += this thread's rows of A E, column j
template <int NN, int RB>
__device__ __forceinline__ void row_times(const cx<float> *A, const cx<float> *E, int n_rt, int i1, int j,
                                          u64 (&s1)[RB], u64 (&s2)[RB]) {
    const int n = NN > 0 ? NN : n_rt, ld = row_ld(n);
    if constexpr (NN > 0 && NN % 2 == 0) {
#pragma unroll 4
        for (int i = 0; i < n; i += 2) {
            const cx<float> e = E[i * ld + j], f = E[(i + 1) * ld + j];
            const u64 ex = f32x2(e.re, e.re), ey = f32x2(e.im, e.im);
            const u64 fx = f32x2(f.re, f.re), fy = f32x2(f.im, f.im);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(A + (i1 + r) * ld + i);
                s1[r] = fma_f32x2(x.y, fx, fma_f32x2(x.x, ex, s1[r]));
                s2[r] = fma_f32x2(x.y, fy, fma_f32x2(x.x, ey, s2[r]));
            }
        }
    } else {
#pragma unroll 8
        for (int i = 0; i < n; ++i) {
            const cx<float> e = E[i * ld + j];
            const u64 bx = f32x2(e.re, e.re), by = f32x2(e.im, e.im);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const u64 x = *reinterpret_cast<const u64 *>(A + (i1 + r) * ld + i);
                s1[r] = fma_f32x2(x, bx, s1[r]);
                s2[r] = fma_f32x2(x, by, s2[r]);
            }
        }
    }
}

// One refinement step by rows: the vectors in s.w.U, the levels in s.lw.
// Returns its largest correction.  NN > 0: n = NN at compile time.
template <int NN, int RB>
__device__ __forceinline__ float oa_refine_rows(SnapSmem<float> &s, int n_rt) {
    const int n = NN > 0 ? NN : n_rt, ld = row_ld(n), tid = threadIdx.x;
    const RowShape sh = row_shape(n, blockDim.x);
    const int rg = tid / n, j = tid - rg * n, i0 = rg * sh.rows;
    // threads past the last group follow along on the first rows and store nothing
    const bool active = rg < sh.groups;
    const int i1 = active ? i0 : 0;
    auto mine = [&](int r) { return active && r < sh.rows && i0 + r < n; };
    cx<float> *X = s.w.U, *R = s.w.H, *T = s.w.H;
    if (tid < 4) s.scal[tid] = 0;  // [0]: amax, [1]: max|l|, [2]: step (float bits), [3]: clusters
    float sx = 0.f;
#pragma unroll
    for (int r = 0; r < RB; ++r)
        if (mine(r)) sx += cabs2(X[(i0 + r) * ld + j]);
    if (active) s.part[tid].x = sx;
    __syncthreads();
    float cn = 0.f;
    for (int g = 0; g < sh.groups; ++g) cn += s.part[g * n + j].x;
    cn = sqrtf(cn);
    // H X
    float4 y[RB];
    {
        u64 s1[RB], c1[RB], s2[RB], c2[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            s1[r] = s2[r] = lm_anchor(s.rn[i1 + r] * cn);
            c1[r] = c2[r] = 0ull;
        }
        const int ldh = row_ldh(n);
        const float4 *H = s.H4 + i1 * ldh;
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            const cx<float> x = X[k * ld + j];
            const u64 bx = f32x2(x.re, x.re), by = f32x2(x.im, x.im);
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const ulonglong2 h = *reinterpret_cast<const ulonglong2 *>(H + r * ldh + k);
                lm_step<true, false>(s1[r], c1[r], s2[r], c2[r], h.x, h.y, bx, by, 0ull, 0ull);
            }
        }
#pragma unroll
        for (int r = 0; r < RB; ++r)
            y[r] = lm_dw<false>(s1[r], c1[r], s2[r], c2[r], lm_anchor(s.rn[i1 + r] * cn));
    }
    // Rayleigh quotients from this thread's rows, then every group's
    {
        float sy = 0.f;
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (mine(r)) sy = fmaf(y[r].x, y[r].x, fmaf(y[r].y, y[r].y, sy));
        const u64 Ky = lm_anchor(sqrtf(sx * sy)), Kx = lm_anchor(sx);
        u64 dy = Ky, cy = 0ull, dx = Kx, cc = 0ull;
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            if (!mine(r)) continue;
            const u64 x = *reinterpret_cast<const u64 *>(X + (i0 + r) * ld + j);
            dw_dot(dy, cy, x, f32x2(y[r].x, y[r].y), f32x2(y[r].z, y[r].w));
            dw_dot(dx, cc, x, x, 0ull);
        }
        const float2 a = dw_dot_value(dy, cy, Ky), b = dw_dot_value(dx, cc, Kx);
        __syncthreads();  // the norms have been read
        if (active) s.part[tid] = make_float4(a.x, a.y, b.x, b.y);
    }
    __syncthreads();
    float4 d = s.part[j];
    for (int g = 1; g < sh.groups; ++g) {
        const float4 e = s.part[g * n + j];
        dw_add(d.x, d.y, e.x, e.y);
        dw_add(d.z, d.w, e.z, e.w);
    }
    const float2 gj = dw_add_f(dw_two_sum(d.z, d.w), -1.0f);
    const float2 lj = dw_rayleigh(dw_two_sum(d.x, d.y), gj);
    if (rg == 0) {
        s.lw[j] = lj;
        atomicMax(&s.scal[1], __float_as_int(fabsf(lj.x)));  // non-negative: int order = float order
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        if (!mine(r)) continue;
        const cx<float> x = X[(i0 + r) * ld + j];
        R[(i0 + r) * ld + j] = mk<float>(fmaf(-lj.x, x.re, y[r].x) + fmaf(-lj.y, x.re, y[r].z),
                                         fmaf(-lj.x, x.im, y[r].y) + fmaf(-lj.y, x.im, y[r].w));
    }
    __syncthreads();
    // B = X^H R
    cx<float> b[RB];
    row_products<NN, RB>(X, R, n, i1, j, b);
    {
        float amax = 0.f;
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            if (mine(r) && i0 + r != j) amax = fmaxf(amax, fmaxf(fabsf(b[r].re), fabsf(b[r].im)));
        }
        const int am = __reduce_max_sync(0xffffffffu, __float_as_int(amax));
        if ((tid & 31) == 0) atomicMax(&s.scal[0], am);
    }
    __syncthreads();
    OaCluster cl;
    cl.rank = s.rk;
    cl.order = s.ord;
    cl.cstart = s.cst;
    cl.scal = s.scal;
    cl.T = T;
    cl.ldt = ld;
    oa_cluster_starts(s.lw, n, cl);
    // E; the couplings inside clusters go to T
    float emax = 0.f, corr = 0.f;
    const int rj = s.rk[j], cj = s.cst[rj];
    bool any = false;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        const int i = i0 + r;
        if (!mine(r)) continue;
        cx<float> E;
        if (i == j) {
            E = mk<float>(-0.5f * (gj.x + gj.y), 0.f);
        } else if (s.cst[s.rk[i]] == cj) {
            any = true;
            T[s.rk[i] * ld + rj] = b[r];
            const cx<float> G = row_gram(X, n, ld, i, j, lm_anchor(1.1f * cn * cn));
            E = mk<float>(-0.5f * G.re, -0.5f * G.im);
        } else {
            const float inv = 1.0f / dw_sub_f(lj, s.lw[i]);
            E = mk<float>(b[r].re * inv, b[r].im * inv);
            corr = fmaf(b[r].re * b[r].re + b[r].im * b[r].im, inv, corr);
            emax = fmaxf(emax, fmaxf(fabsf(E.re), fabsf(E.im)));
        }
        s.SR[i * ld + j] = E;
    }
    if (active) s.part[tid].x = corr;
    if (any) s.scal[3] = 1;
    {
        const int em = __reduce_max_sync(0xffffffffu, __float_as_int(emax));
        if ((tid & 31) == 0) atomicMax(&s.scal[2], em);  // non-negative: int order = float order
    }
    __syncthreads();
    // the same in every thread
    const bool clusters = s.scal[3] != 0;
    const float first = __int_as_float(s.scal[2]);
    const bool second = n > 24 && !clusters && first > 2e-4f && first <= 3e-3f;
    if (rg == 0) {
        float c = 0.f;
        for (int g = 0; g < sh.groups; ++g) c += s.part[g * n + j].x;
        s.corr[j] = c;
    }
    if (second) {
        // The exact E solves E_ij (l'_j - l_i) = (B + B E)_ij, with l'_j - l_j =
        // sum_i conj(B_ij) E_ij: one more pass with the first-order E on the right
        // leaves errors of its third power (no gap is below 30 amax here), where
        // another refinement step would cost a double-word product.  B comes back
        // as E times the gap, so that no register holds it.  Scan of n = 32: 19.4 ms
        // against 21.3.  Not at n <= 24, where nine first steps in ten suffice and
        // the branch alone cost 6% (0.44 ms against 0.41).
        auto coupling = [&](int r) {
            const cx<float> e = s.SR[(i0 + r) * ld + j];
            const float gap = dw_sub_f(lj, s.lw[i0 + r]);
            return mk<float>(e.re * gap, e.im * gap);
        };
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (mine(r)) R[(i0 + r) * ld + j] = coupling(r);
        __syncthreads();
        const float dj = s.corr[j];
        cx<float> q[RB];
        {
            u64 s1[RB], s2[RB];
#pragma unroll
            for (int r = 0; r < RB; ++r) s1[r] = s2[r] = 0ull;
            row_times<NN, RB>(R, s.SR, n, i1, j, s1, s2);
#pragma unroll
            for (int r = 0; r < RB; ++r) q[r] = lm_plain<false>(s1[r], s2[r]);
        }
        float shift = 0.f, norm = 0.f;
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            if (!mine(r) || i0 + r == j) continue;
            const cx<float> b1 = R[(i0 + r) * ld + j];
            const float inv = 1.0f / (dw_sub_f(lj, s.lw[i0 + r]) + dj);
            q[r] = mk<float>((b1.re + q[r].re) * inv, (b1.im + q[r].im) * inv);
            shift = fmaf(b1.re, q[r].re, fmaf(b1.im, q[r].im, shift));
            norm += cabs2(q[r]);
        }
        if (active) {
            s.part[tid].x = shift;
            s.part[tid].y = norm;
        }
        __syncthreads();
        norm = 0.f;
        for (int g = 0; g < sh.groups; ++g) norm += s.part[g * n + j].y;
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (mine(r))
                s.SR[(i0 + r) * ld + j] = i0 + r == j ? mk<float>(-0.5f * (gj.x + gj.y + norm), 0.f) : q[r];
        if (rg == 0) {
            float c = 0.f;
            for (int g = 0; g < sh.groups; ++g) c += s.part[g * n + j].x;
            s.corr[j] = c;
        }
        __syncthreads();
    }
    if (clusters) {
        // T Hermitian
        for (int r = 0; r < sh.rows; ++r) {
            const int i = i0 + r;
            if (!mine(r) || i >= j || s.cst[s.rk[i]] != cj) continue;
            const int ri = s.rk[i];
            const cx<float> u = T[ri * ld + rj], l = T[rj * ld + ri];
            const cx<float> t = mk<float>(0.5f * (u.re + l.re), 0.5f * (u.im - l.im));
            T[ri * ld + rj] = t;
            T[rj * ld + ri] = conj(t);
        }
        __syncthreads();
        oa_cluster_diagonal(s.lw, s.corr, n, cl);
    }
    // X + X E
    {
        u64 s1[RB], s2[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            s1[r] = *reinterpret_cast<const u64 *>(X + (i1 + r) * ld + j);
            s2[r] = 0ull;
        }
        row_times<NN, RB>(X, s.SR, n, i1, j, s1, s2);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (mine(r)) X[(i0 + r) * ld + j] = lm_plain<false>(s1[r], s2[r]);
    }
    __syncthreads();
    if (clusters) {
        const float em = oa_resolve_clusters(X, ld, n, s.lw, s.corr, n, cl, __int_as_float(s.scal[1]));
        atomicMax(&s.scal[2], __float_as_int(em));
    } else if (rg == 0) {
        s.lw[j] = dw_add_f(s.lw[j], s.corr[j]);
    }
    __syncthreads();
    const float step = second ? first * first : __int_as_float(s.scal[2]);
    __syncthreads();
    return step;
}

// Refined eigenpairs (see eigenpairs above) of a two-stage kernel.  One copy for
// all kernels; it carves shared memory itself so that its accesses stay
// shared-memory accesses.
static __noinline__ __device__ int eigenpairs_rows(int n, bool rho, int fac_len, int max_refine) {
    extern __shared__ __align__(16) char smem[];
    SnapSmem<float> s = row_carve(smem, n, rho, fac_len);
    if (max_refine <= 0) max_refine = 4;
    for (int it = 0; it < max_refine; ++it) {
        // n <= 8: a warp has two rows per thread (300 snapshots of n = 8: 18.5 us, 23.4 with
        // the registers and products of four)
        const float step = n == 24   ? oa_refine_rows<24, ROW_MAX>(s, n)
                           : n == 32 ? oa_refine_rows<32, ROW_MAX>(s, n)
                           : n <= 8  ? oa_refine_rows<0, 2>(s, n)
                                     : oa_refine_rows<0, ROW_MAX>(s, n);
        if (step <= 2e-4f) return MSP_ITEM_OK;
    }
    return MSP_ITEM_REFINE_LIMIT;
}

}  // namespace msp
