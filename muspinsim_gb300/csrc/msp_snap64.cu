// FP64 per-snapshot kernels (n <= 64): one CTA per Hamiltonian.  Replaces,
// like msp_snap.cu, ExperimentRunner.Htot (muspinsim/experiment.py:332-341),
// Hermitian.diag (muspinsim/spinop.py:51-82) and the eigenbasis part of
// Hamiltonian.fast_evolve / evolve / integrate_decaying
// (muspinsim/hamiltonian.py:76-87, 149-160, 195-211).
//
// GB300 runs an FP64 FMA at 1/74 of its FP32 rate, so what an FP64 eigensolve
// costs is the number of FP64 operations.  Cyclic Jacobi in FP64 takes some
// 1.5 M of them at n = 24.  Here the bulk runs in FP32 and FP64 only finishes:
//   1. FP32 eigenvectors (warp Jacobi or Householder + QL for batches of
//      n <= 32, else FP32 Jacobi in this CTA);
//   2. their double-word refinement (oa_refine): eigenvalues to ~2^-48,
//      vectors to ~1e-12, kept as hi + lo FP32;
//   3. one FP64 step.  With x_j the vectors and l_j the levels from 2:
//        r_j = H x_j - l_j x_j                (FP64, 4 n FMAs per nonzero entry of H),
//        d_j = x_j^H r_j / x_j^H x_j          (level correction),
//        E_ij = x_i^H r_j / (l_j - l_i),  E_jj = (1 - x_j^H x_j) / 2,
//        x_j += sum_i x_i E_ij.
//      r_j is small (1e-12 |H|), so everything after it except x_j^H x_j runs
//      in FP32 without losing FP64 accuracy: the products of r_j are exact to
//      6e-8 of 1e-12.  Levels closer than 100 times the largest coupling
//      x_i^H r_j form clusters (Ogita and Aishima, Japan J. Indust. Appl.
//      Math. 36 (2019) 435): orthonormalised among themselves and resolved
//      by a Jacobi on their block of couplings.
//   The step is repeated while its largest E exceeds 4e-9 (its error is of
//   order E^2).  A snapshot that does not get there (entries outside the FP32
//   range, no convergence in stage 1) takes the FP64 Jacobi (msp_jacobi.cuh).
// That and the eigenbasis product (n^3 FMAs) are nearly all that the FP64 pipe sees:
// 44 k FMAs for a molecule of n = 24, 83 k with the zeros of H and with the
// product over all n rows.  Powder of n = 24 (10,000): 3.91 -> 3.43 ms in all; scan of
// n = 12 (14,544): 1.63 -> 1.54 ms.
#include "msp_refine.cuh"

namespace msp {

namespace {

// ------------------------------------------------------------------ shared memory

// Small arrays that live through the kernel, then a region that holds the
// FP32 refinement's buffers first (snap_layout and, for n <= 32, the lo words
// of the vectors) and three FP64 buffers D0..D2 of jacobi_buffer(m) complex
// entries after: D1 over the FP32 matrix and vectors, D0 next, D2 last, so
// that D0 can be filled from the FP32 vectors in place.
struct Snap64Layout {
    size_t lam0, lam, gn, tdiag, nz, red, dl, corr, rk, ord, cst, scal, fac;
    size_t region, xl, total;
};

constexpr int S64_LO_MAX = 32;  // largest n whose lo words fit

__host__ __device__ inline Snap64Layout snap64_layout(int n, int fac_len, int nwarps) {
    Snap64Layout L;
    const size_t m = (size_t)(n + (n & 1));
    size_t off = 0;
    L.lam0 = lay_take(off, m * 8);
    L.lam = lay_take(off, m * 8);
    L.gn = lay_take(off, m * 8);
    L.tdiag = lay_take(off, m * 8);
    L.nz = lay_take(off, m * 8);
    L.red = lay_take(off, 2 * (size_t)nwarps * 8);
    L.dl = lay_take(off, m * 4);
    L.corr = lay_take(off, m * 4);
    L.rk = lay_take(off, m * 4);
    L.ord = lay_take(off, m * 4);
    L.cst = lay_take(off, m * 4);
    L.scal = lay_take(off, 16);
    L.fac = lay_take(off, (size_t)fac_len * 16);
    L.region = off = (off + 255) & ~size_t(255);
    const size_t mj = (size_t)jacobi_buffer((int)m) * 16;
    size_t lo = snap_layout(n, 4, true, false, 0, nwarps).total;
    L.xl = 0;
    if (n <= S64_LO_MAX) {
        // past D0, which is filled from it
        if (lo < 2 * mj) lo = 2 * mj;
        L.xl = off + lo;
        lo += m * (m + 1) * 8;
    }
    // the FP64 Jacobi: its two buffers (D0, D1), then its tables
    const size_t jac = snap_layout(n, 8, false, false, 0, nwarps).total;
    size_t hi = 3 * mj;
    if (hi < lo) hi = lo;
    if (hi < jac) hi = jac;
    L.total = off + hi;
    return L;
}

struct S64 {
    cx<double> *D0, *D1, *D2;
    double *lam0, *lam, *gn, *tdiag, *red;
    unsigned long long *nz;  // bit k of row i: H_ik is not zero
    float *dl, *corr;
    int *rk, *ord, *cst, *scal;
    cx<double> *fac;
    cx<float> *xl;
    char *region;
};

__device__ __forceinline__ S64 carve64(char *base, int n, int fac_len) {
    const Snap64Layout L = snap64_layout(n, fac_len, (blockDim.x + 31) >> 5);
    const size_t mj = (size_t)jacobi_buffer(n + (n & 1)) * 16;
    S64 s;
    s.lam0 = reinterpret_cast<double *>(base + L.lam0);
    s.lam = reinterpret_cast<double *>(base + L.lam);
    s.gn = reinterpret_cast<double *>(base + L.gn);
    s.tdiag = reinterpret_cast<double *>(base + L.tdiag);
    s.nz = reinterpret_cast<unsigned long long *>(base + L.nz);
    s.red = reinterpret_cast<double *>(base + L.red);
    s.dl = reinterpret_cast<float *>(base + L.dl);
    s.corr = reinterpret_cast<float *>(base + L.corr);
    s.rk = reinterpret_cast<int *>(base + L.rk);
    s.ord = reinterpret_cast<int *>(base + L.ord);
    s.cst = reinterpret_cast<int *>(base + L.cst);
    s.scal = reinterpret_cast<int *>(base + L.scal);
    s.fac = reinterpret_cast<cx<double> *>(base + L.fac);
    s.xl = L.xl ? reinterpret_cast<cx<float> *>(base + L.xl) : nullptr;
    s.region = base + L.region;
    s.D1 = reinterpret_cast<cx<double> *>(s.region);
    s.D0 = reinterpret_cast<cx<double> *>(s.region + mj);
    s.D2 = reinterpret_cast<cx<double> *>(s.region + 2 * mj);
    return s;
}

// Where a Hamiltonian comes from: Hsys + b . Z, or one matrix (Z = NULL).
// Only the upper triangle is read.
struct HSource {
    const cx<double> *Hsys, *Z;
    const double *b;
};

__device__ __forceinline__ cx<double> h_entry(const HSource &h, size_t nn, size_t o) {
    cx<double> v = h.Hsys[o];
    if (h.Z) {
        const cx<double> z0 = h.Z[o], z1 = h.Z[nn + o], z2 = h.Z[2 * nn + o];
        v.re = v.re + h.b[0] * z0.re + h.b[1] * z1.re + h.b[2] * z2.re;
        v.im = v.im + h.b[0] * z0.im + h.b[1] * z1.im + h.b[2] * z2.im;
    }
    return v;
}

// The full Hermitian matrix (n x n of row stride ld) into dst, zero beyond n
// up to m.
__device__ void load_h64(const HSource &h, int n, int m, int ld, cx<double> *dst) {
    const size_t nn = (size_t)n * n;
    for (int e = threadIdx.x; e < m * (m + 1) / 2; e += blockDim.x) {
        int i, j;
        tri_index(e, j, i);  // j >= i
        cx<double> v = mk<double>(0.0, 0.0);
        if (j < n) v = h_entry(h, nn, (size_t)i * n + j);
        if (i == j) v.im = 0.0;
        dst[i * ld + j] = v;
        if (i != j) dst[j * ld + i] = conj(v);
    }
}

// ------------------------------------------------------------------ 3. FP64 step

// One FP64 step on X = s.D0 (row stride ld) and the levels s.lam0: s.lam and X
// corrected.  Returns the largest |E| (NaN or infinite when the input is
// unusable).
__device__ float step64(S64 &s, const HSource &h, int n, int m) {
    const int tid = threadIdx.x, nt = blockDim.x, ld = m + 1;
    cx<double> *X = s.D0, *H = s.D1;
    cx<float> *XF = reinterpret_cast<cx<float> *>(s.D2), *RF = XF + n * n;
    if (tid < 4) s.scal[tid] = 0;  // [0]: largest coupling, [1]: largest |level|, [2]: |E|
    load_h64(h, n, m, ld, H);
    for (int e = tid; e < n * n; e += nt) {
        const int i = FastDiv(n).div(e), j = e - i * n;
        const cx<double> x = X[i * ld + j];
        XF[e] = mk<float>((float)x.re, (float)x.im);
    }
    __syncthreads();
    for (int i = tid >> 5; i < n; i += nt >> 5) {
        const int lane = tid & 31;
        unsigned w[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int k = 32 * q + lane;
            const cx<double> a = H[i * ld + (k < n ? k : 0)];
            w[q] = __ballot_sync(0xffffffffu, k < n && !(a.re == 0.0 && a.im == 0.0));  // a NaN counts
        }
        if (lane == 0) s.nz[i] = (unsigned long long)w[1] << 32 | w[0];
    }
    __syncthreads();
    // r = H x - l x over the nonzero entries of H: a spin Hamiltonian in the product
    // basis is sparse (13 of 24 entries a row with two nuclei, an electron and a
    // muon), and the FP64 pipe is the bound
    for (int e = tid; e < n * n; e += nt) {
        const int i = FastDiv(n).div(e), j = e - i * n;
        const cx<double> *row = H + i * ld, *col = X + j;
        double r0 = 0.0, r1 = 0.0, i0 = 0.0, i1 = 0.0;
        for (unsigned long long w = s.nz[i]; w != 0; w &= w - 1) {
            const int k = __ffsll((long long)w) - 1;
            const cx<double> a = row[k], x = col[k * ld];
            r0 = fma(a.re, x.re, r0);
            r1 = fma(-a.im, x.im, r1);
            i0 = fma(a.re, x.im, i0);
            i1 = fma(a.im, x.re, i1);
        }
        const double l = s.lam0[j];
        const cx<double> x = X[i * ld + j];
        RF[e] = mk<float>((float)(fma(-l, x.re, r0) + r1), (float)(fma(-l, x.im, i0) + i1));
    }
    __syncthreads();
    // column norms (FP64) and level corrections, four threads per column
    float lmax = 0.f;
    for (int e = tid; e < 4 * ((n + 7) & ~7); e += nt) {
        const int j = e >> 2, part = e & 3;
        const unsigned mask = 0xffffffffu;  // whole warps run the loop
        double g = part == 0 ? -1.0 : 0.0;
        float d = 0.f;
        if (j < n)
            for (int k = part; k < n; k += 4) {
                const cx<double> x = X[k * ld + j];
                const cx<float> xf = XF[k * n + j], r = RF[k * n + j];
                g = fma(x.re, x.re, fma(x.im, x.im, g));
                d = fmaf(xf.re, r.re, fmaf(xf.im, r.im, d));
            }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            g += __shfl_xor_sync(mask, g, o);
            d += __shfl_xor_sync(mask, d, o);
        }
        if (part == 0 && j < n) {
            s.gn[j] = g;
            s.lam[j] = s.lam0[j] + (double)(d / (1.0f + (float)g));
            lmax = fmaxf(lmax, fabsf((float)s.lam[j]));
        }
    }
    if (lmax > 0.f) atomicMax(&s.scal[1], __float_as_int(lmax));
    // couplings B_ij = x_i^H r_j (over H, which nobody reads any more)
    cx<float> *B = reinterpret_cast<cx<float> *>(s.D1);
    float amax = 0.f;
    for (int e = tid; e < n * n; e += nt) {
        const int i = FastDiv(n).div(e), j = e - i * n;
        cx<float> v = mk<float>(0.f, 0.f);
        for (int k = 0; k < n; ++k) {
            const cx<float> x = XF[k * n + i], r = RF[k * n + j];
            v.re = fmaf(x.re, r.re, fmaf(x.im, r.im, v.re));
            v.im = fmaf(x.re, r.im, fmaf(-x.im, r.re, v.im));
        }
        B[e] = v;
        const float w = fabsf(v.re) + fabsf(v.im);
        if (i != j) amax = max_or_nan(amax, w);
    }
    atomicMax(&s.scal[0], __float_as_int(amax));  // NaN: above every number
    __syncthreads();
    const float big = __int_as_float(s.scal[0]);
    if (!(big < CUDART_INF_F)) return CUDART_INF_F;
    // ascending order, ties by index; runs of gaps up to 100 couplings
    for (int i = tid; i < n; i += nt) {
        const int r = level_rank(s.lam, n, i);
        s.rk[i] = r;
        s.ord[r] = i;
    }
    __syncthreads();
    const float gamma = 100.0f * big;
    for (int q = tid; q < n; q += nt) {
        int c = q;
        while (c > 0 && (float)(s.lam[s.ord[c]] - s.lam[s.ord[c - 1]]) <= gamma) --c;
        s.cst[q] = c;
    }
    __syncthreads();
    // couplings inside clusters, sorted coordinates (over r)
    cx<float> *T = RF;
    for (int e = tid; e < n * n; e += nt) {
        const int i = FastDiv(n).div(e), j = e - i * n;
        const int ri = s.rk[i], rj = s.rk[j];
        if (s.cst[ri] != s.cst[rj] || i == j) continue;
        const cx<float> b = B[i * n + j], c = B[j * n + i];
        T[ri * n + rj] = mk<float>(0.5f * (b.re + c.re), 0.5f * (b.im - c.im));
    }
    __syncthreads();
    // E (next to B) and second-order level terms, four threads per column.
    // With c = (B + B^H) / 2, E_ij = c_ij / (l_j - l_i) - (X^H X)_ij / 2: B_ij /
    // (l_j - l_i) is that too, but carries B's rounding (eps |H|) divided by the
    // gap into X's orthonormality, so close levels take X^H X in FP64.
    cx<float> *EX = B + n * n;
    const float close = __int_as_float(s.scal[1]) * (1.0f / 32.0f);
    float emax = 0.f;
    for (int e = tid; e < 4 * ((n + 7) & ~7); e += nt) {
        const int j = e >> 2, part = e & 3;
        const unsigned mask = 0xffffffffu;  // whole warps run the loop
        float corr = 0.f;
        if (j < n) {
            const double lj = s.lam[j];
            const int cj = s.cst[s.rk[j]];
            for (int i = part; i < n; i += 4) {
                const cx<float> b = B[i * n + j];
                const float gap = (float)(lj - s.lam[i]);
                const bool same = s.cst[s.rk[i]] == cj;
                cx<float> E = mk<float>(0.f, 0.f);
                if (i == j) {
                    E.re = -0.5f * (float)s.gn[j];
                } else {
                    const float inv = same ? 0.f : 1.0f / gap;
                    corr += (b.re * b.re + b.im * b.im) * inv;
                    if (same || fabsf(gap) < close) {
                        double gr = 0.0, gi = 0.0;
                        for (int k = 0; k < n; ++k) {
                            const cx<double> x = X[k * ld + i], y = X[k * ld + j];
                            gr = fma(x.re, y.re, fma(x.im, y.im, gr));
                            gi = fma(x.re, y.im, fma(-x.im, y.re, gi));
                        }
                        const cx<float> c = B[j * n + i];
                        E.re = 0.5f * ((b.re + c.re) * inv - (float)gr);
                        E.im = 0.5f * ((b.im - c.im) * inv - (float)gi);
                    } else {
                        E.re = b.re * inv;
                        E.im = b.im * inv;
                    }
                }
                const float w = fabsf(E.re) + fabsf(E.im);
                emax = max_or_nan(emax, w);
                EX[i * n + j] = E;
            }
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) corr += __shfl_xor_sync(mask, corr, o);
        if (part == 0 && j < n) s.corr[j] = corr;
    }
    atomicMax(&s.scal[2], __float_as_int(emax));
    __syncthreads();
    for (int r = tid; r < n; r += nt) {
        const int i = s.ord[r];
        if (oa_in_cluster(s.cst, n, r))
            s.tdiag[r] = (s.lam[i] - s.lam[s.ord[s.cst[r]]]) + (double)s.corr[i];
    }
    // X += X E
    for (int e = tid; e < n * n; e += nt) {
        const int k = FastDiv(n).div(e), j = e - k * n;
        float ar = 0.f, ai = 0.f;
        for (int i = 0; i < n; ++i) {
            const cx<float> x = XF[k * n + i], E = EX[i * n + j];
            ar = fmaf(x.re, E.re, fmaf(-x.im, E.im, ar));
            ai = fmaf(x.re, E.im, fmaf(x.im, E.re, ai));
        }
        X[k * ld + j].re += (double)ar;
        X[k * ld + j].im += (double)ai;
    }
    __syncthreads();
    // levels outside clusters; the clusters' own (reading lam of their first
    // level, which only their warp writes)
    for (int r = tid; r < n; r += nt)
        if (!oa_in_cluster(s.cst, n, r)) s.lam[s.ord[r]] += (double)s.corr[s.ord[r]];
    oa_resolve64(s.cst, s.ord, s.lam, s.tdiag, T, X, n, ld, 1e-15f * __int_as_float(s.scal[1]),
                 tid >> 5, (nt + 31) >> 5);
    __syncthreads();
    const float step = __int_as_float(s.scal[2]);
    __syncthreads();
    return step;
}

// FP64 eigenpairs of one Hamiltonian: levels in s.lam, vectors in s.D0 (row
// stride m + 1).  The FP32 refinement's buffers hold the matrix and, in
// f.w.U, the FP32 eigenvectors, whose status is `st`.  One copy for all
// kernels; it carves shared memory itself so that its accesses stay
// shared-memory accesses.
__noinline__ __device__ int eigenpairs64(int n, int fac_len, const HSource h, int st,
                                         int max_sweeps, bool swapped) {
    extern __shared__ __align__(16) char smem[];
    const int tid = threadIdx.x, nt = blockDim.x, m = n + (n & 1), ld = m + 1;
    S64 s = carve64(smem, n, fac_len);
    SnapSmem<float> f = snap_carve<float, true>(s.region, n, false, 0);
    if (swapped) {  // the FP32 Jacobi leaves its vectors in the other buffer
        cx<float> *t = f.w.H;
        f.w.H = f.w.U;
        f.w.U = t;
    }
    // squares and products of the FP32 stages must neither overflow nor vanish
    float hn = 0.f;
    bool ok = st == MSP_ITEM_OK;
    for (int i = 0; i < n; ++i) {
        ok = ok && f.rn[i] < 1e12f;  // false for a NaN
        hn = fmaxf(hn, f.rn[i]);
    }
    ok = ok && hn > 1e-12f;
    if (ok) {
        for (int it = 0; it < 4; ++it) {
            const float e = s.xl == nullptr ? oa_refine<0>(f, n, m)
                            : n == 24       ? oa_refine<24, true>(f, n, m, s.xl)
                            : n == 32       ? oa_refine<32, true>(f, n, m, s.xl)
                                            : oa_refine<0, true>(f, n, m, s.xl);
            if (e <= 5e-5f) break;
        }
        for (int j = tid; j < n; j += nt) s.lam0[j] = dw_to_double(f.lw[j]);
        __syncthreads();  // lw lies under D0
        for (int e = tid; e < n * n; e += nt) {
            const int i = FastDiv(n).div(e), j = e - i * n;
            const cx<float> x = f.w.U[i * ld + j];
            cx<double> v = mk<double>(x.re, x.im);
            if (s.xl) {
                const cx<float> l = s.xl[i * ld + j];
                v.re += (double)l.re;
                v.im += (double)l.im;
            }
            s.D0[i * ld + j] = v;
        }
        __syncthreads();
        ok = false;
        for (int it = 0; it < 3; ++it) {
            const float e = step64(s, h, n, m);
            if (!(e < 1e-2f)) break;
            if (e <= 4e-9f) {
                ok = true;
                break;
            }
            for (int j = tid; j < n; j += nt) s.lam0[j] = s.lam[j];
            __syncthreads();
        }
    }
    if (ok) return MSP_ITEM_OK;
    // FP64 Jacobi: matrix in D0, vectors in D1 (they swap), tables in D2
    __syncthreads();
    const SnapLayout J = snap_layout(n, 8, false, false, 0, (nt + 31) >> 5);
    JacobiWork<double> w;
    char *t = reinterpret_cast<char *>(s.D2) - J.rot;
    w.H = s.D0;
    w.U = s.D1;
    w.rot = reinterpret_cast<JRot<double> *>(t + J.rot);
    w.dia = reinterpret_cast<double *>(t + J.dia);
    w.red = reinterpret_cast<double *>(t + J.red);
    w.tab = reinterpret_cast<uint2 *>(t + J.tab);
    w.diag = reinterpret_cast<double *>(t + J.diag);
    load_h64(h, n, m, jacobi_ldh(m), w.H);
    __syncthreads();
    st = jacobi_sweeps<double>(w, m, max_sweeps);
    for (int j = tid; j < n; j += nt) s.lam[j] = w.diag[j];
    __syncthreads();
    return st;
}

// The same for n <= S64_DIRECT_MAX: one FP64 rotation, by every warp.
__noinline__ __device__ int eigenpair64(int n, int fac_len, const HSource h, int max_sweeps) {
    extern __shared__ __align__(16) char smem[];
    const S64 s = carve64(smem, n, fac_len);
    const int tid = threadIdx.x, lane = tid & 31;
    cx<double> v = mk<double>(0.0, 0.0);  // entries 00, 01, 11 of lanes 0, 1, 2
    if (lane < n * (n + 1) / 2) v = h_entry(h, (size_t)n * n, lane < 2 ? lane : 3);
    const double h0 = __shfl_sync(0xffffffffu, v.re, 0), h1 = __shfl_sync(0xffffffffu, v.re, 2);
    const cx<double> b =
        mk<double>(__shfl_sync(0xffffffffu, v.re, 1), __shfl_sync(0xffffffffu, v.im, 1));
    const double tol = JacobiConst<double>::tol, off = 2.0 * cabs2(b), fro = h0 * h0 + h1 * h1 + off;
    JRot<double> R;
    double e0, e1;
    jacobi_rotation<double>(h0, h1, b, off <= tol * tol * fro || max_sweeps < 1 ? CUDART_INF : 0.0, 0, 1, R,
                            e0, e1);
    const bool ok = (off <= tol * tol * fro || max_sweeps > 0) && fro >= 0.0;  // false for a NaN
    if (tid == 0) {
        const int ld = n + (n & 1) + 1;
        s.lam[0] = e0;
        s.D0[0] = mk<double>(R.c, 0.0);
        if (n == 2) {
            s.lam[1] = e1;
            s.D0[1] = mk<double>(R.sr, R.si);
            s.D0[ld] = mk<double>(-R.sr, R.si);
            s.D0[ld + 1] = mk<double>(R.c, 0.0);
        }
    }
    __syncthreads();
    return ok ? MSP_ITEM_OK : MSP_ITEM_NOT_CONVERGED;
}

}  // namespace

// ------------------------------------------------------------------ eigh

__global__ void __maxnreg__(128)
    msp_eigh64_kernel(const cx<double> *__restrict__ Hin, int n, int batch, int max_sweeps,
                      double *__restrict__ evals, cx<double> *__restrict__ evecs,
                      int *__restrict__ status) {
    extern __shared__ __align__(16) char smem[];
    const int m = n + (n & 1), ld = m + 1, ldh = jacobi_ldh(m);
    S64 s = carve64(smem, n, 0);
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int bidx = blockIdx.x; bidx < batch; bidx += gridDim.x) {
        const HSource h = {Hin + (size_t)bidx * n * n, nullptr, nullptr};
        int st;
        if (n <= S64_DIRECT_MAX) {
            st = eigenpair64(n, 0, h, max_sweeps);
        } else {
            SnapSmem<float> f = snap_carve<float, true>(s.region, n, false, 0);
            for (int e = tid; e < m * (m + 1) / 2; e += nt) {
                int i, j;
                tri_index(e, j, i);  // j >= i
                cx<double> v = mk<double>(0.0, 0.0);
                if (j < n) v = h.Hsys[(size_t)i * n + j];
                if (i == j) v.im = 0.0;
                const cx<float> hi = mk<float>((float)v.re, (float)v.im);
                const cx<float> lo = mk<float>((float)(v.re - (double)hi.re), (float)(v.im - (double)hi.im));
                f.w.H[i * ldh + j] = hi;
                f.w.H[j * ldh + i] = conj(hi);
                f.Hh[i * ld + j] = hi;
                f.Hl[i * ld + j] = lo;
                if (i != j) {
                    f.Hh[j * ld + i] = conj(hi);
                    f.Hl[j * ld + i] = conj(lo);
                }
            }
            __syncthreads();
            hamiltonian_row_norms(f, n, m);
            st = jacobi_sweeps<float>(f.w, m, max_sweeps);
            st = eigenpairs64(n, 0, h, st, max_sweeps, true);
        }
        // ascending order, ties by index (stable)
        for (int j = tid; j < n; j += nt) {
            const double lj = s.lam[j];
            int r = 0;
            for (int k = 0; k < n; ++k) {
                const double lk = s.lam[k];
                r += (lk < lj) || (lk == lj && k < j);
            }
            evals[(size_t)bidx * n + r] = lj;
            s.rk[j] = r;
        }
        __syncthreads();
        cx<double> *Vb = evecs + (size_t)bidx * n * n;
        for (int e = tid; e < n * n; e += nt) {
            const int i = FastDiv(n).div(e), j = e - i * n;
            Vb[(size_t)i * n + s.rk[j]] = s.D0[i * ld + j];
        }
        if (tid == 0) status[bidx] = st;
        __syncthreads();
    }
}

// ------------------------------------------------------------------ snapshots

namespace {

// Stages 1-3 for snapshot sn of a launch (PRE: stage 1 ran in its own kernel
// and left its vectors and status).
template <bool PRE>
__device__ __forceinline__ int snapshot64(const SnapArgs &a, const SnapSource &src, int sn, S64 &s,
                                          int n, int m, int fac_len) {
    const HSource h = {src.Hsys, src.Z, a.field + 3 * (size_t)src.g};
    if (!PRE && n <= S64_DIRECT_MAX) return eigenpair64(n, fac_len, h, a.max_sweeps);
    SnapSmem<float> f = snap_carve<float, true>(s.region, n, false, 0);
    load_hamiltonian<PRE>(src.Hsys, src.Z, src.Hdw, src.Zdw, h.b, n, m, f);
    const int st = snap_eigvecs<PRE>(a, sn, src.g, n, m, m + 1, f);
    return eigenpairs64(n, fac_len, h, st, a.max_sweeps, !PRE);
}

// V (d x n, row stride ld) from U; `stride` is the muon digit's.  The caller
// follows with a barrier.
__device__ __forceinline__ void muon_project(const double *p, double norm, const cx<double> *U,
                                             cx<double> *V, int n, int ld, int stride) {
    const double px = p[0], py = p[1], pz = p[2];
    const bool up = pz >= 0.0;
    const double c = norm + fabs(pz);
    for (int e = threadIdx.x; e < n / 2 * n; e += blockDim.x) {
        const int i = FastDiv(n).div(e), k = e - i * n;
        const int hi = i / stride, base = (i + hi * stride) * ld + k;  // muon digit 0
        const cx<double> u0 = U[base], u1 = U[base + stride * ld];
        V[i * ld + k] = up ? cadd(cscale(c, u0), cmul(mk<double>(px, -py), u1))
                           : cadd(cmul(mk<double>(px, py), u0), cscale(c, u1));
    }
}

// (V^H V)_jk
__device__ __forceinline__ cx<double> muon_product(const cx<double> *V, int n, int ld, int j, int k) {
    double g0 = 0.0, g1 = 0.0, h0 = 0.0, h1 = 0.0;
#pragma unroll 4
    for (int i = 0; i < n / 2; ++i) {
        const cx<double> a = V[i * ld + j], b = V[i * ld + k];
        g0 = fma(a.re, b.re, g0);
        g1 = fma(a.im, b.im, g1);
        h0 = fma(a.re, b.im, h0);
        h1 = fma(-a.im, b.re, h1);
    }
    return mk<double>(g0 + g1, h0 + h1);
}

// Sum of every thread's v (all threads get it); begins with a barrier.
__device__ __forceinline__ double block_sum64(double v, double *red) {
    double z = 0.0;
    block_sum2(v, z, red);
    return v;
}

}  // namespace

// The muon-first T = inf shortcut (muspinsim/hamiltonian.py:166-217): A =
// |U^dag (sigma_p (x) 1_d) U|^2 and omega_jk = 2 pi (l_j - l_k) for j > k,
// scaled by 0.5 w / d, plus the constant 0.5 sum_j A_jj part.
template <bool PRE>
__global__ void __maxnreg__(80) msp_snap64_fast_kernel(SnapArgs a) {
    extern __shared__ __align__(16) char smem[];
    const int n = a.n, m = n + (n & 1), ld = m + 1, d = n / 2;
    S64 s = carve64(smem, n, 0);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int P = n * (n - 1) / 2, ntri = n * (n + 1) / 2;
    double2 *coef = reinterpret_cast<double2 *>(a.pair_coef);
    __shared__ MuonAxis axis;
    for (int sn = blockIdx.x; sn < a.num_snap; sn += gridDim.x) {
        const SnapSource src = snap_source(a, sn);
        const size_t g = (size_t)src.g;
        if (tid == nt - 1) axis = muon_axis(a.pol + 3 * g);  // read many barriers later
        const int st = snapshot64<PRE>(a, src, sn, s, n, m, 0);
        // sigma_p = p . sigma (Pauli) on the muon (slowest) digit
        cx<double> *V = s.D1;
        muon_project(a.pol + 3 * g, axis.norm, s.D0, V, n, ld, d);
        __syncthreads();
        const double scale = 0.5 * a.wscale[g] / (double)d, inv = axis.inv, norm = axis.norm;
        double diag = 0.0;
        for (int e = tid; e < ntri; e += nt) {
            int j, k;
            tri_index(e, j, k);
            const cx<double> G = muon_product(V, n, ld, j, k);
            const double gr = fma(inv, G.re, j == k ? -norm : 0.0), gi = inv * G.im;
            const double A = gr * gr + gi * gi;
            if (j == k) {
                diag += A;
            } else {
                const size_t o = (size_t)sn * P + pair_index(j, k);
                coef[o] = make_double2(scale * A, 0.0);
                store_frequency(a, o, 6.283185307179586476925 * (s.lam[j] - s.lam[k]));
            }
        }
        diag = block_sum64(diag, s.red);
        if (tid == 0) {
            a.snap_const[sn] = scale * 0.5 * diag;
            a.status[g] = st;
        }
        __syncthreads();
    }
}

// The general path: rho' = U^dag rho0 U, O' = U^dag O U with rho0 = (x)_s
// rho_s (Kronecker factors) and O = p . S_mu.  EVOLVE writes the pair
// coefficients of <O>(t) = sum_ij rho'_ij O'_ji exp(-i w_ij t)
// (muspinsim/hamiltonian.py:80-107); INTEGRAL writes the decaying integral
// divided by tau (muspinsim/hamiltonian.py:150-164, experiment.py:492-496).
// At T = inf rho' follows from O' (rho_is_hot).
template <bool INTEGRAL, bool PRE>
__global__ void __maxnreg__(96) msp_snap64_rho_kernel(SnapArgs a) {
    extern __shared__ __align__(16) char smem[];
    const int n = a.n, m = n + (n & 1), ld = m + 1;
    S64 s = carve64(smem, n, a.fac_len);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int P = n * (n - 1) / 2, ntri = n * (n + 1) / 2;
    double2 *coef = reinterpret_cast<double2 *>(a.pair_coef);
    const double twopi = 6.283185307179586476925, inv_tau = INTEGRAL ? 1.0 / a.tau : 0.0;
    __shared__ MuonAxis axis;
    __shared__ double axis_hot;
    for (int sn = blockIdx.x; sn < a.num_snap; sn += gridDim.x) {
        const bool hot = rho_is_hot(a, sn);
        if (tid == nt - 1) {  // read many barriers later
            axis = muon_axis(a.pol + 3 * (size_t)sn);
            axis_hot = axis.norm > 0.0 ? 2.0 / (axis.norm * n) : 0.0;  // rho_hot_scale
        }
        if (a.rho_fac) {
            for (int e = tid; e < a.fac_len; e += nt)
                s.fac[e] = a.rho_fac[(size_t)sn * a.fac_len + e];
        } else if (!hot) {
            build_rho_factors(a, sn, s.fac);
        }
        SnapSource src;
        src.g = sn;
        src.Hsys = a.Hsys;
        src.Z = a.Z;
        src.Hdw = a.Hsys_dw;
        src.Zdw = a.Z_dw;
        const int st = snapshot64<PRE>(a, src, sn, s, n, m, a.fac_len);
        const cx<double> *U = s.D0;
        const cx<double> *X = s.D1;
        cx<double> *Y = s.D2;
        if (!hot) {
            // rho0 U by Kronecker factors: X ping-pongs between D1 and D2
            X = U;
            Y = s.D1;
            int off = 0;
            for (int sp = 0; sp < a.num_spins; ++sp) {
                const int dim = a.dims[sp];
                apply_digit<double>(s.fac + off, dim, a.strides[sp], X, Y, n, ld);
                off += dim * dim;
                X = Y;
                Y = (Y == s.D1) ? s.D2 : s.D1;
            }
            // rho'_jk (j >= k) into the other buffer
            tri_conj_products<double>(U, X, Y, n);
            __syncthreads();
        }
        // O = p . S on the muon digit: half of sigma_p.  V into the buffer X (free now)
        cx<double> *V = const_cast<cx<double> *>(X);
        muon_project(a.pol + 3 * (size_t)sn, axis.norm, U, V, n, ld, a.strides[a.mu_index]);
        __syncthreads();
        const double scale = a.wscale[sn], hs = axis_hot, inv = 0.5 * axis.inv, norm = 0.5 * axis.norm;
        double local = 0.0;
        for (int e = tid; e < ntri; e += nt) {
            int j, k;
            tri_index(e, j, k);
            // O'_kj
            const cx<double> G = muon_product(V, n, ld, k, j);
            const double orr = fma(inv, G.re, j == k ? -norm : 0.0), oii = inv * G.im;
            // rho'_jk, at T = inf from O'_jk
            const cx<double> r = hot ? mk<double>(fma(hs, orr, j == k ? 1.0 / n : 0.0), -hs * oii)
                                     : Y[j * ld + k];
            // C_jk = rho'_jk O'_kj
            const double cr = r.re * orr - r.im * oii, ci = r.re * oii + r.im * orr;
            if (INTEGRAL) {
                // term = C_jk (-1) / (2 pi i (l_k - l_j) - 1/tau); pairs count twice
                if (j == k) {
                    local += cr * a.tau;
                } else {
                    const double x = twopi * (s.lam[k] - s.lam[j]);
                    // -C / (-1/tau + i x) = C (1/tau + i x) / (1/tau^2 + x^2)
                    const double den = inv_tau * inv_tau + x * x;
                    local += 2.0 * (cr * inv_tau - ci * x) / den;
                }
            } else if (j == k) {
                local += cr;
            } else {
                const size_t o = (size_t)sn * P + pair_index(j, k);
                coef[o] = make_double2(2.0 * scale * cr, 2.0 * scale * ci);
                store_frequency(a, o, twopi * (s.lam[j] - s.lam[k]));
            }
        }
        local = block_sum64(local, s.red);
        if (tid == 0) {
            a.snap_const[sn] = INTEGRAL ? scale * local / a.tau : scale * local;
            a.status[sn] = st;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ launchers

size_t snap64_smem_bytes(int n, int fac_len, int threads) {
    return snap64_layout(n, fac_len, threads / 32).total;
}

template <typename K>
static cudaError_t launch64(K kernel, const SnapArgs &a, int grid, int threads, size_t smem,
                            cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}

int snap64_occupancy(int n, int threads, bool pre) {
    const size_t smem = snap64_smem_bytes(n, 0, threads);
    const void *k = pre ? (const void *)msp_snap64_fast_kernel<true>
                        : (const void *)msp_snap64_fast_kernel<false>;
    int blocks = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return blocks > 0 ? blocks : 1;
}

// pre: the FP32 eigenvectors are in a.evec (launch_jacobi_warp).
cudaError_t launch_snapshots64(const SnapArgs &a, int mode, bool pre, cudaStream_t st, int threads,
                               int grid) {
    const size_t smem = snap64_smem_bytes(a.n, mode == MSP_MODE_FAST ? 0 : a.fac_len, threads);
    if (mode == MSP_MODE_FAST)
        return pre ? launch64(msp_snap64_fast_kernel<true>, a, grid, threads, smem, st)
                   : launch64(msp_snap64_fast_kernel<false>, a, grid, threads, smem, st);
    if (mode == MSP_MODE_EVOLVE)
        return pre ? launch64(msp_snap64_rho_kernel<false, true>, a, grid, threads, smem, st)
                   : launch64(msp_snap64_rho_kernel<false, false>, a, grid, threads, smem, st);
    return pre ? launch64(msp_snap64_rho_kernel<true, true>, a, grid, threads, smem, st)
               : launch64(msp_snap64_rho_kernel<true, false>, a, grid, threads, smem, st);
}

cudaError_t launch_eigh64(const double *H, int n, int batch, int max_sweeps, double *evals,
                          double *evecs, int *status, cudaStream_t st) {
    const int threads = jacobi_threads(n + (n & 1));
    const size_t smem = snap64_smem_bytes(n, 0, threads);
    cudaError_t e = cudaFuncSetAttribute(msp_eigh64_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    msp_eigh64_kernel<<<batch, threads, smem, st>>>(reinterpret_cast<const cx<double> *>(H), n,
                                                    batch, max_sweeps, evals,
                                                    reinterpret_cast<cx<double> *>(evecs), status);
    return cudaGetLastError();
}

}  // namespace msp
