// The fast path for 64 < n <= MSP_MAX_DIM_LARGE (muspinsim/hamiltonian.py:
// 166-217, muspinsim/spinop.py:51-82): refinement of the FP32 eigenvectors of
// msp_large_solve.cu, then M = U^H (sigma_p (x) 1_d) U and the pair records.
//
// Refinement steps (T. Ogita and K. Aishima, Japan J. Indust. Appl. Math. 35
// (2018) 1007, Algorithm 1, Hermitian form, with exact rotations inside
// clusters of near-degenerate levels, msp_cluster.cuh), in residual form:
//   l_j = x_j^H H x_j / x_j^H x_j,  r_j = H x_j - l_j x_j,  B = X^H R,
//   E_ij = B_ij / (l_j - l_i),  E_jj = (1 - x_j^H x_j) / 2,  X <- X + X E,
// eigenvalues l_j plus the second-order term (B_ij is the S_ij + l_j R_ij of
// the paper, with S = X^H H X and R = I - X^H X).  H X and the Rayleigh quotients are
// accumulated in double-word FP32 from an anchor (msp_dw.cuh); H itself is
// held as hi + lo.  r_j is small, so B and X E are plain FP32 sums: one
// double-word product per step where S and R would take two more.
// Eigenvalues come out FP64-accurate, eigenvectors to FP32 rounding: the MIXED
// result.  FP64 keeps the last correction's low words and
// goes on with the FP64 step of the n <= 64 kernels (msp_snap64.cu):
//   r_j = H x_j - l_j x_j in FP64 (4 n FMAs per entry of H that is not zero), everything after it except
//   norms in FP32, because r_j is small,
// until its correction is below 2e-8, and forms M in FP64 (2 n^3
// FMAs).  A snapshot that does not get there is left to the FP64 solver
// (msp_large.cu).
//
// One thread-block cluster of 1 to 8 CTAs works on a snapshot: the tiles of a
// product, the pairs of levels and the clusters of levels are dealt out to its
// CTAs, the matrices pass through the snapshot's global scratch, and vectors
// (norms, levels, sums) lie in every CTA's shared memory, written by whoever
// computes them through distributed shared memory.
#include <cooperative_groups.h>

#include "msp_cluster.cuh"
#include "msp_large.cuh"
#include "msp_large_slots.cuh"
#include "msp_rho.cuh"

namespace msp {

namespace cg = cooperative_groups;

namespace {

// The CTAs of one snapshot.
struct Team {
    int rank, size;
    __device__ __forceinline__ Team() {
        const cg::cluster_group c = cg::this_cluster();
        rank = (int)c.block_rank();
        size = (int)c.num_blocks();
    }
    // All threads of all CTAs; global and shared writes before it are seen
    // after it.
    __device__ __forceinline__ void sync() const {
        if (size == 1) {
            __syncthreads();
        } else {
            __threadfence();
            cg::this_cluster().sync();
        }
    }
    template <typename T>
    __device__ __forceinline__ T *of(T *p, int r) const {
        return size == 1 ? p : cg::this_cluster().map_shared_rank(p, r);
    }
    // *p = v in every CTA
    template <typename T>
    __device__ __forceinline__ void put(T *p, T v) const {
        for (int r = 0; r < size; ++r) *of(p, r) = v;
    }
    // *p = max(*p, bits of v) in every CTA, v >= 0 (or NaN: above every number)
    __device__ __forceinline__ void put_max(int *p, float v) const {
        const int m = __reduce_max_sync(0xffffffffu, __float_as_int(v));
        if ((threadIdx.x & 31) == 0)
            for (int r = 0; r < size; ++r) atomicMax(of(p, r), m);
    }
};

// ------------------------------------------------------------------ shared memory

struct LmVec {
    double *lam64, *lam0, *gn, *tdiag;  // FP64 step
    float2 *lam;                        // eigenvalues as double-words
    int *rank, *order, *cstart;         // clusters of levels (msp_cluster.cuh)
    float *corr, *rn, *cn, *gf;
    int *scal;     // [0]: largest correction, [1]: largest |l_i|, [2]: largest coupling (float
                   // bits), [3]: nonzeros of H's fullest row
    double *dsum;  // one per CTA of the team
    char *slab;    // two stages of GEMM slabs
};

__host__ __device__ inline size_t lm_vec_bytes(int n, bool fp64) {
    return (((fp64 ? 32 : 0) + 36) * (size_t)n + 16 + 8 * 8 + 15) & ~size_t(15);
}

__host__ __device__ inline size_t lm_smem_bytes(int n, int threads, bool fp64) {
    return lm_vec_bytes(n, fp64) + 2 * lm_stage_bytes(threads);
}

__device__ __forceinline__ LmVec lm_vec(char *smem, int n, bool fp64) {
    LmVec v;
    v.dsum = reinterpret_cast<double *>(smem);
    v.lam64 = v.dsum + 8;
    v.lam0 = v.lam64 + n;
    v.gn = v.lam0 + n;
    v.tdiag = v.gn + n;
    v.lam = fp64 ? reinterpret_cast<float2 *>(v.tdiag + n) : reinterpret_cast<float2 *>(v.lam64);
    v.rank = reinterpret_cast<int *>(v.lam + n);
    v.order = v.rank + n;
    v.cstart = v.order + n;
    v.corr = reinterpret_cast<float *>(v.cstart + n);
    v.rn = v.corr + n;
    v.cn = v.rn + n;
    v.gf = v.cn + n;
    v.scal = reinterpret_cast<int *>(v.gf + n);
    v.slab = smem + lm_vec_bytes(n, fp64);
    return v;
}

// Column 2-norms of X into `out` of every CTA: 32 columns per CTA and turn,
// rows over the warps.
__device__ void lm_colnorms(const float2 *X, int n, float *out, const LmVec &v, const Team &team) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float *part = reinterpret_cast<float *>(v.slab);
    for (int g = team.rank; 32 * g < n; g += team.size) {
        const int j = 32 * g + lane;
        float acc = 0.f;
        if (j < n) {
#pragma unroll 8
            for (int k = warp; k < n; k += nw) {
                const float2 e = X[(size_t)k * n + j];
                acc = fmaf(e.x, e.x, fmaf(e.y, e.y, acc));
            }
        }
        part[32 * warp + lane] = acc;
        __syncthreads();
        if (warp == 0 && j < n) {
            for (int w = 1; w < nw; ++w) acc += part[32 * w + lane];
            team.put(out + j, sqrtf(acc));
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ rows of H

// A spin Hamiltonian in the product basis is sparse: a term reaches the states
// that differ in one or two spins (19 of 96 entries a row for five nuclei and
// spins with an electron and a muon, 22 of 192 for six).  H X skips the zeros of H: its
// rows are compacted in place, the nonzero entries first, the column of entry q in
// the 4-byte word 2 + q from the row's end and their number in the last word.
// Only where no row has more than n / 2 of them, so that both fit (fuller ones stay
// dense for the tiled product): 192 snapshots of n = 192 in 8.05 ms at n / 2 - 1
// entries a row against 8.13 for the tiled product at n / 2 + 1, 96 of n = 96 in
// 1.51 against 1.64 (all stages, MIXED).  Batch of 21 systems up to n = 192: 9.6 -> 8.0
// ms; n = 96 in FP64, where the FP64 pipe is the bound: 2.45 -> 2.07 ms.

__device__ __forceinline__ bool lm_nonzero(const float4 &h) {
    return !(h.x == 0.f && h.y == 0.f && h.z == 0.f && h.w == 0.f);  // true for a NaN
}
__device__ __forceinline__ bool lm_nonzero(const cx<double> &h) { return !(h.re == 0.0 && h.im == 0.0); }

// Compacts H (n x n, seen by the team) where it is sparse and says whether it was;
// *most is zero in every CTA.  A warp per row; n <= 1024, so lane c can keep the
// nonzeros of columns 32 c .. 32 c + 31.
template <typename T>
__device__ bool lm_compact(T *H, int n, int *most, const Team &team) {
    static_assert(sizeof(T) == 16, "room for the columns");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int me = team.rank * nw + warp, all = team.size * nw;
    int fullest = 0;
    for (int i = me; i < n; i += all) {
        int cnt = 0;
#pragma unroll 4
        for (int k0 = 0; k0 < n; k0 += 32)
            cnt += __popc(__ballot_sync(0xffffffffu, k0 + lane < n && lm_nonzero(H[(size_t)i * n + min(k0 + lane, n - 1)])));
        fullest = max(fullest, cnt);
    }
    if (lane == 0)
        for (int r = 0; r < team.size; ++r) atomicMax(team.of(most, r), fullest);
    team.sync();
    if (2 * *most > n) return false;  // the same in every CTA
    for (int i = me; i < n; i += all) {
        T *row = H + (size_t)i * n;
        unsigned mine = 0;
        int cnt = 0;
        for (int k0 = 0; k0 < n; k0 += 32) {
            const T h = row[min(k0 + lane, n - 1)];
            const bool nz = k0 + lane < n && lm_nonzero(h);
            const unsigned b = __ballot_sync(0xffffffffu, nz);  // everyone has read
            if (lane == k0 >> 5) mine = b;
            if (nz) row[cnt + __popc(b & ((1u << lane) - 1))] = h;
            cnt += __popc(b);
            __syncwarp();
        }
        int *tail = reinterpret_cast<int *>(row + n);
        int q = 0;
        for (int k0 = 0; k0 < n; k0 += 32) {
            const unsigned b = __shfl_sync(0xffffffffu, mine, k0 >> 5);
            if (b >> lane & 1) tail[-2 - (q + __popc(b & ((1u << lane) - 1)))] = k0 + lane;
            q += __popc(b);
        }
        if (lane == 0) tail[-1] = cnt;
    }
    team.sync();
    return true;
}

// H X by compacted rows: a warp makes 64 columns of a row, two per lane, so that an
// entry of H serves both; X comes through L1 / L2 in whole rows.  init(i, j) starts a
// sum, step(sum, h, x) adds a product, epi(i, j, sum) consumes it.
template <typename T, typename X, typename Init, typename Step, typename Epi>
__device__ __forceinline__ void lm_sparse_rows(const T *H, const X *x, int n, const Team &team,
                                               Init init, Step step, Epi epi) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int groups = (n + 63) >> 6;
    for (int u = team.rank * nw + warp; u < n * groups; u += team.size * nw) {
        const int i = u / groups, j = (u - i * groups) * 64 + lane;
        const bool two = j - lane + 32 < n;  // the same in the whole warp
        const int ja = min(j, n - 1), jb = min(j + 32, n - 1);
        const T *row = H + (size_t)i * n;
        const int *tail = reinterpret_cast<const int *>(row + n);
        const int cnt = tail[-1];
        auto a = init(i, ja), b = init(i, jb);
#pragma unroll 4
        for (int q = 0; q < cnt; ++q) {
            const T h = row[q];
            const X *xk = x + (size_t)tail[-2 - q] * n;
            step(a, h, xk[ja]);
            if (two) step(b, h, xk[jb]);
        }
        if (j < n) epi(i, j, a);
        if (j + 32 < n) epi(i, j + 32, b);
    }
}

// ------------------------------------------------------------------ double-word step

struct LmSum {
    u64 s1, c1, s2, c2;
};

// Rayleigh quotients and residuals from Y = H X: v.lam, v.gf = x_j^H x_j - 1
// (in every CTA) and R = Y - X diag(l), 32 columns per CTA and turn, rows over
// the warps.
__device__ void lm_residuals(const LargeSlot &s, const cx<float> *X, const LmVec &v, int n,
                             const Team &team) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float *part = reinterpret_cast<float *>(v.slab);
    float2 *dots = reinterpret_cast<float2 *>(part + 32 * nw);  // x^H y, then x^H x - 1
    const u64 *Xp = reinterpret_cast<const u64 *>(X);
    for (int g = team.rank; 32 * g < n; g += team.size) {
        const int j = 32 * g + lane, jc = min(j, n - 1);
        float acc = 0.f;
#pragma unroll 8
        for (int k = warp; k < n; k += nw) {
            const float4 y = s.Y[(size_t)k * n + jc];
            acc = fmaf(y.x, y.x, fmaf(y.y, y.y, acc));
        }
        part[32 * warp + lane] = acc;
        __syncthreads();
        acc = 0.f;
        for (int w = 0; w < nw; ++w) acc += part[32 * w + lane];
        const float cn = v.cn[jc];
        const u64 Ky = lm_anchor(cn * sqrtf(acc)), Kx = lm_anchor(cn * cn);
        u64 sy = Ky, cy = 0ull, sx = Kx, cc = 0ull;
#pragma unroll 4
        for (int k = warp; k < n; k += nw) {
            const u64 x = Xp[(size_t)k * n + jc];
            u64 yh, yl;
            lm_pairs(&s.Y[(size_t)k * n + jc], yh, yl);
            dw_dot(sy, cy, x, yh, yl);
            dw_dot(sx, cc, x, x, 0ull);
        }
        dots[64 * warp + lane] = dw_dot_value(sy, cy, Ky);
        dots[64 * warp + 32 + lane] = dw_dot_value(sx, cc, Kx);
        __syncthreads();
        float2 xy = dots[lane], xx = dots[32 + lane];
        for (int w = 1; w < nw; ++w) {
            const float2 a = dots[64 * w + lane], b = dots[64 * w + 32 + lane];
            dw_add(xy.x, xy.y, a.x, a.y);
            dw_add(xx.x, xx.y, b.x, b.y);
        }
        xx = dw_add_f(dw_two_sum(xx.x, xx.y), -1.0f);
        const float2 l = dw_rayleigh(dw_two_sum(xy.x, xy.y), xx);
        if (warp == 0 && j < n) {
            team.put(v.lam + j, l);
            team.put(v.gf + j, xx.x + xx.y);
        }
        if (j < n) {
#pragma unroll 4
            for (int k = warp; k < n; k += nw) {
                const size_t o = (size_t)k * n + j;
                const float4 y = s.Y[o];
                const cx<float> x = X[o];
                s.R[o] = mk<float>(fmaf(-l.x, x.re, y.x) + fmaf(-l.y, x.re, y.z),
                                   fmaf(-l.x, x.im, y.y) + fmaf(-l.y, x.im, y.w));
            }
        }
        __syncthreads();
    }
}

// (X^H X)_ij, i != j, to FP32 rounding, by a warp: rows over the lanes.
__device__ cx<float> lm_gram(const cx<float> *X, int n, int i, int j, float bound) {
    const u64 K = lm_anchor(bound);
    u64 s1 = K, c1 = 0ull, s2 = K, c2 = 0ull;
    for (int k = threadIdx.x & 31; k < n; k += 32) {
        const u64 x = *reinterpret_cast<const u64 *>(X + (size_t)k * n + i);
        const cx<float> y = X[(size_t)k * n + j];
        lm_step<false, false>(s1, c1, s2, c2, x, 0ull, f32x2(y.re, y.re), f32x2(y.im, y.im), 0ull, 0ull);
    }
    float4 r = lm_dw<true>(s1, c1, s2, c2, K);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        dw_add(r.x, r.z, __shfl_xor_sync(0xffffffffu, r.x, o), __shfl_xor_sync(0xffffffffu, r.z, o));
        dw_add(r.y, r.w, __shfl_xor_sync(0xffffffffu, r.y, o), __shfl_xor_sync(0xffffffffu, r.w, o));
    }
    return mk<float>(r.x + r.z, r.y + r.w);
}

// The same in FP64.
__device__ cx<float> lm_gram64(const cx<double> *X, int n, int i, int j) {
    double re = 0.0, im = 0.0;
    for (int k = threadIdx.x & 31; k < n; k += 32) {
        const cx<double> x = X[(size_t)k * n + i], y = X[(size_t)k * n + j];
        re = fma(x.re, y.re, fma(x.im, y.im, re));
        im = fma(x.re, y.im, fma(-x.im, y.re, im));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    return mk<float>((float)re, (float)im);
}

// visit(i, j, gram) for every pair i < j of levels, in this order: the warps of
// the team take the j in turn, the lanes i (in whole groups of 32: on = i < j).
// Where want(i, j) asks for it, gram(i, j), a warp-wide computation, comes first.
template <typename Want, typename Gram, typename Visit>
__device__ __forceinline__ void lm_pairs_of(int n, const Team &team, Want want, Gram gram, Visit visit) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // the longest rows first
    for (int j = n - 1 - (team.rank * nw + warp); j > 0; j -= team.size * nw) {
        for (int i0 = 0; i0 < j; i0 += 32) {
            const int i = i0 + lane;
            const bool on = i < j;
            cx<float> G = mk<float>(0.f, 0.f);
            unsigned need = __ballot_sync(0xffffffffu, on && want(i, j));
            while (need) {
                const int l = __ffs(need) - 1;
                need &= need - 1;
                const cx<float> g = gram(i0 + l, j);
                if (lane == l) G = g;
            }
            if (on) visit(i, j, G);
        }
    }
}

// out[0][j] = sum_i first(i, j), out[1][j] = sum_i second(i, j) (where given) into
// every CTA: 32 columns per CTA and turn, rows over the warps.  The order of the sums
// is fixed, so that results repeat bit for bit.
template <int NS, typename Term>
__device__ void lm_column_sums(int n, float *const (&out)[NS], const LmVec &v, const Team &team, Term term) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float *part = reinterpret_cast<float *>(v.slab);
    for (int g = team.rank; 32 * g < n; g += team.size) {
        const int j = 32 * g + lane;
        float acc[NS] = {};
        if (j < n)
            for (int i = warp; i < n; i += nw) term(i, j, acc);
#pragma unroll
        for (int q = 0; q < NS; ++q) part[(q * nw + warp) * 32 + lane] = acc[q];
        __syncthreads();
        if (warp == 0 && j < n) {
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                for (int w = 1; w < nw; ++w) acc[q] += part[(q * nw + w) * 32 + lane];
                team.put(out[q] + j, acc[q]);
            }
        }
        __syncthreads();
    }
}

// The CTA whose warp resolves the cluster that starts at sorted position q0,
// when the warps of the team take the starts in turn.
__device__ __forceinline__ int lm_owner(int q0, const Team &team) {
    const int nw = blockDim.x >> 5;
    return q0 % (team.size * nw) / nw;
}

// One refinement step of the eigenvector columns X into X2 (LO: its low words
// into Xl) and of the eigenvalues v.lam, clusters resolved as in the n <= 64
// refinement (msp_cluster.cuh).  Y holds the couplings B, then E in their
// place, and T behind them.  Returns the step's largest correction.
// sparse: H is compacted.
template <bool LO>
__device__ float lm_refine(const LargeSlot &s, const cx<float> *X, cx<float> *X2, const LmVec &v,
                           int n, bool sparse, const Team &team) {
    const int tid = threadIdx.x, nt = blockDim.x, nw = nt >> 5, warp = tid >> 5;
    const float2 *Xf = reinterpret_cast<const float2 *>(X);
    if (tid < 3) v.scal[tid] = 0;
    lm_colnorms(Xf, n, v.cn, v, team);
    team.sync();
    // Y = H X
    auto bound = [&](int i, int j) { return v.rn[min(i, n - 1)] * v.cn[min(j, n - 1)]; };
    if (sparse)
        lm_sparse_rows(
            s.H, Xf, n, team,
            [&](int i, int j) {
                const u64 K = lm_anchor(bound(i, j));
                return LmSum{K, 0ull, K, 0ull};
            },
            [](LmSum &t, const float4 &h, const float2 &x) {
                lm_step<true, false>(t.s1, t.c1, t.s2, t.c2, f32x2(h.x, h.y), f32x2(h.z, h.w),
                                     f32x2(x.x, x.x), f32x2(x.y, x.y), 0ull, 0ull);
            },
            [&](int i, int j, const LmSum &t) {
                s.Y[(size_t)i * n + j] = lm_dw<false>(t.s1, t.c1, t.s2, t.c2, lm_anchor(bound(i, j)));
            });
    else
        lm_tiles<LM_DW_ALO, false>(
            n, n, n, s.H, n, Xf, n, v.slab, team.rank, team.size, [](int, int) { return false; },
            [&](int i, int j, u64 &s1, u64 &, u64 &s2, u64 &) { s1 = s2 = lm_anchor(bound(i, j)); },
            [&](int i, int j, u64 s1, u64 c1, u64 s2, u64 c2) {
                s.Y[(size_t)i * n + j] = lm_dw<false>(s1, c1, s2, c2, lm_anchor(bound(i, j)));
            });
    team.sync();
    lm_residuals(s, X, v, n, team);
    team.sync();
    // B, and its transpose in X2, so that both couplings of a pair are read in rows
    cx<float> *B = reinterpret_cast<cx<float> *>(s.Y), *Bt = X2;
    float amax = 0.f;
    lm_tiles<LM_PLAIN_C, true>(
        n, n, n, Xf, n, reinterpret_cast<const float2 *>(s.R), n, v.slab, team.rank, team.size,
        [](int, int) { return false; }, [](int, int, u64 &, u64 &, u64 &, u64 &) {},
        [&](int i, int j, u64 s1, u64, u64 s2, u64) {
            const cx<float> b = lm_plain<true>(s1, s2);
            B[(size_t)i * n + j] = b;
            Bt[(size_t)j * n + i] = b;
            if (i != j) amax = fmaxf(amax, fmaxf(fabsf(b.re), fabsf(b.im)));
        });
    team.put_max(&v.scal[2], amax);
    float lmax = 0.f;
    for (int i = tid; i < n; i += nt) lmax = fmaxf(lmax, fabsf(v.lam[i].x));
    atomicMax(&v.scal[1], __float_as_int(lmax));  // the same in every CTA
    team.sync();
    OaCluster cl;
    cl.rank = v.rank;
    cl.order = v.order;
    cl.cstart = v.cstart;
    cl.scal = v.scal + 2;
    cl.T = B + (size_t)n * n;
    cl.ldt = n;
    oa_cluster_starts(v.lam, n, cl);
    float emax = 0.f;
    auto same = [&](int i, int j) { return v.cstart[v.rank[i]] == v.cstart[v.rank[j]]; };
    lm_pairs_of(
        n, team, same, [&](int i, int j) { return lm_gram(X, n, i, j, v.cn[i] * v.cn[j]); },
        [&](int i, int j, cx<float> G) {
            const size_t lo = (size_t)j * n + i, up = (size_t)i * n + j;
            const cx<float> b = Bt[lo], c = B[lo];  // B_ij, B_ji
            cx<float> Eij, Eji;
            if (same(i, j)) {
                const int ri = v.rank[i], rj = v.rank[j];
                const cx<float> t = mk<float>(0.5f * (b.re + c.re), 0.5f * (b.im - c.im));
                cl.T[(size_t)ri * n + rj] = t;
                cl.T[(size_t)rj * n + ri] = conj(t);
                Eij = mk<float>(-0.5f * G.re, -0.5f * G.im);
                Eji = conj(Eij);
            } else {
                const float inv = 1.0f / dw_sub_f(v.lam[j], v.lam[i]);
                Eij = mk<float>(b.re * inv, b.im * inv);
                Eji = mk<float>(-c.re * inv, -c.im * inv);
                emax = fmaxf(emax, fmaxf(fmaxf(fabsf(Eij.re), fabsf(Eij.im)),
                                         fmaxf(fabsf(Eji.re), fabsf(Eji.im))));
            }
            B[up] = Eij;
            B[lo] = Eji;
        });
    for (int j = team.rank * nt + tid; j < n; j += team.size * nt)
        B[(size_t)j * n + j] = mk<float>(-0.5f * v.gf[j], 0.f);
    team.sync();
    // second-order terms of the levels: |E_ij|^2 (l_j - l_i) over other clusters
    {
        float *const out[1] = {v.corr};
        lm_column_sums<1>(n, out, v, team, [&](int i, int j, float (&acc)[1]) {
            if (!same(i, j))
                acc[0] = fmaf(cabs2(B[(size_t)i * n + j]), dw_sub_f(v.lam[j], v.lam[i]), acc[0]);
        });
    }
    team.sync();
    // every CTA writes the same diagonal of T
    oa_cluster_diagonal(v.lam, v.corr, n, cl);
    // X2 = X + X E
    lm_tiles<LM_PLAIN, false>(
        n, n, n, Xf, n, reinterpret_cast<const float2 *>(B), n, v.slab, team.rank, team.size,
        [](int, int) { return false; },
        [&](int i, int j, u64 &s1, u64 &, u64 &, u64 &) {
            if (LO) return;
            const cx<float> x = i < n && j < n ? X[(size_t)i * n + j] : mk<float>(0.f, 0.f);
            s1 = f32x2(x.re, x.im);
        },
        [&](int i, int j, u64 s1, u64, u64 s2, u64) {
            const size_t o = (size_t)i * n + j;
            const cx<float> y = lm_plain<false>(s1, s2);
            if (LO) {
                const cx<float> x = X[o];
                const float2 re = dw_two_sum(x.re, y.re), im = dw_two_sum(x.im, y.im);
                X2[o] = mk<float>(re.x, im.x);
                s.Xl[o] = mk<float>(re.y, im.y);
            } else {
                X2[o] = y;
            }
        });
    team.sync();
    emax = fmaxf(emax, oa_resolve_clusters(X2, n, n, v.lam, v.corr, n, cl,
                                           __int_as_float(v.scal[1]), LO ? s.Xl : nullptr,
                                           team.rank * nw + warp, team.size * nw));
    team.put_max(&v.scal[0], emax);
    team.sync();
    // the levels of clusters that other CTAs resolved
    for (int r = tid; r < n; r += nt) {
        if (!oa_in_cluster(v.cstart, n, r)) continue;
        const int o = lm_owner(v.cstart[r], team), i = v.order[r];
        if (o != team.rank) v.lam[i] = team.of(v.lam, o)[i];
    }
    const float step = __int_as_float(v.scal[0]);
    team.sync();  // before anyone resets scal or replaces lam
    return step;
}

// ------------------------------------------------------------------ FP64 step

// Products whose FP64 operands come straight out of L1 / L2: a warp makes 4
// rows x 32 columns, 16 FMAs per five loads, and the FP64 pipe (one warp-wide
// FMA per 18 clocks and SM) is the bound.  The warps of the team take the
// blocks in turn; drop(i0, j0) leaves one out, load(i, k) gives an entry of
// the row operand, B[0 .. NB - 1] are row-major column operands of `depth` rows, epi(i, j, re, im)
// consumes their results.
template <int NB, typename Drop, typename Load, typename Epi>
__device__ __forceinline__ void fp64_blocks(int n, int depth, const cx<double> *const (&B)[NB], const Team &team,
                                            Drop drop, Load load, Epi epi) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int ti = (n + 3) >> 2, tj = (n + 31) >> 5, me = team.rank * nw + warp, all = team.size * nw;
    int turn = -1;
    for (int t = 0; t < ti * tj; ++t) {
        const int i0 = t / tj * 4, j = (t % tj) * 32 + lane;
        if (drop(i0, j - lane)) continue;
        if (++turn == all) turn = 0;
        if (turn != me) continue;
        double re[4][NB], im[4][NB];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < NB; ++c) re[q][c] = im[q][c] = 0.0;
        const int jc = min(j, n - 1);
#pragma unroll 2
        for (int k = 0; k < depth; ++k) {
            cx<double> b[NB];
#pragma unroll
            for (int c = 0; c < NB; ++c) b[c] = B[c][(size_t)k * n + jc];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const cx<double> a = load(min(i0 + q, n - 1), k);
#pragma unroll
                for (int c = 0; c < NB; ++c) {
                    re[q][c] = fma(a.re, b[c].re, re[q][c]);
                    im[q][c] = fma(a.re, b[c].im, im[q][c]);
                    re[q][c] = fma(-a.im, b[c].im, re[q][c]);
                    im[q][c] = fma(a.im, b[c].re, im[q][c]);
                }
            }
        }
        if (j < n)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (i0 + q < n) epi(i0 + q, j, re[q], im[q]);
    }
}

// One FP64 step (the maths of step64 in msp_snap64.cu) on the vectors X64 and
// the levels v.lam0: v.lam64 and X64 corrected.  H in FP64; XF the vectors in
// FP32; R, B and Bt n x n scratch (the couplings, which the corrections replace, and
// their transpose; T, the couplings inside clusters, takes R's place).  Returns the largest column norm of E (NaN or infinite when the input is
// unusable): the step leaves an error of that order squared.  sparse: H is compacted.
__device__ float lm_step64(const cx<double> *H, cx<double> *X64, const cx<float> *XF, cx<float> *R,
                           cx<float> *B, cx<float> *Bt, const LmVec &v, int n, bool sparse,
                           const Team &team) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int me = team.rank * nt + tid, all = team.size * nt;
    if (tid < 3) v.scal[tid] = 0;
    // r = H x - l x
    auto residual = [&](int i, int j, double re, double im) {
        const size_t o = (size_t)i * n + j;
        const cx<double> x = X64[o];
        const double l = v.lam0[j];
        R[o] = mk<float>((float)fma(-l, x.re, re), (float)fma(-l, x.im, im));
    };
    if (sparse) {
        lm_sparse_rows(
            H, X64, n, team, [](int, int) { return mk<double>(0.0, 0.0); },
            [](cx<double> &t, const cx<double> &h, const cx<double> &x) {
                t.re = fma(h.re, x.re, t.re);
                t.im = fma(h.re, x.im, t.im);
                t.re = fma(-h.im, x.im, t.re);
                t.im = fma(h.im, x.re, t.im);
            },
            [&](int i, int j, const cx<double> &t) { residual(i, j, t.re, t.im); });
    } else {
        const cx<double> *const x64[1] = {X64};
        fp64_blocks<1>(
            n, n, x64, team, [](int, int) { return false; },
            [&](int i, int k) { return H[(size_t)i * n + k]; },
            [&](int i, int j, const double *re, const double *im) { residual(i, j, re[0], im[0]); });
    }
    team.sync();
    // column norms (FP64) and level corrections, a thread per column and part
    // of the rows
    {
        double *pg = reinterpret_cast<double *>(v.slab);
        float *pd = reinterpret_cast<float *>(pg + nt);
        for (int g = team.rank; 32 * g < n; g += team.size) {
            const int j = 32 * g + lane;
            double gs = warp == 0 ? -1.0 : 0.0;
            float d = 0.f;
            if (j < n)
                for (int k = warp; k < n; k += nw) {
                    const size_t o = (size_t)k * n + j;
                    const cx<double> x = X64[o];
                    const cx<float> xf = XF[o], r = R[o];
                    gs = fma(x.re, x.re, fma(x.im, x.im, gs));
                    d = fmaf(xf.re, r.re, fmaf(xf.im, r.im, d));
                }
            pg[tid] = gs;
            pd[tid] = d;
            __syncthreads();
            if (warp == 0 && j < n) {
                for (int w = 1; w < nw; ++w) {
                    gs += pg[32 * w + lane];
                    d += pd[32 * w + lane];
                }
                team.put(v.gn + j, gs);
                team.put(v.lam64 + j, v.lam0[j] + (double)(d / (1.0f + (float)gs)));
            }
            __syncthreads();
        }
    }
    // couplings B_ij = x_i^H r_j
    float amax = 0.f;
    lm_tiles<LM_PLAIN_C, true>(
        n, n, n, reinterpret_cast<const float2 *>(XF), n, reinterpret_cast<const float2 *>(R), n,
        v.slab, team.rank, team.size, [](int, int) { return false; },
        [](int, int, u64 &, u64 &, u64 &, u64 &) {},
        [&](int i, int j, u64 s1, u64, u64 s2, u64) {
            const cx<float> b = lm_plain<true>(s1, s2);
            B[(size_t)i * n + j] = b;
            Bt[(size_t)j * n + i] = b;
            const float w = fabsf(b.re) + fabsf(b.im);
            if (i != j) amax = max_or_nan(amax, w);
        });
    team.put_max(&v.scal[2], amax);
    team.sync();
    const float big = __int_as_float(v.scal[2]);
    if (!(big < CUDART_INF_F)) return CUDART_INF_F;  // the same in every CTA
    // ascending order, ties by index; runs of gaps up to 100 couplings
    float lmax = 0.f;
    for (int i = tid; i < n; i += nt) {
        const int r = level_rank(v.lam64, n, i);
        v.rank[i] = r;
        v.order[r] = i;
        lmax = fmaxf(lmax, fabsf((float)v.lam64[i]));
    }
    atomicMax(&v.scal[1], __float_as_int(lmax));
    __syncthreads();
    const float gamma = 100.0f * big;
    for (int q = tid; q < n; q += nt) {
        int c = q;
        while (c > 0 && (float)(v.lam64[v.order[c]] - v.lam64[v.order[c - 1]]) <= gamma) --c;
        v.cstart[q] = c;
    }
    __syncthreads();
    // E, T and the second-order level terms.  With c = (B + B^H) / 2, E_ij =
    // c_ij / (l_j - l_i) - (X^H X)_ij / 2; B_ij / (l_j - l_i) is that too, but
    // carries B's rounding divided by the gap into X's orthonormality, so close
    // levels take X^H X in FP64.
    cx<float> *T = R;
    const float close = __int_as_float(v.scal[1]) * (1.0f / 32.0f);
    auto same = [&](int i, int j) { return v.cstart[v.rank[i]] == v.cstart[v.rank[j]]; };
    auto gap_of = [&](int i, int j) { return (float)(v.lam64[j] - v.lam64[i]); };
    lm_pairs_of(
        n, team, [&](int i, int j) { return fabsf(gap_of(i, j)) < close || same(i, j); },
        [&](int i, int j) { return lm_gram64(X64, n, i, j); },
        [&](int i, int j, cx<float> G) {
            const size_t lo = (size_t)j * n + i, up = (size_t)i * n + j;
            const cx<float> b = Bt[lo], c = B[lo];  // B_ij, B_ji
            const float gap = gap_of(i, j);
            const bool one = same(i, j);
            const float inv = one ? 0.f : 1.0f / gap;
            cx<float> Eij = mk<float>(b.re * inv, b.im * inv);
            cx<float> Eji = mk<float>(-c.re * inv, -c.im * inv);
            if (one || fabsf(gap) < close) {
                Eij = mk<float>(0.5f * ((b.re + c.re) * inv - G.re), 0.5f * ((b.im - c.im) * inv - G.im));
                Eji = mk<float>(0.5f * (-(b.re + c.re) * inv - G.re), 0.5f * ((b.im - c.im) * inv + G.im));
            }
            if (one) {
                const int ri = v.rank[i], rj = v.rank[j];
                const cx<float> t = mk<float>(0.5f * (b.re + c.re), 0.5f * (b.im - c.im));
                T[(size_t)ri * n + rj] = t;
                T[(size_t)rj * n + ri] = conj(t);
            }
            B[up] = Eij;
            B[lo] = Eji;
        });
    for (int j = me; j < n; j += all) B[(size_t)j * n + j] = mk<float>(-0.5f * (float)v.gn[j], 0.f);
    team.sync();
    // second-order terms of the levels and squared column norms of E (over cn, which
    // the double-word steps have used)
    float *const norm = v.cn;
    {
        float *const out[2] = {v.corr, norm};
        lm_column_sums<2>(n, out, v, team, [&](int i, int j, float (&acc)[2]) {
            const float e2 = cabs2(B[(size_t)i * n + j]);
            if (!same(i, j)) acc[0] = fmaf(e2, gap_of(i, j), acc[0]);
            acc[1] += e2;
        });
    }
    team.sync();
    float emax = 0.f;
    for (int j = tid; j < n; j += nt) emax = max_or_nan(emax, norm[j]);
    atomicMax(&v.scal[0], __float_as_int(emax));  // the same in every CTA
    for (int r = tid; r < n; r += nt) {
        const int i = v.order[r];
        if (oa_in_cluster(v.cstart, n, r))
            v.tdiag[r] = (v.lam64[i] - v.lam64[v.order[v.cstart[r]]]) + (double)v.corr[i];
    }
    // X += X E
    lm_tiles<LM_PLAIN, false>(
        n, n, n, reinterpret_cast<const float2 *>(XF), n, reinterpret_cast<const float2 *>(B), n,
        v.slab, team.rank, team.size, [](int, int) { return false; },
        [](int, int, u64 &, u64 &, u64 &, u64 &) {},
        [&](int i, int j, u64 s1, u64, u64 s2, u64) {
            const cx<float> y = lm_plain<false>(s1, s2);
            cx<double> &x = X64[(size_t)i * n + j];
            x = mk<double>(x.re + (double)y.re, x.im + (double)y.im);
        });
    team.sync();
    for (int r = tid; r < n; r += nt)
        if (!oa_in_cluster(v.cstart, n, r)) v.lam64[v.order[r]] += (double)v.corr[v.order[r]];
    oa_resolve64(v.cstart, v.order, v.lam64, v.tdiag, T, X64, n, n,
                 1e-15f * __int_as_float(v.scal[1]), team.rank * nw + warp, team.size * nw);
    team.sync();
    for (int r = tid; r < n; r += nt) {
        if (!oa_in_cluster(v.cstart, n, r)) continue;
        const int o = lm_owner(v.cstart[r], team), i = v.order[r];
        if (o != team.rank) v.lam64[i] = team.of(v.lam64, o)[i];
    }
    const float step = sqrtf(__int_as_float(v.scal[0]));
    team.sync();
    return step;
}

// ------------------------------------------------------------------ pair records

// Pair record of the mixed path: FP32 coefficient and, from the level gap
// d (double-word), the double-word phases on a uniform grid or the FP64
// frequency otherwise.
__device__ __forceinline__ void lm_store_pair(const SnapArgs &a, size_t o, float cA, float2 d) {
    reinterpret_cast<float2 *>(a.pair_coef)[o] = make_float2(cA, 0.f);
    if (a.pair_phase) {
        const float2 psi = dw_phase_mod2pi(d, a.c_dt);
        const float2 ph0 = a.t0_zero ? make_float2(0.f, 0.f) : dw_phase_mod2pi(d, a.c_t0);
        a.pair_phase[o] = make_float4(psi.x, psi.y, ph0.x, ph0.y);
    } else {
        a.pair_omega[o] = 6.283185307179586476925 * dw_to_double(d);
    }
}

// W = (sigma_p (x) 1_d) X
template <typename T>
__device__ void lm_pauli(const cx<T> *X, cx<T> *W, int n, const double *pol, const Team &team) {
    const int d = n / 2;
    const T px = (T)pol[0], py = (T)pol[1], pz = (T)pol[2];
    for (int x = team.rank * blockDim.x + threadIdx.x; x < d * n; x += team.size * blockDim.x) {
        const cx<T> u0 = X[x], u1 = X[x + (size_t)d * n];
        W[x] = mk<T>(pz * u0.re + px * u1.re + py * u1.im, pz * u0.im + px * u1.im - py * u1.re);
        W[x + (size_t)d * n] =
            mk<T>(px * u0.re - py * u0.im - pz * u1.re, px * u0.im + py * u0.re - pz * u1.im);
    }
}

// The sum over the team of a thread's share, in thread 0 of CTA 0.
__device__ double team_sum(double x, double *dsum, const Team &team) {
    __shared__ double red[32];
    x = block_sum(x, red);
    if (threadIdx.x == 0) team.of(dsum, 0)[team.rank] = x;
    team.sync();
    double t = 0.0;
    if (team.rank == 0 && threadIdx.x == 0)
        for (int r = 0; r < team.size; ++r) t += dsum[r];
    return t;
}

// ------------------------------------------------------------------ kernel

// MIXED: refinement steps until the correction drops below 2e-4 (at most
// a.max_refine; one step leaves an error of order E^2); M in FP32; pair records
// with frequencies from the refined eigenvalues.  FP64: double-word steps until
// 6e-5 (four at most), then FP64 steps until 2e-8 (three at most); the vectors
// stay in the slot's Y, the levels in its R, for the pair kernels, and
// redo[slot] asks for the FP64 solver.
// Bound by issue in the plain products; H X skips the zeros of H (4.1 ms for 192
// snapshots of n = 192 MIXED where it did not, 2.4 ms now).
template <bool FP64>
__global__ void __maxnreg__(128)
    msp_large_refine_kernel(SnapArgs a, char *scratch, size_t per, int first, int *redo) {
    extern __shared__ __align__(16) char smem[];
    const Team team;
    const int n = a.n, slot = blockIdx.x / team.size;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int me = team.rank * nt + tid, all = team.size * nt, nn = n * n;
    const LargeSlot s = large_slot(scratch, per, slot, n);
    const LmVec v = lm_vec(smem, n, FP64);
    const int sn = first + slot;
    const SnapSource src = snap_source(a, sn);
    const size_t g = (size_t)src.g;
    int st = s.ql->status;
    if (tid == 0) v.scal[3] = 0;
    team.sync();  // every CTA of the team runs before its shared memory is written
    // row norms of H
    for (int i = team.rank * nw + warp; i < n; i += team.size * nw) {
        float acc = 0.f;
        for (int k = lane; k < n; k += 32) {
            const float4 h = s.H[(size_t)i * n + k];
            acc = fmaf(h.x, h.x, fmaf(h.y, h.y, acc));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) team.put(v.rn + i, sqrtf(acc));
    }
    bool sparse = lm_compact(s.H, n, v.scal + 3, team);  // behind a team barrier
    cx<float> *X = s.X, *X2 = s.X2;
    const int max_refine = FP64 || a.max_refine <= 0 ? 4 : a.max_refine;
    bool ok = true;
    if (FP64) {
        // squares and products of the FP32 stages must neither overflow nor vanish
        float hn = 0.f;
        for (int i = 0; i < n; ++i) {
            ok = ok && v.rn[i] < 1e12f;  // false for a NaN
            hn = fmaxf(hn, v.rn[i]);
        }
        ok = ok && hn > 1e-12f && st == MSP_ITEM_OK;
    }
    st |= MSP_ITEM_REFINE_LIMIT;
    for (int it = 0; ok && it < max_refine; ++it) {
        const float step = lm_refine<FP64>(s, X, X2, v, n, sparse, team);
        cx<float> *t = X;
        X = X2;
        X2 = t;
        if (step <= (FP64 ? 6e-5f : 2e-4f)) {
            st &= ~MSP_ITEM_REFINE_LIMIT;
            break;
        }
    }
    if (FP64) {
        cx<double> *H = reinterpret_cast<cx<double> *>(s.H), *X64 = reinterpret_cast<cx<double> *>(s.Y);
        if (ok) {
            if (tid == 0) v.scal[3] = 0;  // read before the first step
            for (int j = tid; j < n; j += nt) v.lam0[j] = dw_to_double(v.lam[j]);
            const double bx = a.field[3 * g], by = a.field[3 * g + 1], bz = a.field[3 * g + 2];
            for (int x = me; x < nn; x += all) {
                const int i = x / n, j = x - i * n;
                const cx<float> hi = X[x], lo = s.Xl[x];
                X64[x] = mk<double>((double)hi.re + (double)lo.re, (double)hi.im + (double)lo.im);
                if (j > i) continue;
                const cx<double> hs = src.Hsys[x], z0 = src.Z[x], z1 = src.Z[nn + x],
                                 z2 = src.Z[2 * (size_t)nn + x];
                cx<double> h = mk<double>(hs.re + bx * z0.re + by * z1.re + bz * z2.re,
                                          hs.im + bx * z0.im + by * z1.im + bz * z2.im);
                if (i == j) h.im = 0.0;
                H[x] = h;
                H[(size_t)j * n + i] = conj(h);
            }
            team.sync();
            sparse = lm_compact(H, n, v.scal + 3, team);
            ok = false;
            for (int it = 0; it < 3; ++it) {
                const float step = lm_step64(H, X64, X, s.R, X2, s.Xl, v, n, sparse, team);
                if (!(step < 1e-2f)) break;
                if (step <= 2e-8f) {
                    ok = true;
                    break;
                }
                for (int j = tid; j < n; j += nt) v.lam0[j] = v.lam64[j];
                for (int x = me; x < nn; x += all) X[x] = mk<float>((float)X64[x].re, (float)X64[x].im);
                team.sync();
            }
        }
        if (team.rank == 0) {
            double *lam = reinterpret_cast<double *>(s.R);
            for (int j = tid; j < n; j += nt) lam[j] = v.lam64[j];
            if (tid == 0) redo[slot] = !ok;
        }
        return;  // the last team barrier is behind every shared access
    }
    // W into X2; G = X^H W (tiles with an entry j >= k only); A_jk = |G_jk|^2
    lm_pauli(X, X2, n, a.pol + 3 * g, team);
    team.sync();
    const double scale = 0.5 * a.wscale[g] / (double)(n / 2);
    double diag = 0.0;
    const float scale_f = (float)scale;
    const int tr = 4 * nw;
    const size_t rec = (size_t)sn * (n * (n - 1) / 2);
    lm_tiles<LM_PLAIN_C, true>(
        n, n, n, reinterpret_cast<const float2 *>(X), n, reinterpret_cast<const float2 *>(X2), n,
        v.slab, team.rank, team.size, [=](int i0, int j0) { return i0 + tr - 1 < j0; },
        [](int, int, u64 &, u64 &, u64 &, u64 &) {},
        [&](int j, int k, u64 s1, u64, u64 s2, u64) {
            if (j < k) return;
            const cx<float> G = lm_plain<true>(s1, s2);
            const float Am = G.re * G.re + G.im * G.im;
            if (j == k)
                diag += (double)Am;
            else
                lm_store_pair(a, rec + (size_t)j * (j - 1) / 2 + k, scale_f * Am,
                              dw_sub(v.lam[j], v.lam[k]));
        });
    diag = team_sum(diag, v.dsum, team);
    if (me == 0) {
        a.snap_const[sn] = scale * 0.5 * diag;
        a.status[g] = st;
    }
}

// FP64 pairs: A_jk = |G_jk|^2 for j >= k, G = V^H V / (|p| + |p_z|) - |p| 1 (MuonAxis) with
// the n / 2 rows of V in the slot's H.  n^3 FP64 FMAs per snapshot, bound by the FP64
// pipe; 2 n^3 as U^H sigma U: 49 of n = 96 2.07 ms in all against 1.85.
__global__ void __maxnreg__(128)
    msp_large_fast_pairs_kernel(SnapArgs a, char *scratch, size_t per, int first, const int *redo) {
    const Team team;
    const int n = a.n, slot = blockIdx.x / team.size, sn = first + slot;
    if (redo[slot]) return;  // the same in the whole team
    const LargeSlot s = large_slot(scratch, per, slot, n);
    const size_t g = (size_t)snap_source(a, sn).g, rec = (size_t)sn * (n * (n - 1) / 2);
    const cx<double> *X = reinterpret_cast<const cx<double> *>(s.Y);
    cx<double> *W = reinterpret_cast<cx<double> *>(s.H);
    const double *lam = reinterpret_cast<const double *>(s.R);
    const int d = n / 2;
    const double *p = a.pol + 3 * g;
    __shared__ MuonAxis axis;
    if (threadIdx.x == 0) axis = muon_axis(p);
    __syncthreads();
    const double norm = axis.norm, inv = axis.inv, c = norm + fabs(p[2]);
    const bool up = p[2] >= 0.0;
    for (int x = team.rank * blockDim.x + threadIdx.x; x < d * n; x += team.size * blockDim.x) {
        const cx<double> u0 = X[x], u1 = X[x + (size_t)d * n];
        W[x] = up ? cadd(cscale(c, u0), cmul(mk<double>(p[0], -p[1]), u1))
                  : cadd(cmul(mk<double>(p[0], p[1]), u0), cscale(c, u1));
    }
    team.sync();
    const double scale = 0.5 * a.wscale[g] / (double)d;
    double diag = 0.0;
    const cx<double> *const w[1] = {W};
    fp64_blocks<1>(
        n, d, w, team, [](int j0, int k0) { return k0 > j0 + 3; },
        [&](int j, int i) { return conj(W[(size_t)i * n + j]); },
        [&](int j, int k, const double *re, const double *im) {
            if (j < k) return;
            const double gr = fma(inv, re[0], j == k ? -norm : 0.0), gi = inv * im[0];
            const double Am = gr * gr + gi * gi;
            if (j == k)
                diag += Am;
            else
                large_store_pair(a, rec + (size_t)j * (j - 1) / 2 + k, scale * Am,
                                 6.283185307179586476925 * (lam[j] - lam[k]));
        });
    __shared__ double dsum[8];
    diag = team_sum(diag, dsum, team);
    if (team.rank == 0 && threadIdx.x == 0) {
        a.snap_const[sn] = scale * 0.5 * diag;
        a.status[g] = MSP_ITEM_OK;
    }
}

// Y = (1 (x) F (x) 1) X on the digit of the given stride and size
__device__ void lm_apply_digit(const cx<double> *F, int dim, int stride, const cx<double> *X,
                               cx<double> *Y, int n, const Team &team) {
    for (int e = team.rank * blockDim.x + threadIdx.x; e < n * n; e += team.size * blockDim.x) {
        const int i = e / n, k = e - i * n;
        const int di = (i / stride) % dim, base = i - di * stride;
        double yr = 0, yi = 0;
        for (int l = 0; l < dim; ++l) {
            const cx<double> f = F[di * dim + l], x = X[(size_t)(base + l * stride) * n + k];
            yr += f.re * x.re - f.im * x.im;
            yi += f.re * x.im + f.im * x.re;
        }
        Y[e] = mk<double>(yr, yi);
    }
    team.sync();
}

// The general path (EVOLVE / INTEGRAL) from the FP64 eigenpairs: rho0's
// Kronecker factors, rho0 U factor by factor, O U on the muon digit (O = p .
// S_mu), then for j >= k rho'_jk = (U^dag rho0 U)_jk and O'_jk together (4 n^3
// FP64 FMAs), C_jk = rho'_jk O'_kj and its frequency, or the decaying integral.
// The slot's H and two more n x n complex matrices behind it hold the products.
template <bool INTEGRAL>
__global__ void __maxnreg__(128)
    msp_large_rho_pairs_kernel(SnapArgs a, char *scratch, size_t per, int first, const int *redo) {
    extern __shared__ __align__(16) char smem[];
    const Team team;
    const int n = a.n, slot = blockIdx.x / team.size, sn = first + slot, tid = threadIdx.x, nt = blockDim.x;
    if (redo[slot]) return;  // the same in the whole team
    const LargeSlot s = large_slot(scratch, per, slot, n);
    const size_t nn = (size_t)n * n, rec = (size_t)sn * (n * (n - 1) / 2);
    const cx<double> *U = reinterpret_cast<const cx<double> *>(s.Y);
    cx<double> *P0 = reinterpret_cast<cx<double> *>(s.H);
    cx<double> *P1 = reinterpret_cast<cx<double> *>(scratch + per * (size_t)slot + 64 * nn), *OU = P1 + nn;
    const double *lam = reinterpret_cast<const double *>(s.R);
    cx<double> *fac = reinterpret_cast<cx<double> *>(smem);
    if (a.rho_fac) {
        for (int e = tid; e < a.fac_len; e += nt) fac[e] = a.rho_fac[(size_t)sn * a.fac_len + e];
    } else {
        build_rho_factors(a, sn, fac);
    }
    __syncthreads();
    {
        const double px = a.pol[3 * (size_t)sn], py = a.pol[3 * (size_t)sn + 1],
                     pz = a.pol[3 * (size_t)sn + 2];
        const int stride = a.strides[a.mu_index];
        const cx<double> o00 = mk<double>(0.5 * pz, 0.0), o01 = mk<double>(0.5 * px, -0.5 * py);
        const cx<double> o10 = mk<double>(0.5 * px, 0.5 * py), o11 = mk<double>(-0.5 * pz, 0.0);
        for (int e = team.rank * nt + tid; e < (int)nn; e += team.size * nt) {
            const int i = e / n, k = e - i * n;
            const int di = (i / stride) & 1, b0 = i - di * stride;
            const cx<double> x0 = U[(size_t)b0 * n + k], x1 = U[(size_t)(b0 + stride) * n + k];
            OU[e] = di == 0 ? cadd(cmul(o00, x0), cmul(o01, x1)) : cadd(cmul(o10, x0), cmul(o11, x1));
        }
    }
    const cx<double> *X = U;
    cx<double> *Y = P0;
    int off = 0;
    for (int sp = 0; sp < a.num_spins; ++sp) {
        const int dim = a.dims[sp];
        lm_apply_digit(fac + off, dim, a.strides[sp], X, Y, n, team);
        off += dim * dim;
        X = Y;
        Y = Y == P0 ? P1 : P0;
    }
    const double twopi = 6.283185307179586476925, scale = a.wscale[sn];
    double local = 0.0;
    const cx<double> *const w[2] = {X, OU};
    fp64_blocks<2>(
        n, n, w, team, [](int j0, int k0) { return k0 > j0 + 3; },
        [&](int j, int i) { return conj(U[(size_t)i * n + j]); },
        [&](int j, int k, const double *re, const double *im) {
            if (j < k) return;
            // C_jk = rho'_jk O'_kj = rho'_jk conj(O'_jk)
            const double cr = re[0] * re[1] + im[0] * im[1], ci = im[0] * re[1] - re[0] * im[1];
            if (INTEGRAL) {
                // term = -C_jk / (2 pi i (l_k - l_j) - 1/tau); pairs count twice
                const double inv_tau = 1.0 / a.tau;
                if (j == k) {
                    local += cr * a.tau;
                } else {
                    const double x = twopi * (lam[k] - lam[j]);
                    local += 2.0 * (cr * inv_tau - ci * x) / (inv_tau * inv_tau + x * x);
                }
            } else if (j == k) {
                local += cr;
            } else {
                large_store_pair(a, rec + (size_t)j * (j - 1) / 2 + k, 2.0 * scale * cr,
                                 twopi * (lam[j] - lam[k]), 2.0 * scale * ci);
            }
        });
    __shared__ double dsum[8];
    local = team_sum(local, dsum, team);
    if (team.rank == 0 && tid == 0) {
        a.snap_const[sn] = INTEGRAL ? scale * local / a.tau : scale * local;
        a.status[sn] = MSP_ITEM_OK;
    }
}

// ------------------------------------------------------------------ host side

// One launch of a team kernel: `count` snapshots, `smem` bytes per CTA.  A CTA's
// share of a snapshot takes about as long alone on its SM as beside the others
// that fit (latency bounds it up to there), so a team of t CTAs takes 1 / t per
// round of teams: the team is the one with the smallest rounds / t.  (n = 192,
// 192 snapshots: 4.8 ms in two rounds of teams of seven, 5.5 ms in two of four or
// in one of two.)
template <typename... Params, typename... Args>
cudaError_t launch_team(void (*kernel)(Params...), int count, int threads, size_t smem,
                        cudaStream_t st, Args... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int occ = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem) != cudaSuccess ||
        occ < 1) {
        cudaGetLastError();
        occ = 1;
    }
    // a cluster lies in one of eight GPCs, taken as equal (if they are not, the choice
    // may cost a wave; the launch is valid either way)
    const int gpc = occ * large_sms() / 8 > 8 ? occ * large_sms() / 8 : 8;
    unsigned team = 1;
    double best = 1e300;
    for (unsigned t = 1; t <= 8; ++t) {
        const int fit = 8 * (gpc / (int)t);
        const double cost = (double)((count + fit - 1) / fit) / t;
        if (cost <= best) {
            best = cost;
            team = t;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)count * team);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = team;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Slots and flags of a run in `bytes` of scratch; 0 when not even one fits.
int fit_slots(int wanted, size_t per, size_t bytes) {
    const size_t fit = bytes / (per + sizeof(int));
    return (size_t)wanted < fit ? wanted : (int)fit;
}

// FP64 eigenpairs of chunk after chunk, each handed to `pairs`, what did not
// converge to `redo`.
template <typename Pairs, typename Redo>
cudaError_t run_fp64(const SnapArgs &a, char *base, size_t per, int slots, int threads,
                     cudaStream_t st, Pairs pairs, Redo redo) {
    int *flag = reinterpret_cast<int *>(base + per * (size_t)slots);
    for (int first = 0; first < a.num_snap; first += slots) {
        const int count = a.num_snap - first < slots ? a.num_snap - first : slots;
        cudaError_t e = launch_large_solve(a, base, per, first, count, st);
        if (e == cudaSuccess)
            e = launch_team(msp_large_refine_kernel<true>, count, threads,
                            lm_smem_bytes(a.n, threads, true), st, a, base, per, first, flag);
        if (e == cudaSuccess) e = pairs(first, count, flag);
        if (e == cudaSuccess) e = redo(first, count, flag);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

cudaError_t launch_large_fast(const SnapArgs &a, void *scratch, size_t bytes, int slots,
                              cudaStream_t st, int threads, int precision) {
    if (threads <= 0) threads = large_threads(a.n);
    if (threads & 31) return cudaErrorInvalidValue;
    const bool mixed = precision == MSP_PREC_MIXED;
    if (mixed && threads > 256) return cudaErrorInvalidValue;
    char *base = static_cast<char *>(scratch);
    const size_t per = large_slot_bytes(a.n, precision);
    if (mixed) {
        for (int first = 0; first < a.num_snap; first += slots) {
            const int count = a.num_snap - first < slots ? a.num_snap - first : slots;
            cudaError_t e = launch_large_solve(a, base, per, first, count, st);
            if (e == cudaSuccess)
                e = launch_team(msp_large_refine_kernel<false>, count, threads,
                                lm_smem_bytes(a.n, threads, false), st, a, base, per, first,
                                (int *)nullptr);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    double *solver = static_cast<double *>(scratch);
    slots = fit_slots(slots, per, bytes);
    if (slots < 1)  // the scratch of one FP64 solver
        return launch_large_fast64(a, solver, 1, st, threads, 0, a.num_snap, nullptr);
    const int nt = threads > 256 ? 256 : threads;
    return run_fp64(
        a, base, per, slots, nt, st,
        [&](int first, int count, const int *flag) {
            return launch_team(msp_large_fast_pairs_kernel, count, nt, 0, st, a, base, per, first, flag);
        },
        [&](int first, int count, const int *flag) {
            return launch_large_fast64(a, solver, count, st, threads, first, count, flag);
        });
}

cudaError_t launch_large_rho(const SnapArgs &a, void *scratch, size_t bytes, int slots,
                             cudaStream_t st, int integral) {
    char *base = static_cast<char *>(scratch);
    const int threads = large_threads(a.n);
    const size_t per = large_rho_slot_bytes(a.n);
    double *solver = static_cast<double *>(scratch);
    slots = fit_slots(slots, per, bytes);
    if (slots < 1) return launch_large_rho64(a, solver, 1, st, integral, 0, a.num_snap, nullptr);
    const size_t fac = (size_t)a.fac_len * sizeof(cx<double>);
    return run_fp64(
        a, base, per, slots, threads, st,
        [&](int first, int count, const int *flag) {
            return integral ? launch_team(msp_large_rho_pairs_kernel<true>, count, threads, fac, st, a,
                                          base, per, first, flag)
                            : launch_team(msp_large_rho_pairs_kernel<false>, count, threads, fac, st, a,
                                          base, per, first, flag);
        },
        [&](int first, int count, const int *flag) {
            return launch_large_rho64(a, solver, count, st, integral, first, count, flag);
        });
}

}  // namespace msp
