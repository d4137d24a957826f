// Shared parts of the fast path for 64 < n <= MSP_MAX_DIM_LARGE: the global
// scratch of one snapshot (a slot), and the tile engine of its n^3 products.
//
// A batch runs in chunks of as many snapshots as there are slots.  Each chunk
// passes through the FP32 eigensolver's kernels (msp_large_solve.cu), then the
// refinement kernel (msp_large_refine.cu), so that every stage has the grid
// that suits it: one CTA with the matrix in shared memory for the
// tridiagonalisation, one warp for the serial QL recurrence, many CTAs for
// everything that is parallel.
#pragma once

#include "msp_dw.cuh"
#include "msp_internal.cuh"

namespace msp {

// A slot, as byte offsets (nn = n^2).  H: the Hamiltonian as double-words
// (FP64 steps: as FP64); Y: H X as double-words, then couplings (FP64 steps:
// the FP64 vectors); R: residuals; X, X2: eigenvectors; Xl (FP64): their low
// words.  While the solver runs: V, row k = reflector k,
// in the first half of Y; the QL rotations over the second half of Y and R
// (the matrix of a global-memory tridiagonalisation lies there before them);
// Z^T in the first half of X2, the solver's vectors in its second half.
struct LargeSlot {
    float4 *H, *Y;
    cx<float> *R, *X, *X2, *Xl;
    cx<float> *V, *A;
    float2 *rot;
    float *Zt;
    float *d, *e;
    cx<float> *tau;
    struct QlState *ql;
};

// What the FP64 solver (msp_large.cu) does for the snapshots first .. first +
// count - 1: all of them (redo = NULL), or those with redo[sn - first] set.
cudaError_t launch_large_fast64(const SnapArgs &a, double *scratch, int grid, cudaStream_t st,
                                int threads, int first, int count, const int *redo);
cudaError_t launch_large_rho64(const SnapArgs &a, double *scratch, int grid, cudaStream_t st,
                               int integral, int first, int count, const int *redo);

// The QL recurrence between two rounds of its kernel.
struct QlState {
    int l, iter, status, done;
    int len;  // entries of the rotation stream of this round
};

constexpr int LARGE_QL_ROUNDS = 2;

__host__ __device__ inline size_t large_slot_bytes(int n, int precision) {
    const size_t nn = (size_t)n * n;
    return ((precision == MSP_PREC_MIXED ? 56 : 64) * nn + 255) & ~size_t(255);
}

// The general path's: two more FP64 matrices.
__host__ __device__ inline size_t large_rho_slot_bytes(int n) {
    return ((size_t)96 * n * n + 255) & ~size_t(255);
}

// Entries of the rotation stream.  QL takes some 0.85 n^2 rotations.
__host__ __device__ inline int large_rot_capacity(int n) { return 2 * n * n; }

__device__ __forceinline__ LargeSlot large_slot(char *scratch, size_t per, int slot, int n) {
    const size_t nn = (size_t)n * n;
    char *b = scratch + per * (size_t)slot;
    LargeSlot s;
    s.H = reinterpret_cast<float4 *>(b);
    s.Y = reinterpret_cast<float4 *>(b + 16 * nn);
    s.R = reinterpret_cast<cx<float> *>(b + 32 * nn);
    s.X = reinterpret_cast<cx<float> *>(b + 40 * nn);
    s.X2 = reinterpret_cast<cx<float> *>(b + 48 * nn);
    s.Xl = reinterpret_cast<cx<float> *>(b + 56 * nn);
    s.V = reinterpret_cast<cx<float> *>(b + 16 * nn);
    s.A = reinterpret_cast<cx<float> *>(b + 24 * nn);
    s.rot = reinterpret_cast<float2 *>(b + 24 * nn);
    s.Zt = reinterpret_cast<float *>(b + 48 * nn);
    char *v = b + ((52 * nn + 15) & ~size_t(15));
    s.d = reinterpret_cast<float *>(v);
    s.e = s.d + n;
    s.tau = reinterpret_cast<cx<float> *>(s.e + n);
    s.ql = reinterpret_cast<QlState *>(s.tau + n);
    return s;
}

// FP32 eigenvectors of H = Hsys + b . Z for snapshots first .. first + count - 1
// of the launch into X of slots 0 .. count - 1; H as double-words beside them.
cudaError_t launch_large_solve(const SnapArgs &a, char *scratch, size_t per, int first, int count,
                               cudaStream_t st);

constexpr int LM_KT = 16;  // k depth of a GEMM slab

// Bytes of one slab stage: A and B at up to 16 bytes per element.
__host__ __device__ inline size_t lm_stage_bytes(int threads) {
    return ((size_t)4 * (threads / 32) * LM_KT + (size_t)LM_KT * 32) * 16;
}

// Asynchronous global -> shared copies of one element (8 or 16 bytes);
// `valid` false writes zeros (nothing is read; src is still a valid
// address).  One commit group per slab; wait_group 1 leaves the newest
// group in flight.
__device__ __forceinline__ void lm_cp8(void *dst, const void *src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src),
                 "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void lm_cp16(void *dst, const void *src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src),
                 "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void lm_cp(float4 *dst, const float4 *src, bool valid) {
    lm_cp16(dst, src, valid);
}
__device__ __forceinline__ void lm_cp(float2 *dst, const float2 *src, bool valid) {
    lm_cp8(dst, src, valid);
}
__device__ __forceinline__ void lm_cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void lm_cp_wait1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// A stored element as its hi and lo lane pairs (lo = 0 for FP32 elements)
__device__ __forceinline__ void lm_pairs(const float4 *p, u64 &h, u64 &l) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
    h = v.x;
    l = v.y;
}
__device__ __forceinline__ void lm_pairs(const float2 *p, u64 &h, u64 &l) {
    h = *reinterpret_cast<const u64 *>(p);
    l = 0ull;
}

// Tiled product C(i, j) = sum_k op(A)(i, k) B(k, j), i < M, j < N, k < K,
// as one CTA-wide kernel body.  The CTA walks output tiles of TR = 4 x
// warps rows by 32 columns; a thread owns rows 4 w .. 4 w + 3 (w its warp)
// of column `lane`.  A and B are staged in shared memory LM_KT deep as they
// are stored in global memory (no conversion), by cp.async in two stages:
// the next slab's copies are in flight while the current one is
// multiplied.  A(i, k) is read from Ag[k * lda + i] (A_KI) or
// Ag[i * lda + k], B(k, j) from Bg[k * ldb + j]; the A reads of the multiply
// are warp broadcasts.  Accumulation (ACC):
//   LM_DW_ALO   anchored double-word, A double-word (float4), B FP32
//   LM_PLAIN    FP32 sums of A B
//   LM_PLAIN_C  FP32 sums of conj(A) B
// (the pair (s1, s2) of lm_step; lm_dw / lm_plain turn it into the value).
// The tiles are dealt out in turn to `nparts` CTAs, of which this is number
// `part`.  skip(i0, j0) drops a whole tile; init(i, j, s1, c1, s2, c2) seeds an
// accumulator (the anchor, or a start value); epi(i, j, s1, c1, s2, c2)
// consumes it (i < M, j < N only).
enum { LM_DW_ALO = 0, LM_PLAIN = 1, LM_PLAIN_C = 2 };

template <int ACC, bool A_KI, typename AT, typename BT, typename Skip, typename Init, typename Epi>
static __device__ void lm_tiles(int M, int N, int K, const AT *Ag, int lda,
                         const BT *Bg, int ldb, char *slab, int part, int nparts,
                         Skip skip, Init init, Epi epi) {
    const int tid = threadIdx.x, nt = blockDim.x, w = tid >> 5, lane = tid & 31;
    const int TR = 4 * (nt >> 5);
    const int ti = (M + TR - 1) / TR, tj = (N + 31) >> 5, nslab = (K + LM_KT - 1) / LM_KT;
    const size_t stage = lm_stage_bytes(nt);
    char *A0 = slab, *B0 = slab + (size_t)TR * LM_KT * 16;
    // this thread's elements of a slab: two of A, (ia, ka) and (ia + di, ka + dk),
    // and B's rows w, w + warps, ... of column `lane`
    const int ia = A_KI ? tid % TR : tid / LM_KT, ka = A_KI ? tid / TR : tid % LM_KT;
    const int di = A_KI ? 0 : nt / LM_KT, dk = A_KI ? 8 : 0, nw = nt >> 5;
    const size_t astep = A_KI ? (size_t)lda : 1;
    auto issue = [&](int i0, int j0, int sl) {
        AT *As = reinterpret_cast<AT *>(A0 + (sl & 1) * stage);
        BT *Bs = reinterpret_cast<BT *>(B0 + (sl & 1) * stage);
        const int k0 = sl * LM_KT, gi = i0 + ia, gk = k0 + ka, gj = j0 + lane;
        const AT *src = Ag + (A_KI ? (size_t)gk * lda + gi : (size_t)gi * lda + gk);
        const bool ok0 = gi < M && gk < K, ok1 = gi + di < M && gk + dk < K;
        lm_cp(As + tid, ok0 ? src : Ag, ok0);
        lm_cp(As + tid + nt, ok1 ? src + (A_KI ? dk * astep : (size_t)di * lda) : Ag, ok1);
        const BT *bsrc = Bg + (size_t)(k0 + w) * ldb + gj;
        for (int k = w; k < LM_KT; k += nw) {
            const bool ok = k0 + k < K && gj < N;
            lm_cp(Bs + k * 32 + lane, ok ? bsrc : Bg, ok);
            bsrc += (size_t)nw * ldb;
        }
        lm_cp_commit();
    };
    int turn = -1;
    for (int t = 0; t < ti * tj; ++t) {  // the same sequence in every thread
        const int it = t / tj, i0 = it * TR, j0 = (t - it * tj) * 32;
        if (skip(i0, j0)) continue;
        if (++turn == nparts) turn = 0;
        if (turn != part) continue;
        const int j = j0 + lane;
        u64 s1[4], c1[4], s2[4], c2[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            s1[q] = c1[q] = s2[q] = c2[q] = 0ull;
            init(i0 + 4 * w + q, j, s1[q], c1[q], s2[q], c2[q]);
        }
        issue(i0, j0, 0);
        for (int sl = 0; sl < nslab; ++sl) {
            if (sl + 1 < nslab)
                issue(i0, j0, sl + 1);
            else
                lm_cp_commit();  // an empty group keeps wait_group 1 exact
            lm_cp_wait1();
            __syncthreads();
            const AT *As = reinterpret_cast<const AT *>(A0 + (sl & 1) * stage);
            const BT *Bs = reinterpret_cast<const BT *>(B0 + (sl & 1) * stage);
#pragma unroll
            for (int k = 0; k < LM_KT; ++k) {
                u64 bh, bl;
                lm_pairs(Bs + k * 32 + lane, bh, bl);
                float b0, b1;
                split_f32x2(bh, b0, b1);
                const u64 bx = f32x2(b0, b0), by = f32x2(b1, b1);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int r = 4 * w + q;
                    u64 ah, al;
                    lm_pairs(As + (A_KI ? k * TR + r : r * LM_KT + k), ah, al);
                    if (ACC == LM_DW_ALO) {
                        lm_step<true, false>(s1[q], c1[q], s2[q], c2[q], ah, al, bx, by, 0ull, 0ull);
                    } else {
                        s1[q] = fma_f32x2(ah, bx, s1[q]);
                        s2[q] = fma_f32x2(ah, by, s2[q]);
                    }
                }
            }
            __syncthreads();  // the stage is refilled two slabs later
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = i0 + 4 * w + q;
            if (i < M && j < N) epi(i, j, s1[q], c1[q], s2[q], c2[q]);
        }
    }
    __syncthreads();
}

}  // namespace msp
