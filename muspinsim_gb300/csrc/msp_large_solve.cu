// FP32 eigenvectors of the Hamiltonians of the fast path for n > 64: the
// start of their refinement (msp_large_refine.cu).  Replaces, with it,
// numpy.linalg.eigh in Hermitian.diag (muspinsim/spinop.py:51-82).
//
// Householder tridiagonalisation, implicit QL with the rotations accumulated
// into Z, back-transformation: the algorithm of msp_large.cuh, one kernel per
// stage.  In one kernel per snapshot each stage waited for the one that suits
// the grid least: a 192 x 192 matrix took 7.6 ms to tridiagonalise out of L2
// with 128 threads, 6.4 ms for the QL iteration, which one thread computes and
// the other warps apply, and 2.0 ms to transform back.  Apart:
//   1. one CTA per matrix, the lower triangle in shared memory (n <= 221;
//      beyond that the blocked reduction out of global memory);
//   2. one warp per matrix for the QL recurrence, a serial chain of some
//      0.85 n^2 rotations; the rotations go to a stream in global memory;
//   3. one warp per 32 rows of Z applies the stream, its rows in shared memory;
//   4. one CTA per 32 columns applies the reflectors, its columns in shared
//      memory.
#include "msp_large.cuh"
#include "msp_large_slots.cuh"

namespace msp {

namespace {

// The Hamiltonian of a snapshot as double-words into s.H; put(i, j, v) gets
// the high words.
template <typename Put>
__device__ __forceinline__ void load_hamiltonian_dw(const SnapArgs &a, int sn, int n,
                                                    const LargeSlot &s, Put put) {
    const SnapSource src = snap_source(a, sn);
    const size_t g = (size_t)src.g, nn = (size_t)n * n;
    const double bx = a.field[3 * g], by = a.field[3 * g + 1], bz = a.field[3 * g + 2];
    for (int x = threadIdx.x; x < (int)nn; x += blockDim.x) {
        const cx<double> hs = src.Hsys[x], z0 = src.Z[x], z1 = src.Z[nn + x], z2 = src.Z[2 * nn + x];
        const double hr = hs.re + bx * z0.re + by * z1.re + bz * z2.re;
        const double hi = hs.im + bx * z0.im + by * z1.im + bz * z2.im;
        const float4 h = dw_split(make_double2(hr, hi));
        s.H[x] = h;
        const int i = x / n;
        put(i, x - i * n, mk<float>(h.x, h.y));
    }
}

// ------------------------------------------------------------------ 1. tridiagonalisation

// Shared memory: the lower triangle by columns, v of this column and the last,
// p, the column sums, the warps' partial products, a partial sum per warp.
__host__ __device__ inline size_t tri_smem_bytes(int n, int threads) {
    return ((size_t)n * (n + 1) / 2 + 4 * (size_t)n + (size_t)(threads / 32) * n + threads / 32) * 8;
}

__host__ __device__ inline int tri_threads(int n) { return n <= 128 ? 256 : 512; }

constexpr size_t TRI_SMEM_MAX = 227 * 1024;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// h - v conj(w) - w conj(v')
__device__ __forceinline__ cx<float> rank2(cx<float> h, cx<float> vi, cx<float> wi, cx<float> vj,
                                           cx<float> wj) {
    h.re = fmaf(-vi.re, wj.re, fmaf(-vi.im, wj.im, fmaf(-wi.re, vj.re, fmaf(-wi.im, vj.im, h.re))));
    h.im = fmaf(-vi.im, wj.re, fmaf(vi.re, wj.im, fmaf(-wi.im, vj.re, fmaf(wi.re, vj.im, h.im))));
    return h;
}

// LAPACK zhetd2, lower form, the rank-2 update A -= v w^H + w v^H of a column
// put off until the product A v of the next, so that one pass over the triangle
// does both; an entry serves its row and, conjugated, its column.  Q = ceil(n /
// 32): a lane keeps rows lane + 32 q of v, w and of its warp's part of A v in
// registers, and warps take whole columns, two at a time, without bank
// conflicts; every warp makes the reflector for itself, so that a column costs
// three barriers.  Bound by instruction issue.  n = 192: 1.0 ms per matrix and SM
// against 7.6 ms out of L2.
template <int Q>
__global__ void __launch_bounds__(512)
    msp_large_tridiag_kernel(SnapArgs a, char *scratch, size_t per, int first) {
    extern __shared__ __align__(16) char smem[];
    const int n = a.n, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int nw = nt >> 5;
    const LargeSlot s = large_slot(scratch, per, blockIdx.x, n);
    cx<float> *P = reinterpret_cast<cx<float> *>(smem);
    cx<float> *vbuf = P + (size_t)n * (n + 1) / 2, *p = vbuf + 2 * n, *pc = p + n, *part = pc + n;
    cx<float> *red = part + (size_t)nw * n;
    auto column = [&](int k) { return P + k * n - k * (k + 1) / 2; };  // [i]: entry (i, k), i >= k
    load_hamiltonian_dw(a, first + blockIdx.x, n, s, [&](int i, int j, cx<float> h) {
        if (j <= i) column(j)[i] = h;
    });
    const cx<float> zero = mk<float>(0.f, 0.f);
    for (int i = tid; i < 3 * n; i += nt) vbuf[i] = zero;  // both v, and p
    __syncthreads();
    cx<float> vo[Q], wo[Q];  // rows of the last column's v and w
#pragma unroll
    for (int q = 0; q < Q; ++q) vo[q] = wo[q] = zero;
    cx<float> a2 = zero;
    for (int k = 0; k < n; ++k) {
        // column k, brought up to date by every warp
        const cx<float> *vold = vbuf + (k & 1) * n;
        cx<float> *vnew = vbuf + ((k + 1) & 1) * n;
        const cx<float> vk = vold[k], wk = cadd(p[k], cmul(a2, vk));
        const cx<float> *ck = column(k);
        cx<float> vn[Q];
        float xn2 = 0.f;
        cx<float> alpha = zero;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int i = 32 * q + lane;
            vn[q] = zero;
            if (i >= k && i < n) {
                const cx<float> x = rank2(ck[i], vo[q], wo[q], vk, wk);
                if (i == k && warp == 0) s.d[k] = x.re;
                if (i > k) vn[q] = x;
                if (i > k + 1) xn2 += cabs2(x);
            }
            if (q == (k + 1) >> 5) {
                alpha.re = __shfl_sync(0xffffffffu, vn[q].re, (k + 1) & 31);
                alpha.im = __shfl_sync(0xffffffffu, vn[q].im, (k + 1) & 31);
            }
        }
        if (k + 1 >= n) break;
        xn2 = warp_sum(xn2);
        float up = 1.f;
        if (alpha.re * alpha.re + alpha.im * alpha.im + xn2 < REFLECT_TINY) {
            up = REFLECT_UP;
            alpha = cscale(up, alpha);
            xn2 = 0.f;
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if (32 * q + lane > k + 1) xn2 += cabs2(cscale(up, vn[q]));
            xn2 = warp_sum(xn2);
            if (cabs2(alpha) + xn2 < REFLECT_TINY) xn2 = alpha.im = 0.f;
        }
        float beta = alpha.re;
        cx<float> tau = zero, sc = zero;
        if (!(xn2 == 0.f && alpha.im == 0.f)) {
            beta = -copysignf(sqrtf(alpha.re * alpha.re + alpha.im * alpha.im + xn2), alpha.re);
            tau = mk<float>((beta - alpha.re) / beta, -alpha.im / beta);
            const cx<float> den = mk<float>(alpha.re - beta, alpha.im);
            const float dd = up / cabs2(den);
            sc = mk<float>(den.re * dd, -den.im * dd);
        }
        if (up != 1.f) beta *= 1.f / REFLECT_UP;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int i = 32 * q + lane;
            vn[q] = i == k + 1 ? mk<float>(1.f, 0.f) : cmul(vn[q], sc);
            if (i > k && i < n && q % nw == warp) {
                vnew[i] = vn[q];
                s.V[(size_t)k * n + i - k - 1] = vn[q];
            }
        }
        if (tid == 0) {
            s.e[k] = beta;
            s.tau[k] = tau;
        }
        __syncthreads();
        // the trailing columns: the last update, and p = A v
        cx<float> pr[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) pr[q] = zero;
        for (int j0 = k + 1 + warp; j0 < n; j0 += 2 * nw) {
            const int j1 = j0 + nw, jc = min(j1, n - 1);
            cx<float> *c0 = column(j0), *c1 = column(jc);
            const cx<float> v0 = vnew[j0], v1 = vnew[jc], u0 = vold[j0], u1 = vold[jc];
            const cx<float> w0 = cadd(p[j0], cmul(a2, u0)), w1 = cadd(p[jc], cmul(a2, u1));
            cx<float> s0 = zero, s1 = zero;
            auto visit = [&](cx<float> *col, int j, int q, int i, const cx<float> &vj,
                             const cx<float> &uj, const cx<float> &wj, cx<float> &sum) {
                cx<float> h = rank2(col[i], vo[q], wo[q], uj, wj);
                if (i == j) h.im = 0.f;
                col[i] = h;
                pr[q].re = fmaf(h.re, vj.re, fmaf(-h.im, vj.im, pr[q].re));
                pr[q].im = fmaf(h.re, vj.im, fmaf(h.im, vj.re, pr[q].im));
                if (i == j) h = zero;
                sum.re = fmaf(h.re, vn[q].re, fmaf(h.im, vn[q].im, sum.re));
                sum.im = fmaf(h.re, vn[q].im, fmaf(-h.im, vn[q].re, sum.im));
            };
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                if (32 * q + 31 < j0) continue;
                const int i = 32 * q + lane;
                if (i < n) {
                    if (i >= j0) visit(c0, j0, q, i, v0, u0, w0, s0);
                    if (i >= j1) visit(c1, j1, q, i, v1, u1, w1, s1);
                }
            }
            // four sums over the warp: lanes 0, 8, 16, 24 get one each
            const bool hi = lane & 16, h8 = lane & 8;
            float x0 = hi ? s1.re : s0.re, x1 = hi ? s1.im : s0.im;
            x0 += __shfl_xor_sync(0xffffffffu, hi ? s0.re : s1.re, 16);
            x1 += __shfl_xor_sync(0xffffffffu, hi ? s0.im : s1.im, 16);
            float x = h8 ? x1 : x0;
            x += __shfl_xor_sync(0xffffffffu, h8 ? x0 : x1, 8);
            x += __shfl_xor_sync(0xffffffffu, x, 4);
            x += __shfl_xor_sync(0xffffffffu, x, 2);
            x += __shfl_xor_sync(0xffffffffu, x, 1);
            const int j = hi ? j1 : j0;
            if ((lane & 7) == 0 && j < n) reinterpret_cast<float *>(pc + j)[h8 ? 1 : 0] = x;
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int i = 32 * q + lane;
            if (i > k && i < n) part[(size_t)warp * n + i] = pr[q];
        }
        __syncthreads();
        // p *= tau; p^H v
        float hr = 0.f, hm = 0.f;
        for (int i = k + 1 + tid; i < n; i += nt) {
            cx<float> x = pc[i];
            for (int w = 0; w < nw; ++w) x = cadd(x, part[(size_t)w * n + i]);
            x = cmul(tau, x);
            p[i] = x;
            const cx<float> c = cmulc(x, vnew[i]);  // conj(p_i) v_i
            hr += c.re;
            hm += c.im;
        }
        hr = warp_sum(hr);
        hm = warp_sum(hm);
        if (lane == 0) red[warp] = mk<float>(hr, hm);
        __syncthreads();
        cx<float> h2 = zero;
        for (int w = 0; w < nw; ++w) h2 = cadd(h2, red[w]);
        a2 = cscale(-0.5f, cmul(tau, h2));
        // w = p + a2 v
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int i = 32 * q + lane;
            vo[q] = vn[q];
            wo[q] = i > k && i < n ? cadd(p[i], cmul(a2, vn[q])) : zero;
        }
    }
    if (tid == 0) s.e[n - 1] = 0.f;
}

// Blocked tridiagonalisation out of global memory (the panel scheme of
// LAPACK zlatrd / zhetrd, lower form, full storage): columns are reduced
// LM_KT at a time.  Within a panel the trailing matrix stays as it was at
// the panel start ("stale"); reflector j of the panel keeps v_j and w_j in
// VW (rows: V in columns 0..15, W in 16..31), so that the true trailing
// matrix is the stale one minus V W^H + W V^H:
//   1. column k (rows k..) is brought up to date from the panel's V, W;
//   2. its reflector (as in the unblocked form; d_k, e_k, tau_k);
//   3. p = A22 v over the stale matrix, in the same column-parallel pass
//      as y = VW^H v (32 extra "columns" read from VW);
//   4. p -= V (W^H v) + W (V^H v), p *= tau, alpha = -tau (p^H v) / 2,
//      w = p + alpha v;
// and after the panel one rank-2 LM_KT update of the trailing matrix,
// A22 += [V W] [-W^H; -V^H], through the tile engine.  The trailing matrix
// is read about 1.2 times per column instead of three times.  Scratch: R
// holds VW (n x 32) and the update's right operand (32 x n).
__global__ void __maxnreg__(96)
    msp_large_tridiag_panel_kernel(SnapArgs a, char *scratch, size_t per, int first) {
    extern __shared__ __align__(16) char smem[];
    const int n = a.n, tid = threadIdx.x, nt = blockDim.x;
    const LargeSlot s = large_slot(scratch, per, blockIdx.x, n);
    const int RW = nt < 64 ? nt : 64, G = nt / RW, pr = tid % RW, pg = tid / RW;
    const LargeSm<float> sm = large_sm<float>(smem, n, nt);
    cx<float> *A = s.A;
    char *slab = smem + ((large_sm_bytes<float>(n, nt) + 15) & ~size_t(15));
    cx<float> *VW = s.R;                   // n x 32
    cx<float> *Bt = s.R + (size_t)n * 32;  // 32 x n
    cx<float> *v = sm.v, *p = sm.p, *part = sm.part, *y = sm.y;
    const size_t pst = (size_t)n + 32;  // stride of the partial sums
    auto noskip = [](int, int) { return false; };
    load_hamiltonian_dw(a, first + blockIdx.x, n, s,
                        [&](int i, int j, cx<float> h) { A[(size_t)i * n + j] = h; });
    __syncthreads();
    for (int k0 = 0; k0 + 1 < n; k0 += LM_KT) {
        const int nbp = min(LM_KT, n - 1 - k0);
        for (size_t x = (size_t)k0 * 32 + tid; x < (size_t)n * 32; x += nt)
            VW[x] = mk<float>(0.f, 0.f);
        __syncthreads();
        for (int j = 0; j < nbp; ++j) {
            const int k = k0 + j, m = n - k - 1;
            // 1. column k, rows k.., minus the panel's V W^H + W V^H
            if (j > 0) {
                const cx<float> *vk = VW + (size_t)k * 32;
                for (int r = k + tid; r < n; r += nt) {
                    const cx<float> *vr = VW + (size_t)r * 32;
                    cx<float> a = A[(size_t)r * n + k];
                    for (int c = 0; c < j; ++c) {
                        const cx<float> t1 = cmul(vr[c], conj(vk[16 + c]));
                        const cx<float> t2 = cmul(vr[16 + c], conj(vk[c]));
                        a = mk<float>(a.re - t1.re - t2.re, a.im - t1.im - t2.im);
                    }
                    A[(size_t)r * n + k] = a;
                }
                __syncthreads();
            }
            // 2. reflector of A[k+1.., k]
            float xn2 = 0.f;
            for (int i = 1 + tid; i < m; i += nt) xn2 += cabs2(A[(size_t)(k + 1 + i) * n + k]);
            xn2 = block_sum(xn2, sm.red);
            cx<float> alpha = A[(size_t)(k + 1) * n + k];
            float up = 1.f;
            if (alpha.re * alpha.re + alpha.im * alpha.im + xn2 < REFLECT_TINY) {
                up = REFLECT_UP;
                alpha = cscale(up, alpha);
                xn2 = 0.f;
                for (int i = 1 + tid; i < m; i += nt)
                    xn2 += cabs2(cscale(up, A[(size_t)(k + 1 + i) * n + k]));
                __syncthreads();  // sm.red again
                xn2 = block_sum(xn2, sm.red);
                if (cabs2(alpha) + xn2 < REFLECT_TINY) xn2 = alpha.im = 0.f;
            }
            cx<float> tau = mk<float>(0.f, 0.f);
            float beta = alpha.re;
            const bool reflect = !(xn2 == 0.f && alpha.im == 0.f);
            if (reflect) {
                beta = -copysignf(sqrtf(alpha.re * alpha.re + alpha.im * alpha.im + xn2), alpha.re);
                tau = mk<float>((beta - alpha.re) / beta, -alpha.im / beta);
                const cx<float> den = mk<float>(alpha.re - beta, alpha.im);
                const float dd = up / cabs2(den);
                const cx<float> sc = mk<float>(den.re * dd, -den.im * dd);
                for (int i = tid; i < m; i += nt)
                    v[i] = i == 0 ? mk<float>(1.f, 0.f) : cmul(A[(size_t)(k + 1 + i) * n + k], sc);
            } else {
                for (int i = tid; i < m; i += nt) v[i] = mk<float>(0.f, 0.f);  // V and W columns stay 0
            }
            if (up != 1.f) beta *= 1.f / REFLECT_UP;
            if (tid == 0) {
                s.d[k] = A[(size_t)k * n + k].re;
                s.e[k] = beta;
                s.tau[k] = tau;
            }
            __syncthreads();
            // 3. p = A22 v (stale A22, Hermitian: p_i = sum_l conj(A22_li) v_l) and
            //    y = VW^H v in extra columns i = m .. m + 31
            if (pg < G) {
                const int lb = (int)((long long)m * pg / G), le = (int)((long long)m * (pg + 1) / G);
                for (int i = pr; i < m + 32; i += RW) {
                    const cx<float> *col = i < m ? A + (size_t)(k + 1) * n + (k + 1 + i)
                                                 : VW + (size_t)(k + 1) * 32 + (i - m);
                    const size_t ld = i < m ? (size_t)n : 32;
                    float r0 = 0.f, i0 = 0.f, r1 = 0.f, i1 = 0.f;
                    int l = lb;
#pragma unroll 4
                    for (; l + 1 < le; l += 2) {
                        const cx<float> a0 = col[(size_t)l * ld], a1 = col[(size_t)(l + 1) * ld];
                        const cx<float> x0 = v[l], x1 = v[l + 1];
                        r0 += a0.re * x0.re + a0.im * x0.im;
                        i0 += a0.re * x0.im - a0.im * x0.re;
                        r1 += a1.re * x1.re + a1.im * x1.im;
                        i1 += a1.re * x1.im - a1.im * x1.re;
                    }
                    if (l < le) {
                        const cx<float> a0 = col[(size_t)l * ld], x0 = v[l];
                        r0 += a0.re * x0.re + a0.im * x0.im;
                        i0 += a0.re * x0.im - a0.im * x0.re;
                    }
                    part[(size_t)pg * pst + i] = mk<float>(r0 + r1, i0 + i1);
                }
            }
            __syncthreads();
            for (int i = tid; i < m + 32; i += nt) {
                float sr = 0.f, si = 0.f;
                for (int g = 0; g < G; ++g) {
                    sr += part[(size_t)g * pst + i].re;
                    si += part[(size_t)g * pst + i].im;
                }
                if (i < m)
                    p[i] = mk<float>(sr, si);
                else
                    y[i - m] = mk<float>(sr, si);  // V^H v in 0..15, W^H v in 16..31
            }
            __syncthreads();
            // 4. p = tau (p - V (W^H v) - W (V^H v)); w = p + alpha v
            float hr = 0.f, hi = 0.f;
            for (int i = tid; i < m; i += nt) {
                cx<float> acc = p[i];
                const cx<float> *vr = VW + (size_t)(k + 1 + i) * 32;
                for (int c = 0; c < j; ++c) {
                    const cx<float> t1 = cmul(vr[c], y[16 + c]), t2 = cmul(vr[16 + c], y[c]);
                    acc = mk<float>(acc.re - t1.re - t2.re, acc.im - t1.im - t2.im);
                }
                acc = cmul(tau, acc);
                p[i] = acc;
                const cx<float> c = cmulc(acc, v[i]);  // conj(p_i) v_i
                hr += c.re;
                hi += c.im;
            }
            hr = block_sum(hr, sm.red);
            hi = block_sum(hi, sm.red);
            const cx<float> a2 = cscale(-0.5f, cmul(tau, mk<float>(hr, hi)));
            for (int i = tid; i < m; i += nt) {
                const cx<float> vi = v[i];
                VW[(size_t)(k + 1 + i) * 32 + j] = vi;
                VW[(size_t)(k + 1 + i) * 32 + 16 + j] = cadd(p[i], cmul(a2, vi));
                s.V[(size_t)k * n + i] = vi;  // for the back-transformation
            }
            __syncthreads();
        }
        // rank-2 LM_KT update of the trailing matrix (rows and columns k1..)
        const int k1 = k0 + nbp, mt = n - k1;
        if (mt > 0) {
            for (int x = tid; x < 32 * mt; x += nt) {
                const int kk = x / mt, jj = x - kk * mt;
                const cx<float> w = VW[(size_t)(k1 + jj) * 32 + (kk < 16 ? 16 + kk : kk - 16)];
                Bt[(size_t)kk * n + jj] = mk<float>(-w.re, w.im);  // -conj
            }
            __syncthreads();
            cx<float> *At = A + (size_t)k1 * n + k1;
            lm_tiles<LM_PLAIN, false>(
                mt, mt, 32, reinterpret_cast<const float2 *>(VW + (size_t)k1 * 32), 32,
                reinterpret_cast<const float2 *>(Bt), n, slab, 0, 1, noskip,
                [&](int i, int j, u64 &s1, u64 &, u64 &, u64 &) {
                    const cx<float> a = i < mt && j < mt ? At[(size_t)i * n + j] : mk<float>(0.f, 0.f);
                    s1 = f32x2(a.re, a.im);
                },
                [&](int i, int j, u64 s1, u64, u64 s2, u64) {
                    At[(size_t)i * n + j] = lm_plain<false>(s1, s2);
                });
        }
    }
    if (tid == 0) {
        s.d[n - 1] = A[(size_t)(n - 1) * n + (n - 1)].re;
        s.e[n - 1] = 0.f;
    }
}

// ------------------------------------------------------------------ 2. QL recurrence

// 1 / sqrt(x) for x in the normal range: the approximation instruction and one
// Newton step
__device__ __forceinline__ float ql_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y * fmaf(-0.5f * x * y, y, 1.5f);
}

// One warp: every lane follows the same recurrence (lane 0 stores), and the
// searches for a split and the shifts of the diagonal run over the lanes.  The
// tridiagonal matrix is scaled to norm 1 .. 2 and split where an off-diagonal
// entry is below 2^-23, the error of the reduction to it; so entries inside a
// step stay in the range of ql_rsqrt.  The rotations of a QL step, for columns
// (i, i + 1) of Z with i = m - 1 .. l, follow a header (m, l) in the stream; a
// round ends early when the next step might not fit.  What bounds it is the
// chain of one rotation: a product sum, a reciprocal square root with one Newton
// step and a product; the next d and e are loaded one rotation ahead.
// n = 192: 1.2 ms, 40 ns per rotation.
__global__ void __launch_bounds__(32) msp_large_ql_kernel(char *scratch, size_t per, int n, int round) {
    extern __shared__ __align__(16) char smem[];
    const LargeSlot s = large_slot(scratch, per, blockIdx.x, n);
    const int lane = threadIdx.x;
    float *d = reinterpret_cast<float *>(smem), *e = d + n;
    QlState st;
    if (round == 0) {
        st.l = st.iter = st.done = 0;
        st.status = MSP_ITEM_OK;
    } else {
        st = *s.ql;
    }
    st.len = 0;
    __syncwarp();
    if (st.done) {
        if (lane == 0) s.ql->len = 0;
        return;
    }
    float norm = 0.f;
    for (int i = lane; i < n; i += 32) norm = fmaxf(norm, fabsf(s.d[i]) + fabsf(s.e[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) norm = fmaxf(norm, __shfl_xor_sync(0xffffffffu, norm, o));
    // 0 for an overflowed matrix: its entries become NaN and split everywhere
    const float inv = round > 0 ? 1.f : norm < 1e37f ? 1.f / pow2_above(norm) : 0.f;
    for (int i = lane; i < n; i += 32) {
        d[i] = 2.f * inv * s.d[i];
        e[i] = 2.f * inv * s.e[i];
        if (round > 0) {
            d[i] = s.d[i];
            e[i] = s.e[i];
        }
    }
    __syncwarp();
    const float small = LargeEps<float>::eps;
    const int cap = large_rot_capacity(n);
    while (st.l < n) {
        const int l = st.l;
        int m = l;
        for (;;) {
            const int i = m + lane;
            const unsigned hit = __ballot_sync(0xffffffffu, i >= n - 1 || !(fabsf(e[min(i, n - 1)]) > small));
            if (hit) {
                m = min(m + __ffs(hit) - 1, n - 1);
                break;
            }
            m += 32;
        }
        if (m == l || st.iter >= 60) {
            if (m != l) st.status = MSP_ITEM_NOT_CONVERGED;
            if (lane == 0) e[l] = 0.f;
            __syncwarp();
            ++st.l;
            st.iter = 0;
            continue;
        }
        if (st.len + 1 + (m - l) > cap) break;
        // shift
        const float g0 = d[l], e0 = e[l];
        float pp = (d[l + 1] - g0) / (2.f * e0);
        const float t = pp + copysignf(sqrtf(fmaf(pp, pp, 1.f)), pp);
        const float dl = e0 / t, dl1 = e0 * t, h0 = g0 - dl;
        __syncwarp();
        for (int i = l + 2 + lane; i < n; i += 32) d[i] -= h0;
        if (lane == 0) {
            d[l] = dl;
            d[l + 1] = dl1;
        }
        __syncwarp();
        const float el1 = e[l + 1];
        float2 *out = s.rot + st.len;
        if (lane == 0) *out = make_float2(__int_as_float(m), __int_as_float(l));
        pp = d[m];
        float c = 1.f, c2 = 1.f, c3 = 1.f, sn = 0.f, s2 = 0.f;
        float ei = e[m - 1], di = d[m - 1];
        const float *dp = d + m - 1, *ep = e + m - 1;
        float *dq = d + m, *eq = e + m;
#pragma unroll 2
        for (int i = m - 1; i >= l; --i) {
            // the entries of the next rotation; the last reads e[l - 1] in vain
            dp -= i > l;
            ep -= i > l;
            const float en = *ep, dn = *dp;
            c3 = c2;
            c2 = c;
            s2 = sn;
            const float g = c * ei, h = c * pp;
            const float x2 = fmaf(pp, pp, ei * ei), u = fmaf(pp, di, -ei * g);
            const float y = ql_rsqrt(x2);
            const float en1 = sn * (x2 * y);
            sn = ei * y;
            c = pp * y;
            pp = u * y;  // c d_i - s g
            const float d1 = fmaf(sn, fmaf(c, g, sn * di), h);
            if (lane == 0) {
                *eq = en1;
                *dq = d1;
                *++out = make_float2(c, sn);
            }
            --eq;
            --dq;
            ei = en;
            di = dn;
        }
        __syncwarp();
        pp = -sn * s2 * c3 * el1 * e[l] / dl1;
        __syncwarp();
        if (lane == 0) {
            e[l] = sn * pp;
            d[l] = c * pp;
        }
        __syncwarp();
        ++st.iter;
        st.len += 1 + (m - l);
    }
    st.done = st.l >= n;
    if (!st.done) {
        st.status = round + 1 < LARGE_QL_ROUNDS ? st.status : MSP_ITEM_NOT_CONVERGED;
        for (int i = lane; i < n; i += 32) {
            s.d[i] = d[i];
            s.e[i] = e[i];
        }
    }
    if (lane == 0) *s.ql = st;
}

// ------------------------------------------------------------------ 3. rotations

constexpr int ROT_WINDOW = 128;  // stream entries staged at a time

// One warp per 32 rows of Z, in shared memory (column-major, a lane per row).
// The stream passes through a window in shared memory, the next window on its
// way from global memory meanwhile.  Bound by issue, some 9 instructions per
// rotation and 32 rows.  192 matrices of n = 192: 0.45 ms.
__global__ void __launch_bounds__(32) msp_large_rotate_kernel(char *scratch, size_t per, int n, int round) {
    extern __shared__ __align__(16) char smem[];
    const LargeSlot s = large_slot(scratch, per, blockIdx.y, n);
    const int lane = threadIdx.x, row = blockIdx.x * 32 + lane;
    const int len = s.ql->len;
    if (round > 0 && len == 0) return;
    float2 *win = reinterpret_cast<float2 *>(smem);
    float *Z = reinterpret_cast<float *>(win + ROT_WINDOW) + lane;  // Z[32 * column]
    for (int c = 0; c < n; ++c)
        Z[32 * c] = round == 0 ? (c == row ? 1.f : 0.f) : (row < n ? s.Zt[(size_t)c * n + row] : 0.f);
    float2 next[ROT_WINDOW / 32];
    auto fetch = [&](int base) {
#pragma unroll
        for (int q = 0; q < ROT_WINDOW / 32; ++q) {
            const int i = base + 32 * q + lane;
            next[q] = i < len ? s.rot[i] : make_float2(0.f, 0.f);
        }
    };
    int base = 0;
    auto advance = [&]() {  // the window at `base`, the one after it under way
        __syncwarp();
#pragma unroll
        for (int q = 0; q < ROT_WINDOW / 32; ++q) win[32 * q + lane] = next[q];
        __syncwarp();
        fetch(base + ROT_WINDOW);
    };
    fetch(0);
    advance();
    int pos = 0;
    while (pos < len) {
        const float2 hd = win[pos - base];
        const int m = __float_as_int(hd.x), l = __float_as_int(hd.y);
        if (++pos == base + ROT_WINDOW) {
            base = pos;
            advance();
        }
        float hc = Z[32 * m];
        int i = m - 1;
        while (i >= l) {
            const int cnt = min(i - l + 1, base + ROT_WINDOW - pos);
            const float2 *w = win + (pos - base);
            int u = 0;
            for (; u + 8 <= cnt; u += 8) {
                float z[8];
                float2 r[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    z[q] = Z[32 * (i - u - q)];
                    r[q] = w[u + q];
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    Z[32 * (i - u - q + 1)] = r[q].y * z[q] + r[q].x * hc;
                    hc = r[q].x * z[q] - r[q].y * hc;
                }
            }
            for (; u < cnt; ++u) {
                const float2 r = w[u];
                const float z = Z[32 * (i - u)];
                Z[32 * (i - u + 1)] = r.y * z + r.x * hc;
                hc = r.x * z - r.y * hc;
            }
            i -= cnt;
            pos += cnt;
            if (pos == base + ROT_WINDOW) {
                base = pos;
                advance();
            }
        }
        Z[32 * l] = hc;
    }
    if (row < n)
        for (int c = 0; c < n; ++c) s.Zt[(size_t)c * n + row] = Z[32 * c];
}

// ------------------------------------------------------------------ 4. back-transformation

constexpr int BACK_THREADS = 256;

// 32 columns of U = Q Z per CTA: reflectors n - 2 .. 0, a thread per column and
// every eighth row, so that one barrier per reflector is enough (the partial
// sums of v^H U and the next reflector change hands there).  NR: rows per thread,
// which then stay in registers; NR = 0 keeps them in shared memory (n > 224).
// 192 matrices of n = 192: 0.9 ms; 1.0 ms with the rows in shared memory.
template <int NR>
__global__ void __launch_bounds__(BACK_THREADS) msp_large_back_kernel(char *scratch, size_t per, int n) {
    constexpr int CB = NR > 0 ? 32 : 16, R = BACK_THREADS / CB;
    extern __shared__ __align__(16) char smem[];
    const LargeSlot s = large_slot(scratch, per, blockIdx.y, n);
    const int tid = threadIdx.x, c = tid % CB, rg = tid / CB, j0 = blockIdx.x * CB;
    const int ld = (n + R - 1) / R * R;
    cx<float> *part = reinterpret_cast<cx<float> *>(smem);  // two of [R][CB]
    cx<float> *v = part + 2 * BACK_THREADS;                 // three reflectors, by absolute row
    cx<float> *U = v + 3 * (size_t)ld;                      // [row][CB]
    cx<float> u[NR > 0 ? NR : 1];
    const cx<float> zero = mk<float>(0.f, 0.f);
    if (NR > 0) {
        const int j = min(j0 + c, n - 1);
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            const int r = rg + R * q;
            u[q] = mk<float>(r < n ? s.Zt[(size_t)j * n + r] : 0.f, 0.f);
        }
    } else {
        for (int e = tid; e < n * CB; e += BACK_THREADS) {
            const int cc = e / n, i = e - cc * n;
            U[i * CB + cc] = mk<float>(j0 + cc < n ? s.Zt[(size_t)(j0 + cc) * n + i] : 0.f, 0.f);
        }
    }
    for (int i = tid; i < 3 * ld; i += BACK_THREADS) v[i] = zero;
    __syncthreads();
    auto stage = [&](int k) {
        const cx<float> tau = s.tau[k];
        const bool none = tau.re == 0.f && tau.im == 0.f;
        cx<float> *dst = v + (size_t)(k % 3) * ld;
        for (int i = k + 1 + tid; i < n; i += BACK_THREADS)
            dst[i] = none ? zero : s.V[(size_t)k * n + i - k - 1];
    };
    stage(n - 2);
    __syncthreads();
    for (int k = n - 2; k >= 0; --k) {
        const cx<float> *vk = v + (size_t)(k % 3) * ld;
        const int r0 = k + 1 + (rg - (k + 1) % R + R) % R;  // first row of this thread
        float sr = 0.f, si = 0.f;
        auto dot = [&](const cx<float> &x, const cx<float> &y) {
            sr = fmaf(x.re, y.re, fmaf(x.im, y.im, sr));
            si = fmaf(x.re, y.im, fmaf(-x.im, y.re, si));
        };
        if (NR > 0) {
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (rg + R * q > k && rg + R * q < ld) dot(vk[rg + R * q], u[q]);
        } else {
            for (int r = r0; r < n; r += R) dot(vk[r], U[r * CB + c]);
        }
        cx<float> *pk = part + (k & 1) * BACK_THREADS;
        pk[rg * CB + c] = mk<float>(sr, si);
        if (k > 0) stage(k - 1);
        const cx<float> tau = s.tau[k];
        __syncthreads();
        cx<float> t = zero;
#pragma unroll
        for (int q = 0; q < R; ++q) t = cadd(t, pk[q * CB + c]);
        t = cmul(tau, t);
        auto take = [&](cx<float> &y, const cx<float> &x) {
            y.re = fmaf(-x.re, t.re, fmaf(x.im, t.im, y.re));
            y.im = fmaf(-x.re, t.im, fmaf(-x.im, t.re, y.im));
        };
        if (NR > 0) {
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (rg + R * q > k && rg + R * q < ld) take(u[q], vk[rg + R * q]);
        } else {
            for (int r = r0; r < n; r += R) take(U[r * CB + c], vk[r]);
        }
    }
    if (NR > 0) {
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            const int r = rg + R * q;
            if (r < n && j0 + c < n) s.X[(size_t)r * n + j0 + c] = u[q];
        }
    } else {
        for (int r = rg; r < n; r += R)
            if (j0 + c < n) s.X[(size_t)r * n + j0 + c] = U[r * CB + c];
    }
}

template <typename F>
cudaError_t allow_smem(F *fn, size_t bytes) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <int Q>
cudaError_t launch_tridiag(const SnapArgs &a, char *scratch, size_t per, int first, int count,
                           int threads, size_t smem, cudaStream_t st) {
    cudaError_t e = allow_smem(msp_large_tridiag_kernel<Q>, smem);
    if (e != cudaSuccess) return e;
    msp_large_tridiag_kernel<Q><<<count, threads, smem, st>>>(a, scratch, per, first);
    return cudaGetLastError();
}

template <int NR>
cudaError_t launch_back(int n, char *scratch, size_t per, int count, cudaStream_t st) {
    const int cb = NR > 0 ? 32 : 16, r = BACK_THREADS / cb, ld = (n + r - 1) / r * r;
    const size_t smem = (2 * (size_t)BACK_THREADS + 3 * (size_t)ld + (NR > 0 ? 0 : (size_t)n * cb)) * 8;
    cudaError_t e = allow_smem(msp_large_back_kernel<NR>, smem);
    if (e != cudaSuccess) return e;
    msp_large_back_kernel<NR><<<dim3((n + cb - 1) / cb, count), BACK_THREADS, smem, st>>>(scratch, per, n);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_large_solve(const SnapArgs &a, char *scratch, size_t per, int first, int count,
                               cudaStream_t st) {
    const int n = a.n;
    cudaError_t e;
    const int threads = tri_threads(n);
    const size_t smem = tri_smem_bytes(n, threads);
    if (smem <= TRI_SMEM_MAX) {
        switch ((n + 31) / 32) {
            case 3: e = launch_tridiag<3>(a, scratch, per, first, count, threads, smem, st); break;
            case 4: e = launch_tridiag<4>(a, scratch, per, first, count, threads, smem, st); break;
            case 5: e = launch_tridiag<5>(a, scratch, per, first, count, threads, smem, st); break;
            case 6: e = launch_tridiag<6>(a, scratch, per, first, count, threads, smem, st); break;
            default: e = launch_tridiag<7>(a, scratch, per, first, count, threads, smem, st); break;
        }
    } else {
        const int nt = 256;
        const size_t sm = ((large_sm_bytes<float>(n, nt) + 15) & ~size_t(15)) + 2 * lm_stage_bytes(nt);
        e = allow_smem(msp_large_tridiag_panel_kernel, sm);
        if (e != cudaSuccess) return e;
        msp_large_tridiag_panel_kernel<<<count, nt, sm, st>>>(a, scratch, per, first);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return e;
    const size_t rot = ROT_WINDOW * 8 + (size_t)n * 128;
    e = allow_smem(msp_large_rotate_kernel, rot);
    for (int round = 0; e == cudaSuccess && round < LARGE_QL_ROUNDS; ++round) {
        msp_large_ql_kernel<<<count, 32, 8 * (size_t)n, st>>>(scratch, per, n, round);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        msp_large_rotate_kernel<<<dim3((n + 31) / 32, count), 32, rot, st>>>(scratch, per, n, round);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return e;
    if (n <= 96) return launch_back<12>(n, scratch, per, count, st);
    if (n <= 128) return launch_back<16>(n, scratch, per, count, st);
    if (n <= 192) return launch_back<24>(n, scratch, per, count, st);
    if (n <= 224) return launch_back<28>(n, scratch, per, count, st);
    return launch_back<0>(n, scratch, per, count, st);
}

}  // namespace msp
