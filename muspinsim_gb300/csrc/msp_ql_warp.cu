// FP32 Householder + implicit-shift QL eigensolver for batches of n <= 32
// Hamiltonians: the first stage of the two-stage snapshot pipeline for large
// batches (the alternative to msp_jacobi_warp.cu's cyclic Jacobi), replacing the
// FP32 part of Hermitian.diag's eigensolve (muspinsim/spinop.py:51-82) for the
// batched snapshots of ExperimentRunner (muspinsim/experiment.py:332-341,
// 434-498).  The second stage (msp_snap.cu, msp_snap64.cu) refines the
// eigenvectors this one leaves in scratch, exactly as it refines the Jacobi's;
// they only have to be orthonormal to FP32 rounding.
//
// Two kernels, so that each has the registers and shared memory it wants (as
// one kernel per four matrices and warp, ten warps fitted an SM and every stage
// waited for its own latency: 20.2 ms for 201,000 matrices of n = 32, 0.52 ms for
// 10,000 of n = 24; now 10.7 and 0.40 ms):
//   1. msp_tri_warp_kernel, tridiagonalisation (LAPACK zhetd2), a warp per
//      matrix, the matrix in registers (a lane holds a row);
//   2. msp_ql_kernel, QL with the rotations accumulated into Z and the
//      back-transformation U = Q Z, a CTA per QlShape::GM matrices: one warp runs
//      the serial recurrences of all of them, a lane per matrix, one QL step
//      ahead of eight warps that apply the rotations to Z in shared memory.
// Between them the reflectors and the tridiagonal matrix lie in the snapshot's
// eigenvector scratch, which U overwrites: row k holds reflector v_k in columns
// k + 1 .. n - 1, (d_k, e_k) in column 0 and tau_k in column 1 (tau_0 in row
// n - 1, column 1).
#include "msp_internal.cuh"

namespace msp {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// ------------------------------------------------------------------ 1. tridiagonalisation

constexpr int TRI_WARPS = 4;

// Lanes per matrix: small ones share a warp.
template <int NM>
struct TriShape {
    static constexpr int LN = NM <= 8 ? 8 : NM <= 16 ? 16 : 32;
    static constexpr int PER_CTA = TRI_WARPS * 32 / LN;
};

__device__ __forceinline__ float fast_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y * fmaf(-0.5f * x * y, y, 1.5f);
}

template <int LN>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
    for (int o = LN / 2; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o, LN);
    return v;
}

// Lane i holds row i.  Step k finds the column it eliminates in register 0: the
// rank-2 update moves every entry one register down, so that no index depends on
// k.  v and w reach the other lanes through shared memory, (v_j, w_j) by row
// relative to k + 1, zero beyond the last.  p^H v = conj(tau) v^H A v with a real
// v^H A v, so one real sum over the lanes does.  Bound by issue: 14 instructions
// per trailing entry and row, some 110 per column.  201,000 matrices of n = 32:
// 3.5 ms, 61% of the issue slots.
template <int NM>
__global__ void __launch_bounds__(TRI_WARPS * 32) msp_tri_warp_kernel(SnapArgs a) {
    constexpr int LN = TriShape<NM>::LN, PER = 32 / LN;
    __shared__ __align__(16) float4 sh_all[TRI_WARPS * PER][LN + 4];
    const int n = a.n, lane = threadIdx.x & (LN - 1), grp = threadIdx.x / LN;
    const int sn = blockIdx.x * TriShape<NM>::PER_CTA + grp;
    const bool live = sn < a.num_snap;
    float4 *sh = sh_all[grp];  // (v_j, w_j)
    const int at = live ? sn : a.num_snap - 1;
    const SnapSource src = snap_source(a, at);
    float2 *out = reinterpret_cast<float2 *>(a.evec) + (size_t)at * n * n;
    cx<float> r[NM];
    {
        const double *b = a.field + 3 * (size_t)src.g;
        const size_t nn = (size_t)n * n;
        const bool on = lane < n;
        if (src.Hdw != nullptr) {
            const float bx = (float)b[0], by = (float)b[1], bz = (float)b[2];
#pragma unroll
            for (int j = 0; j < NM; ++j) {
                r[j] = mk<float>(0.f, 0.f);
                if (j >= n || !on) continue;
                const size_t o = (size_t)j * n + lane;
                auto hi = [](const float4 *p) { return *reinterpret_cast<const float2 *>(p); };
                const float2 h = hi(src.Hdw + o), z0 = hi(src.Zdw + o), z1 = hi(src.Zdw + nn + o),
                             z2 = hi(src.Zdw + 2 * nn + o);
                // A[lane][j] = conj(A[j][lane])
                r[j] = mk<float>(fmaf(bz, z2.x, fmaf(by, z1.x, fmaf(bx, z0.x, h.x))),
                                 -fmaf(bz, z2.y, fmaf(by, z1.y, fmaf(bx, z0.y, h.y))));
            }
        } else {
#pragma unroll
            for (int j = 0; j < NM; ++j) {
                r[j] = mk<float>(0.f, 0.f);
                if (j >= n || !on) continue;
                const size_t o = (size_t)j * n + lane;
                const cx<double> h = src.Hsys[o], z0 = src.Z[o], z1 = src.Z[nn + o], z2 = src.Z[2 * nn + o];
                r[j] = mk<float>((float)(h.re + b[0] * z0.re + b[1] * z1.re + b[2] * z2.re),
                                 -(float)(h.im + b[0] * z0.im + b[1] * z1.im + b[2] * z2.im));
            }
        }
    }
    float2 tau0 = make_float2(0.f, 0.f);
    for (int k = 0; k + 1 < n; ++k) {
        const int m = n - k - 1;
        const bool below = lane > k && lane < n;
        const cx<float> x = below ? r[0] : mk<float>(0.f, 0.f);
        const float dk = __shfl_sync(FULL, r[0].re, k, LN);
        float xn2 = lanes_sum<LN>(lane > k + 1 ? cabs2(x) : 0.f);
        cx<float> alpha =
            mk<float>(__shfl_sync(FULL, x.re, k + 1, LN), __shfl_sync(FULL, x.im, k + 1, LN));
        float s2 = fmaf(alpha.re, alpha.re, fmaf(alpha.im, alpha.im, xn2)), up = 1.f;
        if (__any_sync(FULL, s2 < REFLECT_TINY)) {
            const float u2 = lanes_sum<LN>(lane > k + 1 ? cabs2(cscale(REFLECT_UP, x)) : 0.f);
            if (s2 < REFLECT_TINY) {
                up = REFLECT_UP;
                alpha = cscale(up, alpha);
                xn2 = u2;
                s2 = cabs2(alpha) + xn2;
                if (s2 < REFLECT_TINY) xn2 = alpha.im = 0.f;
            }
        }
        float beta = alpha.re;
        cx<float> tau = mk<float>(0.f, 0.f), sc = tau;
        if (xn2 != 0.f || alpha.im != 0.f) {
            float root, inv;  // |beta| and its reciprocal
            if (s2 > 1e-36f && s2 < 1e36f) {
                inv = fast_rsqrt(s2);
                root = s2 * inv;
            } else {
                root = sqrtf(s2);
                inv = 1.f / root;
            }
            beta = -copysignf(root, alpha.re);
            inv = -copysignf(inv, alpha.re);
            tau = mk<float>(1.f - alpha.re * inv, -alpha.im * inv);
            const cx<float> den = mk<float>(alpha.re - beta, alpha.im);
            const float dd = up / cabs2(den);
            sc = mk<float>(den.re * dd, -den.im * dd);
        }
        if (up != 1.f) beta *= 1.f / REFLECT_UP;
        const cx<float> v = lane == k + 1 ? mk<float>(1.f, 0.f) : cmul(x, sc);
        {
            float2 o = make_float2(v.re, v.im);
            if (lane == 0) o = make_float2(dk, beta);
            if (lane == 1 && k > 0) o = make_float2(tau.re, tau.im);
            if (k == 0) tau0 = make_float2(tau.re, tau.im);
            if (live && lane < n && (lane > k || lane < 2)) out[(size_t)k * n + lane] = o;
        }
        // relative row of this lane; retired ones and padding fill the end with zeros
        const int rel = below ? lane - k - 1 : (lane <= k ? m + lane : lane);
        sh[rel] = make_float4(v.re, v.im, 0.f, 0.f);
        __syncwarp();
        // p = A v
        float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
#pragma unroll
        for (int g = 0; g < NM / 4; ++g) {
            if (4 * g >= m) continue;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int j = 4 * g + t;
                if (j + 1 >= NM) continue;
                const float2 q = *reinterpret_cast<const float2 *>(sh + j);
                p0 = fmaf(r[j + 1].re, q.x, p0);
                p1 = fmaf(-r[j + 1].im, q.y, p1);
                p2 = fmaf(r[j + 1].re, q.y, p2);
                p3 = fmaf(r[j + 1].im, q.x, p3);
            }
        }
        const cx<float> p = mk<float>(p0 + p1, p2 + p3);
        const float vav = lanes_sum<LN>(below ? fmaf(v.re, p.re, v.im * p.im) : 0.f);
        const float half = -0.5f * cabs2(tau) * vav;
        cx<float> w = cmul(tau, p);
        w = below ? mk<float>(fmaf(half, v.re, w.re), fmaf(half, v.im, w.im)) : mk<float>(0.f, 0.f);
        const cx<float> vi = below ? v : mk<float>(0.f, 0.f);
        __syncwarp();
        sh[rel] = make_float4(vi.re, vi.im, w.re, w.im);
        __syncwarp();
        // A -= v w^H + w v^H, one register down
#pragma unroll
        for (int g = 0; g < NM / 4; ++g) {
            if (4 * g >= m) continue;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int j = 4 * g + t;
                if (j + 1 >= NM) continue;
                const float4 q = sh[j];
                cx<float> h = r[j + 1];
                h.re = fmaf(-vi.re, q.z, fmaf(-vi.im, q.w, fmaf(-w.re, q.x, fmaf(-w.im, q.y, h.re))));
                h.im = fmaf(-vi.im, q.z, fmaf(vi.re, q.w, fmaf(-w.im, q.x, fmaf(w.re, q.y, h.im))));
                r[j] = h;
            }
        }
        __syncwarp();
    }
    const float dl = __shfl_sync(FULL, r[0].re, n - 1, LN);
    if (live && lane < 2) out[(size_t)(n - 1) * n + lane] = lane == 0 ? make_float2(dl, 0.f) : tau0;
}

// ------------------------------------------------------------------ 2. QL

constexpr int QL_APPLY = 8;                         // warps that apply rotations
constexpr int QL_THREADS = 32 * (QL_APPLY + 1);
constexpr int QL_AHEAD = 2;  // reflectors fetched ahead of the one that acts

// GM matrices of up to NM x NM per CTA, LN lanes per matrix in the application.
template <int NM>
struct QlShape {
    static constexpr int GM = NM <= 24 ? 32 : 16;
    static constexpr int LN = NM <= 8 ? 8 : NM <= 16 ? 16 : 32;
    static constexpr int LDZ = NM + 1;
    static constexpr int Z_FLOATS = NM * LDZ;
    static constexpr size_t RING = (size_t)2 * NM * GM * 8;  // two steps' rotations
    static constexpr size_t BYTES = (size_t)GM * Z_FLOATS * 4 + RING + (size_t)2 * NM * GM * 4;
    static_assert(RING >= (size_t)(QL_APPLY + 1) * 2 * NM * 8, "reflectors alias the ring");
};

// What bounds it is the chain of one rotation (a product sum, a reciprocal square
// root with one Newton step and a product), of which GM run side by side: a QL
// step takes as long as its longest chain, some 1.4 times the average.  The
// shift of a step is applied as the chain loads the diagonal, and a bit mask per
// matrix, rebuilt as the chain passes, tells where its off-diagonal is
// negligible.  The tridiagonal matrix is scaled to norm 1 .. 2 and split below
// 2^-23, the error of the reduction to it, so the reciprocal square root's operand
// stays in range.  201,000 matrices of n = 32: 7.2 ms, half of the issue
// slots; more CTAs per SM (GM = 8 or 16, n = 24) took as long.
template <int NM>
__global__ void __launch_bounds__(QL_THREADS, 2) msp_ql_kernel(SnapArgs a) {
    using S = QlShape<NM>;
    constexpr int GM = S::GM, LN = S::LN, LDZ = S::LDZ;
    extern __shared__ __align__(16) char smem[];
    float2 *const ring = reinterpret_cast<float2 *>(smem);  // [2][NM][GM]
    float *const d = reinterpret_cast<float *>(smem + S::RING), *const e = d + NM * GM;  // [NM][GM]
    float *const Z = e + NM * GM;  // [GM][column][row]
    __shared__ int head[2][GM], alive[2], status[GM];  // head: m | l << 8, -1: no step
    const int n = a.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sn0 = blockIdx.x * GM, cnt = min(GM, a.num_snap - sn0);
    float2 *const evec = reinterpret_cast<float2 *>(a.evec);
    for (int x = tid; x < n * GM; x += QL_THREADS) {
        const int i = x / GM, g = x - i * GM;
        const float2 v = g < cnt ? evec[((size_t)(sn0 + g) * n + i) * n] : make_float2(0.f, 0.f);
        d[x] = v.x;
        e[x] = v.y;
    }
    for (int x = tid; x < GM * S::Z_FLOATS; x += QL_THREADS) {
        const int y = x % S::Z_FLOATS;
        Z[x] = y / LDZ == y % LDZ ? 1.f : 0.f;
    }
    __syncthreads();
    // the recurrences (warp 0), a lane per matrix
    const bool mine = warp == 0 && lane < cnt;
    const int g0 = warp == 0 ? lane & (GM - 1) : 0;
    float *const dg = d + g0, *const eg = e + g0;  // entry i at [i * GM]
    const float small = 1.1920928955078125e-7f;  // 2^-23
    unsigned mask = 0;  // bit i: entry i of e is negligible
    int l = 0, iter = 0, st = MSP_ITEM_OK;
    if (mine) {
        float norm = 0.f;
        bool nan = false;
        for (int i = 0; i < n; ++i) {
            const float x = fabsf(dg[i * GM]) + fabsf(eg[i * GM]);
            nan |= x != x;
            norm = fmaxf(norm, x);
        }
        // it splits everywhere and would count as converged
        if (nan && a.num_snap < STAGE1_REPORT_NAN) st = MSP_ITEM_NOT_CONVERGED;
        // 0 for an overflowed matrix: its entries become NaN and split everywhere
        const float inv = norm < 1e37f ? 2.f / pow2_above(norm) : 0.f;
        for (int i = 0; i < n; ++i) {
            dg[i * GM] *= inv;
            const float x = eg[i * GM] * inv;
            eg[i * GM] = x;
            if (!(fabsf(x) > small)) mask |= 1u << i;
        }
        mask |= 1u << (n - 1);
    }
    for (int step = 0;; ++step) {
        const int slot = step & 1;
        if (warp == 0) {
            // one QL step of every matrix that is not finished
            bool on = mine && l < n;
            if (on) {
                if (iter >= 60 && !((mask >> l) & 1u)) {
                    st = MSP_ITEM_NOT_CONVERGED;
                    mask |= 1u << l;
                }
                const unsigned rest = ~(mask >> l);
                const int skip = rest ? __ffs(rest) - 1 : 32;  // levels that are done
                if (skip > 0) {
                    l += skip;
                    iter = 0;
                }
                on = l < n;
            }
            const unsigned go = __ballot_sync(FULL, on);
            if (lane == 0) alive[slot] = go != 0;
            int m = 0, len = 0;
            float h = 0.f, dl = 0.f, dl1 = 0.f, el1 = 0.f, e0 = 0.f;
            if (on) {
                ++iter;
                m = l + __ffs(mask >> l) - 1;
                len = m - l;
                const float g = dg[l * GM];
                e0 = eg[l * GM];
                el1 = eg[(l + 1) * GM];
                // the shift only has to be good, not exact
                const float pp = __fdividef(dg[(l + 1) * GM] - g, 2.f * e0);
                const float t1 = fmaf(pp, pp, 1.f), t = pp + copysignf(t1 * fast_rsqrt(t1), pp);
                dl = __fdividef(e0, t);
                dl1 = e0 * t;
                h = g - dl;
            }
            if (lane < GM) head[slot][lane] = on ? m | l << 8 : -1;
            const int longest = __reduce_max_sync(FULL, len);
            float c = 1.f, c2 = 1.f, c3 = 1.f, s = 0.f, s2 = 0.f, pp = 0.f, di = 0.f, ei = 0.f;
            unsigned seen = 0;
            auto diagonal = [&](int i) {
                const float x = dg[i * GM] - h;
                return i == l ? dl : i == l + 1 ? dl1 : x;
            };
            if (on) {
                pp = diagonal(m);
                di = diagonal(m - 1);
                ei = eg[(m - 1) * GM];
            }
            float2 *out = ring + slot * NM * GM + g0;
            for (int t = 0; t < longest; ++t, out += GM) {
                if (t >= len) continue;
                const int i = m - 1 - t, nx = max(i - 1, l);
                const float dn = diagonal(nx), en = eg[nx * GM];
                c3 = c2;
                c2 = c;
                s2 = s;
                const float g = c * ei, hh = c * pp;
                const float x2 = fmaf(pp, pp, ei * ei), u = fmaf(pp, di, -ei * g);
                const float y = fast_rsqrt(x2);
                const float en1 = s * (x2 * y);
                s = ei * y;
                c = pp * y;
                pp = u * y;  // c d_i - s g
                eg[(i + 1) * GM] = en1;
                dg[(i + 1) * GM] = fmaf(s, fmaf(c, g, s * di), hh);
                *out = make_float2(c, s);
                seen = seen << 1 | (fabsf(en1) > small ? 0u : 1u);
                di = dn;
                ei = en;
            }
            if (on) {
                pp = __fdividef(-s * s2 * c3 * el1 * e0, dl1);
                const float x = s * pp;
                eg[l * GM] = x;
                dg[l * GM] = c * pp;
                seen = seen << 1 | (fabsf(x) > small ? 0u : 1u);
                // bits l .. m
                const unsigned span = (2u << len) - 1u;
                mask = (mask & ~(span << l)) | (seen & span) << l;
                mask |= 1u << m;  // e_m = 0 r: the block's end
            }
        } else if (step > 0) {
            // the previous step's rotations, a lane per row of Z
            const int old = slot ^ 1, sub = lane & (LN - 1);
            for (int g = (warp - 1) * (32 / LN) + lane / LN; g < GM; g += QL_APPLY * (32 / LN)) {
                const int hd = head[old][g];
                if (hd < 0 || sub >= n) continue;
                const int m = hd & 255, l = hd >> 8;
                const float2 *rot = ring + old * NM * GM + g;
                float *z = Z + g * S::Z_FLOATS + m * LDZ + sub;
                float hc = *z;
                int len = m - l;
                for (; len >= 8; len -= 8) {
                    float zi[8];
                    float2 q[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        zi[u] = z[-(u + 1) * LDZ];
                        q[u] = rot[u * GM];
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        z[-u * LDZ] = q[u].y * zi[u] + q[u].x * hc;
                        hc = q[u].x * zi[u] - q[u].y * hc;
                    }
                    z -= 8 * LDZ;
                    rot += 8 * GM;
                }
                for (; len > 0; --len) {
                    const float zi = z[-LDZ];
                    const float2 q = *rot;
                    *z = q.y * zi + q.x * hc;
                    hc = q.x * zi - q.y * hc;
                    z -= LDZ;
                    rot += GM;
                }
                *z = hc;
            }
        }
        __syncthreads();
        if (!alive[slot]) break;
    }
    if (mine) status[lane] = st;
    __syncthreads();
    // U = Q Z, a warp per matrix: lane j holds column j and applies the reflectors
    // last to first, each staged in shared memory while the one before it acts
    float2 *const vb = ring + warp * 2 * NM;
    for (int g = warp; g < cnt; g += QL_APPLY + 1) {
        float2 *const V = evec + (size_t)(sn0 + g) * n * n;
        const float *z = Z + g * S::Z_FLOATS + min(lane, NM - 1) * LDZ;
        cx<float> u[NM];
#pragma unroll
        for (int i = 0; i < NM; ++i) u[i] = mk<float>(i < n ? z[i] : 0.f, 0.f);
        auto fetch = [&](int k) {
            return k >= 0 && lane > k && lane < n ? V[(size_t)k * n + lane] : make_float2(0.f, 0.f);
        };
        auto scalar = [&](int k) { return V[(size_t)(k > 0 ? k : n - 1) * n + 1]; };
        float2 next[QL_AHEAD], tn[QL_AHEAD];
#pragma unroll
        for (int q = 0; q < QL_AHEAD; ++q) {
            next[q] = fetch(n - 2 - q);
            tn[q] = scalar(n - 2 - q);
        }
        for (int k = n - 2; k >= 0; --k) {
            float2 *const vk = vb + (k & 1) * NM;
            const float2 tau = tn[0];
            if (lane < NM) vk[lane] = next[0];
#pragma unroll
            for (int q = 0; q + 1 < QL_AHEAD; ++q) {
                next[q] = next[q + 1];
                tn[q] = tn[q + 1];
            }
            next[QL_AHEAD - 1] = fetch(k - QL_AHEAD);
            tn[QL_AHEAD - 1] = scalar(k - QL_AHEAD);
            __syncwarp();
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
            for (int q = 0; q < NM / 4; ++q) {
                if (4 * q + 3 <= k || 4 * q >= n) continue;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int i = 4 * q + t;
                    const float2 v = vk[i];
                    s0 = fmaf(v.x, u[i].re, s0);
                    s1 = fmaf(v.y, u[i].im, s1);
                    s2 = fmaf(v.x, u[i].im, s2);
                    s3 = fmaf(-v.y, u[i].re, s3);
                }
            }
            const cx<float> ts = cmul(mk<float>(tau.x, tau.y), mk<float>(s0 + s1, s2 + s3));
#pragma unroll
            for (int q = 0; q < NM / 4; ++q) {
                if (4 * q + 3 <= k || 4 * q >= n) continue;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const int i = 4 * q + t;
                    const float2 v = vk[i];
                    u[i].re = fmaf(-v.x, ts.re, fmaf(v.y, ts.im, u[i].re));
                    u[i].im = fmaf(-v.x, ts.im, fmaf(-v.y, ts.re, u[i].im));
                }
            }
        }
        __syncwarp();  // every lane has read the reflectors
        if (lane < n) {
#pragma unroll
            for (int i = 0; i < NM; ++i)
                if (i < n) V[(size_t)i * n + lane] = make_float2(u[i].re, u[i].im);
        }
        if (lane == 0) a.status[snap_source(a, sn0 + g).g] = status[g];
    }
}

template <int NM>
cudaError_t launch(const SnapArgs &a, cudaStream_t st) {
    using S = QlShape<NM>;
    msp_tri_warp_kernel<NM><<<(a.num_snap + TriShape<NM>::PER_CTA - 1) / TriShape<NM>::PER_CTA,
                              TRI_WARPS * 32, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(msp_ql_kernel<NM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::BYTES);
    if (e != cudaSuccess) return e;
    msp_ql_kernel<NM><<<(a.num_snap + S::GM - 1) / S::GM, QL_THREADS, S::BYTES, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

bool ql_warp_supported(int n) { return n >= 3 && n <= 32; }

cudaError_t launch_ql_warp(const SnapArgs &a, cudaStream_t st) {
    if (a.num_snap <= 0) return cudaSuccess;
    if (a.n <= 8) return launch<8>(a, st);
    if (a.n <= 16) return launch<16>(a, st);
    if (a.n <= 24) return launch<24>(a, st);
    if (a.n <= 32) return launch<32>(a, st);
    return cudaErrorInvalidValue;
}

}  // namespace msp
