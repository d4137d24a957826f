// Mixed-precision per-snapshot kernels (n <= 64; FP64: msp_snap64.cu): one
// CTA turns one Hamiltonian's eigenbasis into the quantities the time
// evolution needs.  Replaces, per configuration snapshot, ExperimentRunner.Htot
// (muspinsim/experiment.py:332-341), Hermitian.diag (muspinsim/spinop.py:
// 51-82) and the eigenbasis part of Hamiltonian.fast_evolve / evolve /
// integrate_decaying (muspinsim/hamiltonian.py:76-87, 149-160, 195-211).
//
// FP32 eigenvectors (warp Jacobi or Householder + QL for batches of n <= 32,
// else FP32 Jacobi in the CTA), then one Ogita-Aishima refinement step
// evaluated in double-word FP32 arithmetic (msp_refine.cuh): H X (for n > 32 and
// eigensolves also X^H H X and X^H X) to ~2^-44, eigenvalues to FP64 accuracy
// (Rayleigh quotient plus the second-order term), the eigenvectors corrected
// to FP32 rounding.  GB300 runs FP32 at ~60x its FP64 rate, so this costs
// about as much as the FP32 eigenvectors themselves instead of dominating as
// FP64 would.  Also the host-side launch rules of both precisions and the
// FP64 basis changes of the single-Hamiltonian API.
#include "msp_refine.cuh"

namespace msp {

// ------------------------------------------------------------------ eigh

__global__ void msp_eigh_kernel(const cx<double> *__restrict__ Hin, int n, int batch,
                                int max_sweeps, double *__restrict__ evals,
                                cx<double> *__restrict__ evecs, int *__restrict__ status) {
    extern __shared__ __align__(16) char smem[];
    const int m = n + (n & 1), ld = m + 1, ldh = jacobi_ldh(m);
    SnapSmem<float> s = snap_carve<float, true>(smem, n, false, 0);
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int bidx = blockIdx.x; bidx < batch; bidx += gridDim.x) {
        const cx<double> *Hb = Hin + (size_t)bidx * n * n;
        for (int e = tid; e < m * m; e += nt) {
            const int i = FastDiv(m).div(e), j = e - i * m;
            cx<double> h = mk<double>(0.0, 0.0);
            if (i < n && j < n) h = Hb[(size_t)i * n + j];
            const float hr = (float)h.re, hi = (float)h.im;
            s.w.H[i * ldh + j] = mk<float>(hr, hi);
            s.Hh[i * ld + j] = mk<float>(hr, hi);
            s.Hl[i * ld + j] = mk<float>((float)(h.re - (double)hr), (float)(h.im - (double)hi));
        }
        __syncthreads();
        hamiltonian_row_norms(s, n, m);
        int st = jacobi_sweeps<float>(s.w, m, max_sweeps);
        st |= eigenpairs(s, n, m, 4);
        // ascending order, ties by index (stable)
        for (int j = tid; j < n; j += nt) {
            int r = 0;
            const float2 lj = s.lw[j];
            for (int k = 0; k < n; ++k) {
                const float2 lk = s.lw[k];
                r += dw_less(lk, lj) || (dw_equal(lk, lj) && k < j);
            }
            evals[(size_t)bidx * n + r] = dw_to_double(lj);
            s.rank[j] = r;
        }
        __syncthreads();
        cx<double> *Vb = evecs + (size_t)bidx * n * n;
        for (int e = tid; e < n * n; e += nt) {
            const int i = FastDiv(n).div(e), j = e - i * n;
            const cx<float> u = s.w.U[i * ld + j];
            Vb[(size_t)i * n + s.rank[j]] = mk<double>((double)u.re, (double)u.im);
        }
        if (tid == 0) status[bidx] = st;
        __syncthreads();
    }
}

// ------------------------------------------------------------------ fast path

// Mixed fast path: A_jk = |(U^H M)_jk|^2 over the lower triangle j >= k
// (FP32), pair records for j > k, and this thread's share of sum_j A_jj as
// a double-word.
__device__ __forceinline__ float2 amplitudes_mixed(const SnapArgs &a, const SnapSmem<float> &s,
                                                   const cx<float> *U, const cx<float> *M, int n,
                                                   int sn, float scale) {
    const int ld = n + (n & 1) + 1;
    const int P = n * (n - 1) / 2, ntri = n * (n + 1) / 2;
    float2 diag = make_float2(0.f, 0.f);
    for (int e = threadIdx.x; e < ntri; e += blockDim.x) {
        int j, k;
        tri_index(e, j, k);
        float gr = 0.f, gi = 0.f;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const cx<float> u = U[i * ld + j], mm = M[i * ld + k];
            gr += u.re * mm.re + u.im * mm.im;
            gi += u.re * mm.im - u.im * mm.re;
        }
        const float A = gr * gr + gi * gi;
        if (j == k) {
            diag = dw_add_f(diag, A);
        } else {
            const size_t o = (size_t)sn * P + pair_index(j, k);
            reinterpret_cast<float2 *>(a.pair_coef)[o] = make_float2(scale * A, 0.f);
            store_frequency_dw(a, o, dw_sub(s.lw[j], s.lw[k]));
        }
    }
    return diag;
}

// The same in the two-stage kernels: a thread's rows k <= j of column j of the
// Hermitian U^H M (see oa_refine_rows).
template <int NN>
__device__ __forceinline__ float2 amplitudes_rows(const SnapArgs &a, const SnapSmem<float> &s,
                                                  const cx<float> *U, const cx<float> *M, int n_rt,
                                                  int sn, float scale) {
    const int n = NN > 0 ? NN : n_rt;
    const size_t rec = (size_t)sn * (n * (n - 1) / 2);
    const RowShape sh = row_shape(n, blockDim.x);
    const int rg = threadIdx.x / n, j = threadIdx.x - rg * n, i0 = rg * sh.rows;
    float2 diag = make_float2(0.f, 0.f);
    if (rg >= sh.groups || i0 > j) return diag;
    cx<float> b[ROW_MAX];
    row_products<NN, ROW_MAX>(U, M, n, i0, j, b);
#pragma unroll
    for (int r = 0; r < ROW_MAX; ++r) {
        const int k = i0 + r;
        if (r >= sh.rows || k > j) continue;
        const float A = cabs2(b[r]);
        if (j == k) {
            diag = dw_add_f(diag, A);
        } else {
            const size_t o = rec + pair_index(j, k);
            reinterpret_cast<float2 *>(a.pair_coef)[o] = make_float2(scale * A, 0.f);
            store_frequency_dw(a, o, dw_sub(s.lw[j], s.lw[k]));
        }
    }
    return diag;
}

// One snapshot of the muon-first T = inf shortcut (muspinsim/hamiltonian.py:
// 166-217): A = |U^dag (sigma_p (x) 1_d) U|^2 and omega_jk = 2 pi (l_j - l_k)
// for j > k, scaled by 0.5 * w / (d * N_avg), plus the constant
// 0.5 * sum_j A_jj part.
// PRE: the FP32 eigenvectors come from the first stage (n <= 32), refined by
// rows; else (n > 32) Jacobi and oa_refine in this CTA.  At most 64 registers,
// which leaves as many CTAs per SM as shared memory does.
template <bool PRE>
__global__ void __maxnreg__(64) msp_snap_fast_kernel(SnapArgs a) {
    typedef float T;
    extern __shared__ __align__(16) char smem[];
    const int n = a.n, m = n + (n & 1), ld = PRE ? row_ld(n) : m + 1, d = n / 2;
    SnapSmem<T> s = PRE ? row_carve(smem, n, false, 0) : snap_carve<T, true>(smem, n, false, 0);
    const int tid = threadIdx.x, nt = blockDim.x;

    for (int sn = blockIdx.x; sn < a.num_snap; sn += gridDim.x) {
        const SnapSource src = snap_source(a, sn);
        const size_t g = (size_t)src.g;
        if (PRE)
            load_hamiltonian_rows(src, a.field + 3 * g, n, s);
        else
            load_hamiltonian<PRE>(src.Hsys, src.Z, src.Hdw, src.Zdw, a.field + 3 * g, n, m, s);
        int st = snap_eigvecs<PRE>(a, sn, (int)g, n, m, ld, s);
        st |= PRE ? eigenpairs_rows(n, false, 0, a.max_refine) : eigenpairs(s, n, m, a.max_refine);

        // sigma_p = p . sigma (Pauli), applied on the muon (slowest) digit
        T px, py, pz;
        load_vec3<T>(a.pol + 3 * g, px, py, pz);
        const cx<T> s00 = mk<T>(pz, T(0)), s01 = mk<T>(px, -py);
        const cx<T> s10 = mk<T>(px, py), s11 = mk<T>(-pz, T(0));
        cx<T> *M = s.w.H;  // free buffer
        const cx<T> *U = s.w.U;
        for (int e = tid; e < n * n; e += nt) {
            const int i = FastDiv(n).div(e), k = e - i * n;
            cx<T> v;
            if (i < d)
                v = cadd(cmul(s00, U[i * ld + k]), cmul(s01, U[(i + d) * ld + k]));
            else
                v = cadd(cmul(s10, U[(i - d) * ld + k]), cmul(s11, U[i * ld + k]));
            M[i * ld + k] = v;
        }
        __syncthreads();
        // FP32 amplitudes, double-word level gaps and diagonal sum
        const float scale = (float)a.wscale[g] * (0.5f / (float)d);
        const float2 diag = !PRE      ? amplitudes_mixed(a, s, U, M, n, sn, scale)
                            : n == 24 ? amplitudes_rows<24>(a, s, U, M, n, sn, scale)
                            : n == 32 ? amplitudes_rows<32>(a, s, U, M, n, sn, scale)
                                      : amplitudes_rows<0>(a, s, U, M, n, sn, scale);
        const double dsum = dw_block_sum(diag, reinterpret_cast<float2 *>(s.w.red));
        if (tid == 0) {
            a.snap_const[sn] = 0.25 * a.wscale[g] * dsum / (double)d;
            a.status[g] = st;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ general path

// The term C_jk = rho'_jk O'_kj of a pair j >= k: its pair record (EVOLVE) or
// decaying-integral term (INTEGRAL); `local` collects the constant / integral.
template <bool INTEGRAL>
__device__ __forceinline__ void rho_term(const SnapArgs &a, const SnapSmem<float> &s, size_t rec, int j,
                                         int k, cx<float> r, cx<float> o, float scale2, float tau_f,
                                         float itau_f, float2 &local) {
    const float cr = r.re * o.re - r.im * o.im;
    const float ci = r.re * o.im + r.im * o.re;
    if (INTEGRAL) {
        // term = C_jk (-1) / (2 pi i (l_k - l_j) - 1/tau); pairs count twice
        if (j == k) {
            local = dw_add_f(local, cr * tau_f);
        } else {
            const float gap = dw_sub_f(s.lw[k], s.lw[j]);
            const float x = fmaf(gap, MSP_TWOPI_HI, gap * MSP_TWOPI_LO);
            const float den = fmaf(x, x, itau_f * itau_f);
            local = dw_add_f(local, 2.0f * (cr * itau_f - ci * x) / den);
        }
    } else {
        if (j == k) {
            local = dw_add_f(local, cr);
        } else {
            const size_t at = rec + pair_index(j, k);
            reinterpret_cast<float2 *>(a.pair_coef)[at] = make_float2(scale2 * cr, scale2 * ci);
            store_frequency_dw(a, at, dw_sub(s.lw[j], s.lw[k]));
        }
    }
}

// Every term j >= k with O'_kj = sum_i conj(U_ik) (O U)_ij; returns this thread's
// share of the constant / integral as a double-word.  rho' comes from rho0 U in
// X, or (hot) from O' itself: rho'_jk = (delta_jk + hot_scale O'_jk n) / n.
// !ROWS: rho'_jk in X already.
template <bool INTEGRAL, bool ROWS, int NN>
__device__ __forceinline__ float2 rho_terms_mixed(const SnapArgs &a, const SnapSmem<float> &s,
                                                  const cx<float> *U, const cx<float> *OU,
                                                  const cx<float> *X, int n_rt, int sn, float tau_f,
                                                  float itau_f, bool hot, float hot_scale) {
    const int n = NN > 0 ? NN : n_rt, ld = n + (n & 1) + 1;  // !ROWS
    const size_t rec = (size_t)sn * (n * (n - 1) / 2);
    const float scale2 = 2.0f * (float)a.wscale[sn];
    float2 local = make_float2(0.f, 0.f);
    auto rho_hot = [&](cx<float> o, bool diagonal) {
        return mk<float>(fmaf(hot_scale, o.re, diagonal ? 1.0f / (float)n : 0.f), -hot_scale * o.im);
    };
    if (ROWS) {
        // a thread's rows k <= j of column j (see oa_refine_rows)
        const RowShape sh = row_shape(n, blockDim.x);
        const int rg = threadIdx.x / n, j = threadIdx.x - rg * n, i0 = rg * sh.rows;
        if (rg >= sh.groups || i0 > j) return local;
        cx<float> o[ROW_MAX], r[ROW_MAX];
        row_products<NN, ROW_MAX>(U, OU, n, i0, j, o);
        if (!hot) row_products<NN, ROW_MAX>(U, X, n, i0, j, r);  // rho'_kj
#pragma unroll
        for (int q = 0; q < ROW_MAX; ++q) {
            const int k = i0 + q;
            if (q >= sh.rows || k > j) continue;
            rho_term<INTEGRAL>(a, s, rec, j, k, hot ? rho_hot(o[q], j == k) : conj(r[q]), o[q], scale2,
                               tau_f, itau_f, local);
        }
        return local;
    }
    const int ntri = n * (n + 1) / 2;
    for (int e = threadIdx.x; e < ntri; e += blockDim.x) {
        int j, k;
        tri_index(e, j, k);
        float orr = 0.f, oii = 0.f;
#pragma unroll 4
        for (int i = 0; i < n; ++i) {
            const cx<float> u = U[i * ld + k], x = OU[i * ld + j];
            orr += u.re * x.re + u.im * x.im;
            oii += u.re * x.im - u.im * x.re;
        }
        const cx<float> o = mk<float>(orr, oii);
        rho_term<INTEGRAL>(a, s, rec, j, k, hot ? rho_hot(o, j == k) : X[j * ld + k], o, scale2, tau_f,
                           itau_f, local);
    }
    return local;
}

// One snapshot of the general path: rho' = U^dag rho0 U, O' = U^dag O U with
// rho0 = (x)_s rho_s (Kronecker factors) and O = p . S_mu.  EVOLVE writes the
// pair coefficients of <O>(t) = sum_ij rho'_ij O'_ji exp(-i w_ij t)
// (muspinsim/hamiltonian.py:80-107); INTEGRAL writes the decaying integral
// divided by tau (muspinsim/hamiltonian.py:150-164, experiment.py:492-496).
// At T = inf rho' follows from O' (rho_is_hot), which leaves one eigenbasis
// product instead of two and the digit products.
// PRE: as in msp_snap_fast_kernel, 64 registers (four CTAs of 256 threads per SM
// at n = 32; 22.6 ms with 80, 25.5 with 96 where 64 take 22.1).
template <bool INTEGRAL, bool PRE>
__global__ void __maxnreg__(PRE ? 64 : 96) msp_snap_rho_kernel(SnapArgs a) {
    typedef float T;
    extern __shared__ __align__(16) char smem[];
    const int n = a.n, m = n + (n & 1), ld = PRE ? row_ld(n) : m + 1;
    SnapSmem<T> s =
        PRE ? row_carve(smem, n, true, a.fac_len) : snap_carve<T, true>(smem, n, true, a.fac_len);
    const int tid = threadIdx.x, nt = blockDim.x;
    const float tau_f = a.tau_f, itau_f = a.itau_f;
    __shared__ float hot_scale[1];

    for (int sn = blockIdx.x; sn < a.num_snap; sn += gridDim.x) {
        const bool hot = rho_is_hot(a, sn);
        // some forty FP64 operations: one thread's, read many barriers later
        if (hot && tid == nt - 1) *hot_scale = (float)rho_hot_scale(a, sn);
        if (a.rho_fac) {
            for (int e = tid; e < a.fac_len; e += nt)
                s.fac[e] = a.rho_fac[(size_t)sn * a.fac_len + e];
        } else if (!hot) {
            build_rho_factors(a, sn, s.fac);
        }
        if (PRE)
            load_hamiltonian_rows(snap_source(a, sn), a.field + 3 * (size_t)sn, n, s);
        else
            load_hamiltonian<PRE>(a.Hsys, a.Z, a.Hsys_dw, a.Z_dw, a.field + 3 * (size_t)sn, n, m, s);
        // made visible by the eigensolve's barriers
        if (!hot)
            for (int e = tid; e < a.fac_len; e += nt)
                s.facf[e] = mk<float>((float)s.fac[e].re, (float)s.fac[e].im);
        int st = snap_eigvecs<PRE>(a, sn, sn, n, m, ld, s);
        st |= PRE ? eigenpairs_rows(n, true, a.fac_len, a.max_refine)
                  : eigenpairs(s, n, m, a.max_refine);
        const cx<T> *U = s.w.U;

        const cx<T> *X = s.w.H;
        cx<T> *Y = s.B2;
        if (!hot) {
            // rho0 U by Kronecker factors: X ping-pongs between H and B2
            X = U;
            Y = s.w.H;
            int off = 0;
            for (int sp = 0; sp < a.num_spins; ++sp) {
                const int dim = a.dims[sp];
                apply_digit<T>(s.facf + off, dim, a.strides[sp], X, Y, n, ld);
                off += dim * dim;
                X = Y;
                Y = (Y == s.w.H) ? s.B2 : s.w.H;
            }
            if (!PRE) {
                // X holds rho0 U.  rho'_jk (j >= k) -> Y (the other buffer).
                tri_conj_products<T>(U, X, Y, n);
                __syncthreads();
                cx<T> *t = Y;
                Y = const_cast<cx<T> *>(X);
                X = t;
            }
        }
        // O U into the buffer Y (free now): O = sum_a p_a S^a on the muon digit
        cx<T> *OU = Y;
        {
            T px, py, pz;
            load_vec3<T>(a.pol + 3 * (size_t)sn, px, py, pz);
            const T h = T(0.5);
            const int stride = a.strides[a.mu_index];
            const cx<T> o00 = mk<T>(h * pz, T(0));
            const cx<T> o01 = mk<T>(h * px, -h * py);
            const cx<T> o10 = mk<T>(h * px, h * py);
            const cx<T> o11 = mk<T>(-h * pz, T(0));
            for (int e = tid; e < n * n; e += nt) {
                const int i = FastDiv(n).div(e), k = e - i * n;
                const int di = (i / stride) & 1;
                const int base = i - di * stride;
                const cx<T> x0 = U[base * ld + k], x1 = U[(base + stride) * ld + k];
                OU[i * ld + k] = di == 0 ? cadd(cmul(o00, x0), cmul(o01, x1))
                                        : cadd(cmul(o10, x0), cmul(o11, x1));
            }
        }
        __syncthreads();
        // FP32 terms, double-word level gaps and sums
        const float hs = hot ? *hot_scale : 0.f;
        const float2 local =
            PRE && n == 24
                ? rho_terms_mixed<INTEGRAL, PRE, PRE ? 24 : 0>(a, s, U, OU, X, n, sn, tau_f, itau_f, hot, hs)
            : PRE && n == 32
                ? rho_terms_mixed<INTEGRAL, PRE, PRE ? 32 : 0>(a, s, U, OU, X, n, sn, tau_f, itau_f, hot, hs)
                : rho_terms_mixed<INTEGRAL, PRE, 0>(a, s, U, OU, X, n, sn, tau_f, itau_f, hot, hs);
        const double sum = dw_block_sum(local, reinterpret_cast<float2 *>(s.w.red));
        if (tid == 0) {
            a.snap_const[sn] = INTEGRAL ? a.wscale[sn] * sum / a.tau : a.wscale[sn] * sum;
            a.status[sn] = st;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ launchers

int snap_default_threads(int n, int precision) {
    if (precision == MSP_PREC_MIXED && jacobi_warp_supported(n)) return row_threads(n);
    return jacobi_threads(n + (n & 1));
}

// Shared memory of a snapshot kernel launched with `threads` threads.  rows: the
// second stage of the two-stage MIXED form.
static size_t snap_smem_threads(int n, int mode, int precision, int fac_len, int threads, bool rows) {
    const bool rho = mode != MSP_MODE_FAST;
    if (precision != MSP_PREC_MIXED) return snap64_smem_bytes(n, rho ? fac_len : 0, threads);
    if (rows) return row_layout(n, rho, fac_len, threads).total;
    return snap_layout(n, 4, true, rho, fac_len, threads / 32).total;
}

size_t snap_smem_bytes(int n, int mode, int precision, int fac_len) {
    return snap_smem_threads(n, mode, precision, fac_len, jacobi_threads(n + (n & 1)), false);
}

template <typename K>
static cudaError_t launch_snap(K kernel, const SnapArgs &a, int grid, int threads, size_t smem,
                               cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <typename K>
static int occupancy_of(K kernel, int threads, size_t smem) {
    int blocks = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, threads, smem) !=
            cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return blocks > 0 ? blocks : 1;
}

// Threads of a snapshot kernel asked for `threads` (0: the default): the second
// stage of the two-stage MIXED form takes at least what its four rows per
// thread need.
static int stage2_threads(int n, int precision, int threads, bool rows) {
    const int least = rows && precision == MSP_PREC_MIXED ? row_threads(n) : 0;
    if (threads <= 0) threads = rows ? snap_default_threads(n, precision) : jacobi_threads(n + (n & 1));
    return threads < least ? least : threads;
}

int snap_occupancy(int n, int mode, int precision, int threads) {
    const bool pre = jacobi_warp_supported(n);
    threads = stage2_threads(n, precision, threads, pre);
    const size_t smem = snap_smem_threads(n, mode, precision, 0, threads, pre);
    if (mode != MSP_MODE_FAST) return 1;
    if (precision != MSP_PREC_MIXED) return snap64_occupancy(n, threads, pre);
    return pre ? occupancy_of(msp_snap_fast_kernel<true>, threads, smem)
               : occupancy_of(msp_snap_fast_kernel<false>, threads, smem);
}

size_t snap_evec_bytes(int n, long long num_snap) {
    if (!jacobi_warp_supported(n) || num_snap <= 0) return 0;
    return (size_t)num_snap * (size_t)n * (size_t)n * sizeof(float2);
}

// Second stage of the two-stage form: refinement and eigenbasis products from
// the eigenvectors the first stage left in a.evec.
cudaError_t launch_snapshots_refine(const SnapArgs &a, int mode, int precision, cudaStream_t st,
                                    int threads, int grid) {
    if (a.num_snap <= 0) return cudaSuccess;
    threads = stage2_threads(a.n, precision, threads, true);
    if (grid <= 0 || grid > a.num_snap) grid = a.num_snap;
    if (precision != MSP_PREC_MIXED) return launch_snapshots64(a, mode, true, st, threads, grid);
    const size_t smem = snap_smem_threads(a.n, mode, precision, a.fac_len, threads, true);
    if (mode == MSP_MODE_FAST)
        return launch_snap(msp_snap_fast_kernel<true>, a, grid, threads, smem, st);
    if (mode == MSP_MODE_EVOLVE)
        return launch_snap(msp_snap_rho_kernel<false, true>, a, grid, threads, smem, st);
    return launch_snap(msp_snap_rho_kernel<true, true>, a, grid, threads, smem, st);
}

// threads = 0: jacobi_threads(m); grid = 0: one CTA per snapshot.  Any
// other grid runs persistent CTAs that stride over the snapshots.
cudaError_t launch_snapshots(const SnapArgs &a, int mode, int precision, cudaStream_t st,
                             int threads, int grid) {
    if (a.num_snap <= 0) return cudaSuccess;
    if (grid <= 0 || grid > a.num_snap) grid = a.num_snap;
    if (a.evec != nullptr && jacobi_warp_supported(a.n)) {
        // two stages: FP32 eigenvectors, then refinement and eigenbasis products
        const cudaError_t e = launch_jacobi_warp(a, st);
        if (e != cudaSuccess) return e;
        return launch_snapshots_refine(a, mode, precision, st, threads, grid);
    }
    threads = stage2_threads(a.n, precision, threads, false);
    if (precision != MSP_PREC_MIXED) return launch_snapshots64(a, mode, false, st, threads, grid);
    const size_t smem = snap_smem_threads(a.n, mode, precision, a.fac_len, threads, false);
    if (mode == MSP_MODE_FAST)
        return launch_snap(msp_snap_fast_kernel<false>, a, grid, threads, smem, st);
    if (mode == MSP_MODE_EVOLVE)
        return launch_snap(msp_snap_rho_kernel<false, false>, a, grid, threads, smem, st);
    return launch_snap(msp_snap_rho_kernel<true, false>, a, grid, threads, smem, st);
}

__global__ void msp_split_dw_kernel(const cx<double> *__restrict__ Hsys, size_t nh,
                                    const cx<double> *__restrict__ Z, size_t nz,
                                    float4 *__restrict__ dst) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nh + nz; i += stride) {
        const cx<double> v = i < nh ? Hsys[i] : Z[i - nh];
        dst[i] = dw_split(make_double2(v.re, v.im));
    }
}

cudaError_t launch_split_dw(const double *Hsys, size_t nh, const double *Z, size_t nz,
                            float4 *dst, cudaStream_t st) {
    const size_t total = nh + nz;
    if (total == 0) return cudaSuccess;
    size_t grid = (total + 255) / 256;
    if (grid > 1024) grid = 1024;
    msp_split_dw_kernel<<<(unsigned)grid, 256, 0, st>>>(
        reinterpret_cast<const cx<double> *>(Hsys), nh, reinterpret_cast<const cx<double> *>(Z),
        nz, dst);
    return cudaGetLastError();
}

cudaError_t launch_eigh(const double *H, int n, int batch, int precision, int max_sweeps,
                        double *evals, double *evecs, int *status, cudaStream_t st) {
    if (precision != MSP_PREC_MIXED)
        return launch_eigh64(H, n, batch, max_sweeps, evals, evecs, status, st);
    const int threads = jacobi_threads(n + (n & 1));
    const size_t smem = snap_smem_bytes(n, MSP_MODE_FAST, precision, 0);
    const cudaError_t e = cudaFuncSetAttribute(
        msp_eigh_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    msp_eigh_kernel<<<batch, threads, smem, st>>>(reinterpret_cast<const cx<double> *>(H), n, batch,
                                                  max_sweeps, evals,
                                                  reinterpret_cast<cx<double> *>(evecs), status);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ assemble / basis change

__global__ void msp_assemble_kernel(const cx<double> *__restrict__ Hsys,
                                    const cx<double> *__restrict__ Z,
                                    const double *__restrict__ fields, int n, int batch,
                                    cx<double> *__restrict__ H) {
    const size_t nn = (size_t)n * n;
    const size_t total = nn * batch;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
         e += (size_t)gridDim.x * blockDim.x) {
        const size_t b = e / nn, o = e - b * nn;
        const double bx = fields[3 * b], by = fields[3 * b + 1], bz = fields[3 * b + 2];
        const cx<double> hs = Hsys[o], z0 = Z[o], z1 = Z[nn + o], z2 = Z[2 * nn + o];
        H[e] = mk<double>(hs.re + bx * z0.re + by * z1.re + bz * z2.re,
                          hs.im + bx * z0.im + by * z1.im + bz * z2.im);
    }
}

cudaError_t launch_assemble(const double *Hsys, const double *Z, const double *fields, int n,
                            int batch, double *H, cudaStream_t st) {
    const size_t total = (size_t)n * n * batch;
    int grid = (int)((total + 255) / 256);
    if (grid > 152 * 32) grid = 152 * 32;
    if (grid < 1) grid = 1;
    msp_assemble_kernel<<<grid, 256, 0, st>>>(reinterpret_cast<const cx<double> *>(Hsys),
                                              reinterpret_cast<const cx<double> *>(Z), fields, n,
                                              batch, reinterpret_cast<cx<double> *>(H));
    return cudaGetLastError();
}

// out = U^dag M U (adjoint = 0) or U M U^dag (adjoint = 1), FP64, n <= 64.  One
// CTA per MSP_BC_COLS columns of a matrix (few matrices come per call: one
// CTA for all of a 24 x 24 one took 53 us): T = M U (or M U^dag) for these
// columns in shared memory, then U^dag T (or U T).
#define MSP_BC_COLS 4
__global__ void __launch_bounds__(128) msp_basis_change_kernel(
    const cx<double> *__restrict__ U, long long u_stride, const cx<double> *__restrict__ M,
    long long m_stride, int n, int batch, int adjoint, cx<double> *__restrict__ out) {
    extern __shared__ __align__(16) char smem[];
    const int ld = n + 1;  // odd or even, rows and columns both spread over the banks
    cx<double> *sU = reinterpret_cast<cx<double> *>(smem);
    cx<double> *sT = sU + n * ld;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int k0 = blockIdx.y * MSP_BC_COLS, kn = n - k0 < MSP_BC_COLS ? n - k0 : MSP_BC_COLS;
    for (int b = blockIdx.x; b < batch; b += gridDim.x) {
        const cx<double> *Ub = U + (size_t)b * u_stride;
        const cx<double> *Mb = M + (size_t)b * m_stride;
        if (u_stride != 0 || b == (int)blockIdx.x)
            for (int e = tid; e < n * n; e += nt) sU[(e / n) * ld + e % n] = Ub[e];
        __syncthreads();
        for (int e = tid; e < n * kn; e += nt) {
            const int i = e / kn, k = k0 + e - (e / kn) * kn;
            double r0 = 0, r1 = 0, i0 = 0, i1 = 0;
            for (int l = 0; l < n; ++l) {
                const cx<double> mv = Mb[i * n + l];
                // adjoint: (U^dag)_lk = conj(U_kl)
                const cx<double> uv = adjoint ? conj(sU[k * ld + l]) : sU[l * ld + k];
                r0 = fma(mv.re, uv.re, r0);
                r1 = fma(-mv.im, uv.im, r1);
                i0 = fma(mv.re, uv.im, i0);
                i1 = fma(mv.im, uv.re, i1);
            }
            sT[e] = mk<double>(r0 + r1, i0 + i1);
        }
        __syncthreads();
        cx<double> *Ob = out + (size_t)b * n * n;
        for (int e = tid; e < n * kn; e += nt) {
            const int j = e / kn, q = e - (e / kn) * kn;
            double r0 = 0, r1 = 0, i0 = 0, i1 = 0;
            for (int i = 0; i < n; ++i) {
                // row j of U^dag = conj(U_ij); row j of U = U_ji
                const cx<double> uv = adjoint ? sU[j * ld + i] : conj(sU[i * ld + j]);
                const cx<double> tv = sT[i * kn + q];
                r0 = fma(uv.re, tv.re, r0);
                r1 = fma(-uv.im, tv.im, r1);
                i0 = fma(uv.re, tv.im, i0);
                i1 = fma(uv.im, tv.re, i1);
            }
            Ob[(size_t)j * n + k0 + q] = mk<double>(r0 + r1, i0 + i1);
        }
        __syncthreads();
    }
}

// n > 64: the same product from global memory in two launches, one CTA
// per (column j, matrix): T = M op(U) into out (op(U) = U, or U^dag when
// adjoint), then out = op'(U) T (op'(U) = U^dag, or U).  Each CTA first
// stages its column (of op(U), then of T) in shared memory, so the second
// pass overwrites column j in place.
__global__ void msp_basis_change_col1_kernel(const cx<double> *__restrict__ U, long long u_stride,
                                             const cx<double> *__restrict__ M, long long m_stride,
                                             int n, int adjoint, int b0,
                                             cx<double> *__restrict__ out) {
    extern __shared__ __align__(16) char smem[];
    cx<double> *col = reinterpret_cast<cx<double> *>(smem);
    const int j = blockIdx.x, b = b0 + blockIdx.y, tid = threadIdx.x, nt = blockDim.x;
    const cx<double> *Ub = U + (size_t)b * u_stride;
    const cx<double> *Mb = M + (size_t)b * m_stride;
    cx<double> *Ob = out + (size_t)b * n * n;
    for (int l = tid; l < n; l += nt)
        col[l] = adjoint ? conj(Ub[(size_t)j * n + l]) : Ub[(size_t)l * n + j];
    __syncthreads();
    for (int i = tid; i < n; i += nt) {
        const cx<double> *row = Mb + (size_t)i * n;
        double tr = 0, ti = 0;
        for (int l = 0; l < n; ++l) {
            const cx<double> mv = row[l], uv = col[l];
            tr += mv.re * uv.re - mv.im * uv.im;
            ti += mv.re * uv.im + mv.im * uv.re;
        }
        Ob[(size_t)i * n + j] = mk<double>(tr, ti);
    }
}

__global__ void msp_basis_change_col2_kernel(const cx<double> *__restrict__ U, long long u_stride,
                                             int n, int adjoint, int b0,
                                             cx<double> *__restrict__ out) {
    extern __shared__ __align__(16) char smem[];
    cx<double> *col = reinterpret_cast<cx<double> *>(smem);
    const int j = blockIdx.x, b = b0 + blockIdx.y, tid = threadIdx.x, nt = blockDim.x;
    const cx<double> *Ub = U + (size_t)b * u_stride;
    cx<double> *Ob = out + (size_t)b * n * n;
    for (int k = tid; k < n; k += nt) col[k] = Ob[(size_t)k * n + j];
    __syncthreads();
    for (int i = tid; i < n; i += nt) {
        double tr = 0, ti = 0;
        for (int k = 0; k < n; ++k) {
            // row i of U^dag = conj(U_ki); row i of U = U_ik
            const cx<double> uv = adjoint ? Ub[(size_t)i * n + k] : conj(Ub[(size_t)k * n + i]);
            const cx<double> tv = col[k];
            tr += uv.re * tv.re - uv.im * tv.im;
            ti += uv.re * tv.im + uv.im * tv.re;
        }
        Ob[(size_t)i * n + j] = mk<double>(tr, ti);
    }
}

cudaError_t launch_basis_change(const double *U, long long u_stride, const double *M,
                                long long m_stride, int n, int batch, int adjoint, double *out,
                                cudaStream_t st) {
    if (n > MSP_MAX_DIM) {
        const size_t smem = (size_t)n * sizeof(cx<double>);
        const cx<double> *Uc = reinterpret_cast<const cx<double> *>(U);
        cx<double> *Oc = reinterpret_cast<cx<double> *>(out);
        for (int b0 = 0; b0 < batch; b0 += 65535) {
            const dim3 grid(n, batch - b0 < 65535 ? batch - b0 : 65535);
            msp_basis_change_col1_kernel<<<grid, 256, smem, st>>>(
                Uc, u_stride, reinterpret_cast<const cx<double> *>(M), m_stride, n, adjoint, b0,
                Oc);
            msp_basis_change_col2_kernel<<<grid, 256, smem, st>>>(Uc, u_stride, n, adjoint, b0,
                                                                  Oc);
        }
        return cudaGetLastError();
    }
    const size_t smem = ((size_t)n * (n + 1) + (size_t)n * MSP_BC_COLS) * sizeof(cx<double>);
    cudaError_t e = cudaFuncSetAttribute(msp_basis_change_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const dim3 grid(batch < 152 * 8 ? batch : 152 * 8, (n + MSP_BC_COLS - 1) / MSP_BC_COLS);
    msp_basis_change_kernel<<<grid, 128, smem, st>>>(
        reinterpret_cast<const cx<double> *>(U), u_stride,
        reinterpret_cast<const cx<double> *>(M), m_stride, n, batch, adjoint,
        reinterpret_cast<cx<double> *>(out));
    return cudaGetLastError();
}

}  // namespace msp
