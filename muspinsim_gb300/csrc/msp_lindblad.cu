// Dissipative (Lindblad) propagation: the path ExperimentRunner takes when
// the configuration has dissipation terms (muspinsim/experiment.py:272-341)
// and the Lindbladian class it builds (muspinsim/lindbladian.py:17-173).
//
// The reference diagonalises the n^2 x n^2 superoperator L with a dense
// non-Hermitian eig and writes rho(t) = V exp(2 pi Lambda t) V^-1 rho0 and
// the decaying integral as sum_k rho'_k O'_k / (1/tau - 2 pi lambda_k).
// Both are functions of L alone, computed here without an eigensolver:
//   * evolution: E = exp(2 pi L dt) by scaling and squaring of a degree-13
//     Taylor polynomial (Horner form, ||2 pi L dt / 2^s||_1 <= 1/2, truncation
//     below 1e-15), then rho(t_{k+1}) = E rho(t_k); a uniform grid needs
//     exp(2 pi L t0) and exp(2 pi L dt) only, a non-uniform grid one
//     exponential per interval;
//   * integral: O^T-weighted solution of (1/tau - 2 pi L) x = rho0 by
//     Gaussian elimination with partial pivoting (the matrix is regular:
//     Re lambda <= 0 for a Lindbladian and 1/tau > 0).
// Same values up to rounding, and no ill-conditioned eigenvector matrix
// when L is (nearly) defective.  FP64 in both precisions.
//
// One CTA per superoperator problem; its N x N matrices (N = n^2) live in a
// per-CTA slice of the caller's workspace.  The driver's evolution on a
// uniform grid with N <= 64 takes the real form further down instead.
#include <math_constants.h>
#include <string.h>

#include <algorithm>

#include "msp_internal.cuh"
#include "msp_rho.cuh"

namespace msp {
int record_error(int code, const char *msg);
}

using namespace msp;

typedef cx<double> zd;

#define MSP_LB_THREADS 256
#define MSP_LB_MAX_N2 1024  // superoperator dimension (n <= 32)

namespace {

// Per-CTA scratch, complex entries: L, A (LU / spare), X, T (N x N);
// v, w (N); o (num_ops x N); H, Mx, Ax (n x n); pivot row indices (N ints,
// stored in N complex slots).
struct LbWork {
    zd *L, *A, *X, *T, *v, *w, *o, *H, *M, *D;
    int *piv;
};

__host__ __device__ inline size_t lb_entries(int n, int num_ops) {
    const size_t N = (size_t)n * n;
    return 4 * N * N + (2 + (size_t)num_ops) * N + 3 * (size_t)n * n + N + 32;
}

__device__ inline LbWork lb_carve(zd *base, int n, int num_ops) {
    const size_t N = (size_t)n * n;
    LbWork w;
    w.L = base;
    w.A = w.L + N * N;
    w.X = w.A + N * N;
    w.T = w.X + N * N;
    w.v = w.T + N * N;
    w.w = w.v + N;
    w.o = w.w + N;
    w.H = w.o + (size_t)num_ops * N;
    w.M = w.H + (size_t)n * n;
    w.D = w.M + (size_t)n * n;
    w.piv = reinterpret_cast<int *>(w.D + (size_t)n * n);
    return w;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ double warp_sumd(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide maximum (every thread gets it); red: >= 32 doubles.
__device__ double lb_block_max(double v, double *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double m = 0.0;
    for (int k = 0; k < nw; ++k) m = fmax(m, red[k]);
    __syncthreads();
    return m;
}

// Block-wide complex sum (every thread gets it); red: >= 64 doubles.
__device__ zd lb_block_csum(zd v, double *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v.re = warp_sumd(v.re);
    v.im = warp_sumd(v.im);
    __syncthreads();
    if (lane == 0) {
        red[warp] = v.re;
        red[32 + warp] = v.im;
    }
    __syncthreads();
    zd s = mk<double>(0.0, 0.0);
    for (int k = 0; k < nw; ++k) {
        s.re += red[k];
        s.im += red[32 + k];
    }
    __syncthreads();
    return s;
}

// C = A B (N x N, row-major); C aliases neither.
__device__ void lb_gemm(zd *C, const zd *A, const zd *B, int N) {
    const int NN = N * N;
    for (int e = threadIdx.x; e < NN; e += blockDim.x) {
        const int i = e / N, j = e - (e / N) * N;
        const zd *a = A + (size_t)i * N;
        double cr = 0.0, ci = 0.0;
        for (int k = 0; k < N; ++k) {
            const zd x = a[k], y = B[(size_t)k * N + j];
            cr = fma(x.re, y.re, cr);
            cr = fma(-x.im, y.im, cr);
            ci = fma(x.re, y.im, ci);
            ci = fma(x.im, y.re, ci);
        }
        C[e] = mk<double>(cr, ci);
    }
    __syncthreads();
}

// y = E x, a warp per row.
__device__ void lb_matvec(zd *y, const zd *E, const zd *x, int N) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int i = warp; i < N; i += nw) {
        const zd *row = E + (size_t)i * N;
        double cr = 0.0, ci = 0.0;
        for (int k = lane; k < N; k += 32) {
            const zd a = row[k], b = x[k];
            cr = fma(a.re, b.re, cr);
            cr = fma(-a.im, b.im, cr);
            ci = fma(a.re, b.im, ci);
            ci = fma(a.im, b.re, ci);
        }
        cr = warp_sumd(cr);
        ci = warp_sumd(ci);
        if (lane == 0) y[i] = mk<double>(cr, ci);
    }
    __syncthreads();
}

// exp(f L) into the returned buffer (w.X or w.T).
__device__ zd *lb_expm(LbWork &w, int N, double f, double *red) {
    const int tid = threadIdx.x, nt = blockDim.x, NN = N * N;
    double cmax = 0.0;
    for (int j = tid; j < N; j += nt) {
        double s = 0.0;
        for (int i = 0; i < N; ++i) {
            const zd x = w.L[(size_t)i * N + j];
            s += sqrt(x.re * x.re + x.im * x.im);
        }
        cmax = fmax(cmax, s);
    }
    double nrm = lb_block_max(cmax, red) * fabs(f);
    int sq = 0;
    while (nrm > 0.5 && sq < 64) {
        nrm *= 0.5;
        ++sq;
    }
    const double g = ldexp(f, -sq);
    for (int e = tid; e < NN; e += nt) w.X[e] = mk<double>((e / N) == (e % N) ? 1.0 : 0.0, 0.0);
    __syncthreads();
    for (int k = 13; k >= 1; --k) {  // X <- I + (g / k) L X
        lb_gemm(w.T, w.L, w.X, N);
        const double c = g / (double)k;
        for (int e = tid; e < NN; e += nt) {
            const zd t = w.T[e];
            w.X[e] = mk<double>(((e / N) == (e % N) ? 1.0 : 0.0) + c * t.re, c * t.im);
        }
        __syncthreads();
    }
    zd *P = w.X, *Q = w.T;
    for (int s = 0; s < sq; ++s) {
        lb_gemm(Q, P, P, N);
        zd *t = P;
        P = Q;
        Q = t;
    }
    return P;
}

// Expectations (or states) of one time sample.
__device__ void lb_emit(const LbWork &w, int N, int num_ops, const zd *v, double *red,
                        zd *out_c, double *out_r, double weight) {
    if (num_ops == 0) {  // states
        for (int e = threadIdx.x; e < N; e += blockDim.x) out_c[e] = v[e];
        return;
    }
    for (int op = 0; op < num_ops; ++op) {
        zd acc = mk<double>(0.0, 0.0);
        for (int e = threadIdx.x; e < N; e += blockDim.x) acc = cadd(acc, cmul(w.o[(size_t)op * N + e], v[e]));
        const zd s = lb_block_csum(acc, red);
        if (threadIdx.x == 0) {
            if (out_c) out_c[op] = s;
            if (out_r) out_r[op] = s.re * weight;
        }
    }
}

// Time series of rho(t) = exp(2 pi L t) rho0 (w.L, w.v hold L and rho0):
// outputs per time through lb_emit.
__device__ void lb_evolve(LbWork &w, int N, int num_ops, const double *times, int num_times,
                          int uniform, double t0, double dt, double *red, zd *out_c,
                          double *out_r, double weight) {
    zd *v = w.v, *y = w.w;
    zd *E = nullptr;
    double t_prev = 0.0;
    if (uniform && t0 != 0.0) {  // to the first sample
        E = lb_expm(w, N, 2.0 * CUDART_PI * t0, red);
        lb_matvec(y, E, v, N);
        zd *t = v;
        v = y;
        y = t;
        E = nullptr;
    }
    for (int k = 0; k < num_times; ++k) {
        if (uniform) {
            if (k > 0) {
                if (E == nullptr) E = lb_expm(w, N, 2.0 * CUDART_PI * dt, red);
                lb_matvec(y, E, v, N);
                zd *t = v;
                v = y;
                y = t;
            }
        } else {
            const double tk = times[k], step = tk - t_prev;
            if (step != 0.0) {
                E = lb_expm(w, N, 2.0 * CUDART_PI * step, red);
                lb_matvec(y, E, v, N);
                zd *t = v;
                v = y;
                y = t;
            }
            t_prev = tk;
        }
        lb_emit(w, N, num_ops, v, red,
                out_c ? out_c + (size_t)k * (num_ops ? num_ops : N) : nullptr,
                out_r ? out_r + (size_t)k * num_ops : nullptr, weight);
        __syncthreads();
    }
}

// x = (1/tau - 2 pi L)^-1 rho0 into w.v; w.A holds the factors.
__device__ void lb_solve(LbWork &w, int N, double tau, double *red) {
    const int tid = threadIdx.x, nt = blockDim.x, NN = N * N;
    const double inv_tau = 1.0 / tau, tp = 2.0 * CUDART_PI;
    for (int e = tid; e < NN; e += nt) {
        const zd l = w.L[e];
        w.A[e] = mk<double>(((e / N) == (e % N) ? inv_tau : 0.0) - tp * l.re, -tp * l.im);
    }
    __syncthreads();
    __shared__ int s_piv;
    zd *M = w.A, *b = w.v, *f = w.w;
    for (int k = 0; k < N; ++k) {
        // pivot: largest |M[i][k]|, i >= k (warp 0 scans)
        if (threadIdx.x < 32) {
            double best = -1.0;
            int bi = k;
            for (int i = k + (int)threadIdx.x; i < N; i += 32) {
                const zd x = M[(size_t)i * N + k];
                const double a = x.re * x.re + x.im * x.im;
                if (a > best) {
                    best = a;
                    bi = i;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) {
                    best = ob;
                    bi = oi;
                }
            }
            if (threadIdx.x == 0) s_piv = bi;
        }
        __syncthreads();
        const int p = s_piv;
        if (p != k) {
            for (int j = tid; j < N; j += nt) {
                const zd t = M[(size_t)k * N + j];
                M[(size_t)k * N + j] = M[(size_t)p * N + j];
                M[(size_t)p * N + j] = t;
            }
            if (tid == 0) {
                const zd t = b[k];
                b[k] = b[p];
                b[p] = t;
            }
        }
        __syncthreads();
        const zd piv = M[(size_t)k * N + k];
        const double dd = 1.0 / (piv.re * piv.re + piv.im * piv.im);
        const zd inv = mk<double>(piv.re * dd, -piv.im * dd);
        for (int i = k + 1 + tid; i < N; i += nt) f[i] = cmul(M[(size_t)i * N + k], inv);
        __syncthreads();
        const int rows = N - k - 1, cols = N - k - 1;
        for (int e = tid; e < rows * (cols + 1); e += nt) {
            const int i = k + 1 + e / (cols + 1), jj = e - (e / (cols + 1)) * (cols + 1);
            if (jj == cols) {
                const zd t = cmul(f[i], b[k]);
                b[i] = mk<double>(b[i].re - t.re, b[i].im - t.im);
            } else {
                const int j = k + 1 + jj;
                const zd t = cmul(f[i], M[(size_t)k * N + j]);
                M[(size_t)i * N + j] = mk<double>(M[(size_t)i * N + j].re - t.re,
                                                  M[(size_t)i * N + j].im - t.im);
            }
        }
        __syncthreads();
    }
    // back substitution, column oriented
    for (int k = N - 1; k >= 0; --k) {
        if (tid == 0) {
            const zd piv = M[(size_t)k * N + k];
            const double dd = 1.0 / (piv.re * piv.re + piv.im * piv.im);
            b[k] = cmul(b[k], mk<double>(piv.re * dd, -piv.im * dd));
        }
        __syncthreads();
        const zd xk = b[k];
        for (int i = tid; i < k; i += nt) {
            const zd t = cmul(M[(size_t)i * N + k], xk);
            b[i] = mk<double>(b[i].re - t.re, b[i].im - t.im);
        }
        __syncthreads();
    }
    (void)red;
}

// o[op] = vec(O_op^T): o[i n + j] = O[j][i]
__device__ void lb_observables(LbWork &w, const zd *ops, int num_ops, int n) {
    const int N = n * n;
    for (int e = threadIdx.x; e < num_ops * N; e += blockDim.x) {
        const int op = e / N, r = e - op * N, i = r / n, j = r - (r / n) * n;
        w.o[e] = ops[(size_t)op * N + (size_t)j * n + i];
    }
    __syncthreads();
}

__global__ void __launch_bounds__(MSP_LB_THREADS) msp_superop_kernel(
    const zd *__restrict__ L, int n, const zd *__restrict__ rho0, const zd *__restrict__ ops,
    int num_ops, const double *__restrict__ times, int num_times, int uniform, double t0,
    double dt, int integral, double tau, zd *__restrict__ out, zd *__restrict__ scratch) {
    __shared__ double red[64];
    const int N = n * n;
    LbWork w = lb_carve(scratch, n, num_ops);
    for (int e = threadIdx.x; e < N * N; e += blockDim.x) w.L[e] = L[e];
    for (int e = threadIdx.x; e < N; e += blockDim.x) w.v[e] = rho0[e];
    __syncthreads();
    lb_observables(w, ops, num_ops, n);
    if (integral) {
        lb_solve(w, N, tau, red);
        lb_emit(w, N, num_ops, w.v, red, out, nullptr, 1.0);
    } else {
        lb_evolve(w, N, num_ops, times, num_times, uniform, t0, dt, red, out, nullptr, 1.0);
    }
}

// ---------------------------------------------------------------- batched driver path

struct LbArgs {
    SnapArgs sa;             // n, spins, field, pol, temperature, gammas (rho0 factors)
    const zd *spin_ops;      // num_spins x 3 x n x n: S^a_i embedded
    int num_diss;
    int diss_spin[MSP_MAX_SPINS];
    double diss_rate[MSP_MAX_SPINS];
    const double *times;
    int num_times, uniform;
    double t0, dt;
    int integral;
    double *res;             // num_snap x T (real part x wscale)
    zd *scratch;
    size_t scratch_entries;  // per CTA
};

// Two axes orthogonal to z (muspinsim/utils.py:71-93), z a unit vector.
__device__ inline void lb_get_xy(const double *z, double *x, double *y) {
    if (z[0] == 0.0 && z[1] == 0.0) {
        x[0] = 1.0; x[1] = 0.0; x[2] = 0.0;
        y[0] = 0.0; y[1] = z[2]; y[2] = 0.0;
        return;
    }
    const double r = sqrt(z[0] * z[0] + z[1] * z[1]);
    x[0] = z[1] / r; x[1] = -z[0] / r; x[2] = 0.0;
    y[0] = z[1] * x[2] - z[2] * x[1];
    y[1] = z[2] * x[0] - z[0] * x[2];
    y[2] = z[0] * x[1] - z[1] * x[0];
}

__global__ void __launch_bounds__(MSP_LB_THREADS) msp_lindblad_kernel(LbArgs a) {
    __shared__ double red[64];
    __shared__ zd fac[MSP_MAX_SPINS * MSP_FACTOR_MAXD * MSP_FACTOR_MAXD];
    __shared__ double axes[6];
    const SnapArgs &sa = a.sa;
    const int n = sa.n, N = n * n, tid = threadIdx.x, nt = blockDim.x;
    LbWork w = lb_carve(a.scratch + (size_t)blockIdx.x * a.scratch_entries, n, 1);
    const size_t nn = (size_t)n * n;
    for (int s = blockIdx.x; s < sa.num_snap; s += gridDim.x) {
        const double *b = sa.field + 3 * (size_t)s, *p = sa.pol + 3 * (size_t)s;
        const double Bn = sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
        const double T = sa.temperature ? sa.temperature[s] : CUDART_INF;
        // H = Hsys + b . Z; rho0 factors; dissipator axes
        for (size_t e = tid; e < nn; e += nt) {
            const zd hs = sa.Hsys[e], z0 = sa.Z[e], z1 = sa.Z[nn + e], z2 = sa.Z[2 * nn + e];
            w.H[e] = mk<double>(hs.re + b[0] * z0.re + b[1] * z1.re + b[2] * z2.re,
                                hs.im + b[0] * z0.im + b[1] * z1.im + b[2] * z2.im);
        }
        build_rho_factors(sa, s, fac);
        if (tid == 0) {
            double x[3] = {1.0, 0.0, 0.0}, y[3] = {0.0, 1.0, 0.0};
            if (Bn != 0.0) {
                const double z[3] = {b[0] / Bn, b[1] / Bn, b[2] / Bn};
                lb_get_xy(z, x, y);
            }
            for (int k = 0; k < 3; ++k) {
                axes[k] = x[k];
                axes[3 + k] = y[k];
            }
        }
        __syncthreads();
        // rho0 = Kronecker product of the factors (spin 0 the slowest digit)
        for (int e = tid; e < N; e += nt) {
            int i = e / n, j = e - (e / n) * n, off = 0;
            zd r = mk<double>(1.0, 0.0);
            int ri = i, rj = j, stride = n;
            for (int q = 0; q < sa.num_spins; ++q) {
                const int dq = sa.dims[q];
                stride /= dq;
                const int di = ri / stride, dj = rj / stride;
                ri -= di * stride;
                rj -= dj * stride;
                r = cmul(r, fac[off + di * dq + dj]);
                off += dq * dq;
            }
            w.v[e] = r;
        }
        // observable: O = p . S_mu, o = vec(O^T)
        const zd *Smu = a.spin_ops + (size_t)sa.mu_index * 3 * nn;
        for (int e = tid; e < N; e += nt) {
            const int i = e / n, j = e - (e / n) * n;
            const size_t q = (size_t)j * n + i;
            w.o[e] = mk<double>(p[0] * Smu[q].re + p[1] * Smu[nn + q].re + p[2] * Smu[2 * nn + q].re,
                                p[0] * Smu[q].im + p[1] * Smu[nn + q].im + p[2] * Smu[2 * nn + q].im);
        }
        __syncthreads();
        // L: -i (H (x) 1 - 1 (x) H^T)
        for (int e = tid; e < N * N; e += nt) {
            const int r = e / N, c = e - (e / N) * N;
            const int i = r / n, j = r - (r / n) * n, k = c / n, l = c - (c / n) * n;
            zd v = mk<double>(0.0, 0.0);
            if (j == l) v = cadd(v, w.H[(size_t)i * n + k]);
            if (i == k) {
                const zd h = w.H[(size_t)l * n + j];
                v = mk<double>(v.re - h.re, v.im - h.im);
            }
            w.L[e] = mk<double>(v.im, -v.re);  // -i v
        }
        __syncthreads();
        // dissipators: S+ and S- about the field of each dissipative spin
        for (int d = 0; d < a.num_diss; ++d) {
            const int si = a.diss_spin[d];
            const double rate = a.diss_rate[d];
            double Zu = 0.0;
            if (T > 0.0) Zu = exp(-6.62607015e-34 * sa.gammas[si] * Bn * 1e6 / (1.380649e-23 * T));
            const zd *S = a.spin_ops + (size_t)si * 3 * nn;
            for (int pm = 0; pm < 2; ++pm) {
                const double g = pm == 0 ? rate * Zu / (CUDART_PI * (1.0 + Zu))
                                         : rate / (CUDART_PI * (1.0 + Zu));
                const double sg = pm == 0 ? 1.0 : -1.0;
                if (g == 0.0) continue;
                // D = op_x +/- i op_y
                for (size_t e = tid; e < nn; e += nt) {
                    double xr = 0, xi = 0, yr = 0, yi = 0;
                    for (int c = 0; c < 3; ++c) {
                        const zd sc = S[c * nn + e];
                        xr += axes[c] * sc.re;
                        xi += axes[c] * sc.im;
                        yr += axes[3 + c] * sc.re;
                        yi += axes[3 + c] * sc.im;
                    }
                    w.D[e] = mk<double>(xr - sg * yi, xi + sg * yr);
                }
                __syncthreads();
                // M = D^H D
                for (size_t e = tid; e < nn; e += nt) {
                    const int i = (int)(e / n), j = (int)(e - (e / n) * n);
                    double mr = 0, mi = 0;
                    for (int k = 0; k < n; ++k) {
                        const zd x = w.D[(size_t)k * n + i], y = w.D[(size_t)k * n + j];
                        mr += x.re * y.re + x.im * y.im;
                        mi += x.re * y.im - x.im * y.re;
                    }
                    w.M[e] = mk<double>(mr, mi);
                }
                __syncthreads();
                // L += g [D (x) conj(D) - 1/2 (M (x) 1 + 1 (x) M^T)]
                for (int e = tid; e < N * N; e += nt) {
                    const int r = e / N, c = e - (e / N) * N;
                    const int i = r / n, j = r - (r / n) * n, k = c / n, l = c - (c / n) * n;
                    const zd dik = w.D[(size_t)i * n + k], djl = w.D[(size_t)j * n + l];
                    zd v = cmul(dik, mk<double>(djl.re, -djl.im));
                    if (j == l) {
                        const zd m = w.M[(size_t)i * n + k];
                        v = mk<double>(v.re - 0.5 * m.re, v.im - 0.5 * m.im);
                    }
                    if (i == k) {
                        const zd m = w.M[(size_t)l * n + j];
                        v = mk<double>(v.re - 0.5 * m.re, v.im - 0.5 * m.im);
                    }
                    const zd lv = w.L[e];
                    w.L[e] = mk<double>(lv.re + g * v.re, lv.im + g * v.im);
                }
                __syncthreads();
            }
        }
        const double weight = sa.wscale[s];
        double *res = a.res + (size_t)s * a.num_times;
        if (a.integral) {
            lb_solve(w, N, sa.tau, red);
            lb_emit(w, N, 1, w.v, red, nullptr, res, weight / sa.tau);
        } else {
            lb_evolve(w, N, 1, a.times, a.num_times, a.uniform, a.t0, a.dt, red, nullptr, res,
                      weight);
        }
        if (tid == 0 && sa.status) sa.status[s] = MSP_ITEM_OK;
        __syncthreads();
    }
}

// ---------------------------------------------------------------- real form
// Evolution on a uniform grid, N = n^2 <= 64 (both precisions).  What bounds it
// is the FP64 pipe (1/74 of the FP32 rate), so the form with the fewest FP64
// operations is taken:
//   * a Lindbladian maps Hermitian matrices to Hermitian ones, so in the
//     orthonormal Hermitian basis (E_ii, (E_ij + E_ji) / sqrt 2, i (E_ij - E_ji) /
//     sqrt 2) it is a REAL N x N matrix: one FMA per product term instead of
//     four;
//   * exp(A), ||A||_2 <= 0.9 after scaling, is the degree-16 Taylor polynomial
//     (truncation 5e-16) in powers of A^4 (Paterson and Stockmeyer 1973): six
//     products instead of thirteen or more;
//   * samples come from y_{j b + i} = (o^T F^j) (E^i rho0), F = E^b by log2 b
//     further squarings: b + T / b matrix-vector products instead of T.
// One CTA per snapshot, everything in shared memory (six N x N matrices; ld =
// N + 4 keeps the row-parallel matrix-vector product free of bank conflicts);
// a product is 4 x 4 outputs per thread.  mu, e, 1H (N = 64), 200 snapshots x
// 1000 times: 34.4 -> 2.4 ms (FP64 as above) and 4.3 -> 2.4 ms (double-word
// FP32 propagation); 15 products' worth of FMAs on 200 CTAs over 152 SMs.
constexpr int LBR_MAXN = 64, LBR_THREADS = 256, LBR_GIANTS = 128;
constexpr int LBR_FAC = 96;  // rho0 factors: sum of d^2 for a product of d up to 8, and spins 0
constexpr size_t LBR_SMEM_MAX = 224 * 1024;  // beside the kernel's static arrays (3 KB)

struct LbrShape {
    int b, lg;  // samples per giant step, log2
    int skip;   // squarings of the step's exponential left out (b = 1)
};

// Squarings of exp(A) that pay less than its 2^k applications to a vector would, when
// it acts `steps` times: a squaring takes N^3 FMAs, an application N^2 and about as
// long again for its barriers.  n = 8, 2,000 snapshots, 2 samples: 21.3 ms with all
// fifteen squarings, 17.5 without the last of them.
__host__ __device__ inline int lbr_skip(int N, double steps) {
    int skip = 0;
    double best = 2.0 * steps;
    for (int k = 1; k <= 6; ++k) {
        const double c = 2.0 * steps * (double)(1 << k) - k * (double)N;
        if (c < best) {
            best = c;
            skip = k;
        }
    }
    return skip;
}

// b = 2^lg minimises log2(b) N^3 + (b + T / b) N^2.
__host__ __device__ inline LbrShape lbr_shape(int N, int T) {
    LbrShape s = {1, 0, 0};
    double best = 1e300;
    for (int lg = 0; lg <= 6; ++lg) {
        const double b = (double)(1 << lg), c = lg * (double)N + b + (T + b - 1.0) / b;
        if (c < best) {
            best = c;
            s.b = 1 << lg;
            s.lg = lg;
        }
    }
    if (s.lg == 0) s.skip = lbr_skip(N, T - 1.0);
    return s;
}

__host__ __device__ inline size_t lbr_smem_bytes(int n, int num_diss) {
    const size_t N = (size_t)n * n, M = N * (N + 4);
    // four matrices, later b + LBR_GIANTS vectors (stride N + 1); two more
    // matrices; r, o and 3 N of scratch; K and the dissipators
    const size_t vecs = (64 + (size_t)LBR_GIANTS) * (N + 1);
    return ((4 * M > vecs ? 4 * M : vecs) + 2 * M + 5 * N) * 8 +
           (1 + 2 * (size_t)num_diss) * N * 16;
}

// Row and column of basis element e of the Hermitian basis and its kind (0
// diagonal, 1 symmetric, 2 antisymmetric): e = i n + j with the diagonal at i =
// j, symmetric elements above and antisymmetric ones below it.
__device__ __forceinline__ void lbr_basis(int e, int n, int &i, int &j, int &kind) {
    const int r = e / n, c = e - r * n;
    kind = r == c ? 0 : (r < c ? 1 : 2);
    i = r < c ? r : c;
    j = r < c ? c : r;
}

// L_{ij,kl} = K_ik delta_jl + delta_ik conj(K_jl) + sum_d g_d D_ik conj(D_jl).
__device__ __forceinline__ zd lbr_entry(const zd *K, const zd *D, const double *g, int nd, int n,
                                        int i, int j, int k, int l) {
    zd v = mk<double>(0.0, 0.0);
    if (j == l) v = K[i * n + k];
    if (i == k) {
        const zd c = K[j * n + l];
        v.re += c.re;
        v.im -= c.im;
    }
    for (int d = 0; d < nd; ++d) {
        const zd a = cscale(g[d], D[(d * n + i) * n + k]), b = D[(d * n + j) * n + l];
        v.re = fma(a.re, b.re, fma(a.im, b.im, v.re));
        v.im = fma(a.im, b.re, fma(-a.re, b.im, v.im));
    }
    return v;
}

// f x the superoperator in the Hermitian basis into A (row stride ld).
__device__ void lbr_matrix(double *A, const zd *K, const zd *D, const double *g, int nd, int n,
                           int ld, double f) {
    const int N = n * n;
    const double r2 = 1.41421356237309504880, h2 = 0.70710678118654752440;
    for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
        const int a = e / N, b = e - a * N;
        int i, j, ka, k, l, kb;
        lbr_basis(a, n, i, j, ka);
        lbr_basis(b, n, k, l, kb);
        // (L B_b)_ij
        zd v = lbr_entry(K, D, g, nd, n, i, j, k, l);
        if (kb) {
            const zd w = lbr_entry(K, D, g, nd, n, i, j, l, k);
            // symmetric: v + w; antisymmetric: i (v - w)
            v = kb == 1 ? mk<double>(v.re + w.re, v.im + w.im) : mk<double>(w.im - v.im, v.re - w.re);
        }
        // rows: sqrt 2 Re, sqrt 2 Im; columns: 1 / sqrt 2
        const double x = ka == 2 ? v.im : v.re;
        A[a * ld + b] = f * x * (ka ? (kb ? 1.0 : r2) : (kb ? h2 : 1.0));
    }
}

// C = A B, plus c0 I + c1 P1 + c2 P2 + c3 P3 when P1 is given; C aliases none
// of A and B.
__device__ void lbr_gemm(double *C, const double *A, const double *B, int N, int ld,
                         const double *P1 = nullptr, const double *P2 = nullptr,
                         const double *P3 = nullptr, double c0 = 0.0, double c1 = 0.0,
                         double c2 = 0.0, double c3 = 0.0) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int R = (N + 15) >> 4;  // 16-row bands
    double acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.0;
    if (R == 4) {
#pragma unroll 2
        for (int k = 0; k < N; ++k) {
            double a[4], b[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                a[r] = ty + 16 * r < N ? A[(ty + 16 * r) * ld + k] : 0.0;
                b[r] = tx + 16 * r < N ? B[k * ld + tx + 16 * r] : 0.0;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[r][c] = fma(a[r], b[c], acc[r][c]);
        }
    } else {
        for (int k = 0; k < N; ++k) {
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                if (r >= R || ty + 16 * r >= N) continue;
                const double a = A[(ty + 16 * r) * ld + k];
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    if (c < R && tx + 16 * c < N)
                        acc[r][c] = fma(a, B[k * ld + tx + 16 * c], acc[r][c]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = ty + 16 * r, j = tx + 16 * c;
            if (i >= N || j >= N) continue;
            const int o = i * ld + j;
            double v = acc[r][c];
            if (P1) v += fma(c1, P1[o], fma(c2, P2[o], fma(c3, P3[o], i == j ? c0 : 0.0)));
            C[o] = v;
        }
    __syncthreads();
}

// y = E x, four lanes per row.
__device__ void lbr_matvec(double *y, const double *E, const double *x, int N, int ld) {
    const int part = threadIdx.x & 3;
    for (int i = threadIdx.x >> 2; i < ((N + 7) & ~7); i += LBR_THREADS / 4) {
        double s0 = 0.0, s1 = 0.0;
        if (i < N)
            for (int k = part; k < N; k += 8) {
                s0 = fma(E[i * ld + k], x[k], s0);
                if (k + 4 < N) s1 = fma(E[i * ld + k + 4], x[k + 4], s1);
            }
        s0 += s1;
        s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
        s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
        if (i < N && part == 0) y[i] = s0;
    }
    __syncthreads();
}

// y = x^T F: columns across the lanes, four row groups (red: 3 N doubles).
__device__ void lbr_vecmat(double *y, const double *F, const double *x, int N, int ld, double *red) {
    const int j = threadIdx.x & 63, part = threadIdx.x >> 6;
    double s0 = 0.0, s1 = 0.0;
    if (j < N)
        for (int k = part; k < N; k += 8) {
            s0 = fma(F[k * ld + j], x[k], s0);
            if (k + 4 < N) s1 = fma(F[(k + 4) * ld + j], x[k + 4], s1);
        }
    s0 += s1;
    if (part > 0 && j < N) red[(part - 1) * N + j] = s0;
    __syncthreads();
    if (part == 0 && j < N) y[j] = ((s0 + red[j]) + (red[N + j] + red[2 * N + j]));
    __syncthreads();
}

// exp(A 2^-skip) of the matrix A in W[0] (scaled in place); W: six matrices.  Returns
// the one that holds the result; `spare` another, free one.  skip comes back as the
// number of squarings left out.
__device__ double *lbr_expm(double *const *W, int N, int ld, double *red, double **spare, int &skip) {
    const int tid = threadIdx.x;
    double *A = W[0];
    // ||A||_2 <= sqrt(||A||_1 ||A||_inf)
    double c1 = 0.0, ci = 0.0;
    if (tid < N) {
        for (int k = 0; k < N; ++k) {
            c1 += fabs(A[k * ld + tid]);
            ci += fabs(A[tid * ld + k]);
        }
    }
    c1 = lb_block_max(c1, red);
    ci = lb_block_max(ci, red);
    double nrm = sqrt(c1 * ci);
    int sq = 0;
    while (nrm > 0.9 && sq < 64) {
        nrm *= 0.5;
        ++sq;
    }
    const double g = ldexp(1.0, -sq);
    for (int e = tid; e < N * ld; e += LBR_THREADS) A[e] *= g;
    __syncthreads();
    double *A2 = W[1], *A3 = W[2], *A4 = W[3], *X = W[4], *T = W[5];
    lbr_gemm(A2, A, A, N, ld);
    lbr_gemm(A3, A2, A, N, ld);
    lbr_gemm(A4, A2, A2, N, ld);
    // c_k = 1 / k!
    double c[17];
    c[0] = 1.0;
#pragma unroll
    for (int k = 1; k <= 16; ++k) c[k] = c[k - 1] / (double)k;
    for (int e = tid; e < N * N; e += LBR_THREADS) {
        const int i = e / N, j = e - i * N, o = i * ld + j;
        X[o] = fma(c[16], A4[o], fma(c[15], A3[o], fma(c[14], A2[o], fma(c[13], A[o], i == j ? c[12] : 0.0))));
    }
    __syncthreads();
    lbr_gemm(T, A4, X, N, ld, A, A2, A3, c[8], c[9], c[10], c[11]);
    lbr_gemm(X, A4, T, N, ld, A, A2, A3, c[4], c[5], c[6], c[7]);
    lbr_gemm(T, A4, X, N, ld, A, A2, A3, c[0], c[1], c[2], c[3]);
    double *P = T, *Q = X;
    if (skip > sq) skip = sq;
    for (int s = skip; s < sq; ++s) {
        lbr_gemm(Q, P, P, N, ld);
        double *t = P;
        P = Q;
        Q = t;
    }
    *spare = Q;
    return P;
}

__global__ void __launch_bounds__(LBR_THREADS) msp_lindblad_real_kernel(LbArgs a) {
    extern __shared__ __align__(16) unsigned char lbr_smem[];
    __shared__ double red[64];
    __shared__ zd fac[LBR_FAC];
    __shared__ double axes[6], rates[2 * MSP_MAX_SPINS];
    const SnapArgs &sa = a.sa;
    const int n = sa.n, N = n * n, ld = N + 4, tid = threadIdx.x, nt = LBR_THREADS;
    const int s = blockIdx.x, nn = N, nd = 2 * a.num_diss;
    const size_t M = (size_t)N * ld, vs = N + 1, vecs = (64 + LBR_GIANTS) * vs;
    double *const base = reinterpret_cast<double *>(lbr_smem);
    double *const top = base + (4 * M > vecs ? 4 * M : vecs);
    double *const W[6] = {base, base + M, base + 2 * M, base + 3 * M, top, top + M};
    double *r = top + 2 * M, *o = r + N, *tmp = o + N;
    zd *K = reinterpret_cast<zd *>(tmp + 3 * N), *D = K + N;

    const double *b = sa.field + 3 * (size_t)s, *p = sa.pol + 3 * (size_t)s;
    const double Bn = sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
    const double Tk = sa.temperature ? sa.temperature[s] : CUDART_INF;
    build_rho_factors(sa, s, fac);
    if (tid == 32) {
        double x[3] = {1.0, 0.0, 0.0}, y[3] = {0.0, 1.0, 0.0};
        if (Bn != 0.0) {
            const double z[3] = {b[0] / Bn, b[1] / Bn, b[2] / Bn};
            lb_get_xy(z, x, y);
        }
        for (int k = 0; k < 3; ++k) {
            axes[k] = x[k];
            axes[3 + k] = y[k];
        }
    }
    __syncthreads();
    // S+ and S- about the field of each dissipative spin
    for (int d = 0; d < a.num_diss; ++d) {
        const int si = a.diss_spin[d];
        const double rate = a.diss_rate[d];
        double Zu = 0.0;
        if (Tk > 0.0) Zu = exp(-6.62607015e-34 * sa.gammas[si] * Bn * 1e6 / (1.380649e-23 * Tk));
        const double gp = rate * Zu / (CUDART_PI * (1.0 + Zu)), gm = rate / (CUDART_PI * (1.0 + Zu));
        const zd *S = a.spin_ops + (size_t)si * 3 * nn;
        for (int e = tid; e < nn; e += nt) {
            double xr = 0, xi = 0, yr = 0, yi = 0;
            for (int c = 0; c < 3; ++c) {
                const zd sc = S[c * nn + e];
                xr += axes[c] * sc.re;
                xi += axes[c] * sc.im;
                yr += axes[3 + c] * sc.re;
                yi += axes[3 + c] * sc.im;
            }
            D[(2 * d) * nn + e] = mk<double>(xr - yi, xi + yr);
            D[(2 * d + 1) * nn + e] = mk<double>(xr + yi, xi - yr);
        }
        if (tid == 0) {
            rates[2 * d] = gp;
            rates[2 * d + 1] = gm;
        }
    }
    // rho0 and the observable in the Hermitian basis
    const zd *Smu = a.spin_ops + (size_t)sa.mu_index * 3 * nn;
    for (int e = tid; e < N; e += nt) {
        int i, j, kind;
        lbr_basis(e, n, i, j, kind);
        int off = 0, ri = i, rj = j, stride = n;
        zd v = mk<double>(1.0, 0.0);
        for (int q = 0; q < sa.num_spins; ++q) {
            const int dq = sa.dims[q];
            stride /= dq;
            const int di = ri / stride, dj = rj / stride;
            ri -= di * stride;
            rj -= dj * stride;
            v = cmul(v, fac[off + di * dq + dj]);
            off += dq * dq;
        }
        const int q = i * n + j;
        const zd w = mk<double>(
            p[0] * Smu[q].re + p[1] * Smu[nn + q].re + p[2] * Smu[2 * nn + q].re,
            p[0] * Smu[q].im + p[1] * Smu[nn + q].im + p[2] * Smu[2 * nn + q].im);
        const double r2 = kind ? 1.41421356237309504880 : 1.0;
        r[e] = r2 * (kind == 2 ? v.im : v.re);
        o[e] = r2 * (kind == 2 ? w.im : w.re);
    }
    __syncthreads();
    // K = -i H - 1/2 sum_d g_d D^H D
    for (int e = tid; e < nn; e += nt) {
        const zd hs = sa.Hsys[e], z0 = sa.Z[e], z1 = sa.Z[nn + e], z2 = sa.Z[2 * nn + e];
        const double hr = hs.re + b[0] * z0.re + b[1] * z1.re + b[2] * z2.re;
        const double hi = hs.im + b[0] * z0.im + b[1] * z1.im + b[2] * z2.im;
        const int i = e / n, j = e - i * n;
        double kr = hi, ki = -hr;
        for (int d = 0; d < nd; ++d) {
            double mr = 0, mi = 0;
            for (int k = 0; k < n; ++k) {
                const zd x = D[(d * n + k) * n + i], y = D[(d * n + k) * n + j];
                mr += x.re * y.re + x.im * y.im;
                mi += x.re * y.im - x.im * y.re;
            }
            kr -= 0.5 * rates[d] * mr;
            ki -= 0.5 * rates[d] * mi;
        }
        K[e] = mk<double>(kr, ki);
    }
    __syncthreads();
    double *spare;
    if (a.t0 != 0.0) {  // to the first sample
        lbr_matrix(W[0], K, D, rates, nd, n, ld, 2.0 * CUDART_PI * a.t0);
        __syncthreads();
        int skip = lbr_skip(N, 1.0);
        const double *E0 = lbr_expm(W, N, ld, red, &spare, skip);
        double *x = r, *y = tmp;
        for (int k = 0; k < 1 << skip; ++k) {
            lbr_matvec(y, E0, x, N, ld);
            double *t = x;
            x = y;
            y = t;
        }
        if (x != r) {
            for (int e = tid; e < N; e += nt) r[e] = x[e];
            __syncthreads();
        }
    }
    const int Tn = a.num_times;
    LbrShape sh = lbr_shape(N, Tn);
    lbr_matrix(W[0], K, D, rates, nd, n, ld, 2.0 * CUDART_PI * a.dt);
    __syncthreads();
    double *E = lbr_expm(W, N, ld, red, &spare, sh.skip);
    // the result and the spare are W[4] and W[5]: vectors go below them
    double *baby = base, *giant = baby + 64 * vs;
    for (int e = tid; e < N; e += nt) baby[e] = r[e];
    __syncthreads();
    for (int i = 1; i < sh.b; ++i)
        lbr_matvec(baby + i * vs, E, baby + (i - 1) * vs, N, ld);
    for (int q = 0; q < sh.lg; ++q) {
        lbr_gemm(spare, E, E, N, ld);
        double *t = E;
        E = spare;
        spare = t;
    }
    const double weight = sa.wscale[s];
    double *res = a.res + (size_t)s * Tn;
    const int groups = (Tn + sh.b - 1) / sh.b;
    // dst = x^T F (F = E^b; through the baby vectors' place where E is a fraction of a step)
    auto advance = [&](double *dst, const double *x) {
        double *t0 = baby + vs, *t1 = baby + 2 * vs;
        for (int k = (1 << sh.skip) - 1; k > 0; --k) {
            lbr_vecmat(t0, E, x, N, ld, tmp);
            x = t0;
            t0 = t1;
            t1 = const_cast<double *>(x);
        }
        lbr_vecmat(dst, E, x, N, ld, tmp);
    };
    for (int e = tid; e < N; e += nt) giant[e] = o[e];
    __syncthreads();
    for (int g0 = 0; g0 < groups; g0 += LBR_GIANTS) {
        const int cnt = min(LBR_GIANTS, groups - g0);
        if (g0 > 0) {  // continue from the last chunk's final vector
            advance(o, giant + (LBR_GIANTS - 1) * vs);
            for (int e = tid; e < N; e += nt) giant[e] = o[e];
            __syncthreads();
        }
        for (int j = 1; j < cnt; ++j)
            advance(giant + j * vs, giant + (j - 1) * vs);
        for (int e = tid; e < cnt * sh.b; e += nt) {
            const int j = e / sh.b, i = e - j * sh.b;
            const int k = (g0 + j) * sh.b + i;
            if (k >= Tn) continue;
            const double *x = baby + i * vs, *y = giant + j * vs;
            double s0 = 0.0, s1 = 0.0;
            int q = 0;
            for (; q + 1 < N; q += 2) {
                s0 = fma(x[q], y[q], s0);
                s1 = fma(x[q + 1], y[q + 1], s1);
            }
            if (q < N) s0 = fma(x[q], y[q], s0);
            res[k] = (s0 + s1) * weight;
        }
        __syncthreads();
    }
    if (tid == 0 && sa.status) sa.status[s] = MSP_ITEM_OK;
}

// out[slot][t] = sum of the slot's snapshot results, in snapshot order
__global__ void msp_lindblad_reduce_kernel(const double *__restrict__ res,
                                           const int *__restrict__ slot_first, int num_slots,
                                           int T, double *__restrict__ out) {
    const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (e >= (size_t)num_slots * T) return;
    const int sl = (int)(e / T), t = (int)(e - (e / T) * T);
    double acc = 0.0;
    for (int s = slot_first[sl]; s < slot_first[sl + 1]; ++s) acc += res[(size_t)s * T + t];
    out[e] = acc;
}

static int lb_grid(int jobs) {
    int dev = 0, sms = 152;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        sms = 152;
    }
    return jobs < sms ? (jobs > 0 ? jobs : 1) : sms;
}

static int lb_fail(int code, const char *m) { return record_error(code, m); }

static int lb_cuda(cudaError_t e) {
    return e == cudaSuccess ? MSP_OK : record_error(MSP_ERR_CUDA, cudaGetErrorString(e));
}

}  // namespace

extern "C" {

int msp_superop_workspace(int n, int num_ops, size_t *bytes) {
    if (n < 1 || (size_t)n * n > MSP_LB_MAX_N2 || num_ops < 0 || bytes == NULL)
        return lb_fail(MSP_ERR_ARG, "msp_superop_workspace: n outside 1..32 or num_ops < 0");
    *bytes = lb_entries(n, num_ops) * sizeof(zd);
    return MSP_OK;
}

static int superop_common(const double *L, int n, const double *rho0, const double *ops,
                          int num_ops, void *workspace, size_t workspace_bytes) {
    size_t need = 0;
    int rc = msp_superop_workspace(n, num_ops, &need);
    if (rc != MSP_OK) return rc;
    if (L == NULL || rho0 == NULL || (num_ops > 0 && ops == NULL))
        return lb_fail(MSP_ERR_ARG, "msp_superop: a required pointer is NULL");
    if (workspace == NULL || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255))
        return lb_fail(MSP_ERR_WORKSPACE, "msp_superop: workspace too small or not 256-byte aligned");
    return MSP_OK;
}

int msp_superop_evolve(const double *L, int n, const double *rho0, const double *ops, int num_ops,
                       const double *times, int num_times, int uniform, double t0, double dt,
                       double *out, void *workspace, size_t workspace_bytes, void *stream) {
    int rc = superop_common(L, n, rho0, ops, num_ops, workspace, workspace_bytes);
    if (rc != MSP_OK) return rc;
    if (num_times < 0 || out == NULL || (!uniform && num_times > 0 && times == NULL))
        return lb_fail(MSP_ERR_ARG, "msp_superop_evolve: times / out");
    if (num_times == 0) return MSP_OK;
    msp_superop_kernel<<<1, MSP_LB_THREADS, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const zd *>(L), n, reinterpret_cast<const zd *>(rho0),
        reinterpret_cast<const zd *>(ops), num_ops, times, num_times, uniform, t0, dt, 0, 1.0,
        reinterpret_cast<zd *>(out), reinterpret_cast<zd *>(workspace));
    return lb_cuda(cudaGetLastError());
}

int msp_superop_integrate(const double *L, int n, const double *rho0, const double *ops,
                          int num_ops, double tau, double *out, void *workspace,
                          size_t workspace_bytes, void *stream) {
    int rc = superop_common(L, n, rho0, ops, num_ops, workspace, workspace_bytes);
    if (rc != MSP_OK) return rc;
    if (!(tau > 0.0) || num_ops < 1 || out == NULL)
        return lb_fail(MSP_ERR_ARG, "msp_superop_integrate: tau must be > 0, one operator at least");
    msp_superop_kernel<<<1, MSP_LB_THREADS, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const zd *>(L), n, reinterpret_cast<const zd *>(rho0),
        reinterpret_cast<const zd *>(ops), num_ops, nullptr, 0, 1, 0.0, 0.0, 1, tau,
        reinterpret_cast<zd *>(out), reinterpret_cast<zd *>(workspace));
    return lb_cuda(cudaGetLastError());
}

static int check_lindblad(const msp_lindblad_args *a) {
    if (a == NULL) return lb_fail(MSP_ERR_ARG, "msp_lindblad: args is NULL");
    if (a->n < 2 || (size_t)a->n * a->n > MSP_LB_MAX_N2)
        return lb_fail(MSP_ERR_UNSUPPORTED, "msp_lindblad: n outside 2..32");
    if (a->num_spins < 1 || a->num_spins > MSP_MAX_SPINS)
        return lb_fail(MSP_ERR_ARG, "msp_lindblad: num_spins");
    long long prod = 1;
    for (int s = 0; s < a->num_spins; ++s) {
        if (a->dims[s] < 1 || a->dims[s] > MSP_FACTOR_MAXD)
            return lb_fail(MSP_ERR_UNSUPPORTED, "msp_lindblad: a spin multiplicity outside 1..10");
        prod *= a->dims[s];
    }
    if (prod != a->n) return lb_fail(MSP_ERR_ARG, "msp_lindblad: product of dims != n");
    if (a->mu_index < 0 || a->mu_index >= a->num_spins || a->dims[a->mu_index] != 2)
        return lb_fail(MSP_ERR_ARG, "msp_lindblad: mu_index");
    if (a->num_dissipative < 0 || a->num_dissipative > a->num_spins)
        return lb_fail(MSP_ERR_ARG, "msp_lindblad: num_dissipative");
    for (int d = 0; d < a->num_dissipative; ++d)
        if (a->dissipative_spin[d] < 0 || a->dissipative_spin[d] >= a->num_spins)
            return lb_fail(MSP_ERR_ARG, "msp_lindblad: dissipative_spin out of range");
    if (a->num_snap < 0 || a->num_slots < 1) return lb_fail(MSP_ERR_ARG, "msp_lindblad: sizes");
    if (a->mode != MSP_MODE_EVOLVE && a->mode != MSP_MODE_INTEGRAL)
        return lb_fail(MSP_ERR_ARG, "msp_lindblad: mode must be EVOLVE or INTEGRAL");
    if (a->mode == MSP_MODE_INTEGRAL && !(a->tau > 0.0))
        return lb_fail(MSP_ERR_ARG, "msp_lindblad: tau must be > 0");
    if (a->mode == MSP_MODE_EVOLVE && (a->num_times < 1 || (!a->uniform && a->times == NULL)))
        return lb_fail(MSP_ERR_ARG, "msp_lindblad: times");
    if (a->precision != MSP_PREC_FP64 && a->precision != MSP_PREC_MIXED)
        return lb_fail(MSP_ERR_ARG, "msp_lindblad: precision");
    return MSP_OK;
}

struct LbLayout {
    size_t res, slot_first, item_first, scratch, total;
    int T, grid;
    bool real;  // the real form: evolution on a uniform grid, n^2 <= 64
};

static LbLayout lb_layout(const msp_lindblad_args *a) {
    LbLayout L;
    L.T = a->mode == MSP_MODE_INTEGRAL ? 1 : a->num_times;
    L.grid = lb_grid(a->num_snap);
    L.real = a->mode == MSP_MODE_EVOLVE && a->uniform && a->n * a->n <= LBR_MAXN &&
             lbr_smem_bytes(a->n, a->num_dissipative) <= LBR_SMEM_MAX;
    size_t off = 0;
    auto take = [&](size_t b) {
        const size_t o = off;
        off += (b + 255) & ~(size_t)255;
        return o;
    };
    L.res = take((size_t)a->num_snap * L.T * 8);
    L.slot_first = take((size_t)(a->num_slots + 1) * 4);
    L.item_first = take((size_t)(a->num_slots + 1) * 4);
    L.scratch = take(L.real ? 0 : lb_entries(a->n, 1) * sizeof(zd) * L.grid);
    L.total = off;
    return L;
}

int msp_lindblad_workspace(const msp_lindblad_args *a, size_t *bytes) {
    int rc = check_lindblad(a);
    if (rc != MSP_OK) return rc;
    if (bytes == NULL) return lb_fail(MSP_ERR_ARG, "msp_lindblad_workspace: bytes is NULL");
    *bytes = lb_layout(a).total;
    return MSP_OK;
}

int msp_lindblad_run(const msp_lindblad_args *a) {
    int rc = check_lindblad(a);
    if (rc != MSP_OK) return rc;
    if (a->out == NULL) return lb_fail(MSP_ERR_ARG, "msp_lindblad_run: out is NULL");
    if (a->num_snap > 0 && (!a->Hsys || !a->Z || !a->spin_ops || !a->field || !a->pol ||
                            !a->wscale || !a->slot || !a->status))
        return lb_fail(MSP_ERR_ARG, "msp_lindblad_run: a snapshot pointer is NULL");
    const LbLayout Lo = lb_layout(a);
    if (a->workspace == NULL || a->workspace_bytes < Lo.total ||
        (reinterpret_cast<uintptr_t>(a->workspace) & 255))
        return lb_fail(MSP_ERR_WORKSPACE, "msp_lindblad_run: workspace too small or misaligned");
    cudaStream_t st = (cudaStream_t)a->stream;
    char *ws = reinterpret_cast<char *>(a->workspace);
    LbArgs la;
    memset(&la, 0, sizeof(la));
    SnapArgs &sa = la.sa;
    sa.n = a->n;
    sa.num_snap = a->num_snap;
    sa.Hsys = reinterpret_cast<const zd *>(a->Hsys);
    sa.Z = reinterpret_cast<const zd *>(a->Z);
    sa.field = a->field;
    sa.pol = a->pol;
    sa.wscale = a->wscale;
    sa.num_spins = a->num_spins;
    sa.mu_index = a->mu_index;
    for (int s = 0; s < a->num_spins; ++s) {
        sa.dims[s] = a->dims[s];
        sa.gammas[s] = a->gammas[s];
    }
    sa.temperature = a->temperature;
    sa.tau = a->tau;
    sa.status = a->status;
    la.spin_ops = reinterpret_cast<const zd *>(a->spin_ops);
    la.num_diss = a->num_dissipative;
    for (int d = 0; d < a->num_dissipative; ++d) {
        la.diss_spin[d] = a->dissipative_spin[d];
        la.diss_rate[d] = a->dissipative_rate[d];
    }
    la.times = a->times;
    la.num_times = Lo.T;
    la.uniform = a->mode == MSP_MODE_INTEGRAL ? 1 : a->uniform;
    la.t0 = a->t0;
    la.dt = a->dt;
    la.integral = a->mode == MSP_MODE_INTEGRAL;
    la.res = reinterpret_cast<double *>(ws + Lo.res);
    la.scratch = reinterpret_cast<zd *>(ws + Lo.scratch);
    la.scratch_entries = lb_entries(a->n, 1);
    if (a->num_snap > 0 && Lo.real) {
        const size_t smem = lbr_smem_bytes(a->n, a->num_dissipative);
        rc = lb_cuda(cudaFuncSetAttribute(msp_lindblad_real_kernel,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (rc != MSP_OK) return rc;
        msp_lindblad_real_kernel<<<a->num_snap, LBR_THREADS, smem, st>>>(la);
        rc = lb_cuda(cudaGetLastError());
        if (rc != MSP_OK) return rc;
    } else if (a->num_snap > 0) {
        msp_lindblad_kernel<<<Lo.grid, MSP_LB_THREADS, 0, st>>>(la);
        rc = lb_cuda(cudaGetLastError());
        if (rc != MSP_OK) return rc;
    }
    rc = lb_cuda(launch_schedule(a->slot, a->num_snap, a->num_slots, 1, 1, 0,
                                 reinterpret_cast<int *>(ws + Lo.slot_first),
                                 reinterpret_cast<int *>(ws + Lo.item_first), a->status, st));
    if (rc != MSP_OK) return rc;
    const size_t total = (size_t)a->num_slots * Lo.T;
    msp_lindblad_reduce_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
        la.res, reinterpret_cast<const int *>(ws + Lo.slot_first), a->num_slots, Lo.T, a->out);
    return lb_cuda(cudaGetLastError());
}

}  // extern "C"
