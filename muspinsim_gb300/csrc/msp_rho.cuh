// Initial density matrix of a configuration snapshot as Kronecker factors,
// shared by the snapshot kernels and the Lindblad kernels.
#pragma once

#include <math_constants.h>

#include "msp_internal.cuh"

namespace msp {

#define MSP_FACTOR_MAXD 10

// Unit vector along v (z when v = 0) and |v|.
__device__ __forceinline__ double rho_direction(const double *v, double &nx, double &ny,
                                                double &nz) {
    const double vn = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    const double inv = vn > 0.0 ? 1.0 / vn : 0.0;
    nx = v[0] * inv;
    ny = v[1] * inv;
    nz = vn > 0.0 ? v[2] * inv : 1.0;
    return vn;
}

// Factor of a spin with d = 2I + 1 > 2 at a finite temperature T: weights of
// its levels in the field v, times their projectors.  By a warp, Q entries per lane:
// the d (d - 1) products with the tridiagonal n.S are a chain of FP64 latencies
// (3,000 snapshots of mu + e + N at 4 K: 501 us in all with a thread per spin, 201).
template <int Q>
static __noinline__ __device__ void thermal_factor(int d, double T, double gamma, const double *v,
                                                   cx<double> *R) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const double I = 0.5 * (d - 1);
    double nx, ny, nz;
    const double vn = rho_direction(v, nx, ny, nz);
    // lane k: the weight of level m = I - k, and 1 / k
    const double h = 6.62607015e-34, kB = 1.380649e-23;
    const double E = (I - lane) * vn * 1e6 * gamma;
    const bool level = lane < d;
    double w, best, sum;
    if (T > 0.0) {
        const double x = -h * E / (kB * T);
        best = level ? x : -CUDART_INF;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) best = fmax(best, __shfl_xor_sync(full, best, o, 16));
        w = level ? exp(x - best) : 0.0;
    } else {
        best = level ? E : CUDART_INF;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) best = fmin(best, __shfl_xor_sync(full, best, o, 16));
        w = level && E == best ? 1.0 : 0.0;
    }
    sum = w;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o, 16);
    w = sum > 0.0 ? w / sum : (level ? 1.0 / d : 0.0);
    const double rcp = 1.0 / (double)(lane > 0 ? lane : 1);
    // n.S: diagonal n_z m_k, off-diagonal (n_x -/+ i n_y)/2 c_k,
    // c_k = sqrt((k+1)(2I-k)) = <m+1|S+|m>; this lane's columns of it
    int col[Q];
    double up[Q], low[Q];
    cx<double> acc[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int e = lane + 32 * q, c = e % d;
        col[q] = e < d * d ? c : -1;
        up[q] = c > 0 ? 0.5 * sqrt((double)c * (2.0 * I - (c - 1))) : 0.0;
        low[q] = c + 1 < d ? 0.5 * sqrt((double)(c + 1) * (2.0 * I - c)) : 0.0;
        acc[q] = mk<double>(0.0, 0.0);
    }
    for (int k = 0; k < d; ++k) {
        const double wk = __shfl_sync(full, w, k);
        if (wk == 0.0) continue;
        __syncwarp();
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (col[q] >= 0) R[lane + 32 * q] = mk<double>((lane + 32 * q) / d == col[q] ? 1.0 : 0.0, 0.0);
        cx<double> P[Q];
        for (int k2 = 0; k2 < d; ++k2) {
            if (k2 == k) continue;
            // P (nS - m2) / (mk - m2), mk - m2 = k2 - k
            const double inv = k2 > k ? __shfl_sync(full, rcp, k2 - k) : -__shfl_sync(full, rcp, k - k2);
            const double m2 = I - k2;
            __syncwarp();
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int e = lane + 32 * q, c = col[q];
                if (c < 0) continue;
                double tr = 0.0, ti = 0.0;
                if (c > 0) {
                    const cx<double> p = R[e - 1], x = mk<double>(nx * up[q], -ny * up[q]);
                    tr = p.re * x.re - p.im * x.im;
                    ti = p.re * x.im + p.im * x.re;
                }
                const cx<double> p = R[e];
                const double dg = nz * (I - c) - m2;
                tr += p.re * dg;
                ti += p.im * dg;
                if (c + 1 < d) {
                    const cx<double> n = R[e + 1], x = mk<double>(nx * low[q], ny * low[q]);
                    tr += n.re * x.re - n.im * x.im;
                    ti += n.re * x.im + n.im * x.re;
                }
                P[q] = mk<double>(tr * inv, ti * inv);
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if (col[q] >= 0) R[lane + 32 * q] = P[q];
        }
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (col[q] >= 0) {
                acc[q].re += wk * P[q].re;
                acc[q].im += wk * P[q].im;
            }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < Q; ++q)
        if (col[q] >= 0) R[lane + 32 * q] = acc[q];
    __syncwarp();
    double tr = 0.0;
    for (int k = 0; k < d; ++k) tr += R[k * d + k].re;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < Q; ++q)
        if (col[q] >= 0) R[lane + 32 * q] = mk<double>(acc[q].re / tr, acc[q].im / tr);
}

// Whether snapshot s starts from rho0 = (1 + n.sigma_mu) / n_dim: no factors
// given and T = inf.  Then rho'_jk = (delta_jk + 2 O'_jk / |p|) / n_dim with O' the
// muon operator in the eigenbasis, and rho0 needs no product of its own.
__device__ __forceinline__ bool rho_is_hot(const SnapArgs &a, int s) {
    return a.rho_fac == nullptr && (a.temperature == nullptr || a.temperature[s] == CUDART_INF);
}

// 2 / (|p| n), or 0 for p = 0 (O' is zero too).
__device__ __forceinline__ double rho_hot_scale(const SnapArgs &a, int s) {
    const double *p = a.pol + 3 * (size_t)s;
    const double pn = sqrt(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
    return pn > 0.0 ? 2.0 / (pn * a.n) : 0.0;
}

// sigma_p = p . sigma = 2 w w^H / |w|^2 |p| - |p| with w its eigenvector of +|p|,
// (|p| + p_z, p_x + i p_y) or, p_z < 0, (p_x - i p_y, |p| - p_z); |w|^2 = 2 |p| (|p| +
// |p_z|).  With V = w^H on the muon digit of U, the d = n / 2 rows of the other
// digits, U^dag (sigma_p (x) 1) U is V^H V / (|p| + |p_z|) - |p| 1, because U is
// unitary to FP64: half the FP64 FMAs of the product with U.
struct MuonAxis {
    double norm, inv;  // |p|, 1 / (|p| + |p_z|) (0 for p = 0, where sigma_p is too)
};

// One thread's work (a square root and a division in FP64).
__device__ __forceinline__ MuonAxis muon_axis(const double *p) {
    MuonAxis x;
    x.norm = sqrt(p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
    x.inv = x.norm == 0.0 ? 0.0 : 1.0 / (x.norm + fabs(p[2]));
    return x;
}

// Kronecker factors of rho0 for snapshot s (muspinsim/experiment.py:170-236):
// the muon in the pure +1/2 state along its polarisation, every other spin
// thermal in its own Zeeman field gamma_i B (uniform at T = inf, ground
// state at T <= 0): sum_k w_k P_k with P_k the spectral projectors of n.S.
// Spins up to I = 9/2, a thread per spin.  It is a serial chain of FP64 operations
// that the whole CTA waits for, so it takes the closed forms where there are any: 1/d
// at T = inf or without a field, and for spin 1/2 (w_0 + w_1) / 2 + (w_0 - w_1) n.S.
// A larger spin at a finite temperature takes a warp of its own.
__device__ __forceinline__ void build_rho_factors(const SnapArgs &a, int s, cx<double> *fac) {
    const double T = a.temperature ? a.temperature[s] : CUDART_INF;
    const double *pol = a.pol + 3 * (size_t)s, *field = a.field + 3 * (size_t)s;
    const int i = threadIdx.x;
    if (i < a.num_spins) {
        int off = 0;
        for (int k = 0; k < i; ++k) off += a.dims[k] * a.dims[k];
        const int d = a.dims[i];
        cx<double> *R = fac + off;
        const bool is_mu = i == a.mu_index;
        if (d > MSP_FACTOR_MAXD) {  // rejected on the host
            for (int e = 0; e < d * d; ++e) R[e] = mk<double>(0.0, 0.0);
        } else if (!is_mu && (T == CUDART_INF || d == 1)) {
            for (int e = 0; e < d * d; ++e)
                R[e] = mk<double>(e / d == e % d ? 1.0 / (double)d : 0.0, 0.0);
        } else if (d <= 2) {
            double nx, ny, nz;
            const double vn = rho_direction(is_mu ? pol : field, nx, ny, nz);
            double dw = 1.0;  // w_0 - w_1
            if (!is_mu) {
                // levels +-E: w_0 / w_1 = exp(-2 x), x = h E / (k T)
                const double E = 0.5 * vn * 1e6 * a.gammas[i];
                if (T > 0.0)
                    dw = tanh(-6.62607015e-34 * E / (1.380649e-23 * T));
                else
                    dw = E < 0.0 ? 1.0 : (E > 0.0 ? -1.0 : 0.0);
            }
            dw *= 0.5;
            R[0] = mk<double>(0.5 + dw * nz, 0.0);
            R[1] = mk<double>(dw * nx, -dw * ny);
            R[2] = mk<double>(dw * nx, dw * ny);
            R[3] = mk<double>(0.5 - dw * nz, 0.0);
        }
    }
    for (int k = threadIdx.x >> 5, off = 0, at = 0; k < a.num_spins; k += blockDim.x >> 5) {
        const int d = a.dims[k];
        if (d <= 2 || d > MSP_FACTOR_MAXD || (k != a.mu_index && T == CUDART_INF)) continue;
        for (; at < k; ++at) off += a.dims[at] * a.dims[at];
        const double *v = k == a.mu_index ? pol : field;
        if (d * d <= 32)
            thermal_factor<1>(d, T, a.gammas[k], v, fac + off);
        else
            thermal_factor<(MSP_FACTOR_MAXD * MSP_FACTOR_MAXD + 31) / 32>(d, T, a.gammas[k], v, fac + off);
    }
}

}  // namespace msp
