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
// its levels in the field v, times their projectors.
static __noinline__ __device__ void thermal_factor(int d, double T, double gamma, const double *v,
                                                   cx<double> *R) {
    const double I = 0.5 * (d - 1);
    double nx, ny, nz;
    const double vn = rho_direction(v, nx, ny, nz);
    for (int e = 0; e < d * d; ++e) R[e] = mk<double>(0.0, 0.0);
    double w[MSP_FACTOR_MAXD];
    const double h = 6.62607015e-34, kB = 1.380649e-23;
    double E[MSP_FACTOR_MAXD];
    for (int k = 0; k < d; ++k) E[k] = (I - k) * vn * 1e6 * gamma;
    double sum = 0.0;
    if (T > 0.0) {
        double xmax = -CUDART_INF;
        for (int k = 0; k < d; ++k) {
            w[k] = -h * E[k] / (kB * T);
            xmax = fmax(xmax, w[k]);
        }
        for (int k = 0; k < d; ++k) {
            w[k] = exp(w[k] - xmax);
            sum += w[k];
        }
    } else {
        double emin = E[0];
        for (int k = 1; k < d; ++k) emin = fmin(emin, E[k]);
        for (int k = 0; k < d; ++k) {
            w[k] = E[k] == emin ? 1.0 : 0.0;
            sum += w[k];
        }
    }
    for (int k = 0; k < d; ++k) w[k] = sum > 0.0 ? w[k] / sum : 1.0 / d;
    // n.S: diagonal n_z m_k, off-diagonal (n_x -/+ i n_y)/2 c_k,
    // c_k = sqrt((k+1)(2I-k)) = <m+1|S+|m>
    cx<double> nS[MSP_FACTOR_MAXD * MSP_FACTOR_MAXD];
    for (int e = 0; e < d * d; ++e) nS[e] = mk<double>(0.0, 0.0);
    for (int k = 0; k < d; ++k) nS[k * d + k] = mk<double>(nz * (I - k), 0.0);
    for (int k = 0; k + 1 < d; ++k) {
        const double c = sqrt((double)(k + 1) * (2.0 * I - k));
        nS[k * d + k + 1] = mk<double>(0.5 * nx * c, -0.5 * ny * c);
        nS[(k + 1) * d + k] = mk<double>(0.5 * nx * c, 0.5 * ny * c);
    }
    cx<double> P[MSP_FACTOR_MAXD * MSP_FACTOR_MAXD], Tm[MSP_FACTOR_MAXD * MSP_FACTOR_MAXD];
    for (int k = 0; k < d; ++k) {
        if (w[k] == 0.0) continue;
        const double mk_ = I - k;
        for (int e = 0; e < d * d; ++e) P[e] = mk<double>((e / d) == (e % d) ? 1.0 : 0.0, 0.0);
        for (int k2 = 0; k2 < d; ++k2) {
            if (k2 == k) continue;
            const double m2 = I - k2, inv = 1.0 / (mk_ - m2);
            // Tm = P (nS - m2) / (mk - m2)
            for (int r = 0; r < d; ++r)
                for (int c = 0; c < d; ++c) {
                    double tr = 0.0, ti = 0.0;
                    for (int l = 0; l < d; ++l) {
                        cx<double> x = nS[l * d + c];
                        if (l == c) x.re -= m2;
                        const cx<double> p = P[r * d + l];
                        tr += p.re * x.re - p.im * x.im;
                        ti += p.re * x.im + p.im * x.re;
                    }
                    Tm[r * d + c] = mk<double>(tr * inv, ti * inv);
                }
            for (int e = 0; e < d * d; ++e) P[e] = Tm[e];
        }
        for (int e = 0; e < d * d; ++e) {
            R[e].re += w[k] * P[e].re;
            R[e].im += w[k] * P[e].im;
        }
    }
    double tr = 0.0;
    for (int k = 0; k < d; ++k) tr += R[k * d + k].re;
    for (int e = 0; e < d * d; ++e) {
        R[e].re /= tr;
        R[e].im /= tr;
    }
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
// One thread per spin; spins up to I = 9/2.  It is a serial chain of FP64
// operations that the whole CTA waits for, so it takes the closed forms where
// there are any: 1/d at T = inf or without a field, and for spin 1/2 (w_0 +
// w_1) / 2 + (w_0 - w_1) n.S.
__device__ __forceinline__ void build_rho_factors(const SnapArgs &a, int s, cx<double> *fac) {
    const int i = threadIdx.x;
    if (i >= a.num_spins) return;
    int off = 0;
    for (int k = 0; k < i; ++k) off += a.dims[k] * a.dims[k];
    const int d = a.dims[i];
    cx<double> *R = fac + off;
    const bool is_mu = i == a.mu_index;
    const double T = a.temperature ? a.temperature[s] : CUDART_INF;
    if (d > MSP_FACTOR_MAXD) {  // rejected on the host
        for (int e = 0; e < d * d; ++e) R[e] = mk<double>(0.0, 0.0);
        return;
    }
    if (!is_mu && (T == CUDART_INF || d == 1)) {
        for (int e = 0; e < d * d; ++e)
            R[e] = mk<double>(e / d == e % d ? 1.0 / (double)d : 0.0, 0.0);
        return;
    }
    const double *v = is_mu ? a.pol + 3 * (size_t)s : a.field + 3 * (size_t)s;
    if (d > 2) {
        thermal_factor(d, T, a.gammas[i], v, R);
        return;
    }
    double nx, ny, nz;
    const double vn = rho_direction(v, nx, ny, nz);
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

}  // namespace msp
