// Phase sum on a uniform time grid as a nonuniform Fourier transform.
//
// Replaces the per-sample loops of the reference's cosine sum
// (muspinsim/cython/parallel.pyx:59-67) and evolve loop
// (muspinsim/hamiltonian.py:95-107) for output rows that many eigenvalue
// pairs feed.  A row is
//   f(k) = sum_p A_p cos(k psi_p) + B_p sin(k psi_p),  k = 0 .. tt - 1,
// psi_p = w_p dt.  Summed sample by sample it costs pairs x samples; here
// every pair is spread once onto a grid of G = n1 n2 >= 4 tt angles (cosine
// terms are even and sine terms odd in the angle, so only the half circle
// 0 .. m = G / 2 is kept), and one transform of the grid gives all samples:
//   b_g = sum_p A_p phi(g - |psi_p| G / 2 pi)   (folded at 0 and m),
//   f(k) = 1 / phi^(k) sum_{g=0}^{m} b_g cos(2 pi g k / G).
// phi is the Kaiser-Bessel window I0(beta sqrt(1 - (2 x / W)^2)) / I0(beta),
// whose Fourier transform phi^ is W sinh(r) / (r I0(beta)), r^2 = beta^2 -
// (pi W k / G)^2.  With G / (2 tt) = 2 and beta = 0.985 (3 pi / 4) W the
// truncation error, relative to sum |A|, is 6e-16 at W = 16 (FP64 rows) and
// 6e-11 at W = 10 (mixed rows).
//
// Kernels of one run:
//   1. tables: the roots of unity, 1 / phi^ and (FP64) the window's table.
//   2. spread: one CTA per (work item, time tile) holds the whole grid in
//      shared memory as 64-bit fixed-point numbers (scaled by the item's
//      sum |A|, so no cell can overflow; integer sums do not depend on the
//      order of the adds, so the result is reproducible bit for bit).  Low
//      and high words are separate arrays: two native 32-bit shared atomics
//      with the carry taken from the first one's return value (a 64-bit
//      shared atomic is a compare-and-swap loop: half the rate).  FP64: a warp
//      loads 32 pairs, one per lane, then takes 16 lanes per pair and each
//      lane evaluates the window at one cell from a table, in 64-bit fixed
//      point off the slow FP64 pipe.  Mixed: a lane keeps its pair and walks the ten
//      cells, the window as ten polynomials of the offset in the kernel's
//      parameters (even and odd parts shared by mirrored cells).
//   3. reduce: items -> row grid in FP64, fixed order; the row's constant.
//   4. two transform steps, G = n1 n2 (g = g1 + n1 g2):
//      F[g1][q] = sum_g2 b e^{2 pi i g2 q / n2}, then
//      f(k) = Re sum_g1 e^{2 pi i g1 k / G} F[g1][k mod n2].
#include <math.h>
#include <string.h>

#include <type_traits>

#include "msp_internal.cuh"

#include <math_constants.h>

namespace msp {

namespace {

constexpr int NU_THREADS = 1024;
constexpr int NU_DEG = 8;  // Taylor coefficients of the window per table entry

// Window width of each precision.  FP64 table: SUB sub-cells per cell, the
// Taylor expansion about each sub-cell's centre (|d| <= 1 / 64), orders 0..3
// in FP64 and 4..7 in FP32 (order 4 is 4e-9 of the window: its FP32 rounding
// is 3e-16).
constexpr int NU_W64 = 16, NU_W32 = 10;
constexpr int NU_SUB = 32, NU_ENTRIES = NU_SUB * NU_W64;
constexpr int NU_TAB_BYTES = NU_ENTRIES * 48;
// Mixed: Taylor expansion about each cell's centre (|d| <= 1 / 2) to order
// 12 (order 13: 3e-9 of the window); cells c and 9 - c mirror each other.
constexpr int NU_HALF = NU_W32 / 2, NU_EVEN = 7, NU_ODD = 6;
struct NuWindow {
    float even[NU_HALF][NU_EVEN], odd[NU_HALF][NU_ODD];
};

// beta of a window of W cells at twofold oversampling.
__host__ __device__ constexpr double nu_beta(int W) { return 0.985 * 2.35619449019234492885 * W; }

size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// I0(x), power series (all terms positive).
double bessel_i0(double x) {
    double t = 1.0, s = 1.0;
    for (int k = 1; k < 200; ++k) {
        t *= (x * x / 4.0) / ((double)k * k);
        s += t;
        if (t < s * 1e-18) break;
    }
    return s;
}

// Taylor coefficient of offset^d of the window of W cells at cell position x,
// times I0(beta): with q(x) = (beta^2 / 4)(1 - (2x/W)^2) the window is
// f(q) / I0(beta), f^(j)(q) = sum_k q^k / (k! (k + j)!), and q is exactly
// quadratic in the offset, q + a d + b d^2.
double window_taylor(int W, double x, int d) {
    const double beta = nu_beta(W), y = 2.0 * x / W;
    const double q = 0.25 * beta * beta * (1.0 - y * y);
    const double a = -2.0 * beta * beta * x / (W * W), b = -beta * beta / (W * W);
    double coef = 0.0;
    for (int j = (d + 1) / 2; j <= d; ++j) {
        double t = 1.0, f = 0.0, v = 1.0;
        for (int k = 2; k <= j; ++k) t /= k;
        const double fact = t;
        for (int k = 1; k < 72; ++k) {
            f += t;
            t *= q / ((double)k * (k + j));
        }
        for (int i = 0; i < 2 * j - d; ++i) v *= a;
        for (int i = 0; i < d - j; ++i) v *= b * (j - i) / (i + 1);
        coef += f * fact * v;
    }
    return coef;
}

// The mixed window's polynomials (a constant of the library).
const NuWindow &mixed_window() {
    static const NuWindow win = [] {
        NuWindow w;
        const double i0 = bessel_i0(nu_beta(NU_W32));
        for (int c = 0; c < NU_HALF; ++c) {
            const double x = c - NU_W32 / 2 + 0.5;
            for (int k = 0; k < NU_EVEN; ++k) w.even[c][k] = (float)(window_taylor(NU_W32, x, 2 * k) / i0);
            for (int k = 0; k < NU_ODD; ++k) w.odd[c][k] = (float)(window_taylor(NU_W32, x, 2 * k + 1) / i0);
        }
        return w;
    }();
    return win;
}

}  // namespace

// ------------------------------------------------------------------ shape

static int nu_smem(const NufftShape &s, bool f64) {
    return (int)(al256((size_t)(s.two ? 2 : 1) * (s.m + 1) * 8) + (f64 ? NU_TAB_BYTES : 0));
}

// Shape of the transform for S snapshots of P pairs in `slots` rows of T
// uniform samples; `two`: sine terms occur (complex coefficients or t0 != 0).
// False when summing the samples directly is cheaper.
bool nufft_shape(long long S, int P, int slots, int T, int precision, bool two, NufftShape *out) {
    const bool f64 = precision != MSP_PREC_MIXED;
    const long long pairs = S * P;
    if (T < 64 || pairs < 1 || slots < 1) return false;
    NufftShape s;
    // time tiles of at most 4096 samples: the half-circle grid (and the sine
    // grid) fit in shared memory
    s.tiles = (T + 4095) / 4096;
    s.tt = (T + s.tiles - 1) / s.tiles;
    s.two = (two || s.tiles > 1) ? 1 : 0;
    s.n2 = 2 * (int)ceil(sqrt((double)s.tt));
    s.n1 = (4 * s.tt + s.n2 - 1) / s.n2;
    s.m = s.n1 * s.n2 / 2;
    const int grids = s.two ? 2 : 1;
    s.cols = grids * (s.m + 1);
    if ((long long)s.tiles * grids > 65535) return false;  // the transform's launch grid
    // Times of both forms in ns, measured on GB300 (152 SMs) with 10,000 x 276
    // pairs x 4096 samples: the direct FP64 sum 44.3 ms (255 pair-samples per
    // ns), the tensor-core mixed sum 0.617 ms (18,300); spreading 0.80 ms
    // (3.4 pairs per ns) in FP64 and 0.077 ms (36) in mixed precision.  The
    // transform's FMAs run at about 400 per ns; the extra launches and their
    // latencies cost 25 us.  One shape's figures: the FP64 spread is the one with a
    // window in FP64 (nu_spread's takes 0.31 ms), and a direct sum's padded tiles and own
    // launches are not counted, so the transform is taken later than it could be.  No
    // call with 1 to 20,000 rows, 1 to 6,000 snapshots and 64 to 4,096 samples was
    // found to take longer than with the direct sum alone.
    const double direct = (double)pairs * T / (f64 ? 255.0 : 18300.0);
    const double dft = (double)slots * s.tiles * grids *
                       (0.5 * s.n1 * s.n2 * s.n2 + 2.0 * s.tt * s.n1) / 400.0;
    const double spread = (double)pairs * s.tiles * (s.two ? 1.4 : 1.0) / (f64 ? 3.4 : 36.0);
    if (spread + dft + 25000.0 > direct) return false;
    // work items: about one wave of CTAs (registers allow one per SM), shared
    // out over the rows
    const long long target = 152 / s.tiles;
    long long per_slot = target / slots;
    if (per_slot < 1) per_slot = 1;
    const long long per_row = (pairs + slots - 1) / slots;
    long long ip = (per_row + per_slot - 1) / per_slot;
    if (ip < 512) ip = 512;
    if (ip > (1LL << 30)) ip = 1LL << 30;
    s.ip = (int)ip;
    s.max_items = phase_max_items((int)S, slots, P, s.ip);
    size_t off = 0;
    s.off_root = off;
    off += al256((size_t)2 * s.m * 16);
    s.off_win = off;
    off += al256((size_t)s.tt * 8);
    s.off_tab = off;
    off += al256(f64 ? NU_TAB_BYTES : 0);
    s.off_partial = off;
    off += al256((size_t)s.max_items * s.tiles * s.cols * 8);
    s.off_rows = off;
    off += al256((size_t)slots * ((size_t)s.tiles * s.cols + 1) * 8);
    s.off_spec = off;
    off += al256((size_t)slots * s.tiles * grids * s.n1 * (s.n2 / 2 + 1) * 16);
    s.bytes = off;
    *out = s;
    return true;
}

namespace {

struct NuArgs {
    int m, n1, n2, tt, tiles, cols, two;
    double per_rad;     // grid cells per radian
    float2 per_rad_dw;  // the same as a double-word
    double win_norm;    // W / I0(beta)
    double inv_i0;      // 1 / I0(beta)
    double2 *root;      // e^{2 pi i j / G}, j < G
    double *win;        // 1 / phi^(k), k < tt
    char *tab;          // FP64 window table
    double *partial;    // items x tiles x cols
    double *rows;       // slots x (tiles x cols + 1)
    double2 *spec;      // slots x tiles x grids x n1 x (n2 / 2 + 1)
    NuWindow mixed;
};

// ------------------------------------------------------------------ 1. tables

// window_taylor at entry e = sub-cell * W + cell of the FP64 table, one lane
// per order d; inv[k] = 1 / k.
__device__ void nu_table_entry(const NuArgs &na, int e, int d, const double *inv) {
    constexpr int W = NU_W64;
    const int s = e / W, c = e - s * W;
    const double beta = nu_beta(W);
    const double x = c - W / 2 + (s + 0.5) / NU_SUB;
    const double y = 2.0 * x / W;
    const double q = 0.25 * beta * beta * (1.0 - y * y);
    const double a = -2.0 * beta * beta * x / (W * W), b = -beta * beta / (W * W);
    // f^(d)(q) / d!; the terms fall below 1e-19 of the sum before k = 54
    double t = 1.0;
    for (int k = 2; k <= d; ++k) t *= inv[k];
    const double fact = t;
    double f = t;
    for (int k = 1; k < 54; ++k) {
        t *= (q * inv[k]) * inv[k + d];
        f += t;
    }
    f *= fact;
    // coefficient of offset^d: sum_j f_j C(j, d - j) a^(2 j - d) b^(d - j)
    double coef = 0.0;
    for (int j = 0; j < NU_DEG; ++j) {
        const double fj = __shfl_sync(0xffffffffu, f, j, NU_DEG);
        if (j <= d && 2 * j >= d) {
            double v = fj;
            for (int i = 0; i < 2 * j - d; ++i) v *= a;
            for (int i = 0; i < d - j; ++i) v *= b * (double)(j - i) * inv[i + 1];
            coef += v;
        }
    }
    coef *= na.inv_i0;
    if (d < 4)
        reinterpret_cast<double *>(na.tab)[(s * 4 + d) * W + c] = coef;
    else
        reinterpret_cast<float *>(na.tab + NU_ENTRIES * 32)[e * 4 + d - 4] = (float)coef;
}

// One warp per CTA: FP64 latency and issue bound, so spread over the SMs.
// The first CTAs (FP64) fill the window table, the others the roots and
// window factors.
__global__ void __launch_bounds__(32) msp_nufft_tables_kernel(NuArgs na, int W, int tab_blocks) {
    const int tid = threadIdx.x;
    if ((int)blockIdx.x < tab_blocks) {
        __shared__ double inv[64];
        for (int k = tid + 1; k < 64; k += 32) inv[k] = 1.0 / (double)k;
        __syncwarp();
        const int t = blockIdx.x * 32 + tid;
        nu_table_entry(na, t / NU_DEG, t % NU_DEG, inv);
        return;
    }
    const int j = (blockIdx.x - tab_blocks) * 32 + tid, G = 2 * na.m;
    if (j < G) {
        double s, c;
        sincospi(2.0 * (double)j / (double)G, &s, &c);
        na.root[j] = make_double2(c, s);
    }
    if (j < na.tt) {
        const double beta = nu_beta(W);
        const double u = 3.14159265358979323846 * W * (double)j / (double)G;
        const double r = sqrt(beta * beta - u * u);
        na.win[j] = 2.0 * r / (na.win_norm * (exp(r) - exp(-r)));
    }
}

// ------------------------------------------------------------------ 2. spread

__device__ __forceinline__ double nu_block_sum(double v, double *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    v = 0.0;
    for (int w = 0; w < NU_THREADS / 32; ++w) v += red[w];
    return v;
}

// cell += q, mod 2^64 in two words.
__device__ __forceinline__ void nu_add(unsigned *lo, unsigned *hi, int cell, long long q) {
    const unsigned x = (unsigned)q;
    const unsigned old = atomicAdd(&lo[cell], x);
    atomicAdd(&hi[cell], (unsigned)(q >> 32) + (old + x < x ? 1u : 0u));
}

// Cell of grid position j folded onto 0 .. m.
__device__ __forceinline__ int nu_fold(int j, int m) { return j < 0 ? -j : (j > m ? 2 * m - j : j); }

// One pair's place on the grid and its two coefficients.
template <typename T>
struct NuPair {
    T A, B, frac;  // frac: first cell's offset from the window's edge, [0, 1)
    int first;
    bool ok;
};

template <bool TWO>
__device__ __forceinline__ NuPair<double> nu_pair64(const PhaseArgs &a, const NuArgs &na, int p,
                                                    double tb) {
    NuPair<double> r;
    const double2 c = reinterpret_cast<const double2 *>(a.pair_coef)[p];
    const double w = a.pair_omega[p];
    const double ph = w * a.dt;
    double psi = reduce_2pi(ph) + fma(w, a.dt, -ph);
    if (!(fabs(psi) <= 3.2)) psi = remainder(ph, 6.283185307179586476925);
    const double s = fabs(psi) * na.per_rad - 0.5 * NU_W64;
    const double f = ceil(s);
    r.frac = f - s;
    r.ok = s >= -NU_W64 && s <= na.m;  // false: a frequency that is not finite
    r.first = r.ok ? (int)f : 0;
    r.A = c.x;
    r.B = 0.0;
    if (TWO) {
        double sn, cs;
        sincos(reduce_2pi(w * tb), &sn, &cs);
        r.A = c.x * cs + c.y * sn;
        r.B = c.y * cs - c.x * sn;
        if (psi < 0.0) r.B = -r.B;
    }
    return r;
}

template <bool TWO>
__device__ __forceinline__ NuPair<float> nu_pair32(const PhaseArgs &a, const NuArgs &na, int p,
                                                   float tile_steps) {
    NuPair<float> r;
    const float2 c = reinterpret_cast<const float2 *>(a.pair_coef)[p];
    float4 rec = a.pair_phase[p];
    if (!(fabsf(rec.x) <= 3.2f)) {
        const float2 q = dw_of(remainder((double)rec.x + (double)rec.y, 6.283185307179586476925));
        rec.x = q.x;
        rec.y = q.y;
    }
    const bool neg = rec.x < 0.f;
    const float px = fabsf(rec.x), py = neg ? -rec.y : rec.y;
    // |psi| per_rad as a double-word, less W / 2
    const float h0 = __fmul_rn(px, na.per_rad_dw.x);
    float l = fmaf(px, na.per_rad_dw.x, -h0);
    l = fmaf(px, na.per_rad_dw.y, fmaf(py, na.per_rad_dw.x, l));
    const float2 h = dw_two_sum(h0, -0.5f * NU_W32);
    l += h.y;
    const float f = ceilf(h.x);
    r.frac = (f - h.x) - l;
    r.ok = h.x >= (float)-NU_W32 && h.x <= (float)na.m;
    r.first = r.ok ? (int)f : 0;
    r.A = c.x;
    r.B = 0.f;
    if (TWO) {
        float th = rec.z, tl = rec.w;
        if (tile_steps > 0.f) {
            const float ph = rec.x * tile_steps;
            float bh = ph, bl = fmaf(rec.x, tile_steps, -ph) + rec.y * tile_steps;
            dw_reduce_2pi(bh, bl);
            dw_add(th, tl, bh, bl);
            dw_reduce_2pi(th, tl);
        }
        float sn, cs;
        sincosf(th, &sn, &cs);
        const float c2 = fmaf(-sn, tl, cs), s2 = fmaf(cs, tl, sn);
        r.A = c.x * c2 + c.y * s2;
        r.B = c.y * c2 - c.x * s2;
        if (neg) r.B = -r.B;
    }
    return r;
}

// x y / 2^64, rounded to nearest: a truncated sum over pairs would be biased.
__device__ __forceinline__ long long nu_mul_rn(long long x, long long y) {
    return __mul64hi(x, y) + (long long)((unsigned long long)x * (unsigned long long)y >> 63);
}

// Spreads pairs pbeg .. pend - 1, FP64: 16 lanes per pair.  Returns whether a
// frequency was not finite.  Window and product in 64-bit fixed point like the
// grid: seven operations per cell on the FP64 pipe (18 clocks each for a warp and
// SM) were the bound, some forty integer instructions take a fifth of that.  The
// offset has 2^-68, the window 2^-62 (its orders 4 .. 7, below 0.05, come in FP32
// as before; the coefficients of orders 0 .. 3 are below 1), the amplitudes 2^-62
// of the item's sum, where FP64 rounded each product to 2^-53.  2.76 M pairs: powder
// of n = 24 (10,000, 4,096 samples) 3.43 -> 2.94 ms in all, and a quarter of the
// error against 64 bits.
template <bool TWO>
__device__ __forceinline__ bool nu_spread(const PhaseArgs &a, const NuArgs &na, double,
                                          int pbeg, int pend, int ex, unsigned *lo, unsigned *hi,
                                          const char *tab) {
    constexpr int W = NU_W64;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = na.m, cells = m + 1;
    const double tb = a.t0 + (double)((long long)blockIdx.y * na.tt) * a.dt;
    const int sub = lane / W, cell = lane - sub * W;
    bool bad = false;
    for (int pb = pbeg + warp * 32; pb < pend; pb += NU_THREADS) {
        const int p = pb + lane;
        long long A = 0, B = 0, delta = 0;  // 2^(ex + 2), 2^68
        int code = 0;  // (first cell + W) << 8 | sub-cell
        if (p < pend) {
            const NuPair<double> r = nu_pair64<TWO>(a, na, p, tb);
            bad |= !r.ok;
            int k = (int)(r.frac * NU_SUB);
            k = k < 0 ? 0 : (k > NU_SUB - 1 ? NU_SUB - 1 : k);
            delta = __double2ll_rn((r.frac - ((double)k + 0.5) * (1.0 / NU_SUB)) * 295147905179352825856.0);
            code = (r.first + W) << 8 | k;
            A = __double2ll_rn(scalbn(r.A, ex + 2));
            if (TWO) B = __double2ll_rn(scalbn(r.B, ex + 2));
        }
        // pairs below the fixed-point resolution add nothing
        unsigned todo = __ballot_sync(0xffffffffu, A != 0 || (TWO && B != 0));
        while (todo) {
            const int b0 = __ffs(todo) - 1;
            todo &= todo - 1;
            const int b1 = todo ? __ffs(todo) - 1 : 32;
            todo &= todo - 1;
            const int src = sub ? b1 : b0, sl = src & 31;
            const int cd = __shfl_sync(0xffffffffu, code, sl);
            const long long dl = __shfl_sync(0xffffffffu, delta, sl);
            const long long Ap = __shfl_sync(0xffffffffu, A, sl);
            long long Bp = 0;
            if (TWO) Bp = __shfl_sync(0xffffffffu, B, sl);
            if (src == 32) continue;
            const int k = cd & 255;
            const long long *ch = reinterpret_cast<const long long *>(tab) + k * 4 * W + cell;
            const float4 cl = reinterpret_cast<const float4 *>(tab + NU_ENTRIES * 32)[k * W + cell];
            const int dh = (int)(dl >> 32);  // 2^36
            const float df = (float)dh * 1.4551915228366852e-11f;
            const float t = fmaf(df, fmaf(df, fmaf(df, cl.w, cl.z), cl.y), cl.x);
            long long v = ch[3 * W] + ((long long)__float2int_rn(t * 17179869184.f) * dh >> 8);
            v = ch[2 * W] + (__mul64hi(v, dl) >> 4);
            v = ch[W] + (__mul64hi(v, dl) >> 4);
            v = ch[0] + (__mul64hi(v, dl) >> 4);
            const int j = (cd >> 8) - W + cell, g = nu_fold(j, m);
            nu_add(lo, hi, g, nu_mul_rn(Ap, v));
            if (TWO) {
                const long long bv = nu_mul_rn(Bp, v);
                nu_add(lo + cells, hi + cells, g, j == g ? bv : -bv);
            }
        }
    }
    return bad;
}

// The same in FP32: one lane per pair.
template <bool TWO>
__device__ __forceinline__ bool nu_spread(const PhaseArgs &a, const NuArgs &na, float,
                                          int pbeg, int pend, int ex, unsigned *lo, unsigned *hi,
                                          const char *) {
    const int m = na.m, cells = m + 1;
    const float tile_steps = (float)((long long)blockIdx.y * na.tt);  // exact: < 2^24
    bool bad = false;
    for (int p = pbeg + threadIdx.x; p < pend; p += NU_THREADS) {
        const NuPair<float> r = nu_pair32<TWO>(a, na, p, tile_steps);
        bad |= !r.ok;
        const float A = scalbnf(r.A, ex), B = TWO ? scalbnf(r.B, ex) : 0.f;
        if (!(fabsf(A) >= 0.5f || (TWO && fabsf(B) >= 0.5f))) continue;
        const float d = r.frac - 0.5f, d2 = d * d;
#pragma unroll
        for (int c = 0; c < NU_HALF; ++c) {
            float e = na.mixed.even[c][NU_EVEN - 1], o = na.mixed.odd[c][NU_ODD - 1];
#pragma unroll
            for (int k = NU_EVEN - 2; k >= 0; --k) e = fmaf(e, d2, na.mixed.even[c][k]);
#pragma unroll
            for (int k = NU_ODD - 2; k >= 0; --k) o = fmaf(o, d2, na.mixed.odd[c][k]);
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const float v = fmaf(side ? -o : o, d, e);
                const int j = r.first + (side ? NU_W32 - 1 - c : c), g = nu_fold(j, m);
                nu_add(lo, hi, g, __float2ll_rn(A * v));
                if (TWO) nu_add(lo + cells, hi + cells, g, __float2ll_rn((j == g ? B : -B) * v));
            }
        }
    }
    return bad;
}

template <bool F64, bool TWO>
__global__ void __launch_bounds__(NU_THREADS, 1) msp_nufft_spread_kernel(PhaseArgs a, NuArgs na) {
    typedef typename std::conditional<F64, double, float>::type T;
    typedef typename PairCoef<T>::type coef_t;
    extern __shared__ __align__(16) unsigned grid[];
    __shared__ double red[NU_THREADS / 32];
    __shared__ int s_range[2];
    const int tid = threadIdx.x, words = (TWO ? 2 : 1) * (na.m + 1);
    unsigned *lo = grid, *hi = grid + words;
    char *tab = reinterpret_cast<char *>(grid) + ((words * 8 + 255) & ~255);

    if (tid == 0) phase_item_range(a, blockIdx.x, &s_range[0], &s_range[1]);
    __syncthreads();
    const int pbeg = s_range[0], pend = s_range[1];
    if (pbeg < 0) return;
    const coef_t *coef = reinterpret_cast<const coef_t *>(a.pair_coef);

    if (F64) {
        // orders 0 .. 3 with 62 bits, then the FP32 ones
        for (int e = tid; e < NU_ENTRIES * 4; e += NU_THREADS)
            reinterpret_cast<long long *>(tab)[e] =
                __double2ll_rn(reinterpret_cast<const double *>(na.tab)[e] * 4611686018427387904.0);
        for (int e = tid; e < NU_ENTRIES; e += NU_THREADS)
            reinterpret_cast<float4 *>(tab + NU_ENTRIES * 32)[e] =
                reinterpret_cast<const float4 *>(na.tab + NU_ENTRIES * 32)[e];
    }
    for (int e = tid; e < 2 * words; e += NU_THREADS) grid[e] = 0u;
    // fixed-point scale: a power of two with sum |A| scale < 2^61
    double sum = 0.0;
    for (int p = pbeg + tid; p < pend; p += NU_THREADS) {
        const coef_t c = coef[p];
        sum += fabs((double)c.x) + (TWO ? fabs((double)c.y) : 0.0);
    }
    sum = nu_block_sum(sum, red);  // its barrier also covers the grid and the table
    double *out = na.partial + ((size_t)blockIdx.x * na.tiles + blockIdx.y) * na.cols;
    bool bad = !(sum <= 1.7976931348623157e308);
    const int ex = sum > 0.0 && !bad ? 60 - ilogb(sum) : 0;
    if (!bad) bad = nu_spread<TWO>(a, na, T(0), pbeg, pend, ex, lo, hi, tab);
    // amplitudes or frequencies that are not finite: neither is the row
    bad = __syncthreads_or(bad);
    const bool normal = ex <= 1000;  // 2^-ex is a normal number
    const double inv = scalbn(1.0, -ex);
    for (int e = tid; e < words; e += NU_THREADS) {
        const long long q = (long long)((unsigned long long)hi[e] << 32 | lo[e]);
        out[e] = bad ? CUDART_NAN : normal ? (double)q * inv : scalbn((double)q, -ex);
    }
}

// ------------------------------------------------------------------ 3. reduce

#define NU_RED_COLS 8
#define NU_RED_STREAMS 64
__global__ void __launch_bounds__(NU_RED_COLS *NU_RED_STREAMS)
    msp_nufft_reduce_kernel(PhaseArgs a, NuArgs na, const double *__restrict__ snap_const) {
    __shared__ double red[NU_RED_STREAMS][NU_RED_COLS + 1];
    const int sl = blockIdx.y, tid = threadIdx.x;
    const int c0 = tid % NU_RED_COLS, stream = tid / NU_RED_COLS;
    const int width = na.tiles * na.cols;
    double v = 0.0;
    if (blockIdx.x == 0) {
        // the row's constant
        const int s0 = a.slot_first[sl], s1 = a.slot_first[sl + 1];
        for (int s = s0 + tid; s < s1; s += blockDim.x) v += snap_const[s];
    } else {
        const int col = (blockIdx.x - 1) * NU_RED_COLS + c0;
        if (col < width) {
            const int i0 = a.item_first[sl], i1 = a.item_first[sl + 1];
            for (int it = i0 + stream; it < i1; it += NU_RED_STREAMS)
                v += na.partial[(size_t)it * width + col];
        }
    }
    red[stream][c0] = v;
    __syncthreads();
    if (stream == 0) {
        double s = 0.0;
        for (int q = 0; q < NU_RED_STREAMS; ++q) s += red[q][c0];
        double *row = na.rows + (size_t)sl * (width + 1);
        if (blockIdx.x == 0) {
#pragma unroll
            for (int o = NU_RED_COLS / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffu, s, o);
            if (tid == 0) row[width] = s;
        } else {
            const int col = (blockIdx.x - 1) * NU_RED_COLS + c0;
            if (col < width) row[col] = s;
        }
    }
}

// ------------------------------------------------------------------ 4. transform

// F[g1][q], q <= n2 / 2 (the grid is real): one CTA per (g1, tile and grid,
// row).
__global__ void __launch_bounds__(128) msp_nufft_dft1_kernel(NuArgs na) {
    extern __shared__ __align__(16) double sm[];
    const int g1 = blockIdx.x, tg = blockIdx.y, tid = threadIdx.x;
    const int grids = na.two ? 2 : 1, n1 = na.n1, n2 = na.n2, h = n2 / 2 + 1;
    double2 *tw = reinterpret_cast<double2 *>(sm);
    double *u = sm + 2 * n2;
    const double *row = na.rows + (size_t)blockIdx.z * ((size_t)na.tiles * na.cols + 1) +
                        (size_t)(tg / grids) * na.cols + (size_t)(tg % grids) * (na.m + 1);
    const int cnt = (na.m - g1) / n1 + 1;
    for (int i = tid; i < n2; i += 128) tw[i] = na.root[(size_t)i * n1];
    for (int i = tid; i < cnt; i += 128) u[i] = row[g1 + n1 * i];
    __syncthreads();
    double2 *F = na.spec + (((size_t)blockIdx.z * gridDim.y + tg) * n1 + g1) * h;
    for (int q = tid; q < h; q += 128) {
        double re[4] = {0, 0, 0, 0}, im[4] = {0, 0, 0, 0};
        int idx = 0, g2 = 0;
        for (; g2 + 3 < cnt; g2 += 4) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const double2 t = tw[idx];
                const double x = u[g2 + r];
                re[r] = fma(x, t.x, re[r]);
                im[r] = fma(x, t.y, im[r]);
                idx += q;
                if (idx >= n2) idx -= n2;
            }
        }
        for (; g2 < cnt; ++g2) {
            const double2 t = tw[idx];
            re[0] = fma(u[g2], t.x, re[0]);
            im[0] = fma(u[g2], t.y, im[0]);
            idx += q;
            if (idx >= n2) idx -= n2;
        }
        F[q] = make_double2((re[0] + re[1]) + (re[2] + re[3]), (im[0] + im[1]) + (im[2] + im[3]));
    }
}

// out[row][k]: 32 samples per CTA, 8 threads per sample (g1 modulo 8).
#define NU_OUT_K 32
#define NU_OUT_PARTS 8
__global__ void __launch_bounds__(NU_OUT_K *NU_OUT_PARTS)
    msp_nufft_dft2_kernel(PhaseArgs a, NuArgs na, double *__restrict__ out) {
    __shared__ double red[NU_OUT_PARTS][NU_OUT_K];
    const int tid = threadIdx.x, kk = tid % NU_OUT_K, part = tid / NU_OUT_K;
    const int tile = blockIdx.y, sl = blockIdx.z, k = blockIdx.x * NU_OUT_K + kk;
    const int grids = na.two ? 2 : 1, n1 = na.n1, n2 = na.n2, h = n2 / 2 + 1, G = 2 * na.m;
    const long long t = (long long)tile * na.tt + k;
    const bool valid = k < na.tt && t < a.num_times;
    double v = 0.0;
    if (valid) {
        const int qf = k % n2;
        const bool mir = qf >= h;
        const int q = mir ? n2 - qf : qf;
        const double sg = mir ? -1.0 : 1.0;
        const double2 *F = na.spec + ((size_t)(sl * na.tiles + tile) * grids) * n1 * h + q;
        const double2 *Fs = F + (size_t)n1 * h;
        long long j = (long long)part * k % G;
        const long long step = (long long)NU_OUT_PARTS * k % G;
        double c = 0.0, s = 0.0;
        for (int g1 = part; g1 < n1; g1 += NU_OUT_PARTS) {
            const double2 e = na.root[j], f = F[(size_t)g1 * h];
            // Re e F for the cosine grid, Im e F for the sine grid
            c = fma(e.x, f.x, fma(-sg * e.y, f.y, c));
            if (grids == 2) {
                const double2 fs = Fs[(size_t)g1 * h];
                s = fma(e.y, fs.x, fma(sg * e.x, fs.y, s));
            }
            j += step;
            if (j >= G) j -= G;
        }
        v = c + s;
    }
    red[part][kk] = v;
    __syncthreads();
    if (part == 0 && valid) {
        double s = 0.0;
#pragma unroll
        for (int p = 0; p < NU_OUT_PARTS; ++p) s += red[p][kk];
        const size_t width = (size_t)na.tiles * na.cols;
        s = fma(s, na.win[k], na.rows[(size_t)sl * (width + 1) + width]);
        const size_t o = (size_t)(a.slot_row ? a.slot_row[sl] : sl) * a.num_times + t;
        if (a.accumulate)
            out[o] += s;
        else
            out[o] = s;
    }
}

template <bool F64, bool TWO>
cudaError_t nu_launch_spread(const PhaseArgs &a, const NuArgs &na, const NufftShape &s,
                             cudaStream_t st) {
    const int smem = nu_smem(s, F64);
    const cudaError_t e = cudaFuncSetAttribute(msp_nufft_spread_kernel<F64, TWO>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    msp_nufft_spread_kernel<F64, TWO>
        <<<dim3(s.max_items, s.tiles), NU_THREADS, smem, st>>>(a, na);
    return cudaGetLastError();
}

NuArgs nu_args(const NufftShape &s, int precision, char *ws) {
    NuArgs na;
    const int W = precision == MSP_PREC_MIXED ? NU_W32 : NU_W64;
    na.m = s.m;
    na.n1 = s.n1;
    na.n2 = s.n2;
    na.tt = s.tt;
    na.tiles = s.tiles;
    na.cols = s.cols;
    na.two = s.two;
    na.per_rad = s.m / 3.14159265358979323846;
    na.per_rad_dw = dw_of(na.per_rad);
    const double i0 = bessel_i0(nu_beta(W));
    na.win_norm = W / i0;
    na.inv_i0 = 1.0 / i0;
    na.root = reinterpret_cast<double2 *>(ws + s.off_root);
    na.win = reinterpret_cast<double *>(ws + s.off_win);
    na.tab = ws + s.off_tab;
    na.partial = reinterpret_cast<double *>(ws + s.off_partial);
    na.rows = reinterpret_cast<double *>(ws + s.off_rows);
    na.spec = reinterpret_cast<double2 *>(ws + s.off_spec);
    na.mixed = mixed_window();
    return na;
}

// ------------------------------------------------------------------ adjoint direction
//
// G(nu) = sum_k g_k e^{2 pi i nu t_k} and H(nu) = sum_k t_k g_k e^{2 pi i nu
// t_k} of a row of samples g on t_k = t0 + k dt at many frequencies: with the
// same window, U_j = sum_k (g_k / phi^(k)) e^{2 pi i j k / G} and
// G(nu) = e^{2 pi i nu t0} sum_j phi(j - s) U_j, s = nu dt G mod G.  U is
// conjugate-symmetric (g real): only j = 0 .. m is kept.

struct __align__(16) NuCell {
    double gr, gi, hr, hi;  // U of g and of t g
};

// F[k1][q] = sum_k2 h_{k1 + n1 k2} e^{2 pi i k2 q / n2}, q <= n2 / 2; one CTA per
// (k1, which of g and t g, row).
__global__ void __launch_bounds__(64) msp_nufft_adj_dft1_kernel(NuArgs na, const double *__restrict__ g,
                                                                int T, double t0, double dt) {
    extern __shared__ __align__(16) double sm[];
    const int k1 = blockIdx.x, which = blockIdx.y, n1 = na.n1, n2 = na.n2, h = n2 / 2 + 1;
    double2 *tw = reinterpret_cast<double2 *>(sm);
    double *u = sm + 2 * n2;
    const double *row = g + (size_t)blockIdx.z * T;
    const int cnt = k1 < T ? (T - 1 - k1) / n1 + 1 : 0;
    for (int i = threadIdx.x; i < n2; i += 64) tw[i] = na.root[(size_t)i * n1];
    for (int i = threadIdx.x; i < cnt; i += 64) {
        const int k = k1 + n1 * i;
        u[i] = row[k] * na.win[k] * (which ? t0 + (double)k * dt : 1.0);
    }
    __syncthreads();
    double2 *F = na.spec + (((size_t)blockIdx.z * 2 + which) * n1 + k1) * h;
    for (int q = threadIdx.x; q < h; q += 64) {
        double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
        int idx = 0;
        for (int i = 0; i < cnt; ++i) {
            const double2 t = tw[idx];
            re[i & 1] = fma(u[i], t.x, re[i & 1]);
            im[i & 1] = fma(u[i], t.y, im[i & 1]);
            idx += q;
            if (idx >= n2) idx -= n2;
        }
        F[q] = make_double2(re[0] + re[1], im[0] + im[1]);
    }
}

// U_j = sum_k1 e^{2 pi i j k1 / G} F[k1][j mod n2], j = 0 .. m, as (G, H) pairs:
// 32 cells per CTA, 4 threads per cell and quantity.
__global__ void __launch_bounds__(256) msp_nufft_adj_dft2_kernel(NuArgs na, NuCell *__restrict__ grid) {
    __shared__ double2 red[8][32];
    const int kk = threadIdx.x & 31, part = (threadIdx.x >> 5) & 3, which = threadIdx.x >> 7;
    const int n1 = na.n1, n2 = na.n2, h = n2 / 2 + 1, G = 2 * na.m;
    const int j = blockIdx.x * 32 + kk;
    double c = 0.0, s = 0.0;
    if (j <= na.m) {
        const int qf = j % n2;
        const bool mir = qf >= h;
        const int q = mir ? n2 - qf : qf;
        const double sg = mir ? -1.0 : 1.0;
        const double2 *F = na.spec + ((size_t)blockIdx.y * 2 + which) * n1 * h + q;
        long long x = (long long)part * j % G;
        const long long step = 4LL * j % G;
        for (int k1 = part; k1 < n1; k1 += 4) {
            const double2 e = na.root[x], f = F[(size_t)k1 * h];
            c = fma(e.x, f.x, fma(-sg * e.y, f.y, c));
            s = fma(e.y, f.x, fma(sg * e.x, f.y, s));
            x += step;
            if (x >= G) x -= G;
        }
    }
    red[which * 4 + part][kk] = make_double2(c, s);
    __syncthreads();
    if (threadIdx.x < 32 && j <= na.m) {
        double2 v[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            v[w] = make_double2(0.0, 0.0);
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                v[w].x += red[w * 4 + p][kk].x;
                v[w].y += red[w * 4 + p][kk].y;
            }
        }
        grid[(size_t)blockIdx.y * (na.m + 1) + j] = NuCell{v[0].x, v[0].y, v[1].x, v[1].y};
    }
}

// One thread per (snapshot, a <= b): G and 2 pi i H at nu = l_b - l_a into the
// full n x n tables (G(-nu) = conj G(nu), H likewise).
__global__ void __launch_bounds__(128) msp_nufft_adj_eval_kernel(
    NuArgs na, const NuCell *__restrict__ grid, const double *__restrict__ evals, int n, int S,
    const int *__restrict__ slot, double t0, double dt, cx<double> *__restrict__ Gh,
    cx<double> *__restrict__ Gd) {
    extern __shared__ __align__(16) char smtab[];
    constexpr int W = NU_W64;
    for (int e = threadIdx.x; e < NU_TAB_BYTES / 16; e += 128)
        reinterpret_cast<uint4 *>(smtab)[e] = reinterpret_cast<const uint4 *>(na.tab)[e];
    __syncthreads();
    const int ntri = n * (n + 1) / 2, m = na.m;
    const long long items = (long long)S * ntri;
    const double twopi = 6.283185307179586476925;
    for (long long it = (long long)blockIdx.x * 128 + threadIdx.x; it < items;
         it += (long long)gridDim.x * 128) {
        const int s = (int)(it / ntri), e = (int)(it - (long long)s * ntri);
        // e -> (b, a), b >= a, e = b (b + 1) / 2 + a
        int b = (int)((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
        while ((b + 1) * (b + 2) / 2 <= e) ++b;
        while (b * (b + 1) / 2 > e) --b;
        const int a = e - b * (b + 1) / 2;
        const double nu = evals[(size_t)s * n + b] - evals[(size_t)s * n + a];
        // cycles per sample, reduced to [-1/2, 1/2]
        const double p = nu * dt;
        double f = (p - rint(p)) + fma(nu, dt, -p);
        const bool neg = f < 0.0;
        f = fabs(f);
        const double x = f * (2.0 * m) - 0.5 * W;
        cx<double> hg = mk<double>(CUDART_NAN, CUDART_NAN), hd = hg;
        if (x >= -W && x <= m) {
            const double first = ceil(x), frac = first - x;
            int k = (int)(frac * NU_SUB);
            k = k < 0 ? 0 : (k > NU_SUB - 1 ? NU_SUB - 1 : k);
            const double dl = frac - ((double)k + 0.5) * (1.0 / NU_SUB);
            const float df = (float)dl;
            const double *hi = reinterpret_cast<const double *>(smtab) + k * 4 * W;
            const float4 *lo = reinterpret_cast<const float4 *>(smtab + NU_ENTRIES * 32) + k * W;
            const NuCell *row = grid + (size_t)slot[s] * (m + 1);
            double gr = 0.0, gi = 0.0, dr = 0.0, di = 0.0;
#pragma unroll 4
            for (int c = 0; c < W; ++c) {
                const float4 t4 = lo[c];
                const float t = fmaf(df, fmaf(df, fmaf(df, t4.w, t4.z), t4.y), t4.x);
                const double v = fma(dl, fma(dl, fma(dl, fma(dl, (double)t, hi[3 * W + c]), hi[2 * W + c]),
                                             hi[W + c]),
                                     hi[c]);
                const int j = (int)first + c, g = nu_fold(j, m);
                const double vi = j == g ? v : -v;  // folded cells hold the conjugate
                const NuCell u = row[g];
                gr = fma(v, u.gr, gr);
                gi = fma(vi, u.gi, gi);
                dr = fma(v, u.hr, dr);
                di = fma(vi, u.hi, di);
            }
            if (neg) {
                gi = -gi;
                di = -di;
            }
            hg = mk<double>(gr, gi);
            hd = mk<double>(dr, di);
            if (t0 != 0.0) {
                double sn, cs;
                const double q = nu * t0;
                sincospi(2.0 * ((q - rint(q)) + fma(nu, t0, -q)), &sn, &cs);
                const cx<double> w = mk<double>(cs, sn);
                hg = cmul(w, hg);
                hd = cmul(w, hd);
            }
        }
        const cx<double> d2 = mk<double>(-twopi * hd.im, twopi * hd.re);
        const size_t base = (size_t)s * n * n;
        Gh[base + (size_t)a * n + b] = hg;
        Gd[base + (size_t)a * n + b] = d2;
        if (a != b) {
            Gh[base + (size_t)b * n + a] = conj(hg);
            Gd[base + (size_t)b * n + a] = mk<double>(-d2.re, d2.im);
        }
    }
}

}  // namespace

cudaError_t launch_nufft_spread(const PhaseArgs &a, const NufftShape &s, int precision, char *ws,
                                cudaStream_t st) {
    const NuArgs na = nu_args(s, precision, ws);
    const bool f64 = precision != MSP_PREC_MIXED;
    const int tabs = f64 ? NU_ENTRIES * NU_DEG / 32 : 0;
    msp_nufft_tables_kernel<<<tabs + (2 * s.m + 31) / 32, 32, 0, st>>>(na, f64 ? NU_W64 : NU_W32,
                                                                      tabs);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (f64)
        return s.two ? nu_launch_spread<true, true>(a, na, s, st)
                     : nu_launch_spread<true, false>(a, na, s, st);
    return s.two ? nu_launch_spread<false, true>(a, na, s, st)
                 : nu_launch_spread<false, false>(a, na, s, st);
}

cudaError_t launch_nufft_rows(const PhaseArgs &a, const NufftShape &s, int precision, char *ws,
                              const double *snap_const, double *out, cudaStream_t st) {
    const NuArgs na = nu_args(s, precision, ws);
    const int grids = s.two ? 2 : 1, width = s.tiles * s.cols;
    const dim3 rg((width + NU_RED_COLS - 1) / NU_RED_COLS + 1, a.num_slots);
    msp_nufft_reduce_kernel<<<rg, NU_RED_COLS * NU_RED_STREAMS, 0, st>>>(a, na, snap_const);
    msp_nufft_dft1_kernel<<<dim3(s.n1, s.tiles * grids, a.num_slots), 128,
                            (size_t)(2 * s.n2 + s.n2 / 2 + 1) * 8, st>>>(na);
    msp_nufft_dft2_kernel<<<dim3((s.tt + NU_OUT_K - 1) / NU_OUT_K, s.tiles, a.num_slots),
                            NU_OUT_K * NU_OUT_PARTS, 0, st>>>(a, na, out);
    return cudaGetLastError();
}

// Shape of the adjoint transform: `points` frequencies against `slots` rows of
// T uniform samples.  False when the direct sums are cheaper: they run 35
// samples per ns (14 FP64 operations each, 72,000 x 1000 in 1.97 ms), the
// transform costs 25 us of launches, 8 T n1 FMAs per row and 140 per frequency.
bool nufft_adjoint_shape(long long points, int slots, int T, NufftShape *out) {
    if (T < 64 || T > (1 << 22) || points < 1 || slots < 1) return false;
    NufftShape s;
    memset(&s, 0, sizeof(s));
    s.tiles = 1;
    s.tt = T;
    s.n2 = 2 * (int)ceil(sqrt((double)T));
    s.n1 = (4 * T + s.n2 - 1) / s.n2;
    s.m = s.n1 * s.n2 / 2;
    const double direct = (double)points * T / 35.0;
    const double dft = (double)slots * (8.0 * s.m * s.n1 + 1.0 * T * s.n2) / 400.0;
    if (25000.0 + dft + (double)points * 140.0 / 400.0 > direct) return false;
    size_t off = 0;
    s.off_root = off;
    off += al256((size_t)2 * s.m * 16);
    s.off_win = off;
    off += al256((size_t)T * 8);
    s.off_tab = off;
    off += al256(NU_TAB_BYTES);
    s.off_spec = off;
    off += al256((size_t)slots * 2 * s.n1 * (s.n2 / 2 + 1) * 16);
    s.off_rows = off;
    off += al256((size_t)slots * (s.m + 1) * 32);
    s.bytes = off;
    *out = s;
    return true;
}

// Fills the adjoint's tables G(l_b - l_a) and G'(l_b - l_a) of every snapshot.
cudaError_t launch_nufft_adjoint(const NufftShape &s, char *ws, const double *evals, int n, int S,
                                 const int *slot, const double *g, int slots, double t0, double dt,
                                 cx<double> *Gh, cx<double> *Gd, cudaStream_t st) {
    const NuArgs na = nu_args(s, MSP_PREC_FP64, ws);
    NuCell *grid = reinterpret_cast<NuCell *>(ws + s.off_rows);
    const int tabs = NU_ENTRIES * NU_DEG / 32;
    msp_nufft_tables_kernel<<<tabs + (2 * s.m + 31) / 32, 32, 0, st>>>(na, NU_W64, tabs);
    const int depth = (s.tt + s.n1 - 1) / s.n1;
    const size_t smem = (size_t)(2 * s.n2 + depth) * 8;
    cudaError_t e = cudaFuncSetAttribute(msp_nufft_adj_dft1_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    for (int r0 = 0; r0 < slots; r0 += 65535) {
        const int rn = slots - r0 < 65535 ? slots - r0 : 65535;
        NuArgs nr = na;
        nr.spec += (size_t)r0 * 2 * s.n1 * (s.n2 / 2 + 1);
        msp_nufft_adj_dft1_kernel<<<dim3(s.n1, 2, rn), 64, smem, st>>>(nr, g + (size_t)r0 * s.tt, s.tt,
                                                                       t0, dt);
        msp_nufft_adj_dft2_kernel<<<dim3((s.m + 32) / 32, rn), 256, 0, st>>>(
            nr, grid + (size_t)r0 * (s.m + 1));
    }
    e = cudaFuncSetAttribute(msp_nufft_adj_eval_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             NU_TAB_BYTES);
    if (e != cudaSuccess) return e;
    const long long items = (long long)S * (n * (n + 1) / 2);
    long long blocks = (items + 127) / 128;
    if (blocks > 152 * 8) blocks = 152 * 8;
    msp_nufft_adj_eval_kernel<<<(int)blocks, 128, NU_TAB_BYTES, st>>>(na, grid, evals, n, S, slot, t0,
                                                                     dt, Gh, Gd);
    return cudaGetLastError();
}

}  // namespace msp
