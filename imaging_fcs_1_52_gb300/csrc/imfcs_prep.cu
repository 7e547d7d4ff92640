// imfcs_prep.cu -- the passes in front of the correlator:
//   trace_kernel       averaged intensity trace (calcIntensityTrace, java:9822-9855)
//   bleach_*_kernel    polynomial / exponential bleach fits (java:10845-11004)
//   monitor_finalize_kernel  the lags' monitors from the partial sums the
//                      streaming pass (imfcs_stream.cu) wrote (java:9484-9491)
//   block_kernel       lag-1 blocking curve of blockTransform (java:9217-9422),
//                      from the corrected level-0 stream
// The streaming passes split the time axis into segments so that every SM
// has enough loads in flight.
#include <math.h>

#include "imfcs_internal.cuh"
#include "imfcs_ff.cuh"
#include "imfcs_host.h"

namespace imfcs {

// ---------------------------------------------------------------------------
// Averaged trace: out[trace][x] = (int) sum_{ave frames, window} / ave.
// Block (32 traces) x (8 rows); each thread computes 4 points; a shared tile
// transposes the result so both reads and writes are coalesced.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) trace_kernel(Job j, const void *stack, float *trace_out)
{
    __shared__ float tile[32][33];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int trace = blockIdx.x * 32 + tx;
    const int xbase = blockIdx.y * 32;
    int x0 = 0, y0 = 0;
    const bool valid = trace < j.ntrace;
    if (valid) trace_origin(j, trace, x0, y0);
    const int bg = valid ? trace_bg_avg(j, trace) : 0;
    for (int r = 0; r < 4; r++) {
        int xl = ty * 4 + r, x = xbase + xl;
        float val = 0.f;
        if (valid && x < j.nopit) {
            int sum = 0;
            const int fb = x * j.ave, fe = (x + 1) * j.ave;
            for (int f = fb; f < fe; f += 8) {
                float v[8];
                window_values<8>(j, stack, x0, y0, f, fe, bg, v);
#pragma unroll
                for (int u = 0; u < 8; u++) sum += (int)v[u];
            }
            val = (float)(sum / j.ave);
        }
        tile[tx][xl] = val;
    }
    __syncthreads();
    for (int r = 0; r < 4; r++) {
        int tl = ty * 4 + r, tr = blockIdx.x * 32 + tl, x = xbase + tx;
        if (tr < j.ntrace && x < j.nopit) trace_out[(size_t)tr * j.nopit + x] = tile[tl][tx];
    }
}

// The same in two passes where the traces read most of the frames' columns:
// the sums of `ave` frames (and, where the windows' rows do not overlap, of a
// window's rows: ROWS) of every raw pixel of the rows read, once and with wide
// loads, bound by HBM, then the windows of the sums.
struct TraceSums {
    int lines, len, lstride;      // lines of sums (ROWS: one per output row), their length, raw elements between them
    int rows, in_w;               // raw rows added up
};
// sums[x][line][i], VEC raw pixels per thread: 8 (16-byte loads), 2 or 1 by the
// lines' length and alignment.  One pass with a guarded 2-byte load per raw value
// was bound by issue: 0.67 -> 0.28 ms at 128x128x50,000 (read once at 6.8
// TB/s: 0.24), 0.73 -> 0.09 for overlapping 5 x 5 windows at 101x67x12,345.
template <int VEC, bool ROWS>
__global__ void __launch_bounds__(128) trace_sums_kernel(const uint16_t *base, size_t fsz, TraceSums g, int ave,
                                                         unsigned *sums)
{
    const int i = blockIdx.x * 128 + threadIdx.x, per = g.len / VEC;
    if (i >= g.lines * per) return;
    const int line = ROWS ? i / per : 0, x = (i - line * per) * VEC;
    const uint16_t *p = base + (size_t)blockIdx.y * ave * fsz + (size_t)line * g.lstride + x;
    unsigned acc[VEC];
#pragma unroll
    for (int e = 0; e < VEC; e++) acc[e] = 0;
    auto add2 = [](unsigned w, unsigned *a) {         // two 16-bit values, one integer dot product each
        a[0] = __dp2a_lo(w, 0x0001u, a[0]);
        a[1] = __dp2a_lo(w, 0x0100u, a[1]);
    };
    // a window's rows, then the next frame
    const int n = ROWS ? ave * g.rows : ave;
    const size_t back = fsz - (size_t)(g.rows - 1) * g.in_w;
    int row = 0;
    auto next = [&] {
        if (ROWS && ++row < g.rows) {
            p += g.in_w;
        } else {
            p += ROWS ? back : fsz;
            row = 0;
        }
    };
    constexpr int U = VEC == 8 ? 4 : 8;
    // U values (the last time: those left), all loads before their sums
    auto batch = [&](int left) {
        if constexpr (VEC == 8) {
            uint4 v[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = make_uint4(0, 0, 0, 0);
                if (u < left) {
                    v[u] = __ldcs((const uint4 *)p);
                    next();
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                add2(v[u].x, acc);
                add2(v[u].y, acc + 2);
                add2(v[u].z, acc + 4);
                add2(v[u].w, acc + 6);
            }
        } else if constexpr (VEC == 2) {
            unsigned v[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = 0;
                if (u < left) {
                    v[u] = __ldcs((const unsigned *)p);
                    next();
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) add2(v[u], acc);
        } else {
            uint16_t v[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                v[u] = 0;
                if (u < left) {
                    v[u] = __ldcs(p);
                    next();
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) acc[0] += v[u];
        }
    };
    int f = 0;
    for (; f + U <= n; f += U) batch(U);
    if (f < n) batch(n - f);
    unsigned *o = sums + ((size_t)blockIdx.y * g.lines + line) * g.len + x;
#pragma unroll
    for (int e = 0; e < VEC; e++) o[e] = acc[e];
}

// Block (32 traces) x (8 rows), 4 points per thread, transposed through a
// shared tile like trace_kernel.  row0: the first raw row of the sums; they
// are those of points p0 .. p0 + np - 1, nelem to a point.
template <bool ROWS>
__global__ void __launch_bounds__(256) trace_windows_kernel(Job j, const unsigned *sums, int row0, int nelem, int p0,
                                                            int np, float *trace_out)
{
    __shared__ float tile[32][33];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int trace = blockIdx.x * 32 + tx;
    const int xbase = blockIdx.y * 32;
    if (trace < j.ntrace) {
        int x0, y0;
        trace_origin(j, trace, x0, y0);
        // the raw sums may pass 2^31 (bright windows, many frames a point) where
        // the sum above the background does not: modulo 2^32
        const unsigned bg = (unsigned)trace_bg_avg(j, trace) * (unsigned)j.ave;
        const unsigned *w = sums + (size_t)(ROWS ? y0 / j.pixbiny - j.map_y0 : y0 - row0) * j.in_w + x0;
        unsigned acc[4];
#pragma unroll
        for (int r = 0; r < 4; r++) acc[r] = 0;
        for (int k = 0; k < (ROWS ? 1 : j.biny); k++)
            for (int i = 0; i < j.binx; i++)
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int x = min(xbase + ty * 4 + r, np - 1);
                    acc[r] += __ldg(&w[(size_t)x * nelem + k * j.in_w + i]);
                }
#pragma unroll
        for (int r = 0; r < 4; r++) tile[tx][ty * 4 + r] = (float)((int)(acc[r] - bg) / j.ave);
    }
    __syncthreads();
    for (int r = 0; r < 4; r++) {
        const int tl = ty * 4 + r, tr = blockIdx.x * 32 + tl, x = xbase + tx;
        if (tr < j.ntrace && x < np) trace_out[(size_t)tr * j.nopit + p0 + x] = tile[tl][tx];
    }
}

// ---------------------------------------------------------------------------
// Polynomial bleach fit: least squares in the Legendre basis of
// u = t * uscale + uoff (t = averaged-trace time), coefficients = proj * y
// with the FP64 projection matrix proj[(order+1)][nopit] built on the host.
// One warp per trace.  Also writes f0 = f(0), the centre c and flags.  K:
// order + 1, at compile time, so that the coefficients and the basis values stay in
// registers and four points' chains overlap (with run-time counts in local
// memory: 66 us for 441 traces, 190 for 7,938; now 27 and 108, of which FP64
// issue is 87).
// ---------------------------------------------------------------------------

// legendre() with its roundings.
template <int K, int N = 1>
__device__ __forceinline__ void legendre_k(float u, float (&out)[K])
{
    if constexpr (N == 1) {
        out[0] = 1.f;
        out[1] = u;
    }
    if constexpr (N + 1 < K) {
        const float a = (float)(2 * N + 1) * u;
        out[N + 1] = div_small<N + 1>(fmaf(a, out[N], -__fmul_rn((float)N, out[N - 1])));
        legendre_k<K, N + 1>(u, out);
    }
}

template <int K>
__global__ void __launch_bounds__(128) bleach_poly_kernel(Job j, const float *trace, const double *proj, float uscale,
                                                          float uoff, float *bp_out)
{
    const int lane = threadIdx.x & 31;
    const int tr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (tr >= j.ntrace) return;
    const float *y = trace + (size_t)tr * j.nopit;
    double c[K];
#pragma unroll
    for (int i = 0; i < K; i++) c[i] = 0.0;
#pragma unroll 4
    for (int x = lane; x < j.nopit; x += 32) {
        const double yx = f2d(__ldg(&y[x]));
#pragma unroll
        for (int i = 0; i < K; i++) c[i] = fma(__ldg(&proj[(size_t)i * j.nopit + x]), yx, c[i]);
    }
    float cf[K], lb[K];
#pragma unroll
    for (int i = 0; i < K; i++) {
        c[i] = warp_sum_d(c[i]);
        cf[i] = (float)c[i];
    }
    legendre_k<K>(uoff, lb);             // u(0) = uoff
    double f0 = 0.0;
#pragma unroll
    for (int i = 0; i < K; i++) f0 = fma(c[i], (double)lb[i], f0);
    float f0f = (float)f0, inv_f0 = (float)(1.0 / f0);
    // centre: mean of the finite points of the corrected averaged trace (a
    // shift the correlator removes exactly; non-finite points, where the
    // curve crosses zero, are left out so that they cannot spread)
    float csum = 0.f, cnt = 0.f;
#pragma unroll 4
    for (int x = lane; x < j.nopit; x += 32) {
        float t = j.frametime * ((float)x + 0.5f) * (float)j.ave;
        legendre_k<K>(t * uscale + uoff, lb);
        float f = 0.f;
#pragma unroll
        for (int i = 0; i < K; i++) f = fmaf(cf[i], lb[i], f);
        const float v = bleach_correct(__ldg(&y[x]), f, f0f, inv_f0);
        if (isfinite(v)) { csum += v; cnt += 1.f; }
    }
    csum = warp_sum(csum);
    cnt = warp_sum(cnt);
    if (lane == 0) {
        float *bp = bp_out + (size_t)tr * kBleachStride;
#pragma unroll
        for (int i = 0; i < K; i++) bp[i] = cf[i];
        bp[9] = f0f;
        bp[10] = inv_f0;
        bp[11] = (isfinite(f0) && f0 != 0.0) ? 1.f : 0.f;
        bp[12] = cnt > 0.f ? csum / cnt : 0.f;
        bp[13] = uscale;
        bp[14] = uoff;
    }
}

// Centre only (no bleach correction): mean of the averaged trace.
__global__ void center_kernel(Job j, const float *trace, float *bp_out)
{
    const int lane = threadIdx.x & 31;
    const int tr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (tr >= j.ntrace) return;
    const float *y = trace + (size_t)tr * j.nopit;
    float s = 0.f;
    for (int x = lane; x < j.nopit; x += 32) s += __ldg(&y[x]);
    s = warp_sum(s);
    if (lane == 0) {
        float *bp = bp_out + (size_t)tr * kBleachStride;
        bp[11] = 0.f;
        bp[12] = s / j.nopit;
    }
}

// ---------------------------------------------------------------------------
// Exponential bleach fits (SingleExp / DoubleExp, java:13028-13085).
//
// The reference fits A e^{-t/tau} + C (+ A2 e^{-t/tau2}) by Levenberg-
// Marquardt from fixed initial guesses (java:10862-10864, 10917-10921).  The
// same least-squares problem is solved here in the equivalent parameters
//     f0 = f(0),  s_c = A_c / tau_c,  k_c = 1 / tau_c >= 0,
//     f(t) = f0 - sum_c s_c (1 - e^{-k_c t}) / k_c,
// which stay well conditioned when a component is slow (k_c t << 1, where
// the reference's A and C grow without bound while A + C stays finite) and
// are continuous through k_c = 0 (tau = infinity): the fit is the
// least-squares minimum over k_c >= 0 (a rate at its bound whose step points
// below it is held there), whose linear limit stands for the reference's
// A, tau, C stopping in the tau -> infinity valley.
// Scaled variables t / tmax, y / ymax; one warp per trace.
//   start:   single exponential: the global minimum over a grid of rates by
//            variable projection (the oracle scans the same grid); double
//            exponential: the reference's initial guesses;
//   phase 1: FP32 Levenberg-Marquardt until the Gauss-Newton step is below
//            1e-3 sigma + 1e-6 |p| (or no step lowers chi^2);
//   phase 2: Newton with the full Hessian of chi^2/2 (J^T J - sum r d2f; the
//            Gauss-Newton matrix alone does not contract on these
//            large-residual problems), residuals and gradient in float-float
//            (the exponentials by a per-lane recurrence), to the least-squares
//            minimum: until the step is below 1e-9 sigma + 1e-12 |p|.
// ---------------------------------------------------------------------------

// u = (1 - e^{-kt}) / k and du/dk in FP32, x = k t >= 0 (ik = 1/k).
__device__ __forceinline__ void exp_u_f(float k, float ik, float t, float &u, float &dudk)
{
    const float x = k * t;
    if (fabsf(x) < 0.05f) {
        u = slow_exp_term(k, t);
        // du/dk = -t^2 (1/2 - x/3 + x^2/8 - x^3/30 + x^4/144)
        float d = fmaf(x, 1.f / 144.f, -1.f / 30.f);
        d = fmaf(x, d, 1.f / 8.f);
        d = fmaf(x, d, -1.f / 3.f);
        d = fmaf(x, d, 0.5f);
        dudk = -t * t * d;
    } else {
        const float em = (x < 0.7f) ? expm1f(-x) : __expf(-x) - 1.f;
        u = -em * ik;
        dudk = (t * (1.f + em) - u) * ik;
    }
}

// du/dk from an FP32 copy of e = e^{-kt} and u (series for small x).
__device__ __forceinline__ float exp_dudk(float k, float ik, float t, float e, float u)
{
    const float x = k * t;
    if (fabsf(x) < 0.05f) {
        float d = fmaf(x, 1.f / 144.f, -1.f / 30.f);
        d = fmaf(x, d, 1.f / 8.f);
        d = fmaf(x, d, -1.f / 3.f);
        d = fmaf(x, d, 0.5f);
        return -t * t * d;
    }
    return (t * e - u) * ik;
}

// (A + lambda diag(A) + ridge) x = b on the Jacobi-scaled system, FP32;
// parameters in `fix` (bit mask) are held: x_i = 0.
template <int K>
__device__ bool solve_scaled_k(const float *A, const float *b, float lambda, unsigned fix, float *x)
{
    float sc[K], L[K * K];
    for (int i = 0; i < K; i++) sc[i] = ((fix >> i) & 1) ? 0.f : rsqrtf(fmaxf(A[i * K + i], 1e-30f));
    for (int r = 0; r < K; r++)
        for (int c = 0; c < K; c++) L[r * K + c] = A[r * K + c] * sc[r] * sc[c];
    for (int i = 0; i < K; i++) L[i * K + i] = ((fix >> i) & 1) ? 1.f : 1.f + lambda + 1e-6f;
    for (int c = 0; c < K; c++) {
        float d = L[c * K + c];
        for (int m = 0; m < c; m++) d -= L[c * K + m] * L[c * K + m];
        if (!(d > 0.f) || !isfinite(d)) return false;
        d = sqrtf(d);
        L[c * K + c] = d;
        for (int r = c + 1; r < K; r++) {
            float s = L[r * K + c];
            for (int m = 0; m < c; m++) s -= L[r * K + m] * L[c * K + m];
            L[r * K + c] = s / d;
        }
    }
    float yv[K], z[K];
    for (int r = 0; r < K; r++) {
        float s = b[r] * sc[r];
        for (int m = 0; m < r; m++) s -= L[r * K + m] * yv[m];
        yv[r] = s / L[r * K + r];
    }
    for (int r = K - 1; r >= 0; r--) {
        float s = yv[r];
        for (int m = r + 1; m < K; m++) s -= L[m * K + r] * z[m];
        z[r] = s / L[r * K + r];
    }
    for (int r = 0; r < K; r++) x[r] = z[r] * sc[r];
    return true;
}

// d2u/dk2 of u = (1 - e^{-kt}) / k from e = e^{-kt} and u_k (series for
// small |x|, x = kt: t^3 (1/3 - x/4 + x^2/10 - x^3/36 + x^4/168)).
__device__ __forceinline__ float exp_d2udk2(float k, float ik, float t, float e, float uk)
{
    const float x = k * t;
    if (fabsf(x) < 0.05f) {
        float d = fmaf(x, 1.f / 168.f, -1.f / 36.f);
        d = fmaf(x, d, 0.1f);
        d = fmaf(x, d, -0.25f);
        d = fmaf(x, d, 1.f / 3.f);
        return t * t * t * d;
    }
    return (-t * t * e - 2.f * uk) * ik;
}

// One evaluation of the scaled model at p over the trace (warp): residuals in
// float-float (the exponentials by a per-lane recurrence e <- e q seeded in
// FP64), A = the full Hessian of chi^2/2, J^T J - sum_i r_i d2f_i (FP32),
// g = J^T r accumulated in float-float and reduced in FP64.  VALUE: chi^2
// alone.  Returns chi^2 (float-float summed).
template <int K, bool VALUE>
__device__ __noinline__ double exp_normal(const float *y, int n, float dts, float iy, const double *p, float *A,
                                          double *g, int lane)
{
    constexpr int NC = (K - 1) / 2;
    constexpr int NA = K * (K + 1) / 2;
    float acc[NA];
    f2 gp[K];
    for (int i = 0; i < NA; i++) acc[i] = 0.f;
    for (int i = 0; i < K; i++) gp[i] = {0.f, 0.f};
    float pf[K], ik[NC];
    for (int i = 0; i < K; i++) pf[i] = (float)p[i];
    for (int c = 0; c < NC; c++) ik[c] = 1.f / pf[2 + 2 * c];
    f2 e[NC], q[NC], invk[NC], sp[NC];
    bool slow[NC];
    const f2 f0 = f2_from_d(p[0]);
    for (int c = 0; c < NC; c++) {
        const double k = p[2 + 2 * c];
        e[c] = f2_from_d(exp(-k * ((double)lane + 0.5) * (double)dts));
        q[c] = f2_from_d(exp(-k * 32.0 * (double)dts));
        slow[c] = fabs(k * (double)n * (double)dts) < 1e-4;
        invk[c] = f2_from_d(slow[c] ? 0.0 : 1.0 / k);
        sp[c] = f2_from_d(p[1 + 2 * c]);
    }
    f2 c2 = {0.f, 0.f};
    for (int x = lane; x < n; x += 32) {
        const float t = ((float)x + 0.5f) * dts;
        float gr[K];
        float hsk[NC], hkk[NC];   // d2f/(ds dk), d2f/dk2 per component
        gr[0] = 1.f;
        const f2 tf = f2_two_prod((float)x + 0.5f, dts);
        f2 f = f0;
        for (int c = 0; c < NC; c++) {
            f2 u;
            if (slow[c]) {
                // u = t (1 - corr), corr = x/2 - x^2/6 + x^3/24 (|x| < 1e-4)
                const float xx = pf[2 + 2 * c] * t;
                const float corr = xx * (0.5f - xx * (1.f / 6.f - xx * (1.f / 24.f)));
                u = f2_add(tf, f2_neg(f2_two_prod(tf.hi, corr)));
            } else {
                u = f2_mul(f2_add({1.f, 0.f}, f2_neg(e[c])), invk[c]);
            }
            f = f2_add(f, f2_neg(f2_mul(sp[c], u)));
            if (!VALUE) {
                const float uf = u.hi + u.lo, ef = e[c].hi + e[c].lo;
                const float uk = exp_dudk(pf[2 + 2 * c], ik[c], t, ef, uf);
                gr[1 + 2 * c] = -uf;
                gr[2 + 2 * c] = -pf[1 + 2 * c] * uk;
                hsk[c] = -uk;
                hkk[c] = -pf[1 + 2 * c] * exp_d2udk2(pf[2 + 2 * c], ik[c], t, ef, uk);
            }
            e[c] = f2_mul(e[c], q[c]);
        }
        const f2 rr = f2_add(f2_two_prod(__ldg(&y[x]), iy), f2_neg(f));
        c2 = f2_add(c2, f2_mul(rr, rr));
        if (VALUE) continue;
        const float r = rr.hi + rr.lo;
        for (int a = 0; a < K; a++) gp[a] = f2_add(gp[a], f2_two_prod(gr[a], rr.hi));
        for (int a = 0; a < K; a++) gp[a] = f2_add(gp[a], f2_two_prod(gr[a], rr.lo));
        int qa = 0;
        for (int a = 0; a < K; a++)
            for (int b = 0; b <= a; b++) acc[qa++] += gr[a] * gr[b];
        // - r d2f: the only nonzero second derivatives are (s_c, k_c) and (k_c, k_c)
        for (int c = 0; c < NC; c++) {
            const int is = 1 + 2 * c, ikk = 2 + 2 * c;
            acc[ikk * (ikk + 1) / 2 + is] -= r * hsk[c];
            acc[ikk * (ikk + 1) / 2 + ikk] -= r * hkk[c];
        }
    }
    if (!VALUE) {
        int qa = 0;
        for (int a = 0; a < K; a++)
            for (int b = 0; b <= a; b++) {
                float v = warp_sum(acc[qa++]);
                A[a * K + b] = v;
                A[b * K + a] = v;
            }
        for (int a = 0; a < K; a++) g[a] = warp_sum_d((double)gp[a].hi + (double)gp[a].lo);
    }
    return warp_sum_d((double)c2.hi + (double)c2.lo);
}

// FP32 evaluation for phase 1 (no FP64 operation: GB300 issues FP64 at 1/64
// of the FP32 rate): chi^2, A = J^T J, g = J^T r at the FP32 parameters.
template <int K>
__device__ __noinline__ float exp_normal32(const float *y, int n, float dts, float iy, const float *pf, float *A,
                                           float *g, int lane)
{
    constexpr int NC = (K - 1) / 2;
    constexpr int NA = K * (K + 1) / 2;
    float acc[NA], gf[K], ik[NC];
    for (int i = 0; i < NA; i++) acc[i] = 0.f;
    for (int i = 0; i < K; i++) gf[i] = 0.f;
    for (int c = 0; c < NC; c++) ik[c] = 1.f / pf[2 + 2 * c];
    float c2f = 0.f;
    for (int x = lane; x < n; x += 32) {
        const float t = ((float)x + 0.5f) * dts;
        float gr[K];
        gr[0] = 1.f;
        float f = pf[0];
        for (int c = 0; c < NC; c++) {
            float u, du;
            exp_u_f(pf[2 + 2 * c], ik[c], t, u, du);
            f -= pf[1 + 2 * c] * u;
            gr[1 + 2 * c] = -u;
            gr[2 + 2 * c] = -pf[1 + 2 * c] * du;
        }
        const float r = __ldg(&y[x]) * iy - f;
        c2f = fmaf(r, r, c2f);
        int qa = 0;
        for (int a = 0; a < K; a++)
            for (int b = 0; b <= a; b++) acc[qa++] += gr[a] * gr[b];
        for (int a = 0; a < K; a++) gf[a] += gr[a] * r;
    }
    int qa = 0;
    for (int a = 0; a < K; a++)
        for (int b = 0; b <= a; b++) {
            const float v = warp_sum(acc[qa++]);
            A[a * K + b] = v;
            A[b * K + a] = v;
        }
    for (int a = 0; a < K; a++) g[a] = warp_sum(gf[a]);
    return warp_sum(c2f);
}

// solve_scaled_k for phase 1, its first subtractions spelled out (where the
// compiler fuses a scaling product into them depends on the code around the
// call): x = z sc, factors apart.
template <int K>
__device__ __forceinline__ bool exp_solve(const float *A, const float *b, float lambda, unsigned fix, float (&z)[K],
                                          float (&sc)[K])
{
    float L[K * K];
#pragma unroll
    for (int i = 0; i < K; i++) sc[i] = ((fix >> i) & 1) ? 0.f : rsqrtf(fmaxf(A[i * K + i], 1e-30f));
#pragma unroll
    for (int c = 0; c < K; c++) {
        float d = ((fix >> c) & 1) ? 1.f : 1.f + lambda + 1e-6f;
#pragma unroll
        for (int m = 0; m < c; m++) d = fmaf(-L[c * K + m], L[c * K + m], d);
        if (!(d > 0.f) || !isfinite(d)) return false;
        d = sqrtf(d);
        L[c * K + c] = d;
#pragma unroll
        for (int r = c + 1; r < K; r++) {
            const float t = __fmul_rn(A[r * K + c], sc[r]);
            float sum = __fmul_rn(t, sc[c]);
            if (c > 0)
                sum = fmaf(t, sc[c], -__fmul_rn(L[r * K], L[c * K]));
#pragma unroll
            for (int m = 1; m < c; m++) sum = fmaf(-L[r * K + m], L[c * K + m], sum);
            L[r * K + c] = sum / d;
        }
    }
    float yv[K];
#pragma unroll
    for (int r = 0; r < K; r++) {
        float sum = __fmul_rn(b[r], sc[r]);
        if (r > 0) sum = fmaf(b[r], sc[r], -__fmul_rn(L[r * K], yv[0]));
#pragma unroll
        for (int m = 1; m < r; m++) sum = fmaf(-L[r * K + m], yv[m], sum);
        yv[r] = sum / L[r * K + r];
    }
#pragma unroll
    for (int r = K - 1; r >= 0; r--) {
        float sum = yv[r];
#pragma unroll
        for (int m = r + 1; m < K; m++) sum = fmaf(-L[m * K + r], z[m], sum);
        z[r] = sum / L[r * K + r];
    }
    return true;
}

// The undamped (Gauss-)Newton step on A h = g, with a rate at its bound
// k = 0 held there (bit set in `fix`) when its step points below it.  The
// rate form is continuous through k = 0 (tau = infinity), so a trace whose
// minimum over k >= 0 is the linear limit reaches it exactly; the
// reference's A, tau, C cannot cross tau = infinity either and stop in that
// valley, on the k -> 0+ side.
template <int K>
__device__ __forceinline__ bool exp_newton_step(const float *A, const double *gd, const double *p, unsigned &fix,
                                                float *h)
{
    constexpr int NC = (K - 1) / 2;
    float g[K];
    for (int a = 0; a < K; a++) g[a] = (float)gd[a];
    fix = 0;
    bool ok = solve_scaled_k<K>(A, g, 0.f, 0u, h);
    for (int c = 0; c < NC; c++)
        if (p[2 + 2 * c] <= 0.0 && (!ok || h[2 + 2 * c] < 0.f)) fix |= 1u << (2 + 2 * c);
    if (fix) ok = solve_scaled_k<K>(A, g, 0.f, fix, h);
    return ok;
}

// Scaled time per trace point; tmax: the last point's time (s).
__host__ __device__ inline float bleach_dts(const Job &j, float &tmax)
{
    const double dt_pt = (double)j.frametime * (double)j.ave;
    tmax = (float)(dt_pt * ((double)j.nopit - 0.5));
    return (float)(dt_pt / (double)tmax);
}

// Start of the single-exponential fit: global search by variable projection.
// For each rate of the grid x = k tmax in {0} and 96 log-spaced values 1e-3 ..
// 1e4 (the oracle's grid), c0 + c1 e^{-kt} (k = 0: c0 + c1 t) is linear in c0,
// c1 and chi^2 is minimised over them exactly; the best rate starts the LM.
//
// The centred basis b = e^{-kt} - mean and its square sum are the same for
// every trace: bleach_grid_table_kernel lays them out once per plan, and what is
// left per trace are 97 dot products of 1000 points.  A CTA takes T traces; a
// warp takes eight rates at a time, a lane its points lane, lane + 32, ... in
// that order (sums as one rate of one trace at a time gives them), so a loaded
// basis value serves T traces and a loaded sample eight rates.  Bound by FP32
// issue and the loads of the table (430 KB, in L2): 16,384 traces in 0.15 ms,
// against 0.7 ms of the fit kernel when each trace's warp made its own basis.
constexpr int kGridRates = 97, kGridPad = 104, kGridPts = 1024;

// Position of point x in the table: a lane's four successive points adjoin.
__device__ __forceinline__ int grid_pos(int x) { return ((x >> 7) * 32 + (x & 31)) * 4 + ((x >> 5) & 3); }

// tab: [rate][1024] centred basis (0 past the trace), then [3][kGridPad]: mean, square sum, rate.
__global__ void __launch_bounds__(32) bleach_grid_table_kernel(int n, float dts, float *tab)
{
    const int lane = threadIdx.x, jg = blockIdx.x;
    float *row = tab + (size_t)jg * kGridPts, *stat = tab + (size_t)kGridPad * kGridPts + jg;
    const float kx = (jg == 0 || jg >= kGridRates) ? 0.f : exp10f(-3.f + 7.f * (float)(jg - 1) / 95.f);
    const float q = __expf(-kx * 32.f * dts), e0 = __expf(-kx * ((float)lane + 0.5f) * dts);
    float se = 0.f, e = e0;
    for (int x = lane; x < n; x += 32) {
        const float tt = ((float)x + 0.5f) * dts;
        se += jg == 0 ? tt : e;
        e *= q;
    }
    const float me = warp_sum(se) / (float)n;
    float see = 0.f;
    e = e0;
    for (int x = lane; x < kGridPts; x += 32) {
        const float tt = ((float)x + 0.5f) * dts;
        const float b = x < n ? (jg == 0 ? tt : e) - me : 0.f;
        see = fmaf(b, b, see);
        row[grid_pos(x)] = b;
        e *= q;
    }
    const float sE = warp_sum(see);
    if (lane == 0) {
        stat[0] = me;
        stat[kGridPad] = sE;
        stat[2 * kGridPad] = kx;
    }
}

template <int T>
__global__ void __launch_bounds__(128) bleach_grid_kernel(Job j, const float *trace, const float *tab, float *bp_out)
{
    constexpr int RB = 8;                         // rates of a warp's pass
    constexpr int NS = T * RB, NW = NS > 32 ? 32 : NS;
    __shared__ float4 yc[T][kGridPts / 4];        // centred samples, table order
    __shared__ float sy[T][kGridPad];             // dot products
    __shared__ float my[T], syy[T];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int tr0 = blockIdx.x * T, n = j.nopit;
    for (int m = wid; m < T; m += 4) {
        float *out = reinterpret_cast<float *>(yc[m]);
        const int tr = tr0 + m;
        if (tr >= j.ntrace) {
            for (int x = lane; x < kGridPts; x += 32) out[x] = 0.f;
            continue;
        }
        const float *y = trace + (size_t)tr * n;
        float ym = 0.f;
        for (int x = lane; x < n; x += 32) ym = fmaxf(ym, fabsf(__ldg(&y[x])));
        for (int o = 16; o > 0; o >>= 1) ym = fmaxf(ym, __shfl_xor_sync(0xffffffffu, ym, o));
        if (ym == 0.f) ym = 1.f;
        const float iy = 1.f / ym;
        float s = 0.f;
        for (int x = lane; x < n; x += 32) s += __ldg(&y[x]) * iy;
        const float mean = warp_sum(s) / (float)n;
        float s2 = 0.f;
        for (int x = lane; x < kGridPts; x += 32) {
            const float v = x < n ? __ldg(&y[x]) * iy - mean : 0.f;
            s2 = fmaf(v, v, s2);
            out[grid_pos(x)] = v;
        }
        s2 = warp_sum(s2);
        if (lane == 0) { my[m] = mean; syy[m] = s2; }
    }
    __syncthreads();
    const float4 *tab4 = reinterpret_cast<const float4 *>(tab);
    for (int jb = wid * RB; jb < kGridPad; jb += 4 * RB) {
        float acc[NS];
#pragma unroll
        for (int i = 0; i < NS; i++) acc[i] = 0.f;
#pragma unroll 1
        for (int i = lane; i < kGridPts / 4; i += 32) {
            float4 b[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) b[r] = __ldg(&tab4[(size_t)(jb + r) * (kGridPts / 4) + i]);
#pragma unroll
            for (int m = 0; m < T; m++) {
                const float4 v = yc[m][i];
#pragma unroll
                for (int r = 0; r < RB; r++) {
                    float a = acc[m * RB + r];
                    a = fmaf(v.x, b[r].x, a);
                    a = fmaf(v.y, b[r].y, a);
                    a = fmaf(v.z, b[r].z, a);
                    acc[m * RB + r] = fmaf(v.w, b[r].w, a);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < NS; h += NW) {
            float part[NW];
#pragma unroll
            for (int i = 0; i < NW; i++) part[i] = acc[h + i];
            int pos;
            const float v = warp_sums<NW, 16>(part, lane, pos);
            if (pos >= 0) sy[(h + pos) / RB][jb + (h + pos) % RB] = v;
        }
    }
    __syncthreads();
    const float *stat = tab + (size_t)kGridPad * kGridPts;
    for (int m = wid; m < T; m += 4) {
        if (tr0 + m >= j.ntrace) break;
        // the first rate of least chi^2 (below 3.4e38)
        float bc = 3.4e38f, b1 = 0.f;
        int bj = kGridPad;
        for (int jg = lane; jg < kGridRates; jg += 32) {
            const float sE = __ldg(&stat[kGridPad + jg]), sY = sy[m][jg];
            const float c1 = sE > 0.f ? sY / sE : 0.f;
            const float c2 = syy[m] - c1 * sY;
            if (c2 < bc) { bc = c2; b1 = c1; bj = jg; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float oc = __shfl_xor_sync(0xffffffffu, bc, o), o1 = __shfl_xor_sync(0xffffffffu, b1, o);
            const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
            if (oc < bc || (oc == bc && oj < bj)) { bc = oc; b1 = o1; bj = oj; }
        }
        if (lane == 0) {
            float *bp = bp_out + (size_t)(tr0 + m) * kBleachStride;
            const bool any = bj < kGridPad;
            bp[0] = any ? my[m] - b1 * __ldg(&stat[bj]) : 0.f;
            bp[1] = b1;
            bp[2] = any ? __ldg(&stat[2 * kGridPad + bj]) : 0.f;
        }
    }
}

template <int K>
__global__ void __launch_bounds__(128, 4) bleach_exp_kernel(Job j, const float *trace, float *bp_out)
{
    constexpr int NC = (K - 1) / 2;
    const int lane = threadIdx.x & 31;
    const int tr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (tr >= j.ntrace) return;
    const int n = j.nopit;
    const float *y = trace + (size_t)tr * n;
    const double dt_pt = (double)j.frametime * (double)j.ave;      // time per trace point (s)
    float tmax;
    const float dts = bleach_dts(j, tmax);
    float ym = 0.f;
    for (int x = lane; x < n; x += 32) ym = fmaxf(ym, fabsf(__ldg(&y[x])));
    for (int o = 16; o > 0; o >>= 1) ym = fmaxf(ym, __shfl_xor_sync(0xffffffffu, ym, o));
    if (ym == 0.f) ym = 1.f;
    const float iy = 1.f / ym;
    double p[K];
    if constexpr (K == 3) {
        // bleach_grid_kernel's start: c0 + c1 e^{-kt} (k = 0: c0 + c1 t)
        const float *st = bp_out + (size_t)tr * kBleachStride;
        const float b0 = st[0], b1 = st[1], bk = st[2];
        if (bk == 0.f) { p[0] = b0; p[1] = -b1; p[2] = 0.0; }                  // f = c0 + c1 t
        else { p[0] = (double)b0 + b1; p[1] = (double)b1 * bk; p[2] = bk; }       // f = c0 + c1 e^{-kt}
    } else {
        // reference initial guesses (java:10917-10921) in f0, s, k
        const double y1 = (double)__ldg(&y[1]) * (double)iy;
        const double thalf = ((double)(n / 2) + 0.5) * (double)dts;
        {
            const double t10 = ((double)(n / 10) + 0.5) * (double)dts;
            p[0] = y1; p[1] = 0.5 * y1 / t10; p[2] = 1.0 / t10; p[3] = 0.5 * y1 / thalf; p[4] = 1.0 / thalf;
        }
    }
    // Phase 1: FP32 Levenberg-Marquardt (FP32 parameters, no FP64 operation)
    // until the Gauss-Newton step is below 1e-3 sigma + 1e-6 |p| (or, with
    // that step within 0.05 sigma, two steps in a row fail to lower chi^2,
    // or no step lowers it up to lambda 1e10): inside the region where the Newton
    // phase converges quadratically; FP32 sums over 1000 points cannot
    // resolve much smaller steps anyway.
    float A[K * K], lambda = 1e-3f;
    double g[K];
    float pf[K], gf[K];
    for (int a = 0; a < K; a++) pf[a] = (float)p[a];
    float chi2f = exp_normal32<K>(y, n, dts, iy, pf, A, gf, lane);
    const bool ok = isfinite(chi2f);
    int evals = 1, rejected = 0;
    for (int it_n = 0; ok && it_n < 100; it_n++) {
        // the undamped step of the stopping test in the warp's lower half and
        // the damped one in the upper: a solve is one long chain (2,304
        // double-exponential traces 1.73 -> 1.53 ms, 16,384 single 0.95 ->
        // 0.89).  A rate at its bound whose undamped step points below it is
        // held (second pass).
        float hz[K], sc[K];
        unsigned fix = 0, votes;
#pragma unroll 1
        for (;;) {
            votes = __ballot_sync(0xffffffffu, exp_solve<K>(A, gf, lane < 16 ? 0.f : lambda, fix, hz, sc));
            if (fix) break;
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const float hk = __shfl_sync(0xffffffffu, __fmul_rn(hz[2 + 2 * c], sc[2 + 2 * c]), 0);
                if (pf[2 + 2 * c] <= 0.f && (!(votes & 1) || hk < 0.f)) fix |= 1u << (2 + 2 * c);
            }
            if (!fix) break;
        }
        bool gn_near = false;      // Gauss-Newton step within 0.05 sigma
        if (votes & 1) {
            bool conv = true;
            gn_near = true;
#pragma unroll
            for (int a = 0; a < K; a++) {
                const float ha = __shfl_sync(0xffffffffu, __fmul_rn(hz[a], sc[a]), 0);
                if ((fix >> a) & 1) continue;
                const float sig = rsqrtf(fmaxf(A[a * K + a], 1e-30f));
                conv = conv && fabsf(ha) <= 1e-6f * fabsf(pf[a]) + 1e-3f * sig;
                gn_near = gn_near && fabsf(ha) <= 0.05f * sig;
            }
            if (conv) break;
        }
        if (!(votes >> 16 & 1)) {
            lambda *= 10.f;
            if (lambda > 1e10f) break;
            continue;
        }
        float pn[K];
#pragma unroll
        for (int a = 0; a < K; a++) {
            const float z = __shfl_sync(0xffffffffu, hz[a], 16);
            pn[a] = __fadd_rn(pf[a], __fmul_rn(z, sc[a]));
        }
        for (int c = 0; c < NC; c++) pn[2 + 2 * c] = fmaxf(pn[2 + 2 * c], 0.f);
        float An[K * K], gn[K];
        const float c2n = exp_normal32<K>(y, n, dts, iy, pn, An, gn, lane);
        evals++;
        if (isfinite(c2n) && c2n < chi2f) {
            for (int a = 0; a < K; a++) { pf[a] = pn[a]; gf[a] = gn[a]; }
            for (int a = 0; a < K * K; a++) A[a] = An[a];
            chi2f = c2n;
            lambda = fmaxf(lambda * 0.1f, 1e-12f);
            rejected = 0;
        } else {
            // two rejected steps in a row while the Gauss-Newton step is
            // within 0.05 sigma: FP32 chi^2 no longer resolves the descent
            // this close to the minimum -- the Newton phase takes over
            // (elsewhere rejections raise the damping as usual)
            rejected = gn_near ? rejected + 1 : 0;
            lambda *= 10.f;
            if (lambda > 1e10f || rejected >= 2) break;
        }
    }
    for (int a = 0; a < K; a++) p[a] = (double)pf[a];
    double chi2 = chi2f;
    // Phase 2: Newton with the full Hessian, float-float residuals and
    // gradient, to the least-squares minimum: until the step is below
    // 1e-9 sigma + 1e-12 |p|, while chi^2 does not increase.
    if (ok) {
        chi2 = exp_normal<K, false>(y, n, dts, iy, p, A, g, lane);
        evals++;
        for (int it_n = 0; it_n < 20 && isfinite(chi2); it_n++) {
            float h[K];
            unsigned fix;
            if (!exp_newton_step<K>(A, g, p, fix, h)) break;   // Hessian not positive definite
            bool conv = true;
            for (int a = 0; a < K; a++) {
                if ((fix >> a) & 1) continue;
                const float sig = rsqrtf(fmaxf(A[a * K + a], 1e-30f));
                conv = conv && fabsf(h[a]) <= 1e-12f * (float)fabs(p[a]) + 1e-9f * sig;
            }
            double pn[K];
            for (int a = 0; a < K; a++) pn[a] = p[a] + (double)h[a];
            for (int c = 0; c < NC; c++) pn[2 + 2 * c] = fmax(pn[2 + 2 * c], 0.0);
            float An[K * K];
            double gn[K];
            // the last step only has to show that chi^2 does not rise
            const double c2n = conv ? exp_normal<K, true>(y, n, dts, iy, pn, An, gn, lane)
                                    : exp_normal<K, false>(y, n, dts, iy, pn, An, gn, lane);
            evals++;
            if (!(isfinite(c2n) && c2n <= chi2)) break;
            for (int a = 0; a < K; a++) p[a] = pn[a];
            if (conv) break;
            for (int a = 0; a < K; a++) g[a] = gn[a];
            for (int a = 0; a < K * K; a++) A[a] = An[a];
            chi2 = c2n;
        }
    }
    // back to data units: y = y_s / iy, t = t_s tmax
    const double st = (double)dts / dt_pt;            // 1 / tmax
    const double f0d = p[0] / (double)iy;
    double sd[NC], kd[NC];
    bool valid = ok && isfinite(f0d);
    for (int c = 0; c < NC; c++) {
        sd[c] = p[1 + 2 * c] * st / (double)iy;
        kd[c] = p[2 + 2 * c] * st;
        valid = valid && isfinite(sd[c]) && isfinite(kd[c]) && sd[c] != 0.0;  // java:9689, 9714
    }
    // curve evaluation form per component (exp form unless slow over the run)
    const double t_end = (double)j.frametime * ((double)j.num + 2.0);
    float bpl[kBleachStride];
    for (int a = 0; a < kBleachStride; a++) bpl[a] = 0.f;
    double cconst = f0d, csum_amp = 0.0;
    int flags = 0;
    for (int c = 0; c < NC; c++) {
        const double amp = sd[c] / kd[c];               // A_c (inf when k_c = 0)
        bpl[5 + c] = (float)kd[c];
        if (fabs(kd[c]) * t_end <= 0.5) {
            flags |= 1 << c;
            bpl[7 + c] = (float)sd[c];
        } else {
            bpl[7 + c] = (float)amp;
            cconst -= amp;
        }
        csum_amp += amp;
        // reference form: A_c, tau_c
        bpl[2 * c] = (float)amp;
        bpl[2 * c + 1] = (float)(1.0 / kd[c]);
    }
    bpl[2 * NC] = (float)(f0d - csum_amp);               // C
    bpl[13] = (float)cconst;
    bpl[14] = (float)flags;
    const float f0 = (float)f0d, inv_f0 = (float)(1.0 / f0d);
    float csum = 0.f, cnt = 0.f;     // centre over the finite corrected points
    for (int x = lane; x < n; x += 32) {
        float yx = __ldg(&y[x]);
        if (valid) {
            float t = j.frametime * ((float)x + 0.5f) * (float)j.ave;
            yx = bleach_correct(yx, bleach_f(bpl, j.bleach, 0, t, nullptr), f0, inv_f0);
        }
        if (isfinite(yx)) { csum += yx; cnt += 1.f; }
    }
    csum = warp_sum(csum);
    cnt = warp_sum(cnt);
    if (lane == 0) {
        float *bp = bp_out + (size_t)tr * kBleachStride;
        for (int a = 0; a < kBleachStride; a++) bp[a] = bpl[a];
        bp[9] = f0;
        bp[10] = inv_f0;
        bp[11] = valid ? 1.f : 0.f;
        bp[12] = cnt > 0.f ? csum / cnt : 0.f;
        bp[15] = (float)evals;      // model evaluations (diagnostic)
    }
}

// Finalise monitors: one warp per output pixel.  Exclusive scan of the
// segment totals (FP64), snapshot prefixes, then for every lag
//   a = sum(direct window)/n - 2^k c0,  b = sum(delayed window)/n - 2^k c1,
// dm = a + 2^k c0, Dm = b + 2^k c1  (java:9484-9491), plus the lag-1 monitors
// of the zero-led sequence blockTransform reads (java:9259-9272).
//
// Non-finite corrected frames entered the sums as 0 and are counted; a
// window that contains one gives a NaN monitor, so exactly the lags whose
// windows hold a bad frame become non-finite, as calculateCF's sums do
// (java:9484-9491).
// Bound by FP64 issue (1/64 of the FP32 rate): conversions on the integer
// pipe, the divisions by the product counts from their reciprocals in the lag
// table, the counts of non-finite frames as integers (0.31 -> 0.13 ms at
// 16,384 pixels x 50,000 frames).
__global__ void __launch_bounds__(128) monitor_finalize_kernel(Job j, const LagInfo *li, const float *bparams,
                                        int nseg, const float2 *segtot, const float2 *snap_part,
                                        const int *segbad, const int *snap_bad, float4 *mon, float4 *blkmon)
{
    extern __shared__ double sh[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int pix = blockIdx.x * nw + wid;
    if (pix >= j.npix) return;
    double *scan = sh + (size_t)wid * (nseg + 1 + 2 * j.nsnap);
    double *pre0 = scan + nseg + 1;
    double *pre1 = pre0 + j.nsnap;
    // the same for the counts of non-finite frames
    int *bscan = (int *)(sh + (size_t)nw * (nseg + 1 + 2 * j.nsnap)) + (size_t)wid * (nseg + 1 + 2 * j.nsnap);
    int *bad0 = bscan + nseg + 1, *bad1 = bad0 + j.nsnap;
    for (int which = 0; which < (j.is_ccf ? 2 : 1); which++) {
        const size_t tr = which ? j.npix + pix : pix;
        double *pre = which ? pre1 : pre0;
        int *bpre = which ? bad1 : bad0;
        // exclusive scans of the segment totals and counts, then the snapshot prefixes
        double carry = 0.0;
        int bcarry = 0;
        for (int s0 = 0; s0 < nseg; s0 += 32) {
            const int s = s0 + lane;
            double v = 0.0;
            int bv = 0;
            if (s < nseg) {
                const float2 t = __ldg(&segtot[tr * nseg + s]);
                v = f2d(t.x) + f2d(t.y);
                bv = __ldg(&segbad[tr * nseg + s]);
            }
            double incl = v;
            int bincl = bv;
            for (int o = 1; o < 32; o <<= 1) {
                const double u = __shfl_up_sync(0xffffffffu, incl, o);
                const int bu = __shfl_up_sync(0xffffffffu, bincl, o);
                if (lane >= o) { incl += u; bincl += bu; }
            }
            if (s < nseg) { scan[s] = carry + incl - v; bscan[s] = bcarry + bincl - bv; }
            carry += __shfl_sync(0xffffffffu, incl, 31);
            bcarry += __shfl_sync(0xffffffffu, bincl, 31);
        }
        __syncwarp();
        for (int sj = lane; sj < j.nsnap; sj += 32) {
            const int p = li->snap_pos[sj];
            double v = 0.0;
            int bv = 0;
            if (p > 0) {
                const int seg = (p - 1) / kSeg;
                const float2 t = __ldg(&snap_part[tr * j.nsnap + sj]);
                v = scan[seg] + f2d(t.x) + f2d(t.y);
                bv = bscan[seg] + __ldg(&snap_bad[tr * j.nsnap + sj]);
            }
            pre[sj] = v;
            bpre[sj] = bv;
        }
        __syncwarp();
    }
    if (!j.is_ccf) { pre1 = pre0; bad1 = bad0; }
    const double c0 = f2d(bparams[(size_t)pix * kBleachStride + 12]);
    const double c1 = f2d(bparams[(size_t)(j.is_ccf ? j.npix + pix : pix) * kBleachStride + 12]);
    const float qnan = __int_as_float(0x7fc00000);
    for (int x = lane; x < j.chanum; x += 32) {
        const int k = li->level[x];
        const double n = li->prodnum[x], in = li->inv_prodnum[x];
        const int de = li->snap_dir_end[x], lb = li->snap_del_beg[x], le = li->snap_del_end[x];
        const double a = div_by(pre0[de], n, in), b = div_by(pre1[le] - pre1[lb], n, in);
        const double sc = __hiloint2double((1023 + k) << 20, 0);        // 2^k
        float4 m = make_float4((float)a, (float)b, (float)fma(sc, c0, a), (float)fma(sc, c1, b));
        if (bad0[de] > 0) m.x = m.z = qnan;
        if (bad1[le] - bad1[lb] > 0) m.y = m.w = qnan;
        mon[(size_t)pix * j.chanum + x] = m;
    }
    if (lane == 0) {
        const double T1 = j.num - 1, iT1 = li->blk_inv_n[0];
        double dm1 = div_by(fma((double)(j.num - 2), c0, pre0[li->snap_tm2]), T1, iT1);   // zero-led direct window
        double Dm1 = div_by(fma((double)(j.num - 1), c1, pre1[li->snap_tm1]), T1, iT1);
        if (bad0[li->snap_tm2] > 0) dm1 = nan("");
        if (bad1[li->snap_tm1] > 0) Dm1 = nan("");
        blkmon[pix] = make_float4((float)(dm1 - c0), (float)(Dm1 - c1), (float)dm1, (float)Dm1);
    }
}

// ---------------------------------------------------------------------------
// Blocking pass (blockTransform, java:9217-9422).  The lag-1 products of the
// zero-led sequence J = [0, v_0, ..., v_{T-2}] are
//   p_j = (J_j - dm1) (J_{j+1} - Dm1),  j = 0 .. T-2,
// blocked pairwise (block means, java:9308-9316).  One thread per (pixel,
// segment of 256 products) computes, for levels 0..8, the sums of block means
// and squared block means of the complete blocks inside its segment, and the
// segment sum for the higher levels.
// ---------------------------------------------------------------------------
// One product into a level-0 sum pair, one block into a level's.
__device__ __forceinline__ void blk_add(float &S1, float &S2, float m)
{
    S1 = __fadd_rn(S1, m);
    S2 = fmaf(m, m, S2);
}

// A whole segment is sixteen steps of sixteen products: levels 1 to 4 are
// sums inside a step, levels 5 to 8 are carried between steps (the same
// branches for every thread).  Run-time carries for every product took 58
// instructions each; HBM-bound now (4 B a frame-pixel): 1.45 -> 0.59 ms at
// 16,384 pixels x 50,000 frames.  Four segments a thread, to halve the
// statistics written, gained nothing (0.62 + 0.18 against 0.59 + 0.22 ms).
template <bool CCF>
__global__ void __launch_bounds__(128) block_kernel(Job j, const float *s0a, const float *s0b,
                                                    const float4 *blkmon, int nbseg, float *s1, float *s2,
                                                    float *segsum)
{
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    const int seg = blockIdx.y;
    if (pix >= j.npix) return;
    const float4 bm = blkmon[pix];   // a1 = dm1 - c0, b1 = Dm1 - c1, dm1, Dm1
    const int nprod = j.num - 1;
    const int j0 = seg * kBlkSeg, j1 = min(j0 + kBlkSeg, nprod);
    float S1[kBlkSegLog + 1], S2[kBlkSegLog + 1], pend[kBlkSegLog + 1];
#pragma unroll
    for (int y = 0; y <= kBlkSegLog; y++) { S1[y] = 0.f; S2[y] = 0.f; pend[y] = 0.f; }
    // direct element of product jj is J_jj = v_{jj-1} (J_0 = 0); s0 holds the
    // corrected values centred on c, so J - dm1 = s0 - (dm1 - c)
    const float *pa = s0a + (size_t)j0 * j.npix + pix, *pb = s0b + (size_t)j0 * j.npix + pix;
    float u_prev = (j0 == 0) ? -bm.z : __ldg(pa - j.npix) - bm.x;
    float segv = 0.f;
    int t = j0;
    constexpr int kStep = 16, kStepLog = 4;
#pragma unroll 1
    for (; t + kStep <= j1; t += kStep) {
        float v[kStep], w[kStep];
#pragma unroll
        for (int u = 0; u < kStep; u++) {
            v[u] = __ldg(&pa[(size_t)u * j.npix]);
            w[u] = CCF ? __ldg(&pb[(size_t)u * j.npix]) : v[u];
        }
        pa += (size_t)kStep * j.npix;
        pb += (size_t)kStep * j.npix;
#pragma unroll
        for (int u = 0; u < kStep; u++) {
            const float p = __fmul_rn(u_prev, w[u] - bm.y);
            u_prev = v[u] - bm.x;    // next direct element J_{t+u+1} = v_{t+u}
            blk_add(S1[0], S2[0], p);
            v[u] = p;
        }
#pragma unroll
        for (int y = 1; y <= kStepLog; y++)
#pragma unroll
            for (int i = 0; i < (kStep >> y); i++) {
                v[i] = __fadd_rn(v[2 * i], v[2 * i + 1]);
                blk_add(S1[y], S2[y], v[i] * (1.f / (float)(1 << y)));
            }
        float c = v[0];
        const int rel = (t - j0) >> kStepLog;
        bool carry = true;
#pragma unroll
        for (int y = kStepLog; y < kBlkSegLog; y++) {
            if (carry) {
                if ((rel >> (y - kStepLog)) & 1) {
                    c = __fadd_rn(pend[y], c);
                    blk_add(S1[y + 1], S2[y + 1], c * (1.f / (float)(1 << (y + 1))));
                } else {
                    pend[y] = c;
                    carry = false;
                }
            }
        }
        if (carry) segv = c;
    }
    // the last segment's remaining products, one by one
#pragma unroll 1
    for (; t < j1; t++) {
        const float va = __ldg(pa), vb = CCF ? __ldg(pb) : va;
        pa += j.npix;
        pb += j.npix;
        const float p = __fmul_rn(u_prev, vb - bm.y);
        u_prev = va - bm.x;
        blk_add(S1[0], S2[0], p);
        const int rel = t - j0;
        float c = p;
        bool carry = true;
#pragma unroll
        for (int y = 0; y < kBlkSegLog; y++) {
            if (carry) {
                if ((rel >> y) & 1) {
                    c = __fadd_rn(pend[y], c);
                    blk_add(S1[y + 1], S2[y + 1], c * (1.f / (float)(1 << (y + 1))));
                } else {
                    pend[y] = c;
                    carry = false;
                }
            }
        }
        if (carry) segv = c;
    }
    // [level][segment][pixel]: coalesced here and in the finaliser
#pragma unroll
    for (int y = 0; y <= kBlkSegLog; y++) {
        const size_t o = ((size_t)y * nbseg + seg) * j.npix + pix;
        s1[o] = S1[y];
        s2[o] = S2[y];
    }
    segsum[(size_t)seg * j.npix + pix] = segv;     // used only for complete segments
}

// Blocking decision.  A CTA serves 32 pixels with 16 threads each: thread
// (pixel, y) sums the segments' statistics of level y (and y + 16) in three
// FP32 terms, no less precise than FP64 (coalesced across pixels, in segment
// order), the levels above the segment size from segment sums, and takes the
// level's standard deviation in FP64; then one thread per pixel applies the overlap / monotonic-increase
// criteria of java:9339-9380.  FP64 sums by 8 threads a pixel: 0.39 ms at
// 16,384 pixels x 50,000 frames, this 0.07.
constexpr int kBlkFinPix = 32, kBlkFinLev = 16;

// f(value, value) over n pairs `stride` apart, the loads of U at a time.
template <int U, class F>
__device__ __forceinline__ void blk_walk(const float *p1, const float *p2, size_t stride, int n, F f)
{
    int i = 0;
    for (; i + U <= n; i += U) {
        float v[U], w[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            v[u] = __ldg(&p1[u * stride]);
            w[u] = __ldg(&p2[u * stride]);
        }
        p1 += U * stride;
        p2 += U * stride;
#pragma unroll
        for (int u = 0; u < U; u++) f(v[u], w[u]);
    }
    for (; i < n; i++) {
        f(__ldg(p1), __ldg(p2));
        p1 += stride;
        p2 += stride;
    }
}

// Sums a1, a2 of the means and squared means of nb blocks of S * parts segment
// sums each (inv: 1 / products of a block, a power of two), loads of 16 at a
// time: whole blocks where S < 16.
template <int S>
__device__ __forceinline__ void blk_upper(const float *p, size_t stride, int nb, int parts, float inv, ff3 &a1,
                                          ff3 &a2)
{
    constexpr int G = 16 / S;             // blocks per batch
    for (int b = 0; b < nb; b += G) {
        ff3 sb[G];
#pragma unroll
        for (int g = 0; g < G; g++) sb[g] = {0.f, 0.f, 0.f};
        for (int q = 0; q < parts; q++, p += 16 * stride) {
            float v[16];
#pragma unroll
            for (int u = 0; u < 16; u++) v[u] = b + u / S < nb ? __ldg(&p[u * stride]) : 0.f;
#pragma unroll
            for (int u = 0; u < 16; u++) ff3_add(sb[u / S], v[u] * inv);
        }
#pragma unroll
        for (int g = 0; g < G; g++) {     // (past the last block: zeros)
            ff3_add(a1, sb[g].hi);
            ff3_add_low(a1, sb[g].mid);
            a1.lo = __fadd_rn(a1.lo, sb[g].lo);
            ff3_add_square(a2, sb[g]);
        }
    }
}

// The same sums of level y in FP64, for statistics that left the FP32 range.
static __device__ __noinline__ void blk_plain_sums(const float *s1, const float *s2, const float *segsum, int y,
                                                   int nbseg, int full_segs, size_t npix, int pix, double &A1,
                                                   double &A2)
{
    A1 = A2 = 0.0;
    if (y <= kBlkSegLog) {
        for (int seg = 0; seg < nbseg; seg++) {
            A1 += (double)s1[((size_t)y * nbseg + seg) * npix + pix];
            A2 += (double)s2[((size_t)y * nbseg + seg) * npix + pix];
        }
        return;
    }
    const int span = 1 << (y - kBlkSegLog);
    for (int seg = 0; seg + span <= full_segs; seg += span) {
        double sb = 0.0;
        for (int k = 0; k < span; k++) sb += (double)segsum[(size_t)(seg + k) * npix + pix];
        sb /= (double)(1 << y);
        A1 += sb;
        A2 += sb * sb;
    }
}

__global__ void __launch_bounds__(kBlkFinPix * kBlkFinLev)
block_finalize_kernel(Job j, const LagInfo *li, int q, int nbseg, const float *s1, const float *s2, const float *segsum,
                      const float4 *blkmon, int *ind_out, int *ok_out)
{
    // the levels' standard deviations and their error bars' ends
    __shared__ double vb[kMaxBlockLevels][kBlkFinPix], up[kMaxBlockLevels][kBlkFinPix], lo[kMaxBlockLevels][kBlkFinPix];
    const int pl = threadIdx.x % kBlkFinPix, ty = threadIdx.x / kBlkFinPix;
    const int pix = blockIdx.x * kBlkFinPix + pl;
    const int blocknum = j.blocknum;
    const int full_segs = (j.num - 1) / kBlkSeg;   // segments holding kBlkSeg products
    if (pix < j.npix && ty < blocknum) {
        const float4 bm = blkmon[pix];
        const double dmDm = f2d(bm.z) * f2d(bm.w), idm = rcp_near(dmDm, bm.z * bm.w);
        for (int y = ty; y < blocknum; y += kBlkFinLev) {
            if (bm.x != bm.x || bm.y != bm.y) {     // a non-finite frame: every product is non-finite
                vb[y][pl] = up[y][pl] = lo[y][pl] = __longlong_as_double(0x7ff8000000000000ll);
                continue;
            }
            ff3 a1 = {0.f, 0.f, 0.f}, a2 = a1;
            if (y <= kBlkSegLog) {
                const size_t o = (size_t)y * nbseg * j.npix + pix;
                blk_walk<16>(s1 + o, s2 + o, j.npix, nbseg, [&](float v, float w) {
                    ff3_add(a1, v);
                    ff3_add(a2, w);
                });
            } else {
                // levels above the segment: block y spans 2^(y-8) consecutive
                // complete segments (a non-finite segment sum, from a
                // non-finite frame, propagates like the Java sums)
                const int span = 1 << (y - kBlkSegLog), nb = full_segs / span;
                const float inv = 1.f / (float)(1 << y);
                const float *p = segsum + pix;
                if (span == 2) blk_upper<2>(p, j.npix, nb, 1, inv, a1, a2);
                else if (span == 4) blk_upper<4>(p, j.npix, nb, 1, inv, a1, a2);
                else if (span == 8) blk_upper<8>(p, j.npix, nb, 1, inv, a1, a2);
                else blk_upper<16>(p, j.npix, nb, span / 16, inv, a1, a2);
            }
            double A1 = ff3_val(a1), A2 = ff3_val(a2);
            if (!(isfinite(a1.hi) && isfinite(a2.hi)))
                blk_plain_sums(s1, s2, segsum, y, nbseg, full_segs, j.npix, pix, A1, A2);
            const double n = f2d((float)((j.num - 1) >> y)), in = li->blk_inv_n[y];
            const double m1 = div_by(A1, n, in), m2 = div_by(A2, n, in);
            const double v = newton_sqrt(div_near(fma(-m1, m1, m2), n * dmDm * dmDm, in * idm * idm));
            const double e = div_by(v, li->blk_root[y], li->blk_inv_root[y]);
            vb[y][pl] = v;
            up[y][pl] = v + e;
            lo[y][pl] = v - e;
        }
    }
    __syncthreads();
    if (ty != 0 || pix >= j.npix) return;
    // criteria as bit masks over the levels: error bars of neighbours overlap
    // (crt), the deviation grows (pos)
    unsigned crt = 0, pos = 0;
    for (int x = 0; x + 1 < blocknum; x++) {
        if (up[x][pl] > lo[x + 1][pl] && up[x + 1][pl] > lo[x][pl]) crt |= 1u << x;
        if (vb[x + 1][pl] > vb[x][pl]) pos |= 1u << x;
    }
    const unsigned below = (1u << (blocknum - 2)) - 1;
    unsigned cr12 = crt & (crt >> 1) & below;
    const unsigned rise = pos & (pos >> 1) & below & ~cr12;
    const int last0 = rise ? 31 - __clz(rise) : 0;
    cr12 &= ~((2u << last0) - 1);
    cr12 &= ~(3u << (blocknum - 4));
    cr12 &= (1u << (blocknum - 4)) - 2;              // levels 1 .. blocknum - 5
    const int ok = cr12 != 0;
    int ind = ok ? __ffs(cr12) : (blocknum - 3 > 0 ? blocknum - 3 : blocknum - 1);
    if (ind < q - 1) ind = q - 1;
    ind_out[pix] = ind;
    ok_out[pix] = ok;
}

// Centre of traces whose bleach parameters were supplied by the caller
// (reference calcACF path): mean of the corrected averaged trace.
__global__ void center_given_kernel(Job j, const float *trace, float *bp_out)
{
    const int lane = threadIdx.x & 31;
    const int tr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (tr >= j.ntrace) return;
    float *bp = bp_out + (size_t)tr * kBleachStride;
    const float *y = trace + (size_t)tr * j.nopit;
    float bpl[kBleachStride];
    for (int i = 0; i < kBleachStride; i++) bpl[i] = bp[i];
    float s = 0.f, cnt = 0.f, lb[kMaxPoly + 1];
    for (int x = lane; x < j.nopit; x += 32) {
        float v = __ldg(&y[x]);
        if (j.bleach != IMFCS_BLEACH_NONE && bpl[11] != 0.f) {
            float t = j.frametime * ((float)x + 0.5f) * (float)j.ave;
            if (j.bleach == IMFCS_BLEACH_POLYNOMIAL) legendre(t * bpl[13] + bpl[14], j.poly_order, lb);
            v = bleach_correct(v, bleach_f(bpl, j.bleach, j.poly_order, t, lb), bpl[9], bpl[10]);
        }
        if (isfinite(v)) { s += v; cnt += 1.f; }
    }
    s = warp_sum(s);
    cnt = warp_sum(cnt);
    if (lane == 0) bp[12] = cnt > 0.f ? s / cnt : 0.f;
}

// Stride-1 box-sum binning of a float stack (calc_binning, agpufitjni.cu:4560-4586).
__global__ void binning_kernel(const float *in, float *out, int win, int hin, int wt, int ht,
                               int frames, int bx, int by)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)wt * ht * frames;
    if (i >= n) return;
    int x = (int)(i % wt);
    int y = (int)((i / wt) % ht);
    size_t t = i / ((size_t)wt * ht);
    const float *f = in + t * (size_t)win * hin;
    float s = 0.f;
    for (int a = 0; a < bx; a++)
        for (int b = 0; b < by; b++) s += f[(size_t)(y + b) * win + x + a];
    out[i] = s;
}

// Averages of `ave` frames per pixel of a float stack [t][h][w] -> [h][w][nopit]
// with the Java CPU's truncating division (java:9852).
__global__ void bleach_average_kernel(const float *in, float *out, int w, int h, int nopit, int ave)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)w * h * nopit) return;
    int pix = (int)(i / nopit), x = (int)(i % nopit);
    double s = 0.0;
    for (int f = x * ave; f < (x + 1) * ave; f++) s += in[(size_t)f * w * h + pix];
    out[i] = (float)trunc(s / ave);
}

// Explicit instantiations used by the host side.
template __global__ void bleach_exp_kernel<3>(Job, const float *, float *);
template __global__ void bleach_exp_kernel<5>(Job, const float *, float *);

}  // namespace imfcs

namespace imfcs {

// How the averaged trace is taken: the raw rows read, from row0 on, the lines
// of sums, and the points whose sums s0 holds at a time (0: the one-pass
// kernel, which needs no scratch).  Times of the stage in us, one pass / two:
//   regions narrower than half the frame, or using a third of its values or
//     less (every second pixel of every second row at 128x128x20,000: 99 /
//     132, the left half of the frame at 12,345: 130 / 107): one pass;
//   single pixels: two (64x64x1,999 46 / 38, 128x128x10,000 241 / 130,
//     256x256x4,500 576 / 391), but in parts 79 / 89 (half the frame, 1,500);
//   windows whose rows do not overlap: two from two frames a point on (128x128,
//     3 x 3: 36 / 52 at one frame, 54 / 50 at two, 89 / 50 at four; 512x512, 5 x
//     5: 189 / 237, 316 / 294, 573 / 417), from three on where s0 holds less than
//     a third of the sums (128x128, 16 x 16: 128 / 153 at two, 236 / 131 at four),
//     from one on where a value is used twice (2 x 2 cross-correlation at
//     128x128x1,500: 74 / 59);
//   other windows, whose sums are as many as the raw values: where s0 holds them
//     (overlapping 5 x 5 windows at 101x67: 95 / 87 at one frame, 738 / 105 at
//     twelve), else with half as many frames again a point as parts, each of
//     which adds up its windows anew (128x128, 8 x 8 in steps of 4: 113 / 152 at
//     four frames and four parts, 183 / 135 at seven and three; 16 x 16 in steps
//     of 8: 419 / 617 at seven and eleven, 1,160 / 327 at twenty and four).
struct TracePlan {
    TraceSums g;
    int row0, points;
    bool rows;
};
static TracePlan trace_plan(const Job &j)
{
    TracePlan p;
    p.row0 = j.map_y0 * j.pixbiny + (j.cfy < 0 ? j.cfy : 0);
    const int row1 = (j.map_y0 + j.out_h - 1) * j.pixbiny + j.biny + (j.cfy > 0 ? j.cfy : 0);
    const int cols = (j.out_w - 1) * j.pixbinx + j.binx + (j.cfx < 0 ? -j.cfx : j.cfx);
    const size_t raw = (size_t)(row1 - p.row0) * j.in_w;
    p.points = 0;
    if (j.input_float || 2 * cols < j.in_w || raw > (1u << 30)) return p;
    p.rows = j.biny > 1 && j.pixbiny >= j.biny && !j.cfy;
    p.g.lines = p.rows ? j.out_h : 1;
    p.g.len = p.rows ? j.in_w : (int)raw;
    p.g.lstride = j.pixbiny * j.in_w;
    p.g.rows = p.rows ? j.biny : 1;
    p.g.in_w = j.in_w;
    const size_t area = (size_t)j.binx * j.biny, values = (size_t)j.ntrace * area;
    if (3 * values <= raw) return p;
    const size_t points = level0_stream_floats(j) / ((size_t)p.g.lines * p.g.len), all = j.nopit;
    bool one;
    if (area == 1) one = points < all;
    else if (j.ave < 2 && values < 2 * raw) one = true;
    else if (p.rows) one = j.ave < 3 && 3 * points < all;
    else one = points < all && 2 * j.ave * points <= 3 * all;
    if (one) return p;
    p.points = points < (size_t)j.nopit ? (int)points : j.nopit;
    return p;
}

int trace_kernel_count(const Job &j)
{
    const TracePlan p = trace_plan(j);
    return p.points ? 2 * ((j.nopit + p.points - 1) / p.points) : 1;
}

cudaError_t launch_trace(const Job &j, const void *stack, float *scratch, float *trace, cudaStream_t s)
{
    const dim3 block(32, 8);
    const unsigned gx = (j.ntrace + 31) / 32;
    const TracePlan p = trace_plan(j);
    if (!p.points) {
        trace_kernel<<<dim3(gx, (j.nopit + 31) / 32), block, 0, s>>>(j, stack, trace);
        return cudaGetLastError();
    }
    unsigned *sums = (unsigned *)scratch;
    const size_t fsz = (size_t)j.in_w * j.in_h;
    const int n = p.g.lines * p.g.len;
    for (int p0 = 0; p0 < j.nopit; p0 += p.points) {
        const int np = p.points < j.nopit - p0 ? p.points : j.nopit - p0;
        const uint16_t *base =
            (const uint16_t *)stack + ((size_t)j.first + (size_t)p0 * j.ave) * fsz + (size_t)p.row0 * j.in_w;
        // whole vectors of a line, aligned in every row (ROWS: of in_w elements) and frame
        auto fits = [&](int vec) { return (uintptr_t)base % (2 * vec) == 0 && fsz % vec == 0 && p.g.len % vec == 0; };
#define SUMS(vec, rows) \
    trace_sums_kernel<vec, rows><<<dim3((n / vec + 127) / 128, np), 128, 0, s>>>(base, fsz, p.g, j.ave, sums)
        if (p.rows) {
            if (fits(8)) SUMS(8, true);
            else if (fits(2)) SUMS(2, true);
            else SUMS(1, true);
        } else {
            if (fits(8)) SUMS(8, false);
            else if (fits(2)) SUMS(2, false);
            else SUMS(1, false);
        }
#undef SUMS
        const dim3 grid(gx, (np + 31) / 32);
        if (p.rows) trace_windows_kernel<true><<<grid, block, 0, s>>>(j, sums, p.row0, n, p0, np, trace);
        else trace_windows_kernel<false><<<grid, block, 0, s>>>(j, sums, p.row0, n, p0, np, trace);
    }
    return cudaGetLastError();
}

size_t bleach_grid_floats() { return (size_t)kGridPad * (kGridPts + 3); }

cudaError_t launch_bleach_grid_table(const Job &j, float *tab, cudaStream_t s)
{
    float tmax;
    bleach_grid_table_kernel<<<kGridPad, 32, 0, s>>>(j.nopit, bleach_dts(j, tmax), tab);
    return cudaGetLastError();
}

cudaError_t launch_bleach(const Job &j, const float *trace, const double *proj, float uscale,
                          float uoff, const float *grid, float *bparams, cudaStream_t s)
{
    const int threads = 128;
    const int blocks = (j.ntrace * 32 + threads - 1) / threads;
    switch (j.bleach) {
    case IMFCS_BLEACH_POLYNOMIAL:
        switch (j.poly_order) {
#define POLY(o) case o: bleach_poly_kernel<o + 1><<<blocks, threads, 0, s>>>(j, trace, proj, uscale, uoff, bparams); break
            POLY(1); POLY(2); POLY(3); POLY(4); POLY(5); POLY(6); POLY(7); POLY(8);
#undef POLY
        }
        break;
    case IMFCS_BLEACH_SINGLE_EXP:
        // eight traces a CTA reuse a basis value most (0.15 ms for 16,384); with
        // fewer than two such CTAs per SM (152) two a CTA fill the chip better
        if (j.ntrace >= 8 * 304) bleach_grid_kernel<8><<<(j.ntrace + 7) / 8, 128, 0, s>>>(j, trace, grid, bparams);
        else bleach_grid_kernel<2><<<(j.ntrace + 1) / 2, 128, 0, s>>>(j, trace, grid, bparams);
        bleach_exp_kernel<3><<<blocks, threads, 0, s>>>(j, trace, bparams);
        break;
    case IMFCS_BLEACH_DOUBLE_EXP:
        bleach_exp_kernel<5><<<blocks, threads, 0, s>>>(j, trace, bparams);
        break;
    default:
        center_kernel<<<blocks, threads, 0, s>>>(j, trace, bparams);
    }
    return cudaGetLastError();
}

cudaError_t launch_center_given(const Job &j, const float *trace, float *bparams, cudaStream_t s)
{
    const int threads = 128;
    center_given_kernel<<<(j.ntrace * 32 + threads - 1) / threads, threads, 0, s>>>(j, trace, bparams);
    return cudaGetLastError();
}

cudaError_t launch_monitor_finalize(const Job &j, const LagInfo *li_dev, const float *bparams, int nseg,
                                    const float2 *segtot, const float2 *snap_part, const int *segbad,
                                    const int *snap_bad, float4 *mon, float4 *blkmon, cudaStream_t s)
{
    // four pixels a block; fewer where a recording's segments leave no room for
    // their scans (from 1.1 million frames on, to 4.9 million with one)
    constexpr size_t kMaxSmem = 227 * 1024;
    const size_t one = (size_t)(nseg + 1 + 2 * j.nsnap) * (sizeof(double) + sizeof(int));
    int wpb = 4;
    while (wpb > 1 && wpb * one > kMaxSmem) wpb /= 2;
    const size_t smem = wpb * one;
    if (smem > 48 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(monitor_finalize_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    monitor_finalize_kernel<<<(j.npix + wpb - 1) / wpb, wpb * 32, smem, s>>>(j, li_dev, bparams, nseg, segtot,
                                                                           snap_part, segbad, snap_bad, mon,
                                                                           blkmon);
    return cudaGetLastError();
}

cudaError_t launch_block(const Job &j, const LagInfo *li, const float *s0, const float4 *blkmon, int nbseg, float *s1, float *s2,
                         float *segsum, int *ind, int *ok, cudaStream_t s)
{
    dim3 grid((j.npix + 127) / 128, nbseg);
    const float *s0b = j.is_ccf ? s0 + (size_t)j.npix * j.num : s0;
    if (j.is_ccf) block_kernel<true><<<grid, 128, 0, s>>>(j, s0, s0b, blkmon, nbseg, s1, s2, segsum);
    else block_kernel<false><<<grid, 128, 0, s>>>(j, s0, s0b, blkmon, nbseg, s1, s2, segsum);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    block_finalize_kernel<<<(j.npix + kBlkFinPix - 1) / kBlkFinPix, kBlkFinPix * kBlkFinLev, 0, s>>>(
        j, li, j.q, nbseg, s1, s2, segsum, blkmon, ind, ok);
    return cudaGetLastError();
}

cudaError_t launch_binning(const float *in, float *out, int win, int hin, int wt, int ht,
                           int frames, int bx, int by, cudaStream_t s)
{
    size_t n = (size_t)wt * ht * frames;
    binning_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, out, win, hin, wt, ht, frames, bx, by);
    return cudaGetLastError();
}

cudaError_t launch_bleach_average(const float *in, float *out, int w, int h, int nopit, int ave,
                                  cudaStream_t s)
{
    size_t n = (size_t)w * h * nopit;
    bleach_average_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, out, w, h, nopit, ave);
    return cudaGetLastError();
}

}  // namespace imfcs
