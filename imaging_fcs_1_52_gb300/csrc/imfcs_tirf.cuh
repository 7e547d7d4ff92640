// imfcs_tirf.cuh -- the N-free part a(D, tau) of the one-component FCS_3p model
// (java:13131-13408) without flow and triplet, for the specialised fit kernels:
// FP32 with da/dD, FP64, and float-float.
#pragma once

#include "imfcs_ff.cuh"
#include "imfcs_lm.cuh"

namespace imfcs {

struct TirfC {
    float ax, ay, rx, ry, s2, inv_sz2, inv_norm;
    double axd, ayd, rxd, ryd, sd, inv_sz2d, inv_normd;
    f2 s2f, inv_normf;   // float-float copies for the precise residuals
    bool square;         // ax == ay (and rx == ry): the two lateral factors coincide
    bool axial;          // the axial factor can differ from 1 in FP64 (finite sz)
};

__device__ __forceinline__ TirfC tirf_consts(const ModelConst &mc)
{
    TirfC c;
    c.ax = mc.ax; c.ay = mc.ay; c.rx = mc.rx; c.ry = mc.ry;
    c.s2 = mc.s * mc.s; c.inv_sz2 = 1.f / (mc.sz * mc.sz);
    c.inv_norm = mc.inv_norm;
    c.axd = mc.ax; c.ayd = mc.ay; c.rxd = mc.rx; c.ryd = mc.ry;
    c.sd = mc.s; c.inv_normd = mc.inv_norm;
    c.inv_sz2d = 1.0 / ((double)mc.sz * (double)mc.sz);
    c.square = mc.ay == mc.ax && mc.ry == mc.rx;
    c.s2f = f2_two_prod(mc.s, mc.s);
    c.inv_normf = f2_from_f(mc.inv_norm);
    // 4 D tau / sz^2 at the largest D and lag time a fit can reach is far
    // below FP64 resolution for a TIRF sz; the axial factor is then exactly 1
    c.axial = !(c.inv_sz2d * 4e6 < 1e-17);
    return c;
}

// Lateral factor of a square-pixel window without offset or flow (the
// two-term form of lateral_1d_f).
__device__ __forceinline__ void tirf_lat(float a, float p0, float inv_p0, float &L, float &dL)
{
    const float inv_sqrtpi = 0.5641895835477563f;
    const float u = a * inv_p0;
    const float m = expm1f(-u * u), er = erff(u);
    L = 2.f * (p0 * inv_sqrtpi * m + a * er);
    dL = 2.f * m * inv_sqrtpi;
}

// The N-free part of the model a(D, tau) = lateral x axial factor and
// da/dD in FP32, internal units (the model is a / N + G).
template <bool OFF>
static __device__ __noinline__ void tirf_terms(float D, const TirfC &c, float tau, float &a, float &da)
{
    const float p0 = sqrtf(fmaf(4.f * D, tau, c.s2));
    const float inv_p0 = 1.f / p0;
    float Lx, dLx, Ly, dLy;
    if (OFF) {
        float dv;
        lateral_1d_f(c.ax, c.rx, 0.f, tau, p0, inv_p0, Lx, dLx, dv);
        if (c.square) { Ly = Lx; dLy = dLx; }
        else lateral_1d_f(c.ay, c.ry, 0.f, tau, p0, inv_p0, Ly, dLy, dv);
    } else {
        tirf_lat(c.ax, p0, inv_p0, Lx, dLx);
        if (c.square) { Ly = Lx; dLy = dLx; }
        else tirf_lat(c.ay, p0, inv_p0, Ly, dLy);
    }
    const float dp0 = 2.f * tau * inv_p0;
    const float lat = Lx * Ly * c.inv_norm;
    const float dlat = (dLx * Ly + Lx * dLy) * dp0 * c.inv_norm;
    const float psp = rsqrtf(fmaf(4.f * D * tau, c.inv_sz2, 1.f));
    const float dpsp = -2.f * tau * c.inv_sz2 * psp * psp * psp;
    a = lat * psp;
    da = dlat * psp + lat * dpsp;
}

// The same inline, without offset, for the points of a lane side by side.
__device__ __forceinline__ void tirf_terms_plain(float D, const TirfC &c, float tau, float &a, float &da)
{
    const float p0 = sqrtf(fmaf(4.f * D, tau, c.s2));
    const float inv_p0 = 1.f / p0;
    float Lx, dLx, Ly, dLy;
    tirf_lat(c.ax, p0, inv_p0, Lx, dLx);
    if (c.square) { Ly = Lx; dLy = dLx; }
    else tirf_lat(c.ay, p0, inv_p0, Ly, dLy);
    const float dp0 = 2.f * tau * inv_p0;
    const float lat = Lx * Ly * c.inv_norm;
    const float dlat = fmaf(dLx, Ly, __fmul_rn(Lx, dLy)) * dp0 * c.inv_norm;   // rounded as in tirf_terms
    const float psp = rsqrtf(fmaf(4.f * D * tau, c.inv_sz2, 1.f));
    const float dpsp = -2.f * tau * c.inv_sz2 * psp * psp * psp;
    a = lat * psp;
    da = dlat * psp + lat * dpsp;
}

// Model value and gradient (d/dN, d/dD; d/dG = 1) in FP32, internal units;
// mag = |a/N| + |G|, the magnitude of the summed terms (the rounding error
// of the value is relative to it).
template <bool OFF, bool INLINE = false>
__device__ __forceinline__ float tirf_f(float N, float D, float G, const TirfC &c, float tau, float &gN, float &gD,
                                        float &mag)
{
    float a, da;
    if (INLINE) tirf_terms_plain(D, c, tau, a, da);
    else tirf_terms<OFF>(D, c, tau, a, da);
    const float iN = 1.f / N;
    gN = -a * iN * iN;
    gD = iN * da;
    const float aN = __fmul_rn(a, iN);
    mag = fabsf(aN) + fabsf(G);
    return aN + G;
}

// FP64 N-free model part a (the precise residuals: a / N + G), with as few
// FP64 divisions and square roots as the accuracy allows (GB300 issues FP64
// at 1/64 of the FP32 rate): 1/p0 from one reciprocal square root, and the
// axial factor (1 + 4 D tau / sz^2)^(-1/2) only where it differs from 1 in
// FP64 (a TIRF model's sz is ~1e6 um: 4 D tau / sz^2 < 1e-17 and the factor
// rounds to exactly 1).  The offset lateral factor (OFF) divides by p0.
template <bool OFF>
static __device__ __noinline__ double tirf_a_d(double D, const TirfC &c, double tau)
{
    const double inv_sqrtpi = 0.56418958354775628695;
    const double p2 = 4.0 * D * tau + c.sd * c.sd;
    const double ip0 = rsqrt(p2);
    const double p0 = p2 * ip0;
    double lx, ly;
    if (OFF) {
        lx = lateral_1d_d(c.axd, c.rxd, 0.0, tau, p0);
        ly = c.square ? lx : lateral_1d_d(c.ayd, c.ryd, 0.0, tau, p0);
    } else {
        double u = c.axd * ip0;
        lx = 2.0 * (p0 * inv_sqrtpi * expm1(-u * u) + c.axd * erf(u));
        ly = lx;
        if (!c.square) {
            u = c.ayd * ip0;
            ly = 2.0 * (p0 * inv_sqrtpi * expm1(-u * u) + c.ayd * erf(u));
        }
    }
    double a1 = lx * ly * c.inv_normd;
    const double ax = 4.0 * D * tau * c.inv_sz2d;
    if (ax > 1e-17) a1 *= rsqrt(1.0 + ax);
    return a1;
}

// Float-float model value for the precise residuals: about 1e-12 relative,
// far below what the residuals need (the data are FP32), on the FP32 pipes.
// erf(u) = u sum_n e_n x^n with e_n = (2/sqrt(pi)) (-1)^n / (n! (2n+1)) and
// expm1(-x) = -x sum_n q_n x^n with q_n = (-1)^n / (n+1)!, x = u^2, are the
// Taylor series, truncated at n = 15: for u <= 1 the first omitted terms are
// below 3e-14 and 5e-14.  Points with u > 1 (windows much wider than the
// PSF) or an axial factor different from 1 in FP64 (SPIM) take the FP64
// model instead.
constexpr int kSeriesN = 16;

// The series coefficients as float-float (hi = the float nearest the FP64
// value, lo = the float nearest the remainder), evaluated at compile time.
struct SeriesTab {
    float eh[kSeriesN], el[kSeriesN], qh[kSeriesN], ql[kSeriesN];
};
constexpr SeriesTab make_series_tab()
{
    SeriesTab t{};
    const double two_sqrtpi = 1.1283791670955125739;   // 2 / sqrt(pi)
    double fact = 1.0;                                 // n!
    for (int n = 0; n < kSeriesN; n++) {
        if (n > 0) fact *= n;
        const double en = ((n & 1) ? -1.0 : 1.0) * two_sqrtpi / (fact * (2 * n + 1));
        const double qn = ((n & 1) ? -1.0 : 1.0) / (fact * (n + 1));
        t.eh[n] = (float)en;
        t.el[n] = (float)(en - (double)t.eh[n]);
        t.qh[n] = (float)qn;
        t.ql[n] = (float)(qn - (double)t.qh[n]);
    }
    return t;
}
static __constant__ SeriesTab kSeries = make_series_tab();

__device__ __forceinline__ f2 ff_const(const float *hi, const float *lo, int n) { return {hi[n], lo[n]}; }

// L = 2 (p0 / sqrt(pi) expm1(-u^2) + a erf(u)), u = a / p0 (float-float);
// false when u > 1
__device__ __forceinline__ bool tirf_lat_ff(float a, f2 p0, f2 ip0, f2 &L)
{
    const f2 u = f2_mul_f(ip0, a);
    if (!(u.hi <= 1.f)) return false;
    const f2 x = f2_mul(u, u);
    f2 pe = ff_const(kSeries.eh, kSeries.el, kSeriesN - 1), pq = ff_const(kSeries.qh, kSeries.ql, kSeriesN - 1);
#pragma unroll
    for (int n = kSeriesN - 2; n >= 0; n--) {
        pe = f2_add(f2_mul(pe, x), ff_const(kSeries.eh, kSeries.el, n));
        pq = f2_add(f2_mul(pq, x), ff_const(kSeries.qh, kSeries.ql, n));
    }
    const f2 er = f2_mul(u, pe);                     // erf(u)
    const f2 m = f2_neg(f2_mul(x, pq));               // expm1(-u^2)
    const f2 inv_sqrtpi = {5.641896129e-01f, -2.931769139e-08f};   // 1/sqrt(pi) as float-float
    const f2 t1 = f2_mul(f2_mul(p0, inv_sqrtpi), m);
    const f2 t2 = f2_mul_f(er, a);
    const f2 sum = f2_add(t1, t2);
    L = {2.f * sum.hi, 2.f * sum.lo};
    return true;
}

// N-free model part a in float-float at D; false where the FP64 model is
// needed (see above).
__device__ __forceinline__ bool tirf_a_ff(f2 D, const TirfC &c, float tau, f2 &lat)
{
    if (c.axial) return false;
    // p0^2 = 4 D tau + s^2 (4 tau exact), 1/p0 by one Newton step on
    // rsqrtf: e = 1 - p2 r^2, 1/p0 = r + r e / 2 (error ~e^2)
    const f2 p2 = f2_add(f2_mul_f(D, 4.f * tau), c.s2f);
    const float r = rsqrtf(p2.hi);
    const f2 pr2 = f2_mul_f(f2_mul_f(p2, r), r);
    const float e = (1.f - pr2.hi) - pr2.lo;
    const f2 ip0 = f2_two_sum(r, 0.5f * r * e);
    const f2 p0 = f2_mul(p2, ip0);
    f2 Lx, Ly;
    if (!tirf_lat_ff(c.ax, p0, ip0, Lx)) return false;
    if (c.square) Ly = Lx;
    else if (!tirf_lat_ff(c.ay, p0, ip0, Ly)) return false;
    lat = f2_mul(f2_mul(Lx, Ly), c.inv_normf);
    return true;
}

// solve_scaled with its roundings spelled out (where its products are fused
// into the sums depends on the code around it).
__device__ __forceinline__ bool tirf_solve(const float (&A)[9], const float (&g)[3], float lambda, float (&h)[3])
{
    float sc[3], L[9];
#pragma unroll
    for (int i = 0; i < 3; i++) sc[i] = rsqrtf(fmaxf(A[i * 3 + i], 1e-30f));
#pragma unroll
    for (int c = 0; c < 3; c++) {
        float d = 1.f + lambda;
#pragma unroll
        for (int m = 0; m < c; m++) d = fmaf(-L[c * 3 + m], L[c * 3 + m], d);
        if (!(d > 0.f) || !isfinite(d)) return false;
        d = sqrtf(d);
        L[c * 3 + c] = d;
        const float id = 1.f / d;
#pragma unroll
        for (int r = c + 1; r < 3; r++) {
            float sum = __fmul_rn(__fmul_rn(A[r * 3 + c], sc[r]), sc[c]);
#pragma unroll
            for (int m = 0; m < c; m++) sum = fmaf(-L[r * 3 + m], L[c * 3 + m], sum);
            L[r * 3 + c] = __fmul_rn(sum, id);
        }
    }
    float yv[3], z[3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        float sum = r ? fmaf(g[r], sc[r], -__fmul_rn(L[r * 3], yv[0])) : __fmul_rn(g[0], sc[0]);
#pragma unroll
        for (int m = 1; m < r; m++) sum = fmaf(-L[r * 3 + m], yv[m], sum);
        yv[r] = sum / L[r * 3 + r];
    }
#pragma unroll
    for (int r = 2; r >= 0; r--) {
        float sum = yv[r];
#pragma unroll
        for (int m = r + 1; m < 3; m++) sum = fmaf(-L[m * 3 + r], z[m], sum);
        z[r] = sum / L[r * 3 + r];
    }
#pragma unroll
    for (int r = 0; r < 3; r++) h[r] = __fmul_rn(z[r], sc[r]);
    return true;
}

}  // namespace imfcs
