// imfcs_gls.cu -- regularised covariance of the ACF and its Cholesky factor
// for the GLS fit.  One CTA per pixel.
//
// Restates the GLS branch of calculateCF (Imaging_FCS_1_52.java:9524-9610):
// the blocked products of lags 1..C-1 (first pnum blocks, from the
// correlator) normalised by dm*Dm, their mean mcov, the sample covariance,
// the shrinkage weights lamvar (variance towards the median, which includes
// the unset zero-lag slot, java:9563-9573) and lamcov (correlations towards
// zero, with the Java accumulation order, java:9592-9603), then the FP64
// Cholesky with commons-math's thresholds (dataTransform, java:13705-13729)
// and L^-1.
//
// One pass over the centred samples e_xz gives, per lag pair (x >= y),
// S1 = sum_z e_x e_y and S2 = sum_z (e_x e_y)^2 (FP32 per chunk of samples,
// float-float across chunks; each thread owns a 4x4 tile of pairs, so a
// sample loaded from shared memory serves four pairs).  The shrinkage sums follow
// without a second pass:
//   sum_z (e_x^2 - c_xx)^2               = S2_xx - (pnum - 2) c_xx^2
//   sum_z (e_x e_y / (sd_x sd_y) - r_xy)^2 = (S2_xy - (pnum - 2) c_xy^2) / (c_xx c_yy)
// with c = S1 / (pnum - 1) and r = c / (sd_x sd_y).  Divisions by per-lag
// quantities are multiplications by their reciprocals; the median is a
// parallel rank selection on the variances' bits; the FP64 Cholesky runs in
// panels of 8 columns on the packed lower triangle in shared memory.  GB300
// issues FP64 at 1/64 of the FP32 rate, so what needs more than FP32 but not
// the FP64 Cholesky -- the centred samples, the sums across chunks,
// L^-1 (one column per lane) and L^-1 mcov -- runs in float-float
// (compensated products and sums, about 44 bits) on the FP32 pipe; L^-1
// leaves the kernel as FP32.
//
// Bound by FP64 issue (6,200 FP64 warp instructions a pixel at 72 lags, 1.4 ms
// of 2.2 at 4,096 pixels) and the factorisation's serial panels: 2.71 -> 2.21
// ms by panels in one warp's registers instead of three barriers a column,
// uniform loops for L^-1 and four CTAs per SM.  Shrinkage and regularisation
// in float-float would save a tenth more, but L^-1 magnifies its last bits
// past FP32 rounding and weakly determined fits take other steps.
#include <math.h>

#include "imfcs_internal.cuh"
#include "imfcs_args.h"
#include "imfcs_ff.cuh"

namespace imfcs {

constexpr int kGlsThreads = 192;                // 171 tiles of pairs at 72 lags
constexpr int kGlsZChunk = 80;                  // samples summed in FP32 before float-float
constexpr int kGlsZStage = 20;                  // samples staged at a time (four CTAs per SM)
constexpr int kGlsZStride = kGlsZStage + 1;     // odd row stride: rows in distinct banks
constexpr int kMaxN1 = 96;                      // chanum - 1 limit of this kernel
constexpr int kGlsTile = 4;                     // pairs per thread: 4 x 4

__device__ __forceinline__ int tri(int r, int c) { return r * (r + 1) / 2 + c; }   // c <= r

// Compensated dot-product step (float-float operands a, b; sum (sh, sl)):
// the error of the product and of the running sum go to sl, so the result
// carries about twice the FP32 precision, on the FP32 pipe.  Explicitly
// rounded operations: a contracted sh + ah*bh would break the two-sum.
__device__ __forceinline__ void ff_dot_step(float ah, float al, float bh, float bl, float &sh, float &sl)
{
    const float p = __fmul_rn(ah, bh);
    const float pe = __fadd_rn(fmaf(ah, bh, -p), fmaf(ah, bl, __fmul_rn(al, bh)));
    const float t = __fadd_rn(sh, p);
    const float bb = __fsub_rn(t, sh);
    const float e = __fadd_rn(__fsub_rn(sh, __fsub_rn(t, bb)), __fsub_rn(p, bb));
    sl = __fadd_rn(sl, __fadd_rn(e, pe));
    sh = t;
}

// Columns k0 .. k0 + kPanel - 1 of the Cholesky factor, one warp: lane l holds
// rows k0 + l, k0 + l + 32, ... of the panel.  Per pivot: 1/sqrt by
// Newton-Raphson from an FP32 estimate (two steps: ~1e-16), sqrt(d) =
// d / sqrt(d) corrected once, the column scaled, the panel's later columns
// updated.  False where a pivot is not above commons-math's threshold.
constexpr int kPanel = 8;
constexpr int kPanelRows = (kMaxN1 + 31) / 32;
__device__ __forceinline__ bool chol_panel(double *lp, int n1, int k0, double *rdiag, int lane)
{
    double a[kPanelRows][kPanel];
#pragma unroll
    for (int t = 0; t < kPanelRows; t++)
#pragma unroll
        for (int j = 0; j < kPanel; j++) {
            const int r = k0 + lane + 32 * t;
            a[t][j] = r < n1 && k0 + j <= r ? lp[tri(r, k0 + j)] : 0.0;
        }
#pragma unroll
    for (int j = 0; j < kPanel; j++) {
        if (k0 + j >= n1) break;
        const double d = __shfl_sync(0xffffffffu, a[0][j], j);
        if (!(d > 1e-10)) return false;
        double rs, r;
        if (d < 1e30) {
            const double h = -0.5 * d;
            rs = f2d(rsqrtf((float)d));
            rs = rs * fma(h * rs, rs, 1.5);
            rs = rs * fma(h * rs, rs, 1.5);
            r = d * rs;
            r = fma(0.5 * rs, fma(-r, r, d), r);
        } else {
            r = sqrt(d);
            rs = 1.0 / r;
        }
        if (lane == j) rdiag[k0 + j] = rs;
#pragma unroll
        for (int t = 0; t < kPanelRows; t++) {
            if (k0 + 32 * t >= n1) break;
            a[t][j] = t == 0 && lane == j ? r : a[t][j] * rs;
        }
#pragma unroll
        for (int c = j + 1; c < kPanel; c++) {
            const double m = __shfl_sync(0xffffffffu, a[0][j], c);      // L[k0 + c][k0 + j]
#pragma unroll
            for (int t = 0; t < kPanelRows; t++) {
                if (k0 + 32 * t >= n1) break;
                a[t][c] = fma(-a[t][j], m, a[t][c]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < kPanelRows; t++)
#pragma unroll
        for (int j = 0; j < kPanel; j++) {
            const int r = k0 + lane + 32 * t;
            if (r < n1 && k0 + j <= r) lp[tri(r, k0 + j)] = a[t][j];
        }
    return true;
}

__global__ void __launch_bounds__(kGlsThreads, 4) gls_kernel(GlsArgs g)
{
    extern __shared__ double gsh[];
    const int n1 = g.chanum - 1;
    const int npairs = n1 * (n1 + 1) / 2;
    const int nrt = (n1 + kGlsTile - 1) / kGlsTile;    // tile rows
    // [npairs] each, 8 bytes a pair: S1 (float-float) -> covariance (FP64) ->
    // correlation -> regularised covariance -> Cholesky factor (FP64, then
    // float-float), and S2 (float-float) -> t_xy (FP64) -> L^-1 (float-float)
    f2 *cf = (f2 *)gsh, *s2f = (f2 *)(gsh + npairs);
    double *lp = gsh, *s2 = gsh + npairs;
    float *eb = (float *)(gsh + 2 * npairs);   // [nrt*4][kGlsZStride] a stage of centred samples
    __shared__ double cdiag[kMaxN1], isd[kMaxN1], sq[kMaxN1], rdiag[kMaxN1];
    __shared__ f2 inv_dmf[kMaxN1], mcovf[kMaxN1], rdf[kMaxN1];
    __shared__ double red[2][kGlsThreads / 32];
    __shared__ double s_med[2], s_lamvar, s_lamcov, s_inv[2], s_f;
    __shared__ int s_fail;

    const int pix = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pnum = g.pnum_by_ind[g.blk_ind[pix]];
    const float *bp = g.bprod + (size_t)pix * n1 * g.pnum_stride;
    if (tid < n1) {
        const float4 m = g.mon[(size_t)pix * g.chanum + tid + 1];
        rdiag[tid] = 1.0 / (f2d(m.z) * f2d(m.w));
        inv_dmf[tid] = f2_from_d(rdiag[tid]);
    } else if (tid == kGlsThreads - 1) {               // a warp of its own
        s_fail = 0;
        s_inv[0] = 1.0 / (double)(pnum - 1);
        s_inv[1] = 1.0 / (double)pnum;
        s_f = (double)pnum / pow((double)pnum - 1.0, 3);
    }
    for (int i = tid; i < npairs; i += kGlsThreads) cf[i] = s2f[i] = {0.f, 0.f};
    // rows past n1 of the staging buffer stay zero
    for (int i = n1 * kGlsZStride + tid; i < nrt * kGlsTile * kGlsZStride; i += kGlsThreads) eb[i] = 0.f;
    // mcov (java:9526-9531): sum of the blocked products (float-float per
    // lane and across the warp), one warp per lag
    for (int x = warp; x < n1; x += kGlsThreads / 32) {
        float sh = 0.f, sl = 0.f;
        for (int z = lane; z < pnum; z += 32) {
            const f2 t = f2_two_sum(sh, bp[(size_t)x * g.pnum_stride + z]);
            sh = t.hi;
            sl = __fadd_rn(sl, t.lo);
        }
        f2 sum = f2_two_sum(sh, sl);
        for (int o = 16; o > 0; o >>= 1) {
            const f2 other = {__shfl_xor_sync(0xffffffffu, sum.hi, o), __shfl_xor_sync(0xffffffffu, sum.lo, o)};
            sum = f2_add(sum, other);
        }
        if (lane == 0) mcovf[x] = sum;
    }
    __syncthreads();                  // 1 / dm Dm (threads < n1), the constants and the sums (warps)
    const double inv_pm1 = s_inv[0], inv_pnum = s_inv[1];
    if (tid < n1) mcovf[tid] = f2_from_d((f2d(mcovf[tid].hi) + f2d(mcovf[tid].lo)) * rdiag[tid] * inv_pnum);
    __syncthreads();

    // S1, S2 per pair: thread t owns tile (bx, by), bx >= by, of the pairs
    // x in [4 bx, 4 bx + 4), y in [4 by, 4 by + 4)
    const int ntiles = nrt * (nrt + 1) / 2;
    for (int t0 = 0; t0 < ntiles; t0 += kGlsThreads) {
        const int t = t0 + tid;
        int bx = 0, by = 0;
        if (t < ntiles) {
            bx = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
            while ((bx + 1) * (bx + 2) / 2 <= t) bx++;
            while (bx * (bx + 1) / 2 > t) bx--;
            by = t - bx * (bx + 1) / 2;
        }
        for (int z0 = 0; z0 < pnum; z0 += kGlsZChunk) {
            float a1[kGlsTile][kGlsTile], a2[kGlsTile][kGlsTile];
#pragma unroll
            for (int i = 0; i < kGlsTile; i++)
#pragma unroll
                for (int j = 0; j < kGlsTile; j++) { a1[i][j] = 0.f; a2[i][j] = 0.f; }
            for (int zs = z0; zs < min(z0 + kGlsZChunk, pnum); zs += kGlsZStage) {
                const int zn = min(kGlsZStage, pnum - zs);
                __syncthreads();
                // centred sample e = b / (dm Dm) - mcov in float-float: the
                // product exactly as hi + lo, then the subtraction of the mean
                for (int i = tid; i < n1 * kGlsZStage; i += kGlsThreads) {
                    const int x = i / kGlsZStage, z = i - x * kGlsZStage;
                    if (z < zn) {
                        const float b = bp[(size_t)x * g.pnum_stride + zs + z];
                        const f2 iv = inv_dmf[x], mc = mcovf[x];
                        const float ph = __fmul_rn(b, iv.hi);
                        const float pl = fmaf(b, iv.lo, fmaf(b, iv.hi, -ph));
                        eb[x * kGlsZStride + z] = __fadd_rn(__fsub_rn(ph, mc.hi), __fsub_rn(pl, mc.lo));
                    }
                }
                __syncthreads();
                if (t >= ntiles) continue;
                const float *ex = eb + (kGlsTile * bx) * kGlsZStride, *ey = eb + (kGlsTile * by) * kGlsZStride;
                for (int z = 0; z < zn; z++) {
                    float vx[kGlsTile], vy[kGlsTile];
#pragma unroll
                    for (int i = 0; i < kGlsTile; i++) { vx[i] = ex[i * kGlsZStride + z]; vy[i] = ey[i * kGlsZStride + z]; }
#pragma unroll
                    for (int i = 0; i < kGlsTile; i++)
#pragma unroll
                        for (int j = 0; j < kGlsTile; j++) {
                            const float u = __fmul_rn(vx[i], vy[j]);
                            a1[i][j] = __fadd_rn(a1[i][j], u);
                            a2[i][j] = fmaf(u, u, a2[i][j]);
                        }
                }
            }
            if (t >= ntiles) continue;
#pragma unroll
            for (int i = 0; i < kGlsTile; i++)
#pragma unroll
                for (int j = 0; j < kGlsTile; j++) {
                    const int x = kGlsTile * bx + i, y = kGlsTile * by + j;
                    if (x < n1 && y <= x) {
                        f2 v = cf[tri(x, y)], sv = f2_two_sum(v.hi, a1[i][j]);
                        cf[tri(x, y)] = {sv.hi, __fadd_rn(v.lo, sv.lo)};
                        v = s2f[tri(x, y)];
                        sv = f2_two_sum(v.hi, a2[i][j]);
                        s2f[tri(x, y)] = {sv.hi, __fadd_rn(v.lo, sv.lo)};
                    }
                }
        }
    }
    __syncthreads();
    // covariance (java:9534-9542), S2 in FP64, standard deviations
    for (int i = tid; i < npairs; i += kGlsThreads) {
        const f2 v = cf[i], w = s2f[i];
        lp[i] = (f2d(v.hi) + f2d(v.lo)) * inv_pm1;
        s2[i] = f2d(w.hi) + f2d(w.lo);
    }
    __syncthreads();
    if (tid < n1) {
        const double c = lp[tri(tid, tid)];
        cdiag[tid] = c;
        isd[tid] = 1.0 / sqrt(c);
    }
    // where more than half of the variances are NaN no lag has the median's
    // rank: not what the CTA before left here
    if (tid == 0) s_med[0] = s_med[1] = 0.0;
    __syncthreads();
    // median of the chanum diagonal entries incl. the zero-lag slot that
    // stays 0 (java:9563-9573): rank selection, ties ordered by index
    if (tid <= n1) {
        // (variances order like their bits: no FP64 comparison; a NaN, above
        // all numbers here, compares with nothing and takes rank 0)
        const long long above = 0x7fffffffffffffffll;
        auto key_of = [&](int j) {
            const double w = j == 0 ? 0.0 : cdiag[j - 1];
            return w != w ? above : __double_as_longlong(w);
        };
        const double v = tid == 0 ? 0.0 : cdiag[tid - 1];
        const long long key = key_of(tid);
        int rank = 0;
        for (int j = 0; j <= n1; j++) {
            const long long w = key_of(j);
            rank += (w < key) || (w == key && j < tid);
        }
        if (key == above) rank = 0;
        const int c = n1 + 1;
        const int pos1 = (c - 1) / 2, pos2 = c / 2;     // floor / ceil of (c - 1) / 2
        if (rank == pos1) s_med[0] = v;
        if (rank == pos2) s_med[1] = v;
    }
    // t_xy and correlations; lamvar's and lamcov's sums
    const double f = s_f;
    const double pm2 = (double)(pnum - 2);
    for (int i = tid; i < npairs; i += kGlsThreads) {
        int x = (int)((sqrtf(8.f * i + 1.f) - 1.f) * 0.5f);
        while ((x + 1) * (x + 2) / 2 <= i) x++;
        while (x * (x + 1) / 2 > i) x--;
        const int y = i - x * (x + 1) / 2;
        const double c = lp[i];
        const double t = s2[i] - pm2 * c * c;        // sum_z (e_x e_y - c_xy)^2 terms
        if (x == y) {
            s2[i] = t;                               // lamvar numerator term
        } else {
            const double k = isd[x] * isd[y];
            s2[i] = t * k * k;                       // t_xy
            lp[i] = c * k;                           // correlation
        }
    }
    __syncthreads();
    if (tid == 0) {
        const double med = (s_med[0] + s_med[1]) * 0.5;
        s_med[0] = med;
    }
    {
        double num = 0.0, den = 0.0;
        if (tid < n1) num = s2[tri(tid, tid)] * f;
        __syncthreads();                              // the median's average
        if (tid < n1) {
            const double d = cdiag[tid] - s_med[0];
            den = d * d;
        }
        num = warp_sum_d(num);
        den = warp_sum_d(den);
        if (lane == 0) { red[0][warp] = num; red[1][warp] = den; }
        __syncthreads();
        if (tid == 0) {
            double a = 0.0, b = 0.0;
            for (int w = 0; w < kGlsThreads / 32; w++) { a += red[0][w]; b += red[1][w]; }
            s_lamvar = fmax(fmin(1.0, a / b), 0.0);
        }
        __syncthreads();
    }
    // lamcov: per x, T_y = (T_{y-1} + t_xy) f summed over y < x
    {
        double num = 0.0, den = 0.0;
        if (tid < n1) {
            const int x = tid;
            double T = 0.0;
            for (int y = 0; y < x; y++) {
                T = (T + s2[tri(x, y)]) * f;
                num += T;
                const double r = lp[tri(x, y)];
                den += r * r;
            }
        }
        num = warp_sum_d(num);
        den = warp_sum_d(den);
        if (lane == 0) { red[0][warp] = num; red[1][warp] = den; }
        __syncthreads();
        if (tid == 0) {
            double a = 0.0, b = 0.0;
            for (int w = 0; w < kGlsThreads / 32; w++) { a += red[0][w]; b += red[1][w]; }
            s_lamcov = fmax(fmin(1.0, a / b), 0.0);
        }
        __syncthreads();
    }
    // regularised covariance (java:9605-9615), FP64, packed lower triangle
    const double lv = s_lamvar, lc = s_lamcov, med = s_med[0];
    if (tid < n1) {
        const double d = lv * med + (1.0 - lv) * cdiag[tid];
        sq[tid] = sqrt(d);
        rdiag[tid] = d * inv_pnum;
    }
    __syncthreads();
    for (int i = tid; i < npairs; i += kGlsThreads) {
        int x = (int)((sqrtf(8.f * i + 1.f) - 1.f) * 0.5f);
        while ((x + 1) * (x + 2) / 2 <= i) x++;
        while (x * (x + 1) / 2 > i) x--;
        const int y = i - x * (x + 1) / 2;
        lp[i] = (x == y) ? rdiag[x] : (1.0 - lc) * lp[i] * sq[x] * sq[y] * inv_pnum;
    }
    __syncthreads();
    if (g.covmats_out) {
        for (int i = tid; i < n1 * n1; i += kGlsThreads) {
            const int x = i / n1, y = i - x * n1;
            g.covmats_out[(size_t)pix * n1 * n1 + i] = x >= y ? lp[tri(x, y)] : lp[tri(y, x)];
        }
        __syncthreads();              // every warp has copied its share before warp 0 factors lp in place
    }
    // Cholesky in panels of kPanel columns: warp 0 factors a panel in
    // registers, then all warps subtract its columns' products from the rest
    // (18 barriers instead of 216; a panel ahead, with the other warps at the
    // columns behind, was no faster: warp 0 is the critical path).  Every
    // element sees the pivots' updates A[q][p] -= A[q][i] A[p][i] in
    // commons-math's order (java:13717).
    for (int k0 = 0; k0 < n1; k0 += kPanel) {
        if (warp == 0 && !chol_panel(lp, n1, k0, rdiag, lane) && lane == 0) s_fail = 1;
        __syncthreads();
        if (s_fail) break;
        // 2 x 2 elements per thread, q >= p, both past the panel
        const int k1 = k0 + kPanel, half = n1 > k1 ? (n1 - k1 + 1) / 2 : 0;
        for (int e = tid; e < half * (half + 1) / 2; e += kGlsThreads) {
            int bq = (int)((sqrtf(8.f * e + 1.f) - 1.f) * 0.5f);
            while ((bq + 1) * (bq + 2) / 2 <= e) bq++;
            while (bq * (bq + 1) / 2 > e) bq--;
            const int q0 = k1 + 2 * bq, p0 = k1 + 2 * (e - bq * (bq + 1) / 2);
            const bool two_q = q0 + 1 < n1, upper = p0 + 1 <= q0;   // rows q0 + 1; element (q0, p0 + 1)
            const int rq0 = tri(q0, 0), rq1 = two_q ? tri(q0 + 1, 0) : rq0;
            const int rp0 = tri(p0, 0), rp1 = p0 + 1 < n1 ? tri(p0 + 1, 0) : rp0;
            double a00 = lp[rq0 + p0], a01 = upper ? lp[rq0 + p0 + 1] : 0.0;
            double a10 = lp[rq1 + p0], a11 = two_q ? lp[rq1 + p0 + 1] : 0.0;
#pragma unroll
            for (int i = 0; i < kPanel; i++) {
                const double x0 = lp[rq0 + k0 + i], x1 = lp[rq1 + k0 + i], y0 = lp[rp0 + k0 + i], y1 = lp[rp1 + k0 + i];
                a00 = fma(-x0, y0, a00);
                a01 = fma(-x0, y1, a01);
                a10 = fma(-x1, y0, a10);
                a11 = fma(-x1, y1, a11);
            }
            lp[rq0 + p0] = a00;
            if (upper) lp[rq0 + p0 + 1] = a01;
            if (two_q) {
                lp[rq1 + p0] = a10;
                lp[rq1 + p0 + 1] = a11;
            }
        }
        __syncthreads();
    }
    if (s_fail) {
        if (tid == 0) g.ok[pix] = 0;
        return;
    }
    // L and 1/diag(L) in float-float for the triangular inverse on the FP32
    // pipe (the output L^-1 is FP32), in the place of the FP64 factor
    f2 *L = cf, *X = s2f;
    for (int i = tid; i < npairs; i += kGlsThreads) L[i] = f2_from_d(lp[i]);
    if (tid < n1) rdf[tid] = f2_from_d(rdiag[tid]);
    __syncthreads();
    // L^-1, column c on lane c of a warp's 32 columns: X[c][c] = 1/L[c][c],
    // X[r][c] = -(sum_{m=c}^{r-1} L[r][m] X[m][c]) / L[r][r].  All lanes are at
    // the same (r, m) -- L is a broadcast, a row of X consecutive -- and take
    // zeros up to their column (with r starting at each lane's own column
    // both loads were spread over the banks, and bound the kernel).
    if (tid < ((n1 + 31) & ~31)) {
        const int c = tid, c0 = tid & ~31;
        for (int r = c0; r < n1; r++) {
            float sh = 0.f, sl = 0.f;
            const f2 *Lr = L + tri(r, 0), *Xc = X + tri(c0, 0) + c;
            int m = c0;
            for (; m < min(r, c0 + 32); m++) {          // the warp's own columns: zeros above the diagonal
                const f2 x = c <= m ? *Xc : f2{0.f, 0.f};
                Xc += m + 1;
                ff_dot_step(Lr[m].hi, Lr[m].lo, x.hi, x.lo, sh, sl);
            }
            for (; m + 8 <= r; m += 8) {
                f2 xv[8], lv[8];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    xv[u] = Xc[u * m + u * (u + 1) / 2];
                    lv[u] = Lr[m + u];
                }
                Xc += 8 * m + 36;
#pragma unroll
                for (int u = 0; u < 8; u++) ff_dot_step(lv[u].hi, lv[u].lo, xv[u].hi, xv[u].lo, sh, sl);
            }
            for (; m < r; m++) {
                const f2 x = *Xc;
                Xc += m + 1;
                ff_dot_step(Lr[m].hi, Lr[m].lo, x.hi, x.lo, sh, sl);
            }
            if (c < r) X[tri(r, c)] = f2_neg(f2_mul(f2_two_sum(sh, sl), rdf[r]));
            else if (c == r) X[tri(r, r)] = rdf[r];
            __syncwarp();
        }
    }
    __syncthreads();
    float *lo = g.linv + (size_t)pix * npairs;
    for (int i = tid; i < npairs; i += kGlsThreads) lo[i] = __fadd_rn(X[i].hi, X[i].lo);
    // transformed data L^-1 mcov
    if (tid < n1) {
        const f2 *Xr = X + tri(tid, 0);
        float sh = 0.f, sl = 0.f;
        for (int c = 0; c <= tid; c++) ff_dot_step(Xr[c].hi, Xr[c].lo, mcovf[c].hi, mcovf[c].lo, sh, sl);
        g.ytrans[(size_t)pix * n1 + tid] = sh + sl;
    }
    if (tid == 0) g.ok[pix] = 1;
}

size_t gls_smem_bytes(int chanum)
{
    const int n1 = chanum - 1;
    const size_t npairs = (size_t)n1 * (n1 + 1) / 2;
    const size_t rows = (size_t)((n1 + kGlsTile - 1) / kGlsTile) * kGlsTile;
    return 2 * npairs * sizeof(double) + rows * kGlsZStride * sizeof(float);
}

cudaError_t launch_gls(const GlsArgs &g, cudaStream_t stream)
{
    if (g.chanum - 1 > kMaxN1) return cudaErrorInvalidValue;
    size_t smem = gls_smem_bytes(g.chanum);
    cudaFuncSetAttribute(gls_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    gls_kernel<<<g.npix, kGlsThreads, smem, stream>>>(g);
    return cudaGetLastError();
}

}  // namespace imfcs
