// imfcs_fit.cu -- batched Levenberg-Marquardt fits, one warp per fit.
//
//   * FCS model (FCS_3p, java:13131-13408 / Gpufit ACF_1D, agpufitjni.cu:427-543)
//     weighted by 1/blocked variance over lags fitstart..fitend (standardFit,
//     java:10288-10471) or, for GLS, on the data and model transformed by
//     L^-1 of the regularised covariance (GLSFit, java:10622-10789).
//   * LINEAR_1D polynomial model (agpufitjni.cu:362-420).
//
// Lanes own fit points; J^T W J, J^T W r and chi^2 are warp reductions; the
// small K x K damped system is solved redundantly in every lane.  The grid is
// persistent: each warp strides over fits.  The solver stops on a small step
// (undamped Gauss-Newton step |h_i| <= 1e-7 |p_i| + 1e-5 sigma_i) once the
// residuals come from the FP64 model value, or when no step lowers chi^2 any
// more, or on the Gpufit criterion |dchi2| < tol max(1, chi2) when a
// tolerance is given through the reference fit API.
#include <math.h>

#include "imfcs_internal.cuh"
#include "imfcs_args.h"

namespace imfcs {

constexpr int kMaxPts = 160;

// lm_kernel (imfcs_lm.cuh): launchers in imfcs_lm{3,5,11}.cu
cudaError_t launch_lm_k3(const FitArgs &a, bool big, int blocks, int threads, size_t smem, cudaStream_t s);
cudaError_t launch_lm_k5(const FitArgs &a, bool big, int blocks, int threads, size_t smem, cudaStream_t s);
cudaError_t launch_lm_k11(const FitArgs &a, bool big, int blocks, int threads, size_t smem, cudaStream_t s);
// specialised kernel of the default fit (imfcs_lm_tirf.cu)
bool lm_tirf_applies(const FitArgs &a, bool tirf_zero_held);
// specialised kernels of the plain one- and two-component fits (imfcs_lm_comp.cu)
bool lm_comp_applies(const FitArgs &a);
cudaError_t launch_lm_comp(const FitArgs &a, cudaStream_t s);
cudaError_t launch_lm_tirf(const FitArgs &a, int blocks, int threads, cudaStream_t s);
cudaError_t launch_lm_gls(const FitArgs &a, cudaStream_t s);   // the same on whitened data (imfcs_lm_gls.cu)

size_t lm_smem_bytes(const FitArgs &a, int km, int warps)
{
    if (!a.linv) return 0;
    return (size_t)warps * ((size_t)a.npts * (a.npts + 1) / 2 + km * a.npts + 2 * a.npts + 2) * sizeof(float);
}

cudaError_t launch_lm(const FitArgs &a, int num_sms, cudaStream_t stream)
{
    if (a.nfits <= 0) return cudaSuccess;
    const bool big = a.npts > kMaxPts;
    if (big && a.linv) return cudaErrorInvalidValue;
    const int warps = 4;
    int km = a.k <= 3 ? 3 : (a.k <= 5 ? 5 : 11);
    size_t smem = lm_smem_bytes(a, km, warps);
    int blocks = (a.nfits + warps - 1) / warps;
    int cap = num_sms * 16;
    if (blocks > cap) blocks = cap;
    const bool tirf = lm_tirf_applies(a, a.tirf_zero_held != 0);
    if (lm_comp_applies(a)) return launch_lm_comp(a, stream);
    if (tirf && a.linv) return launch_lm_gls(a, stream);
    if (a.counter) {
        const cudaError_t e = cudaMemsetAsync(a.counter, 0, sizeof(int), stream);
        if (e != cudaSuccess) return e;
    }
    if (tirf) return launch_lm_tirf(a, blocks, warps * 32, stream);
    if (km == 3) return launch_lm_k3(a, big, blocks, warps * 32, smem, stream);
    if (km == 5) return launch_lm_k5(a, big, blocks, warps * 32, smem, stream);
    return launch_lm_k11(a, big, blocks, warps * 32, smem, stream);
}

// ---------------------------------------------------------------------------
// Pipeline glue: OLS data from the correlator outputs (double [pix][chanum])
// over lags fitstart..fitend, weights 1/var (java:10372).
// ---------------------------------------------------------------------------
__global__ void ols_prepare_kernel(int npix, int chanum, int fitstart, int npts, const double *acf,
                                   const double *var, float *y, float *w)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)npix * npts) return;
    size_t pix = i / npts;
    int p = (int)(i % npts);
    y[i] = (float)acf[pix * chanum + fitstart + p];
    w[i] = (float)(1.0 / var[pix * chanum + fitstart + p]);
}

// ---------------------------------------------------------------------------
// Fit epilogue (FP64, one thread per pixel): SI parameters, reduced chi^2 as
// the Java code reports it, the parameter covariance with commons-math's
// singularity threshold 1 (a singular covariance fails the fit exactly like
// the catch block of standardFit, java:10412, 10441), and the Bayes terms
// (java:10171-10207).
//
// A few hundred dependent FP64 operations per thread and nothing to overlap them
// with, on every call's critical path: the parameter count is a template
// argument (K = 3, 5; 0: at run time), so that matrices stay in registers
// (30 -> 19 us), and the Bayes residuals, 72 model values a pixel, are a kernel
// of their own with a warp per pixel (105 -> 41 us at 1,600 pixels, K = 3; 168 ->
// 87, K = 5).
// ---------------------------------------------------------------------------

template <int K>
__device__ __forceinline__ double det_lu(const double *ain, int n_)
{
    const int n = K ? K : n_;
    // determinant by LU with partial pivoting (equal, up to rounding, to the
    // cofactor expansion of java:14752-14770)
    constexpr int M = K ? K : IMFCS_NPARAM;
    double a[M * M];
#pragma unroll
    for (int i = 0; i < n * n; i++) a[i] = ain[i];
    double det = 1.0;
#pragma unroll
    for (int c = 0; c < n; c++) {
        int p = c;
        double top = fabs(a[c * n + c]);
#pragma unroll
        for (int r = c + 1; r < n; r++)
            if (fabs(a[r * n + c]) > top) { p = r; top = fabs(a[r * n + c]); }
        double piv = a[c * n + c];
#pragma unroll
        for (int r = c + 1; r < n; r++)
            if (r == p) piv = a[r * n + c];
        if (piv == 0.0) return 0.0;
#pragma unroll
        for (int r = c + 1; r < n; r++)
            if (r == p) {
#pragma unroll
                for (int q = 0; q < n; q++) { double t = a[c * n + q]; a[c * n + q] = a[r * n + q]; a[r * n + q] = t; }
            }
        if (p != c) det = -det;
        det *= a[c * n + c];
#pragma unroll
        for (int r = c + 1; r < n; r++) {
            double f = a[r * n + c] / a[c * n + c];
#pragma unroll
            for (int q = c; q < n; q++) a[r * n + q] -= f * a[c * n + q];
        }
    }
    return det;
}

// Householder QR inverse with |R_ii| <= threshold -> singular.
template <int K>
__device__ __forceinline__ bool qr_inverse_d(const double *ain, int k_, double threshold, double *inv)
{
    constexpr int M = K ? K : IMFCS_NPARAM;
    const int k = K ? K : k_;
    double a[M * M], rdiag[M];
#pragma unroll
    for (int i = 0; i < k * k; i++) a[i] = ain[i];
#pragma unroll
    for (int minor = 0; minor < k; minor++) {
        double xn = 0.0;
#pragma unroll
        for (int r = minor; r < k; r++) xn += a[r * k + minor] * a[r * k + minor];
        double alpha = a[minor * k + minor] > 0 ? -sqrt(xn) : sqrt(xn);
        rdiag[minor] = alpha;
        if (alpha != 0.0) {
            a[minor * k + minor] -= alpha;
#pragma unroll
            for (int c = minor + 1; c < k; c++) {
                double ac = 0.0;
#pragma unroll
                for (int r = minor; r < k; r++) ac -= a[r * k + c] * a[r * k + minor];
                ac /= alpha * a[minor * k + minor];
#pragma unroll
                for (int r = minor; r < k; r++) a[r * k + c] -= ac * a[r * k + minor];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < k; i++)
        if (!(fabs(rdiag[i]) > threshold)) return false;
#pragma unroll
    for (int col = 0; col < k; col++) {
        double y[M];
#pragma unroll
        for (int i = 0; i < k; i++) y[i] = (i == col) ? 1.0 : 0.0;
#pragma unroll
        for (int minor = 0; minor < k; minor++) {
            double dot = 0.0;
#pragma unroll
            for (int r = minor; r < k; r++) dot += y[r] * a[r * k + minor];
            dot /= rdiag[minor] * a[minor * k + minor];
#pragma unroll
            for (int r = minor; r < k; r++) y[r] += dot * a[r * k + minor];
        }
#pragma unroll
        for (int i = k - 1; i >= 0; i--) {
            y[i] /= rdiag[i];
#pragma unroll
            for (int r = 0; r < i; r++) y[r] -= y[i] * a[r * k + i];
        }
#pragma unroll
        for (int i = 0; i < k; i++) inv[i * k + col] = y[i];
    }
    return true;
}

// Bayes: log-residual term of every converged pixel (left in logp), a warp per
// pixel; the sums in the order of one thread.
constexpr int kResWarps = 4;
__global__ void __launch_bounds__(32 * kResWarps) bayes_residual_kernel(EpilogueArgs e)
{
    __shared__ double tres_sh[kResWarps][kMaxChan], z_sh[kResWarps][kMaxChan];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int pix = blockIdx.x * kResWarps + wid;
    if (pix >= e.npix) return;
    // a failed fit has no residuals, a failed factorisation no L^-1
    if (e.state[pix] != IMFCS_STATE_CONVERGED || (e.pre_ok && !e.pre_ok[pix])) return;
    double *tres = tres_sh[wid], *z = z_sh[wid];
    float par[IMFCS_NPARAM];
#pragma unroll
    for (int i = 0; i < IMFCS_NPARAM; i++) par[i] = e.par_int[(size_t)pix * IMFCS_NPARAM + i];
    const bool c2 = par[5] != 0.f, c3 = par[7] != 0.f;
    // unweighted residuals of the fitted lags (tres)
    for (int i = 1 + lane; i < e.chanum; i += 32) {
        const bool in = e.gls || (i >= e.fitstart && i <= e.fitend);
        const double v = in ? (double)fcs_model_f(par, e.mc, e.lagtime[i], nullptr, c2, c3) : 0.0;
        tres[i - 1] = in ? e.acf[(size_t)pix * e.chanum + i] - v : 0.0;
    }
    __syncwarp();
    double sum = 0.0;
    if (!e.gls) {
        if (lane == 0)
            for (int i = 1; i < e.chanum - 1; i++) sum += tres[i] * tres[i];   // from index 1 (java:10170)
    } else {
        // tres^T covmats^-1 tres = |L^-1 tres|^2
        const int n = e.chanum - 1;
        const float *L = e.linv + (size_t)pix * n * (n + 1) / 2;
        for (int i = lane; i < n; i += 32) {
            const float *row = L + (size_t)i * (i + 1) / 2;
            double zi = 0.0;
            for (int c = 0; c <= i; c++) zi += (double)row[c] * tres[c];
            z[i] = zi;
        }
        __syncwarp();
        if (lane == 0)
            for (int i = 0; i < n; i++) sum += z[i] * z[i];
    }
    if (lane == 0) e.logp[pix] = -0.5 * sum;
}

template <int K>
__global__ void fit_epilogue_kernel(EpilogueArgs e)
{
    constexpr int M = K ? K : IMFCS_NPARAM;
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= e.npix) return;
    const float *pi = e.par_int + (size_t)pix * IMFCS_NPARAM;
    int st = e.state[pix];
    bool ok = (st == IMFCS_STATE_CONVERGED) && (!e.pre_ok || e.pre_ok[pix]);
    double cov[M * M], jtj[M * M];
    const int k = K ? K : e.k;
#pragma unroll
    for (int aa = 0; aa < k; aa++)
#pragma unroll
        for (int bb = 0; bb < k; bb++)
            jtj[aa * k + bb] = (double)e.hess[(size_t)pix * k * k + aa * k + bb] /
                               (param_unit(e.idx[aa]) * param_unit(e.idx[bb]));
    if (ok) ok = qr_inverse_d<K>(jtj, k, 1.0, cov);
#pragma unroll
    for (int i = 0; i < k; i++) ok = ok && isfinite(cov[i * k + i]) && cov[i * k + i] > 0.0;
    float *fr = e.fitres + (size_t)pix * IMFCS_NPARAM;
#pragma unroll
    for (int i = 0; i < IMFCS_NPARAM; i++) {
        bool is_free = false;
#pragma unroll
        for (int q = 0; q < k; q++) is_free |= (e.idx[q] == i);
        fr[i] = (ok || !is_free) ? (float)((double)pi[i] * param_unit(i)) : nanf("");
    }
    if (e.chi2) e.chi2[pix] = ok ? (float)((double)e.chi2_raw[pix] / e.chi2_div) : nanf("");
    if (e.fitted) e.fitted[pix] = ok ? 1 : 0;
    if (e.logp) {
        // Bayes model-probability exponent (java:10171-10207):
        //   0.5 k ln(2 pi) + 0.5 ln det(cov) + logresid - ln(prod sigma * (2*200)^k)
        const double pi_j = 3.14159265359;
        double logresid, det, prodsig = 1.0;
        if (ok) {
            logresid = e.logp[pix];                   // bayes_residual_kernel
            det = det_lu<K>(cov, k);
#pragma unroll
            for (int i = 0; i < k; i++) prodsig *= sqrt(cov[i * k + i]);
        } else {
            // failed fit: ones (java:10441-10466) -> det of the all-ones matrix
            logresid = 0.0;
            for (int i = 1; i < e.chanum - 1; i++) logresid += 1.0;
            logresid *= -0.5;
            det = (k == 1) ? 1.0 : 0.0;
            prodsig = 1.0;
        }
        e.logp[pix] = 0.5 * k * log(2 * pi_j) + 0.5 * log(det) + logresid - log(prodsig * pow(400.0, k));
    }
}

__global__ void bayes_combine_kernel(int npix, const double *lp1, const double *lp2, float *prob)
{
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= npix) return;
    double m1 = exp(lp1[pix]), m2 = exp(lp2[pix]);
    double nrm = m1 + m2;
    prob[2 * pix] = (float)(m1 / nrm);
    prob[2 * pix + 1] = (float)(m2 / nrm);
}

cudaError_t launch_fit_epilogue(const EpilogueArgs &e, cudaStream_t stream)
{
    if (e.logp) bayes_residual_kernel<<<(e.npix + kResWarps - 1) / kResWarps, 32 * kResWarps, 0, stream>>>(e);
    const int blocks = (e.npix + 63) / 64;
    if (e.k == 3) fit_epilogue_kernel<3><<<blocks, 64, 0, stream>>>(e);
    else if (e.k == 5) fit_epilogue_kernel<5><<<blocks, 64, 0, stream>>>(e);
    else fit_epilogue_kernel<0><<<blocks, 64, 0, stream>>>(e);
    return cudaGetLastError();
}
cudaError_t launch_ols_prepare(int npix, int chanum, int fitstart, int npts, const double *acf,
                               const double *var, float *y, float *w, cudaStream_t stream)
{
    size_t n = (size_t)npix * npts;
    ols_prepare_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(npix, chanum, fitstart, npts, acf, var, y, w);
    return cudaGetLastError();
}
cudaError_t launch_bayes_combine(int npix, const double *lp1, const double *lp2, float *prob,
                                 cudaStream_t stream)
{
    bayes_combine_kernel<<<(npix + 127) / 128, 128, 0, stream>>>(npix, lp1, lp2, prob);
    return cudaGetLastError();
}

}  // namespace imfcs
