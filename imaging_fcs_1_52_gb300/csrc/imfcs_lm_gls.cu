// imfcs_lm_gls.cu -- the LM fit of the plugin's default model (one component,
// no flow, no triplet, N, D and G free; window offsets: OFF) on the data and
// model whitened by L^-1 of the regularised covariance (GLSFit,
// java:10622-10789), up to 96 points.  The model enters through u = L^-1 a and
// v = L^-1 da/dD of its N-free part a: L^-1 f = u / N + G L^-1 1, so an
// evaluation is triangular products per warp (L^-1 in shared memory), and the
// precise residuals transform the FP64 values of a.  Algorithm, stopping rules
// and operation order are those of lm_tirf_kernel.
//
// The evaluations are drawn to one place, driven by a state machine, so that
// the code stays near the instruction caches, and chi^2 comes first: a rejected
// step (about half of them) ends there, on the FP64 model without the FP32
// model and its products.  Bound by FP64 issue where fits end in many FP64
// steps (weak correlations), else by latency.  4,096 fits of 72 points: 0.67
// ms with one row of a lane at a time, 0.54 with three side by side, 0.40 in
// this form; 9,120 with an offset 5.47 -> 4.6 ms.  (The same machine gave the
// OLS fits nothing: they take few steps and no products.)
#include "imfcs_tirf.cuh"

namespace imfcs {

// Per-warp shared memory of a GLS fit: L^-1 (packed lower, float), its row
// sums (L^-1 1, float and FP64), and the staged N-free model part a, da/dD
// (FP32) and a (FP64) of the points.
struct GlsSh {
    float *L, *l1, *sa, *sda;
    double *sfd, *l1d;
};
constexpr int kGlsRows = 3;           // rows of a lane: at most 96 points

// Rows lane, lane + 32, lane + 64 of the whitened model, side by side: a
// column's values are read once for all of them, and three chains of products
// run at a time.  PREC = false: u = (L^-1 a)_r, v = (L^-1 da/dD)_r; true:
// U = (L^-1 a)_r in FP64 (float-float for U was 10 % faster but sent weakly
// determined fits along other LM steps).
template <bool PREC>
__device__ __forceinline__ void gls_rows(const GlsSh &g, int n, int lane, float (&u)[kGlsRows], float (&v)[kGlsRows],
                                         double (&U)[kGlsRows])
{
    const float *L[kGlsRows];
    int r[kGlsRows];
#pragma unroll
    for (int m = 0; m < kGlsRows; m++) {
        r[m] = lane + 32 * m < n ? lane + 32 * m : -1;
        L[m] = g.L + (r[m] >= 0 ? r[m] * (r[m] + 1) / 2 : 0);
        if (PREC) U[m] = 0.0;
        else u[m] = v[m] = 0.f;
    }
    // columns 32 p .. 32 p + 31 reach the lane's rows p and up
#pragma unroll
    for (int p = 0; p < kGlsRows; p++)
#pragma unroll 4
        for (int k = 32 * p; k < min(32 * (p + 1), n); k++) {
            const float a = PREC ? 0.f : g.sa[k], da = PREC ? 0.f : g.sda[k];
            const double ad = PREC ? g.sfd[k] : 0.0;
#pragma unroll
            for (int m = p; m < kGlsRows; m++)
                if (k <= r[m]) {
                    const float l = L[m][k];
                    if (PREC) {
                        U[m] = fma(f2d(l), ad, U[m]);
                    } else {
                        u[m] = fmaf(l, a, u[m]);
                        v[m] = fmaf(l, da, v[m]);
                    }
                }
        }
}

// Floats of shared memory of a GLS fit with n points: L^-1, l1, a, da/dD,
// then (8-byte aligned) a in FP64 and l1 in FP64.
__host__ __device__ __forceinline__ int gls_warp_floats(int n)
{
    return ((n * (n + 1) / 2 + 3 * n + 1) & ~1) + 4 * n;
}

constexpr int kGlsSums = 9;

struct GlsFitSh {
    float x[32 * kGlsRows], r[32 * kGlsRows];
    float s[2][kGlsSums];             // lower triangle of J^T J by rows, then J^T r: the fit's, a probe's
    float H[9];
};

__device__ __forceinline__ float gls_sig(const float *s, int i)
{
    return rsqrtf(fmaxf(s[i * (i + 3) / 2], 1e-30f));
}

// One warp, one block per fit.
template <bool OFF>
__global__ void __launch_bounds__(32, 16) lm_gls_kernel(FitArgs a)
{
    extern __shared__ __align__(16) float tsh[];   // holds FP64 arrays too
    __shared__ GlsFitSh sh;
    const int lane = threadIdx.x;
    const int n = a.npts;
    const TirfC c = tirf_consts(a.mc);
    for (int i = lane; i < n; i += 32) sh.x[i] = __ldg(&a.x[i]);
    const int npairs = n * (n + 1) / 2;
    GlsSh g;
    g.L = tsh;
    g.l1 = g.L + npairs;
    g.sa = g.l1 + n;
    g.sda = g.sa + n;
    g.sfd = (double *)(tsh + ((npairs + 3 * n + 1) & ~1));
    g.l1d = g.sfd + n;
    for (int fit = blockIdx.x; fit < a.nfits; fit += gridDim.x) {
        if (a.todo && !__ldg(&a.todo[fit])) continue;
        // this fit's L^-1 and its row sums (the whitened constant G)
        const float *src = a.linv + (size_t)fit * npairs;
        for (int i = lane; i < npairs; i += 32) g.L[i] = __ldg(&src[i]);
        __syncwarp();
        for (int r = lane; r < n; r += 32) {
            const float *Lr = g.L + r * (r + 1) / 2;
            float s1 = 0.f;
            double s1d = 0.0;
#pragma unroll 4
            for (int k = 0; k <= r; k++) { s1 += Lr[k]; s1d += f2d(Lr[k]); }
            g.l1[r] = s1;
            g.l1d[r] = s1d;
        }
        float yl[kGlsRows];
#pragma unroll
        for (int m = 0; m < kGlsRows; m++) {
            const int i = lane + 32 * m;
            yl[m] = i < n ? __ldg(&a.y[(size_t)fit * n + i]) : 0.f;
        }
        __syncwarp();
        const float *ip = a.init + (size_t)fit * a.init_stride;
        // free parameters N, D, G (vector indices 0, 1, 4): FP32 in the FP32
        // phases, FP64 from the FP64-residual Newton steps on; pe, pde: the
        // ones to evaluate
        float pf[3] = {__ldg(&ip[0]), __ldg(&ip[1]), __ldg(&ip[4])}, pe[3] = {pf[0], pf[1], pf[2]};
        double pd[3] = {0.0, 0.0, 0.0}, pde[3] = {0.0, 0.0, 0.0};
        bool precise = false;     // parameters and chi^2 held in FP64
        bool retried = false;     // Newton left its region once: FP32 LM to 1e-4 sigma, then Newton again
        bool fresh = true;
        int state = IMFCS_STATE_MAX_ITERATIONS, it = 0, nprec = 0, ni = 0, col = 0;
        float lambda = 1e-3f, de = 0.f, schif = 0.f;
        double schi = 0.0;
        // what the evaluation under way is for
        enum { INIT, TRIAL, HESSIAN, NEWTON32, NEWTON64, RESTART } mode = INIT;
        for (;;) {
            // --- chi^2 at pe (precise: pde), and the sums unless a rejected
            // step.  FP32: no FP64 operation (GB300 issues FP64 at 1/64 of the
            // FP32 rate, and the FP32 phases evaluate the model some twenty
            // times per fit).  Precise: residuals of the whitened model in
            // FP64, the Jacobian in FP32.
            const float N = pe[0], D = pe[1], G = pe[2], iN = 1.f / N;
            double chi2;
            float chi2f;
            bool take;
            float acc[kGlsSums];
#pragma unroll
            for (int i = 0; i < kGlsSums; i++) acc[i] = 0.f;
            if (precise) {
                const double inv_Nd = 1.0 / pde[0];
#pragma unroll 1
                for (int i = lane; i < n; i += 32) {
                    f2 lat;
                    g.sfd[i] = (!OFF && tirf_a_ff(f2_from_d(pde[1]), c, sh.x[i], lat))
                                   ? (double)lat.hi + (double)lat.lo
                                   : tirf_a_d<OFF>(pde[1], c, (double)sh.x[i]);
                }
                __syncwarp();
                float u[kGlsRows], v[kGlsRows];
                double U[kGlsRows], c2 = 0.0;
                gls_rows<true>(g, n, lane, u, v, U);
#pragma unroll
                for (int m = 0; m < kGlsRows; m++) {
                    const int r = lane + 32 * m;
                    if (r < n) {
                        const double rr = (double)yl[m] - fma(U[m], inv_Nd, pde[2] * g.l1d[r]);
                        c2 = fma(rr, rr, c2);
                        sh.r[r] = (float)rr;
                    }
                }
                chi2 = warp_sum_d(c2);
                chi2f = (float)chi2;
                take = mode != TRIAL || (isfinite(chi2) && chi2 < schi);
            }
            if (!precise || take) {
                float gN[kGlsRows], gD[kGlsRows], r[kGlsRows];
#pragma unroll 1
                for (int i = lane; i < n; i += 32) {
                    float av, da;
                    tirf_terms<OFF>(D, c, sh.x[i], av, da);
                    g.sa[i] = av;
                    g.sda[i] = da;
                }
                __syncwarp();
                float u[kGlsRows], v[kGlsRows];
                double U[kGlsRows];
                gls_rows<false>(g, n, lane, u, v, U);
#pragma unroll
                for (int m = 0; m < kGlsRows; m++) {
                    const int i = lane + 32 * m;
                    gN[m] = -u[m] * iN * iN;
                    gD[m] = iN * v[m];
                    r[m] = i < n ? yl[m] - (__fmul_rn(u[m], iN) + G * g.l1[min(i, n - 1)]) : 0.f;
                }
                if (!precise) {
                    float c2f = 0.f;
#pragma unroll
                    for (int m = 0; m < kGlsRows; m++)
                        if (lane + 32 * m < n) c2f = fmaf(r[m], r[m], c2f);
                    chi2f = warp_sum(c2f);
                    chi2 = (double)chi2f;
                    take = mode != TRIAL || (isfinite(chi2f) && chi2f < schif);
                }
                if (take) {
#pragma unroll
                    for (int m = 0; m < kGlsRows; m++) {
                        const int i = lane + 32 * m;
                        if (i < n) {
                            const float gr[3] = {gN[m], gD[m], g.l1[i]};
                            const float rm = precise ? sh.r[i] : r[m];
                            int q = 0;
#pragma unroll
                            for (int p = 0; p < 3; p++)
#pragma unroll
                                for (int t = 0; t <= p; t++) acc[q++] += gr[p] * gr[t];
#pragma unroll
                            for (int p = 0; p < 3; p++) acc[q++] += gr[p] * rm;
                        }
                    }
                    int pos;
                    const float sum = warp_sums<kGlsSums, 16>(acc, lane, pos);
                    if (pos >= 0) sh.s[mode == HESSIAN][pos] = sum;
                    __syncwarp();
                }
            }

            bool newton = false, evald = false, to_precise = false, done = false;
            if (mode == TRIAL) {
                if (precise) nprec++;
                if (take) {
                    schi = chi2;
                    schif = chi2f;
                    fresh = true;
#pragma unroll
                    for (int i = 0; i < 3; i++) { pf[i] = pe[i]; pd[i] = pde[i]; }
                    lambda = fmaxf(lambda * 0.1f, 1e-9f);
                } else {
                    lambda *= 10.f;
                    if (lambda > (precise ? 1e10f : 1e6f)) {
                        if (precise) { state = IMFCS_STATE_CONVERGED; done = true; }
                        else to_precise = true;
                    }
                }
                if (nprec > 60) { state = IMFCS_STATE_CONVERGED; done = true; }
                if (!to_precise) it++;
            } else if (mode == HESSIAN) {
                // column `col` of the Newton finish's Hessian of chi^2/2, from
                // forward differences of the FP32 gradient (see lm_kernel)
                if (lane < 3) sh.H[lane * 3 + col] = (sh.s[0][6 + lane] - sh.s[1][6 + lane]) / de;
                __syncwarp();
                if (++col < 3) {
                    to_precise = true;
                } else {
                    float v = 0.f;
                    const int r = lane / 3, q = lane % 3;
                    if (lane < 9 && q < r) v = 0.5f * (sh.H[r * 3 + q] + sh.H[q * 3 + r]);
                    __syncwarp();
                    if (lane < 9 && q < r) { sh.H[r * 3 + q] = v; sh.H[q * 3 + r] = v; }
                    __syncwarp();
                    newton = true;
                }
            } else {
                schi = chi2;
                schif = chi2f;
                if (mode == INIT) {
                    if (!isfinite(chi2f)) { state = IMFCS_STATE_SINGULAR_HESSIAN; done = true; }
                } else if (mode == NEWTON32) {
                    ni++;
                    newton = true;
                } else if (mode == NEWTON64) {
                    newton = evald = true;
                } else {             // RESTART
                    lambda = 1e-3f;
                    fresh = true;
                    it++;
                }
            }
            if (done) break;

            // --- next LM step: the stopping test on the undamped step (once:
            // it stays what it is after a rejected step), then the damped one
            while (!newton && !to_precise) {
                if (it >= a.max_iter) { done = true; break; }
                float A[9], gv[3], h[3];
                {
                    int q = 0;
#pragma unroll
                    for (int i = 0; i < 3; i++)
#pragma unroll
                        for (int t = 0; t <= i; t++) { A[i * 3 + t] = A[t * 3 + i] = sh.s[0][q]; q++; }
#pragma unroll
                    for (int i = 0; i < 3; i++) gv[i] = sh.s[0][q++];
                }
                // the undamped solve in the warp's lower half beside the damped
                // one in the upper: a solve is one long chain
                const bool test = fresh;
                float hs[3];
                const bool oks = tirf_solve(A, gv, test && lane < 16 ? 0.f : lambda, hs);
                const unsigned votes = __ballot_sync(0xffffffffu, oks);
                const bool ok = votes >> 16 & 1;
#pragma unroll
                for (int i = 0; i < 3; i++) h[i] = __shfl_sync(0xffffffffu, hs[i], 16);
                if (test && (votes & 1)) {
                    bool conv = true;
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const float sig = gls_sig(sh.s[0], i);
                        const float tol = precise ? 1e-7f * fabsf(pf[i]) + 1e-5f * sig
                                                  : (retried ? 1e-4f : 1e-3f) * sig;
                        const float hg = __shfl_sync(0xffffffffu, hs[i], 0);
                        conv = conv && (fabsf(hg) <= tol);
                    }
                    if (conv) {
                        if (precise) { state = IMFCS_STATE_CONVERGED; done = true; }
                        else to_precise = true;
                    }
                }
                if (done || to_precise) break;
                fresh = false;
                if (!ok) {
                    lambda *= 10.f;
                    if (lambda > 1e15f) { state = IMFCS_STATE_SINGULAR_HESSIAN; done = true; break; }
                    it++;
                    continue;
                }
                mode = TRIAL;
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    if (precise) {
                        pde[i] = pd[i] + (double)h[i];
                        pe[i] = (float)pde[i];
                    } else {
                        pe[i] = pf[i] + h[i];
                    }
                }
                break;
            }
            if (done) break;

            if (to_precise) {
                if (mode != HESSIAN) col = 0;
                mode = HESSIAN;
                const float eps = 0.1f * gls_sig(sh.s[0], col);
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    pe[i] = pf[i];
                    if (i == col) {
                        pe[i] = pf[i] + eps;
                        de = pe[i] - pf[i];
                    }
                }
            } else if (newton) {
                // Newton steps: up to 3 on the FP32 gradient to its stationary
                // point, then on that of the FP64 residuals until the step is
                // below 1e-4 sigma + 1e-7 |p|
                if (mode == HESSIAN) ni = 0;
                bool left = false;
#pragma unroll 1
                for (;;) {
                    if (ni >= 7) { left = true; break; }
                    const bool fp64 = ni >= 3;
                    if (fp64 && !evald) {
                        if (!precise) {
#pragma unroll
                            for (int i = 0; i < 3; i++) pd[i] = (double)pf[i];
                            precise = true;
                        }
                        mode = NEWTON64;
                        break;
                    }
                    if (fp64 && !isfinite(schi)) { left = true; break; }
                    evald = false;
                    float H[9], gv[3], hn[3];
#pragma unroll
                    for (int i = 0; i < 9; i++) H[i] = sh.H[i];
#pragma unroll
                    for (int i = 0; i < 3; i++) gv[i] = sh.s[0][6 + i];
                    if (!tirf_solve(H, gv, 0.f, hn)) { left = true; break; }
                    bool small = true;
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const float sig = gls_sig(sh.s[0], i);
                        if (!(fabsf(hn[i]) <= 0.05f * sig)) left = true;
                        small = small && (fabsf(hn[i]) <= 1e-4f * sig + (fp64 ? 1e-7f * fabsf(pf[i]) : 0.f));
                    }
                    if (left) break;
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        if (fp64) {
                            pd[i] += (double)hn[i];
                            pf[i] = (float)pd[i];
                        } else {
                            pf[i] += hn[i];
                        }
                    }
                    if (fp64 && small) { state = IMFCS_STATE_CONVERGED; it++; done = true; break; }
                    if (!fp64) {
                        if (!small) { mode = NEWTON32; break; }
                        ni = 2;
                    }
                    ni++;
                }
                if (done) break;
                if (left) {
                    mode = RESTART;
                    if (!retried) {
                        // Newton left its quadratic region (a step above 0.05
                        // sigma) or met an indefinite Hessian: back to FP32 LM,
                        // to the tighter 1e-4 sigma, and Newton from there -- an
                        // LM on FP64-residual evaluations costs ~10x an FP32
                        // iteration and runs for tens of iterations, and the few
                        // fits that take it set the duration of the whole launch
                        retried = true;
                        precise = false;
                    } else if (!precise) {
                        // LM on the FP64-residual model
#pragma unroll
                        for (int i = 0; i < 3; i++) pd[i] = (double)pf[i];
                        precise = true;
                    }
                }
#pragma unroll
                for (int i = 0; i < 3; i++) { pde[i] = pd[i]; pe[i] = pf[i]; }
            }
        }
        if (lane == 0) {
            float *o = a.out_par + (size_t)fit * a.out_stride;
            for (int i = 0; i < a.np; i++) o[i] = __ldg(&ip[i]);
            o[0] = precise ? (float)pd[0] : pf[0];
            o[1] = precise ? (float)pd[1] : pf[1];
            o[4] = precise ? (float)pd[2] : pf[2];
            if (a.out_chi2) a.out_chi2[fit] = schif;
            if (a.out_state) a.out_state[fit] = state;
            if (a.out_iter) a.out_iter[fit] = it;
            if (a.out_hess)
                for (int i = 0; i < 9; i++) {
                    const int r = max(i / 3, i % 3), q = min(i / 3, i % 3);
                    a.out_hess[(size_t)fit * 9 + i] = sh.s[0][r * (r + 1) / 2 + q];
                }
        }
        __syncwarp();
    }
}

// One fit per block, handed out by the hardware as fits end.
cudaError_t launch_lm_gls(const FitArgs &a, cudaStream_t s)
{
    const int blocks = a.nfits < (1 << 20) ? a.nfits : 1 << 20;
    const size_t smem = (size_t)gls_warp_floats(a.npts) * sizeof(float);
    auto kern = a.mc.rx != 0.f || a.mc.ry != 0.f ? lm_gls_kernel<true> : lm_gls_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<blocks, 32, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace imfcs
