// imfcs_lm_comp.cu -- LM fits of the plain one- and two-component models,
// specialised: FCS_3p (java:13131-13408) without flow, triplet, third
// component or window offset, OLS, up to 96 points.  Two uses:
//   K = 5  N, D, G, F2, D2 free, shared constants, step-mode stopping rule:
//          the second model of the plugin's Bayes comparison (bayesFit,
//          java:10191-10220);
//   K = 3  N, D, G free, constants of each fit, Gpufit's stopping rule: the
//          plugin's call of Gpufit (agpufitjni.cu:2289-2320, 2458-2487).
// Same algorithm, stopping rules and operation order as lm_kernel
// (imfcs_lm.cuh), which gives the same bits.
//
// The Bayes fits take some 80 accepted and 80 rejected FP32 steps and 45
// steps on the FP64 model each (a few take 900), one warp per fit, so a
// warp's time is its instruction count times a latency of about ten cycles, and the
// longest fits set the launch's.  Against lm_kernel:
//   - one evaluation site, driven by a state machine, and loops over the
//     components instead of copies: the code stays near the instruction
//     caches (a third of the stalls were instruction fetches);
//   - parameters in registers, the normal matrix in shared memory;
//   - chi^2 first: a rejected step ends there, without the sums of the
//     normal equations and, on the FP64 model, without the gradient;
//   - the undamped step behind the stopping test is not solved again after a
//     rejected step, and beside the damped one where it is (5.15 -> 4.87 ms);
//   - the sums over the warp as one transposed reduction (same tree);
//   - FP64 model values two lanes a point, one component each: 5 rounds for
//     72 points, not 6.
// 1,600 fits of 72 points, K = 5: 14.2 -> 4.9 ms, then bound by the FP64 pipe
// (60 % busy) and the longest fits.  16,384 fits, K = 3: 3.05 -> 1.09 ms.
#include "imfcs_lm.cuh"

namespace imfcs {

constexpr int kCompPts = 96;
constexpr int kSide = kCompPts / 32;   // points of a lane, evaluated side by side

template <int K>
struct CompSh {
    static constexpr int NC = (K - 1) / 2;               // components
    static constexpr int NS = K * (K + 1) / 2 + K;       // sums of the normal equations
    double a[NC * kCompPts];   // FP64 component terms [point][component]
    double x[kCompPts];
    float s[2][NS];            // lower triangle of J^T W J by rows, then J^T W r: the fit's, a probe's
    float H[K * K];
};

// lat x axial factor of one component and its derivative (component_f).
__device__ __forceinline__ void plain_component_f(float d, const ModelConst &c, bool square, float tau, float &a,
                                                float &da)
{
    const float p0 = sqrtf(fmaf(4.f * d, tau, c.s * c.s));
    const float inv_p0 = 1.f / p0;
    float Lx, Ly, dLx, dLy, dv;
    lateral_1d_f(c.ax, 0.f, 0.f, tau, p0, inv_p0, Lx, dLx, dv);
    if (square) { Ly = Lx; dLy = dLx; }
    else lateral_1d_f(c.ay, 0.f, 0.f, tau, p0, inv_p0, Ly, dLy, dv);
    const float cross = fmaf(dLx, Ly, __fmul_rn(Lx, dLy));   // as component_f is rounded
    const float dp0 = 2.f * tau * inv_p0;
    const float lat = Lx * Ly * c.inv_norm;
    const float dlat = cross * dp0 * c.inv_norm;
    const float inv_sz2 = 1.f / (c.sz * c.sz);
    const float psp = rsqrtf(fmaf(4.f * d * tau, inv_sz2, 1.f));
    const float dpsp = -2.f * tau * inv_sz2 * psp * psp * psp;
    a = lat * psp;
    da = dlat * psp + lat * dpsp;
}

// Values and gradients (d/dN, D, G[, F2, D2]) of the lane's points.  `one` is
// 1.f, a run-time value: products with it stay where the general model
// multiplies by the triplet factor, and round as they do there.
template <int K>
__device__ __forceinline__ void plain_model_f(const float (&p)[K], const ModelConst &c, bool square, float one,
                                              const float (&x)[kSide], float (&f)[kSide], float (&g)[kSide][K])
{
    const float N = p[0], G = p[2];
    const float iN = 1.f / N;
    if constexpr (K == 3) {
#pragma unroll
        for (int m = 0; m < kSide; m++) {
            float a, d;
            plain_component_f(p[1], c, square, x[m], a, d);
            g[m][0] = -a * one * iN * iN;
            g[m][1] = iN * d;
            g[m][2] = one;
            f[m] = __fmul_rn(a, iN) + G;
        }
    } else {
        const float F2 = p[3];
        float a1[kSide], a2[kSide], d1[kSide], d2[kSide];
#pragma unroll
        for (int m = 0; m < kSide; m++) a2[m] = d2[m] = 0.f;
#pragma unroll 1
        for (int q = 0; q < 2; q++) {
            const float D = q ? p[4] : p[1];
#pragma unroll
            for (int m = 0; m < kSide; m++) {
                a1[m] = a2[m];
                d1[m] = d2[m];
                plain_component_f(D, c, square, x[m], a2[m], d2[m]);
            }
        }
        const float Z = 1.f - F2 + c.q2 * F2;
        const float w1 = 1.f - F2, w2 = c.q2 * c.q2 * F2;
        const float iZ = 1.f / Z;
        const float k = one * iN * iZ * iZ;
#pragma unroll
        for (int m = 0; m < kSide; m++) {
            const float S = w1 * a1[m] + w2 * a2[m];
            const float base = S * iZ * iZ;
            g[m][0] = -base * one * iN * iN;
            g[m][1] = k * w1 * d1[m];
            g[m][2] = one;
            g[m][3] = one * iN * ((c.q2 * c.q2 * a2[m] - a1[m]) * iZ * iZ - 2.f * S * (c.q2 - 1.f) * iZ * iZ * iZ);
            g[m][4] = k * w2 * d2[m];
            f[m] = base * iN * one + G;
        }
    }
}

// FP64 values of the lane's points.
template <int K>
__device__ __forceinline__ void plain_model_d(const double (&p)[K], const ModelConstD &c, double one, int n, int lane,
                                              CompSh<K> &sh, double (&f)[kSide])
{
    constexpr int NC = CompSh<K>::NC;
    const double N = p[0], G = p[2];
    const double D = NC == 2 && (lane & 1) ? p[K - 1] : p[1];
#pragma unroll 1
    for (int i = lane; i < ((NC * n + 31) & ~31); i += 32)
        sh.a[i] = component_d(D, 0.0, 0.0, c, sh.x[min(i / NC, n - 1)]);
    __syncwarp();
    double F2 = 0.0, Z = 1.0;
    if constexpr (K == 5) {
        F2 = p[3];
        Z = 1.0 - F2 + c.q2 * F2;
    }
#pragma unroll
    for (int m = 0; m < kSide; m++) {
        const int i = lane + 32 * m;
        f[m] = 0.0;
        if (i < n) {
            if constexpr (K == 5) {
                const double S = (1.0 - F2) * sh.a[2 * i] + c.q2 * c.q2 * F2 * sh.a[2 * i + 1];
                f[m] = S / (Z * Z) / N * one + G;
            } else {
                f[m] = sh.a[i] / N + G;
            }
        }
    }
    __syncwarp();
}

// solve_scaled for K parameters, its products and sums rounded as they are
// there for a run-time parameter count (without the branches).
template <int K>
__device__ __forceinline__ bool comp_solve(const float (&A)[K * K], const float (&g)[K], float lambda, float (&h)[K])
{
    float sc[K], L[K * K];
#pragma unroll
    for (int i = 0; i < K; i++) sc[i] = rsqrtf(fmaxf(A[i * K + i], 1e-30f));
#pragma unroll
    for (int c = 0; c < K; c++) {
        float d = 1.f + lambda;
#pragma unroll
        for (int m = 0; m < c; m++) d = fmaf(-L[c * K + m], L[c * K + m], d);
        if (!(d > 0.f) || !isfinite(d)) return false;
        d = sqrtf(d);
        L[c * K + c] = d;
        const float id = 1.f / d;
#pragma unroll
        for (int r = c + 1; r < K; r++) {
            float sum = __fmul_rn(__fmul_rn(A[r * K + c], sc[r]), sc[c]);
#pragma unroll
            for (int m = 0; m < c; m++) sum = fmaf(-L[r * K + m], L[c * K + m], sum);
            L[r * K + c] = __fmul_rn(sum, id);
        }
    }
    float yv[K], z[K];
#pragma unroll
    for (int r = 0; r < K; r++) {
        float sum = r ? fmaf(g[r], sc[r], -__fmul_rn(L[r * K], yv[0])) : __fmul_rn(g[0], sc[0]);
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
#pragma unroll
    for (int r = 0; r < K; r++) h[r] = __fmul_rn(z[r], sc[r]);
    return true;
}

// GPUFIT: per-fit constants and Gpufit's stopping rule.
template <int K, bool GPUFIT>
__global__ void __launch_bounds__(32) lm_comp_kernel(FitArgs a)
{
    constexpr int NS = CompSh<K>::NS;
    __shared__ CompSh<K> sh;
    const int lane = threadIdx.x, n = a.npts;
    float xl[kSide];
#pragma unroll
    for (int m = 0; m < kSide; m++) {
        const int i = lane + 32 * m;
        xl[m] = __ldg(&a.x[min(i, n - 1)]);
        sh.x[i] = (double)xl[m];
    }
    __syncwarp();
    constexpr int kPar[5] = {0, 1, 4, 5, 6};

    for (int fit = blockIdx.x; fit < a.nfits; fit += gridDim.x) {
        if (a.todo && !__ldg(&a.todo[fit])) continue;
        const ModelConst mc = GPUFIT ? load_consts(a.cst + (size_t)fit * IMFCS_NCONST) : a.mc;
        ModelConstD mcd = to_double(mc);
        mcd.rx = mcd.ry = 0.0;
        const bool square = mc.ay == mc.ax;
        float yl[kSide], wl[kSide];
#pragma unroll
        for (int m = 0; m < kSide; m++) {
            const int i = lane + 32 * m;
            yl[m] = i < n ? __ldg(&a.y[(size_t)fit * n + i]) : 0.f;
            wl[m] = i < n ? (a.w ? __ldg(&a.w[(size_t)fit * n + i]) : 1.f) : 0.f;
        }
        const float *ip = a.init + (size_t)fit * a.init_stride;
        float p[K], pe[K];         // the fit's parameters, the ones to evaluate
        double pd[K], pde[K];
#pragma unroll
        for (int i = 0; i < K; i++) {
            p[i] = pe[i] = __ldg(&ip[kPar[i]]);
            pd[i] = pde[i] = p[i];
        }
        // lm_kernel's control flow with its evaluations drawn to one place:
        // what the evaluation under way is for
        enum { INIT, TRIAL, HESSIAN, NEWTON32, NEWTON64, RESTART } mode = INIT;
        bool precise = false, fresh = true;
        int state = IMFCS_STATE_MAX_ITERATIONS, it = 0, nprec = 0, ni = 0, col = 0;
        float lambda = 1e-3f, de = 0.f;
        double schi = 0.0;
        for (;;) {
            // --- chi^2 at pe, and J^T W J, J^T W r unless a rejected step ---
            const bool prec = mode == NEWTON64 || (precise && mode != HESSIAN);
            double chi2;
            bool take;
            {
                float g[kSide][K], r[kSide];
                if (prec) {
                    double f[kSide], c2 = 0.0;
                    plain_model_d<K>(pde, mcd, (double)a.one, n, lane, sh, f);
#pragma unroll
                    for (int m = 0; m < kSide; m++) {
                        r[m] = 0.f;
                        if (lane + 32 * m < n) {
                            const double rd = f2d(yl[m]) - f[m];
                            r[m] = (float)rd;
                            c2 += f2d(wl[m]) * rd * rd;
                        }
                    }
                    chi2 = warp_sum_d(c2);
                    take = mode != TRIAL || (isfinite(chi2) && chi2 < schi);
                }
                if (!prec || take) {
                    float f[kSide];
                    plain_model_f<K>(pe, mc, square, a.one, xl, f, g);
                    if (!prec) {
                        float c2f = 0.f;
#pragma unroll
                        for (int m = 0; m < kSide; m++)
                            if (lane + 32 * m < n) {
                                r[m] = yl[m] - f[m];
                                c2f = fmaf(wl[m] * r[m], r[m], c2f);
                            }
                        chi2 = (double)warp_sum(c2f);
                        take = mode != TRIAL || (isfinite(chi2) && chi2 < schi);
                    }
                }
                if (take) {
                    float acc[NS];
#pragma unroll
                    for (int i = 0; i < NS; i++) acc[i] = 0.f;
#pragma unroll
                    for (int m = 0; m < kSide; m++)
                        if (lane + 32 * m < n) {
                            const float w = wl[m];
                            int q = 0;
#pragma unroll
                            for (int i = 0; i < K; i++)
#pragma unroll
                                for (int t = 0; t <= i; t++) acc[q++] += w * g[m][i] * g[m][t];
#pragma unroll
                            for (int i = 0; i < K; i++) acc[q++] += w * g[m][i] * r[m];
                        }
                    int pos;
                    const float sum = warp_sums<NS, 16>(acc, lane, pos);
                    if (pos >= 0) sh.s[mode == HESSIAN][pos] = sum;
                    __syncwarp();
                }
            }

            bool newton = false, evald = false, to_precise = false, done = false;
            if (mode == TRIAL) {
                if (precise) nprec++;
                const bool found = GPUFIT && isfinite(chi2) && fabs(chi2 - schi) < (double)a.tol * fmax(1.0, chi2);
                if (take) {
                    schi = chi2;
                    fresh = true;
#pragma unroll
                    for (int i = 0; i < K; i++) { p[i] = pe[i]; pd[i] = pde[i]; }
                    lambda = GPUFIT ? lambda * 0.1f : fmaxf(lambda * 0.1f, 1e-9f);
                } else {
                    lambda *= 10.f;
                }
                if (GPUFIT ? found || lambda > 1e30f : !take && lambda > (precise ? 1e10f : 1e6f)) {
                    if (precise) { state = IMFCS_STATE_CONVERGED; done = true; }
                    else to_precise = true;
                }
                if (!GPUFIT && nprec > 60) { state = IMFCS_STATE_CONVERGED; done = true; }
                if (!to_precise) it++;
            } else if (mode == HESSIAN) {
                // column `col` of the Newton finish's Hessian (see lm_kernel)
                if (lane < K) sh.H[lane * K + col] = (sh.s[0][NS - K + lane] - sh.s[1][NS - K + lane]) / de;
                __syncwarp();
                if (++col < K) {
                    to_precise = true;
                } else {
                    float v = 0.f;
                    const int r = lane / K, q = lane % K;
                    if (lane < K * K && q < r) v = 0.5f * (sh.H[r * K + q] + sh.H[q * K + r]);
                    __syncwarp();
                    if (lane < K * K && q < r) { sh.H[r * K + q] = v; sh.H[q * K + r] = v; }
                    __syncwarp();
                    newton = true;
                }
            } else {
                schi = chi2;
                if (mode == INIT) {
                    if (!isfinite(chi2)) { state = IMFCS_STATE_SINGULAR_HESSIAN; done = true; }
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

            // --- next LM step: the stopping test on the undamped step, then
            // the damped one; one copy of the solver for both
            while (!newton && !to_precise) {
                if (it >= a.max_iter) { done = true; break; }
                float A[K * K], gv[K], h[K];
                {
                    int q = 0;
#pragma unroll
                    for (int i = 0; i < K; i++)
#pragma unroll
                        for (int t = 0; t <= i; t++) { A[i * K + t] = A[t * K + i] = sh.s[0][q]; q++; }
#pragma unroll
                    for (int i = 0; i < K; i++) gv[i] = sh.s[0][q++];
                }
                // the undamped solve in the warp's lower half beside the damped
                // one in the upper: a solve is one long chain
                const bool test = fresh && !GPUFIT;
                float hs[K];
                const bool oks = comp_solve<K>(A, gv, test && lane < 16 ? 0.f : lambda, hs);
                const unsigned votes = __ballot_sync(0xffffffffu, oks);
                const bool ok = votes >> 16 & 1;
#pragma unroll
                for (int i = 0; i < K; i++) h[i] = __shfl_sync(0xffffffffu, hs[i], 16);
                if (test && (votes & 1)) {
                    bool conv = true;
#pragma unroll
                    for (int i = 0; i < K; i++) {
                        const float sig = rsqrtf(fmaxf(A[i * K + i], 1e-30f));
                        const float tol = precise ? 1e-7f * fabsf(p[i]) + 1e-5f * sig : 1e-3f * sig;
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
                for (int i = 0; i < K; i++) {
                    pde[i] = pd[i] + (double)h[i];
                    pe[i] = (float)pde[i];
                }
                break;
            }
            if (done) break;

            if (to_precise) {
                // a forward difference (0.1 sigma) in parameter `col`
                if (mode != HESSIAN) col = 0;
                mode = HESSIAN;
                const int diag = col * (col + 3) / 2;
                const float eps = 0.1f * rsqrtf(fmaxf(sh.s[0][diag], 1e-30f));
#pragma unroll
                for (int i = 0; i < K; i++) {
                    pde[i] = pd[i];
                    pe[i] = p[i];
                    if (i == col) {
                        pde[i] += (double)eps;
                        pe[i] = (float)pde[i];
                        de = (float)(pde[i] - pd[i]);
                    }
                }
            } else if (newton) {
                // Newton steps: up to 3 on the FP32 gradient, then on that of
                // the FP64 residuals
                if (mode == HESSIAN) ni = 0;
                bool left = false;
#pragma unroll 1
                for (;;) {
                    if (ni >= 7) { left = true; break; }
                    const bool fp64 = ni >= 3;
                    if (fp64 && !evald) { mode = NEWTON64; break; }
                    if (fp64 && !isfinite(schi)) { left = true; break; }
                    evald = false;
                    float H[K * K], gv[K], hn[K];
#pragma unroll
                    for (int i = 0; i < K * K; i++) H[i] = sh.H[i];
#pragma unroll
                    for (int i = 0; i < K; i++) gv[i] = sh.s[0][NS - K + i];
                    if (!comp_solve<K>(H, gv, 0.f, hn)) { left = true; break; }
                    bool small = true;
#pragma unroll
                    for (int i = 0; i < K; i++) {
                        const float sig = rsqrtf(fmaxf(sh.s[0][i * (i + 3) / 2], 1e-30f));
                        if (!(fabsf(hn[i]) <= 0.05f * sig)) left = true;   // not in the quadratic region
                        small = small && (fabsf(hn[i]) <= 1e-4f * sig + (fp64 ? 1e-7f * fabsf(p[i]) : 0.f));
                    }
                    if (left) break;
#pragma unroll
                    for (int i = 0; i < K; i++) {
                        pd[i] += (double)hn[i];
                        p[i] = (float)pd[i];
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
                    // Levenberg-Marquardt on the FP64-residual model
                    precise = true;
                    mode = RESTART;
                }
#pragma unroll
                for (int i = 0; i < K; i++) { pde[i] = pd[i]; pe[i] = p[i]; }
            }
        }
        if (lane == 0) {
            float *o = a.out_par + (size_t)fit * a.out_stride;
            for (int i = 0; i < IMFCS_NPARAM; i++) o[i] = __ldg(&ip[i]);
#pragma unroll
            for (int i = 0; i < K; i++) o[kPar[i]] = (float)pd[i];
            if (a.out_chi2) a.out_chi2[fit] = (float)schi;
            if (a.out_state) a.out_state[fit] = state;
            if (a.out_iter) a.out_iter[fit] = it;
            if (a.out_hess)
                for (int i = 0; i < K * K; i++) {
                    const int r = max(i / K, i % K), q = min(i / K, i % K);
                    a.out_hess[(size_t)fit * K * K + i] = sh.s[0][r * (r + 1) / 2 + q];
                }
        }
        __syncwarp();
    }
}

// The fits of lm_comp_kernel: everything but the free parameters without
// effect (plain_held: the held flow, F3, Ftrip -- and F2 with one component --
// are zero for every fit, and no fit's window has an offset), points that
// three registers of a lane hold.  The rest -- GLS, other free parameters,
// more points -- stays with lm_kernel.
bool lm_comp_applies(const FitArgs &a)
{
    const bool common = a.plain_held && a.model == IMFCS_MODEL_ACF_1D && !a.linv && a.npts >= 1 &&
                        a.npts <= kCompPts && a.np == IMFCS_NPARAM && a.idx[0] == 0 && a.idx[1] == 1 && a.idx[2] == 4;
    if (!common) return false;
    if (a.k == 3) return a.tol > 0.f && a.cst;
    return a.k == 5 && a.idx[3] == 5 && a.idx[4] == 6 && a.tol == 0.f && !a.cst && a.mc.rx == 0.f && a.mc.ry == 0.f;
}

// One warp per block and one fit per block, handed out by the hardware as
// fits end: 1,600 fits spread as 10 or 11 over every SM.
cudaError_t launch_lm_comp(const FitArgs &a, cudaStream_t s)
{
    const int blocks = a.nfits < (1 << 20) ? a.nfits : 1 << 20;
    if (a.k == 3) lm_comp_kernel<3, true><<<blocks, 32, 0, s>>>(a);
    else lm_comp_kernel<5, false><<<blocks, 32, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace imfcs
