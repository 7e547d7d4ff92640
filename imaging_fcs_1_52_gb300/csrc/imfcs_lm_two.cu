// imfcs_lm_two.cu -- the LM fit of the two-component model, specialised:
// FCS_3p (java:13131-13408) without flow, third component, triplet or window
// offset, N, D, G, F2 and D2 free, OLS, up to 96 points, step-mode stopping
// rule.  It is the second model of the plugin's Bayes comparison
// (bayesFit, java:10191-10220).  Same algorithm, stopping rules and operation order as
// lm_kernel (imfcs_lm.cuh), which gives the same bits.
//
// These fits take some 80 accepted and 80 rejected FP32 steps and 45 steps on
// the FP64 model each (a few take 900), one warp per fit, so a warp's time is
// its instruction count times a latency of about ten cycles, and the longest fits
// set the launch's.  Against lm_kernel<5>:
//   - one evaluation site, driven by a state machine, and loops over the
//     components instead of copies: the code stays near the instruction
//     caches (a third of the stalls were instruction fetches);
//   - parameters in registers, the normal matrix in shared memory;
//   - chi^2 first: a rejected step ends there, without the 20 sums of the
//     normal equations and, on the FP64 model, without the gradient;
//   - the undamped step behind the stopping test is not solved again after a
//     rejected step;
//   - the 20 sums over the warp as one transposed reduction (same tree);
//   - FP64 model values two lanes a point, one component each: 5 rounds for
//     72 points, not 6.
// 1,600 fits of 72 points: 14.2 -> 5.0 ms, then bound by the FP64 pipe (60 %
// busy) and the longest fits.
#include "imfcs_lm.cuh"

namespace imfcs {

constexpr int kTwoPts = 96;
constexpr int kTwoSide = kTwoPts / 32;   // points of a lane, evaluated side by side

struct TwoSh {
    double a[2 * kTwoPts];   // FP64 component terms [point][component]
    double x[kTwoPts];
    float s[2][20];          // lower triangle of J^T W J by rows, then J^T W r: the fit's, a probe's
    float H[25];
};

// lat x axial factor of one component and its derivative (component_f).
__device__ __forceinline__ void two_component_f(float d, const ModelConst &c, bool square, float tau, float &a,
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

// Values and gradients (d/dN, D, G, F2, D2) of the lane's points.  `one` is
// 1.f, a run-time value: products with it stay where the general model
// multiplies by the triplet factor, and round as they do there.
__device__ __forceinline__ void two_model_f(const float (&p)[5], const ModelConst &c, bool square, float one,
                                            const float (&x)[kTwoSide], float (&f)[kTwoSide],
                                            float (&g)[kTwoSide][5])
{
    const float N = p[0], G = p[2], F2 = p[3];
    float a1[kTwoSide], a2[kTwoSide], d1[kTwoSide], d2[kTwoSide];
#pragma unroll
    for (int m = 0; m < kTwoSide; m++) a2[m] = d2[m] = 0.f;
#pragma unroll 1
    for (int q = 0; q < 2; q++) {
        const float D = q ? p[4] : p[1];
#pragma unroll
        for (int m = 0; m < kTwoSide; m++) {
            a1[m] = a2[m];
            d1[m] = d2[m];
            two_component_f(D, c, square, x[m], a2[m], d2[m]);
        }
    }
    const float Z = 1.f - F2 + c.q2 * F2;
    const float w1 = 1.f - F2, w2 = c.q2 * c.q2 * F2;
    const float iZ = 1.f / Z, iN = 1.f / N;
    const float k = one * iN * iZ * iZ;
#pragma unroll
    for (int m = 0; m < kTwoSide; m++) {
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

// FP64 values of the lane's points.
__device__ __forceinline__ void two_model_d(const double (&p)[5], const ModelConstD &c, double one, int n, int lane,
                                            TwoSh &sh, double (&f)[kTwoSide])
{
    const double N = p[0], G = p[2], F2 = p[3];
    const double D = lane & 1 ? p[4] : p[1];
#pragma unroll 1
    for (int i = lane; i < ((2 * n + 31) & ~31); i += 32)
        sh.a[i] = component_d(D, 0.0, 0.0, c, sh.x[min(i >> 1, n - 1)]);
    __syncwarp();
    const double Z = 1.0 - F2 + c.q2 * F2;
#pragma unroll
    for (int m = 0; m < kTwoSide; m++) {
        const int i = lane + 32 * m;
        f[m] = 0.0;
        if (i < n) {
            const double S = (1.0 - F2) * sh.a[2 * i] + c.q2 * c.q2 * F2 * sh.a[2 * i + 1];
            f[m] = S / (Z * Z) / N * one + G;
        }
    }
    __syncwarp();
}

// solve_scaled for five parameters, its products and sums rounded as they are
// there for a run-time parameter count (without the branches).
__device__ __forceinline__ bool two_solve(const float (&A)[25], const float (&g)[5], float lambda, float (&h)[5])
{
    float sc[5], L[25];
#pragma unroll
    for (int i = 0; i < 5; i++) sc[i] = rsqrtf(fmaxf(A[i * 5 + i], 1e-30f));
#pragma unroll
    for (int c = 0; c < 5; c++) {
        float d = 1.f + lambda;
#pragma unroll
        for (int m = 0; m < c; m++) d = fmaf(-L[c * 5 + m], L[c * 5 + m], d);
        if (!(d > 0.f) || !isfinite(d)) return false;
        d = sqrtf(d);
        L[c * 5 + c] = d;
        const float id = 1.f / d;
#pragma unroll
        for (int r = c + 1; r < 5; r++) {
            float sum = __fmul_rn(__fmul_rn(A[r * 5 + c], sc[r]), sc[c]);
#pragma unroll
            for (int m = 0; m < c; m++) sum = fmaf(-L[r * 5 + m], L[c * 5 + m], sum);
            L[r * 5 + c] = __fmul_rn(sum, id);
        }
    }
    float yv[5], z[5];
#pragma unroll
    for (int r = 0; r < 5; r++) {
        float sum = r ? fmaf(g[r], sc[r], -__fmul_rn(L[r * 5], yv[0])) : __fmul_rn(g[0], sc[0]);
#pragma unroll
        for (int m = 1; m < r; m++) sum = fmaf(-L[r * 5 + m], yv[m], sum);
        yv[r] = sum / L[r * 5 + r];
    }
#pragma unroll
    for (int r = 4; r >= 0; r--) {
        float sum = yv[r];
#pragma unroll
        for (int m = r + 1; m < 5; m++) sum = fmaf(-L[m * 5 + r], z[m], sum);
        z[r] = sum / L[r * 5 + r];
    }
#pragma unroll
    for (int r = 0; r < 5; r++) h[r] = __fmul_rn(z[r], sc[r]);
    return true;
}

// Sums over the warp of 20 values, each in the order of warp_sum (the lane
// pairs 16, 8, 4, 2, 1 apart): every exchange halves the values a lane still
// carries, 21 shuffles instead of 100.  out[i] (shared) = sum of v[i].
__device__ __forceinline__ void warp_sums20(float (&v)[20], int lane, float *out)
{
    // lane's values after each exchange: 10, 5, 3, 2, 1
    float a[10], b[6], c[4], d[2];
    bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 10; i++) {
        const float keep = up ? v[i + 10] : v[i], send = up ? v[i] : v[i + 10];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
    up = lane & 8;
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const float keep = up ? a[i + 5] : a[i], send = up ? a[i] : a[i + 5];
        b[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    b[5] = 0.f;
    up = lane & 4;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const float keep = up ? b[i + 3] : b[i], send = up ? b[i] : b[i + 3];
        c[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
    c[3] = 0.f;
    up = lane & 2;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float keep = up ? c[i + 2] : c[i], send = up ? c[i] : c[i + 2];
        d[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    up = lane & 1;
    const float keep = up ? d[1] : d[0], send = up ? d[0] : d[1];
    const float r = keep + __shfl_xor_sync(0xffffffffu, send, 1);
    // which sum this lane holds (padding: none)
    const int e3 = 2 * ((lane >> 1) & 1) + (lane & 1);    // of 4, 3 used
    const int e5 = 3 * ((lane >> 2) & 1) + e3;            // of 6, 5 used
    if (e3 < 3 && e5 < 5) out[10 * (lane >> 4) + 5 * ((lane >> 3) & 1) + e5] = r;
    __syncwarp();
}

__global__ void __launch_bounds__(32) lm_two_kernel(FitArgs a)
{
    __shared__ TwoSh sh;
    const int lane = threadIdx.x, n = a.npts;
    const bool square = a.mc.ay == a.mc.ax;
    ModelConstD mcd = to_double(a.mc);
    float xl[kTwoSide];
#pragma unroll
    for (int m = 0; m < kTwoSide; m++) {
        const int i = lane + 32 * m;
        xl[m] = __ldg(&a.x[min(i, n - 1)]);
        sh.x[i] = (double)xl[m];
    }
    __syncwarp();
    constexpr int kPar[5] = {0, 1, 4, 5, 6};

    for (int fit = a.counter ? lm_next_fit(a, 0, 0, lane) : blockIdx.x; fit < a.nfits;
         fit = lm_next_fit(a, fit, gridDim.x, lane)) {
        if (a.todo && !__ldg(&a.todo[fit])) continue;
        float yl[kTwoSide], wl[kTwoSide];
#pragma unroll
        for (int m = 0; m < kTwoSide; m++) {
            const int i = lane + 32 * m;
            yl[m] = i < n ? __ldg(&a.y[(size_t)fit * n + i]) : 0.f;
            wl[m] = i < n ? (a.w ? __ldg(&a.w[(size_t)fit * n + i]) : 1.f) : 0.f;
        }
        const float *ip = a.init + (size_t)fit * a.init_stride;
        float p[5], pe[5];         // the fit's parameters, the ones to evaluate
        double pd[5], pde[5];
#pragma unroll
        for (int i = 0; i < 5; i++) {
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
                float g[kTwoSide][5], r[kTwoSide];
                if (prec) {
                    double f[kTwoSide], c2 = 0.0;
                    two_model_d(pde, mcd, (double)a.one, n, lane, sh, f);
#pragma unroll
                    for (int m = 0; m < kTwoSide; m++) {
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
                    float f[kTwoSide];
                    two_model_f(pe, a.mc, square, a.one, xl, f, g);
                    if (!prec) {
                        float c2f = 0.f;
#pragma unroll
                        for (int m = 0; m < kTwoSide; m++)
                            if (lane + 32 * m < n) {
                                r[m] = yl[m] - f[m];
                                c2f = fmaf(wl[m] * r[m], r[m], c2f);
                            }
                        chi2 = (double)warp_sum(c2f);
                        take = mode != TRIAL || (isfinite(chi2) && chi2 < schi);
                    }
                }
                if (take) {
                    float acc[20];
#pragma unroll
                    for (int i = 0; i < 20; i++) acc[i] = 0.f;
#pragma unroll
                    for (int m = 0; m < kTwoSide; m++)
                        if (lane + 32 * m < n) {
                            const float w = wl[m];
                            int q = 0;
#pragma unroll
                            for (int i = 0; i < 5; i++)
#pragma unroll
                                for (int t = 0; t <= i; t++) acc[q++] += w * g[m][i] * g[m][t];
#pragma unroll
                            for (int i = 0; i < 5; i++) acc[q++] += w * g[m][i] * r[m];
                        }
                    warp_sums20(acc, lane, sh.s[mode == HESSIAN]);
                }
            }

            bool newton = false, evald = false, to_precise = false, done = false;
            if (mode == TRIAL) {
                if (precise) nprec++;
                if (take) {
                    schi = chi2;
                    fresh = true;
#pragma unroll
                    for (int i = 0; i < 5; i++) { p[i] = pe[i]; pd[i] = pde[i]; }
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
                // column `col` of the Newton finish's Hessian (see lm_kernel)
                if (lane < 5) sh.H[lane * 5 + col] = (sh.s[0][15 + lane] - sh.s[1][15 + lane]) / de;
                __syncwarp();
                if (++col < 5) {
                    to_precise = true;
                } else {
                    float v = 0.f;
                    const int r = lane / 5, q = lane % 5;
                    if (lane < 25 && q < r) v = 0.5f * (sh.H[r * 5 + q] + sh.H[q * 5 + r]);
                    __syncwarp();
                    if (lane < 25 && q < r) { sh.H[r * 5 + q] = v; sh.H[q * 5 + r] = v; }
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
                float A[25], gv[5], h[5], sig[5];
                {
                    int q = 0;
#pragma unroll
                    for (int i = 0; i < 5; i++)
#pragma unroll
                        for (int t = 0; t <= i; t++) { A[i * 5 + t] = A[t * 5 + i] = sh.s[0][q]; q++; }
#pragma unroll
                    for (int i = 0; i < 5; i++) gv[i] = sh.s[0][q++];
                }
                bool ok = false;
#pragma unroll 1
                for (int pass = fresh ? 0 : 1; pass < 2; pass++) {
                    ok = two_solve(A, gv, pass ? lambda : 0.f, h);
                    if (pass == 0 && ok) {
                        bool conv = true;
#pragma unroll
                        for (int i = 0; i < 5; i++) {
                            sig[i] = rsqrtf(fmaxf(A[i * 5 + i], 1e-30f));
                            const float tol = precise ? 1e-7f * fabsf(p[i]) + 1e-5f * sig[i] : 1e-3f * sig[i];
                            conv = conv && (fabsf(h[i]) <= tol);
                        }
                        if (conv) {
                            if (precise) { state = IMFCS_STATE_CONVERGED; done = true; }
                            else to_precise = true;
                            break;
                        }
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
                for (int i = 0; i < 5; i++) {
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
                for (int i = 0; i < 5; i++) {
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
                    float H[25], gv[5], hn[5];
#pragma unroll
                    for (int i = 0; i < 25; i++) H[i] = sh.H[i];
#pragma unroll
                    for (int i = 0; i < 5; i++) gv[i] = sh.s[0][15 + i];
                    if (!two_solve(H, gv, 0.f, hn)) { left = true; break; }
                    bool small = true;
#pragma unroll
                    for (int i = 0; i < 5; i++) {
                        const float sig = rsqrtf(fmaxf(sh.s[0][i * (i + 3) / 2], 1e-30f));
                        if (!(fabsf(hn[i]) <= 0.05f * sig)) left = true;   // not in the quadratic region
                        small = small && (fabsf(hn[i]) <= 1e-4f * sig + (fp64 ? 1e-7f * fabsf(p[i]) : 0.f));
                    }
                    if (left) break;
#pragma unroll
                    for (int i = 0; i < 5; i++) {
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
                for (int i = 0; i < 5; i++) { pde[i] = pd[i]; pe[i] = p[i]; }
            }
        }
        if (lane == 0) {
            float *o = a.out_par + (size_t)fit * a.out_stride;
            for (int i = 0; i < IMFCS_NPARAM; i++) o[i] = __ldg(&ip[i]);
#pragma unroll
            for (int i = 0; i < 5; i++) o[kPar[i]] = (float)pd[i];
            if (a.out_chi2) a.out_chi2[fit] = (float)schi;
            if (a.out_state) a.out_state[fit] = state;
            if (a.out_iter) a.out_iter[fit] = it;
            if (a.out_hess)
                for (int i = 0; i < 25; i++) {
                    const int r = max(i / 5, i % 5), q = min(i / 5, i % 5);
                    a.out_hess[(size_t)fit * 25 + i] = sh.s[0][r * (r + 1) / 2 + q];
                }
        }
        __syncwarp();
    }
}

// The fits of lm_two_kernel: shared constants, everything but the five free
// parameters without effect (two_zero_held: the held flow, F3 and Ftrip are
// zero for every fit), points that three registers of a lane hold.  The rest
// -- GLS, Gpufit's stopping rule, more points -- stays with lm_kernel<5>.
bool lm_two_applies(const FitArgs &a)
{
    return a.two_zero_held && a.model == IMFCS_MODEL_ACF_1D && !a.cst && !a.linv && a.npts >= 1 &&
           a.npts <= kTwoPts && a.tol == 0.f && a.np == IMFCS_NPARAM && a.k == 5 && a.idx[0] == 0 && a.idx[1] == 1 &&
           a.idx[2] == 4 && a.idx[3] == 5 && a.idx[4] == 6 && a.mc.rx == 0.f && a.mc.ry == 0.f;
}

// One warp per block: 1,600 fits spread as 10 or 11 over every SM.
cudaError_t launch_lm_two(const FitArgs &a, int num_sms, cudaStream_t s)
{
    const int cap = num_sms * 32;
    lm_two_kernel<<<a.nfits < cap ? a.nfits : cap, 32, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace imfcs
