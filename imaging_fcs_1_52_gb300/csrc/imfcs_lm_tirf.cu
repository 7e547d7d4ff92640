// imfcs_lm_tirf.cu -- the LM fit of the plugin's default model, specialised:
// FCS_3p (java:13131-13408) with one component, no flow, no triplet, N, D and
// G free (the other parameters held at zero), up to kMaxPts points,
// step-mode stopping rule.  Same algorithm, stopping rules and FP32
// operation order as lm_kernel (imfcs_lm.cuh): phase 1 LM on FP32 model
// values, Newton finish with a forward-difference Hessian, FP32 then FP64
// residuals.  The model is evaluated from three scalars instead of the
// 11-parameter vector, so the parameters live in registers (no local-memory
// arrays indexed at run time) and the executed code is a few kilobytes --
// the generic kernel stalls on instruction fetch and local-memory loads.
//
// A compile-time variant widens it to the spatial cross-correlation model
// (OFF: window offsets rx, ry, the three-term lateral factor).  The fit on
// whitened data is imfcs_lm_gls.cu's.
#include "imfcs_tirf.cuh"

namespace imfcs {

struct Tirf3 {
    float A[9];
    float g[3];
    float chi2;      // FP32 phases
    double chi2d;    // FP64-residual evaluations
    float fmag;      // sum w (|a/N| + |G|)^2: scale of the model values (FP32 phases)
};

__device__ __forceinline__ void tirf_reduce(float (&acc)[9], Tirf3 &s)
{
    int q = 0;
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
        for (int t = 0; t <= p; t++) {
            const float v = warp_sum(acc[q++]);
            s.A[p * 3 + t] = v;
            s.A[t * 3 + p] = v;
        }
#pragma unroll
    for (int p = 0; p < 3; p++) s.g[p] = warp_sum(acc[q++]);
}

__device__ __forceinline__ void tirf_accumulate(float (&acc)[9], const float (&gr)[3], float w, float r)
{
    int q = 0;
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
        for (int t = 0; t <= p; t++) acc[q++] += w * gr[p] * gr[t];
#pragma unroll
    for (int p = 0; p < 3; p++) acc[q++] += w * gr[p] * r;
}

// One evaluation over the fit's points (warp): chi^2, J^T W J, J^T W r with
// FP32 residuals.  No FP64 operation: GB300 issues FP64 at 1/64 of the FP32
// rate, and the FP32 phases evaluate the model some twenty times per fit.
template <bool OFF, bool SIDE>
__device__ __noinline__ void tirf_eval32(const TirfC &c, float N, float D, float G, const float *yl,
                                         const float *wl, const float *xl, int n, int lane, Tirf3 &s,
                                         float bound)       // a trial step's: chi^2 to be lowered (else NaN)
{
    float acc[9];
#pragma unroll
    for (int i = 0; i < 9; i++) acc[i] = 0.f;
    float c2f = 0.f, fm = 0.f;
    constexpr int kSide = SIDE && !OFF ? 3 : 0;     // a lane's first points, their chains side by side
    float sf[3], sN[3], sD[3], sm[3];
#pragma unroll
    for (int m = 0; m < kSide; m++) sf[m] = tirf_f<OFF, true>(N, D, G, c, xl[m], sN[m], sD[m], sm[m]);
#pragma unroll
    for (int m = 0; m < kPtsPerLane; m++) {
        const int i = lane + 32 * m;
        if (i < n) {
            float gr[3], mag;
            gr[2] = 1.f;
            float f;
            if (m < kSide) {
                f = sf[m];
                gr[0] = sN[m];
                gr[1] = sD[m];
                mag = sm[m];
            } else {
                f = tirf_f<OFF>(N, D, G, c, xl[m], gr[0], gr[1], mag);
            }
            const float w = wl[m];
            const float r = yl[m] - f;
            c2f = fmaf(w * r, r, c2f);
            fm = fmaf(w * mag, mag, fm);
            tirf_accumulate(acc, gr, w, r);
        }
    }
    s.chi2 = warp_sum(c2f);
    s.chi2d = 0.0;
    // a rejected trial step: nobody reads the sums (those of every other
    // evaluation are read, whatever chi^2 is)
    if (!isnan(bound) && !(s.chi2 < bound)) return;
    tirf_reduce(acc, s);
    s.fmag = warp_sum(fm);
}

// The same with residuals of the model value in float-float at the FP64
// parameters (Nd, Dd, Gd) -- FP64 model where the series do not apply --
// the Jacobian in FP32 at their FP32 copies; chi^2 reduced in float-float.
template <bool OFF, bool SIDE>
__device__ __noinline__ void tirf_eval64(const TirfC &c, double Nd, double Dd, double Gd, const float *yl,
                                         const float *wl, const float *xl, int n, int lane, Tirf3 &s)
{
    const float N = (float)Nd, D = (float)Dd, G = (float)Gd;
    const double inv_Nd = 1.0 / Nd;
    float acc[9];
#pragma unroll
    for (int i = 0; i < 9; i++) acc[i] = 0.f;
    const f2 inv_Nf = f2_from_d(inv_Nd), Df = f2_from_d(Dd), Gf = f2_from_d(Gd);
    f2 c2acc = {0.f, 0.f};
#pragma unroll
    for (int m = 0; m < kPtsPerLane; m++) {
        const int i = lane + 32 * m;
        if (i < n) {
            float gr[3], mag;
            gr[2] = 1.f;
            tirf_f<OFF>(N, D, G, c, xl[m], gr[0], gr[1], mag);
            const float w = wl[m];
            f2 fv, lat;
            if (!OFF && tirf_a_ff(Df, c, xl[m], lat)) fv = f2_add(f2_mul(lat, inv_Nf), Gf);
            else fv = f2_from_d(fma(tirf_a_d<OFF>(Dd, c, (double)xl[m]), inv_Nd, Gd));
            const f2 rr = f2_add(f2_from_f(yl[m]), f2_neg(fv));
            const float r = f2_val(rr);
            c2acc = f2_add(c2acc, f2_mul_f(f2_mul(rr, rr), w));
            tirf_accumulate(acc, gr, w, r);
        }
    }
    tirf_reduce(acc, s);
    for (int o = 16; o > 0; o >>= 1) {
        const f2 other = {__shfl_xor_sync(0xffffffffu, c2acc.hi, o), __shfl_xor_sync(0xffffffffu, c2acc.lo, o)};
        c2acc = f2_add(c2acc, other);
    }
    s.chi2d = (double)c2acc.hi + (double)c2acc.lo;
    s.chi2 = c2acc.hi + c2acc.lo;
    s.fmag = 0.f;
}

// dispatch by phase
template <bool OFF, bool SIDE>
__device__ __forceinline__ void tirf_eval(const TirfC &c, float N, float D, float G, double Nd, double Dd, double Gd,
                                          const float *yl, const float *wl, const float *xl, int n, int lane,
                                          bool precise, Tirf3 &s, float bound = NAN)
{
    if (precise) tirf_eval64<OFF, SIDE>(c, Nd, Dd, Gd, yl, wl, xl, n, lane, s);
    else tirf_eval32<OFF, SIDE>(c, N, D, G, yl, wl, xl, n, lane, s, bound);
}

__device__ __forceinline__ float tirf_sig(const Tirf3 &s, int i) { return rsqrtf(fmaxf(s.A[i * 3 + i], 1e-30f)); }

// Bound on the relative rounding error of the FP32 model value (erff and
// expm1f within a few ulp, ~15 roundings of the lateral, axial and final
// terms): 4e-6, some 70 ulp.
constexpr float kModelRound = 4e-6f;

template <bool OFF, bool SIDE>
__global__ void __launch_bounds__(128) lm_tirf_kernel(FitArgs a)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int wpb = blockDim.x >> 5;
    const int n = a.npts;
    const int gw = blockIdx.x * wpb + wib, nw = gridDim.x * wpb;
    const TirfC c = tirf_consts(a.mc);
    float xl[kPtsPerLane];
#pragma unroll
    for (int m = 0; m < kPtsPerLane; m++) {
        const int i = lane + 32 * m;
        xl[m] = i < n ? __ldg(&a.x[i]) : 0.f;
    }
    for (int fit = a.counter ? lm_next_fit(a, 0, 0, lane) : gw; fit < a.nfits; fit = lm_next_fit(a, fit, nw, lane)) {
        if (a.todo && !__ldg(&a.todo[fit])) continue;
        float yl[kPtsPerLane], wl[kPtsPerLane];
#pragma unroll
        for (int m = 0; m < kPtsPerLane; m++) {
            const int i = lane + 32 * m;
            yl[m] = i < n ? __ldg(&a.y[(size_t)fit * n + i]) : 0.f;
            wl[m] = i < n ? (a.w ? __ldg(&a.w[(size_t)fit * n + i]) : 1.f) : 0.f;
        }
        const float *ip = a.init + (size_t)fit * a.init_stride;
        // free parameters N, D, G (vector indices 0, 1, 4): FP32 in the FP32
        // phases, FP64 from the FP64-residual Newton steps on
        float pf[3] = {__ldg(&ip[0]), __ldg(&ip[1]), __ldg(&ip[4])};
        double pd[3] = {0.0, 0.0, 0.0};
        bool precise = false;     // parameters and chi^2 held in FP64 (pd, chi2d)
        bool retried = false;     // Newton left its region once: FP32 LM to 1e-4 sigma, then Newton again
        Tirf3 s;
        tirf_eval<OFF, SIDE>(c, pf[0], pf[1], pf[2], 0.0, 0.0, 0.0, yl, wl, xl, n, lane, false, s);
        int state = IMFCS_STATE_MAX_ITERATIONS, it = 0, nprec = 0;
        float lambda = 1e-3f;
        if (!isfinite(s.chi2)) state = IMFCS_STATE_SINGULAR_HESSIAN;
        for (it = 0; state == IMFCS_STATE_MAX_ITERATIONS && it < a.max_iter; it++) {
            float h[3];
            bool to_precise = false, ok;
            {
                // the undamped step of the stopping test and the damped one,
                // each in half of the warp: a solve is one long chain
                float hs[3], hg[3];
                const bool oks = tirf_solve(s.A, s.g, lane < 16 ? 0.f : lambda, hs);
                const unsigned votes = __ballot_sync(0xffffffffu, oks);
                ok = votes >> 16 & 1;
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    hg[i] = __shfl_sync(0xffffffffu, hs[i], 0);
                    h[i] = __shfl_sync(0xffffffffu, hs[i], 16);
                }
                if (votes & 1) {
                    bool conv = true;
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const float sig = tirf_sig(s, i);
                        const float tol = precise ? 1e-7f * fabsf(pf[i]) + 1e-5f * sig : (retried ? 1e-4f : 1e-3f) * sig;
                        conv = conv && (fabsf(hg[i]) <= tol);
                    }
                    if (conv) {
                        if (precise) { state = IMFCS_STATE_CONVERGED; break; }
                        to_precise = true;
                    }
                }
            }
            if (!to_precise) {
                if (!ok) {
                    lambda *= 10.f;
                    if (lambda > 1e15f) { state = IMFCS_STATE_SINGULAR_HESSIAN; break; }
                    continue;
                }
                Tirf3 sn;
                float pnf[3];
                double pnd[3] = {0.0, 0.0, 0.0};
                bool better;
                if (precise) {
#pragma unroll
                    for (int i = 0; i < 3; i++) { pnd[i] = pd[i] + (double)h[i]; pnf[i] = (float)pnd[i]; }
                    tirf_eval<OFF, SIDE>(c, pnf[0], pnf[1], pnf[2], pnd[0], pnd[1], pnd[2], yl, wl, xl, n, lane, true, sn);
                    nprec++;
                    better = isfinite(sn.chi2d) && sn.chi2d < s.chi2d;
                } else {
#pragma unroll
                    for (int i = 0; i < 3; i++) pnf[i] = pf[i] + h[i];
                    tirf_eval<OFF, SIDE>(c, pnf[0], pnf[1], pnf[2], 0.0, 0.0, 0.0, yl, wl, xl, n, lane, false, sn, s.chi2);
                    better = isfinite(sn.chi2) && sn.chi2 < s.chi2;
                }
                if (better) {
#pragma unroll
                    for (int i = 0; i < 3; i++) { pd[i] = pnd[i]; pf[i] = pnf[i]; }
                    s = sn;
                    lambda = fmaxf(lambda * 0.1f, 1e-9f);
                } else {
                    lambda *= 10.f;
                    if (lambda > (precise ? 1e10f : 1e6f)) {
                        if (precise) { state = IMFCS_STATE_CONVERGED; it++; break; }
                        to_precise = true;
                    }
                }
                if (nprec > 60) { state = IMFCS_STATE_CONVERGED; it++; break; }
            }
            if (to_precise) {
                // Newton finish (see lm_kernel): forward-difference Hessian
                // of chi^2/2 from the FP32 gradient, FP32 steps to its
                // stationary point, then FP64-residual steps until the step
                // is below 1e-4 sigma + 1e-7 |p|.
                float H[9];
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    const float eps = 0.1f * tirf_sig(s, i);
                    float pe[3] = {pf[0], pf[1], pf[2]};
                    pe[i] = pf[i] + eps;
                    const float de = pe[i] - pf[i];
                    Tirf3 se;
                    tirf_eval<OFF, SIDE>(c, pe[0], pe[1], pe[2], 0.0, 0.0, 0.0, yl, wl, xl, n, lane, false, se);
#pragma unroll
                    for (int r = 0; r < 3; r++) H[r * 3 + i] = (s.g[r] - se.g[r]) / de;
                }
#pragma unroll
                for (int r = 0; r < 3; r++)
#pragma unroll
                    for (int q = 0; q < r; q++) {
                        const float v = 0.5f * (H[r * 3 + q] + H[q * 3 + r]);
                        H[r * 3 + q] = v;
                        H[q * 3 + r] = v;
                    }
                bool newton_done = false, left = false, stationary = false;
#pragma unroll 1
                for (int ni = 0; ni < 7 && !left; ni++) {
                    const bool fp64 = ni >= 3;
                    if (!OFF && fp64 && !precise && stationary) {
                        // At the FP32 gradient's stationary point.  The FP32
                        // model value's rounding error (below kModelRound of
                        // the summed terms' magnitude, |a/N| + |G|) moves
                        // the minimum by at most B sigma_i in parameter i,
                        // B = kModelRound sqrt(sum w (|a/N| + |G|)^2)
                        // (Cauchy-Schwarz in the metric of J^T W J).  Where
                        // that is below 1e-5 of N and of D, the FP64 step
                        // cannot matter at the 1e-4 parity bar: skip it.
                        // (Not for the offset lateral factor, whose terms
                        // cancel.)
                        const float B = kModelRound * sqrtf(s.fmag);
                        if (B * tirf_sig(s, 0) <= 1e-5f * fabsf(pf[0]) && B * tirf_sig(s, 1) <= 1e-5f * fabsf(pf[1])) {
                            newton_done = true;
                            break;
                        }
                    }
                    if (fp64) {
                        if (!precise) {
#pragma unroll
                            for (int i = 0; i < 3; i++) pd[i] = (double)pf[i];
                            precise = true;
                        }
                        tirf_eval<OFF, SIDE>(c, pf[0], pf[1], pf[2], pd[0], pd[1], pd[2], yl, wl, xl, n, lane, true, s);
                        if (!isfinite(s.chi2d)) { left = true; break; }
                    }
                    float hn[3];
                    if (!solve_scaled<3>(H, s.g, 3, 0.f, hn)) { left = true; break; }
                    bool small = true;
#pragma unroll
                    for (int i = 0; i < 3; i++) {
                        const float sig = tirf_sig(s, i);
                        if (!(fabsf(hn[i]) <= 0.05f * sig)) left = true;
                        small = small && (fabsf(hn[i]) <= 1e-4f * sig + (fp64 ? 1e-7f * fabsf(pf[i]) : 0.f));
                    }
                    if (left) break;
                    if (fp64) {
#pragma unroll
                        for (int i = 0; i < 3; i++) { pd[i] += (double)hn[i]; pf[i] = (float)pd[i]; }
                        if (small) { newton_done = true; break; }
                    } else {
#pragma unroll
                        for (int i = 0; i < 3; i++) pf[i] += hn[i];
                        if (small) {
                            ni = 2;
                            stationary = true;
                        } else {
                            tirf_eval<OFF, SIDE>(c, pf[0], pf[1], pf[2], 0.0, 0.0, 0.0, yl, wl, xl, n, lane, false, s);
                        }
                    }
                }
                if (newton_done) { state = IMFCS_STATE_CONVERGED; it++; break; }
                if (!retried) {
                    // Newton left its quadratic region (a step above 0.05
                    // sigma) or met an indefinite Hessian: back to FP32 LM,
                    // to the tighter 1e-4 sigma, and Newton from there -- an
                    // LM on FP64-residual evaluations costs ~10x an FP32
                    // iteration and runs for tens of iterations, and the few
                    // fits that take it set the duration of the whole launch
                    retried = true;
                    if (precise) {
#pragma unroll
                        for (int i = 0; i < 3; i++) pf[i] = (float)pd[i];
                        precise = false;
                    }
                    tirf_eval<OFF, SIDE>(c, pf[0], pf[1], pf[2], 0.0, 0.0, 0.0, yl, wl, xl, n, lane, false, s);
                    lambda = 1e-3f;
                    continue;
                }
                // otherwise LM on the FP64-residual model
                if (!precise) {
#pragma unroll
                    for (int i = 0; i < 3; i++) pd[i] = (double)pf[i];
                    precise = true;
                }
                tirf_eval<OFF, SIDE>(c, pf[0], pf[1], pf[2], pd[0], pd[1], pd[2], yl, wl, xl, n, lane, true, s);
                lambda = 1e-3f;
            }
        }
        if (lane == 0) {
            float *o = a.out_par + (size_t)fit * a.out_stride;
            for (int i = 0; i < a.np; i++) o[i] = __ldg(&ip[i]);
            o[0] = precise ? (float)pd[0] : pf[0];
            o[1] = precise ? (float)pd[1] : pf[1];
            o[4] = precise ? (float)pd[2] : pf[2];
            if (a.out_chi2) a.out_chi2[fit] = s.chi2;
            if (a.out_state) a.out_state[fit] = state;
            if (a.out_iter) a.out_iter[fit] = it;
            if (a.out_hess)
                for (int i = 0; i < 9; i++) a.out_hess[(size_t)fit * 9 + i] = s.A[i];
        }
        __syncwarp();
    }
}

// Whether a fit can take the specialised kernels: ACF model, step mode,
// shared constants (window offsets allowed: OFF), OLS or GLS, N, D, G free
// in that order and every other parameter held at zero (tirf_zero_held:
// checked by the caller on the host copy of the initial values).
bool lm_tirf_applies(const FitArgs &a, bool tirf_zero_held)
{
    return tirf_zero_held && a.model == IMFCS_MODEL_ACF_1D && a.npts <= kMaxPts && a.tol == 0.f && !a.cst &&
           (!a.linv || a.npts <= 96) && a.k == 3 && a.idx[0] == 0 && a.idx[1] == 1 && a.idx[2] == 4 &&
           a.np == IMFCS_NPARAM;
}

cudaError_t launch_lm_tirf(const FitArgs &a, int blocks, int threads, cudaStream_t s)
{
    // Three points of a lane side by side shorten a fit's chain but fill the
    // instruction caches: 64 fits 78 -> 72 us, 441 97 -> 89, 2,304 510 -> 507,
    // 16,384 (the SMs full) 401 -> 449
    if (a.mc.rx != 0.f || a.mc.ry != 0.f) lm_tirf_kernel<true, false><<<blocks, threads, 0, s>>>(a);
    else if (a.nfits <= 4096) lm_tirf_kernel<false, true><<<blocks, threads, 0, s>>>(a);
    else lm_tirf_kernel<false, false><<<blocks, threads, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace imfcs
