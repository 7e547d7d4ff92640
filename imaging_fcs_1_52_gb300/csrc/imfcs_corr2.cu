// imfcs_corr2.cu -- multi-tau correlator with blocked variance as a chain of
// streaming kernels, no block-wide synchronisation.
//
// Restates calculateCF (Imaging_FCS_1_52.java:9425-9648) with the same
// per-lag block statistics and outputs as corr_kernel:
//
//   values    the binned, background-subtracted, bleach-corrected and
//             centred value of every (trace, frame) is written once as FP32,
//             frame-major ([t][pixel]): the level-0 sample stream s0;
//   pair k    one thread per (pixel, frame segment) streams the level-k
//             samples and correlates levels k and k+1 (lags 0..16 at level 0,
//             delays 9..16 above) in registers: a window of 32 samples that
//             moves by register copies every 16, so that one step's code
//             serves every step; it writes the level-(k+2) samples (pair sums
//             of its level-(k+1) samples) for the next kernel;
//   tail      levels k0..Q-1 (blocks possibly one sample long): one level per
//             thread, samples built from the level-k0 stream, block
//             statistics in registers;
//   finalise  per (pixel, lag): segments combined at FP64 precision, outputs.
//
// Products are grouped by their direct sample y (processed when the delayed
// samples y..y+16 are present), so the blocks of the blocked variance
// (2^(ind-k) products, java:9502-9511) end at the same y for every lag of a
// level.  With the window means a, b of the centred samples from the monitor
// pass, the blocked product of block z is
//   P_z = (A_z - b B_z - a D_z + L a b) / L
// (A_z: sum of products, B_z: sum of direct samples, D_z: sum of the delayed
// samples y+d over the block, from the block's running sum and the "heads",
// the sums of the first d delayed samples of a block).  Frame segments are
// multiples of every pixel's block length (2^ind frames), so no block spans
// two threads; each segment keeps its own statistics.
#include "imfcs_corr.cuh"

namespace imfcs {

constexpr int kC2Threads = 64;       // pixels per CTA unless the tile says 32
constexpr int kMaxSegExtra = 4;

// Arguments shared by the pair, tail and finalise kernels.
struct C2Args {
    CorrOut o;
    const float4 *mon;        // [pix][chanum] (a, b, dm, Dm)
    const int *blk_ind;       // [pix]
    const LagInfo *li;
    int npix, chanum, p, q, num;
    int numbin[kMaxLevels];
    int seg_log[kMaxLevels];  // frame segment (log2) of the kernel owning each level
    size_t stat_stride;       // floats per segment in o.stats
};

// The blocked product of one block of one lag, (A - b B - a D + L a b) / L,
// with L a power of two (iL = 1/L and L a are exact).
__device__ __forceinline__ float block_product(float A, float B, float D, float a, float b, float L, float iL)
{
    return fmaf(L * a, b, fmaf(-a, D, fmaf(-b, B, A))) * iL;
}

// ---------------------------------------------------------------------------
// Pair kernel: levels k (first) and k+1 (second) of one (pixel, segment).
// FIRST17: the first level is level 0 (lags 0..16); otherwise its lags are
// delays 9..16.  TWO: the second level exists (k+1 < Q).
//
// A step takes the 16 first-level direct samples from y0 on with the 32
// samples from y0 on in registers (the next 16 already loading), and the
// eight second-level direct samples of the step before, whose delayed samples
// are then complete.  Both windows move by register copies, so one step's
// code, 336 FMAs for levels 0-1, serves every step and block ends are in it
// once.  What only block ends touch -- totals, statistics, heads -- is in
// shared memory, the monitors and the statistics' shift in the L1.
// Bound by issue (60 % active at 12 warps an SM, 44 instructions a frame and
// pixel of which 25 are the products): 2.90 -> 1.48 ms for levels 0-1 and 0.85
// -> 0.46 for 2-3 at 16,384 pixels x 50,000 frames against four unrolled
// copies of the step with 32-entry rings and per-lag head sums.
// ---------------------------------------------------------------------------
constexpr int kPairFields = 5;    // per lag in shared memory: Ahi, Alo, S1, S2, head

// Fields of one thread: lag l of the pass, field f at sm[(l * kPairFields + f) * NT].
template <int NT>
struct PairBlocks {
    float *sm;
    const float4 *mon;        // this pixel's monitors from the pass's first lag on
    float *rst;               // this (segment, pixel)'s shift of the first lag's statistics
    float *bprod;             // this pixel's products of the first lag, or nullptr
    int npix, pnum_stride, pnum, zfirst;
    bool skip0;               // the pass's first lag is lag 0 (no product kept)
    __device__ __forceinline__ float &at(int l, int f) { return sm[(l * kPairFields + f) * NT]; }

    // The block z of N lags from lag l0 of the pass on: acc the products' sums
    // (cleared), B and Bd the sums of the direct and undelayed samples, nh the
    // sums of the first d samples of the next block per lag.
    template <int N>
    __device__ __forceinline__ void end(int l0, float (&acc)[N], float B, float Bd, const float (&nh)[N], int L, int z)
    {
        const float fL = (float)L, iL = 1.f / fL;
        const bool stat = z < pnum, first = z == zfirst;
        constexpr int kBatch = 6;          // lags whose monitors and shifts load together
#pragma unroll
        for (int lb = 0; lb < N; lb += kBatch) {
            float2 m[kBatch];
            float r[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                if (lb + u >= N) break;
                m[u] = __ldg((const float2 *)&mon[l0 + lb + u]);
                r[u] = stat && !first ? rst[(size_t)(l0 + lb + u) * kStatN * npix] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                if (lb + u >= N) break;
                const int l = lb + u, s = l0 + l;
                const float P = block_product(acc[l], B, Bd - at(s, 4) + nh[l], m[u].x, m[u].y, fL, iL);
                ff t = {at(s, 0), at(s, 1)};
                ff_add(t, acc[l]);
                at(s, 0) = t.hi;
                at(s, 1) = t.lo;
                at(s, 4) = nh[l];
                acc[l] = 0.f;
                if (stat) {
                    if (first) {                    // the segment's shift of the block statistics
                        rst[(size_t)s * kStatN * npix] = P;
                    } else {
                        const float dv = P - r[u];
                        at(s, 2) += dv;
                        at(s, 3) = fmaf(dv, dv, at(s, 3));
                    }
                    if (bprod && !(skip0 && s == 0)) bprod[(size_t)s * pnum_stride + z] = P;
                }
            }
        }
    }
};

// Sixteen samples n .. n+15 of a level's stream (0 from nk on).
__device__ __forceinline__ void load16(float (&v)[16], const float *in, int n, int nk, int npix)
{
    const float *p = in + (size_t)n * npix;
    if (n + 16 <= nk) {
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = __ldg(&p[(size_t)i * npix]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = n + i < nk ? __ldg(&p[(size_t)i * npix]) : 0.f;
    }
}

// PART: the pass's share of the lags -- 0 all, 1 the first level's (level 0:
// its lags 0..8), 2 the second level's, with the samples it passes on, 3 lags
// 9..16 of level 0.
template <bool CCF, bool FIRST17, bool TWO, int NT, int PART>
struct PairShare {
    static constexpr int FB = PART == 3 ? 9 : 0;                      // first-level lags: from FB on,
    static constexpr int NF = PART == 2 ? 0 : PART == 3 ? 8 : PART == 1 && FIRST17 ? 9 : FIRST17 ? kP + 1 : 8;
    static constexpr int DF = (FIRST17 ? 0 : 9) + FB;                 // the delay of the first of them
    static constexpr bool SECOND = TWO && (PART == 0 || PART == 2);
    static constexpr int NS = SECOND ? 8 : 0;
    static constexpr int LAG = PART == 2 ? (FIRST17 ? kP + 1 : 8) : FB;   // the share's first lag in the pair's
    static constexpr int SMEM = (NF + NS) * kPairFields * NT;
};

template <bool CCF, bool FIRST17, bool TWO, int NT, int PART>
__device__ __forceinline__ void pair_body(const C2Args &a, const float *inA, const float *inB, float *outA,
                                          float *outB, int k, float *sm)
{
    using Share = PairShare<CCF, FIRST17, TWO, NT, PART>;
    constexpr int NF = Share::NF, DF = Share::DF, NS = Share::NS;
    constexpr bool SECOND = Share::SECOND;
    constexpr int NFA = NF ? NF : 1;
    const int tid = threadIdx.x;
    const int pix = blockIdx.x * NT + tid, seg = blockIdx.y;
    const int s0 = seg << a.seg_log[k];
    if (pix >= a.npix || s0 >= a.num) return;          // no block-wide synchronisation below
    const int s1 = s0 + (1 << a.seg_log[k]);
    const int nk = a.numbin[k], nk1 = TWO ? a.numbin[k + 1] : 0;
    const int nk2 = (TWO && k + 2 < a.q) ? a.numbin[k + 2] : 0;
    const int y0 = s0 >> k, y1 = s1 >= a.num ? nk : (s1 >> k);      // direct samples of level k
    const int ind = a.blk_ind[pix];
    const int LF = 1 << (ind - k), LS = 1 << (ind - k - 1);
    const int lag0 = (FIRST17 ? 0 : (kP + 1) + (k - 1) * 8) + Share::LAG;
    float *gst = a.o.stats + (size_t)seg * a.stat_stride;
    PairBlocks<NT> pb;
    pb.sm = sm + tid;
    pb.mon = a.mon + (size_t)pix * a.chanum + lag0;
    pb.rst = &stat_ref(gst, a.npix, lag0, 4, pix);
    pb.bprod = a.o.gls ? a.o.bprod + ((ptrdiff_t)pix * (a.chanum - 1) + (lag0 - 1)) * a.o.pnum_stride : nullptr;
    pb.npix = a.npix;
    pb.pnum_stride = a.o.pnum_stride;
    pb.pnum = a.li->pnum_by_ind[ind];
    pb.zfirst = s0 >> ind;
    pb.skip0 = FIRST17 && Share::LAG == 0;
#pragma unroll
    for (int l = 0; l < NF + NS; l++)
#pragma unroll
        for (int f = 0; f < kPairFields; f++) pb.at(l, f) = 0.f;
    // a segment without a counted block leaves its shift zero
    if (pb.zfirst >= pb.pnum)
        for (int l = 0; l < NF + NS; l++) pb.rst[(size_t)l * kStatN * a.npix] = 0.f;
    inA += pix;
    inB += pix;
    if (outB) {
        outA += pix;
        outB += pix;
    }

    float w[32], cur[16];              // first-level samples y .. y+31; the next 16, loading
    float x[16];                       // CCF: direct-trace samples y .. y+15
    float r[24], rx[8];                // second-level samples y/2-8 .. y/2+15; CCF: direct ones y/2-8 .. y/2-1
    float accF[NFA], accS[8];
    float bF = 0.f, bFd = 0.f, bS = 0.f, bSd = 0.f;
#pragma unroll
    for (int l = 0; l < NF; l++) accF[l] = 0.f;
#pragma unroll
    for (int l = 0; l < 8; l++) accS[l] = 0.f;
#pragma unroll
    for (int i = 0; i < 24; i++) r[i] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) rx[i] = 0.f;
    load16(cur, inB, y0, nk, a.npix);
#pragma unroll
    for (int i = 0; i < 16; i++) w[16 + i] = cur[i];
    load16(cur, inB, y0 + 16, nk, a.npix);
    // heads of the first blocks, and the second level's first eight samples
    {
        float h = 0.f;
        if (DF == 0 && NF) pb.at(0, 4) = 0.f;
#pragma unroll
        for (int d = 1; d <= kP; d++) {
            h += w[16 + d - 1];
            if (d >= DF && d < DF + NF) pb.at(d - DF, 4) = h;
        }
        if (SECOND)
#pragma unroll
            for (int i = 0; i < 8; i++) r[16 + i] = (y0 >> 1) + i < nk1 ? w[16 + 2 * i] + w[17 + 2 * i] : 0.f;
    }
    // one step more than first-level steps: the second level is a step behind
    const int ysteps = y0 + ((y1 - y0 + 15) & ~15);
#pragma unroll 1
    for (int y = y0; y < ysteps + (SECOND ? 16 : 0); y += 16) {
        const bool first_level = y < ysteps;
        const bool second_level = SECOND && y > y0;
        float xn[8];                   // CCF: second-level direct samples of this step
#pragma unroll
        for (int i = 0; i < 16; i++) {
            w[i] = w[16 + i];
            w[16 + i] = cur[i];
        }
        if (CCF) load16(x, inA, y, nk, a.npix);
        load16(cur, inB, y + 32, nk, a.npix);
        if (SECOND) {
#pragma unroll
            for (int i = 0; i < 16; i++) r[i] = r[i + 8];
#pragma unroll
            for (int i = 0; i < 8; i++) r[16 + i] = (y >> 1) + 8 + i < nk1 ? w[16 + 2 * i] + w[17 + 2 * i] : 0.f;
            if (CCF)
#pragma unroll
                for (int i = 0; i < 8; i++) xn[i] = (y >> 1) + i < nk1 ? x[2 * i] + x[2 * i + 1] : 0.f;
        }
        if (first_level) {
            if (NF)
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const float d = CCF ? x[j] : w[j];
#pragma unroll
                for (int l = 0; l < NF; l++) accF[l] = fmaf(d, w[j + DF + l], accF[l]);
                bF += d;
                if (CCF) bFd += w[j];
            }
            if (SECOND && outB) {      // level k+2: pair sums of second-level samples y/2 .. y/2+7
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int m = (y >> 2) + i;
                    if (m < nk2 && m < (s1 >> (k + 2))) {
                        outB[(size_t)m * a.npix] = r[8 + 2 * i] + r[9 + 2 * i];
                        if (CCF) outA[(size_t)m * a.npix] = xn[2 * i] + xn[2 * i + 1];
                    }
                }
            }
            if (NF && ((y + 16) & (LF - 1)) == 0) {
                float nh[NFA], h = 0.f;
                if (DF == 0) nh[0] = 0.f;
#pragma unroll
                for (int d = 1; d <= kP; d++) {
                    h += w[16 + d - 1];
                    if (d >= DF && d < DF + NF) nh[d - DF] = h;
                }
                pb.template end<NFA>(0, accF, bF, CCF ? bFd : bF, nh, LF, (y + 16) / LF - 1);
                bF = 0.f;
                bFd = 0.f;
            }
        }
        if (second_level) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float d = CCF ? rx[i] : r[i];
#pragma unroll
                for (int l = 0; l < 8; l++) accS[l] = fmaf(d, r[i + 9 + l], accS[l]);
                bS += d;
                if (CCF) bSd += r[i];
            }
            if (((y >> 1) & (LS - 1)) == 0) {
                float nh[8], h = 0.f;
#pragma unroll
                for (int d = 1; d <= 16; d++) {
                    h += r[8 + d - 1];
                    if (d >= 9) nh[d - 9] = h;
                }
                pb.template end<8>(NF, accS, bS, CCF ? bSd : bS, nh, LS, (y >> 1) / LS - 1);
                bS = 0.f;
                bSd = 0.f;
            }
        } else if (SECOND) {           // the first step: heads of the second level's first block
            float h = 0.f;
#pragma unroll
            for (int d = 1; d <= 16; d++) {
                h += r[8 + d - 1];
                if (d >= 9) pb.at(NF + d - 9, 4) = h;
            }
        }
        if (CCF && SECOND)
#pragma unroll
            for (int i = 0; i < 8; i++) rx[i] = xn[i];
    }
    // the partial blocks at the end into the totals; everything out
#pragma unroll
    for (int l = 0; l < NF + NS; l++) {
        ff t = {pb.at(l, 0), pb.at(l, 1)};
        ff_add(t, l < NF ? accF[l < NF ? l : 0] : accS[l < NF ? 0 : l - NF]);
        stat_ref(gst, a.npix, lag0 + l, 0, pix) = t.hi;
        stat_ref(gst, a.npix, lag0 + l, 1, pix) = t.lo;
        stat_ref(gst, a.npix, lag0 + l, 2, pix) = pb.at(l, 2);
        stat_ref(gst, a.npix, lag0 + l, 3, pix) = pb.at(l, 3);
    }
}

template <bool CCF, bool FIRST17, bool TWO, int NT>
__global__ void __launch_bounds__(NT, 384 / NT) c2_pair_kernel(C2Args a, const float *inA, const float *inB,
                                                     float *outA, float *outB, int k)
{
    __shared__ float sm[PairShare<CCF, FIRST17, TWO, NT, 0>::SMEM];
    pair_body<CCF, FIRST17, TWO, NT, 0>(a, inA, inB, outA, outB, k, sm);
}

// The same with a pair's lags dealt out to two or three blocks (blockIdx.z),
// each reading the samples for itself: for grids that leave the SMs part-empty,
// where a block's time is the latency of its instructions.  The sums are per
// lag, so they stay what they are.
template <bool CCF, bool FIRST17, int NT>
__global__ void __launch_bounds__(NT, 384 / NT) c2_pair_split_kernel(C2Args a, const float *inA, const float *inB,
                                                           float *outA, float *outB, int k)
{
    __shared__ float sm[9 * kPairFields * NT];
    if (blockIdx.z == 0) pair_body<CCF, FIRST17, true, NT, 2>(a, inA, inB, outA, outB, k, sm);
    else if (blockIdx.z == 1) pair_body<CCF, FIRST17, true, NT, 1>(a, inA, inB, outA, outB, k, sm);
    else if (FIRST17) pair_body<CCF, FIRST17, true, NT, FIRST17 ? 3 : 1>(a, inA, inB, outA, outB, k, sm);
}

// ---------------------------------------------------------------------------
// Tail kernel: one level k >= k0 of one (pixel, segment) per thread, for the
// top levels whose blocks may be as short as one sample.  The thread builds
// its level-k samples from the level-k0 stream (pairwise sums of 2^(k-k0)
// samples), 16 a step, with the 32 samples from the step's first on, its lags'
// block sums and block statistics in registers; the statistics are written
// once.  1.65 -> 0.73 ms at 16,384 pixels x 50,000 frames against a ring in
// shared memory read sample by sample.
// ---------------------------------------------------------------------------
// Samples n .. n+15 of level k0 + LM (0 from nkk on), pairwise sums of the
// level-k0 stream (java:9467-9476).
template <int LM>
__device__ __forceinline__ void tail_samples(float *v, const float *in, int n, int nkk, int npix)
{
    constexpr int M = 1 << LM;
#pragma unroll
    for (int u = 0; u < 16; u++) {
        float t[M];
        const bool inside = n + u < nkk;
        const float *p = in + (size_t)(n + u) * M * npix;
#pragma unroll
        for (int i = 0; i < M; i++) t[i] = inside ? __ldg(&p[(size_t)i * npix]) : 0.f;
#pragma unroll
        for (int h = M / 2; h >= 1; h /= 2)
#pragma unroll
            for (int i = 0; i < h; i++) t[i] = t[2 * i] + t[2 * i + 1];
        v[u] = t[0];
    }
}
__device__ __forceinline__ void tail_load(float *v, const float *in, int n, int lm, int nkk, int npix)
{
    if (lm == 0) tail_samples<0>(v, in, n, nkk, npix);
    else if (lm == 1) tail_samples<1>(v, in, n, nkk, npix);
    else if (lm == 2) tail_samples<2>(v, in, n, nkk, npix);
    else tail_samples<3>(v, in, n, nkk, npix);
}

template <bool CCF, int NT>
__global__ void __launch_bounds__(NT, 512 / NT) c2_tail_kernel(C2Args a, const float *inA, const float *inB, int k0)
{
    __shared__ float2 mon_sm[8 * NT];               // the lags' monitors
    const int tid = threadIdx.x;
    const int pix = blockIdx.x * NT + tid, seg = blockIdx.y, k = k0 + blockIdx.z;
    const int s0 = seg << a.seg_log[k];
    if (pix >= a.npix || k >= a.q || s0 >= a.num) return;          // no block-wide synchronisation below
    const int s1 = min(s0 + (1 << a.seg_log[k]), a.num);
    const int nkk = a.numbin[k], lm = k - k0;
    const int ys0 = s0 >> k, ys1 = (s1 >= a.num) ? nkk : (s1 >> k);
    const int lag0 = (kP + 1) + (k - 1) * 8;
    const int ind = a.blk_ind[pix], pnum = a.li->pnum_by_ind[ind], zfirst = s0 >> ind;
    const int L = ind > k ? 1 << (ind - k) : 1, logL = ind > k ? ind - k : 0;
    const float fL = (float)L, iL = 1.f / fL;
    float *bprod = a.o.gls ? a.o.bprod + ((size_t)pix * (a.chanum - 1) + (lag0 - 1)) * a.o.pnum_stride : nullptr;
    inA += pix;
    inB += pix;
    float2 *ms = mon_sm + tid;
#pragma unroll
    for (int l = 0; l < 8; l++) ms[l * NT] = __ldg((const float2 *)&a.mon[(size_t)pix * a.chanum + lag0 + l]);

    float acc[8], head[8], thi[8], tlo[8], S1[8], S2[8], rr[8];
#pragma unroll
    for (int l = 0; l < 8; l++) acc[l] = thi[l] = tlo[l] = S1[l] = S2[l] = rr[l] = 0.f;
    float b0 = 0.f, b1 = 0.f;
    float w[32], x[16];
    tail_load(w + 16, inB, ys0, lm, nkk, a.npix);
    {
        float h = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            h += w[16 + i];
            if (i + 1 >= 9) head[i + 1 - 9] = h;
        }
    }
#pragma unroll 1
    for (int y = ys0; y < ys1; y += 16) {
#pragma unroll
        for (int i = 0; i < 16; i++) w[i] = w[16 + i];
        tail_load(w + 16, inB, y + 16, lm, nkk, a.npix);
        if (CCF) tail_load(x, inA, y, lm, nkk, a.npix);
        // a segment may end inside the step
        const int left = ys1 - y;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            if (j >= left) break;
            const float d = CCF ? x[j] : w[j];
#pragma unroll
            for (int l = 0; l < 8; l++) acc[l] = fmaf(d, w[j + 9 + l], acc[l]);
            b0 += d;
            if (CCF) b1 += w[j];
            if (((y + j + 1) & (L - 1)) == 0) {
                // heads of the next block: sums of the delayed samples y+j+1 .. y+j+d
                float h = 0.f;
#pragma unroll
                for (int i = 1; i <= 8; i++) h += w[j + i];
                const int z = (y + j) >> logL;
                const bool stat = z < pnum;
#pragma unroll
                for (int l = 0; l < 8; l++) {
                    h += w[j + 9 + l];
                    const float2 m = ms[l * NT];
                    const float P = block_product(acc[l], b0, (CCF ? b1 : b0) - head[l] + h, m.x, m.y, fL, iL);
                    ff t = {thi[l], tlo[l]};
                    ff_add(t, acc[l]);
                    thi[l] = t.hi;
                    tlo[l] = t.lo;
                    if (stat) {
                        if (z == zfirst) rr[l] = P;
                        const float dv = P - rr[l];
                        S1[l] += dv;
                        S2[l] = fmaf(dv, dv, S2[l]);
                        if (bprod) bprod[(size_t)l * a.o.pnum_stride + z] = P;
                    }
                    head[l] = h;
                    acc[l] = 0.f;
                }
                b0 = 0.f;
                b1 = 0.f;
            }
        }
    }
    float *gst = a.o.stats + (size_t)seg * a.stat_stride;
#pragma unroll
    for (int l = 0; l < 8; l++) {
        ff t = {thi[l], tlo[l]};
        ff_add(t, acc[l]);
        stat_ref(gst, a.npix, lag0 + l, 0, pix) = t.hi;
        stat_ref(gst, a.npix, lag0 + l, 1, pix) = t.lo;
        stat_ref(gst, a.npix, lag0 + l, 2, pix) = S1[l];
        stat_ref(gst, a.npix, lag0 + l, 3, pix) = S2[l];
        stat_ref(gst, a.npix, lag0 + l, 4, pix) = rr[l];
    }
}

// ---------------------------------------------------------------------------
// P = 32 (java:1022-1024): level 0 has delays 0..32, every upper level delays
// 17..32 (java:7391-7424), more than the pair kernels' rings hold.  Pixels go
// in chunks whose scratch stays bounded; per chunk
//   cg_levels_kernel    the binned sample streams of levels 1..Q-1 from s0;
//   cg_blocks_kernel    one (pixel, frame segment, level, up to 17 delays) per
//                       thread: the blocked products P_z of every block and
//                       the segment's product totals;
//   cg_finalize_kernel  per (pixel, lag) the block statistics over all blocks
//                       in order, the totals, the outputs.
// Blocks are independent of each other, so the frame segments run in
// parallel; only the statistics, a few operations per block, follow the order
// of the blocks.  48x48x20,000: 10.4 ms with one thread per (pixel, level,
// 8 delays) over the whole recording -- two warps an SM at work, each summing
// its samples from s0 again -- to 0.56 ms (blocks) + 0.06 (levels) + 0.08
// (finalise).  A chunk's scratch (level streams and products, some 400 KB a
// pixel at 50,000 frames and Q = 8) stays below 512 MB, with 64 pixels at
// least; bands under a tight budget grant it what is left.
// ---------------------------------------------------------------------------
constexpr int kCgDelays = 17;                 // delays per thread: 0..16 and 17..32
constexpr int kCgStep = 16;                   // samples per step of a thread
constexpr size_t kCgChunkBytes = (size_t)512 << 20;   // scratch of a pixel chunk

struct CgArgs {
    CorrOut o;
    const float4 *mon;        // [pix][chanum]
    const int *blk_ind;       // [pix]
    const LagInfo *li;
    int npix, p0, np, cs;     // all pixels; the chunk's first pixel, pixels and stride
    int chanum, p, q, num, nseg, pnum_max;
    int numbin[kMaxLevels], seg_log[kMaxLevels];
    const float *s0a, *s0b;   // [frame][npix]
    float *lva, *lvb;         // levels 1..Q-1 of the chunk: [sample][cs] at lv_off
    size_t lv_off[kMaxLevels];
    float *pz;                // [lag][pnum_max][cs] blocked products
    float2 *tot;              // [segment][lag][cs] product totals
};

// Level-k samples (k = 1..3 pairwise, java:9467-9476; above, the level-3
// samples of a sample added in order), 2^(Q-1) frames at a time per thread;
// the blocks of grid.y stride over a long recording's spans.
template <bool CCF>
__global__ void __launch_bounds__(128) cg_levels_kernel(CgArgs a)
{
    const int pc = blockIdx.x * 128 + threadIdx.x;
    if (pc >= a.np) return;
    const int span = 1 << max(a.q - 1, 3);
    for (int f0 = blockIdx.y * span; f0 < a.num; f0 += gridDim.y * span)
        for (int tr = 0; tr < (CCF ? 2 : 1); tr++) {
            const float *in = (tr ? a.s0b : a.s0a) + a.p0 + pc;
            float *lv = (tr ? a.lvb : a.lva) + pc;
            float up[kMaxLevels];             // running sums of levels 4..Q-1
#pragma unroll
            for (int k = 4; k < 8; k++) up[k] = 0.f;
            for (int f = f0; f < f0 + span && f < a.num; f += 8) {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = f + i < a.num ? __ldg(&in[(size_t)(f + i) * a.npix]) : 0.f;
#pragma unroll
                for (int k = 1; k <= 3; k++) {
#pragma unroll
                    for (int i = 0; i < (8 >> k); i++) {
                        v[i] = v[2 * i] + v[2 * i + 1];
                        const int n = (f >> k) + i;
                        if (k < a.q && n < a.numbin[k]) lv[a.lv_off[k] + (size_t)n * a.cs] = v[i];
                    }
                }
#pragma unroll
                for (int k = 4; k < 8; k++) {
                    if (k >= a.q) break;
                    up[k] += v[0];
                    if (((f + 8) & ((1 << k) - 1)) == 0) {
                        const int n = f >> k;
                        if (n < a.numbin[k]) lv[a.lv_off[k] + (size_t)n * a.cs] = up[k];
                        up[k] = 0.f;
                    }
                }
            }
        }
}

// One level's samples of one pixel.
struct CgStream {
    const float *p;
    int n, stride;
    __device__ __forceinline__ float at(int i) const { return i < n ? __ldg(&p[(size_t)i * stride]) : 0.f; }
};

// State of one thread: block sums of its delays dlo .. dlo + nd - 1.  What
// only block ends touch -- the heads and the product totals -- is in shared
// memory (this thread's column of [field][delay][thread]).
constexpr int kCgThreads = 64;
struct CgThread {
    float acc[kCgDelays];
    float b0, b1;
    float *sm;
    int dlo, nd, lag0, L, pnum, pc;
    __device__ __forceinline__ float &head(int l) { return sm[l * kCgThreads]; }
    __device__ __forceinline__ float &thi(int l) { return sm[(kCgDelays + l) * kCgThreads]; }
    __device__ __forceinline__ float &tlo(int l) { return sm[(2 * kCgDelays + l) * kCgThreads]; }
    // sums of the d samples after sample y, for every delay d of the thread
    __device__ __forceinline__ void heads(const CgStream &b, int y, float (&h)[kCgDelays]) const
    {
        float v[kCgDelays], s = 0.f;
        if (dlo) {                        // all loads before their sums: one latency, not one each
#pragma unroll
            for (int i = 1; i < kCgDelays; i++) v[i] = b.at(y + i);
#pragma unroll
            for (int i = 1; i < kCgDelays; i++) s += v[i];
        }
#pragma unroll
        for (int l = 0; l < kCgDelays; l++) v[l] = l < nd && dlo + l > 0 ? b.at(y + dlo + l) : 0.f;
#pragma unroll
        for (int l = 0; l < kCgDelays; l++) {
            s += v[l];
            h[l] = s;
        }
    }
    // the block ending at direct sample y
    __device__ __forceinline__ void block_end(const CgArgs &a, const CgStream &b, const float4 *mon, int y)
    {
        float nh[kCgDelays];
        heads(b, y, nh);
        const int z = y / L;
        float2 mw[kCgDelays];
#pragma unroll
        for (int l = 0; l < kCgDelays; l++) mw[l] = __ldg((const float2 *)&mon[lag0 + min(l, nd - 1)]);
#pragma unroll
        for (int l = 0; l < kCgDelays; l++) {
            if (l < nd) {
                const float2 mm = mw[l];
                const float D = b1 - head(l) + nh[l];
                const float Pz = (acc[l] - mm.y * b0 - mm.x * D + (float)L * mm.x * mm.y) / (float)L;
                ff t = {thi(l), tlo(l)};
                ff_add(t, acc[l]);
                thi(l) = t.hi;
                tlo(l) = t.lo;
                if (z < pnum) a.pz[((size_t)(lag0 + l) * a.pnum_max + z) * a.cs + pc] = Pz;
                head(l) = nh[l];
                acc[l] = 0.f;
            }
        }
        b0 = 0.f;
        b1 = 0.f;
    }
};

// Grid (pixel blocks, level items, frame segments).  Item 0, 1: level 0,
// delays 0..16 and 17..32; item 1 + k: level k.  Sixteen samples at a time
// with the delayed samples in registers where no block ends inside them
// (blocks of 16 samples and more); shorter blocks, at the upper levels, take
// their samples one by one.  Issue-bound: 17 FMAs and 3 loads a sample.
template <bool CCF>
__global__ void __launch_bounds__(kCgThreads, 6) cg_blocks_kernel(CgArgs a)
{
    __shared__ float sm[3 * kCgDelays * kCgThreads];
    const int pc = blockIdx.x * kCgThreads + threadIdx.x;
    const int item = blockIdx.y, seg = blockIdx.z;
    const int k = item < 2 ? 0 : item - 1;
    const int s0 = seg << a.seg_log[k];
    if (pc >= a.np || s0 >= a.num) return;
    const int pix = a.p0 + pc;
    const int s1 = min(s0 + (1 << a.seg_log[k]), a.num);
    const int nk = a.numbin[k];
    const int ys0 = s0 >> k, ys1 = (s1 >= a.num) ? nk : (s1 >> k);
    CgStream sb, sa;
    if (k == 0) {
        sb = {a.s0b + pix, nk, a.npix};
        sa = {a.s0a + pix, nk, a.npix};
    } else {
        sb = {a.lvb + a.lv_off[k] + pc, nk, a.cs};
        sa = {a.lva + a.lv_off[k] + pc, nk, a.cs};
    }
    const int ind = a.blk_ind[pix];
    CgThread t;
    t.sm = sm + threadIdx.x;
    t.pc = pc;
    t.dlo = item == 0 ? 0 : a.p / 2 + 1;
    t.nd = item == 0 ? a.p / 2 + 1 : a.p / 2;
    t.lag0 = item < 2 ? t.dlo : (a.p + 1) + (k - 1) * (a.p / 2);
    t.L = ind > k ? 1 << (ind - k) : 1;
    t.pnum = a.li->pnum_by_ind[ind];
    t.b0 = t.b1 = 0.f;
#pragma unroll
    for (int l = 0; l < kCgDelays; l++) t.acc[l] = t.thi(l) = t.tlo(l) = 0.f;
    {
        float h[kCgDelays];
        t.heads(sb, ys0 - 1, h);
#pragma unroll
        for (int l = 0; l < kCgDelays; l++) t.head(l) = h[l];
    }
    const float4 *mon = a.mon + (size_t)pix * a.chanum;

    float w[kCgDelays - 1 + kCgStep];      // delayed samples y + dlo ...
#pragma unroll
    for (int i = 0; i < kCgDelays - 1; i++) w[i] = sb.at(ys0 + t.dlo + i);
#pragma unroll 1
    for (int y = ys0; y < ys1; y += kCgStep) {
#pragma unroll
        for (int j = 0; j < kCgStep; j++) w[kCgDelays - 1 + j] = sb.at(y + t.dlo + kCgDelays - 1 + j);
        if (t.L >= kCgStep && y + kCgStep <= ys1) {
            float x[kCgStep], v[kCgStep];
#pragma unroll
            for (int j = 0; j < kCgStep; j++) {
                v[j] = sb.at(y + j);
                x[j] = CCF ? sa.at(y + j) : v[j];
            }
#pragma unroll
            for (int j = 0; j < kCgStep; j++) {
#pragma unroll
                for (int l = 0; l < kCgDelays; l++) t.acc[l] = fmaf(x[j], w[j + l], t.acc[l]);
                t.b0 += x[j];
                t.b1 += v[j];
            }
            if (((y + kCgStep) & (t.L - 1)) == 0) t.block_end(a, sb, mon, y + kCgStep - 1);
        } else {
            const int ye = min(y + kCgStep, ys1);
#pragma unroll 1
            for (int yy = y; yy < ye; yy++) {
                float d[kCgDelays];
                const float x = sa.at(yy), v = sb.at(yy);
#pragma unroll
                for (int l = 0; l < kCgDelays; l++) d[l] = sb.at(yy + t.dlo + l);
#pragma unroll
                for (int l = 0; l < kCgDelays; l++) t.acc[l] = fmaf(x, d[l], t.acc[l]);
                t.b0 += x;
                t.b1 += v;
                if (((yy + 1) & (t.L - 1)) == 0) t.block_end(a, sb, mon, yy);
            }
        }
#pragma unroll
        for (int i = 0; i < kCgDelays - 1; i++) w[i] = w[i + kCgStep];
    }
#pragma unroll
    for (int l = 0; l < kCgDelays; l++)
        if (l < t.nd) {
            ff u = {t.thi(l), t.tlo(l)};
            ff_add(u, t.acc[l]);                 // the partial block at the end
            a.tot[((size_t)seg * a.chanum + t.lag0 + l) * a.cs + pc] = make_float2(u.hi, u.lo);
        }
}

// ---------------------------------------------------------------------------
// Finalise: segments combined per (pixel, lag): product totals, block
// statistics brought to one shift (FP64), outputs as calculateCF
// (java:9491-9531).
// ---------------------------------------------------------------------------
// Outputs of one (pixel, lag) from its product total A and the statistics of
// its pnum blocked products (sums S1, S2 shifted by r), FP64.
__device__ __forceinline__ void write_lag(const CorrOut &o, const float4 *mon, const LagInfo *li, int chanum, int pix,
                                          int lag, int ind, double A, double S1, double S2, double r)
{
    const float4 m = mon[(size_t)pix * chanum + lag];
    // a non-finite frame in the lag's windows: NaN, whatever the sums
    double acf = __longlong_as_double(0x7ff8000000000000ll), bv = acf, cov = acf;
    if (m.x == m.x && m.y == m.y) {
        const int pnum = li->pnum_by_ind[ind];
        const double n = f2d((float)li->prodnum[lag]), pn = f2d((float)pnum), ip = li->inv_pnum[ind];
        const double dmDm = f2d(m.z) * f2d(m.w), idm = rcp_near(dmDm, m.z * m.w);
        const double sumprod = fma(-(n * f2d(m.x)), f2d(m.y), A), in = li->inv_prodnum[lag];   // centred products
        const double mean = div_by(S1, pn, ip);
        if (lag == 1) cov = div_by(sumprod, n, in);
        bv = div_near(fma(-mean, mean, div_by(S2, pn, ip)), f2d((float)(pnum - 1)) * dmDm * dmDm,
                      li->inv_pnum1[ind] * idm * idm);
        if (o.gls) acf = div_near(fma(pn, r, S1), pn * dmDm, ip * idm);    // mcov (java:9526-9531)
        else acf = div_near(sumprod, n * dmDm, in * idm);
    }
    if (o.gls && lag == 0) acf = 0.0;
    if (o.acf) o.acf[(size_t)pix * chanum + lag] = acf;
    if (o.var) o.var[(size_t)pix * chanum + lag] = bv;
    if (o.sd) o.sd[(size_t)pix * chanum + lag] = bv == bv ? newton_sqrt(bv) : bv;
    if (lag == 1) {
        if (o.nb_mean) o.nb_mean[pix] = m.z;
        if (o.nb_cov) o.nb_cov[pix] = cov;
    }
}

// The segments combined in FP64 alone, for sums that left the FP32 range.
static __device__ __noinline__ void plain_segments(const float *st, size_t np, size_t stride, int nseg, int sl, int num,
                                                   int ind, int pnum, double r0, double &A, double &S1, double &S2)
{
    A = S1 = S2 = 0.0;
    for (int sg = 0; sg < nseg; sg++, st += stride) {
        A += (double)st[0] + (double)st[np];
        const int f0 = sg << sl, f1 = min(f0 + (1 << sl), num);
        const int cnt = min(pnum, (f1 + (1 << ind) - 1) >> ind) - (f0 >> ind);
        if (cnt <= 0) continue;
        const double d1 = st[2 * np], dr = (double)st[4 * np] - r0;
        S1 += d1 + cnt * dr;
        S2 += st[3 * np] + 2.0 * dr * d1 + cnt * dr * dr;
    }
}

// Grid (pixel blocks, lags).  Bound by FP64 issue (1/64 of the FP32 rate):
// plain sums of FP32 values run in three FP32 terms, no less precise than FP64,
// the products with the segments' shifts are FP64, conversions go to the
// integer pipe, quotients are corrected products with reciprocals.  0.56 -> 0.19
// ms at 16,384 pixels x 50,000 frames.  Float-float for those products too was
// no faster and moved results by 1e-13, enough to round some of the fits' FP32
// data and weights the other way.
__global__ void __launch_bounds__(128) c2_finalize_kernel(C2Args a)
{
    const int pix = blockIdx.x * 128 + threadIdx.x, lag = blockIdx.y;
    if (pix >= a.npix) return;
    const int ind = a.blk_ind[pix];
    const int pnum = a.li->pnum_by_ind[ind];
    const int level = lag <= a.p ? 0 : 1 + (lag - (a.p + 1)) / (a.p / 2);
    const int sl = a.seg_log[level];
    const int nseg = (a.num + (1 << sl) - 1) >> sl;
    const float *st = &stat_ref(a.o.stats, a.npix, lag, 0, pix);
    const size_t np = a.npix;
    const double r0 = f2d(__ldg(&st[4 * np]));      // segment 0 always has a counted block
    ff3 A = {0.f, 0.f, 0.f}, s1 = A, s2 = A;
    double S1 = 0.0, S2 = 0.0;
    const float4 m = a.mon[(size_t)pix * a.chanum + lag];
    const bool bad = m.x != m.x || m.y != m.y;      // a non-finite frame in the lag's windows: NaN, whatever the sums
    constexpr int U = 4;                            // segments whose statistics load together
    for (int sb = 0; sb < nseg && !bad; sb += U) {
        float v[U][kStatN];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int f = 0; f < kStatN; f++)
                v[u][f] = sb + u < nseg ? __ldg(&st[(size_t)u * a.stat_stride + f * np]) : 0.f;
        st += U * a.stat_stride;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int sg = sb + u;
            if (sg >= nseg) break;
            ff3_add(A, v[u][0]);
            ff3_add_low(A, v[u][1]);
            // the segment's blocks that count
            const int f0 = sg << sl, f1 = min(f0 + (1 << sl), a.num);
            const int cnt = min(pnum, (f1 + (1 << ind) - 1) >> ind) - (f0 >> ind);
            if (cnt <= 0) continue;
            // sums of P - r0 from those of P - r: with dr = r - r0,
            // S1 += s1 + cnt dr and S2 += s2 + dr (2 s1 + cnt dr)
            ff3_add(s1, v[u][2]);
            ff3_add(s2, v[u][3]);
            const double dr = f2d(v[u][4]) - r0, c = f2d((float)cnt);
            S1 = fma(c, dr, S1);
            S2 = fma(dr, fma(c, dr, f2d(2.f * v[u][2])), S2);
        }
    }
    S1 += ff3_val(s1);
    S2 += ff3_val(s2);
    double Ad = ff3_val(A);
    if (!(isfinite(A.hi) && isfinite(s1.hi) && isfinite(s2.hi)) && !bad)
        plain_segments(&stat_ref(a.o.stats, a.npix, lag, 0, pix), np, a.stat_stride, nseg, sl, a.num, ind, pnum, r0, Ad,
                       S1, S2);
    write_lag(a.o, a.mon, a.li, a.chanum, pix, lag, ind, Ad, S1, S2, r0);
}

// P = 32: the block statistics of one (pixel, lag) over its blocks in order
// (FP32, shifted by the first block), the segments' totals in three FP32 terms.
__global__ void __launch_bounds__(128) cg_finalize_kernel(CgArgs a)
{
    const int pc = blockIdx.x * 128 + threadIdx.x, lag = blockIdx.y;
    if (pc >= a.np) return;
    const int pix = a.p0 + pc;
    const int ind = a.blk_ind[pix];
    const int pnum = a.li->pnum_by_ind[ind];
    const float *pz = a.pz + (size_t)lag * a.pnum_max * a.cs + pc;
    const float r = pnum > 0 ? pz[0] : 0.f;
    // GLS takes the products themselves (lags 1 and up, [pixel][lag][block])
    float *bprod = a.o.gls && lag > 0
                       ? a.o.bprod + ((size_t)pix * (a.chanum - 1) + (lag - 1)) * a.o.pnum_stride : nullptr;
    float S1 = 0.f, S2 = 0.f;
    for (int z = 0; z < pnum; z += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = z + u < pnum ? pz[(size_t)(z + u) * a.cs] : r;
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (z + u < pnum) {
                const float dv = v[u] - r;
                S1 += dv;
                S2 = fmaf(dv, dv, S2);
                if (bprod) bprod[z + u] = v[u];
            }
    }
    const int sl = a.seg_log[lag <= a.p ? 0 : 1 + (lag - (a.p + 1)) / (a.p / 2)];
    const int nseg = (a.num + (1 << sl) - 1) >> sl;
    const float2 *tot = a.tot + (size_t)lag * a.cs + pc;
    const size_t tstride = (size_t)a.chanum * a.cs;
    ff3 At = {0.f, 0.f, 0.f};
    for (int sg = 0; sg < nseg; sg++) {
        const float2 t = tot[sg * tstride];
        ff3_add(At, t.x);
        ff3_add_low(At, t.y);
    }
    double A = ff3_val(At);
    if (!isfinite(At.hi)) {                         // beyond the FP32 range
        A = 0.0;
        for (int sg = 0; sg < nseg; sg++) {
            const float2 t = tot[sg * tstride];
            A += f2d(t.x) + f2d(t.y);
        }
    }
    write_lag(a.o, a.mon, a.li, a.chanum, pix, lag, ind, A, f2d(S1), f2d(S2), f2d(r));
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
// The chain needs blocks of at least 16 level-0 and 8 level-1 samples
// (ind >= Q-1 >= 4).
bool corr2_supported(const Job &j) { return j.p == kP && j.q >= 5; }
// P = 32 (any Q)
bool corrg_supported(const Job &j) { return j.p == 32; }

namespace {
struct Plan2 {
    int npair;                // pair kernels (levels 0-1, then 2-3 when Q >= 7)
    int k_tail;               // first level of the tail kernel (Q: none)
    int seg_log[kMaxLevels];
    int nseg_max;
};

Plan2 plan2(const Job &j)
{
    Plan2 p;
    // every pixel's block length divides 2^base0 frames; the tile multiplies
    // the pair kernels' segments by 2^c2_seg_extra and the tail kernel's by
    // 2^c2_tail_extra
    const int base0 = max(j.blocknum - 1, j.q - 1);
    const int base = base0 + min(max(j.c2_seg_extra, 0), kMaxSegExtra);
    const int base_tail = base0 + min(max(j.c2_tail_extra, 0), kMaxSegExtra);
    p.npair = (j.q >= 7) ? 2 : 1;
    p.k_tail = 2 * p.npair;
    for (int k = 0; k < kMaxLevels; k++) p.seg_log[k] = 0;
    for (int i = 0; i < p.npair; i++) {
        const int k = 2 * i;
        const int sl = max(base, k + 6);            // segments start at multiples of 64 level-k samples
        p.seg_log[k] = p.seg_log[k + 1] = sl;
    }
    if (p.k_tail < j.q) {
        const int sl = max(base_tail, p.k_tail);
        for (int k = p.k_tail; k < j.q; k++) p.seg_log[k] = sl;
    }
    p.nseg_max = 1;
    for (int k = 0; k < j.q; k++)
        p.nseg_max = max(p.nseg_max, (j.num + (1 << p.seg_log[k]) - 1) >> p.seg_log[k]);
    return p;
}
}  // namespace

int corr2_nseg(const Job &j) { return plan2(j).nseg_max; }

// The P = 32 path's scratch: bytes per pixel, and the pixels of a chunk.
struct CgPlan {
    int chunk, nseg, pnum_max, seg_log[kMaxLevels], numbin[kMaxLevels];
    size_t lv, pz, tot;                   // floats per pixel: level streams, products, totals
};
static CgPlan cg_plan(const Job &j)
{
    CgPlan p;
    p.pnum_max = max((j.num - (j.p << (j.q - 1))) >> (j.q - 1), 1);
    const int base = max(j.blocknum - 1, j.q - 1);     // every pixel's block length divides 2^base frames
    p.lv = 0;
    int nb = j.num;
    p.nseg = 1;
    for (int k = 0; k < j.q; k++, nb /= 2) {
        p.numbin[k] = nb;
        if (k) p.lv += nb;
        p.seg_log[k] = max(base, k + 4);               // whole steps of 16 samples
        p.nseg = max(p.nseg, (j.num + (1 << p.seg_log[k]) - 1) >> p.seg_log[k]);
    }
    p.lv *= j.is_ccf ? 2 : 1;
    p.pz = (size_t)j.chanum * p.pnum_max;
    p.tot = (size_t)2 * j.chanum * p.nseg;
    const size_t pixel = (p.lv + p.pz + p.tot) * sizeof(float);
    size_t c = kCgChunkBytes / pixel;
    c = c < 64 ? 64 : c & ~(size_t)63;
    if (j.cg_bytes) c = j.cg_bytes / pixel > 1 ? j.cg_bytes / pixel : 1;
    p.chunk = (int)(c < (size_t)j.npix ? c : (size_t)j.npix);
    return p;
}

int corr_kernel_count(const Job &j)
{
    if (corrg_supported(j)) {
        const int c = cg_plan(j).chunk;
        return 3 * ((j.npix + c - 1) / c);
    }
    if (!corr2_supported(j)) return 1;
    const Plan2 p = plan2(j);
    return p.npair + (p.k_tail < j.q ? 1 : 0) + 1;   // pair kernels, tail, finalise
}

size_t corr_stats_floats(const Job &j)
{
    if (corrg_supported(j)) {
        const CgPlan p = cg_plan(j);
        return (p.pz + p.tot) * p.chunk;
    }
    const size_t one = (size_t)j.chanum * kStatN * j.npix;
    return corr2_supported(j) ? one * corr2_nseg(j) : one;
}

// Binned sample streams, per trace: s2 (num/4 x npix) and s4 (num/16 x
// npix), written by the pair kernels for the next level pair.
size_t corr_stream_floats(const Job &j)
{
    if (corrg_supported(j)) {
        const CgPlan p = cg_plan(j);
        return p.lv * p.chunk;
    }
    if (!corr2_supported(j)) return 1;
    const size_t tr = j.is_ccf ? 2 : 1;
    return tr * (size_t)j.npix * ((size_t)(j.num >> 2) + (size_t)(j.num >> 4) + 3);
}

// The corrected level-0 stream s0[trace][frame][pixel] (imfcs_stream.cu).
size_t level0_stream_floats(const Job &j) { return (size_t)(j.is_ccf ? 2 : 1) * j.npix * j.num; }

// Threads up to which a grid takes the split pair kernels (levels 0-1: three
// blocks, above: two; 152 SMs hold 58,368).  Measured, whole -> split: levels
// 0-1, 2,560 threads 144 -> 83 us (20,000 frames), 13,312 277 -> 188 (50,000),
// 23,040 158 -> 199 (20,000); levels 2-3, 2,560 46 -> 30, 23,040 56 -> 37,
// 40,960 62 -> 69.
constexpr int kSplitThreads[2] = {256 * 64, 480 * 64};

// One pair kernel of the chain: variant 0 = levels 0-1, 1 = two upper
// levels, 2 = one upper level (the last).
template <int NT>
static void launch_pair(bool ccf, int variant, dim3 grid, cudaStream_t stream, const C2Args &a, const float *ia,
                        const float *ib, float *oa, float *ob, int k)
{
    if (variant < 2 && (long long)grid.x * grid.y * NT <= kSplitThreads[variant]) {
        grid.z = variant == 0 ? 3 : 2;
        if (ccf) {
            if (variant == 0) c2_pair_split_kernel<true, true, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
            else c2_pair_split_kernel<true, false, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
        } else {
            if (variant == 0) c2_pair_split_kernel<false, true, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
            else c2_pair_split_kernel<false, false, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
        }
    } else if (ccf) {
        if (variant == 0) c2_pair_kernel<true, true, true, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
        else if (variant == 1) c2_pair_kernel<true, false, true, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
        else c2_pair_kernel<true, false, false, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
    } else {
        if (variant == 0) c2_pair_kernel<false, true, true, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
        else if (variant == 1) c2_pair_kernel<false, false, true, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
        else c2_pair_kernel<false, false, false, NT><<<grid, NT, 0, stream>>>(a, ia, ib, oa, ob, k);
    }
}

// The P = 32 correlator, one pixel chunk after the other.
cudaError_t launch_corrg(const Job &j, const LagInfo *li, const float *s0, const float4 *mon, const int *blk_ind,
                         const CorrOut &o, float *streams, cudaStream_t stream)
{
    const CgPlan p = cg_plan(j);
    CgArgs a;
    memset(&a, 0, sizeof(a));
    a.o = o;
    a.mon = mon;
    a.blk_ind = blk_ind;
    a.li = li;
    a.npix = j.npix;
    a.cs = p.chunk;
    a.chanum = j.chanum;
    a.p = j.p;
    a.q = j.q;
    a.num = j.num;
    a.nseg = p.nseg;
    a.pnum_max = p.pnum_max;
    size_t off = 0;
    for (int k = 0; k < j.q; k++) {
        a.numbin[k] = p.numbin[k];
        a.seg_log[k] = p.seg_log[k];
        if (k) {
            a.lv_off[k] = off;
            off += (size_t)p.numbin[k] * p.chunk;
        }
    }
    a.s0a = s0;
    a.s0b = j.is_ccf ? s0 + (size_t)j.npix * j.num : s0;
    a.lva = streams;
    a.lvb = j.is_ccf ? streams + off : streams;
    a.tot = (float2 *)o.stats;
    a.pz = o.stats + p.tot * p.chunk;
    const int span = 1 << max(j.q - 1, 3);
    for (a.p0 = 0; a.p0 < j.npix; a.p0 += p.chunk) {
        a.np = min(p.chunk, j.npix - a.p0);
        const dim3 gl((a.np + 127) / 128, min((j.num + span - 1) / span, 65535));
        const dim3 gb((a.np + kCgThreads - 1) / kCgThreads, j.q + 1, p.nseg);
        if (j.is_ccf) {
            cg_levels_kernel<true><<<gl, 128, 0, stream>>>(a);
            cg_blocks_kernel<true><<<gb, kCgThreads, 0, stream>>>(a);
        } else {
            cg_levels_kernel<false><<<gl, 128, 0, stream>>>(a);
            cg_blocks_kernel<false><<<gb, kCgThreads, 0, stream>>>(a);
        }
        cg_finalize_kernel<<<dim3((a.np + 127) / 128, j.chanum), 128, 0, stream>>>(a);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_corr2(const Job &j, const LagInfo *li, const float *s0, const float4 *mon, const int *blk_ind,
                         const CorrOut &o, float *streams, cudaStream_t stream)
{
    const Plan2 pl = plan2(j);
    C2Args a;
    memset(&a, 0, sizeof(a));
    a.o = o;
    a.mon = mon;
    a.blk_ind = blk_ind;
    a.li = li;
    a.npix = j.npix;
    a.chanum = j.chanum;
    a.p = j.p;
    a.q = j.q;
    a.num = j.num;
    {
        int nb = j.num;
        for (int k = 0; k < j.q; k++) { a.numbin[k] = nb; nb /= 2; }
    }
    for (int k = 0; k < kMaxLevels; k++) a.seg_log[k] = pl.seg_log[k];
    a.stat_stride = (size_t)j.chanum * kStatN * j.npix;

    const size_t tr = j.is_ccf ? 2 : 1;
    const size_t np = j.npix;
    const float *s0a = s0, *s0b = j.is_ccf ? s0 + np * j.num : s0;
    float *s2a = streams, *s2b = j.is_ccf ? s2a + np * (j.num >> 2) : s2a;
    float *s4a = s2a + tr * np * (j.num >> 2), *s4b = j.is_ccf ? s4a + np * (j.num >> 4) : s4a;
    cudaError_t e = cudaSuccess;

    const int nt = j.c2_cta == 32 ? 32 : kC2Threads;
    const int pgx = (j.npix + nt - 1) / nt;
    for (int i = 0; i < pl.npair; i++) {
        const int k = 2 * i;
        const float *ia = i ? s2a : s0a, *ib = i ? s2b : s0b;
        float *oa = (k + 2 < j.q) ? (i ? s4a : s2a) : nullptr;
        float *ob = (k + 2 < j.q) ? (i ? s4b : s2b) : nullptr;
        const dim3 grid(pgx, (j.num + (1 << pl.seg_log[k]) - 1) >> pl.seg_log[k]);
        const int variant = (i == 0) ? 0 : (k + 1 < j.q ? 1 : 2);
        if (nt == 32) launch_pair<32>(j.is_ccf, variant, grid, stream, a, ia, ib, oa, ob, k);
        else launch_pair<kC2Threads>(j.is_ccf, variant, grid, stream, a, ia, ib, oa, ob, k);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (pl.k_tail < j.q) {
        const int k0 = pl.k_tail;
        const float *ia = (k0 == 2) ? s2a : s4a, *ib = (k0 == 2) ? s2b : s4b;
        const dim3 grid(pgx, (j.num + (1 << pl.seg_log[k0]) - 1) >> pl.seg_log[k0], j.q - k0);
        if (nt == 32) {
            if (j.is_ccf) c2_tail_kernel<true, 32><<<grid, 32, 0, stream>>>(a, ia, ib, k0);
            else c2_tail_kernel<false, 32><<<grid, 32, 0, stream>>>(a, ia, ib, k0);
        } else {
            if (j.is_ccf) c2_tail_kernel<true, kC2Threads><<<grid, kC2Threads, 0, stream>>>(a, ia, ib, k0);
            else c2_tail_kernel<false, kC2Threads><<<grid, kC2Threads, 0, stream>>>(a, ia, ib, k0);
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    c2_finalize_kernel<<<dim3((j.npix + 127) / 128, j.chanum), 128, 0, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace imfcs
