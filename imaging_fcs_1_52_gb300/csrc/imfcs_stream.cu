// imfcs_stream.cu -- the one streaming pass over the raw uint16 stack after
// the bleach fit: every (trace, frame) is binned, background-subtracted,
// bleach-corrected (java:9682-9769) and centred once, written as the FP32
// level-0 sample stream s0[t][pixel] that the blocking transform and the
// correlator chain read, and summed into the monitor partials (float-float
// segment totals, the partial sums at every snapshot position the lags'
// windows need, and the count of non-finite frames) in the same pass.
//
// Staging: one CTA covers a tile of tr rows x tc columns of output pixels (up
// to 128, one thread per pixel) and a few monitor segments of kSeg = 256
// frames.  Its raw frames arrive as boxes [fbox frames][bh rows][bw columns]
// in a ring of kStRing buffers: by TMA (cp.async.bulk.tensor, each box
// completing on its own mbarrier) where the frames' rows are 16-byte aligned,
// by 4-byte cp.async otherwise (any row length; each row is copied from its
// start rounded down to a word).  The threads walk the staged frames in order,
// eight at a time.  Float input, a stack that is not 4-byte aligned and shapes
// for which cp.async does not pay (stream_plan) are read with plain loads
// instead.
//
// The exponential bleach curve is advanced by a recurrence e <- e q within
// each 64-frame stage (reseeded with exp() per stage: at most 64 FP32
// factors, ~4e-6 relative, a smooth factor that the normalised correlation
// does not see).  Non-finite corrected frames (a bleach curve through zero)
// are written as 0 and counted, so that the monitor finaliser makes exactly
// the lags whose windows hold one non-finite (calculateCF's NaN propagation,
// java:9484-9511).
//
// Waits are bounded (imfcs_tma.cuh): on a timeout the CTA records the error
// flag, waits (bounded) for its own copies and leaves.
#include <string.h>

#include "imfcs_host.h"
#include "imfcs_internal.cuh"
#include "imfcs_tma.cuh"

namespace imfcs {

constexpr int kStReseed = 64;                  // frames between reseeds of the exponential recurrence
constexpr int kStRing = 3;                     // boxes in flight / being processed per CTA
constexpr int kStMaxThreads = 128;
static_assert(kSeg % kStReseed == 0, "monitor segments must hold whole reseeding spans");

struct StreamArgs {
    Job j;
    const void *stack;
    const float *bparams, *basis;
    const int *snap_pos;
    int nseg;
    float *s0a, *s0b;
    float2 *segtot, *snap_part;
    int *segbad, *snap_bad;
    int *err;
    // staged kernels: output tile (tc x tr pixels), box (fbox frames of `rows`
    // raw rows, elements between frames and rows), one run per frame, the
    // monitor segments of a CTA, and the column-sum stage (0: none)
    int tc, tr, tiles_x, fbox, rows, fs, rs, run, segs;
    int col_rows, col_w;
};

// Correction state of one trace (bleach parameters, centre, recurrence).
template <int MODE>
struct StreamCorr {
    float f0, inv_f0, centre, c, k0, a0, k1, a1, q0, q1, e0, e1;
    int flags;
    bool on;
    float coef[(kMaxPoly + 4) & ~3];
    __device__ __forceinline__ void load(const float *bp, float frametime, int order)
    {
        centre = __ldg(&bp[12]);
        on = MODE != IMFCS_BLEACH_NONE && __ldg(&bp[11]) != 0.f;
        f0 = __ldg(&bp[9]);
        inv_f0 = __ldg(&bp[10]);
        if (MODE == IMFCS_BLEACH_SINGLE_EXP || MODE == IMFCS_BLEACH_DOUBLE_EXP) {
            c = __ldg(&bp[13]);
            flags = (int)__ldg(&bp[14]);
            k0 = __ldg(&bp[5]);
            a0 = __ldg(&bp[7]);
            k1 = __ldg(&bp[6]);
            a1 = __ldg(&bp[8]);
            q0 = __expf(-k0 * frametime);
            q1 = __expf(-k1 * frametime);
        }
        if (MODE == IMFCS_BLEACH_POLYNOMIAL)
#pragma unroll
            for (int i = 0; i < ((kMaxPoly + 4) & ~3); i++) coef[i] = i <= order ? __ldg(&bp[i]) : 0.f;
    }
    __device__ __forceinline__ void seed(int t, float frametime)
    {
        if (MODE == IMFCS_BLEACH_SINGLE_EXP || MODE == IMFCS_BLEACH_DOUBLE_EXP) {
            const float ft = frametime * ((float)t + 1.5f);   // java:9747, 1-based frame number
            e0 = __expf(-k0 * ft);
            if (MODE == IMFCS_BLEACH_DOUBLE_EXP) e1 = __expf(-k1 * ft);
        }
    }
    // The exponential bleach curve at frame t; form0: the component's form is
    // the slow series (the flag of component 0), known by the caller.
    __device__ __forceinline__ float curve(int t, float frametime, bool form0) const
    {
        const float ft = frametime * ((float)t + 1.5f);
        float f = __fadd_rn(c, form0 ? __fmul_rn(-a0, slow_exp_term(k0, ft)) : __fmul_rn(a0, e0));
        if (MODE == IMFCS_BLEACH_DOUBLE_EXP)
            f = __fadd_rn(f, ((flags >> 1) & 1) ? __fmul_rn(-a1, slow_exp_term(k1, ft)) : __fmul_rn(a1, e1));
        return f;
    }
    __device__ __forceinline__ void advance()
    {
        if (MODE == IMFCS_BLEACH_SINGLE_EXP || MODE == IMFCS_BLEACH_DOUBLE_EXP) {
            e0 *= q0;
            if (MODE == IMFCS_BLEACH_DOUBLE_EXP) e1 *= q1;
        }
    }
    // Corrected, centred values of the raw window values of N consecutive
    // frames from t on (the frames after the previous call's, or the seeded
    // one).  The tests of `on` and of the curve's form stay outside the loop.
    template <int N>
    __device__ __forceinline__ void apply(float (&v)[N], int t, float frametime, int order, const float *basis)
    {
        if (MODE != IMFCS_BLEACH_NONE && on) {
            if constexpr (MODE == IMFCS_BLEACH_POLYNOMIAL) {
                // the N frames' basis values four at a time (rows padded with
                // zeros), all loads before their use
                const int nq = basis_stride(order) / 4;
                const float4 *b = (const float4 *)basis + (size_t)t * nq;
                float f[N];
#pragma unroll
                for (int u = 0; u < N; u++) f[u] = 0.f;
#pragma unroll
                for (int q = 0; q < (kMaxPoly + 4) / 4; q++) {
                    if (q >= nq) break;
                    float4 w[N];
#pragma unroll
                    for (int u = 0; u < N; u++) w[u] = __ldg(&b[u * nq + q]);
#pragma unroll
                    for (int u = 0; u < N; u++) {
                        f[u] = fmaf(coef[4 * q], w[u].x, f[u]);
                        if (4 * q + 1 <= kMaxPoly) f[u] = fmaf(coef[4 * q + 1], w[u].y, f[u]);
                        if (4 * q + 2 <= kMaxPoly) f[u] = fmaf(coef[4 * q + 2], w[u].z, f[u]);
                        if (4 * q + 3 <= kMaxPoly) f[u] = fmaf(coef[4 * q + 3], w[u].w, f[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < N; u++) v[u] = bleach_correct(v[u], f[u], f0, inv_f0);
            } else if (flags & 1) {
#pragma unroll
                for (int u = 0; u < N; u++) {
                    v[u] = bleach_correct(v[u], curve(t + u, frametime, true), f0, inv_f0);
                    advance();
                }
            } else {
#pragma unroll
                for (int u = 0; u < N; u++) {
                    v[u] = bleach_correct(v[u], curve(t + u, frametime, false), f0, inv_f0);
                    advance();
                }
            }
        }
#pragma unroll
        for (int u = 0; u < N; u++) v[u] -= centre;
    }
};

// Monitor partials of one trace over its segment.  pos: the snapshot
// positions, in shared memory (a thread near the end of the recording passes
// a hundred of them, each compared after the one before).
struct MonAcc {
    ff acc;
    int bad, sj, next;
    const int *pos;
    __device__ __forceinline__ void init(const int *snaps, int nsnap, int t0)
    {
        acc = {0.f, 0.f};
        bad = 0;
        pos = snaps;
        int lo = 0, hi = nsnap;     // first snapshot with position > t0
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (snaps[mid] <= t0) lo = mid + 1; else hi = mid;
        }
        sj = lo;
        next = sj < nsnap ? snaps[sj] : 0x7fffffff;
    }
    __device__ __forceinline__ void snapshot(const StreamArgs &a, int trace, const ff &s)
    {
        a.snap_part[(size_t)trace * a.j.nsnap + sj] = make_float2(s.hi, s.lo);
        a.snap_bad[(size_t)trace * a.j.nsnap + sj] = bad;
        sj++;
        next = sj < a.j.nsnap ? pos[sj] : 0x7fffffff;
    }
    // Values x of N frames from t on, replaced by the values to store (0
    // where non-finite).  With no snapshot among them the sums run without a
    // test per value: a non-finite value leaves the running sum non-finite,
    // and the values are then taken one by one from the sum before them.
    template <int N>
    __device__ __forceinline__ void add(const StreamArgs &a, int trace, int t, float (&x)[N])
    {
        ff s = acc;
#pragma unroll
        for (int u = 0; u < N; u++) ff_add(s, x[u]);
        if (isfinite(s.hi)) {
            if (next > t + N) {
                acc = s;
                return;
            }
#pragma unroll
            for (int u = 0; u < N; u++) {
                ff_add(acc, x[u]);
                while (t + u + 1 == next) snapshot(a, trace, acc);
            }
            return;
        }
#pragma unroll
        for (int u = 0; u < N; u++) {
            if (isfinite(x[u])) {
                ff_add(acc, x[u]);
            } else {
                bad++;
                x[u] = 0.f;
            }
            while (t + u + 1 == next) snapshot(a, trace, acc);
        }
    }
    __device__ __forceinline__ void store(const StreamArgs &a, int trace, int seg)
    {
        a.segtot[(size_t)trace * a.nseg + seg] = make_float2(acc.hi, acc.lo);
        a.segbad[(size_t)trace * a.nseg + seg] = bad;
    }
};

// One trace's N frames from t on: correct, sum, store.
template <int MODE, int N>
__device__ __forceinline__ void stream_frames(const StreamArgs &a, StreamCorr<MODE> &c, MonAcc &m, int trace, int t,
                                              float (&v)[N], float *dst)
{
    c.template apply<N>(v, t, a.j.frametime, a.j.poly_order, a.basis);
    m.template add<N>(a, trace, t, v);
#pragma unroll
    for (int u = 0; u < N; u++) dst[(size_t)u * a.j.npix] = v[u];
}

__device__ __forceinline__ void cp_async4(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Where a CTA's raw frames sit: the element (frame f of the box, row y,
// column x, all relative to the tile's first row and column) is at
// tile[f * fs + y * rs + x + xoff + par], with xoff the columns TMA's 16-byte
// rounding put in front and par the element a word-aligned copy put in front
// of this row (rows of odd length start at odd elements).  A tile as wide as
// the frame is copied as one run per frame: rs is then the frame's width and
// only the frame's first element has a parity.
template <bool TMA>
struct BoxGeo {
    int fs, rs, xoff;
    int par0, par_f, par_y;      // parity of the box's first row; what a frame and a row add
    __device__ __forceinline__ int par(int f, int y) const
    {
        return TMA ? 0 : (par0 ^ (f & par_f) ^ (y & par_y)) & 1;
    }
    __device__ __forceinline__ int at(int f, int y, int x) const { return f * fs + y * rs + x + xoff + par(f, y); }
};

// cp.async of one box: nf frames from frame t (absolute) on, one warp per row
// (per frame where the tile is as wide as the frame).
__device__ __forceinline__ void copy_box(const StreamArgs &a, uint16_t *tile, int t, int nf, int rx0, int ry0,
                                         int ncols)
{
    const Job &j = a.j;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const size_t total = (size_t)(j.first + j.num) * j.in_h * j.in_w;      // elements of the frames read
    int nrow = min(a.rows, j.in_h - ry0), n = ncols;
    if (a.run) {
        n = nrow * j.in_w;
        nrow = 1;
    }
    for (int y = 0; y < nrow; y++)
        for (int f = warp; f < nf; f += nwarp) {
            const size_t e0 = ((size_t)(t + f) * j.in_h + ry0 + y) * j.in_w + rx0;
            const size_t w0 = e0 >> 1;
            const int words = ((int)(e0 & 1) + n + 1) >> 1;
            uint16_t *dst = tile + f * a.fs + y * a.rs;
            const uint32_t *src = (const uint32_t *)a.stack + w0;
            // the last word of an odd number of elements has one that is not there
            const int whole = 2 * (w0 + words) <= total ? words : words - 1;
            for (int w = lane; w < whole; w += 32) cp_async4(dst + 2 * w, src + w);
            if (whole < words && lane == 0) dst[2 * whole] = ((const uint16_t *)a.stack)[2 * (w0 + whole)];
        }
}

// Raw window sums of frames f .. f+N-1 of the box (N = 8, f a multiple of 8,
// or one frame), window at tile row y, column x.
template <bool TMA, bool BIN1, int N>
__device__ __forceinline__ void window_sums(const Job &j, const BoxGeo<TMA> &g, const uint16_t *tile, const int *cols,
                                            int cstride, int f, int y, int x, int (&s)[N])
{
    if constexpr (BIN1) {
#pragma unroll
        for (int u = 0; u < N; u++) s[u] = tile[g.at(f + u, y, x)];
    } else {
#pragma unroll
        for (int u = 0; u < N; u++) s[u] = 0;
        if (cols) {                   // column sums over the window's rows are staged
            const int *p = cols + f * cstride;
            for (int i = 0; i < j.binx; i++)
#pragma unroll
                for (int u = 0; u < N; u++) s[u] += p[u * cstride + i];
        } else {
            for (int k = 0; k < j.biny; k++)
                for (int i = 0; i < j.binx; i++)
#pragma unroll
                    for (int u = 0; u < N; u++) s[u] += tile[g.at(f + u, y + k, x + i)];
        }
    }
}

// Staged stream pass: grid (output tiles, ceil(nseg / segs)).  Bound by HBM
// and issue about equally: 2 B in and 4 B out a frame-pixel take 0.72 ms at the
// copy rate for 128x128x50,000, the kernel 1.09 ms (1.76 before eight frames
// went at a time, with the tests of the curve's form, of non-finite values and
// of snapshots out of the frame loop); whole-row tiles of up to 128 threads with short boxes, and
// the polynomial's coefficients in registers, 7.6 -> 0.59 ms for 2 x 2 binned
// cross-correlation at 128x128x20,000 (32-thread CTAs with 83 KB each before)
// and 1.50 -> 0.76 ms for overlapping 5 x 5 windows of rows of 101 (25 plain
// loads a value before).  A CTA walks
// its monitor segments through a ring of kStRing boxes: while one box is
// processed the next ones are in flight; a CTA barrier frees a box before it
// is filled again.  The outcome of every bounded wait is made uniform across
// the CTA (__syncthreads_or), so no thread is left waiting at a barrier.
// Windows of nine or more raw pixels first become column sums (the rows of
// the window added up) in shared memory, by all threads of the CTA.
template <int MODE, bool CCF, bool BIN1, bool TMA>
__global__ void __launch_bounds__(kStMaxThreads) stream_box_kernel(StreamArgs a,
                                                                   const __grid_constant__ CUtensorMap tmap)
{
    extern __shared__ __align__(128) unsigned char ssm[];
    __shared__ uint64_t full[kStRing];
    __shared__ int snaps[kMaxSnap];
    const Job &j = a.j;
    const int tid = threadIdx.x;
    for (int i = tid; i < j.nsnap; i += blockDim.x) snaps[i] = __ldg(&a.snap_pos[i]);
    const int ty = blockIdx.x / a.tiles_x;
    const int ox0 = (blockIdx.x - ty * a.tiles_x) * a.tc, oy0 = ty * a.tr;
    const int seg0 = blockIdx.y * a.segs, seg1 = min(seg0 + a.segs, a.nseg);
    const int t0 = seg0 * kSeg, t1 = min(seg1 * kSeg, j.num);
    const int F = a.fbox, box = F * a.fs;
    uint16_t *tiles = (uint16_t *)ssm;
    int *cols = BIN1 || a.col_rows == 0 ? nullptr : (int *)(tiles + (size_t)kStRing * box);
    const int cstride = a.col_rows * a.col_w;
    const int rx0 = (j.map_x0 + ox0) * j.pixbinx + min(0, j.cfx);
    const int ry0 = (j.map_y0 + oy0) * j.pixbiny + min(0, j.cfy);
    const int ncols = min((a.tc - 1) * j.pixbinx + j.binx + abs(j.cfx), j.in_w - rx0);
    BoxGeo<TMA> g;
    g.fs = a.fs;
    g.rs = a.rs;
    g.xoff = TMA ? rx0 & 7 : 0;                       // x rounded down to 16 bytes
    g.par_f = (j.in_w * j.in_h) & 1;
    g.par_y = a.run ? 0 : j.in_w & 1;
    g.par0 = 0;
    const int nbox = (t1 - t0 + F - 1) / F;
    if (TMA) {
        if (tid == 0) {
            for (int b = 0; b < kStRing; b++) mbar_init(&full[b], 1);
            for (int b = 0; b < nbox && b < kStRing; b++)
                tma_load_box(&tmap, tiles + (size_t)b * box, &full[b], rx0 & ~7, ry0, j.first + t0 + b * F,
                             (uint32_t)box * 2);
        }
        __syncthreads();
    } else {
        for (int b = 0; b < kStRing; b++) {
            if (b < nbox)
                copy_box(a, tiles + (size_t)b * box, j.first + t0 + b * F, min(F, t1 - t0 - b * F), rx0, ry0, ncols);
            cp_async_commit();
        }
    }
    const int r = tid / a.tc, c = tid - r * a.tc;
    const bool valid = r < a.tr && ox0 + c < j.out_w && oy0 + r < j.out_h;
    const int pix = valid ? (oy0 + r) * j.out_w + ox0 + c : oy0 * j.out_w + ox0;
    // the windows inside the tile; with column sums x, y index those
    const int xa = c * j.pixbinx + (j.cfx < 0 ? -j.cfx : 0), xb = xa + j.cfx;
    const int ya = r * j.pixbiny + (j.cfy < 0 ? -j.cfy : 0), yb = ya + j.cfy;
    const int *ca_cols = cols ? cols + r * a.col_w + xa : nullptr;
    const int *cb_cols = cols ? cols + (r + (j.cfy ? a.tr : 0)) * a.col_w + xb : nullptr;
    const int bga = trace_bg(j, pix), bgb = CCF ? trace_bg(j, j.npix + pix) : 0;
    StreamCorr<MODE> ca, cb;
    ca.load(a.bparams + (size_t)pix * kBleachStride, j.frametime, j.poly_order);
    if (CCF) cb.load(a.bparams + (size_t)(j.npix + pix) * kBleachStride, j.frametime, j.poly_order);
    MonAcc ma, mb;
    int issued = nbox < kStRing ? nbox : kStRing;
    for (int b = 0; b < nbox; b++) {
        const int slot = b % kStRing;
        uint16_t *tile = tiles + (size_t)slot * box;
        if (TMA) {
            const bool waited = mbar_wait(&full[slot], (uint32_t)((b / kStRing) & 1));
            if (__syncthreads_or(!waited)) {
                if (tid == 0) {
                    atomicExch(a.err, 1);
                    // the copies still in flight land before the CTA leaves
                    for (int q = b; q < issued; q++) mbar_wait(&full[q % kStRing], (uint32_t)((q / kStRing) & 1));
                }
                return;
            }
        } else {
            cp_async_wait<kStRing - 1>();
            __syncthreads();
        }
        const int tb = t0 + b * F;
        const int seg = tb / kSeg;
        const int n = min(F, t1 - tb);
        if (!TMA) g.par0 = (int)((((size_t)(j.first + tb) * j.in_h + ry0) * j.in_w + rx0) & 1);
        if (!BIN1 && cols) {
            for (int q = tid; q < a.col_rows * a.col_w; q += blockDim.x) {
                const int row = q / a.col_w, x = q - row * a.col_w;
                const int y = row < a.tr ? row * j.pixbiny + (j.cfy < 0 ? -j.cfy : 0)
                                         : (row - a.tr) * j.pixbiny + (j.cfy < 0 ? 0 : j.cfy);
                if (x >= ncols) continue;
                for (int f = 0; f < n; f += 8) {          // past n: frames of the buffer that nothing reads
                    int s[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) s[u] = 0;
                    for (int k = 0; k < j.biny; k++)
#pragma unroll
                        for (int u = 0; u < 8; u++) s[u] += tile[g.at(f + u, y + k, x)];
#pragma unroll
                    for (int u = 0; u < 8; u++) cols[(f + u) * cstride + q] = s[u];
                }
            }
            __syncthreads();
        }
        if (valid) {
            if (tb % kSeg == 0) {
                ma.init(snaps, j.nsnap, tb);
                if (CCF) mb.init(snaps, j.nsnap, tb);
            }
            if (tb % kStReseed == 0) {
                ca.seed(tb, j.frametime);
                if (CCF) cb.seed(tb, j.frametime);
            }
            float *da = a.s0a + (size_t)tb * j.npix + pix, *db = a.s0b + (size_t)tb * j.npix + pix;
            int f = 0;
#pragma unroll 1
            for (; f + 8 <= n; f += 8) {
                int w[8];
                float v[8];
                window_sums<TMA, BIN1, 8>(j, g, tile, ca_cols, cstride, f, ya, xa, w);
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = (float)(w[u] - bga);
                stream_frames<MODE, 8>(a, ca, ma, pix, tb + f, v, da);
                da += (size_t)8 * j.npix;
                if (CCF) {
                    window_sums<TMA, BIN1, 8>(j, g, tile, cb_cols, cstride, f, yb, xb, w);
#pragma unroll
                    for (int u = 0; u < 8; u++) v[u] = (float)(w[u] - bgb);
                    stream_frames<MODE, 8>(a, cb, mb, j.npix + pix, tb + f, v, db);
                    db += (size_t)8 * j.npix;
                }
            }
#pragma unroll 1
            for (; f < n; f++) {
                int w[1];
                float v[1];
                window_sums<TMA, BIN1, 1>(j, g, tile, ca_cols, cstride, f, ya, xa, w);
                v[0] = (float)(w[0] - bga);
                stream_frames<MODE, 1>(a, ca, ma, pix, tb + f, v, da);
                da += j.npix;
                if (CCF) {
                    window_sums<TMA, BIN1, 1>(j, g, tile, cb_cols, cstride, f, yb, xb, w);
                    v[0] = (float)(w[0] - bgb);
                    stream_frames<MODE, 1>(a, cb, mb, j.npix + pix, tb + f, v, db);
                    db += j.npix;
                }
            }
            if (tb + F >= min((seg + 1) * kSeg, t1)) {   // last box of the segment
                ma.store(a, pix, seg);
                if (CCF) mb.store(a, j.npix + pix, seg);
            }
        }
        __syncthreads();                                    // box `slot` is free
        if (TMA) {
            if (tid == 0 && b + kStRing < nbox) {
                tma_load_box(&tmap, tile, &full[slot], rx0 & ~7, ry0, j.first + t0 + (b + kStRing) * F,
                             (uint32_t)box * 2);
                issued = b + kStRing + 1;
            }
        } else {
            const int q = b + kStRing;
            if (q < nbox) copy_box(a, tile, j.first + t0 + q * F, min(F, t1 - t0 - q * F), rx0, ry0, ncols);
            cp_async_commit();
        }
    }
}

// Plain-load stream pass (float input, a stack at an odd address, or by
// stream_plan's rule): grid
// (ceil(npix/128), nseg), one thread per (pixel, segment).
template <int MODE, bool CCF>
__global__ void __launch_bounds__(128) stream_plain_kernel(StreamArgs a)
{
    const Job &j = a.j;
    __shared__ int snaps[kMaxSnap];
    for (int i = threadIdx.x; i < j.nsnap; i += blockDim.x) snaps[i] = __ldg(&a.snap_pos[i]);
    __syncthreads();
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= j.npix) return;
    const int seg = blockIdx.y, t0 = seg * kSeg, t1 = min(t0 + kSeg, j.num);
    for (int tr = 0; tr < (CCF ? 2 : 1); tr++) {
        const int trace = tr ? j.npix + pix : pix;
        int x0, y0;
        trace_origin(j, trace, x0, y0);
        StreamCorr<MODE> c;
        c.load(a.bparams + (size_t)trace * kBleachStride, j.frametime, j.poly_order);
        MonAcc m;
        m.init(snaps, j.nsnap, t0);
        float *dst = (tr ? a.s0b : a.s0a) + (size_t)t0 * j.npix + pix;
        const int bg = trace_bg(j, trace);
        int t = t0;
        for (; t + 8 <= t1; t += 8) {
            if ((t & (kStReseed - 1)) == 0) c.seed(t, j.frametime);
            float v[8];
            window_values<8>(j, a.stack, x0, y0, t, t1, bg, v);
            stream_frames<MODE, 8>(a, c, m, trace, t, v, dst);
            dst += (size_t)8 * j.npix;
        }
        for (; t < t1; t++) {
            if ((t & (kStReseed - 1)) == 0) c.seed(t, j.frametime);
            float v[1];
            window_values<1>(j, a.stack, x0, y0, t, t1, bg, v);
            stream_frames<MODE, 1>(a, c, m, trace, t, v, dst);
            dst += j.npix;
        }
        m.store(a, trace, seg);
    }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
struct StreamPlan {
    int ok, tma, threads, tc, tr, tiles_x, tiles_y, fbox, bw, rows, rs, fs, run, segs, col_rows, col_w;
    size_t smem;
};

// The tile and box of a job.  Tiles are up to 128 pixels, whole rows where
// the output is narrow (a 21-pixel row alone would leave 107 of 128 threads
// idle).  Boxes are as long as fits 56 KB for the ring (four CTAs per SM),
// shorter for tiles that read many raw pixels; what does not fit at 8 frames
// gets a smaller tile.
//
// The cp.async boxes cost a warp's turn per row and frame (per frame where the
// tile is as wide as the frame), whatever the row's length.  Windows of several
// pixels are worth up to four such rows a warp (plain / boxes, us: overlapping 5
// x 5 at 11x6x15,253 404 / 58, 2 x 2 steps at 439x4x37,510 345 / 136; narrow
// outputs of many rows, 1x158 of 3 x 1 windows at 4,242 frames 218 / 1,680, 6x47
// of 2 x 1 at 6,441 130 / 295).  Single pixels gain where all four warps share
// one copy a frame and the plain kernel's blocks leave the SMs part-empty,
// from 100 pixels up to 600 blocks (123x8x18,566 71 / 57); else the plain kernel is faster
// (13x1x2,627 36 / 67, a third of 25x44x7,172 52 / 218, 85x75x39,755 966 /
// 1,605).
static StreamPlan stream_plan(const Job &j, const void *stack, int nseg)
{
    StreamPlan sp;
    memset(&sp, 0, sizeof(sp));
    if (j.input_float || ((uintptr_t)stack % 4) != 0) return sp;
    sp.tma = ((uintptr_t)stack % 16) == 0 && (j.in_w % 8) == 0;   // 16-byte base and row stride
    const bool col = j.binx * j.biny >= 9;
    const int across = (j.out_w + kStMaxThreads - 1) / kStMaxThreads;
    int tc = (j.out_w + across - 1) / across, tr = kStMaxThreads / tc;
    if (tr > j.out_h) tr = j.out_h;
    for (;;) {
        const int need = (tc - 1) * j.pixbinx + j.binx + abs(j.cfx);
        const int rows = (tr - 1) * j.pixbiny + j.biny + abs(j.cfy);
        // one run per frame: the only tile of a row, reading every column
        const int run = !sp.tma && tc == j.out_w && need == j.in_w;
        const int bw = sp.tma ? (need + 7 + 7) & ~7 : (need + 2) & ~1;
        const int rs = run ? j.in_w : bw;
        const int fs = run ? (rows * j.in_w + 2) & ~1 : rows * bw;
        const int col_rows = col ? tr * (j.cfy ? 2 : 1) : 0;
        for (int f = kStReseed; f >= 8 && (!sp.tma || (bw <= 256 && rows <= 256)); f /= 2) {
            const size_t smem = (size_t)kStRing * f * fs * 2 + (size_t)f * col_rows * need * 4;
            if (smem > (f > 8 ? 56u : 75u) * 1024) continue;
            sp.ok = 1;
            sp.tc = tc;
            sp.tr = tr;
            sp.tiles_x = (j.out_w + tc - 1) / tc;
            sp.tiles_y = (j.out_h + tr - 1) / tr;
            sp.threads = col ? kStMaxThreads : (tc * tr + 31) & ~31;
            sp.fbox = f;
            sp.bw = bw;
            sp.rows = rows;
            sp.rs = rs;
            sp.fs = fs;
            sp.run = run;
            sp.col_rows = col_rows;
            sp.col_w = need;
            sp.smem = smem;
            if (!sp.tma) {
                const int warps = sp.threads / 32, copies = run ? 1 : rows;
                const bool boxes = j.binx * j.biny > 1
                                       ? run || rows <= 4 * warps
                                       : 4 * copies <= warps && j.npix >= 100 && (j.npix + 127) / 128 * nseg <= 600;
                if (!boxes) {
                    sp.ok = 0;
                    return sp;
                }
            }
            // several monitor segments per CTA keep its ring busy; one each
            // where that would leave SMs without a CTA
            sp.segs = 4;
            while (sp.segs > 1 && (long)sp.tiles_x * sp.tiles_y * ((nseg + sp.segs - 1) / sp.segs) < 4 * 152) sp.segs /= 2;
            return sp;
        }
        if (tr > 1) tr = (tr + 1) / 2;
        else if (tc > 1) tc = (tc + 1) / 2;
        else return sp;
    }
}

template <int MODE, bool CCF, bool BIN1>
static cudaError_t launch_stream_box(const StreamArgs &a, const StreamPlan &sp, const CUtensorMap &map, cudaStream_t s)
{
    auto kern = sp.tma ? stream_box_kernel<MODE, CCF, BIN1, true> : stream_box_kernel<MODE, CCF, BIN1, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sp.smem);
    if (e != cudaSuccess) return e;
    kern<<<dim3(sp.tiles_x * sp.tiles_y, (a.nseg + sp.segs - 1) / sp.segs), sp.threads, sp.smem, s>>>(a, map);
    return cudaGetLastError();
}

template <int MODE, bool CCF>
static cudaError_t launch_stream_t(const StreamArgs &a, const StreamPlan &sp, const CUtensorMap &map, cudaStream_t s)
{
    const Job &j = a.j;
    if (!sp.ok) {
        stream_plain_kernel<MODE, CCF><<<dim3((j.npix + 127) / 128, a.nseg), 128, 0, s>>>(a);
        return cudaGetLastError();
    }
    if (j.binx == 1 && j.biny == 1) return launch_stream_box<MODE, CCF, true>(a, sp, map, s);
    return launch_stream_box<MODE, CCF, false>(a, sp, map, s);
}

cudaError_t launch_stream(const Job &j, const void *stack, const float *bparams, const float *basis,
                          const int *snap_pos, int nseg, float *s0, float2 *segtot, float2 *snap_part, int *segbad,
                          int *snap_bad, int *err, cudaStream_t s)
{
    StreamArgs a;
    memset(&a, 0, sizeof(a));
    a.j = j;
    a.stack = stack;
    a.bparams = bparams;
    a.basis = basis;
    a.snap_pos = snap_pos;
    a.nseg = nseg;
    a.s0a = s0;
    a.s0b = j.is_ccf ? s0 + (size_t)j.npix * j.num : s0;
    a.segtot = segtot;
    a.snap_part = snap_part;
    a.segbad = segbad;
    a.snap_bad = snap_bad;
    a.err = err;
    StreamPlan sp = stream_plan(j, stack, nseg);
    CUtensorMap map;
    memset(&map, 0, sizeof(map));
    if (sp.ok && sp.tma) {
        PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
        cuuint64_t dims[3] = {(cuuint64_t)j.in_w, (cuuint64_t)j.in_h, (cuuint64_t)(j.first + j.num)};
        cuuint64_t strides[2] = {(cuuint64_t)j.in_w * 2, (cuuint64_t)j.in_w * j.in_h * 2};
        cuuint32_t box[3] = {(cuuint32_t)sp.bw, (cuuint32_t)sp.rows, (cuuint32_t)sp.fbox};
        cuuint32_t es[3] = {1, 1, 1};
        if (!enc || enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void *>(stack), dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            sp.ok = 0;
    }
    a.tc = sp.tc;
    a.tr = sp.tr;
    a.tiles_x = sp.tiles_x;
    a.fbox = sp.fbox;
    a.rows = sp.rows;
    a.fs = sp.fs;
    a.rs = sp.rs;
    a.run = sp.run;
    a.segs = sp.segs;
    a.col_rows = sp.col_rows;
    a.col_w = sp.col_w;
    switch (j.bleach) {
    case IMFCS_BLEACH_SINGLE_EXP:
        return j.is_ccf ? launch_stream_t<1, true>(a, sp, map, s) : launch_stream_t<1, false>(a, sp, map, s);
    case IMFCS_BLEACH_DOUBLE_EXP:
        return j.is_ccf ? launch_stream_t<2, true>(a, sp, map, s) : launch_stream_t<2, false>(a, sp, map, s);
    case IMFCS_BLEACH_POLYNOMIAL:
        return j.is_ccf ? launch_stream_t<3, true>(a, sp, map, s) : launch_stream_t<3, false>(a, sp, map, s);
    default:
        return j.is_ccf ? launch_stream_t<0, true>(a, sp, map, s) : launch_stream_t<0, false>(a, sp, map, s);
    }
}

// ---------------------------------------------------------------------------
// N&B mode (isNBcalculation, agpufitjni.cu:5719-5720 and calcacf2b
// 5167-5180): only lag 1 is evaluated.  NBmean = the mean of the direct
// window's first num-1 samples, NBcov = <I(t) I'(t+1)> - NBmean <I'>, over
// the same num-1 products -- from the corrected, centred level-0 stream
// (shift-invariant) and the lag-1 monitors.  Grid (pixel blocks, frame
// segments); float-float segment sums combined by FP64 atomics.
// ---------------------------------------------------------------------------
constexpr int kNbSeg = 2048;

__global__ void nb_lag1_kernel(int npix, int num, const float *s0a, const float *s0b, double *sum)
{
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= npix) return;
    const int t0 = blockIdx.y * kNbSeg, t1 = min(t0 + kNbSeg, num - 1);
    ff acc = {0.f, 0.f};
    for (int t = t0; t < t1; t++)
        ff_add(acc, __ldg(&s0a[(size_t)t * npix + pix]) * __ldg(&s0b[(size_t)(t + 1) * npix + pix]));
    atomicAdd(&sum[pix], ff_val(acc));
}

__global__ void nb_finalize_kernel(int npix, int chanum, int num, const float4 *mon, const double *sum,
                                   double *nb_mean, double *nb_cov)
{
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= npix) return;
    const float4 m = mon[(size_t)pix * chanum + 1];   // (a, b, dm, Dm) of lag 1
    const double n = (double)(num - 1);
    if (nb_mean) nb_mean[pix] = m.z;
    if (nb_cov) nb_cov[pix] = sum[pix] / n - (double)m.x * (double)m.y;
}

cudaError_t launch_nb_lag1(const Job &j, const float *s0, const float4 *mon, double *sum, double *nb_mean,
                           double *nb_cov, cudaStream_t s)
{
    const float *s0a = s0, *s0b = j.is_ccf ? s0 + (size_t)j.npix * j.num : s0;
    cudaError_t e = cudaMemsetAsync(sum, 0, sizeof(double) * j.npix, s);
    if (e != cudaSuccess) return e;
    dim3 grid((j.npix + 127) / 128, (j.num - 1 + kNbSeg - 1) / kNbSeg);
    nb_lag1_kernel<<<grid, 128, 0, s>>>(j.npix, j.num, s0a, s0b, sum);
    nb_finalize_kernel<<<(j.npix + 127) / 128, 128, 0, s>>>(j.npix, j.chanum, j.num, mon, sum, nb_mean, nb_cov);
    return cudaGetLastError();
}

}  // namespace imfcs
