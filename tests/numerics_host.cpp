// The device's number helpers (imfcs_num.cuh) on the host: its intrinsics as
// the IEEE operations they are, rsqrtf two ulps off (its stated error).
// Compiled with -ffp-contract=off by test_numerics.py.
#include <math.h>
#include <stdint.h>
#include <string.h>

#define __device__
#define __forceinline__ inline
#define __noinline__
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline unsigned __float_as_uint(float x) { unsigned u; memcpy(&u, &x, 4); return u; }
static inline double __hiloint2double(int hi, int lo)
{
    const uint64_t u = (uint64_t)(unsigned)hi << 32 | (unsigned)lo;
    double d;
    memcpy(&d, &u, 8);
    return d;
}
static inline int __double2hiint(double x)
{
    uint64_t u;
    memcpy(&u, &x, 8);
    return (int)(u >> 32);
}
static int rsqrt_ulps = 0;
static inline float rsqrtf(float x)
{
    float r = (float)(1.0 / sqrt((double)x));
    for (int i = 0; i < rsqrt_ulps; i++) r = nextafterf(r, INFINITY);
    for (int i = 0; i > rsqrt_ulps; i--) r = nextafterf(r, 0.f);
    return r;
}
#include "imfcs_num.cuh"

extern "C" {
double num_sum2(const float *x, int n)
{
    imfcs::ff a = {0.f, 0.f};
    for (int i = 0; i < n; i++) imfcs::ff_add(a, x[i]);
    return imfcs::ff_val(a);
}
double num_sum3(const float *x, int n)
{
    imfcs::ff3 a = {0.f, 0.f, 0.f};
    for (int i = 0; i < n; i++) imfcs::ff3_add(a, x[i]);
    return imfcs::ff3_val(a);
}
double num_f2d(float x) { return imfcs::f2d(x); }
double num_sum3_low(const float *x, const float *low, int n)
{
    imfcs::ff3 a = {0.f, 0.f, 0.f};
    for (int i = 0; i < n; i++) {
        imfcs::ff3_add(a, x[i]);
        imfcs::ff3_add_low(a, low[i]);
    }
    return imfcs::ff3_val(a);
}
// sum of the squares of the sums of runs of k values
double num_sum3_squares(const float *x, int n, int k)
{
    imfcs::ff3 s = {0.f, 0.f, 0.f};
    for (int i = 0; i < n; i += k) {
        imfcs::ff3 a = {0.f, 0.f, 0.f};
        for (int u = 0; u < k; u++) imfcs::ff3_add(a, x[i + u]);
        imfcs::ff3_add_square(s, a);
    }
    return imfcs::ff3_val(s);
}
// the FP32 start of the reciprocal a few ulps off
double num_rcp(double x, int ulps)
{
    float f = (float)x;
    for (int i = 0; i < ulps; i++) f = nextafterf(f, INFINITY);
    for (int i = 0; i > ulps; i--) f = nextafterf(f, -INFINITY);
    return imfcs::rcp_near(x, f);
}
double num_div(double x, double y, int ulps) { return imfcs::div_near(x, y, num_rcp(y, ulps)); }
double num_div_by(double x, double n) { return imfcs::div_by(x, n, 1.0 / n); }
double num_sqrt(double x, int ulps)
{
    rsqrt_ulps = ulps;
    return imfcs::newton_sqrt(x);
}
// mantissas for which div_small<D> is not x / D
int num_div_small_misses()
{
    int miss = 0;
    for (unsigned m = 0; m < 1u << 23; m++) {
        const unsigned u = 0x3f800000u | m;
        float x;
        memcpy(&x, &u, 4);
        miss += imfcs::div_small<2>(x) != x / 2 || imfcs::div_small<3>(x) != x / 3 || imfcs::div_small<4>(x) != x / 4 ||
                imfcs::div_small<5>(x) != x / 5 || imfcs::div_small<6>(x) != x / 6 || imfcs::div_small<7>(x) != x / 7 ||
                imfcs::div_small<8>(x) != x / 8;
    }
    return miss;
}
}
