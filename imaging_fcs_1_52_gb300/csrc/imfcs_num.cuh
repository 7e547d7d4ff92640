// imfcs_num.cuh -- sums, quotients and roots at FP64 precision with few
// operations on the FP64 pipe, which GB300 issues at 1/64 of the FP32 rate.
#pragma once

namespace imfcs {

// ---------------------------------------------------------------------------
// Compensated accumulation of FP32 values: exact two-sums (Knuth).
// ---------------------------------------------------------------------------
// Two terms, about 48 bits.
struct ff {
    float hi, lo;
};
__device__ __forceinline__ float two_sum_err(float a, float b, float s)     // a + b - s, s = fl(a + b)
{
    const float bb = __fsub_rn(s, a);
    return __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
__device__ __forceinline__ void ff_add(ff &a, float b)
{
    const float s = __fadd_rn(a.hi, b);
    const float err = two_sum_err(a.hi, b, s);
    a.hi = s;
    a.lo = __fadd_rn(a.lo, err);
}
__device__ __forceinline__ double ff_val(const ff &a) { return (double)a.hi + (double)a.lo; }

// Three terms: the errors of the first sum are summed with their own errors
// kept, so that thousands of values add up to less than an FP64 rounding (an
// FP64 running sum makes one per value; two terms lose up to n 2^-48).
struct ff3 {
    float hi, mid, lo;
};
__device__ __forceinline__ void ff3_add(ff3 &a, float b)
{
    const float s = __fadd_rn(a.hi, b);
    const float e = two_sum_err(a.hi, b, s);
    const float m = __fadd_rn(a.mid, e);
    a.lo = __fadd_rn(a.lo, two_sum_err(a.mid, e, m));
    a.hi = s;
    a.mid = m;
}
// b: below the last place of the values (the low term of one)
__device__ __forceinline__ void ff3_add_low(ff3 &a, float b)
{
    const float m = __fadd_rn(a.mid, b);
    a.lo = __fadd_rn(a.lo, two_sum_err(a.mid, b, m));
    a.mid = m;
}

// the square of a
__device__ __forceinline__ void ff3_add_square(ff3 &s, const ff3 &a)
{
    const float p = __fmul_rn(a.hi, a.hi), pe = fmaf(a.hi, a.hi, -p);
    const float h2 = 2.f * a.hi, q = __fmul_rn(h2, a.mid), qe = fmaf(h2, a.mid, -q);
    ff3_add(s, p);
    ff3_add_low(s, pe);
    ff3_add_low(s, q);
    s.lo = __fadd_rn(s.lo, fmaf(h2, a.lo, fmaf(a.mid, a.mid, qe)));
}

// float -> double off the FP64 pipe, where the conversion instruction runs at
// 1/64 of the FP32 rate (exact): the exponent rebiased, the fraction moved.
// Subnormal values are scaled by 2^64 first; selects, no branch, so that the
// instruction is never issued beside them.
__device__ __forceinline__ double f2d(float x)
{
    unsigned m = __float_as_uint(x) & 0x7fffffffu;
    unsigned bias = m >= 0x7f800000u ? 0x70000000u : 0x38000000u;
    const unsigned scaled = __float_as_uint(fabsf(x) * 18446744073709551616.f);
    if (m < 0x00800000u) {
        m = scaled;
        bias = m ? 0x34000000u : 0u;
    }
    const unsigned hi = ((m >> 3) + bias) | (__float_as_uint(x) & 0x80000000u);
    return __hiloint2double((int)hi, (int)(m << 29));
}

__device__ __forceinline__ double ff3_val(const ff3 &a) { return f2d(a.hi) + (f2d(a.mid) + f2d(a.lo)); }

// 1/x to 46 bits (for div_near) and sqrt(x) within 0.5 ulp and 1e-15, by
// Newton's iteration from an FP32 start: two and six FP64 operations.  xf: x
// within a few FP32 ulps, from a caller that has it without a conversion.
// Arguments outside [1e-30, 1e30] (and non-finite, zero, negative ones) take
// the plain operation.
static __device__ __noinline__ double plain_div(double x, double y) { return x / y; }
static __device__ __noinline__ double plain_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ double rcp_near(double x, float xf)
{
    const float f = fabsf(xf);
    if (!(f > 1e-30f && f < 1e30f)) return plain_div(1.0, x);
    const double r = f2d(1.f / xf);
    return fma(fma(-x, r, 1.0), r, r);
}
__device__ __forceinline__ double newton_sqrt(double x)
{
    const float f = (float)x;
    if (!(f > 1e-30f && f < 1e30f)) return plain_sqrt(x);
    const float yf = rsqrtf(f);
    const double y = f2d(yf), h = f2d(0.5f * yf);
    double s = x * y;                      // sqrt(x) (1 - e), h = 1 / (2 sqrt(x))
    s = fma(s, fma(-s, h, 0.5), s);
    return fma(fma(-s, s, x), h, s);
}

// x / n, correctly rounded, from inv = 1 / n correctly rounded (n a small
// whole number): the quotient's remainder corrects it (Markstein).  The means
// of unbleached recordings are ratios of short numbers that sit on FP32
// rounding ties, so x * inv alone would round some of them the other way.
__device__ __forceinline__ double div_by(double x, double n, double inv)
{
    const double q = x * inv;
    return fma(fma(-q, n, x), inv, q);
}

// x / y the same way from a reciprocal `inv` of y good to 40 bits (its error
// enters squared): within 0.5 ulp and 1e-9.  The plain division where the
// quotient is zero, non-finite or tiny (y outside the range of its reciprocal
// among them).
__device__ __forceinline__ double div_near(double x, double y, double inv)
{
    const double q = x * inv;
    const unsigned e = ((unsigned)__double2hiint(q) >> 20 & 0x7ffu) - 300u;      // 2^-723 .. 2^577
    if (e > 1300u) return plain_div(x, y);
    return fma(fma(-q, y, x), inv, q);
}

// x / d for d = 2 .. 8, the bits of the division: the same correction in FP32.
template <int D>
__device__ __forceinline__ float div_small(float x)
{
    if constexpr ((D & (D - 1)) == 0) return x * (1.f / D);
    constexpr float inv = 1.f / D;
    const float q = __fmul_rn(x, inv);
    return fmaf(fmaf(-q, (float)D, x), inv, q);
}

}  // namespace imfcs
