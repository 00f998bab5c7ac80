// df64.cuh -- double-float arithmetic on the FP32 pipe.
//
// GB300 issues FP32 at 64 times its FP64 rate, so element arithmetic that
// the step would otherwise spend FP64 issue slots on runs here as pairs of
// floats: a value is the unevaluated sum hi + lo of two floats with
// |lo| <= ulp(hi)/2, which carries about 48 significant bits (relative
// rounding near 2^-47 per operation, against 2^-53 in FP64).
//
// The algorithms are the published error-free transformations and the
// double-word operations built on them, restated:
//   - two_sum: Knuth's two-sum (TAOCP vol. 2, 4.2.2), s + e == a + b exactly;
//   - fast_two_sum: Dekker's (1971) variant for |a| >= |b|;
//   - two_prod: the product and its exact remainder through one fused
//     multiply-add;
//   - df_add / df_mul / df_fma: the "sloppy" double-word sum and the
//     double-word product of Hida, Li and Bailey's QD library (2001) --
//     addition through two_sum of the high words, product through two_prod
//     plus the cross terms, each renormalised by fast_two_sum;
//   - reciprocal, quotient and square roots: an FP32 estimate corrected by
//     one step of its power series, the residual formed exactly.
// Every operation is written with the _rn intrinsics, which the compiler
// neither contracts nor reorders, so any kernel that inlines them rounds the
// same way.
//
// Conversions never touch the FP64 pipe: to_df splits a double's bit
// pattern with integer operations (hi = its leading 24 significand bits, lo
// = the next 24 of the remaining 29, both truncated), and to_double joins
// the two words with one FP64 addition.
#pragma once

#include <cuda_runtime.h>

namespace lulesh {

using ::fabs;
using ::fma;
using ::fmax;

struct df64 {
    float hi, lo;
    df64() = default;
    __host__ __device__ constexpr df64(float h, float l) : hi(h), lo(l) {}
    // compile-time constants only (a run-time double goes through to_df)
    __host__ __device__ constexpr explicit df64(double v) : hi((float)v), lo((float)(v - (double)(float)v)) {}
};

__device__ __forceinline__ df64 two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}

__device__ __forceinline__ df64 fast_two_sum(float a, float b)
{
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ df64 two_prod(float a, float b)
{
    const float p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ df64 df_add(df64 a, df64 b)
{
    const df64 s = two_sum(a.hi, b.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}

__device__ __forceinline__ df64 df_mul(df64 a, df64 b)
{
    const df64 p = two_prod(a.hi, b.hi);
    return fast_two_sum(p.hi, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, p.lo)));
}

// a * b + c with one renormalisation
__device__ __forceinline__ df64 df_fma(df64 a, df64 b, df64 c)
{
    const df64 p = two_prod(a.hi, b.hi);
    const float t = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, p.lo));
    const df64 s = two_sum(p.hi, c.hi);
    return fast_two_sum(s.hi, __fadd_rn(__fadd_rn(s.lo, t), c.lo));
}

// a times a float (exact in hi)
__device__ __forceinline__ df64 df_mul_f(df64 a, float b)
{
    const df64 p = two_prod(a.hi, b);
    return fast_two_sum(p.hi, __fmaf_rn(a.lo, b, p.lo));
}

// a times a power of two: exact
__device__ __forceinline__ df64 df_scale(df64 a, float pow2) { return {__fmul_rn(a.hi, pow2), __fmul_rn(a.lo, pow2)}; }

__device__ __forceinline__ df64 operator+(df64 a, df64 b) { return df_add(a, b); }
__device__ __forceinline__ df64 operator-(df64 a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ df64 operator-(df64 a, df64 b) { return df_add(a, -b); }
__device__ __forceinline__ df64 operator*(df64 a, df64 b) { return df_mul(a, b); }
__device__ __forceinline__ df64 fma(df64 a, df64 b, df64 c) { return df_fma(a, b, c); }
// the sign of a renormalised pair is the sign of its high word
__device__ __forceinline__ df64 fabs(df64 a) { return a.hi < 0.f ? -a : a; }
__device__ __forceinline__ bool df_gt(df64 a, df64 b) { return a.hi > b.hi || (a.hi == b.hi && a.lo > b.lo); }
__device__ __forceinline__ df64 fmax(df64 a, df64 b) { return df_gt(b, a) ? b : a; }

// The FP32 estimates that the functions below refine (the hardware's
// approximate reciprocal and inverse square root, a few units in the last
// place; subnormal arguments included).
__device__ __forceinline__ float rcp_estimate(float b)
{
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(b));
    return r;
}
__device__ __forceinline__ float rsqrt_estimate(float a)
{
    float r;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// Reciprocal, quotient and roots: one series step from the FP32 estimate
// instead of two Newton steps carried out in pairs.  The estimate is first
// refined to a correctly rounded float y or next to one; then its residual,
// 1 - b y or 1 - a y^2 and so on, below 2^-22, is formed by fused
// multiply-adds whose large terms cancel exactly, as a float t and a
// remainder g that also holds the series' second term, and y (t + g) is added
// to y with one rounding of each word.  The first neglected term is of order
// t^3; what remains is a rounding or two of the low word, near 2^-49.  Each
// takes 12-16 FP32 operations where the Newton forms take 72-110 and the
// reciprocal's correctly rounded estimate is a software routine of its own.
// Errors over 2^20 pairs (lulesh_probe_pairs), root mean square and largest,
// the Newton forms' in brackets: 1/b 2^-49.6 and 2^-47.1 (-48.8, -46.0), a/b
// 2^-49.5 and 2^-46.7 (-48.5, -45.5), 1/sqrt(a) 2^-49.4 and 2^-46.4 (-49.2,
// -46.3), sqrt(a) 2^-49.1 and 2^-46.0 (-48.3, -45.5).  With the residual in
// one float, three operations fewer, 1/b and 1/sqrt(a) were a fifth of a bit
// above the Newton forms' instead, sqrt(a) a quarter at worst; the material
// kernel takes 504 us for 486 at s=192 with the remainders (68.0 for 67.6 at
// s=96), the kinematics kernel 1221 for 1228.

// y + s (t + g), |s t| << |y|, |g| << |t|, with one rounding of each word
__device__ __forceinline__ df64 df_corrected(float y, float s, float t, float g)
{
    const float hi = __fmaf_rn(s, t, y);
    return {hi, __fmaf_rn(s, g, __fmaf_rn(s, t, __fsub_rn(y, hi)))};
}

// 1/b = y (1 + e + e^2 + ...)
__device__ __forceinline__ df64 df_rcp(df64 b)
{
    const float y0 = rcp_estimate(b.hi);
    const float y = __fmaf_rn(y0, __fmaf_rn(-b.hi, y0, 1.f), y0);
    const float e = __fmaf_rn(-b.hi, y, 1.f), t = __fmaf_rn(-b.lo, y, e);
    return df_corrected(y, y, t, __fmaf_rn(t, t, __fmaf_rn(-b.lo, y, __fsub_rn(e, t))));
}

// a/b: the FP32 quotient q by the refined reciprocal y, then its remainder
// a - b q (exact in its high words) times y (1 + e)
__device__ __forceinline__ df64 df_div(df64 a, df64 b)
{
    const float y0 = rcp_estimate(b.hi);
    const float y = __fmaf_rn(y0, __fmaf_rn(-b.hi, y0, 1.f), y0);
    const float e = __fmaf_rn(-b.lo, y, __fmaf_rn(-b.hi, y, 1.f));
    const float q = __fmul_rn(a.hi, y);
    const float r = __fmaf_rn(-b.hi, q, a.hi), f = __fmaf_rn(-b.lo, q, a.lo), t = __fadd_rn(r, f);
    return df_corrected(q, y, t, __fmaf_rn(t, e, __fadd_rn(__fsub_rn(r, t), f)));
}

// 1/sqrt(a) = y (1 + e/2 + 3 e^2/8 + ...), a > 0
__device__ __forceinline__ df64 df_rsqrt(df64 a)
{
    const float y0 = rsqrt_estimate(a.hi);
    const float y = __fmaf_rn(__fmul_rn(0.5f, y0), __fmaf_rn(-a.hi, __fmul_rn(y0, y0), 1.f), y0);
    const df64 s = two_prod(y, y);
    const float e = __fmaf_rn(-a.hi, s.hi, 1.f), f = __fmaf_rn(-a.lo, s.hi, __fmul_rn(-a.hi, s.lo));
    const float t = __fadd_rn(e, f);
    return df_corrected(y, __fmul_rn(0.5f, y), t, __fmaf_rn(__fmul_rn(0.75f, t), t, __fadd_rn(__fsub_rn(e, t), f)));
}

// sqrt(a), a > 0: the FP32 root x by the refined inverse root y, then its
// remainder r = a - x^2 (exact in its high words) times y/2 (1 + 3 u/4), u =
// 1 - x y: of the factor's own error, that much and a quarter of x's rounding
// is left
__device__ __forceinline__ df64 df_sqrt(df64 a)
{
    const float y0 = rsqrt_estimate(a.hi);
    const float y = __fmaf_rn(__fmul_rn(0.5f, y0), __fmaf_rn(-a.hi, __fmul_rn(y0, y0), 1.f), y0);
    const float x = __fmul_rn(a.hi, y), u = __fmaf_rn(-x, y, 1.f);
    const float r = __fmaf_rn(-x, x, a.hi), t = __fadd_rn(r, a.lo), h = __fmul_rn(0.5f, y);
    const float hi = __fmaf_rn(h, t, x);
    // (r and a.lo apart: this one needs no exact remainder of their sum)
    return {hi, __fmaf_rn(h, __fmaf_rn(t, __fmul_rn(0.75f, u), a.lo), __fmaf_rn(h, r, __fsub_rn(x, hi)))};
}

// The Newton forms: two steps r <- r + r (1 - b r) or y <- y + y (1 - a y^2)/2
// in pairs from the FP32 value.  The split-precision kernels keep them: their
// FP32 forces magnify a change in the last bit of a time step or volume to
// 1e-7 of the state within tens of cycles, so these kernels' results stay
// bit for bit what they were.  Written out with what is known about the
// operands: 1 - m with m near 1 is exact in its high words, the correction
// is smaller than what it corrects (fast_two_sum), and the first step's
// low word is zero; the same bits as the general operations in 43-50 FP32
// operations instead of 66-80.
__device__ __forceinline__ df64 df_one_minus(df64 m) { return fast_two_sum(__fsub_rn(1.f, m.hi), -m.lo); }

// c + a b, |a b| < |c|
__device__ __forceinline__ df64 df_fma_small(df64 a, df64 b, df64 c)
{
    const df64 p = two_prod(a.hi, b.hi);
    const float t = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, p.lo));
    const df64 s = fast_two_sum(c.hi, p.hi);
    return fast_two_sum(s.hi, __fadd_rn(__fadd_rn(s.lo, t), c.lo));
}

// c + c e for a float c, |e| < 1
__device__ __forceinline__ df64 df_fma_small(float a, df64 b, float c)
{
    const df64 p = two_prod(a, b.hi);
    const df64 s = fast_two_sum(c, p.hi);
    return fast_two_sum(s.hi, __fadd_rn(s.lo, __fmaf_rn(a, b.lo, p.lo)));
}

__device__ __forceinline__ df64 df_rcp_newton(df64 b)
{
    const float r0 = __frcp_rn(b.hi);
    const df64 r = df_fma_small(r0, df_one_minus(df_mul_f(b, r0)), r0);
    return df_fma_small(r, df_one_minus(df_mul(b, r)), r);
}

// a / b: the quotient through the reciprocal, corrected once by the
// remainder a - q b
__device__ __forceinline__ df64 df_div_newton(df64 a, df64 b)
{
    const df64 r = df_rcp_newton(b);
    const df64 q = df_mul(a, r);
    const df64 rem = df_add(a, -df_mul(q, b));
    return df_fma(rem, r, q);
}

__device__ __forceinline__ df64 df_rsqrt_newton(df64 a)
{
    const float y0 = rsqrtf(a.hi);
    const df64 y = df_fma_small(__fmul_rn(0.5f, y0), df_one_minus(df_mul(a, two_prod(y0, y0))), y0);
    return df_fma_small(df_scale(y, 0.5f), df_one_minus(df_mul(a, df_mul(y, y))), y);
}

// The two sets, for the code that both precisions share
struct SeriesFn {
    static __device__ __forceinline__ df64 rcp(df64 b) { return df_rcp(b); }
    static __device__ __forceinline__ df64 div(df64 a, df64 b) { return df_div(a, b); }
    static __device__ __forceinline__ df64 rsqrt(df64 a) { return df_rsqrt(a); }
    static __device__ __forceinline__ df64 sqrt(df64 a) { return df_sqrt(a); }
};
struct NewtonFn {
    static __device__ __forceinline__ df64 rcp(df64 b) { return df_rcp_newton(b); }
    static __device__ __forceinline__ df64 div(df64 a, df64 b) { return df_div_newton(a, b); }
    static __device__ __forceinline__ df64 rsqrt(df64 a) { return df_rsqrt_newton(a); }
    static __device__ __forceinline__ df64 sqrt(df64 a) { return df_mul(a, df_rsqrt_newton(a)); }
};

// ---- conversions --------------------------------------------------------

// double -> pair without the FP64 pipe.  hi takes the 24 leading
// significand bits, lo the next 24 of the remaining 29, both truncated:
// |v - (hi + lo)| < 2^-47 |v|.  For an exponent e of v (v = 1.f 2^e) the
// float exponent field of hi is e + 127, which the bits 60..29 of v plus
// 2^30 give directly (the low nine bits of v's biased exponent, minus 384,
// modulo 2^32); lo is the 29-bit remainder r, signed, converted to float
// rounding toward zero (its 24 leading bits) and scaled by 2^(e-52).
// Magnitudes outside [2^-74, 2^128), where lo or hi would leave the normal
// float range, keep hi only (an error below 2^-98 absolute): zeros,
// infinities and NaNs map to themselves.  The small ones by selects in the
// same instructions, not in a path of their own: zeros stand in most warps
// (differences along the axes, gas at rest), and a second path took each of
// those warps through both (at s=192 the plain kinematics kernel 1267 -> 1222
// us, the split one 921 -> 891).
__device__ __forceinline__ df64 to_df(double v)
{
    const unsigned lo32 = (unsigned)__double2loint(v), hi32 = (unsigned)__double2hiint(v);
    const unsigned sign = hi32 & 0x80000000u;
    const unsigned de = (hi32 >> 20) & 0x7ffu;   // biased exponent, e + 1023
    unsigned hb = (__funnelshift_r(lo32, hi32, 29) + 0x40000000u) | sign;
    const int m = (int)hi32 >> 31;            // 0 or -1
    const int r = (int)(((lo32 & 0x1fffffffu) ^ (unsigned)m) - (unsigned)m);   // +-remainder
    unsigned scale = (max(de, 948u) - 948u) << 23;
    if (de < 897u) hb = sign;
    if (de > 1150u) {
        hb = de == 0x7ffu && ((hi32 & 0xfffffu) | lo32) != 0u ? sign | 0x7fc00000u : sign | 0x7f800000u;
        scale = 0u;
    }
    return {__uint_as_float(hb), __int2float_rz(r) * __uint_as_float(scale)};
}

// float -> double with integer operations (normal floats and zeros exact;
// subnormals flush to a signed zero, infinities and NaNs kept).
__device__ __forceinline__ double df_f2d(float f)
{
    const unsigned u = __float_as_uint(f);
    const unsigned fe = u & 0x7f800000u;
    unsigned hi = (((int)u >> 3) & 0x8fffffffu) + 0x38000000u, lo = u << 29;   // the exponent rebiased by 896
    if (fe == 0u) {
        hi = u & 0x80000000u;
        lo = 0u;
    }
    if (fe == 0x7f800000u) hi |= 0x7ff00000u;
    return __hiloint2double((int)hi, (int)lo);
}

// pair -> double: one FP64 addition (the correctly rounded sum of the words)
__device__ __forceinline__ double to_double(df64 a) { return df_f2d(a.hi) + df_f2d(a.lo); }

__device__ __forceinline__ float2 as_float2(df64 a) { return make_float2(a.hi, a.lo); }
__device__ __forceinline__ df64 as_df(float2 f) { return {f.x, f.y}; }

}  // namespace lulesh
