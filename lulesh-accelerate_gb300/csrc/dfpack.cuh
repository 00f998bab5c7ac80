// dfpack.cuh -- double-float arithmetic two values at a time.
//
// sm_103a has FP32 add, subtract, multiply and fused multiply-add on pairs of
// floats held in one 64-bit register.  They run at the scalar instructions'
// rate per float (measured 59-64 instructions, 118-128 floats, per SM and
// clock against 120-122), so they raise no FP32 peak, but they take half the
// issue slots, and the double-float kernels are bound by issue: ~12 FP32
// operations per multiply-add, beside conversions, moves and addresses.
// Every operation rounds each half exactly as the scalar one does.
//
// df2 holds two double-float values (df64.cuh): hi and lo are pairs of
// floats, one half per value.  The pairing is chosen by the data flow -- two
// modes, two vectors, two corners that take the same operations -- so that
// the halves rarely move between registers.  The pair instructions have no
// operand negation (a scalar one is free), so the products below take one
// operand with its negative at hand (df2n).
#pragma once

#include "df64.cuh"

namespace lulesh {

typedef unsigned long long f2;   // two floats, .x in the low word

__device__ __forceinline__ f2 f2_add(f2 a, f2 b)
{
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b)
{
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// The product as a fused multiply-add with zero (a zero product comes out as
// +0): the assembler contracts a pair multiplication and an addition of its
// result into one fused operation even where both say .rn, which would round
// two_sum's operands differently from place to place.
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b)
{
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(0ULL));
    return d;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 f2_pack(float x, float y)
{
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ float f2_x(f2 a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    (void)y;
    return x;
}
__device__ __forceinline__ float f2_y(f2 a)
{
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    (void)x;
    return y;
}
__device__ __forceinline__ f2 f2_neg(f2 a) { return a ^ 0x8000000080000000ULL; }

struct df2 {
    f2 hi, lo;
};
// a value with its high word's negative
struct df2n {
    f2 hi, lo, nhi;
};

__device__ __forceinline__ df2 df2_pack(df64 x, df64 y) { return {f2_pack(x.hi, y.hi), f2_pack(x.lo, y.lo)}; }
__device__ __forceinline__ df2 df2_dup(df64 x) { return df2_pack(x, x); }
__device__ __forceinline__ df64 df2_x(df2 a) { return {f2_x(a.hi), f2_x(a.lo)}; }
__device__ __forceinline__ df64 df2_y(df2 a) { return {f2_y(a.hi), f2_y(a.lo)}; }
__device__ __forceinline__ df2n df2_both(df2 a) { return {a.hi, a.lo, f2_neg(a.hi)}; }

__device__ __forceinline__ df2 f2_two_sum(f2 a, f2 b)
{
    const f2 s = f2_add(a, b);
    const f2 bb = f2_sub(s, a);
    return {s, f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb))};
}
__device__ __forceinline__ df2 f2_two_diff(f2 a, f2 b)
{
    const f2 s = f2_sub(a, b);
    const f2 bb = f2_sub(s, a);   // -b, rounded
    return {s, f2_sub(f2_sub(a, f2_sub(s, bb)), f2_add(b, bb))};
}
__device__ __forceinline__ df2 df2_renorm(df2 a) { return f2_two_sum(a.hi, a.lo); }

// Sums whose low word gathers the low words and the exact rounding error of
// the high words' sum, not renormalised: eight operations where a
// renormalised sum takes eleven.  A chain of them is renormalised once at
// its end.
__device__ __forceinline__ df2 df2_add(df2 a, df2 b)
{
    const df2 s = f2_two_sum(a.hi, b.hi);
    return {s.hi, f2_add(s.lo, f2_add(a.lo, b.lo))};
}
__device__ __forceinline__ df2 df2_sub(df2 a, df2 b)
{
    const df2 s = f2_two_diff(a.hi, b.hi);
    return {s.hi, f2_add(s.lo, f2_sub(a.lo, b.lo))};
}
__device__ __forceinline__ df64 df_sum(df64 a, df64 b)
{
    const df64 s = two_sum(a.hi, b.hi);
    return {s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo))};
}
__device__ __forceinline__ df64 df_renorm(df64 a) { return two_sum(a.hi, a.lo); }
__device__ __forceinline__ df64 df_tidy(df64 a) { return fast_two_sum(a.hi, a.lo); }

// Sums of products (the compensated dot product of Ogita, Rump and Oishi,
// 2005, on pairs) in both halves: each product's high word joins the running
// high word through two_sum and every low-order term collects in one word;
// 12 operations per term, renormalised once at the end.  The low-order words
// are added before the rounding error of the high words' sum, so that two
// terms, or two partial sums, give the same bits in either order.  The high
// word is held negated: -a b and its exact remainder a b - (-(-a b)) then
// need no more than the factor's negative, once for all of its products.
struct Dot2 {
    f2 ns, e;   // the sum is e - ns
    // a b, the first term
    __device__ __forceinline__ Dot2(df2 a, df2n b)
    {
        ns = f2_mul(a.hi, b.nhi);
        e = f2_fma(a.hi, b.lo, f2_fma(a.lo, b.hi, f2_fma(a.hi, b.hi, ns)));
    }
    __device__ __forceinline__ Dot2(f2 minus_hi, f2 lo) : ns(minus_hi), e(lo) {}
    __device__ __forceinline__ Dot2 &plus(Dot2 t)
    {
        const df2 q = f2_two_sum(ns, t.ns);
        ns = q.hi;
        e = f2_sub(f2_add(e, t.e), q.lo);
        return *this;
    }
    __device__ __forceinline__ Dot2 &minus(Dot2 t)
    {
        const df2 q = f2_two_diff(ns, t.ns);
        ns = q.hi;
        e = f2_sub(f2_sub(e, t.e), q.lo);
        return *this;
    }
    __device__ __forceinline__ Dot2 &minus(df2 c)
    {
        const df2 q = f2_two_sum(ns, c.hi);
        ns = q.hi;
        e = f2_sub(f2_sub(e, c.lo), q.lo);
        return *this;
    }
    __device__ __forceinline__ Dot2 &add(df2 a, df2n b) { return plus(Dot2(a, b)); }
    __device__ __forceinline__ Dot2 &sub(df2 a, df2n b) { return minus(Dot2(a, b)); }
    // the sum and its negative, renormalised for |ns| >= |e|; when the high
    // words cancel further than that, the error stays at 2^-24 |e|, the
    // sum's own
    __device__ __forceinline__ df2 value() const
    {
        const f2 h = f2_sub(e, ns);
        return {h, f2_sub(e, f2_add(h, ns))};
    }
    __device__ __forceinline__ df2 negative() const
    {
        const f2 h = f2_sub(ns, e);
        return {h, f2_sub(f2_sub(ns, h), e)};
    }
    __device__ __forceinline__ df2 raw_negative() const { return {ns, f2_neg(e)}; }
};

// a times b, renormalised
__device__ __forceinline__ df2 df2_mul(df2 a, df2n b) { return Dot2(a, b).value(); }

// The scalar counterpart, one value.
struct Dot1 {
    float s, e;   // the sum is s + e
    __device__ __forceinline__ Dot1(df64 a, df64 b)
    {
        const df64 p = two_prod(a.hi, b.hi);
        s = p.hi;
        e = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, p.lo));
    }
    __device__ __forceinline__ Dot1(float hi, float lo) : s(hi), e(lo) {}
    __device__ __forceinline__ Dot1 &plus(Dot1 t)
    {
        const df64 q = two_sum(s, t.s);
        s = q.hi;
        e = __fadd_rn(__fadd_rn(e, t.e), q.lo);
        return *this;
    }
    __device__ __forceinline__ Dot1 &add(df64 a, df64 b) { return plus(Dot1(a, b)); }
    __device__ __forceinline__ Dot1 &sub(df64 a, df64 b) { return add(a, -b); }
    __device__ __forceinline__ df64 value() const { return fast_two_sum(s, e); }
};
// the two halves of a sum
__device__ __forceinline__ Dot1 dot_x(const Dot2 &d) { return {-f2_x(d.ns), f2_x(d.e)}; }
__device__ __forceinline__ Dot1 dot_y(const Dot2 &d) { return {-f2_y(d.ns), f2_y(d.e)}; }
__device__ __forceinline__ Dot1 minus(const Dot1 &d) { return {-d.s, -d.e}; }
__device__ __forceinline__ Dot1 joined(const Dot2 &d) { return dot_x(d).plus(dot_y(d)); }
__device__ __forceinline__ Dot1 difference(const Dot2 &d) { return dot_x(d).plus(minus(dot_y(d))); }

// ---- vectors ------------------------------------------------------------
struct V2x3 {   // two vectors
    df2 x, y, z;
};
struct V2x3n {
    df2n x, y, z;
};
struct V1x3 {   // one
    df64 x, y, z;
};
__device__ __forceinline__ V2x3n both(const V2x3 &a) { return {df2_both(a.x), df2_both(a.y), df2_both(a.z)}; }
__device__ __forceinline__ V2x3 first_of(const V2x3n &a) { return {{a.x.hi, a.x.lo}, {a.y.hi, a.y.lo}, {a.z.hi, a.z.lo}}; }
__device__ __forceinline__ V1x3 half_x(const V2x3 &a) { return {df2_x(a.x), df2_x(a.y), df2_x(a.z)}; }
__device__ __forceinline__ V1x3 half_y(const V2x3 &a) { return {df2_y(a.x), df2_y(a.y), df2_y(a.z)}; }
__device__ __forceinline__ V2x3 pack3(const V1x3 &a, const V1x3 &b)
{
    return {df2_pack(a.x, b.x), df2_pack(a.y, b.y), df2_pack(a.z, b.z)};
}
__device__ __forceinline__ V1x3 minus(const V1x3 &a) { return {-a.x, -a.y, -a.z}; }

__device__ __forceinline__ V2x3 dup3(const V1x3 &a) { return {df2_dup(a.x), df2_dup(a.y), df2_dup(a.z)}; }
__device__ __forceinline__ V2x3n swapped(const V2x3n &a)
{
    auto sw = [](f2 v) { return f2_pack(f2_y(v), f2_x(v)); };
    auto comp = [&](const df2n &v) { return df2n{sw(v.hi), sw(v.lo), sw(v.nhi)}; };
    return {comp(a.x), comp(a.y), comp(a.z)};
}

// Cross products.  In cross2/cross1 exchanging the two products of a
// component negates it exactly; in the _even forms each product also rounds
// alike with its factors exchanged (two operations more), so that b x a is
// exactly -(a x b).
__device__ __forceinline__ V2x3 cross2(const V2x3 &a, const V2x3n &b)
{
    return {Dot2(a.y, b.z).sub(a.z, b.y).value(), Dot2(a.z, b.x).sub(a.x, b.z).value(),
            Dot2(a.x, b.y).sub(a.y, b.x).value()};
}
__device__ __forceinline__ V1x3 cross1(const V1x3 &a, const V1x3 &b)
{
    return {Dot1(a.y, b.z).sub(a.z, b.y).value(), Dot1(a.z, b.x).sub(a.x, b.z).value(),
            Dot1(a.x, b.y).sub(a.y, b.x).value()};
}
__device__ __forceinline__ Dot2 even_product(df2 u, df2n v)
{
    const f2 np = f2_mul(u.hi, v.nhi);
    return {np, f2_add(f2_fma(u.hi, v.hi, np), f2_add(f2_mul(u.hi, v.lo), f2_mul(u.lo, v.hi)))};
}
__device__ __forceinline__ Dot1 even_product(df64 u, df64 v)
{
    const df64 p = two_prod(u.hi, v.hi);
    return {p.hi, __fadd_rn(p.lo, __fadd_rn(__fmul_rn(u.hi, v.lo), __fmul_rn(u.lo, v.hi)))};
}
__device__ __forceinline__ V2x3 cross2_even(const V2x3 &a, const V2x3n &b)
{
    auto minor = [](df2 u, df2n v, df2 w, df2n x) { return even_product(u, v).minus(even_product(w, x)).value(); };
    return {minor(a.y, b.z, a.z, b.y), minor(a.z, b.x, a.x, b.z), minor(a.x, b.y, a.y, b.x)};
}
__device__ __forceinline__ V1x3 cross1_even(const V1x3 &a, const V1x3 &b)
{
    auto minor = [](df64 u, df64 v, df64 w, df64 x) { return even_product(u, v).plus(even_product(w, -x)).value(); };
    return {minor(a.y, b.z, a.z, b.y), minor(a.z, b.x, a.x, b.z), minor(a.x, b.y, a.y, b.x)};
}
// a x b + c x d
__device__ __forceinline__ V1x3 cross1_sum(const V1x3 &a, const V1x3 &b, const V1x3 &c, const V1x3 &d)
{
    return {Dot1(a.y, b.z).sub(a.z, b.y).plus(Dot1(c.y, d.z).sub(c.z, d.y)).value(),
            Dot1(a.z, b.x).sub(a.x, b.z).plus(Dot1(c.z, d.x).sub(c.x, d.z)).value(),
            Dot1(a.x, b.y).sub(a.y, b.x).plus(Dot1(c.x, d.y).sub(c.y, d.x)).value()};
}
__device__ __forceinline__ V2x3 cross2_sum(const V2x3 &a, const V2x3n &b, const V2x3 &c, const V2x3n &d)
{
    return {Dot2(a.y, b.z).sub(a.z, b.y).plus(Dot2(c.y, d.z).sub(c.z, d.y)).value(),
            Dot2(a.z, b.x).sub(a.x, b.z).plus(Dot2(c.z, d.x).sub(c.x, d.z)).value(),
            Dot2(a.x, b.y).sub(a.y, b.x).plus(Dot2(c.x, d.y).sub(c.y, d.x)).value()};
}
// a . b, x and y exchangeable
__device__ __forceinline__ Dot2 dot2(const V2x3 &a, const V2x3n &b) { return Dot2(a.x, b.x).add(a.y, b.y).add(a.z, b.z); }
__device__ __forceinline__ Dot1 dot1(const V1x3 &a, const V1x3 &b) { return Dot1(a.x, b.x).add(a.y, b.y).add(a.z, b.z); }
__device__ __forceinline__ V1x3 sum1(const V1x3 &a, const V1x3 &b)
{
    return {df_tidy(df_sum(a.x, b.x)), df_tidy(df_sum(a.y, b.y)), df_tidy(df_sum(a.z, b.z))};
}

// ---- Walsh modes ----------------------------------------------------------
// One field's 8 corner values relative to corner 0: FP64 differences (exact
// for neighbouring values) split into pairs, r = (r1, r5), (r3, r7),
// (r2, r6) and r4.  to_df truncates, so its low words reach a whole unit of
// the high word and share its sign; renormalised, they are half that with
// either sign, and the sums of them below round four times finer.
struct CornerPacks {
    df2 r15, r37, r26;
    df64 r4;
};
__device__ __forceinline__ CornerPacks corners_of(const double c[8])
{
    auto pair = [](double x, double y) {
        const df2 a = df2_pack(to_df(x), to_df(y));
        const f2 h = f2_add(a.hi, a.lo);
        return df2{h, f2_sub(a.lo, f2_sub(h, a.hi))};
    };
    return {pair(c[1] - c[0], c[5] - c[0]), pair(c[3] - c[0], c[7] - c[0]), pair(c[2] - c[0], c[6] - c[0]),
            df_tidy(to_df(c[4] - c[0]))};
}

// The modes M1..M7 of one field (hexmodes.cuh) in the pairs that the
// butterfly leaves them in: m12 = (M1, M2), m56 = (M5, M6), m73 = (M7, M3)
// and M4.
//
// The order of the sums follows the element's symmetry, here and in the
// kernels that use these packs.  Exchanging the xi and eta axes (and x and
// y) exchanges corners 1 and 3 and corners 5 and 7, modes 1 and 2 and modes 5
// and 6, and every sum goes over into another one, or into itself, with
// operands or terms commuted in a way that changes no bit.  A mirrored
// element's results are its image's, to the last bit, and a flow that starts
// symmetric about the x = y plane stays exactly symmetric: without that, the
// rounding errors of the volumes, 2^-48, are 1e-7 of the volume changes ahead
// of a shock, and the small energies there lose their symmetry at 1e-9.
struct ModePacks {
    df2 m12, m56, m73;
    df64 m4;
};
struct FaceSums {
    df2 u, w;     // c + a, c - a and d + b, d - b: the xi and eta parts of the two zeta faces
    df2 t, s;     // c - g, c + g and k - h, k + h
};
__device__ __forceinline__ df2 plus_minus(df64 a, df64 b) { return df2_add(df2_dup(a), df2_pack(b, -b)); }
__device__ __forceinline__ df2 minus_plus(df64 a, df64 b) { return df2_add(df2_dup(a), df2_pack(-b, b)); }
__device__ __forceinline__ FaceSums face_sums(const CornerPacks &r)
{
    const df2 ag = minus_plus(df2_x(r.r15), df2_x(r.r37));   // a = r1 - r3, g = r1 + r3
    const df2 bh = minus_plus(df2_y(r.r15), df2_y(r.r37));   // b = r5 - r7, h = r5 + r7
    const df2 dk = minus_plus(df2_y(r.r26), r.r4);           // d = r6 - r4, k = r6 + r4
    const df64 c = df2_x(r.r26);
    return {plus_minus(c, df2_x(ag)), plus_minus(df2_x(dk), df2_x(bh)), minus_plus(c, df2_y(ag)),
            minus_plus(df2_y(dk), df2_y(bh))};
}
__device__ __forceinline__ ModePacks walsh_packs(const CornerPacks &r)
{
    const FaceSums f = face_sums(r);
    return {df2_renorm(df2_add(f.u, f.w)), df2_renorm(df2_sub(f.w, f.u)), df2_renorm(df2_sub(f.s, f.t)),
            df_renorm(df_sum(df2_x(f.t), df2_x(f.s)))};
}

// The corner values sum_i s_i(c) F_i of modes F1..F7 in the pairs (F1, F2),
// (F5, F6), F3, F4 and F7, not renormalised: v[0] = corners 2 and 1, v[1] =
// 0 and 3, v[2] = 6 and 5, v[3] = 4 and 7.
__device__ __forceinline__ void inverse_walsh_packs(df2 f12, df2 f56, df64 f3, df64 f4, df64 f7, df2 v[4])
{
    const df2 a[2] = {df2_sub(f12, f56), df2_add(f12, f56)};   // the xi and eta parts at zeta = -1, +1
    const df2 b4 = minus_plus(f4, f7);                         // the xi eta part
#pragma unroll
    for (int z = 0; z < 2; ++z) {
        const df2 p = plus_minus(df2_x(a[z]), df2_y(a[z]));                              // xi = +1, eta = +-1
        const df2 q = plus_minus(z ? f3 : -f3, z ? df2_y(b4) : df2_x(b4));
        v[2 * z] = df2_add(q, p);
        v[2 * z + 1] = df2_sub(q, p);
    }
}

}  // namespace lulesh
