// Float-pair ("df32") arithmetic for FP64 grids on GB300.
//
// GB300's FP64 pipe issues about 2 operations per clock per SM (measured:
// 600 G DFMA/s on 152 SMs), while its FP32 pipes issue 128 FFMA and its
// integer pipes 64 operations per clock per SM.  A 7-point FP64 sweep done
// in native DFMA is therefore capped near 86 GStencil/s, a fifth of what HBM
// could feed.  This header keeps FP64 values as an unevaluated sum of two
// floats, value = h + l, and does all arithmetic on the FP32 pipes:
//
//   * split_f64: double -> (h, l) with integer bit operations and one
//     integer-to-float conversion (the double-to-float conversion runs on
//     the FP64 pipe, so it is avoided).  h holds the top 24 significant bits
//     (truncated), l the remaining 29 rounded to 24, so
//     |x - (h + l)| <= 2^-48 |x| for 2^-74 <= |x| < 2^128.  Below 2^-74 the
//     low part is dropped and below 2^-126 the value flushes to zero
//     (absolute error under 2^-74, about 5e-23); 2^128 and above sets the
//     range flag.
//   * Scaling: a pair may hold x * 2^s instead of x.  The split then
//     rebiases the exponent by 896 - s instead of 896 (1023 - 127) and the
//     join by the same amount back, so the window above applies to x * 2^s:
//     a run can place any 2^202 range of FP64 magnitudes inside it.  A
//     linear sweep commutes with the power-of-two scale exactly (every
//     product and sum of scaled values is the scaled product or sum, as long
//     as nothing leaves the window), so results do not depend on s.
//   * df_fma: acc += c * x with the product's rounding error recovered by an
//     FMA (Dekker/Veltkamp product via fused multiply-add) and the running
//     sum's by Knuth's TwoSum; error terms are gathered in acc.l.
//   * join_f64: (h, l) -> the double nearest h + l: each float is widened
//     exactly by bit construction and the two are added by one DADD, the
//     only FP64 instruction per point (the FP64 pipe is otherwise idle).
// Every operation is written with the _rn intrinsics so the compiler cannot
// contract or reassociate it; the error-free transformations depend on each
// product and sum being rounded exactly once.
#pragma once
#include <cstdint>

namespace uhs {

struct df {
    float h, l;
};

// Exponent rebias between a double x and the float pair of x * 2^shift.
__host__ __device__ constexpr int pair_bias(int shift) { return 896 - shift; }

// x -> the pair of x * 2^shift (bias = pair_bias(shift)).
__device__ __forceinline__ float2 split_f64(double x, unsigned &range_err, int bias = 896) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(x)), lo = static_cast<unsigned>(__double2loint(x));
    const unsigned sign = hi & 0x80000000u;
    // biased float exponent of x * 2^shift (E + 127 + shift, E = eb - 1023)
    const int fe = static_cast<int>((hi >> 20) & 0x7ffu) - bias;
    // h: exponent rebiased and the top 23 fraction bits funnel-shifted in
    // from both words.
    const unsigned f = __funnelshift_l(lo, hi - (static_cast<unsigned>(bias) << 20), 3);
    const unsigned hb = (f & 0x7fffffffu) | sign;
    // l: the remaining 29 fraction bits (weight 2^(fe-127-52)), rounded to 24
    // bits by the integer-to-float conversion and scaled by that weight.
    const float lm = __uint2float_rn(lo & 0x1fffffffu);
    const float sc = __uint_as_float((hb & 0x7f800000u) - (52u << 23));
    float l = __uint_as_float(__float_as_uint(__fmul_rn(lm, sc)) | sign);
    float h = __uint_as_float(hb);
    if (static_cast<unsigned>(fe - 1) >= 254u) {  // scaled exponent outside [-126, 127] (or x zero)
        if (fe > 254) range_err = 1u;
        h = __uint_as_float(sign);
    }
    if (fe < 53) l = 0.0f;  // the low part's weight below the float range: drop it
    return make_float2(h, l);
}

// Exact float -> double of v * 2^-shift by bit construction (normal floats
// and zero; a subnormal float becomes zero).  No FP64 instruction.
__device__ __forceinline__ double f2d_bits(float v, int bias = 896) {
    const unsigned b = __float_as_uint(v);
    const unsigned s = b & 0x80000000u;
    const unsigned hi = s | (((b & 0x7fffffffu) >> 3) + (static_cast<unsigned>(bias) << 20));
    const unsigned lo = b << 29;
    return (b & 0x7f800000u) ? __hiloint2double(static_cast<int>(hi), static_cast<int>(lo))
                             : __hiloint2double(static_cast<int>(s), 0);
}

// The pair of x * 2^shift -> the double nearest x = (h + l) * 2^-shift: both
// halves converted exactly, then one correctly rounded FP64 addition (the
// only FP64 instruction per point).
__device__ __forceinline__ double join_f64(float h, float l, int bias = 896) {
    return __dadd_rn(f2d_bits(h, bias), f2d_bits(l, bias));
}

// acc = c * x  (first term)
__device__ __forceinline__ void df_mul(df &acc, float ch, float cl, float2 x) {
    const float p = __fmul_rn(ch, x.x);
    float e = __fmaf_rn(ch, x.x, -p);
    e = __fmaf_rn(ch, x.y, e);
    e = __fmaf_rn(cl, x.x, e);
    acc.h = p;
    acc.l = e;
}

// acc += c * x
__device__ __forceinline__ void df_fma(df &acc, float ch, float cl, float2 x) {
    const float p = __fmul_rn(ch, x.x);
    float e = __fmaf_rn(ch, x.x, -p);
    e = __fmaf_rn(ch, x.y, e);
    e = __fmaf_rn(cl, x.x, e);
    const float s = __fadd_rn(acc.h, p);
    const float v = __fsub_rn(s, acc.h);
    const float t = __fadd_rn(__fsub_rn(acc.h, __fsub_rn(s, v)), __fsub_rn(p, v));
    acc.h = s;
    acc.l = __fadd_rn(acc.l, __fadd_rn(t, e));
}

// (h, l) -> the same value with |l| <= ulp(h) / 2 (TwoSum).
__device__ __forceinline__ float2 renorm(df a) {
    const float s = __fadd_rn(a.h, a.l);
    const float v = __fsub_rn(s, a.h);
    const float t = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, v)), __fsub_rn(a.l, v));
    return make_float2(s, t);
}

// ---- packed float pairs: two points' sums per instruction ----------------
// sm_100-family GPUs issue FP32 add/mul/fma on register pairs (.f32x2): one
// instruction per two lanes' worth of operations, at the same pipe rate.  A
// sweep bound by instruction issue sums two points (two rows of a thread's
// column) in packed accumulators.  The products stay scalar: a packed
// instruction takes no constant-bank operand, so packed products would move
// every coefficient into a register pair at each use, while the scalar ones
// read it where it lies.  Products and their errors are formed per point
// (8 scalar operations for the two points of a term), the two points' results
// are paired by the register allocator (they come from separate
// instructions), and the error-free sum runs packed (8 operations): 16
// instructions per term for two points instead of 24.  Each operation is the
// scalar one of df_mul / df_fma / renorm in the same order with the same
// rounding, so the results are bit-identical to the scalar sweep's.
// A u64 holds {point 0, point 1}; df2 holds the pairs' hi and lo parts.
typedef unsigned long long u64;

struct df2 {
    u64 h, l;
};

__device__ __forceinline__ u64 pk2(float a, float b) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk2(u64 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
    u64 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// c * x of one point: the product's hi and its error with the cross terms
// (as in df_mul / df_fma).
__device__ __forceinline__ void df_prod(float ch, float cl, float2 x, float &p, float &e) {
    p = __fmul_rn(ch, x.x);
    e = __fmaf_rn(ch, x.x, -p);
    e = __fmaf_rn(ch, x.y, e);
    e = __fmaf_rn(cl, x.x, e);
}

// acc = c * {x0, x1} (df_mul of both points).
__device__ __forceinline__ void df2_mul_s(df2 &acc, float ch, float cl, float2 x0, float2 x1) {
    float p0, p1, e0, e1;
    df_prod(ch, cl, x0, p0, e0);
    df_prod(ch, cl, x1, p1, e1);
    acc.h = pk2(p0, p1);
    acc.l = pk2(e0, e1);
}

// acc += c * {x0, x1} (df_fma of both points; TwoSum and the low-part
// accumulation packed).
__device__ __forceinline__ void df2_fma_s(df2 &acc, float ch, float cl, float2 x0, float2 x1) {
    float p0, p1, e0, e1;
    df_prod(ch, cl, x0, p0, e0);
    df_prod(ch, cl, x1, p1, e1);
    const u64 p = pk2(p0, p1), e = pk2(e0, e1);
    const u64 s = add2(acc.h, p);
    const u64 v = sub2(s, acc.h);
    const u64 t = add2(sub2(acc.h, sub2(s, v)), sub2(p, v));
    acc.h = s;
    acc.l = add2(acc.l, add2(t, e));
}

// renorm of both points: {hi, lo} pairs with |lo| <= ulp(hi) / 2.
__device__ __forceinline__ void renorm2(const df2 &a, u64 &h, u64 &l) {
    const u64 s = add2(a.h, a.l);
    const u64 v = sub2(s, a.h);
    l = add2(sub2(a.h, sub2(s, v)), sub2(a.l, v));
    h = s;
}

}  // namespace uhs

namespace uhs {

// ---- anchored sums: one stencil point's sum on a running anchor -----------
// A point's sum  s = sum_k c_k * x_k  (float pairs c = ch + cl, x = xh + xl)
// in 7 FP32 operations per term, against df_fma's 12.  The running sum T
// starts at an anchor sigma that dominates the sum, so each step's rounding
// error follows from Dekker's Fast2Sum (no TwoSum):
//   B = sum_k |ch_k| |xh_k|;  sigma = 2 B (1 + 2^-15)        (anchor_add)
//   T_0 = sigma;  T_k = fma(ch, xh, T_{k-1})
//   q = T_k - T_{k-1}          exact: T_{k-1}/2 <= T_k <= 2 T_{k-1}
//   r = fma(ch, xh, -q)        the product's part that T_k did not take
//   hi += r;  lo = fma(ch, xl, lo);  lo = fma(cl, xh, lo)
// and the point's value is (T_n - sigma) + (hi + lo).
// Why q is exact: at step k the terms before it took at most B - |p_k| from
// the anchor, so T_{k-1} >= 2 B - (B - |p_k|) >= 2 |p_k| and T_k lies within
// a factor of two of T_{k-1} (Sterbenz' lemma); the 2^-15 covers the
// roundings of B and of the T's for the 3 to 19 terms that sums have here (and
// well beyond).  The same bound puts T_n
// between sigma / 2 and 2 sigma, so T_n - sigma is exact too.  All error is
// in the three low-order accumulations: |r| <= ulp(3 B) / 2, and keeping the
// r's apart from the cross terms (hi, lo) rounds each at its own size.
// tests/c/anchored_sum_check.c holds the exact steps and the largest error of
// random sums to these bounds on the host.  Compared once on random sums of 5-19
// terms (error / B, rms, in units of 2^-49): 3.7-15 against 4.3-24 for an extraction
// on a power-of-two grid (9 operations per term, one low-order accumulator).
// sum |c| enters as 2 (1 + 2^-15) |ch| from the host (fill_coef_anchor), so
// the anchor is one FMA per term and needs no further rounding.
//
// T reaches 3 B, which would overflow for points whose B lies between 2^126.4
// and 2^128.  So the sums run on coefficients times 2^-2 (fill_coef_anchor) and
// their results are multiplied by 4 (dfa_up, dfa_renorm_up): exact, and every
// rounding the same but for low parts below 2^-124, which keep 2^-147.  It costs
// one or two packed operations for two points.
__device__ __forceinline__ float anchor_add(float b, float cabs, float2 x) {  // cabs = 2 (1 + 2^-15) |ch|
    return __fmaf_rn(cabs, fabsf(x.x), b);
}

// Running state of an anchored sum.
struct dfa {
    float t, sg, hi, lo;
};

// first term, on the anchor sigma
__device__ __forceinline__ void dfa_first(dfa &a, float sigma, float ch, float cl, float2 x) {
    a.sg = sigma;
    a.t = __fmaf_rn(ch, x.x, sigma);
    a.hi = __fmaf_rn(ch, x.x, -__fsub_rn(a.t, sigma));
    a.lo = __fmaf_rn(cl, x.x, __fmul_rn(ch, x.y));
}

// += c * x
__device__ __forceinline__ void dfa_add(dfa &a, float ch, float cl, float2 x) {
    const float t = __fmaf_rn(ch, x.x, a.t);
    const float q = __fsub_rn(t, a.t);
    a.t = t;
    a.hi = __fadd_rn(a.hi, __fmaf_rn(ch, x.x, -q));
    a.lo = __fmaf_rn(cl, x.x, __fmaf_rn(ch, x.y, a.lo));
}

// the sum as an (unnormalised) pair: h is a multiple of T's last place
__device__ __forceinline__ df dfa_end(const dfa &a) {
    return df{__fsub_rn(a.t, a.sg), __fadd_rn(a.hi, a.lo)};
}

// (h, l) of dfa_end -> the same value with |l| <= ulp(h) / 2.  h is a multiple
// of T's last place and |l| a few such places, so h is a multiple of ulp(l)
// whichever of the two is larger, and Fast2Sum is exact.
__device__ __forceinline__ float2 dfa_renorm(df a) {
    const float s = __fadd_rn(a.h, a.l);
    return make_float2(s, __fsub_rn(a.l, __fsub_rn(s, a.h)));
}

// the sum of the unscaled coefficients, and its renormalised pair: the four-fold
// high part is fused into the two additions that dfa_renorm has
__device__ __forceinline__ df dfa_up(df a) { return df{__fmul_rn(a.h, 4.0f), __fmul_rn(a.l, 4.0f)}; }
__device__ __forceinline__ float2 dfa_renorm_up(df a) {
    const float l = __fmul_rn(a.l, 4.0f), s = __fmaf_rn(a.h, 4.0f, l);
    return make_float2(s, __fsub_rn(l, __fmaf_rn(a.h, -4.0f, s)));
}

// The same for two points at once: the subtractions and the hi additions
// packed (.f32x2), the fused products per point (they read the coefficient
// from the constant bank, which a packed instruction cannot).  Per point the
// same operations as above, so bit-identical to them.
struct dfa2 {
    u64 t, sg, hi;
    float lo0, lo1;
};

__device__ __forceinline__ u64 anchored_step2(u64 &t, float ch, float2 x0, float2 x1) {
    float t0, t1, q0, q1;
    upk2(t, t0, t1);
    const u64 tn = pk2(__fmaf_rn(ch, x0.x, t0), __fmaf_rn(ch, x1.x, t1));
    upk2(sub2(tn, t), q0, q1);
    t = tn;
    return pk2(__fmaf_rn(ch, x0.x, -q0), __fmaf_rn(ch, x1.x, -q1));
}

__device__ __forceinline__ void dfa2_first(dfa2 &a, u64 sigma, float ch, float cl, float2 x0, float2 x1) {
    a.sg = a.t = sigma;
    a.hi = anchored_step2(a.t, ch, x0, x1);
    a.lo0 = __fmaf_rn(cl, x0.x, __fmul_rn(ch, x0.y));
    a.lo1 = __fmaf_rn(cl, x1.x, __fmul_rn(ch, x1.y));
}

__device__ __forceinline__ void dfa2_add(dfa2 &a, float ch, float cl, float2 x0, float2 x1) {
    a.hi = add2(a.hi, anchored_step2(a.t, ch, x0, x1));
    a.lo0 = __fmaf_rn(cl, x0.x, __fmaf_rn(ch, x0.y, a.lo0));
    a.lo1 = __fmaf_rn(cl, x1.x, __fmaf_rn(ch, x1.y, a.lo1));
}

__device__ __forceinline__ df2 dfa2_end(const dfa2 &a) {
    return df2{sub2(a.t, a.sg), add2(a.hi, pk2(a.lo0, a.lo1))};
}

__device__ __forceinline__ void dfa2_renorm(const df2 &a, u64 &h, u64 &l) {
    h = add2(a.h, a.l);
    l = sub2(a.l, sub2(h, a.h));
}
__device__ __forceinline__ df2 dfa2_up(const df2 &a) {
    const u64 four = pk2(4.0f, 4.0f);
    return df2{mul2(a.h, four), mul2(a.l, four)};
}
__device__ __forceinline__ void dfa2_renorm_up(const df2 &a, u64 &h, u64 &l) {
    const u64 four = pk2(4.0f, 4.0f), l4 = mul2(a.l, four);
    h = fma2(a.h, four, l4);
    l = sub2(l4, fma2(a.h, pk2(-4.0f, -4.0f), h));
}

// acc += g, an (unnormalised) pair: TwoSum of the high parts.  Adds a group of
// terms summed on its own anchor to a longer sum.
__device__ __forceinline__ void df_add(df &acc, df g) {
    const float s = __fadd_rn(acc.h, g.h);
    const float v = __fsub_rn(s, acc.h);
    const float t = __fadd_rn(__fsub_rn(acc.h, __fsub_rn(s, v)), __fsub_rn(g.h, v));
    acc.h = s;
    acc.l = __fadd_rn(acc.l, __fadd_rn(t, g.l));
}
__device__ __forceinline__ void df2_add(df2 &acc, const df2 &g) {
    const u64 s = add2(acc.h, g.h);
    const u64 v = sub2(s, acc.h);
    const u64 t = add2(sub2(acc.h, sub2(s, v)), sub2(g.h, v));
    acc.h = s;
    acc.l = add2(acc.l, add2(t, g.l));
}

}  // namespace uhs
