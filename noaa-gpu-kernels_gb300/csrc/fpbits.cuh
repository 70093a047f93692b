// IEEE double comparisons, minimum and maximum evaluated on the integer
// pipes from the bit patterns. On GB300 every FP64 instruction -- compares
// and min/max included -- occupies an SMSP's FP64 pipe for 64 cycles per
// warp, while the integer pipes are idle; the secant pass makes ~30 such
// decisions. Each helper returns exactly what the IEEE comparison returns for
// every input, NaN and signed zeros included (IEEE ordering of doubles is the
// ordering of their sign-magnitude bit patterns, with NaN unordered and
// +0 == -0).
#pragma once

#include <cuda_runtime.h>

namespace tr {

constexpr long long kInfBits = 0x7ff0000000000000ll;

__device__ __forceinline__ long long dbits(double x) { return __double_as_longlong(x); }

// x > 0
__device__ __forceinline__ bool fp_gt0(double x)
{
    const long long b = dbits(x);
    return b > 0 && b <= kInfBits;
}

// x < 0
__device__ __forceinline__ bool fp_lt0(double x)
{
    const unsigned long long b = (unsigned long long)dbits(x);
    return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull;
}

// x <= 0
__device__ __forceinline__ bool fp_le0(double x)
{
    const long long b = dbits(x);
    return b <= 0 && (unsigned long long)b <= 0xfff0000000000000ull;
}

// x == 0 (either sign)
__device__ __forceinline__ bool fp_eq0(double x) { return ((unsigned long long)dbits(x) << 1) == 0; }

// x > c for a constant or value c > 0 that is not NaN
__device__ __forceinline__ bool fp_gt_pos(double x, double c)
{
    const long long b = dbits(x);
    return b > dbits(c) && b <= kInfBits;
}

// x >= c for c >= +0 (not NaN, not -0); x >= +0 is true for x = -0 as well
__device__ __forceinline__ bool fp_ge_nonneg(double x, double c)
{
    const long long b = dbits(x);
    if (((unsigned long long)b << 1) == 0) return dbits(c) == 0;  // x = +-0: only c = 0 qualifies
    return b >= dbits(c) && b <= kInfBits;
}

// x < c for a constant or value c > 0 that is not NaN
__device__ __forceinline__ bool fp_lt_pos(double x, double c)
{
    const long long b = dbits(x);
    // sign set: -0 and negative numbers are below c, a negative NaN is not
    return b < 0 ? (unsigned long long)b <= 0xfff0000000000000ull : b < dbits(c);
}

// |a| > b for any a, b (false when either is NaN)
__device__ __forceinline__ bool fp_abs_gt(double a, double b)
{
    const long long ma = dbits(a) & 0x7fffffffffffffffll;
    const long long bb = dbits(b);
    const long long mb = bb & 0x7fffffffffffffffll;
    if (ma > kInfBits || mb > kInfBits) return false;
    if (bb < 0) return ma != 0 || mb != 0;  // b <= -0: |a| > b unless both are zeros
    return ma > mb;
}

// fmax(x, 0.0) and fmax(0.0, x): the positive value, otherwise +0 (NaN -> +0,
// as IEEE maxNum returns the non-NaN operand)
__device__ __forceinline__ double fp_max0(double x) { return fp_gt0(x) ? x : 0.0; }

// fmax(c, x) for c > 0 not NaN and any x (x <= c or NaN gives c)
__device__ __forceinline__ double fp_max_pos(double c, double x) { return fp_gt_pos(x, c) ? x : c; }

__device__ __forceinline__ int dexp(double x) { return (int)(((unsigned long long)dbits(x) >> 52) & 0x7ff); }

// Quotients with three FP64 instructions each on a shared reciprocal of two.
//
// near_rcp: y = 1/b within (1/2 + 2^-28) ulp. The single-precision reciprocal of
// the leading 24 bits of b's significand, corrected by its residual against the
// whole significand (first-order, in single precision: |1 - m s| < 2^-22, so that
// the second-order term, the rounding of the correction to 2^-43 and those of the
// residual leave a relative error below 2^-42), is scaled on the integer pipe to
// y0; with e = RN(1 - b y0) the step y = RN(y0 + y0 e) leaves e^2 < 2^-84 before its
// own rounding (the Newton-Raphson family, e.g. Muller et al., Handbook of
// Floating-Point Arithmetic, chapter on division with an FMA). From the plain
// single-precision seed the step has to be cubic, one FP64 instruction of 64 cycles
// more; the correction is a chain of seven instructions of 4 to 5.
//
// near_quot: q0 = RN(a y), r = RN(a - b q0), q = RN(q0 + r y). y's error and
// q0's rounding put q0 at most 1.5 ulp (+2^-11) from a/b (1 ulp when a's
// significand is at least b's), r carries a relative error of at most 2^-53,
// so q0 + r y before the last rounding is a/b to within 2^-50 ulp and q is the
// IEEE quotient unless a/b lies that close to a rounding midpoint. Seen from
// q0 the midpoints lie at +-1/2 and +-3/2 ulp, i.e. at |r| = T and 3 T with
// T = |b| ulp(q0) / 2, whose bit pattern is b's with q0's exponent added. The
// high words of |r| and T (20 significand bits) tell when r is within 2^-19 of
// T; the difference of two high words is a piecewise linear logarithm, and
// |r| >= 3 T always shows as a difference of at least 1.5 * 2^20 (1.49 is
// tested; below 3 T it is met only by b's with a significand above 1.96 and a
// next to them). When q0's significand starts with 20 zeros the quotient may
// lie in the binade below, with midpoints elsewhere. In these cases -- a few
// per million quotients -- the caller must divide instead: `doubt` is set
// and never cleared. Zero residuals never doubt: q0 is then the quotient.
// Operands: b normal, |b| < 2^1022; a = +0 or |a| >= 2^-900; q0 normal (nothing
// underflows in y or r). The IEEE division takes about 10 FP64
// instructions; the correctly rounded reciprocal and two Markstein
// corrections used before took 8 per divisor and 5 per quotient.
constexpr int kHalfUlp = 1076 << 20;   // exponent bias plus 53
constexpr int kThreeHalves = (int)(1.49 * 1048576);

struct NearRcp {
    double b, y;
};

// y0: single-precision 1/b as a double
__device__ __forceinline__ double rcp_seed(double b)
{
    const int hi = __double2hiint(b), lo = __double2loint(b);
    const float m = __int_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffff) | 0x3f800000);
    float s;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(m));
    const int sb = __float_as_int(s);
    // exponent field 1023 + (field(s) - 127) - (field(b) - 1023), b's sign
    const int yh = ((sb >> 3) + (1919 << 20) - (hi & 0x7ff00000)) | (hi & 0x80000000);
    return __hiloint2double(yh, sb << 29);
}

// 1/b with a relative error below 2^-42
__device__ __forceinline__ double rcp_seed_fine(double b)
{
    const int hi = __double2hiint(b), lo = __double2loint(b);
    const float m = __int_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffff) | 0x3f800000);
    const float ml = __fadd_rn(__int_as_float(((lo & 0x1fffffff) >> 6) | 0x3f800000), -1.0f);   // the rest times 2^23
    float s;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(m));
    s = fmaxf(s, 0.5f);
    const float d = __fmaf_rn(ml, __fmul_rn(s, -0x1p-23f), __fmaf_rn(-m, s, 1.0f));
    // s d in units of 2^-43, which are 2^10 units in the last place of a double in
    // [1/2, 1) (s = 1 only for m = 1, where d <= 0 and the sum lies there too)
    const int c = __float_as_int(__fmaf_rn(__fmul_rn(s, 0x1p43f), d, 12582912.0f)) - 0x4b400000;
    const int sb = __float_as_int(s);
    const int yh = ((sb >> 3) + (1919 << 20) - (hi & 0x7ff00000)) | (hi & 0x80000000);
    return __longlong_as_double((((long long)yh << 32) | (unsigned)(sb << 29)) + (long long)c * 1024);
}

__device__ __forceinline__ NearRcp near_rcp(double b)
{
    const double y0 = rcp_seed_fine(b);
    return {b, __fma_rn(y0, __fma_rn(-b, y0, 1.0), y0)};
}

// Whether the quotient near q0 with residual r may round differently (see above).
__device__ __forceinline__ bool quot_doubt(double b, double q0, double r)
{
    const int hq = __double2hiint(q0), hr = __double2hiint(r) & 0x7fffffff;
    const int t = max((__double2hiint(b) & 0x7fffffff) - kHalfUlp + (hq & 0x7ff00000), 4);
    const int d = hr - t;
    return ((unsigned)(d + 1) <= 2u) | (d >= kThreeHalves) | (((hq & 0xfffff) == 0) & (hr != 0));
}

__device__ __forceinline__ double near_quot(double a, const NearRcp& d, bool& doubt)
{
    const double q0 = a * d.y;
    const double r = __fma_rn(-d.b, q0, a);
    doubt |= quot_doubt(d.b, q0, r);
    return __fma_rn(r, d.y, q0);
}

// 1 / b: the reciprocal itself takes q0's place.
__device__ __forceinline__ double near_one_over(double b, bool& doubt)
{
    const double q0 = near_rcp(b).y;
    const double r = __fma_rn(-b, q0, 1.0);
    doubt |= quot_doubt(b, q0, r);
    return __fma_rn(r, q0, q0);
}

// |x| in [2^-n, 2^n) by the exponent field
__device__ __forceinline__ bool fp_within(double x, int n)
{
    return (unsigned)((__double2hiint(x) & 0x7fffffff) - ((1023 - n) << 20)) < ((unsigned)n << 21);
}

// The IEEE quotient a / b for any operands, by near_quot where it applies.
__device__ __forceinline__ double quot_ieee(double a, double b)
{
    if (fp_within(b, 400) && fp_within(a, 400)) {
        bool doubt = false;
        const double q = near_quot(a, near_rcp(b), doubt);
        if (!doubt) return q;
    }
    return a / b;
}

// RN(a / b) > c -- the IEEE quotient compared with c -- for any a, b > 0 and
// c > 0 (neither NaN), mostly without the division. RN(a/b) > c exactly when
// a/b lies above the midpoint m = c + u between c and the next double
// (u = ulp(c)/2, a power of two), up to the tie a/b = m. With x = a - c b and
// y = u b (exact for b and c normal, y normal): a/b > m <=> x > y. The FMA
// gives e = RN(x) with one rounding, and rounding is monotone with y
// representable, so e > y implies x > y and e < y implies x < y. Only e == y
// (a tie, or x within half an ulp of y), NaN and operands outside the normal
// range take the division.
__device__ __forceinline__ bool quot_gt_pos(double a, double b, double c)
{
    const int eb = dexp(b), ec = dexp(c);
    const int k = ec - 1023 - 53;  // u = 2^k
    if ((unsigned)(eb - 1) < 0x7feu && (unsigned)(ec - 1) < 0x7feu && (unsigned)(eb + k - 1) < 0x7feu) {
        const double y = __longlong_as_double(dbits(b) + ((long long)k << 52));
        const double e = __fma_rn(-c, b, a);
        if (fp_gt_pos(e, y)) return true;
        if (fp_lt_pos(e, y)) return false;
    }
    return fp_gt_pos(a / b, c);
}

// |x| on the integer pipe
__device__ __forceinline__ double fp_abs(double x) { return __longlong_as_double(dbits(x) & 0x7fffffffffffffffll); }

}  // namespace tr
