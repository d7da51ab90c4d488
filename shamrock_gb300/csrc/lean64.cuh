// Correctly rounded FP64 square roots, reciprocals and quotients that use few FP64
// instructions.
//
// GB300 executes two FP64 lanes per clock and SM against 128 FP32 lanes, so the FP64 pair
// loops are bound by the number of FP64 instructions, and each of the compiler's divisions
// and square roots is eight or more of them.  Here the start value comes from the FP32
// pipes: a hardware estimate of the normalised operand refined once in double-float
// arithmetic (about 2^-45), then one FP64 residual correction, then one residual that
// proves the rounding.  The residual x - g^2 (or a - b q) of a value within one unit in the
// last place is exact in an FMA, and g is the correctly rounded root if and only if
//     -g u < x - g^2 <= g u,        u = ulp(g)     (the square (g +- u/2)^2 expanded),
// q the correctly rounded quotient if and only if |a - b q| < b ulp(q) / 2 (a quotient of
// two doubles never lies half-way).  A value that fails the proof (one root in 10^5 and three
// quotients in 10^6 of ordinary size, tests/native/narrow64_check.cpp), and
// operands outside the normal range, report `bad` and the caller evaluates the expression
// with the plain operators, so results are those of the plain operators always.
// For a denominator known per particle the reciprocal is kept as y = RN(1/b) and the
// residual y_lo: q = RN(a y + a y_lo) is a faithful quotient, and then RN(q + (a - b q) y)
// is the correctly rounded one (Markstein, IBM J. Res. Dev. 34, 1990; Muller et al.,
// Handbook of Floating-Point Arithmetic, on division with an FMA), three FP64 instructions
// and no proof needed.
//
// Plain C++ on the host (tests/native/lean64_check.cpp runs it there against the
// operators).  The including unit must not contract or reassociate.
#pragma once

#include "split64.cuh"

#include <cmath>

namespace gbsph {

GBSPH_HD uint64_t bits64(double v) {
    uint64_t b;
    std::memcpy(&b, &v, 8);
    return b;
}
GBSPH_HD double from64(uint64_t b) {
    double v;
    std::memcpy(&v, &b, 8);
    return v;
}
GBSPH_HD uint32_t hi64(double v) { return (uint32_t) (bits64(v) >> 32); }

// +-0, on 32-bit words (as one 64-bit test the compiler makes it an FP64 comparison)
GBSPH_HD bool zero64(uint64_t b) { return ((((uint32_t) (b >> 32)) << 1) | (uint32_t) b) == 0u; }

#ifdef __CUDA_ARCH__
__device__ __forceinline__ double fma64(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma32(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float rsqrt_est(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_est(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
#else
inline double fma64(double a, double b, double c) { return std::fma(a, b, c); }
inline float fma32(float a, float b, float c) { return std::fma(a, b, c); }
// the host check runs with estimates as coarse as the hardware's
inline float rsqrt_est(float x) { return (float) (1.0 / std::sqrt((double) x) * (1.0 + 1.5e-7)); }
inline float rcp_est(float x) { return (float) (1.0 / (double) x * (1.0 - 1.0e-7)); }
#endif

// exact widening of a float whose exponent is in the normal range (a zero gives 2^-127, far
// below the precision the callers keep)
GBSPH_HD double widen_near(float f) {
    uint32_t b;
    std::memcpy(&b, &f, 4);
    return from64(((uint64_t) (b >> 31) << 63) | (((uint64_t) (b & 0x7FFFFFFFu) << 29) + (896ull << 52)));
}

// a positive normal double as m 2^e, m in [1, 2); its float cut m_hi and the rest m_lo
struct Mant {
    double m;
    float hi, lo;
    int e;
};
GBSPH_HD bool normal64(uint32_t h) { return (h & 0x7FFFFFFFu) - 0x00100000u < 0x7FE00000u; }
GBSPH_HD Mant mantissa(double v) { // of |v|
    const uint64_t b  = bits64(v);
    const uint64_t fr = b & 0xFFFFFFFFFFFFFull;
    Mant r;
    r.e  = (int) ((uint32_t) (b >> 52) & 0x7ffu) - 1023;
    r.m  = from64(fr | (1023ull << 52));
    r.hi = split64_bits_to_float(0x3F800000u | (uint32_t) (fr >> 29));
    r.lo = (float) ((uint32_t) fr & 0x1FFFFFFFu) * 2.220446049250313e-16f; // 2^-52
    return r;
}
// v 2^k, v normal; bad when the result is not
GBSPH_HD double scale64(double v, int k, bool &bad) {
    const uint64_t b = bits64(v);
    const int e      = (int) ((uint32_t) (b >> 52) & 0x7ffu) + k;
    bad |= (uint32_t) (e - 1) >= 2046u;
    return from64(b + ((uint64_t) (int64_t) k << 52));
}

// |v| as a float cut towards zero, for comparisons with a margin; NaN from 2^128 on
GBSPH_HD float cut32(double v) {
    const uint64_t b = bits64(v);
    const uint32_t h = (uint32_t) (b >> 32), a = h & 0x7FFFFFFFu;
    uint32_t f = ((a - 0x38000000u) << 3) | ((uint32_t) b >> 29);
    f          = a < 0x38100000u ? 0u : f;
    f          = a >= 0x47F00000u ? 0x7FC00000u : f;
    return split64_bits_to_float(f | (h & 0x80000000u));
}

// sqrt(x) for normal x > 0 (bad otherwise), and what a reciprocal of it needs
struct Root {
    double g;      // RN(sqrt(m)), m = x 4^-k in [1, 4)
    float y, c;    // y + c = 1 / sqrt(m) to about 2^-45
    int k;
};
GBSPH_HD Root root64(double x, bool &bad) {
    const uint64_t b = bits64(x);
    const uint32_t h = (uint32_t) (b >> 32);
    bad |= !(h - 0x00100000u < 0x7FE00000u);
    const uint32_t par = ((h >> 20) & 1u) ^ 1u; // odd exponents: m in [2, 4)
    const uint64_t fr  = b & 0xFFFFFFFFFFFFFull;
    const double m  = from64(fr | ((uint64_t) (1023u + par) << 52));
    const float mh  = split64_bits_to_float((0x3F800000u + (par << 23)) | (uint32_t) (fr >> 29));
    const float ml  = (float) ((uint32_t) fr & 0x1FFFFFFFu)
                     * (par ? 4.440892098500626e-16f : 2.220446049250313e-16f);
    Root r;
    r.k = ((int) (h >> 20) - 1023 - (int) par) / 2;
    // y0 (1 + t/2 + 3 t^2 / 8), t = 1 - m y0^2
    const float y = rsqrt_est(mh);
    const float p = y * y, pe = fma32(y, y, -p);
    float t = fma32(-mh, p, 1.f);
    t       = fma32(-mh, pe, t);
    t       = fma32(-ml, p, t);
    const float c = y * t * fma32(t, 0.375f, 0.5f);
    r.y = y, r.c = c;
    // m (y + c), assembled in FP64
    const float s = mh * y;
    float se = fma32(mh, y, -s);
    se       = fma32(mh, c, se);
    se       = fma32(ml, y, se);
    const double g0 = widen_near(s) + widen_near(se);
    const double d0 = fma64(-g0, g0, m);
    r.g             = fma64(d0, widen_near(0.5f * y), g0);
    // proof: -g u < m - g^2 <= g u, u = 2^-52
    const double d1   = fma64(-r.g, r.g, m);
    const uint64_t ad = bits64(d1) & 0x7FFFFFFFFFFFFFFFull, gu = bits64(r.g) - (52ull << 52);
    bad |= ad > gu || (ad == gu && (hi64(d1) >> 31));
    return r;
}
GBSPH_HD double root_value(const Root &r) {
    return from64(bits64(r.g) + ((uint64_t) (int64_t) r.k << 52));
}
// RN(1 / sqrt value): y1 with |1 - g y1| < g ulp(y1) / 2; y and lo as in Denominator
GBSPH_HD double root_reciprocal(const Root &r, bool &bad, double &y, float &lo) {
    const double y0 = widen_near(r.y) + widen_near(r.c);
    const double e0 = fma64(-r.g, y0, 1.0);
    y               = fma64(e0, y0, y0);
    const double e1 = fma64(-r.g, y, 1.0);
    bad |= (bits64(e1) & 0x7FFFFFFFFFFFFFFFull) >= bits64(r.g) - (54ull << 52);
    lo = cut32(e1) * r.y;
    return from64(bits64(y) - ((uint64_t) (int64_t) r.k << 52));
}
GBSPH_HD double root_reciprocal(const Root &r, bool &bad) {
    double y;
    float lo;
    return root_reciprocal(r, bad, y, lo);
}

// a / b of positive normal doubles
GBSPH_HD double quotient64(double a, double b, bool &bad) {
    bad |= !(hi64(a) - 0x00100000u < 0x7FE00000u) || !(hi64(b) - 0x00100000u < 0x7FE00000u);
    const Mant A = mantissa(a), B = mantissa(b);
    const float y = rcp_est(B.hi);
    float t       = fma32(-B.hi, y, 1.f);
    t             = fma32(-B.lo, y, t);
    const float c = y * fma32(t, t, t);
    const float q = A.hi * y;
    float qe      = fma32(A.hi, y, -q);
    qe            = fma32(A.hi, c, qe);
    qe            = fma32(A.lo, y, qe);
    const double q0 = widen_near(q) + widen_near(qe);
    const double r0 = fma64(-B.m, q0, A.m);
    const double q1 = fma64(r0, widen_near(y), q0);
    const double r1 = fma64(-B.m, q1, A.m);
    // ulp(q1) / 2 is 2^-53 from 1 on, 2^-54 below
    const uint64_t half = bits64(B.m) - ((hi64(q1) >= 0x3FF00000u ? 53ull : 54ull) << 52);
    bad |= (bits64(r1) & 0x7FFFFFFFFFFFFFFFull) >= half;
    return scale64(q1, A.e - B.e, bad);
}

// A denominator kept per particle: y = RN(1/|m|) of its mantissa and the float residual
// 1/|m| - y; lo = NaN where the denominator is zero, subnormal, infinite or NaN.
struct Denominator {
    double b, y;
    float lo;
};
GBSPH_HD Denominator denominator(double b) {
    Denominator d;
    d.b            = b;
    const double m = from64((bits64(b) & 0xFFFFFFFFFFFFFull) | (1023ull << 52));
    d.y            = 1.0 / m;
    d.lo           = (float) (fma64(-m, d.y, 1.0) * d.y);
    if (!normal64(hi64(b))) d.lo = split64_bits_to_float(0x7FC00000u);
    return d;
}
// a / d.b; an exact zero for a == 0
GBSPH_HD double divide_by(double a, const Denominator &d, bool &bad) {
    const uint64_t ab = bits64(a), bb = bits64(d.b);
    const uint64_t fa = ab & 0xFFFFFFFFFFFFFull;
    const double am   = from64(fa | (1023ull << 52));
    const double bm   = from64((bb & 0xFFFFFFFFFFFFFull) | (1023ull << 52));
    const float t     = split64_bits_to_float(0x3F800000u | (uint32_t) (fa >> 29)) * d.lo;
    const double q0   = fma64(am, d.y, widen_near(t));
    const double r0   = fma64(-bm, q0, am);
    const double q1   = fma64(r0, d.y, q0);
    const int k = (int) ((uint32_t) (ab >> 52) & 0x7ffu) - (int) ((uint32_t) (bb >> 52) & 0x7ffu);
    bool odd    = !normal64((uint32_t) (ab >> 32)) || !(d.lo == d.lo);
    const double v = scale64(q1, k, odd);
    const uint64_t sign = (ab ^ bb) & 0x8000000000000000ull;
    const bool zero     = zero64(ab) && d.lo == d.lo;
    bad |= odd && !zero;
    return from64(zero ? sign : (bits64(v) | sign));
}

// The correctly rounded product a b on the integer pipes, about 40 instructions: the 53-bit
// significands are multiplied exactly in 32-bit limbs and rounded to nearest, ties to even.
// Zeros, subnormals, infinities, NaN and results outside the normal range take the FP64
// instruction.  One FP64 instruction occupies the SM for 16 cycles, in which its four
// schedulers issue 64 others, so a loop bound by the FP64 pipe runs faster with part of its
// products here.
static GBSPH_HD_RARE double mul64_plain(double a, double b) { return a * b; }
GBSPH_HD double mul64i(double a, double b) {
    const uint64_t ab = bits64(a), bb = bits64(b);
    const uint32_t ah = (uint32_t) (ab >> 32), bh = (uint32_t) (bb >> 32);
    const uint32_t ea = (ah >> 20) & 0x7ffu, eb = (bh >> 20) & 0x7ffu;
    const uint64_t ma = (ab | (1ull << 52)) << 11, mb = (bb | (1ull << 52)) << 11; // hidden bit at 63
    const uint32_t a1 = (uint32_t) (ma >> 32), a0 = (uint32_t) ma;
    const uint32_t b1 = (uint32_t) (mb >> 32), b0 = (uint32_t) mb;
    const uint64_t p0 = (uint64_t) a0 * b0;
    const uint64_t t  = (uint64_t) a0 * b1 + (p0 >> 32);
    const uint64_t u  = (uint64_t) a1 * b0 + (uint32_t) t;
    uint64_t hi       = (uint64_t) a1 * b1 + (t >> 32) + (u >> 32);
    uint32_t lo       = (uint32_t) u; // then p0's low word, for the sticky bit
    const bool top    = (int64_t) hi < 0;
    if (!top) {
        hi = (hi << 1) | (lo >> 31);
        lo <<= 1;
    }
    const uint32_t e = ea + eb - (top ? 1022u : 1023u);
    if (ea - 1u >= 2046u || eb - 1u >= 2046u || e - 1u >= 2045u) {
        // zeros are common (a state at rest); zero times a finite value is a signed zero
        if ((zero64(ab) || zero64(bb)) && ea != 2047u && eb != 2047u)
            return from64((ab ^ bb) & 0x8000000000000000ull);
        return mul64_plain(a, b);
    }
    const uint32_t rest = ((uint32_t) hi & 0x7ffu) | ((lo | (uint32_t) p0) != 0 ? 1u : 0u);
    uint64_t m          = hi >> 11;
    m += rest + ((uint32_t) m & 1u) > 0x400u ? 1u : 0u;
    // the hidden bit of m adds one to the exponent field
    return from64(m + ((uint64_t) (e - 1u) << 52) + ((uint64_t) ((ah ^ bh) & 0x80000000u) << 32));
}

// The Morton grid cell of a coordinate: min(trunc(RN((clamp(p, lo, hi) - lo) / step)), top),
// inv = 1 / step (0: step is not a normal number in the middle of the range).  The quotient
// comes from one FMA that adds 2^28: it leaves the cell above bit 24 of the significand and
// 24 fraction bits below, in error by less than 0.6 of the last, so a fraction other than
// zero proves the cell (the correctly rounded quotient lies in the same cell); a zero
// fraction, infinities and NaN take the quotient itself.  Two FP64 instructions instead of
// about 25 with the clamps and the division.
// The device's own conversion (saturating, NaN to 2^31) decides what is no cell: a quotient of
// 0 / 0 or inf / inf, in a box without extent along the axis or an unbounded one, takes the
// top cell.  The host check's twin, where such a conversion is undefined, takes cell 0.
static GBSPH_HD_RARE uint32_t grid_cell_plain(double p, double lo, double hi, double step, uint32_t top) {
    const double r = fmin(fmax(p, lo), hi);
    const double q = (r - lo) / step;
#ifdef __CUDA_ARCH__
    return min(__double2uint_rz(q), top);
#else
    if (!(q > 0.)) return 0u;
    return q < (double) top ? (uint32_t) q : top;
#endif
}
GBSPH_HD uint32_t grid_cell(double p, double lo, double hi, double step, double inv, uint32_t top) {
    const double d    = p - lo;
    const uint64_t tb = bits64(fma64(d, inv, 268435456.0));
    const int32_t th  = (int32_t) (uint32_t) (tb >> 32);
    const uint32_t tl = (uint32_t) tb;
    if ((tl & 0xFFFFFFu) == 0u || (hi64(d) & 0x7FF00000u) == 0x7FF00000u)
        return grid_cell_plain(p, lo, hi, step, top);
    if (th < 0x41B00000) return 0u;   // below 2^28: left of the box
    if (th >= 0x41C00000) return top; // at 2^29 and above
    const uint32_t cell = ((uint32_t) (th - 0x41B00000) << 8) | (tl >> 24);
    return cell < top ? cell : top;
}

} // namespace gbsph
