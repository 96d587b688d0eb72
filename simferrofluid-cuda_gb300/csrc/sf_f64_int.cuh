// Double-precision arithmetic on the integer and FP32 pipes, rounded as IEEE 754 rounds it (to nearest, ties to
// even), for kernels that are bound by the FP64 pipe.
//
// This GPU issues one FP64 warp instruction per SM every 16 clocks (2 lanes a clock), against 0.25-0.5 clocks for
// a 32-bit integer or FP32 one, and the two run side by side.  A division, which the compiler builds from about
// ten FP64 instructions, therefore costs far more there than its integer form, and even a multiplication is worth
// moving while the FP64 pipe is the one that is full.
//
// The functions take finite operands whose results stay in the normal range; each says which zeros it accepts.
// Callers test the range of what they feed in (a few integer instructions for a whole stencil) and keep the plain
// FP64 expression for everything else (subnormals, infinities, NaN).  Host and device compile the same code, and
// tests compare it with the host's own arithmetic bit for bit.
//
// Methods: a quotient is found by long division in three digits (two from a 24-bit reciprocal in FP32, one from the
// exact integer remainder), and the exact integer remainder decides the rounding, so the result does not depend on
// the reciprocal's last bits; a square root goes the same way; a third is floor((N + 1) / 3) of the scaled significand
// N, which is its nearest integer because N mod 3 is never a half.
#pragma once
#include <cmath>

#include "sf_convert.cuh"

namespace sf {

#if defined(__CUDA_ARCH__)
SF_CONV_FN float f32_rcp(float x) {  // 1 ulp
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
SF_CONV_FN float f32_rsqrt(float x) {  // within 2^-22
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
SF_CONV_FN float f32_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
SF_CONV_FN float f32_mul(float a, float b) { return __fmul_rn(a, b); }
SF_CONV_FN float f32_add(float a, float b) { return __fadd_rn(a, b); }
SF_CONV_FN int f32_nearest_int(float a) { return __float2int_rn(a); }
SF_CONV_FN double f64_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
SF_CONV_FN uint32_t mulhi_u32(uint32_t a, uint32_t b) { return __umulhi(a, b); }
SF_CONV_FN uint32_t shf_l(uint32_t lo, uint32_t hi, int n) { return __funnelshift_l(lo, hi, n); }
SF_CONV_FN uint32_t shf_r(uint32_t lo, uint32_t hi, int n) { return __funnelshift_r(lo, hi, n); }
SF_CONV_FN int clz_u64(uint64_t v) { return __clzll((long long)v); }
// v >> n of a signed integer, n >= 0 of any size (PTX clamps the amount; in C++ 64 and more are undefined)
SF_CONV_FN int64_t shr_s64(int64_t v, int n) {
    int64_t r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
}
#else
#if defined(SF_F64_TEST_RCP)
// a test's own approximations, off by as much as the device's may be
float SF_F64_TEST_RCP(float y);
SF_CONV_FN float f32_rcp(float x) { return SF_F64_TEST_RCP(1.0f / x); }
SF_CONV_FN float f32_rsqrt(float x) { return SF_F64_TEST_RCP((float)(1.0 / std::sqrt((double)x))); }
#else
SF_CONV_FN float f32_rcp(float x) { return 1.0f / x; }
SF_CONV_FN float f32_rsqrt(float x) { return (float)(1.0 / std::sqrt((double)x)); }
#endif
SF_CONV_FN float f32_fma(float a, float b, float c) { return std::fmaf(a, b, c); }
SF_CONV_FN float f32_mul(float a, float b) { return a * b; }
SF_CONV_FN float f32_add(float a, float b) { return a + b; }
SF_CONV_FN int f32_nearest_int(float a) { return (int)std::nearbyintf(a); }
SF_CONV_FN double f64_fma(double a, double b, double c) { return std::fma(a, b, c); }
SF_CONV_FN uint32_t mulhi_u32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
// the high / low word of (hi:lo) shifted left / right by n in [0, 31]
SF_CONV_FN uint32_t shf_l(uint32_t lo, uint32_t hi, int n) {
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << n) >> 32);
}
SF_CONV_FN uint32_t shf_r(uint32_t lo, uint32_t hi, int n) { return (uint32_t)((((uint64_t)hi << 32) | lo) >> n); }
SF_CONV_FN int clz_u64(uint64_t v) { return v ? __builtin_clzll(v) : 64; }
SF_CONV_FN int64_t shr_s64(int64_t v, int n) { return v >> (n < 63 ? n : 63); }
#endif

constexpr uint32_t kF64Exp = 0x7ff00000u, kF64Frac = 0xfffffu, kF64One = 0x100000u, kF64Sign = 0x80000000u;

// |v| == 0
SF_CONV_FN bool f64_is_zero(double v) {
    uint32_t h, l;
    f64_words(v, h, l);
    return ((h << 1) | l) == 0u;
}

// True when v is zero or 2^lo <= |v| < 2^hi (-1022 <= lo < hi <= 1023): the operands the functions below accept.
SF_CONV_FN bool f64_in_range(double v, int lo, int hi) {
    uint32_t h, l;
    f64_words(v, h, l);
    return (h & kF64Exp) - ((uint32_t)(lo + 1023) << 20) < ((uint32_t)(hi - lo) << 20) || ((h << 1) | l) == 0u;
}

// (M 2^s0 / 3) for a significand M in [2^52, 2^53] with sign and exponent bits `se` above it, packed.
SF_CONV_FN double f64_third_sig(uint32_t m, uint32_t l, uint32_t se) {
    // N = M 2^s in [2^53.58, 2^54.58): N / 3 has 53 bits
    const int s = m >= 0x180000u ? 1 : 2;
    const uint32_t nh = shf_l(l, m, s), nl = l << s;
    // in digits of 30 bits, so that the second digit's dividend (r 2^30 + low digit + 1) fits a word
    const uint32_t d1 = shf_l(nl, nh, 2), d0 = nl & 0x3fffffffu;
    const uint32_t q1 = mulhi_u32(d1, 0x55555556u);  // d1 / 3, exact below 2^31
    const uint32_t z = ((d1 - 3u * q1) << 30) + d0 + 1u;
    const uint32_t q0 = mulhi_u32(z, 0xaaaaaaabu) >> 1;
    const uint64_t q = ((uint64_t)q1 << 30) + q0;
    // x / 3 = q 2^(e - s); q carries the implicit bit
    return f64_from_words((uint32_t)(q >> 32) + se - ((uint32_t)(s + 1) << 20), (uint32_t)q);
}

// x / 3; x zero or normal with a normal result.
SF_CONV_FN double f64_third(double x) {
    uint32_t h, l;
    f64_words(x, h, l);
    const double r = f64_third_sig((h & kF64Frac) | kF64One, l, h & (kF64Sign | kF64Exp));
    return ((h << 1) | l) == 0u ? x : r;
}

// (K x) / 3 with K x rounded first, 2 <= K <= 15; x zero or normal with normal results.
template <int K>
SF_CONV_FN double f64_times_third(double x) {
    uint32_t h, l;
    f64_words(x, h, l);
    const uint32_t m = (h & kF64Frac) | kF64One;
    const uint64_t lo = (uint64_t)l * (uint32_t)K;
    const uint64_t p = lo + ((uint64_t)(m * (uint32_t)K) << 32);
    constexpr int s0 = K >= 8 ? 3 : (K >= 4 ? 2 : 1);
    const int s = s0 + (int)(p >> (53 + s0));
    // round to nearest even at bit s; the sum may reach 2^53, which the third takes
    const uint32_t odd = ((uint32_t)p >> s) & 1u;
    const uint64_t q = p + ((1u << (s - 1)) - 1u + odd);
    const uint32_t ql = shf_r((uint32_t)q, (uint32_t)(q >> 32), s), qh = (uint32_t)(q >> 32) >> s;
    const double r = f64_third_sig(qh, ql, (h & (kF64Sign | kF64Exp)) + ((uint32_t)s << 20));
    return ((h << 1) | l) == 0u ? x : r;
}

// The FP32 digits of a significand (hi word with the implicit bit, low word) in [1, 2): leading 24 bits exactly,
// next 24 bits exactly; the last 5 are left to the remainder.
struct F64Digits {
    float hi, lo;
};
SF_CONV_FN F64Digits f64_digits(uint32_t h, uint32_t l) {
    F64Digits d;
    d.hi = f32_from_bits((shf_l(l, h, 3) & 0x7fffffu) | 0x3f800000u);
    // bits 28..5 of the low word: the leading one of an FP32 at 2^-23 scale, then taken off again (exact)
    d.lo = f32_add(f32_from_bits((((l << 3) >> 9) & 0x7fffffu) | 0x34000000u), -f32_from_bits(0x34000000u));
    return d;
}

// a / b; b normal, a zero or normal, the quotient normal.
SF_CONV_FN double f64_div(double a, double b) {
    uint32_t ah, al, bh, bl;
    f64_words(a, ah, al);
    f64_words(b, bh, bl);
    const uint32_t am = (ah & kF64Frac) | kF64One, bm = (bh & kF64Frac) | kF64One;
    const bool less = am < bm || (am == bm && al < bl);
    const F64Digits x = f64_digits(am, al), y = f64_digits(bm, bl);
    // quotient of the significands to about 2^-44: first digit q0, second digit q1 from the remainder
    float y0 = f32_rcp(y.hi);
    y0 = f32_fma(f32_fma(-y.hi, y0, 1.0f), y0, y0);  // within 2^-24 whatever the approximation's last bits
    const float q0 = f32_mul(x.hi, y0);
    const float r = f32_add(f32_fma(-q0, y.hi, x.hi), f32_fma(-q0, y.lo, x.lo));
    const float q1 = f32_mul(r, y0);  // |q1| < 2^-22: its integer below is less than 2^31
    // Q = quotient * 2^s, s = 53 where a's significand is the smaller and 52 otherwise: 53 bits
    const uint32_t qb = f32_bits(q0);
    const int sh = (int)(qb >> 23) - (127 + 23 - 52) + (less ? 1 : 0);  // 28 .. 30: q0's significand to 2^s
    const uint32_t qm = (qb & 0x7fffffu) | 0x800000u;
    const int c1 = f32_nearest_int(f32_mul(q1, less ? 9007199254740992.0f : 4503599627370496.0f));
    int64_t q = (int64_t)((uint64_t)qm << sh) + c1;
    // exact remainder a 2^s - Q b (its size fits 64 bits, so the low 64 bits of the products suffice); s >= 52, so
    // only a's low bits reach the upper word
    const uint64_t B = ((uint64_t)bm << 32) | bl;
    int64_t rem = (int64_t)(((uint64_t)(al << (less ? 21 : 20)) << 32) - (uint64_t)q * B);
    // third digit: the remainder over b, |digit| < 2^11, by the usual add of 1.5 2^23
    const float rf = f32_fma((float)(int32_t)(rem >> 32), f32_mul(y0, 9.5367431640625e-7f), 12582912.0f);
    const int c2 = (int)(f32_bits(rf) - 0x4b400000u);
    q += c2;
    rem -= (int64_t)((uint64_t)(int64_t)c2 * B);
    // |rem| is now barely above b / 2 at most: the nearest quotient (a tie cannot occur)
    const int64_t twice = rem * 2;
    q += (twice > (int64_t)B ? 1 : 0) - (twice < -(int64_t)B ? 1 : 0);
    const uint32_t ex = (ah & kF64Exp) - (bh & kF64Exp) + ((1023u - 1u) << 20) - (less ? kF64One : 0u);
    const uint32_t sign = (ah ^ bh) & kF64Sign;
    const uint32_t rh = (uint32_t)((uint64_t)q >> 32) + ex;
    return ((ah << 1) | al) == 0u ? f64_from_words(sign, 0u) : f64_from_words(rh | sign, (uint32_t)q);
}

// A product of two significands, each taken times 2^6 (so that the middle sums stay below 2^64): hi:lh:ll is
// A B 2^12, whose upper word pair holds 53 or 54 bits.  Rounded to nearest even and packed with the exponent bits
// `ex` of the 54-bit case less one (the implicit bit adds one) and the sign.
SF_CONV_FN double f64_round_product(uint64_t hi, uint32_t lh, uint32_t ll, uint32_t ex, uint32_t sign) {
    // a 54-bit product drops one bit more (the lowest 12 bits of ll are zero: none is lost below lh)
    const int c = (int)(hi >> 53);
    const uint32_t h1 = (uint32_t)(hi >> 32) >> c, h0 = shf_r((uint32_t)hi, (uint32_t)(hi >> 32), c);
    lh = shf_r(lh, (uint32_t)hi, c);
    // add just under a half, plus one where the kept part is odd or a lower bit is set
    const uint32_t st = ((h0 & 1u) | ll) ? 1u : 0u;
    const uint64_t t = (uint64_t)lh + 0x7fffffffu + st;
    const uint64_t m = (((uint64_t)(h1 + ex + ((uint32_t)c << 20)) << 32) | h0) + (t >> 32);
    return f64_from_words((uint32_t)(m >> 32) | sign, (uint32_t)m);
}

// a * b; each zero (where A0, B0 allow it) or normal, the product zero or normal.
template <bool A0 = true, bool B0 = true>
SF_CONV_FN double f64_mul(double a, double b) {
    uint32_t ah, al, bh, bl;
    f64_words(a, ah, al);
    f64_words(b, bh, bl);
    const uint32_t x1 = shf_l(al, (ah & kF64Frac) | kF64One, 6), x0 = al << 6;
    const uint32_t y1 = shf_l(bl, (bh & kF64Frac) | kF64One, 6), y0 = bl << 6;
    const uint64_t p00 = (uint64_t)x0 * y0;
    const uint64_t mid = (uint64_t)x1 * y0 + ((uint64_t)x0 * y1 + (p00 >> 32));
    const uint64_t hi = (uint64_t)x1 * y1 + (mid >> 32);
    const uint32_t sign = (ah ^ bh) & kF64Sign;
    const double r = f64_round_product(hi, (uint32_t)mid, (uint32_t)p00,
                                       (ah & kF64Exp) + (bh & kF64Exp) - (1024u << 20), sign);
    const bool zero = (A0 && ((ah << 1) | al) == 0u) || (B0 && ((bh << 1) | bl) == 0u);
    return zero ? f64_from_words(sign, 0u) : r;
}

// a * a; a zero or normal with a normal square.
template <bool NONZERO = false>
SF_CONV_FN double f64_sqr(double a) {
    uint32_t ah, al;
    f64_words(a, ah, al);
    const uint32_t x1 = shf_l(al, (ah & kF64Frac) | kF64One, 6), x0 = al << 6;
    const uint64_t p00 = (uint64_t)x0 * x0;
    const uint64_t mid = (uint64_t)x1 * (2u * x0) + (((uint64_t)x1 * (x0 >> 31)) << 32) + (p00 >> 32);
    const uint64_t hi = (uint64_t)x1 * x1 + (mid >> 32);
    const double r = f64_round_product(hi, (uint32_t)mid, (uint32_t)p00, 2u * (ah & kF64Exp) - (1024u << 20), 0u);
    return !NONZERO && ((ah << 1) | al) == 0u ? 0.0 : r;
}

// sqrt(a); a positive and normal.
SF_CONV_FN double f64_sqrt(double a) {
    uint32_t ah, al;
    f64_words(a, ah, al);
    const uint32_t am = (ah & kF64Frac) | kF64One;
    const uint32_t odd = ((ah >> 20) & 1u) ^ 1u;  // exponent 2 k + odd
    // the radicand in [1, 4) as FP32 digits, root to about 2^-45: s0, then s1 from the remainder
    const F64Digits x = f64_digits(am, al);
    const float xh = f32_from_bits(f32_bits(x.hi) + (odd << 23)), xl = odd ? f32_add(x.lo, x.lo) : x.lo;
    float y = f32_rsqrt(xh);
    y = f32_fma(f32_mul(0.5f, y), f32_fma(f32_mul(-xh, y), y, 1.0f), y);
    const float s0 = f32_mul(xh, y);
    const float r = f32_add(f32_fma(-s0, s0, xh), xl);
    const float s1 = f32_mul(r, f32_mul(0.5f, y));
    // S = root * 2^52 in [2^52, 2^53); remainder a 2^(52 + odd) - S^2 in the low 64 bits
    const uint32_t sb = f32_bits(s0);
    uint64_t s = (uint64_t)((sb & 0x7fffffu) | 0x800000u) << ((int)(sb >> 23) - 98);
    s += (int64_t)f32_nearest_int(f32_mul(s1, 4503599627370496.0f));
    int64_t rem = (int64_t)(((uint64_t)(al << (20 + odd)) << 32) - s * s);
    // third digit: remainder / (2 S)
    const float rf = f32_fma((float)(int32_t)(rem >> 32), f32_mul(y, 4.76837158203125e-7f), 12582912.0f);
    const int64_t c = (int64_t)(int)(f32_bits(rf) - 0x4b400000u);
    rem -= (int64_t)((uint64_t)c * (2 * s + (uint64_t)c));
    s += (uint64_t)c;
    // (S + 1/2)^2 = S^2 + S + 1/4: up where the remainder exceeds S, down where it is -S or less
    s += (rem > (int64_t)s ? 1 : 0) - (rem <= -(int64_t)s ? 1 : 0);
    const uint32_t ex = (((ah >> 20) + 1021u - odd) >> 1) << 20;
    return f64_from_words((uint32_t)(s >> 32) + ex, (uint32_t)s);
}

// floor(x) as an integer and as a double, as (int)floor(x) gives it; |x| < 2^31, else (and for NaN) the conversion's own
// result.  The conversions and the rounding all issue on the FP64 pipe.
SF_CONV_FN int f64_floor(double x, double &fl) {
    uint32_t h, l;
    f64_words(x, h, l);
    const int e = (int)((h >> 20) & 0x7ffu) - 1023;
    if (e > 30) {  // infinities and NaN among them
        const int v = (int)std::floor(x);
        fl = (double)v;
        return v;
    }
    if ((int)h >= 0) {
        if (e < 0) {
            fl = 0.0;
            return 0;
        }
        const uint32_t m = (h & kF64Frac) | kF64One;
        if (e <= 20) {
            fl = f64_from_words(h & ~(kF64Frac >> e), 0u);
            return (int)(m >> (20 - e));
        }
        fl = f64_from_words(h, l & ~(0xffffffffu >> (e - 20)));
        return (int)shf_l(l, m, e - 20);
    }
    if (((h << 1) | l) == 0u) {
        fl = 0.0;
        return 0;
    }
    const uint32_t m = (h & kF64Frac) | kF64One;
    uint32_t t = 0, rest = 1;
    if (e >= 0) {
        t = e <= 20 ? m >> (20 - e) : shf_l(l, m, e - 20);
        rest = e < 20 ? (m << (12 + e)) | l : (e == 20 ? l : l << (e - 20));
    }
    const int v = -(int)t - (rest ? 1 : 0);
    // 2^52 + 2^31 + v exactly, less the constant
    fl = f64_from_words(0x43300000u, (uint32_t)v ^ 0x80000000u) - 4503601774854144.0;
    return v;
}

// The distance of v's exponent above 2^lo, for a test against (hi - lo) << 20: below it exactly when 2^lo <= |v| < 2^hi.
// Zeros are outside, so several values are tested by their largest distance.
SF_CONV_FN uint32_t f64_above(double v, int lo) {
    uint32_t h, l;
    f64_words(v, h, l);
    return (h & kF64Exp) - ((uint32_t)(lo + 1023) << 20);
}

// v <= 0, v < 0 and v < 1 on the bits, false for NaN as the comparisons are
SF_CONV_FN bool f64_le0(double v) {
    uint32_t h, l;
    f64_words(v, h, l);
    const uint64_t b = ((uint64_t)h << 32) | l;
    return b == 0 || (b >= 0x8000000000000000ull && b <= 0xfff0000000000000ull);
}
SF_CONV_FN bool f64_lt0(double v) {
    uint32_t h, l;
    f64_words(v, h, l);
    const uint64_t b = ((uint64_t)h << 32) | l;
    return b > 0x8000000000000000ull && b <= 0xfff0000000000000ull;
}
SF_CONV_FN bool f64_lt1(double v) {
    uint32_t h, l;
    f64_words(v, h, l);
    return (int)h < 0 ? (h < 0xfff00000u || (h == 0xfff00000u && l == 0u)) : h < 0x3ff00000u;
}
SF_CONV_FN bool f64_is_one(double v) {
    uint32_t h, l;
    f64_words(v, h, l);
    return h == 0x3ff00000u && l == 0u;
}

// x / 2, or -x / 2 (NEG); x zero or normal with a normal half.
template <bool NEG = false>
SF_CONV_FN double f64_half(double x) {
    uint32_t h, l;
    f64_words(x, h, l);
    const uint32_t r = ((h << 1) | l) == 0u ? h : h - kF64One;
    return f64_from_words(NEG ? r ^ kF64Sign : r, l);
}

// a / b, sqrt(a) and a / 3 for any operands: the integer form where the operands allow it, else the plain one.
SF_CONV_FN double f64_div_any(double a, double b) {
    return f64_in_range(a, -400, 400) && f64_in_range(b, -400, 400) && !f64_is_zero(b) ? f64_div(a, b) : a / b;
}
SF_CONV_FN double f64_sqrt_any(double a) {
    return !f64_lt0(a) && f64_in_range(a, -1000, 1000) && !f64_is_zero(a) ? f64_sqrt(a) : std::sqrt(a);
}
SF_CONV_FN double f64_third_any(double a) { return f64_in_range(a, -1000, 1000) ? f64_third(a) : a / 3; }

// A double as its significand times 2^6, with the sign, and its exponent field: v = m 2^(e - 1081), |m| < 2^59 (a zero or a
// subnormal number, of field 0, comes out as one near 2^-1023).
struct F64Fixed {
    int64_t m;
    int e;
};
SF_CONV_FN F64Fixed f64_fixed(double v) {
    uint32_t h, l;
    f64_words(v, h, l);
    const int64_t t = (int64_t)(((uint64_t)shf_l(l, (h & kF64Frac) | kF64One, 6) << 32) | (l << 6));
    return F64Fixed{(int)h < 0 ? -t : t, (int)((h >> 20) & 0x7ffu)};
}
// In units of 2^(e - 1081), towards minus infinity; e at least the value's own field.
SF_CONV_FN int64_t fixed_at(const F64Fixed &v, int e) { return shr_s64(v.m, e - v.e); }

// t 2^(e - 1081), rounded to nearest even, |t| < 2^63 (the conversion instruction takes the FP64 pipe twice).
SF_CONV_FN double fixed_to_f64(int64_t t, int e) {
    const uint64_t m = t < 0 ? 0ull - (uint64_t)t : (uint64_t)t;
    const int z = clz_u64(m);          // >= 1
    const uint64_t a = m << (z & 63);  // 64-bit significand, the top bit set
    // the 53 kept bits and the exponent field of 2^(e - 1081) 2^(63 - z), less the implicit bit, rounded by adding just
    // under a half of the eleven dropped bits and the kept part's parity
    const uint64_t kept = (a >> 11) + ((uint64_t)(uint32_t)(e + 4 - z) << 52);
    const uint64_t up = ((a & 0x7ffull) + 0x3ffull + ((a >> 11) & 1ull)) >> 11;
    const uint64_t bits = (kept + up) | ((uint64_t)t & 0x8000000000000000ull);
    return m == 0 ? 0. : f64_from_words((uint32_t)(bits >> 32), (uint32_t)bits);
}

// s = n x - (a + b + c + d + e + f), n <= 6, in 64-bit integers of one unit, 2^-58 of the largest magnitude M of the seven:
// what is lost is less than a unit a value, 6 2^-58 M in all, and the last rounding, against a rounding of up to
// 2^-53 of the partial sum at each of seven FP64 operations.  The unit is this sum's own, so that holds wherever
// the seven stand in a field of any range.  False (s unset) where M is below 2^-823, infinite or NaN.
SF_CONV_FN bool fixed_stencil(int n, const F64Fixed &x, const F64Fixed &a, const F64Fixed &b, const F64Fixed &c,
                              const F64Fixed &d, const F64Fixed &e, const F64Fixed &f, double &s) {
    int top = x.e > a.e ? x.e : a.e;
    top = top > b.e ? top : b.e;
    top = top > c.e ? top : c.e;
    top = top > d.e ? top : d.e;
    top = top > e.e ? top : e.e;
    top = top > f.e ? top : f.e;
    if (top < 200 || top > 2040) return false;
    s = fixed_to_f64(fixed_at(x, top) * n - (fixed_at(a, top) + fixed_at(b, top) + fixed_at(c, top) + fixed_at(d, top) +
                                             fixed_at(e, top) + fixed_at(f, top)),
                     top);
    return true;
}

}  // namespace sf
