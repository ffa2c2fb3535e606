// knc_fp64.cuh — FP64 division, square root and comparisons with few FP64
// instructions.
//
// GB300's FP64 pipe takes 64 to 76 cycles per warp instruction and SM
// partition whatever the operation (add, multiply, fused multiply-add,
// comparison, minimum, conversion) and however many lanes are active
// (measured); the FP32 pipe takes 1 and the integer pipe 2. Of those 76-cycle
// slots `a / b` takes 7.2, sqrt 7.5, 1 / b 4.5 and a comparison 1. Here these
// operations leave the FP64 pipe:
//   - a start: the FP32 hardware estimate of 1 / b (or 1 / sqrt(x)) and one
//     Newton step, kept as a 53-bit integer;
//   - the quotient (root) as an integer Q, from the upper words of the
//     mantissa times the start, a few units off at most;
//   - the exact remainder a 2^t - Q b (x - Q^2) from the low words of the
//     products, whose leading words cancel: over b (2 Q) it is the correction
//     of Q and decides the rounding. Where its FP32 value lies next to a
//     midpoint the remainder is compared in 64 bits.
// That is the long-division argument (quotient estimate, exact remainder,
// correction: Knuth, The Art of Computer Programming vol. 2, section 4.3.1;
// Cornea, Harrison and Tang, Scientific Computing on Itanium, 2002), so every
// result is the correctly rounded one, the bits of the plain operators.
// Cycles per warp operation and partition, with 4 warps on it: division 117
// (70 with a shared start) against 548, reciprocal 75 against 344, square root
// 104 against 572.
// The fast forms hold for operands inside an exponent range; callers collect
// range checks (fp64_odd_*) and send a zone or face that fails one through the
// plain operators.
#pragma once

#include <stdint.h>

namespace knc {

// The words of a double. Through asm: integer tests on the bits of a double
// that the compiler can see (x & 0x7ff..f == 0) come out as FP64 comparisons,
// about 45 of 315 FP64 instructions of an update row.
__device__ __forceinline__ uint32_t hi_word(double x) {
    uint32_t hi;
    asm("{.reg .b32 t; mov.b64 {t, %0}, %1;}" : "=r"(hi) : "d"(x));
    return hi;
}
__device__ __forceinline__ uint32_t lo_word(double x) {
    uint32_t lo;
    asm("{.reg .b32 t; mov.b64 {%0, t}, %1;}" : "=r"(lo) : "d"(x));
    return lo;
}
__device__ __forceinline__ double words(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }

// Operands of the fast forms. A divisor (and the operand of a reciprocal or
// square root) lies in 2^[-400, 400]; a numerator in 2^[-600, 600] or is zero:
// the result's exponent stays in the normal range.
__device__ __forceinline__ bool fp64_odd_divisor(double b) {
    return (hi_word(b) & 0x7fffffffu) - (623u << 20) > (800u << 20);
}
__device__ __forceinline__ bool fp64_odd_positive(double b) { return hi_word(b) - (623u << 20) > (800u << 20); }
__device__ __forceinline__ bool fp64_odd_numerator(double a) {
    const uint32_t h = hi_word(a) & 0x7fffffffu;
    return h - (423u << 20) > (1200u << 20) && (h | lo_word(a)) != 0u;
}

// The start of a division or square root: Y 2^-53, Y a 53-bit integer (hi:lo)
// in [2^52, 2^53], approximates 1 / m; r is an FP32 1 / m.
struct Start64 {
    uint32_t lo, hi;
    float r;
};

// R 2^29 + c in units of 2^-53: the FP32 estimate R 2^-24 and its correction
__device__ __forceinline__ Start64 start_sum(uint32_t R, int32_t c, float r) {
    Start64 s;
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, %5;"
        : "=r"(s.lo), "=r"(s.hi)
        : "r"(R << 29), "r"((uint32_t)c), "r"(R >> 3), "r"((uint32_t)(c >> 31)));
    s.r = r;
    return s;
}

// 1 / m to 3 units of 2^-53 for the mantissa m in [1, 2) of b. Mh:Ml the
// mantissa as a fraction of 2^63; R 2^-24 the FP32 estimate of 1 / m, in
// [0.5, 1); the residual e = 1 - m R 2^-24 (below 1.5 2^-23) in units of 2^-53
// from the exact product's low words (its leading bits cancel); then
// 1 / m = R 2^-24 (1 + e + e^2). The estimate of a 24-bit number between 2^31
// and 2^32 is never below 2^-32, as R's bits assume (its 2^23 operands, and
// the 2^24 of the root's, are swept by tests/test_fp64_starts.py); a lower
// clamp beside the upper one cost 0.3% of the FP64 step.
__device__ __forceinline__ Start64 rcp_start(double b) {
    const uint32_t hi = hi_word(b), lo = lo_word(b);
    const uint32_t Mh = __funnelshift_l(lo, hi, 11) | 0x80000000u, Ml = lo << 11;
    float r0;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"((float)Mh));
    r0 = fminf(r0, 4.656612595521637e-10f);   // below 2^-31: R below 2^24
    const uint32_t R = (__float_as_uint(r0) & 0x7fffffu) | 0x800000u;
    const unsigned long long P = (unsigned long long)Mh * R + (__umulhi(Ml, R) + 2u);
    const int32_t e = -(int32_t)__funnelshift_r((uint32_t)P, (uint32_t)(P >> 32), 2);
    const float ef = (float)e;
    const int32_t ee = e + __float2int_rn(ef * (ef * 1.1102230246251565e-16f));   // e + e^2
    const long long c = (long long)ee * (int32_t)(R << 7) + (1ll << 30);
    return start_sum(R, (int32_t)__funnelshift_r((uint32_t)c, (uint32_t)(c >> 32), 31), r0 * 2147483648.0f);
}

// 1 / sqrt(m) to about 2^-44 for m in [1, 4), x = m 4^k > 0: also the start of
// divisions by sqrt(x), whose mantissa is sqrt(m).
__device__ __forceinline__ Start64 rsqrt_start(double x) {
    const uint32_t hi = hi_word(x), lo = lo_word(x);
    const uint32_t odd = (~hi >> 20) & 1u;   // bias 1023 is odd: an even biased exponent is an odd power of two
    const float f0 = __uint_as_float(((__funnelshift_l(lo, hi, 3) & 0x7fffffu) | 0x3f800000u) + (odd << 23));
    const float f1 = (float)(lo & 0x1fffffffu) * __uint_as_float((75u + odd) << 23);   // 2^(-52 + odd)
    float r0;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(f0));
    r0 = fminf(r0, 0.99999994f);
    const float g = f0 * r0;
    float e = __fmaf_rn(-g, r0, 1.0f);
    e = __fmaf_rn(-__fmaf_rn(f0, r0, -g), r0, e);
    e = __fmaf_rn(-f1 * r0, r0, e);
    const float t = __fmaf_rn(0.375f * e, e, 0.5f * e);
    const uint32_t R = (__float_as_uint(r0) & 0x7fffffu) | 0x800000u;
    return start_sum(R, __float2int_rn(r0 * (t * 9007199254740992.0f)), r0);
}

// k = R / D rounded to the nearest integer, f its FP32 value: the quotient
// Q + k is the correctly rounded one unless f lies next to a midpoint, which
// `near` says. |k| is a few units after rcp_start and up to 2^9 after
// rsqrt_start (2^-44 of 2^53), and stays below 2^10 (a remainder's upper word
// is an int32); f is good to 2^-22 |k| + 2^-20 < 2^-11, the guard below.
__device__ __forceinline__ int nearest(float f, bool& near) {
    const float kf = rintf(f);
    near = fabsf(f - kf) > 0.4995f;
    return (int)kf;
}

// a / b, s = rcp_start(b) (or rsqrt_start(x) with b = sqrt(x)). The quotient's
// integer Q = Ma 2^t / Mb in [2^52, 2^53) from the upper words of Ma Y; its
// exact remainder Ma 2^t - Q Mb from the low words (the leading ones cancel);
// Q moves by the remainder over Mb rounded to the nearest integer.
__device__ __forceinline__ double fp64_div(double a, double b, const Start64& s) {
    const uint32_t ahi = hi_word(a), alo = lo_word(a), bhi = hi_word(b), bl = lo_word(b);
    const uint32_t bh = (bhi & 0xfffffu) | 0x100000u, am = (ahi & 0xfffffu) | 0x100000u;
    const bool less = am < bh || (am == bh && alo < bl);   // Ma < Mb: t = 53, else 52
    const uint32_t Ah = __funnelshift_l(alo, am, 11), Al = alo << 11;
    const uint32_t Yh = __funnelshift_l(s.lo, s.hi, 10), Yl = s.lo << 10;
    const unsigned long long p =
        (unsigned long long)Ah * Yh + __umulhi(Ah, Yl) + (unsigned long long)__umulhi(Al, Yh);   // Ma / Mb 2^62
    const unsigned long long Q = p >> (less ? 9 : 10);
    const uint32_t Qh = (uint32_t)(Q >> 32), Ql = (uint32_t)Q;
    const unsigned long long prod = (unsigned long long)Ql * bl;
    const uint32_t ph = (uint32_t)(prod >> 32) + Ql * bh + Qh * bl;
    const uint32_t th = alo << (less ? 21 : 20);
    // upper word of the remainder: its sign and 2^-20 Mb are enough
    const int32_t Rh = (int32_t)(th - ph - ((uint32_t)prod != 0u ? 1u : 0u));
    const float f = (float)Rh * (s.r * 9.5367431640625e-07f);   // 2^32 / (2^52 m)
    bool near;
    int k = nearest(f, near);
    if (near) {
        // R - k Mb against Mb / 2 in 64 bits
        const unsigned long long Mb = ((unsigned long long)bh << 32) | bl;
        const long long R = (long long)(((unsigned long long)th << 32) - Q * Mb) - (long long)k * (long long)Mb;
        if (2 * R > (long long)Mb) ++k;
        if (2 * R < -(long long)Mb) --k;
    }
    const uint32_t e = (ahi & 0x7ff00000u) - (bhi & 0x7ff00000u) + ((less ? 1021u : 1022u) << 20);
    const unsigned long long z = Q + (long long)k;
    const uint32_t sign = (ahi ^ bhi) & 0x80000000u;
    if (((ahi << 1) | alo) == 0u) return words(sign, 0u);
    return words(((uint32_t)(z >> 32) + e) | sign, (uint32_t)z);
}

// 1 / b from s = rcp_start(b)
__device__ __forceinline__ double fp64_rcp(double b, const Start64& s) {
    const uint32_t bhi = hi_word(b), bl = lo_word(b);
    const uint32_t bh = (bhi & 0xfffffu) | 0x100000u;
    const unsigned long long prod = (unsigned long long)s.lo * bl;
    const uint32_t ph = (uint32_t)(prod >> 32) + s.lo * bh + s.hi * bl;   // 2^105 - Y Mb
    const int32_t Rh = (int32_t)(0u - ph - ((uint32_t)prod != 0u ? 1u : 0u));
    const float f = (float)Rh * (s.r * 9.5367431640625e-07f);
    bool near;
    int k = nearest(f, near);
    const unsigned long long Q = ((unsigned long long)s.hi << 32) | s.lo;
    if (near) {
        const unsigned long long Mb = ((unsigned long long)bh << 32) | bl;
        const long long R = (long long)(0ull - Q * Mb) - (long long)k * (long long)Mb;
        if (2 * R > (long long)Mb) ++k;
        if (2 * R < -(long long)Mb) --k;
    }
    const unsigned long long z = Q + (long long)k;
    // biased exponent 2045 - E, the hidden bit of z adds one
    return words((uint32_t)(z >> 32) + ((2044u << 20) - (bhi & 0xfff00000u)), (uint32_t)z);
}

// x / 2 on the integer pipe, x a normal number well above the smallest
__device__ __forceinline__ double fp64_half(double x) { return words(hi_word(x) - (1u << 20), lo_word(x)); }

// sqrt(x), s = rsqrt_start(x): Q = sqrt(m) 2^52 from the upper words of m Y,
// remainder m 2^104 - Q^2 from the low words.
__device__ __forceinline__ double fp64_sqrt(double x, const Start64& s) {
    const uint32_t hi = hi_word(x), lo = lo_word(x);
    const uint32_t sh = 11u - ((hi >> 20) & 1u);   // m 2^62: mantissa << 10, or << 11 for an odd power of two
    const uint32_t m = (hi & 0xfffffu) | 0x100000u;
    const uint32_t Xh = __funnelshift_l(lo, m, sh), Xl = lo << sh;
    const uint32_t Yh = __funnelshift_l(s.lo, s.hi, 10), Yl = s.lo << 10;
    const unsigned long long p =
        (unsigned long long)Xh * Yh + __umulhi(Xh, Yl) + (unsigned long long)__umulhi(Xl, Yh);   // sqrt(m) 2^61
    const unsigned long long Q = p >> 9;
    const uint32_t Qh = (uint32_t)(Q >> 32), Ql = (uint32_t)Q;
    const unsigned long long sq = (unsigned long long)Ql * Ql;
    const uint32_t ph = (uint32_t)(sq >> 32) + 2u * Ql * Qh;
    const uint32_t th = Xl << 10;
    const int32_t Rh = (int32_t)(th - ph - ((uint32_t)sq != 0u ? 1u : 0u));
    const float f = (float)Rh * (s.r * 4.76837158203125e-07f);   // 2^32 / (2 2^52 sqrt(m))
    bool near;
    int k = nearest(f, near);
    if (near) {
        const long long R =
            (long long)(((unsigned long long)th << 32) - Q * Q) - (long long)k * (long long)(2 * Q + (long long)k);
        const long long q = (long long)Q + k;
        if (R > q) ++k;
        if (R <= -q) --k;
    }
    const unsigned long long z = Q + (long long)k;
    // biased exponent (E + 1023) >> 1, the hidden bit of z adds one
    return words((uint32_t)(z >> 32) + ((((hi + (1023u << 20)) >> 1) & 0x7ff00000u) - (1u << 20)), (uint32_t)z);
}

// ---- comparisons on the integer pipe
__device__ __forceinline__ bool is_nan_bits(double x) { return (hi_word(x) & 0x7fffffffu) >= 0x7ff80000u; }   // quiet NaNs
__device__ __forceinline__ long long order_key(double x) {
    const long long b = (long long)(((unsigned long long)hi_word(x) << 32) | lo_word(x));
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
// a < b ? a : b and a > b ? a : b as the plain operators give them (b when
// either is a NaN)
__device__ __forceinline__ double fp64_min(double a, double b) {
    return order_key(a) < order_key(b) && !is_nan_bits(a) && !is_nan_bits(b) ? a : b;
}
__device__ __forceinline__ double fp64_max(double a, double b) {
    return order_key(a) > order_key(b) && !is_nan_bits(a) && !is_nan_bits(b) ? a : b;
}
// |x| as an ordered integer
__device__ __forceinline__ unsigned long long magnitude(double x) {
    return ((unsigned long long)(hi_word(x) & 0x7fffffffu) << 32) | lo_word(x);
}
// x < 0, x >= 0 and x <= 0 (false for a NaN)
__device__ __forceinline__ bool fp64_negative(double x) {
    const uint32_t h = hi_word(x);
    return h - 0x80000000u < 0x7ff80000u && ((h << 1) | lo_word(x)) != 0u;
}
__device__ __forceinline__ bool fp64_ge0(double x) {
    const uint32_t h = hi_word(x);
    return h < 0x7ff80000u || (h == 0x80000000u && lo_word(x) == 0u);
}
__device__ __forceinline__ bool fp64_le0(double x) {
    const uint32_t h = hi_word(x);
    return (h >= 0x80000000u && h < 0xfff80000u) || (h | lo_word(x)) == 0u;
}

}  // namespace knc
