// Double-float ("df64") arithmetic: a value is the unevaluated sum hi + lo of
// two binary32 numbers (|lo| <= ulp(hi)), about 48 significant bits.
//
// Why: on GB300 the FP64 pipe runs at 1/71 of the FP32 rate (1.0 vs 71.9
// TFLOP/s measured) and f64<->f32 conversions occupy that same pipe. The
// FP64-accurate assembly therefore computes with error-free transformations
// on the FP32 pipes (Dekker / Knuth TwoSum and an FMA-based TwoProduct), and
// converts between double and df64 with integer bit manipulation.
//
// All operations use explicitly rounded intrinsics on the device (never
// contracted or re-associated by the compiler); on the host the same code runs
// with plain float operations and must be compiled with -ffp-contract=off.
//
// Accuracy (unit roundoff u = 2^-24; bounds checked against exact rationals by
// tests/test_df64.py, which also covers the conversions below):
//   two_sum, two_prod     exact
//   df_add (sloppy)       |err| <= 2u^2 (|x| + |y|)
//   df_mul                |err| <= 4u^2 |x y|
//   df_recip              |err| <= 2^-46 |1/x|  (one Newton step from the rounded binary32 reciprocal)
//   df_rsqrt              |err| <= 2^-47 x^(-1/2)
//   d2df                  |err| <= 2^-48 |x|   for 2^-100 <= |x| <= 2^127 (both halves normal)
//   df2d                  |err| <= 2^-53 |hi + lo|
#pragma once
#include <cstdint>
#include <cstring>
#include <cmath>

#if defined(__CUDACC__)
#define FGPU_HD __host__ __device__ __forceinline__
#else
#define FGPU_HD inline
#endif

namespace fgpu {

struct df {
    float hi, lo;
};

FGPU_HD float f_add(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
FGPU_HD float f_sub(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
}
FGPU_HD float f_mul(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
FGPU_HD float f_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
FGPU_HD uint32_t f_bits(float x) {
#if defined(__CUDA_ARCH__)
    return __float_as_uint(x);
#else
    uint32_t u;
    std::memcpy(&u, &x, 4);
    return u;
#endif
}
FGPU_HD float f_from_bits(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float x;
    std::memcpy(&x, &u, 4);
    return x;
#endif
}
FGPU_HD uint64_t d_bits(double x) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}
FGPU_HD double d_from_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}
FGPU_HD int clz64(uint64_t x) {
#if defined(__CUDA_ARCH__)
    return __clzll((long long)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}

// Knuth TwoSum: s + e == a + b exactly.
FGPU_HD df two_sum(float a, float b) {
    float s = f_add(a, b);
    float bb = f_sub(s, a);
    float e = f_add(f_sub(a, f_sub(s, bb)), f_sub(b, bb));
    return {s, e};
}
// Dekker FastTwoSum, requires |a| >= |b| (or a == 0).
FGPU_HD df quick_two_sum(float a, float b) {
    float s = f_add(a, b);
    float e = f_sub(b, f_sub(s, a));
    return {s, e};
}
FGPU_HD df df_add(df x, df y) {
    df s = two_sum(x.hi, y.hi);
    float e = f_add(s.lo, f_add(x.lo, y.lo));
    return quick_two_sum(s.hi, e);
}
FGPU_HD df df_neg(df x) { return {-x.hi, -x.lo}; }
FGPU_HD df df_sub(df x, df y) { return df_add(x, df_neg(y)); }
FGPU_HD df df_mul(df x, df y) {
    float p = f_mul(x.hi, y.hi);
    float e = f_fma(x.hi, y.hi, -p);
    e = f_fma(x.hi, y.lo, e);
    e = f_fma(x.lo, y.hi, e);
    return quick_two_sum(p, e);
}
// x * 2^k for a small exact power of two given as a float
FGPU_HD df df_scale(df x, float pow2) { return {f_mul(x.hi, pow2), f_mul(x.lo, pow2)}; }
// 1 / x: Newton step in df64 from the correctly rounded binary32 reciprocal.
FGPU_HD df df_recip(df x) {
#if defined(__CUDA_ARCH__)
    float r = __frcp_rn(x.hi);
#else
    float r = 1.0f / x.hi;
#endif
    df xr = df_mul(x, df{r, 0.0f});
    df e = df_sub(df{1.0f, 0.0f}, xr);
    df t = df_mul(df{r, 0.0f}, e);
    return df_add(df{r, 0.0f}, t);
}
// x^(-1/2), x > 0: r (1 + e / 2 + 3 e^2 / 8) from the binary32 value r, with e = 1 - x r^2 (at most some 2^-22)
// summed from exact products: x r^2 is near 1, so 1 minus its high part is exact.
FGPU_HD df df_rsqrt(df x) {
#if defined(__CUDA_ARCH__)
    float r = __frsqrt_rn(x.hi);
#else
    float r = 1.0f / std::sqrt(x.hi);
#endif
    const float p = f_mul(r, r), q = f_fma(r, r, -p);        // r^2 = p + q
    const float a = f_mul(x.hi, p), b = f_fma(x.hi, p, -a);  // x.hi p = a + b
    const df u = two_sum(f_sub(1.0f, a), -b);
    const df v = two_sum(u.hi, -f_fma(x.hi, q, f_mul(x.lo, p)));
    const float th = f_mul(0.5f, v.hi), tl = f_fma(f_mul(0.375f, v.hi), v.hi, f_mul(0.5f, f_add(u.lo, v.lo)));
    const float m = f_mul(r, th);
    const df y = quick_two_sum(r, m);
    return quick_two_sum(y.hi, f_add(y.lo, f_fma(r, tl, f_fma(r, th, -m))));
}

// double -> df64 with integer operations only. Zero, subnormal doubles and
// magnitudes below 2^-126 map to 0; magnitudes above the binary32 range map to inf.
FGPU_HD df d2df_any(double x) {
    uint64_t b = d_bits(x);
    uint32_t sign = (uint32_t)(b >> 63);
    int e = (int)((b >> 52) & 0x7FF);
    uint64_t m = b & 0xFFFFFFFFFFFFFull;
    int fe = e - 1023 + 127;
    if (e == 0 || fe <= 0) return {sign ? -0.0f : 0.0f, 0.0f};
    if (fe >= 255) return {f_from_bits((sign << 31) | 0x7F800000u), 0.0f};
    float hi = f_from_bits((sign << 31) | ((uint32_t)fe << 23) | (uint32_t)(m >> 29));
    uint32_t rest = (uint32_t)(m & ((1ull << 29) - 1));      // value rest * 2^(e - 1075)
    float lo = 0.0f;
    if (rest) {
        int pe = e - 1075 + 127;                               // biased exponent of 2^(e - 1075)
        float r = (float)rest;                                 // rounds 29 -> 24 bits
        if (pe >= 1) {
            lo = f_mul(r, f_from_bits((uint32_t)pe << 23));
        } else {
            lo = std::ldexp(r, e - 1075);
        }
        if (sign) lo = -lo;
    }
    return quick_two_sum(hi, lo);
}

FGPU_HD float f_from_int(int x) { return (float)x; }
// double -> df64: for 2^-74 <= |x| < 2^127 the high part is the truncated binary32 pattern (exponent
// rebiased in place) and the low part the remaining 29 bits, one integer conversion: 16 instructions
// (about 45 on the general path, which takes everything else).
FGPU_HD df d2df(double x) {
    const uint64_t b = d_bits(x);
    const uint32_t w1 = (uint32_t)(b >> 32), w0 = (uint32_t)b, sign = w1 & 0x80000000u;
    if ((w1 & 0x7FFFFFFFu) - (949u << 20) >= (201u << 20)) return d2df_any(x);      // biased exponent 949 .. 1149
    const uint32_t h = ((w1 << 3) | (w0 >> 29)) - (896u << 23);
    const float scale = f_from_bits((((h & 0x7F800000u) - (52u << 23))) | sign);    // 2^(e - 1075), x's sign
    return quick_two_sum(f_from_bits(h | sign), f_mul(f_from_int((int)(w0 & 0x1FFFFFFFu)), scale));
}

// df64 -> double with integer operations only, any pair (hi normal or zero; lo below 2^-126 ignored).
FGPU_HD double df2d_any(df x) {
    uint32_t hb = f_bits(x.hi);
    int he = (int)((hb >> 23) & 0xFF);
    if (he == 0) return (hb >> 31) ? -0.0 : 0.0;
    if (he == 255) return (hb >> 31) ? -INFINITY : INFINITY;
    int64_t mh = (int64_t)((hb & 0x7FFFFFu) | 0x800000u);     // value mh * 2^(he - 150)
    if (hb >> 31) mh = -mh;
    uint32_t lb = f_bits(x.lo);
    int le = (int)((lb >> 23) & 0xFF);
    int64_t M = mh * ((int64_t)1 << 29);                      // value M * 2^(he - 179)
    if (le != 0 && le != 255) {
        int64_t ml = (int64_t)((lb & 0x7FFFFFu) | 0x800000u);
        if (lb >> 31) ml = -ml;
        int d = he - le;
        if (d <= 29) M += ml * ((int64_t)1 << (29 - d));
        else if (d - 29 < 63) M += ml >> (d - 29);
    }
    uint64_t sign = 0;
    if (M < 0) { sign = 1; M = -M; }
    if (M == 0) return 0.0;
    uint64_t U = (uint64_t)M;
    int top = 63 - clz64(U);                                  // highest set bit
    int shift = top - 52;
    if (shift > 0) {
        uint64_t half = (uint64_t)1 << (shift - 1);
        U = (U + half) >> shift;
        if (U >> 53) { U >>= 1; ++shift; }
    } else if (shift < 0) {
        U <<= -shift;
    }
    int64_t de = (int64_t)he - 179 + shift + 52 + 1023;
    return d_from_bits((sign << 63) | ((uint64_t)de << 52) | (U & 0xFFFFFFFFFFFFFull));
}

FGPU_HD int f_rint(float x) {
#if defined(__CUDA_ARCH__)
    return __float2int_rn(x);
#else
    return (int)std::nearbyint(x);
#endif
}
// df64 -> double, correctly rounded. Binary64 values of one sign are ordered like their bit patterns, so
// hi + lo is hi's pattern plus lo counted in units of hi's last binary64 place (twice as many where lo
// points below a power of two). A normalised pair has |lo| at most 2^28 such units; anything else takes
// the general path. 14 integer and conversion instructions against about 45 there: the assembly's gather
// converts every CSR entry once.
FGPU_HD double df2d(df x) {
    const uint32_t hb = f_bits(x.hi), lb = f_bits(x.lo), sign = hb & 0x80000000u, he = (hb >> 23) & 0xFFu;
    // |lo| in units of 2^(he - 179), positive where it has hi's sign
    float t = f_mul(f_mul(f_from_bits(lb ^ sign), f_from_bits((254u - he) << 23)), 4503599627370496.0f);
    if ((hb & 0x7FFFFFu) == 0u && t < 0.0f) t = f_add(t, t);
    if (he - 1u >= 253u || !(t <= 536870912.0f && t >= -536870912.0f)) return df2d_any(x);
    const uint64_t m = ((uint64_t)(hb ^ sign) << 29) + ((uint64_t)896 << 52) + (uint64_t)(int64_t)f_rint(t);
    return d_from_bits(m | ((uint64_t)sign << 32));
}

}  // namespace fgpu
