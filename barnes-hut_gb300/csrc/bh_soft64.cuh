// FP64 operations on the integer pipes, rounded as IEEE 754 rounds them
// (to nearest, ties to even), for the exact walk's interaction terms.
//
// An FP64 instruction of a warp holds the SM's FP64 pipe for 16 cycles here
// (two lanes per cycle), in which the four schedulers issue 64 instructions.
// A correctly rounded product of two 53-bit significands takes about 20
// integer instructions, and a square root with the reciprocal of its result
// about 80, so most of a term's operations cost less as integer code, and
// they run beside the FP64 pipe instead of in it.
//
// A normal double is carried as Sig{a, e}: value = a 2^(e - 63), a in
// [2^63, 2^64) with its low 11 bits zero.  Host builds of this header (the
// CPU tests) supply the same functions with 128-bit products.
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define BH_SOFT __host__ __device__ __forceinline__
#else
#include <cmath>
#define BH_SOFT inline
#endif

namespace bh {
namespace soft {

struct Sig {
    uint64_t a;
    int e;
};

BH_SOFT uint64_t bits_of(double v)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t b;
    std::memcpy(&b, &v, 8);
    return b;
#endif
}

BH_SOFT double from_bits(uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double v;
    std::memcpy(&v, &b, 8);
    return v;
#endif
}

// High 64 bits of the 128-bit product.
BH_SOFT uint64_t mulhi(uint64_t a, uint64_t b)
{
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// The same with b = y 2^32.
BH_SOFT uint64_t mulhi32(uint64_t a, uint32_t y)
{
    return (a >> 32) * y + (((a & 0xFFFFFFFFull) * y) >> 32);
}

BH_SOFT float float_of(uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __int_as_float((int)b);
#else
    float f;
    std::memcpy(&f, &b, 4);
    return f;
#endif
}

BH_SOFT uint32_t bits_of(float f)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__float_as_int(f);
#else
    uint32_t b;
    std::memcpy(&b, &f, 4);
    return b;
#endif
}

BH_SOFT float fma32(float a, float b, float c)
{
#ifdef __CUDA_ARCH__
    return fmaf(a, b, c);
#else
    return std::fmaf(a, b, c);
#endif
}

// Integers to and from FP32 by adding 2^23 (1.5 2^23 for signed ones) on the
// bit patterns: the conversion instructions take the FP64 pipe here.
BH_SOFT float small_float(uint32_t v) { return float_of(0x4B000000u + v) - 8388608.0f; }     // v < 2^23
BH_SOFT uint32_t small_round(float f) { return bits_of(f + 8388608.0f) - 0x4B000000u; }        // 0 <= f <= 2^23
BH_SOFT float small_float_s(int v) { return float_of(0x4B400000u + (uint32_t)v) - 12582912.0f; }  // |v| < 2^22
BH_SOFT int small_round_s(float f) { return (int)(bits_of(f + 12582912.0f) - 0x4B400000u); }      // |f| < 2^22

// The estimate of 1/sqrt(f) everything below starts from: within 2^-22.
// (f is far from subnormal; rsqrtf puts a scaling for those around it.)
#ifdef __CUDACC__
__device__ __forceinline__ float rsqrt_hw(float f)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    return y;
}
#endif
#ifndef BH_SOFT_RSQRT
#ifdef __CUDA_ARCH__
#define BH_SOFT_RSQRT(f) rsqrt_hw(f)
#else
#define BH_SOFT_RSQRT(f) (1.0f / std::sqrt(f))
#endif
#endif

// +-0, from the two 32-bit words (a test of the shifted 64-bit pattern is
// compiled to an FP64 comparison, which takes the FP64 pipe).
BH_SOFT bool is_zero(uint64_t b) { return (((uint32_t)(b >> 32) & 0x7FFFFFFFu) | (uint32_t)b) == 0u; }

// Significand and exponent of a normal positive or negative double.
BH_SOFT Sig unpack(uint64_t b)
{
    return Sig{(b << 11) | 0x8000000000000000ull, (int)((b >> 52) & 0x7FF) - 1023};
}

// Products.  The high half p of the 128-bit product holds the 53-bit
// significand and 10 or 11 bits below it.  Adding half a last place and
// truncating rounds to nearest; only a product exactly half way between two
// significands would need to go to the even one, and such a product has at
// least 64 trailing zeros, so that one of its factors ends in 32 zero bits.
// `odd_case` is raised for those factors (and for a result that rounds up to
// a power of two); the caller then takes the IEEE operations.
BH_SOFT bool low_zero(const Sig& x) { return (uint32_t)x.a == 0u; }

// RN(x y), to go on with.
BH_SOFT Sig mul(const Sig& x, const Sig& y, bool& odd_case)
{
    uint64_t p = mulhi(x.a, y.a);
    const int top = (int)(p >> 63);
    p = ((p << (1 - top)) + 0x400u) & ~0x7FFull;
    odd_case = odd_case || (int64_t)p >= 0;
    return Sig{p, x.e + y.e + top};
}

// RN(x y) as the bit pattern of a positive double; exponents in the normal
// range.  A significand that rounds up to 2^53 carries into the exponent.
BH_SOFT uint64_t mul_bits(uint64_t a, uint64_t b, int e)
{
    const uint64_t p = mulhi(a, b);
    const int top = (int)(p >> 63);
    return ((p + (uint64_t)(0x200u << top)) >> (10 + top)) + ((uint64_t)(uint32_t)(e + top + 1022) << 52);
}

// RN(1 / RN(sqrt(x))).  x = X 2^(2k) with X in [2^62, 2^64); s = sqrt(X) 2^21
// in [2^31+21, 2^53) is the square root in units of its own last place.
//  * Y = 2^38 (1 - d) / sqrt(X 2^-32) from the FP32 estimate (within 2^-22 of
//    its argument's, the argument truncated by less than 2^-23), scaled down
//    by 2^-20.68 so that Y is never above the true value: d in (0, 2^-20).
//    e = 1 - X Y^2 2^-108 in (0, 2^-18.9) to 2^-62 from integer products, and
//    (1 - e)^(-1/2) = 1 + e/2 + 3/8 e^2 + 5/16 e^3 (next term below 2^-77).
//  * s follows as X Y (1 - e)^(-1/2) to about 2^-9 of a last place.  With
//    q = floor(s), RN is q or q + 1 as s lies below or above q + 1/2 (never
//    on it: the square of an odd multiple of 1/2 is no integer), decided by
//    the exact integer X 2^44 - (2 q + 1)^2, whose magnitude stays below 2^63
//    so that its low 64 bits carry it; an estimate that falls on the wrong
//    side of an integer ends at the same result.
//  * 1/R for the rounded root R: 2^105 / s from the same Y and e, corrected
//    by the rounding of the root, (s - R) / R, in FP32, then rounded by the
//    exact sign of 2^106 - R (2 v + 1) in the same way.
// odd_case: the reciprocal is a power of two.
BH_SOFT Sig rcp_sqrt(const Sig& x, bool& odd_case)
{
    const int odd = x.e & 1;
    const uint64_t X = x.a >> (1 - odd);
    const int k = (x.e + 1 - odd - 63) >> 1;  // exact: the sum is even
    // X 2^-32 truncated to FP32 (24 bits), on the bit patterns
    const float xf = float_of(((uint32_t)(127 + 30 + odd) << 23) | ((uint32_t)(x.a >> 40) & 0x7FFFFFu));
    // 2^38 (1 - 2^-20.68) / sqrt(X 2^-32) rounded to an integer
    const float v = fma32(BH_SOFT_RSQRT(xf), 274877743104.0f, 8388608.0f);
    const float Yf = v - 8388608.0f;
    const uint64_t Y = bits_of(v) - 0x4B000000u;
    const uint64_t Y2 = Y * Y;  // below 2^46
    const uint64_t E = 0x4000000000000000ull - mulhi(X, Y2 << 18);  // e 2^62, e > 0
    const float ef = small_float((uint32_t)(E >> 21)) * 0x1p-41f;
    // the e^2 and e^3 terms in units of 2^-62 (below 2^23)
    const uint32_t quad = small_round(ef * ef * fma32(0.3125f, ef, 0.375f) * 0x1p62f);
    const uint64_t D = (E >> 1) + quad;  // delta 2^62, below 2^43
    const uint64_t A = mulhi32(X, (uint32_t)Y << 9);  // X Y 2^-23 = s 2^10 (1 - e)^(1/2)
    const uint64_t S = A + mulhi(A, D << 2);  // s 2^10
    uint64_t R = S >> 10;
    const uint64_t odd2 = 2 * R + 1;
    if ((int64_t)((X << 44) - odd2 * odd2) > 0) ++R;
    const int f = (int)(int64_t)(S - (R << 10));  // (s - R) 2^10
    const uint64_t T = ((Y * (D >> 2)) >> 20) + (Y << 40);  // 2^105 / s, times 2^10
    // 2^105 / s (s - R) / R, times 2^10: 2^105 / R^2 is Y^2 2^-45 up to 2^-18
    const int c = small_round_s(small_float_s(f) * (Yf * Yf) * 0x1p-45f);
    uint64_t V = (T + (uint64_t)(int64_t)c) >> 10;
    if ((int64_t)(0ull - R * (2 * V + 1)) > 0) ++V;
    odd_case = odd_case || (V >> 53) != 0;
    return Sig{V << 11, -32 - k};
}

// d d rounded, for d = 0 or |d| in [2^-400, 2^400] with a significand that
// does not end in 32 zero bits.  Larger |d|, infinities and NaN give at least
// 2^800 or no number, as the exponent stops at 511: an r^2 with such a square
// in it is outside term()'s range.  (The bound here, not on term()'s components:
// forces at 19,054 bodies 1.105 ms, 1.123 there, 1.100 without one.)
BH_SOFT double square(uint64_t d)
{
    const Sig s = unpack(d);
    const int e = s.e < 511 ? s.e : 511;
    return from_bits(is_zero(d) ? 0ull : mul_bits(s.a, s.a, 2 * e));
}

// The reference's interaction term (src/traversal.cpp:82-88) from the
// displacement, r^2 and G m, all rounded as it rounds them:
//   i = RN(1/RN(sqrt(r2))), i3 = RN(RN(i i) i), sc = RN(gm i3),
//   t = RN(sc d) per component (0 where d = +-0).
// Returns false (t unset) outside r^2 in 2^+-200, G m in 2^+-300 and |d| = 0
// or at least 2^-300 (where every product stays in the normal range; r^2 bounds
// |d| from above), and in the odd cases above.
BH_SOFT bool term(double dx, double dy, double dz, double r2, double gm, double& tx, double& ty, double& tz)
{
    const uint64_t br = bits_of(r2), bg = bits_of(gm);
    bool odd_case = (uint32_t)(br >> 32) - ((uint32_t)(1023 - 200) << 20) >= (uint32_t)400 << 20 ||
                    (uint32_t)(bg >> 32) - ((uint32_t)(1023 - 300) << 20) >= (uint32_t)600 << 20;
    const Sig i = rcp_sqrt(unpack(br), odd_case);
    const Sig i2 = mul(i, i, odd_case);
    const Sig i3 = mul(i2, i, odd_case);
    const Sig g = unpack(bg);
    const Sig sc = mul(g, i3, odd_case);
    odd_case = odd_case || low_zero(i) || low_zero(i2) || low_zero(i3) || low_zero(g) || low_zero(sc);
    auto component = [&](double dk) {
        const uint64_t d = bits_of(dk);
        const bool zero = is_zero(d);
        const Sig s = unpack(d);
        odd_case = odd_case || (!zero && (low_zero(s) || s.e < -300));
        const uint64_t v = mul_bits(sc.a, s.a, sc.e + s.e) | (d & 0x8000000000000000ull);
        return from_bits(zero ? 0ull : v);
    };
    tx = component(dx);
    ty = component(dy);
    tz = component(dz);
    return !odd_case;
}

// Leading zeros of a non-zero 32-bit word.
BH_SOFT int clz32(uint32_t v)
{
#ifdef __CUDA_ARCH__
    return __clz((int)v);
#else
    return __builtin_clz(v);
#endif
}

// G m r^-3 for the FP64 list form, which needs no particular rounding: within
// an ulp of the exact value for the displacement given (the FP64 sequence it
// replaces: three FMAs, rcube_hh and a product, within 6 ulps), with the
// result's rounding the only one to 53 bits.
//  * The components as 63-bit integers M with one exponent; r^2 = sum of the
//    high halves of M^2, S, to 2^-58; S moved up by 0 or 2 bits into
//    [2^62, 2^64) (any scale left is an even power of two).
//  * Y = 2^38 (1 - d) / sqrt(S 2^-32) from the FP32 estimate, never above the
//    true value, as in rcp_sqrt, with d below 2^-19.9 (S 2^-41 is an FP32
//    integer of 22 or 23 bits); e = 1 - S Y^2 2^-108 below 2^-18.9, and
//    (1 - e)^(-3/2) = 1 + 3/2 e + 15/8 e^2 + 35/16 e^3 (+ 2^-72).
//  * Y^3 is exact in 69 bits; P is its leading part times the series, to
//    2^-57.
// Returns false (value unset) outside: largest component in 2^+-100, G m a
// normal number in 2^+-300.
BH_SOFT bool scale(double dx, double dy, double dz, double gm, double& sc)
{
    const uint64_t b[3] = {bits_of(dx), bits_of(dy), bits_of(dz)};
    const uint64_t bg = bits_of(gm);
    int e[3];
    for (int k = 0; k < 3; ++k) e[k] = (int)((uint32_t)(b[k] >> 52) & 0x7FFu);
    int emax = e[0] > e[1] ? e[0] : e[1];
    emax = emax > e[2] ? emax : e[2];
    const bool ok = (uint32_t)(emax - 923) <= 200u &&
                    (uint32_t)(bg >> 32) - ((uint32_t)(1023 - 300) << 20) < (uint32_t)600 << 20;
    uint64_t S = 0;
    for (int k = 0; k < 3; ++k) {
        int sh = emax - e[k];
        if (sh > 63) sh = 63;
        const uint64_t M = (((b[k] << 10) & 0x3FFFFFFFFFFFFFFFull) | 0x4000000000000000ull) >> sh;
        const uint64_t h = M >> 32, l = M & 0xFFFFFFFFull;
        S += h * h + ((h * l) >> 31);
    }
    const int z = (S >> 62) == 0 ? 1 : 0;
    S <<= 2 * z;
    // r^2 = S 2^(2 q)
    const int q = emax - 1085 + 32 - z;
    // 2^38 (1 - 2^-20.5) / sqrt(S 2^-32): sqrt(2^-9) of the estimate's argument
    // in the scale
    const float v = fma32(BH_SOFT_RSQRT(small_float((uint32_t)(S >> 41))), 12147993600.0f, 8388608.0f);
    const uint64_t Y = bits_of(v) - 0x4B000000u;
    const uint64_t Y2 = Y * Y;
    const uint64_t E = 0x4000000000000000ull - mulhi(S, Y2 << 18);  // e 2^62
    const float ef = small_float((uint32_t)(E >> 21)) * 0x1p-41f;
    const uint64_t quad = (uint64_t)small_round(ef * ef * fma32(2.1875f, ef, 1.875f) * 0x1p57f) << 5;
    const uint64_t D = E + (E >> 1) + quad;
    uint64_t P = mulhi32(Y2 << 18, (uint32_t)Y << 8);  // Y^3 2^-6
    P += mulhi(P, D << 2);
    // sc = w 2^(eg - 155 - 3 q), eg the exponent of G m
    uint64_t w = mulhi((bg << 11) | 0x8000000000000000ull, P);
    const int n = clz32((uint32_t)(w >> 32));
    w <<= n;
    const int eg = (int)((uint32_t)(bg >> 52) & 0x7FFu) - 1023;
    // value w 2^(x): leading bit 2^63; significand rounded to 53 bits
    const int x = eg - 155 - 3 * q - n + 63;
    sc = from_bits(((w + 0x400u) >> 11) + (w + 0x400u < w ? 0x0020000000000000ull : 0ull) +
                   ((uint64_t)(uint32_t)(x + 1022) << 52));
    return ok;
}

}  // namespace soft
}  // namespace bh
