// FP64 division and square root in integer arithmetic.
//
// GB300 has one FP64 lane pair per SM. Measured on it (2070 MHz, cycles of one
// warp): any FP64 add, multiply, fma, compare or conversion takes 45-64 and
// overlaps with no other of its warp, so that a division takes 564 and a square
// root 600, and an SM at full load completes one of either per 143 cycles. A
// 32-bit integer add takes 1.5 cycles (0.35 of the SM), a 32 x 32 -> 64 bit
// multiply 6.6 (1.4). The functions here compute the same IEEE results (round to
// nearest even) with 32- and 64-bit integer operations, so every caller's value
// is unchanged to the last bit; operands outside the range they cover (zeros,
// subnormals, infinities, NaN, results near the ends of the exponent range) take
// the hardware's operation.
//
// Division and square root: a 31-bit reciprocal (or reciprocal square root) from
// the hardware's FP32 approximation and one Newton step, two quotient (root)
// digits of 29 and 25 bits taken from exact remainders, and the exact final
// remainder. A quotient or a root of 53-bit numbers is never a midpoint of two
// 53-bit numbers, so the first 54 bits decide the rounding.
//
// Both are functions of their own: 307 and 339 cycles of a warp with the call
// (28 and 31 of the SM), against 250 and 283 inlined. Inlined at their ~200 call
// sites they made a transport slower, not faster (one 100 MeV shower in FP64 14.3
// ms against 13.3 with the hardware's operations and 12.2 with calls): with few
// tracks a launch runs through its code once, and its time is that of fetching
// it. A call also leaves the caller's basic blocks as an operation does, so that
// the compiler contracts the mixed build's multiply-adds as before and its results
// stay the same. Transports: c2's physics in FP64, 300 electrons, 552 -> 484 ms;
// one c3-like event in FP64 1153 -> 1058 ms; 3000 c2 electrons in the mixed build
// 244 -> 226 ms.
//
// The host compiles the plain operations, which give the same values.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include "Macros.hh"

namespace gbx
{
namespace fp64
{
// Approximations of 1 / f, f in [1, 2), and 1 / sqrt(f), f in [1, 4), as FP32
// bits, off by at most 2^-22.4 relative; the host's stand-ins serve the tests
GBX_FORCEINLINE std::uint32_t approx_rcp(std::uint32_t f)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
    return __float_as_uint(r);
#else
    float x, y;
    std::memcpy(&x, &f, sizeof(x));
    y = 1 / x;
    std::uint32_t u;
    std::memcpy(&u, &y, sizeof(u));
    return u;
#endif
}
GBX_FORCEINLINE std::uint32_t approx_rsqrt(std::uint32_t f)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
    return __float_as_uint(r);
#else
    float x, y;
    std::memcpy(&x, &f, sizeof(x));
    y = 1 / std::sqrt(x);
    std::uint32_t u;
    std::memcpy(&u, &y, sizeof(u));
    return u;
#endif
}

//! High 32 bits of a product
GBX_FORCEINLINE std::uint32_t mul_hi(std::uint32_t a, std::uint32_t b)
{
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return static_cast<std::uint32_t>((std::uint64_t(a) * b) >> 32);
#endif
}
GBX_FORCEINLINE std::int32_t mul_hi_s(std::int32_t a, std::int32_t b)
{
#if defined(__CUDA_ARCH__)
    return __mulhi(a, b);
#else
    return static_cast<std::int32_t>((std::int64_t(a) * b) >> 32);
#endif
}
//! 32 x 32 -> 64 bits
GBX_FORCEINLINE std::uint64_t mul_wide(std::uint32_t a, std::uint32_t b)
{
    return std::uint64_t(a) * b;
}
//! Low 64 bits of a 32 x 64 bit product
GBX_FORCEINLINE std::uint64_t mul_lo(std::uint32_t a, std::uint64_t b)
{
    return mul_wide(a, static_cast<std::uint32_t>(b))
           + (std::uint64_t(a * static_cast<std::uint32_t>(b >> 32)) << 32);
}

constexpr std::uint64_t mantissa_mask = 0x000fffffffffffffull;
constexpr std::uint64_t hidden_bit = 0x0010000000000000ull;

//! Significand of a / b for significands ma, mb in [2^52, 2^53): the 53-bit
//! correctly rounded quotient of ma (or, when ma < mb, 2 ma) by mb. 'y' is
//! approx_rcp of mb's leading 24 bits as a float in [1, 2).
GBX_FORCEINLINE std::uint64_t div_significand(std::uint64_t ma, std::uint64_t mb, std::uint32_t y)
{
    // a / b in [1, 2)
    std::uint64_t const num = ma << (ma < mb ? 1 : 0);
    // 1 / b, b in [1, 2): r0 * 2^-24 (23 bits), then one Newton step,
    // r1 * 2^-31 <= 1 / b with an error below 2^-28
    std::uint32_t const r0 = 0x800000u + (y - 0x3f000000u);
    std::uint64_t const p = mul_wide(static_cast<std::uint32_t>(mb >> 21), r0);
    auto const e = static_cast<std::int32_t>(static_cast<std::int64_t>((1ull << 55) - p) >> 3);
    std::uint32_t const r1 = (r0 << 7) + (mul_hi_s(static_cast<std::int32_t>(r0), e) >> 13) - 4;
    // First digit: floor of the quotient times 2^29, or just below; the
    // remainder num 2^29 - q1 mb is nonnegative and below 2^55
    std::uint32_t const q1 = mul_hi(static_cast<std::uint32_t>(num >> 22), r1);
    std::uint64_t const rem1 = (num << 29) - mul_lo(q1, mb);
    // Second digit: 24 more bits, at most one below the floor
    std::uint32_t const q2 = mul_hi(static_cast<std::uint32_t>(rem1 >> 24), r1) >> 3;
    std::uint64_t const rem2 = (rem1 << 24) - mul_lo(q2, mb);
    std::uint64_t const q = (std::uint64_t(q1) << 24) + q2 + (rem2 >= mb ? 1 : 0);
    return (q + 1) >> 1;
}

//! Significand of sqrt(m 2^-52), m in [2^52, 2^54): the 53-bit correctly
//! rounded root times 2^52. 'y' is approx_rsqrt of m's leading 24 bits as a
//! float in [1, 4).
GBX_FORCEINLINE std::uint64_t sqrt_significand(std::uint64_t m, std::uint32_t y)
{
    // 1 / sqrt: r0 * 2^-24, one Newton step, r1 * 2^-31 below the value by
    // less than 2^-28
    std::uint32_t const r0 = 0x800000u + (y - 0x3f000000u);
    auto const sq = static_cast<std::uint32_t>(mul_wide(r0, r0) >> 18);  // times 2^30
    std::uint64_t const p = mul_wide(static_cast<std::uint32_t>(m >> 22), sq);
    auto const e = static_cast<std::int32_t>(static_cast<std::int64_t>((1ull << 60) - p) >> 9);
    std::uint32_t const r1 = (r0 << 7) + (mul_hi_s(static_cast<std::int32_t>(r0), e) >> 13) - 4;
    // First digit: root times 2^29, rounded down; exact remainder times 2^58
    std::uint32_t const s1 = mul_hi(static_cast<std::uint32_t>(m >> 22), r1);
    std::uint64_t const rem1 = (m << 6) - mul_wide(s1, s1);
    // Second digit: rem1 / (2 s1), 24 more bits, at most two below the floor
    std::uint32_t const s2 = mul_hi(static_cast<std::uint32_t>(rem1 >> 4), r1) >> 1;
    std::uint64_t const rem2 = (rem1 << 48) - mul_lo(s2, (std::uint64_t(s1) << 25) + s2);
    std::uint64_t s = (std::uint64_t(s1) << 24) + s2;
    s += (rem2 > 2 * s ? 1 : 0) + (static_cast<std::int64_t>(rem2 - 4 * s - 4) >= 0 ? 1 : 0);
    return (s + 1) >> 1;
}


//! a / b, correctly rounded, inlined: for a loop that one track waits for
GBX_FORCEINLINE double div_inline(double a, double b)
{
#if defined(__CUDA_ARCH__)
    std::uint64_t const ua = __double_as_longlong(a);
    std::uint64_t const ub = __double_as_longlong(b);
    auto const ah = static_cast<std::uint32_t>(ua >> 32);
    auto const bh = static_cast<std::uint32_t>(ub >> 32);
    std::uint32_t const ea = (ah >> 20) & 0x7ffu;
    std::uint32_t const eb = (bh >> 20) & 0x7ffu;
    std::uint64_t const ma = (ua & mantissa_mask) | hidden_bit;
    std::uint64_t const mb = (ub & mantissa_mask) | hidden_bit;
    // Biased exponent of the quotient, less one
    std::uint32_t const e = ea - eb + 1022u - (ma < mb ? 1u : 0u);
    if (ea - 1u < 2046u && eb - 1u < 2046u && e < 2045u)
    {
        std::uint32_t const f = 0x3f800000u | (static_cast<std::uint32_t>(mb >> 29) & 0x7fffffu);
        std::uint64_t const q = div_significand(ma, mb, approx_rcp(f));
        // The hidden bit adds the one to the exponent
        std::uint32_t const top = ((ah ^ bh) & 0x80000000u) | (e << 20);
        return __longlong_as_double(q + (std::uint64_t(top) << 32));
    }
    return a / b;
#else
    return a / b;
#endif
}

//! Square root, correctly rounded, inlined
GBX_FORCEINLINE double sqrt_inline(double a)
{
#if defined(__CUDA_ARCH__)
    std::uint64_t const ua = __double_as_longlong(a);
    auto const ah = static_cast<std::uint32_t>(ua >> 32);
    // Positive and normal
    if (ah - 0x00100000u < 0x7fe00000u)
    {
        std::uint32_t const e = ah >> 20;
        // a = m 2^(2 k - 52), m in [2^52, 2^54)
        std::uint32_t const odd = (e & 1u) ^ 1u;
        std::uint64_t const m = ((ua & mantissa_mask) | hidden_bit) << odd;
        std::uint32_t const f
            = ((127u + odd) << 23) | (static_cast<std::uint32_t>(ua >> 29) & 0x7fffffu);
        std::uint64_t const s = sqrt_significand(m, approx_rsqrt(f));
        std::uint32_t const k = ((e + 1023u - odd) >> 1) - 1u;
        return __longlong_as_double(s + (std::uint64_t(k) << 52));
    }
    return ::sqrt(a);
#else
    return std::sqrt(a);
#endif
}

//! The FP32 value nearest to a positive double (ties to even)
GBX_FORCEINLINE float narrow(double a)
{
#if defined(__CUDA_ARCH__)
    std::uint64_t const u = __double_as_longlong(a);
    auto const hi = static_cast<std::uint32_t>(u >> 32);
    // In the range of FP32's normal numbers: rebias, round to 24 bits
    if (hi - 0x38100000u < 0x0fe00000u)
    {
        std::uint64_t const t = u - (std::uint64_t(0x38000000u) << 32) + 0x0fffffffu
                                + ((u >> 29) & 1u);
        return __uint_as_float(static_cast<std::uint32_t>(t >> 29));
    }
#endif
    return static_cast<float>(a);
}

//! The double equal to a positive FP32 number
GBX_FORCEINLINE double widen(float a)
{
#if defined(__CUDA_ARCH__)
    std::uint32_t const u = __float_as_uint(a);
    // Normal numbers: rebias
    if (u - 0x00800000u < 0x7f000000u)
    {
        return __hiloint2double(static_cast<int>((u >> 3) + 0x38000000u),
                                static_cast<int>(u << 29));
    }
#endif
    return a;
}
}  // namespace fp64

//! a / b, correctly rounded
GBX_NOINLINE double div(double a, double b)
{
    return fp64::div_inline(a, b);
}
//! Square root, correctly rounded
GBX_NOINLINE double sqrt(double a)
{
    return fp64::sqrt_inline(a);
}
GBX_FORCEINLINE float div(float a, float b)
{
    return a / b;
}
GBX_FORCEINLINE float sqrt(float a)
{
    return std::sqrt(a);
}
}  // namespace gbx
