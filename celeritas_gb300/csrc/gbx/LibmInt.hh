// exp, log, sin, cos, expm1 and log1p of the FP64 build in fixed-point integers.
//
// Libm.hh's functions are correctly rounded, so any evaluation that decides the
// rounding returns the same double. On GB300 a fixed-point one is far cheaper than
// one in double-doubles: an FP64 instruction takes one warp 64 cycles and 19 of
// the SM (a logarithm has about 40 of them), a 32 x 32 -> 64 bit multiply 6.6 and
// 1.4, an integer add 1.5 and 0.35. Each function here reduces its argument exactly
// in 64- and 128-bit integers, sums a Taylor series whose terms are held to as
// many bits as they contribute (32 or 64), and rounds the 128-bit result when an
// error of 2^-66 (exp, log, log1p), 2^-64 (sin, cos) or 2^-62 (expm1) of the power of two
// at or below the result cannot change the rounding. Otherwise, for about one argument
// in 2^13, 2^11 or 2^9, and outside the range covered, it returns false and the caller
// evaluates in double-doubles.
//
// The truncations of every operation, the rounded coefficients and the terms dropped,
// all at their worst and in one direction, sum to at most these parts of the error
// allowed: 0.48 (exp), 0.65 (log, log1p; near |log| = 2^-7), 0.62 (sin, cos; near pi/4) and
// 0.59 (expm1; below 2^-12).
//
// Sizes: 128-entry tables as Libm.hh's (log: C_j 2^-10 near 1/m, so that m C_j - 1
// is exact in 64 bits; exp: 2^(j/128)) leave |z| <= 2^-7 and |r| <= 2^-8.5, of which
// nine and seven terms reach 2^-69.
//
// Transports of the FP64 build with these and with double-doubles on the device:
// 100 electrons of 1 GeV in the calorimeter 102 -> 49 ms, c2's physics with 300
// electrons 484 -> 309 ms, a c3-like event 466 -> 398 ms.
//
// The functions compile on the host too, for the tests; the host's callers keep
// the double-doubles.
#pragma once

#include <cstdint>

#include "Fp64.hh"
#include "LibmTables.hh"

namespace gbx
{
namespace libm
{
namespace fixed
{
using i64 = std::int64_t;
using u64 = std::uint64_t;
using i32 = std::int32_t;
using u32 = std::uint32_t;
using u128 = unsigned __int128;

struct Words
{
    u64 hi, lo;
};
#if defined(__CUDACC__)
__device__ const u64 d_ilog_table[] = {GBX_LIBM_ILOG_TABLE};
__device__ const u64 d_iexp_table[] = {GBX_LIBM_IEXP_TABLE};
#endif
inline constexpr u64 h_ilog_table[] = {GBX_LIBM_ILOG_TABLE};
inline constexpr u64 h_iexp_table[] = {GBX_LIBM_IEXP_TABLE};
#if defined(__CUDA_ARCH__)
#    define GBX_LIBM_ILOAD(table, i) __ldg(&fixed::d_##table[i])
#else
#    define GBX_LIBM_ILOAD(table, i) fixed::h_##table[i]
#endif
constexpr Words ln2_q117{GBX_LIBM_LN2_Q117};
constexpr Words ln2_n_q96{GBX_LIBM_LN2_N_Q96};
constexpr Words pio2_q117{GBX_LIBM_PIO2_Q117};

GBX_FORCEINLINE u128 make128(u64 hi, u64 lo)
{
    return (u128(hi) << 64) | lo;
}
GBX_FORCEINLINE i64 mulhi(i64 a, i64 b)
{
#if defined(__CUDA_ARCH__)
    return __mul64hi(a, b);
#else
    return static_cast<i64>((static_cast<__int128>(a) * b) >> 64);
#endif
}
GBX_FORCEINLINE u64 mulhi_u(u64 a, u64 b)
{
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return static_cast<u64>((u128(a) * b) >> 64);
#endif
}
GBX_FORCEINLINE int count_leading_zeros(u64 x)
{
#if defined(__CUDA_ARCH__)
    return __clzll(static_cast<long long>(x));
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}
//! v << n, 0 <= n < 64
GBX_FORCEINLINE u128 shift_left(u128 v, int n)
{
    u64 const hi = static_cast<u64>(v >> 64);
    u64 const lo = static_cast<u64>(v);
    return make128((hi << n) | ((lo >> 1) >> (63 - n)), lo << n);
}
//! Low 128 bits of k times a 128-bit number, 0 <= k < 2^32
GBX_FORCEINLINE u128 mul_u32(u32 k, Words w)
{
    using fp64::mul_wide;
    u64 const p0 = mul_wide(k, static_cast<u32>(w.lo));
    u64 const p1 = mul_wide(k, static_cast<u32>(w.lo >> 32)) + (p0 >> 32);
    u64 const p2 = fp64::mul_lo(k, w.hi) + (p1 >> 32);
    return make128(p2, (p1 << 32) | static_cast<u32>(p0));
}

#if defined(GBX_LIBM_RECORD)
//! What round_result() was last given (host tests)
struct Rounded
{
    u128 v;
    int e;
    int bits;
};
inline Rounded last_rounded{};
#endif

//! v 2^-127 times 2^e, v in [2^127, 2^128), with its sign, rounded to a double;
//! false when an error of 2^-Bits times 2^127 in v could change the rounding
template<int Bits>
GBX_FORCEINLINE bool round_result(u128 v, int e, u64 sign, u64* y)
{
#if defined(GBX_LIBM_RECORD)
    last_rounded = {v, e, Bits};
#endif
    u64 const hi = static_cast<u64>(v >> 64);
    // The 32 bits below the 53-bit significand (half: 2^31), the error in them
    u32 const rest = static_cast<u32>((hi & 0x7ffu) << 21)
                     | static_cast<u32>(static_cast<u64>(v) >> 43);
    constexpr u32 error = 1u << (84 - Bits);
    *y = sign + (u64(e + 1022) << 52) + ((hi >> 11) + (rest >> 31));
    return rest - (0x80000000u - error) >= 2 * error;
}

//! q of log1p(z) = z - z q, times 2^69, for z times 2^70, |z| <= 2^-7:
//! q = z (1/2 - z (1/3 - z (1/4 - ...)))
GBX_FORCEINLINE i64 log1p_series(i64 z)
{
    i32 const zs = static_cast<i32>(z >> 32);  // times 2^38
    constexpr double p32 = 4294967296.0;
    constexpr i32 c10 = static_cast<i32>(p32 / 10), c9 = static_cast<i32>(p32 / 9),
                  c8 = static_cast<i32>(p32 / 8), c7 = static_cast<i32>(p32 / 7),
                  c6 = static_cast<i32>(2 * p32 / 6);
    i32 t = c9 - (fp64::mul_hi_s(zs, c10) >> 6);  // times 2^32
    t = c8 - (fp64::mul_hi_s(zs, t) >> 6);
    t = c7 - (fp64::mul_hi_s(zs, t) >> 6);
    t = c6 - (fp64::mul_hi_s(zs, t) >> 5);  // times 2^33
    // From here times 2^63. zs is up to 2^-38 below z, which raises w by up to 2^25 / 6;
    // the last product of the series lowers it by up to 2^-69, which is 2^22 in w at
    // |z| = 2^-7. Half of each is taken off here, so that the errors near there, the
    // largest, are on both sides: 0.65 of the error allowed instead of 0.90 (and a
    // wider one costs 100 electrons of 1 GeV in the calorimeter 2%: more arguments are left
    // to the double-doubles).
    constexpr i64 one = 0x7fffffffffffffffll;
    constexpr i64 center = (1ll << 24) / 6 + (1ll << 21);
    i64 w = one / 5 - center - ((static_cast<i64>(zs) * t) >> 8);
    w = one / 4 - (mulhi(z, w) >> 6);
    w = one / 3 - (mulhi(z, w) >> 6);
    w = one / 2 - (mulhi(z, w) >> 6);
    return mulhi(z, w);
}

//! z - z q, z = zn 2^-k with 2^61 <= |zn| < 2^62, q times 2^69
GBX_FORCEINLINE bool round_log1p(i64 zn, int k, i64 q, u64* y)
{
    u128 v = make128(static_cast<u64>(zn), 0)
             - static_cast<u128>((static_cast<__int128>(zn) * q) >> 5);
    u64 const sign = static_cast<u64>(zn) & 0x8000000000000000ull;
    if (sign)
        v = -v;
    int const lz = count_leading_zeros(static_cast<u64>(v >> 64));
    return round_result<66>(shift_left(v, lz), 63 - k - lz, sign, y);
}

//! log(m 2^(e - 59)), m in [2^59, 2^60)
GBX_FORCEINLINE bool log_normalized(u64 m, i32 e, u64* y)
{
    u32 const j = static_cast<u32>(m >> 52) & 127u;
    e += (j >= 53 ? 1 : 0);
    u64 const th = GBX_LIBM_ILOAD(ilog_table, 3 * j);
    u64 const tl = GBX_LIBM_ILOAD(ilog_table, 3 * j + 1);
    u32 const c = static_cast<u32>(GBX_LIBM_ILOAD(ilog_table, 3 * j + 2));
    // z = m C_j - 1 (times 2^69, exact: the 1 is a multiple of 2^64)
    i64 const zi = static_cast<i64>(fp64::mul_lo(c, m));
    i64 const q = log1p_series(zi << 1);
    if (e == 0 && (j == 0 || j == 127))
    {
        // Near 1: the result is log1p(z), to its relative precision
        if (zi == 0)
            return false;
        int const s = count_leading_zeros(static_cast<u64>(zi < 0 ? -zi : zi)) - 2;
        return round_log1p(zi << s, 69 + s, q, y);
    }
    // e ln 2 - log(C_j) + z - z q times 2^117
    u128 const el = mul_u32(static_cast<u32>(e < 0 ? -e : e), ln2_q117);
    u128 v = (e < 0 ? -el : el) + make128(th, tl)
             + static_cast<u128>(static_cast<__int128>(zi) << 48)
             - static_cast<u128>((static_cast<__int128>(zi) * q) >> 21);
    u64 const sign = static_cast<u64>(v >> 64) & 0x8000000000000000ull;
    if (sign)
        v = -v;
    int const lz = count_leading_zeros(static_cast<u64>(v >> 64));
    return round_result<66>(shift_left(v, lz), 10 - lz, sign, y);
}

//! log(x) for x positive, normal and not 1
GBX_FORCEINLINE bool log(u64 x, u64* y)
{
    u32 const xh = static_cast<u32>(x >> 32);
    if (xh - 0x00100000u >= 0x7fe00000u)
        return false;
    return log_normalized(((x & fp64::mantissa_mask) | fp64::hidden_bit) << 7,
                          static_cast<i32>(xh >> 20) - 1023,
                          y);
}

//! log(1 + x) for 2^-54 <= |x| < 2^-7 and -1 < x <= -2^-7
GBX_FORCEINLINE bool log1p(u64 x, u64* y)
{
    u32 const xh = static_cast<u32>(x >> 32) & 0x7fffffffu;
    bool const negative = static_cast<i64>(x) < 0;
    if (xh - 0x3c900000u >= (negative ? 0x3ff00000u : 0x3f800000u) - 0x3c900000u)
        return false;
    i64 const m = static_cast<i64>((x & fp64::mantissa_mask) | fp64::hidden_bit);
    int const e = static_cast<int>(xh >> 20) - 1023;
    if (xh < 0x3f800000u)
    {
        // z = x: times 2^70 truncated for the series, exact in the sum
        i64 const zn = negative ? -m : m;
        int const s = e + 18;  // -36 .. 10
        i64 const z = s >= 0 ? zn << s : zn >> -s;
        return round_log1p(zn << 9, 61 - e, log1p_series(z), y);
    }
    // 1 + x in (0, 1 - 2^-7], exact times 2^59
    u64 const u = (1ull << 59) - (static_cast<u64>(m) << (e + 7));
    int const lz = count_leading_zeros(u) - 4;
    return log_normalized(u << lz, -lz, y);
}

//! exp(x) - 1 for 2^-54 <= |x| < 0.35
GBX_FORCEINLINE bool expm1(u64 x, u64* y)
{
    u32 const xh = static_cast<u32>(x >> 32) & 0x7fffffffu;
    // The leading words of 2^-54 and of 0.35
    if (xh - 0x3c900000u >= 0x3fd66666u - 0x3c900000u)
        return false;
    i64 const m = static_cast<i64>((x & fp64::mantissa_mask) | fp64::hidden_bit);
    i64 const xn = static_cast<i64>(x) < 0 ? -m : m;
    int const e = static_cast<int>(xh >> 20) - 1023;
    int const s = e + 12;  // -42 .. 10
    i64 const z = s >= 0 ? xn << s : xn >> -s;  // x times 2^64
    i32 const zs = static_cast<i32>(z >> 32);
    // expm1(x) = x + x v, v = x / 2 + x^2 (1/3! + x (1/4! + ...))
    constexpr i32 a[] = {GBX_LIBM_EXPM1_32};  // times 2^52
    constexpr i64 b[] = {GBX_LIBM_EXPM1_64};  // times 2^65
    i32 t = a[0];
    t = a[1] + fp64::mul_hi_s(zs, t);
    t = a[2] + fp64::mul_hi_s(zs, t);
    t = a[3] + fp64::mul_hi_s(zs, t);
    t = a[4] + fp64::mul_hi_s(zs, t);
    t = a[5] + fp64::mul_hi_s(zs, t);
    t = a[6] + fp64::mul_hi_s(zs, t);
    i64 w = b[0] + ((static_cast<i64>(zs) * t) >> 19);
    w = b[1] + mulhi(z, w);
    w = b[2] + mulhi(z, w);
    w = b[3] + mulhi(z, w);
    w = b[4] + mulhi(z, w);
    w = b[5] + mulhi(z, w);
    w = b[6] + mulhi(z, w);
    i64 const v1 = z + mulhi(mulhi(z, z), w);  // v times 2^65
    i64 const zn = xn << 9;
    u128 v = make128(static_cast<u64>(zn), 0)
             + static_cast<u128>((static_cast<__int128>(zn) * v1) >> 1);
    u64 const sign = static_cast<u64>(zn) & 0x8000000000000000ull;
    if (sign)
        v = -v;
    int const lz = count_leading_zeros(static_cast<u64>(v >> 64));
    return round_result<62>(shift_left(v, lz), 2 + e - lz, sign, y);
}

//! exp(x) for 2^-54 <= |x| < 708.375 (normal results)
GBX_FORCEINLINE bool exp(u64 x, u64* y)
{
    u32 const xh = static_cast<u32>(x >> 32) & 0x7fffffffu;
    // The leading words of 2^-54 and of 708.375
    if (xh - 0x3c900000u >= 0x40862300u - 0x3c900000u)
        return false;
    bool const negative = static_cast<i64>(x) < 0;
    u64 const m = (x & fp64::mantissa_mask) | fp64::hidden_bit;
    // |x| times 2^96
    int const s = static_cast<int>(xh >> 20) - 1023 + 44;
    u128 const f = s >= 0 ? shift_left(m, s) : u128(m >> -s);
    // k = 128 |x| / ln 2 to the nearest integer (or next to it at a tie);
    // 128 / ln 2 times 2^24
    u32 const k = (fp64::mul_hi(static_cast<u32>(f >> 76), 3098164009u) + 2048u) >> 12;
    i64 r = static_cast<i64>(static_cast<u64>((f - mul_u32(k, ln2_n_q96)) >> 25));  // times 2^71
    i32 n = static_cast<i32>(k);
    if (negative)
    {
        r = -r;
        n = -n;
    }
    // exp(r) - 1 = r + r^2 (1/2 + r (1/6 + r (1/24 + ...)))
    i32 const rs = static_cast<i32>(r >> 32);  // times 2^39
    constexpr double p32 = 4294967296.0;
    constexpr i32 c7 = static_cast<i32>(p32 / 5040), c6 = static_cast<i32>(p32 / 720),
                  c5 = static_cast<i32>(p32 / 120), c4 = static_cast<i32>(8 * p32 / 24);
    i32 t = c6 + (fp64::mul_hi_s(rs, c7) >> 7);  // times 2^32
    t = c5 + (fp64::mul_hi_s(rs, t) >> 7);
    t = c4 + (fp64::mul_hi_s(rs, t) >> 4);  // times 2^35
    // From here times 2^63
    constexpr i64 one = 0x7fffffffffffffffll;
    i64 w = one / 6 + (mulhi(r, static_cast<i64>(t) << 28) >> 7);
    w = one / 2 + (mulhi(r, w) >> 7);
    i64 const r2 = mulhi(r, r);  // times 2^78
    i64 const em1 = r + (mulhi(r2, w) >> 6);  // times 2^71
    u32 const j = static_cast<u32>(n) & 127u;
    u64 const th = GBX_LIBM_ILOAD(iexp_table, 2 * j);
    u64 const tl = GBX_LIBM_ILOAD(iexp_table, 2 * j + 1);
    // 2^(j/128) exp(r) times 2^126
    u128 const v = make128(th, tl)
                   + static_cast<u128>((static_cast<__int128>(static_cast<i64>(th)) * em1) >> 7);
    int const lz = count_leading_zeros(static_cast<u64>(v >> 64));
    return round_result<66>(shift_left(v, lz), (n >> 7) + 1 - lz, 0, y);
}

//! sin (offset 0) or cos (offset 1) of x for 2^-26 <= |x| < 2^10
GBX_FORCEINLINE bool sin_cos(u64 x, int offset, u64* y)
{
    u32 const xh = static_cast<u32>(x >> 32) & 0x7fffffffu;
    if (xh - 0x3e500000u >= 0x40900000u - 0x3e500000u)
        return false;
    u64 const m = (x & fp64::mantissa_mask) | fp64::hidden_bit;
    // |x| times 2^117, exact
    int const s = static_cast<int>(xh >> 20) - 1023 + 65;
    u128 const f = s >= 64 ? make128(m << (s - 64), 0) : shift_left(m, s);
    // k = 2 |x| / pi to the nearest integer (or next to it at a tie);
    // 2 / pi times 2^32
    u32 const k = static_cast<u32>(
        (fp64::mul_wide(static_cast<u32>(f >> 96), 2734261102u) + (1ull << 52)) >> 53);
    u128 r = f - mul_u32(k, pio2_q117);
    bool const r_negative = static_cast<i64>(static_cast<u64>(r >> 64)) < 0;
    if (r_negative)
        r = -r;
    u32 const quadrant = (k + static_cast<u32>(offset)) & 3u;
    bool const sine = (quadrant & 1u) == 0;
    // Quadrants 2 and 3 change the sign; a sine is odd in r, sin(x) in x
    bool const x_negative = offset == 0 && static_cast<i64>(x) < 0;
    u64 const sign = u64(((quadrant & 2u) != 0) ^ (sine && r_negative) ^ x_negative) << 63;
    // |r| <= pi/4 (plus the rounding of k) times 2^64, and r^2 times 2^128
    u64 const rh = static_cast<u64>(r >> 53);
    u32 const rl = static_cast<u32>(static_cast<u64>(r) >> 21);  // next 32 bits
    u128 const rsq = u128(rh) * rh
                     + (u128(fp64::mul_wide(static_cast<u32>(rh >> 32), rl)) << 1);
    u64 const u = static_cast<u64>((rsq + (u128(1) << 63)) >> 64);
    u32 const us = static_cast<u32>(u >> 32);
    u128 v;
    int top;
    if (sine)
    {
        // sin(r) = r - r u (1/3! - u (1/5! - ...))
        constexpr u32 a[] = {GBX_LIBM_SIN_32};  // times 2^64
        constexpr u64 b[] = {GBX_LIBM_SIN_64};  // times 2^70
        u32 t = a[1] - fp64::mul_hi(us, a[0]);
        t = a[2] - fp64::mul_hi(us, t);
        t = a[3] - fp64::mul_hi(us, t);
        u64 w = b[0] - (fp64::mul_wide(us, t) >> 26);
        w = b[1] - mulhi_u(u, w);
        w = b[2] - mulhi_u(u, w);
        w = b[3] - mulhi_u(u, w);
        // 1 - sin(r) / r times 2^67; 1/6 times 2^66
        u64 const d = static_cast<u64>((u128(u) * 12297829382473034411ull) >> 63)
                      - (mulhi_u(u, mulhi_u(u, w)) >> 3);
        int const lz = count_leading_zeros(static_cast<u64>(r >> 64));
        if (lz > 50)
            return false;  // below 2^-40: too few bits of r
        v = shift_left(r, lz);
        v -= (u128(static_cast<u64>(v >> 64)) * d) >> 3;
        top = 10 - lz;
    }
    else
    {
        // cos(r) = 1 - u / 2 + u^2 (1/4! - u (1/6! - ...))
        constexpr u32 a[] = {GBX_LIBM_COS_32};  // times 2^64
        constexpr u64 b[] = {GBX_LIBM_COS_64};  // times 2^68
        u32 t = a[1] - fp64::mul_hi(us, a[0]);
        t = a[2] - fp64::mul_hi(us, t);
        t = a[3] - fp64::mul_hi(us, t);
        u64 w = b[0] - (fp64::mul_wide(us, t) >> 28);
        w = b[1] - mulhi_u(u, w);
        w = b[2] - mulhi_u(u, w);
        w = b[3] - mulhi_u(u, w);
        w = b[4] - mulhi_u(u, w);
        w = mulhi_u(mulhi_u(u, u), w);  // times 2^68
        v = make128(1ull << 63, 0) - (rsq >> 2) + (u128(w) << 59);
        top = 0;
    }
    int const lz = count_leading_zeros(static_cast<u64>(v >> 64));
    return round_result<64>(shift_left(v, lz), top - lz, sign, y);
}
}  // namespace fixed
}  // namespace libm
}  // namespace gbx
