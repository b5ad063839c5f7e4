// bmxg_fp64.cuh -- correctly rounded FP64 square root and division in integer
// arithmetic, and FP64 comparisons on the bits.
//
// GB300 issues FP64 at 2 thread-operations per clock per SM, 1/64 of the FP32
// and integer rate, and an IEEE square root or division is a sequence of about
// ten dependent FP64 instructions.  Here they run on the integer pipe: the
// significands as 64-bit fixed point, a reciprocal (or reciprocal square root)
// from the FP32 approximation unit refined by Newton's iteration, and a last
// rounding that is exact -- where the refined value lies too close to a
// rounding boundary the remainder decides -- so every result is the IEEE
// round-to-nearest one, bit for bit.  Operands or results outside the normal
// range (zeros, subnormals, infinities, NaN) take the FP64 instructions.
//
// The refinement is the textbook one: r <- r (2 - x r) for the reciprocal,
// y <- y (3 - m y^2) / 2 for the reciprocal square root, s <- s + (m - s^2) y / 2
// for the root, each error bounded beside the code.  Neither a quotient nor a
// square root of 53-bit significands can lie exactly halfway between two
// doubles (within the normal range), so "nearest" has no tie.
//
// Measured (GB300): 500 trees of 100 segments, FP64, 10 steps and the load 3.35 ->
// 2.96 ms, FP32F, 20 steps 4.33 -> 4.05 ms; 64 colonies of 500..50 000 spheres,
// FP64, 10 steps 4.72 -> 4.40 ms (k_sphere64 1.51 -> 1.42 ms on 2.73 M spheres:
// its FP64 pipe falls from 58 to 44 % busy, and the walk's latency bounds it).
//
// Also compiled for the host (tests), where FP32 approximations of the same
// accuracy stand in for the device's.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define BMXG_HD __host__ __device__ __forceinline__
#else
#define BMXG_HD inline
#endif

namespace bmxg {

#if !defined(__CUDA_ARCH__)
// host stand-ins; a test moves the approximations to the ends of their error range
namespace host_approx {
inline int &ulps() { static int u = 0; return u; }
inline float nudge(float v)
{
    int32_t b;
    std::memcpy(&b, &v, 4);
    b += ulps();
    std::memcpy(&v, &b, 4);
    return v;
}
}  // namespace host_approx
#endif

BMXG_HD float approx_rcp(float x)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return host_approx::nudge(1.0f / x);
#endif
}

BMXG_HD float approx_rsqrt(float x)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return host_approx::nudge((float)(1.0 / std::sqrt((double)x)));
#endif
}

BMXG_HD uint64_t mulhi64(uint64_t a, uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

BMXG_HD uint64_t bits64(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}

BMXG_HD double from_bits64(uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}

BMXG_HD uint32_t bits32(float x)
{
#if defined(__CUDA_ARCH__)
    return __float_as_uint(x);
#else
    uint32_t b;
    std::memcpy(&b, &x, 4);
    return b;
#endif
}

BMXG_HD float from_bits32(uint32_t b)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float x;
    std::memcpy(&x, &b, 4);
    return x;
#endif
}

// The FP64 instructions, out of line: operands or results outside the normal
// range only.
#if defined(__CUDACC__)
static __host__ __device__ __noinline__ double div_fp64(double a, double b) { return a / b; }
static __host__ __device__ __noinline__ double sqrt_fp64(double x) { return sqrt(x); }
#else
inline double div_fp64(double a, double b) { return a / b; }
inline double sqrt_fp64(double x) { return std::sqrt(x); }
#endif

// A divisor: its sign, biased exponent, significand m in [2^52, 2^53) and
// R = 2^127 / (m 2^11), at most 8 units below the exact value and never above.
struct Divisor {
    double v;
    uint64_t m, R;
    int e;   // biased exponent; 0: outside the normal range (the FP64 division)
    uint32_t sign;
};

// A value in (2^31, 2^32] / 2^32 given as an FP32 number in (1/2, 1], as a
// 32-bit fraction lowered by 2^-20 of itself: below the exact value the number
// approximates to 2^-21 (the units' errors are below 2^-22).
BMXG_HD uint32_t lowered_fraction(float y)
{
    uint32_t u = bits32(y);
    if (u < 0x3f000000u) u = 0x3f000000u;  // (an approximation rounded below 1/2)
    const uint32_t f = (u >= 0x3f800000u) ? 0xffffffffu : ((u << 8) | 0x80000000u);
    return f - (f >> 20);
}

// One Newton step of the reciprocal R of x = m 2^11 in [2^63, 2^64) from an R
// within 2^-38 of 2^127 / x: the error term 2^63 - x R / 2^64 is below 2^26 in
// size, its truncation and the product's cost at most three units, and two
// more are subtracted so that R stays below the exact value (at most 8 below).
BMXG_HD uint64_t newton_rcp(uint64_t x, uint64_t R)
{
    const int64_t E = (int64_t)(0x8000000000000000ull - mulhi64(x, R));
    const int64_t c = (E * (int64_t)(R >> 32)) >> 31;
    const uint64_t r = R + (uint64_t)c - 4ull;
    return (r >> 62) ? r : 0xfffffffffffffff8ull;  // (x = 2^63: 2^64 wraps)
}

BMXG_HD Divisor divisor(double b)
{
    Divisor D;
    const uint64_t u = bits64(b);
    D.v = b;
    D.sign = (uint32_t)(u >> 63);
    D.e = (int)((u >> 52) & 0x7ffu);
    if (D.e == 0x7ff) D.e = 0;
    D.m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const uint64_t x = D.m << 11;
    // 1 / X for X = x / 2^63 in [1, 2): from the top 24 bits, 2^-22 (unit) +
    // 2^-23 (truncation) from the exact value, lowered by 2^-20: e in (0, 2^-19)
    const float X = from_bits32(0x3f800000u | ((uint32_t)(D.m >> 29) & 0x7fffffu));
    const uint32_t R0 = lowered_fraction(approx_rcp(X));
    // x R0 / 2^32 = 2^63 (1 - e)
    const uint64_t P = (x >> 32) * (uint64_t)R0 + (((x & 0xffffffffull) * (uint64_t)R0) >> 32);
    const uint64_t E = 0x8000000000000000ull - P;                       // 2^63 e < 2^44
    const uint64_t R1 = ((uint64_t)R0 << 32) + (((uint64_t)R0 * (E >> 13)) >> 18);  // (1 - e^2) of it, 2^-38
    D.R = newton_rcp(x, R1);
    return D;
}

// a / D, correctly rounded.
BMXG_HD double div_by(double a, const Divisor &D)
{
    const uint64_t u = bits64(a);
    const int ea = (int)((u >> 52) & 0x7ffu);
    const uint64_t ma = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const int lt = ma < D.m ? 1 : 0;             // quotient of the significands in (1/2, 1) or [1, 2)
    const int er = ea - D.e + 1023 - lt;
    // the FP64 division outside the normal range (a zero or non-finite operand,
    // a result at the ends of the exponent range)
    if (D.e == 0 || ea == 0 || ea == 0x7ff || er < 1 || er > 2045) return div_fp64(a, D.v);
    // (ma / m) 2^63 (doubled below 1), at most 9 (18) units too small
    const uint64_t q = mulhi64(ma << 11, D.R) << lt;
    // 53 bits and 11 bits below them
    uint64_t r = q >> 11;
    const uint32_t low = (uint32_t)q & 0x7ffu;
    if (low >= 1024u) {
        ++r;
    } else if (low + 18u >= 1024u) {
        // too close to halfway: up when ma 2^(52 + lt) > (r + 1/2) m; the
        // difference fits in 64 bits (it is within a few units of m / 2^10)
        const int64_t rem = (int64_t)((ma << (53 + lt)) - (2ull * r + 1ull) * D.m);
        if (rem > 0) ++r;
    }
    const uint64_t s = ((u >> 63) ^ (uint64_t)D.sign) << 63;
    return from_bits64((s | ((uint64_t)(er - 1) << 52)) + r);  // (a carry of r raises the exponent)
}

BMXG_HD double div_rn(double a, double b)
{
    return div_by(a, divisor(b));
}

// The square root of x, correctly rounded, and the divisor of the result (for
// quotients by it: its reciprocal starts from the root's own).
BMXG_HD double sqrt_rn(double x, Divisor *by = nullptr)
{
    const uint64_t u = bits64(x);
    const int eb = (int)(u >> 52);
    if (eb == 0 || eb >= 0x7ff) {  // zero, subnormal, infinite, NaN or negative
        const double s = sqrt_fp64(x);
        if (by) *by = divisor(s);
        return s;
    }
    const int odd = (eb & 1) ^ 1;  // unbiased exponent eb - 1023 odd
    const uint64_t M = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const uint64_t X = M << (10 + odd);  // m 2^62, m in [1, 4)
    // y = 1 / sqrt(m) in (1/2, 1]: from the top 24 bits, lowered: e in (0, 2^-19)
    const float mf = from_bits32((0x3f800000u + ((uint32_t)odd << 23)) | ((uint32_t)(M >> 29) & 0x7fffffu));
    const uint32_t Y0 = lowered_fraction(approx_rsqrt(mf));
    // m y^2 = 1 - d, d in (0, 2^-18): y (1 + d / 2) is within 2^-37 below
    const uint64_t D = 0x4000000000000000ull - mulhi64(X, (uint64_t)Y0 * Y0);  // 2^62 d < 2^44
    const uint64_t Y1 = ((uint64_t)Y0 << 32) + (((uint64_t)Y0 * (D >> 13)) >> 18);
    // s = m y within 2^-36 below; s + (m - s^2) y / 2 within 2^-73 and a few
    // units of 2^-62
    const uint64_t S0 = mulhi64(X, Y1);                    // s 2^62
    const uint64_t Rm = (X >> 2) - mulhi64(S0, S0);        // (m - s^2) 2^60 < 2^26
    const uint64_t S = S0 + ((Rm * (Y1 >> 32)) >> 31);
    uint64_t r = S >> 10;  // 53 bits and 10 bits below them
    const uint32_t low = (uint32_t)S & 0x3ffu;
    if (low >= 512u - 6u) {
        if (low > 512u + 6u) {
            ++r;
        } else {
            // too close to halfway: up when m 2^106 > (2 r + 1)^2
            const uint64_t h = 2ull * r + 1ull;
            const uint64_t hh = mulhi64(h, h), hl = h * h;
            const uint64_t xh = X >> 20, xl = X << 44;
            if (xh > hh || (xh == hh && xl > hl)) ++r;
        }
    }
    const int er = ((eb - 1023 - odd) >> 1) + 1023;
    const double s = from_bits64(((uint64_t)(er - 1) << 52) + r);
    if (by) {
        by->v = s;
        by->sign = 0;
        const uint32_t carry = (uint32_t)(r >> 53);  // r = 2^53: the next power of two
        by->e = er + (int)carry;
        by->m = carry ? 0x10000000000000ull : r;
        // 2^127 / (m 2^11) = 2^64 / s: y itself, within 2^-36
        by->R = newton_rcp(by->m << 11, carry ? 0xfffffffffffffff8ull : Y1);
    }
    return s;
}

// The quotient and the root in either precision (templates over the pair math).
BMXG_HD float qdiv(float a, float b) { return a / b; }
BMXG_HD double qdiv(double a, double b) { return div_rn(a, b); }
BMXG_HD float qsqrt(float x) { return sqrtf(x); }
BMXG_HD double qsqrt(double x) { return sqrt_rn(x); }

// a < b and a <= b for two doubles on their bits (a comparison is an FP64
// instruction): false with a NaN among them, zeros of either sign equal.
BMXG_HD int64_t order_key(double x)
{
    const int64_t b = (int64_t)bits64(x);
    return b < 0 ? (int64_t)(0x8000000000000000ull - (uint64_t)b) : b;
}
BMXG_HD bool is_nan_bits(double x) { return (bits64(x) & 0x7fffffffffffffffull) > 0x7ff0000000000000ull; }
BMXG_HD bool lt_bits(double a, double b) { return order_key(a) < order_key(b) && !is_nan_bits(a) && !is_nan_bits(b); }
BMXG_HD bool le_bits(double a, double b) { return order_key(a) <= order_key(b) && !is_nan_bits(a) && !is_nan_bits(b); }
// a <= b for values that are not negative (or NaN: false)
BMXG_HD bool le_nonneg(double a, double b)
{
    return bits64(a) <= bits64(b) && bits64(b) <= 0x7ff0000000000000ull;
}
// The comparisons in either precision (templates over the pair math).
BMXG_HD bool lt_q(float a, float b) { return a < b; }
BMXG_HD bool lt_q(double a, double b) { return lt_bits(a, b); }
BMXG_HD bool le_q(float a, float b) { return a <= b; }
BMXG_HD bool le_q(double a, double b) { return le_bits(a, b); }
BMXG_HD bool zero_q(float a) { return a == 0.0f; }
BMXG_HD bool zero_q(double a) { return (bits64(a) << 1) == 0; }
// x + 0.0: a negative zero becomes zero, anything else stays
BMXG_HD double plus_zero(double x) { return (bits64(x) << 1) ? x : 0.0; }

}  // namespace bmxg
