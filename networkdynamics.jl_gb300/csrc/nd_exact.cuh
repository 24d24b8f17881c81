// Exact IEEE-754 binary64 addition (round to nearest, ties to even) in integer
// arithmetic.
//
// On GB300 the FP64 pipe retires about two lanes per clock per SM (1/64 of FP32), and a
// DADD holds its sub-partition's FP64 pipe for the whole warp even with one lane active.
// The per-vertex sums of the RHS are long chains of dependent additions that must round
// exactly like the reference's sequential `aggbuf[i] += o[k]`.  Running those chains on
// the integer pipes keeps the FP64 pipe for the edge functions.
//
// Method (textbook binary floating-point addition): order the operands by magnitude,
// align the smaller significand with 8 guard bits and a sticky bit, add or subtract,
// normalise (left shifts are exact because no bit was shifted out when the exponents
// differ by at most one), round to nearest even on the guard bits, repack.  Zeros,
// subnormals and the signs of exact-zero results follow IEEE-754 round-to-nearest.
// NaN / infinity operands are handed to the hardware adder.
//
// The header compiles as CUDA (device) and as plain C++ (host, for the CPU self-test).
#pragma once

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define ND_HD __host__ __device__ __forceinline__
#else
#define ND_HD inline
#endif

namespace nd {
namespace exact {

constexpr uint64_t kSign = 0x8000000000000000ull;
constexpr uint64_t kFrac = 0x000FFFFFFFFFFFFFull;
constexpr uint64_t kHidden = 0x0010000000000000ull;
constexpr int kGuard = 8;

ND_HD uint64_t to_bits(double x) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, sizeof u);
    return u;
#endif
}

ND_HD double from_bits(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double x;
    memcpy(&x, &u, sizeof x);
    return x;
#endif
}

ND_HD int clz64(uint64_t x) {
#if defined(__CUDA_ARCH__)
    return __clzll((long long)x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}

ND_HD int clz32(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __clz((int)x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}

// Hardware addition for the rare inputs the integer path hands off (inf, nan, overflow).
// On the device it is a volatile asm statement: a plain __dadd_rn behind the branch gets
// if-converted and issued on every call (measured: two DADDs per call), which costs a
// full FP64 warp slot each time.
ND_HD double hw_add(double a, double b) {
#if defined(__CUDA_ARCH__)
    double s;
    asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(s) : "d"(a), "d"(b));
    return s;
#else
    volatile double s = a + b;
    return s;
#endif
}

// a + b rounded to nearest even, computed with integer operations.  Written with selects
// instead of branches so that the lanes of a warp stay converged; only non-finite inputs
// and overflow leave the straight-line path.
ND_HD double add_rn(double a, double b) {
    const uint64_t ia0 = to_bits(a), ib0 = to_bits(b);
    const uint64_t ma0 = ia0 & ~kSign, mb0 = ib0 & ~kSign;
    if (ma0 >= 0x7FF0000000000000ull || mb0 >= 0x7FF0000000000000ull) return hw_add(a, b);  // inf / nan
    const bool sw = ma0 < mb0;  // order so that |a| >= |b|
    const uint64_t ia = sw ? ib0 : ia0, ib = sw ? ia0 : ib0;
    const uint64_t ma = sw ? mb0 : ma0, mb = sw ? ma0 : mb0;
    int ea = (int)(ma >> 52), eb = (int)(mb >> 52);
    uint64_t fa = ((ma & kFrac) | (ea ? kHidden : 0)) << kGuard;  // < 2^61
    uint64_t fb = ((mb & kFrac) | (eb ? kHidden : 0)) << kGuard;
    ea += (ea == 0);  // subnormals share exponent 1 with the smallest normals
    eb += (eb == 0);
    // align b: shift by d with a sticky bit; d >= 63 leaves only the sticky bit (fb < 2^61)
    const int d = ea - eb < 63 ? ea - eb : 63;
    const uint64_t sticky = d ? (uint64_t)((fb << (64 - d)) != 0) : 0;
    const uint64_t fbs = (fb >> d) | sticky;
    const bool sub = ((ia ^ ib) & kSign) != 0;
    uint64_t r = sub ? fa - fbs : fa + fbs;
    int e = ea;
    const int carry = (int)(r >> (52 + kGuard + 1));  // 0 or 1
    r = (r >> carry) | (r & (uint64_t)carry);
    e += carry;
    // normalise left (exact: nothing was shifted out when a left shift is needed by more
    // than one bit); stop at the subnormal range
    int s = clz64(r) - (63 - 52 - kGuard);
    s = s < 0 ? 0 : s;
    s = s > e - 1 ? e - 1 : s;
    r <<= s;
    e -= s;
    const uint64_t half = 1ull << (kGuard - 1);
    const uint64_t g = r & ((1ull << kGuard) - 1);
    r >>= kGuard;
    r += (uint64_t)((g > half) | ((g == half) & (r & 1)));
    const int ov = (int)(r >> 53);  // rounding carried into a new binade
    r >>= ov;
    e += ov;
    if (e >= 0x7FF) return hw_add(a, b);  // overflow to infinity
    const uint64_t efield = (r >= kHidden) ? (uint64_t)e : 0;  // subnormal result keeps field 0
    uint64_t out = (ia & kSign) | (efield << 52) | (r & kFrac);
    out = (r == 0) ? 0ull : out;        // exact cancellation: +0 in round-to-nearest
    out = (ma == 0) ? (ia & ib) : out;  // both zero: -0 only for (-0) + (-0)
    return from_bits(out);
}

// ---- division ----------------------------------------------------------------------------------
ND_HD uint32_t mulhi32(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// The upper 64 bits of a · b, up to two units too small (the low partial product and the
// carries out of the middle ones are left out).
ND_HD uint64_t mulhi64(uint64_t a, uint64_t b) {
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    return (uint64_t)ah * bh + mulhi32(ah, bl) + mulhi32(al, bh);
}

#if defined(__CUDACC__)
#define ND_SLOW static __host__ __device__ __noinline__
#else
#define ND_SLOW static inline
#endif
ND_SLOW double hw_div(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __ddiv_rn(a, b);
#else
    return a / b;
#endif
}

// a / b rounded to nearest even, computed with integer operations: a 60-bit reciprocal of b's
// significand by two Newton steps from a float one, the quotient to 60 bits, and the rounded
// quotient settled by the sign of the exact remainder (a quotient of two 53-bit significands is
// never halfway between two others).  An FP64 division is some ten operations on the FP64
// pipe, 19 clocks each per warp and SM, this about 70 on the integer pipes (17 clocks).  Zeros,
// subnormals, infinities, NaN and results outside the normal range take the hardware division.
ND_HD double div_rn(double a, double b) {
    const uint64_t ia = to_bits(a), ib = to_bits(b);
    const int ea = (int)(ia >> 52) & 0x7ff, eb = (int)(ib >> 52) & 0x7ff;
    const uint64_t ma = (ia & kFrac) | kHidden, mb = (ib & kFrac) | kHidden;
    const int less = ma < mb;
    const int e = ea - eb + 1023 - less;  // exponent field of the quotient
    if ((unsigned)(ea - 1) >= 0x7feu || (unsigned)(eb - 1) >= 0x7feu || (unsigned)(e - 1) >= 0x7fdu) return hw_div(a, b);
    // R ~ 2^126 / B, B = mb · 2^11 in [2^63, 2^64): 1 / (B / 2^64) in (1, 2] in units of 2^-62
    const uint64_t B = mb << 11;
#if defined(__CUDA_ARCH__)
    const float y = __frcp_rn(__uint2float_rn((uint32_t)(B >> 32)));
#else
    const float y = 1.0f / (float)(uint32_t)(B >> 32);
#endif
    uint64_t R = (uint64_t)(uint32_t)(y * 4611686018427387904.0f) << 32;  // y · 2^62: 24 significant bits, below 2^32
    const int64_t e0 = (int64_t)((1ull << 62) - mulhi64(B, R));           // 1 - b r, below 2^-21
    const uint64_t c0 = mulhi64(R, (uint64_t)(e0 < 0 ? -e0 : e0) << 20) >> 18;
    R = e0 < 0 ? R - c0 : R + c0;
    const int32_t e1 = (int32_t)(int64_t)((1ull << 62) - mulhi64(B, R));  // below 2^-40
    R += (uint64_t)(((int64_t)e1 * (int64_t)(uint32_t)(R >> 32)) >> 30);
    // the quotient ma / mb (times 2 where it is below 1) in units of 2^-52, rounded, and its remainder
    const uint64_t Q = mulhi64(ma << 10, R);  // units of 2^-61
    const int s = 9 - less;
    uint64_t q = (Q + (1ull << (s - 1))) >> s;
    const int64_t D = (int64_t)((ma << (52 + less)) - q * mb);
    q += (uint64_t)(int64_t)((2 * D > (int64_t)mb) - (2 * D < -(int64_t)mb));
    return from_bits(((ia ^ ib) & kSign) | ((((uint64_t)e - 1) << 52) + q));
}

}  // namespace exact
}  // namespace nd
