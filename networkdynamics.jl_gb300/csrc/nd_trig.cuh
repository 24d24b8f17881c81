// FP64 sine and cosine of phase differences in integer arithmetic.
//
// GB300 retires 2 FP64 lanes per clock and SM, 1/64 of its FP32 / integer rate, and a sine
// through the FP64 pipe is some fifteen dependent operations on it: the edges of Kuramoto,
// swing and power-grid networks, their Jacobians and the ensembles spent most of their time
// there.  The version below uses 32-bit integer multiplies and adds only.  Measured on the
// whole GPU (2.5 million threads, arguments in [-π, π]): 142 G sines/s against 28 G/s for the
// library's, 148 against 28 for the cosine; both are bound by their pipe.
//
// Method (fixed point, from the Taylor series; no table):
//   |x| as an integer multiple X of 2^-95 (exact for 2^-27 <= |x| < 2^17);
//   r = X - n π/2 with n even and nearest for the sine, n odd for the cosine
//     (cos x = ± sin(x - n π/2)), so |r| <= π/2 up to 2^-13 and the result is ± sin r;
//   w = r² / 4 and V = sin(r) / r = 1 - w (c1 - w (c2 - ...)), c_k = 4^k / (2k + 1)!, in
//     units of 2^-64 (k <= 11: the first omitted term is below 2^-67);
//   the leading 64 bits of r times V, rounded once to 53 bits.
// Errors: V within a few units of 2^-64 of values in [0.63, 1], r within n 2^-96, and r is
// used only where that is below 2^-61 of it, so the result is within 0.51 ulp of the exact
// one (the tests hold 0.51; the library's sine has up to 1 ulp).  Arguments of 2^17 and
// beyond, infinities, NaN and reduced arguments too close to zero for their error (one in
// about 10^5) go to the library function; so do the products with a factor of 0, below 2^-959, of
// 2^960 and beyond, or not finite (a line of weight 0 costs a library sine), whose exponents the
// product in one rounding does not cover.  Both functions are exactly odd / even.
//
// The header compiles as CUDA (device) and as plain C++ (host, for the CPU self-test), with
// the same bits on both for every argument that does not go to the library function.
#pragma once

#include <math.h>
#include <stdint.h>

#include "nd_exact.cuh"

namespace nd {
namespace trig {

using exact::mulhi32;
using exact::mulhi64;
using exact::clz32;

ND_SLOW double sin_library(double x) { return ::sin(x); }
ND_SLOW double cos_library(double x) { return ::cos(x); }
ND_HD double times(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
template <bool kCos, bool kTimes>
ND_HD double library(double x, double f) {
    const double y = kCos ? cos_library(x) : sin_library(x);
    return kTimes ? times(f, y) : y;
}

// f · sin x (kCos = false) or f · cos x (kCos = true); with kTimes = false f is not used (1).
// The product is rounded once, from the 64-bit significand of the sine.
template <bool kCos, bool kTimes>
ND_HD double sincos_fixed(double x, double f) {
    constexpr uint32_t P2 = 0xc90fdaa2u, P1 = 0x2168c234u, P0 = 0xc4c6628cu;  // π/2 · 2^95
    const uint64_t b = exact::to_bits(x);
    const int e = (int)(b >> 52) & 0x7ff;
    const uint64_t fb = exact::to_bits(f);
    const int fe = (int)(fb >> 52) & 0x7ff;
    // x - x³/6 rounds to x, 1 - x²/2 to 1; a factor near the ends of the exponent range takes
    // the plain product
    if (e < 1023 - 27) return kTimes ? times(f, kCos ? 1.0 : x) : (kCos ? 1.0 : x);
    if (e >= 1023 + 17 || (kTimes && (unsigned)(fe - 64) >= 0x7ffu - 128)) return library<kCos, kTimes>(x, f);
    // X = |x| · 2^95 = m · 2^s, 16 <= s <= 59, in two 64-bit words
    const uint64_t m = (b & exact::kFrac) | exact::kHidden;
    const int s = e - 980;
    const uint64_t Xl = m << s, Xh = m >> (64 - s);
    // n: t = floor(|x| · 2^14), round(|x| / π) or floor(|x| / π) up to 2^-13
    const uint32_t t = mulhi32((uint32_t)(Xh >> 17), 0x517cc1b7u);  // 2^32 / π
    const uint32_t k = kCos ? t >> 14 : (t + (1u << 13)) >> 14;
    const uint32_t n = kCos ? 2 * k + 1 : 2 * k;
    // r = X - n · π/2 (two's complement, 128 bits)
    const uint64_t q0 = (uint64_t)n * P0;
    const uint64_t q1 = (uint64_t)n * P1 + (q0 >> 32);
    const uint64_t q2 = (uint64_t)n * P2 + (q1 >> 32);
    const uint64_t ql = (q1 << 32) | (uint32_t)q0;
    uint64_t rl = Xl - ql, rh = Xh - q2 - (Xl < ql);
    const bool neg = (int64_t)rh < 0;
    if (neg) {
        rh = ~rh + (rl == 0);
        rl = 0 - rl;
    }
    // |r| < 2 in 96 bits: r2 r1 r0
    const uint32_t r2 = (uint32_t)rh, r1 = (uint32_t)(rl >> 32), r0 = (uint32_t)rl;
    if (r2 < (1u << 13) && n != 0) return library<kCos, kTimes>(x, f);
    // w = r² / 4 and V = sin(r) / r, units of 2^-64
    const uint64_t r = ((uint64_t)r2 << 32) | r1;
    const uint64_t w = mulhi64(r, r);
    const uint32_t wh = (uint32_t)(w >> 32);
    uint32_t h = 0x5c6e4u - mulhi32(0xbb1u, wh);
    h = 0x25e9369u - mulhi32(h, wh);
    h = 0xca963b82u - mulhi32(h, wh);
    uint64_t a = 0x35cfe7ce67ull - mulhi32(h, wh);
    a = 0xb092309d437ull - ((uint64_t)(uint32_t)(a >> 32) * wh + mulhi32((uint32_t)a, wh));
    a = 0x1ae64567f544eull - mulhi64(a, w);
    a = 0x2e3bc74aad8e67ull - mulhi64(a, w);
    a = 0x340340340340340ull - mulhi64(a, w);
    a = 0x2222222222222222ull - mulhi64(a, w);
    a = 0xaaaaaaaaaaaaaaabull - mulhi64(a, w);
    const uint64_t V = ~mulhi64(a, w);
    // the leading 64 bits of r (r2 >= 2^4 here), times V, rounded to 53 bits
    const int lz = clz32(r2);
    const uint64_t M = (r << lz) | (((uint64_t)r0 << lz) >> 32);
    uint64_t p = mulhi64(M, V);
    int sh = (int)(~p >> 63);
    p <<= sh;
    int ex = 1022 - lz - sh;
    if (kTimes) {  // p · 2^-64 in [1/2, 1) times the factor's significand in [1/2, 1)
        p = mulhi64(p, ((fb & exact::kFrac) | exact::kHidden) << 11);
        sh = (int)(~p >> 63);
        p <<= sh;
        ex += fe - 1022 - sh;
    }
    const uint64_t mag = ((uint64_t)ex << 52) + (p >> 11) + ((p >> 10) & 1);
    // sin(x) = sign(x) (-1)^k sin(r);  cos(x) = -(-1)^k sin(r)
    const uint64_t sign = ((uint64_t)((k & 1) ^ (uint32_t)neg ^ (uint32_t)kCos) << 63) ^
                          (kCos ? 0 : b & exact::kSign) ^ (kTimes ? fb & exact::kSign : 0);
    return exact::from_bits(mag | sign);
}

ND_HD double sin(double x) { return sincos_fixed<false, false>(x, 1.0); }
ND_HD double cos(double x) { return sincos_fixed<true, false>(x, 1.0); }
// f sin x and f cos x, rounded once: one FP64 operation less, and within 0.51 ulp of the exact
// product (a rounded sine times f can be a whole ulp off)
ND_HD double times_sin(double f, double x) { return sincos_fixed<false, true>(x, f); }
ND_HD double times_cos(double f, double x) { return sincos_fixed<true, true>(x, f); }

}  // namespace trig
}  // namespace nd
