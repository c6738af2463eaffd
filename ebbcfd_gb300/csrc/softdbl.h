// softdbl.h -- IEEE double products, quotients and square roots on the integer pipe.
//
// GB300 issues one FP64 instruction per warp every 64 cycles of a scheduler, and a
// plain FP64 stage kernel kept that pipe ~85% busy while 90% of the issue slots stayed
// empty.  These functions return the correctly rounded (to nearest, ties to even) IEEE
// result bit for bit from 32-bit integer instructions, so part of a kernel's FP64
// operations can run beside the FP64 pipe.  Measured on GB300 (16 warps per SM), per warp
// operation of an SM: a product 6.3 ns against 9.6 ns on the FP64 pipe, and 4.8 ns when
// every second product is taken here; a quotient 11 ns against 71 ns (CUDA's division), a
// square root 16 ns against 72 ns.
//
//   product     the 106-bit product of the significands in four 32x32-bit products,
//               its leading 53 bits rounded by a carry from the discarded ones;
//   reciprocal  an FP32 seed y0 of 1/b refined once in fixed point with the exact
//               residual 1 - b y0 (its low 64 bits are all of it): never above 1/b,
//               relative error below 2^-42;
//   quotient    Q = a y truncated, at most a few hundred units in the last place below
//               a/b; the remainder a - b Q is exact in 64 bits (it is small, so the low
//               64 bits of both terms are all of it); remainder * y gives the whole
//               units missing, and what remains is compared with half a divisor (a
//               quotient never is a half exactly);
//   square root the same scheme from an FP32 seed of 1/sqrt(x): one Heron step, the
//               exact remainder x - S^2, and its quotient by 2 S.
// The remainder-corrected rounding is the principle of P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1),
// 1990, carried out on integers.
//
// Every function is branch-free and takes normal numbers and zeros only, results
// included; the caller sees to that with `check` and `divisor_ok` on its inputs, which
// (like `root` itself) record in `bad` -- never cleared -- that it has to evaluate with
// the plain operators instead.  Plain C++ on the
// host, where tests compare every function with the IEEE operators.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define EBB_SOFT_HD __host__ __device__ __forceinline__
#else
#define EBB_SOFT_HD inline
#endif
// the host's seeds (a host test puts the device's errors in their place)
#ifndef EBB_HOST_RCP
#define EBB_HOST_RCP(x) (1.0f / (x))
#define EBB_HOST_RSQRT(x) (1.0f / sqrtf(x))
#endif

namespace ebbsoft {

EBB_SOFT_HD uint32_t hi_of(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return (uint32_t)(u >> 32);
#endif
}
EBB_SOFT_HD uint32_t lo_of(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return (uint32_t)u;
#endif
}
EBB_SOFT_HD double make(uint32_t hi, uint32_t lo)
{
#if defined(__CUDA_ARCH__)
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t u = ((uint64_t)hi << 32) | lo;
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
EBB_SOFT_HD float as_float(uint32_t u)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}
EBB_SOFT_HD uint32_t as_bits(float f)
{
#if defined(__CUDA_ARCH__)
    return __float_as_uint(f);
#else
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
#endif
}
// the high word of (hi:lo) << s, 0 <= s < 32
EBB_SOFT_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s)
{
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, s);
#else
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << s) >> 32);
#endif
}
// the low word of (hi:lo) >> s, 0 <= s < 32
EBB_SOFT_HD uint32_t shr_lo(uint32_t lo, uint32_t hi, uint32_t s)
{
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, s);
#else
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> s);
#endif
}
EBB_SOFT_HD uint32_t mul_hi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// FP32 seeds of 1/x and 1/sqrt(x); relative error below 2^-22.9 (the device's
// approximate instructions), on the host correctly rounded operations
EBB_SOFT_HD float rcp_seed(float x)
{
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return EBB_HOST_RCP(x);
#endif
}
EBB_SOFT_HD float rsqrt_seed(float x)
{
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return EBB_HOST_RSQRT(x);
#endif
}
// significand of a seed in (0.5, 1) as an integer of 24 bits (1 taken as 1 - 2^-24).  The
// error of a seed of a value within 2^-24 of 0.5 may take it below: 0.5 is as near.
EBB_SOFT_HD uint32_t seed_bits(float y)
{
    const float c = fminf(fmaxf(y, 0.5f), 0.99999994f);
    return (as_bits(c) & 0x7fffffu) | 0x800000u;
}

constexpr uint32_t kExp = 0x7ff00000u;

// Records in `bad` a value that is neither zero nor within 2^-R <= |x| < 2^R
template <int R> EBB_SOFT_HD void check(double x, bool &bad)
{
    const uint32_t m = hi_of(x) & 0x7fffffffu;
    bad |= (m - ((1023u - R) << 20) >= ((2u * R) << 20)) && ((m | lo_of(x)) != 0u);
}

constexpr uint32_t kTop = 0xfff00000u;  // sign and exponent

// a 2 for a normal a
EBB_SOFT_HD double twice(double a) { return make(hi_of(a) + 0x100000u, lo_of(a)); }

// RN(a b) for a and b zero or normal whose product is zero or normal; NZ: a is not zero
template <bool NZ = false> EBB_SOFT_HD double mul(double a, double b)
{
    const uint32_t ah = hi_of(a), al = lo_of(a), bh = hi_of(b), bl = lo_of(b);
    const uint32_t Ah = (ah & 0xfffffu) | 0x100000u, Bh = (bh & 0xfffffu) | 0x100000u;
    // the 106-bit product of the significands, w3:w2:w1:w0 (the middle terms fit 64 bits)
    const uint64_t t = (uint64_t)al * bl;
    uint64_t m = (uint64_t)Ah * bl + (uint32_t)(t >> 32);
    m = (uint64_t)al * Bh + m;
    const uint64_t top = (uint64_t)Ah * Bh + (uint32_t)(m >> 32);
    const uint32_t w0 = (uint32_t)t, w1 = (uint32_t)m, w2 = (uint32_t)top, w3 = (uint32_t)(top >> 32);
    // its leading 53 bits in h:l, the rest in r:w0; signs add modulo 2
    const uint32_t n = 12u - (w3 >> 9);
    const uint32_t l = shl_hi(w1, w2, n), r = w1 << n;
    const uint32_t h = shl_hi(w2, w3, n) + (ah & kTop) + (bh & kTop) - ((1012u + n) << 20);
    // to nearest, ties to even: r is a multiple of 2^11, so r:w0 plus (half - 1, or half
    // when l is odd) carries out exactly when it rounds up
    const uint32_t half = 0x7fffffffu + (l & 1u);
    uint32_t lo, hi;
#if defined(__CUDA_ARCH__)
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, 0xffffffff;\n\taddc.cc.u32 t, %3, %4;\n\t"
        "addc.cc.u32 %0, %5, 0;\n\taddc.u32 %1, %6, 0;\n\t}"
        : "=r"(lo), "=r"(hi)
        : "r"(w0), "r"(r), "r"(half), "r"(l), "r"(h));
#else
    const uint64_t v = (((uint64_t)h << 32) | l) + (((uint64_t)r + half + (w0 != 0u)) >> 32);
    lo = (uint32_t)v;
    hi = (uint32_t)(v >> 32);
#endif
    const bool zero = (!NZ && (ah & kExp) == 0u) || (bh & kExp) == 0u;
    return make(zero ? (ah ^ bh) & 0x80000000u : hi, zero ? 0u : lo);
}

// a divisor's reciprocal: Y (scaled by 2^63, significand in [1, 2)) <= 1/b
struct Recip {
    uint32_t bh, bl;  // the divisor's bits
    uint32_t Yh, Yl;
};

// divisors 2^-125 <= |b| < 2^126
EBB_SOFT_HD bool divisor_ok(double b) { return (hi_of(b) & 0x7fffffffu) - (898u << 20) < (251u << 20); }

EBB_SOFT_HD Recip recip(double b)
{
    Recip R;
    R.bh = hi_of(b);
    R.bl = lo_of(b);
    const uint32_t Bh = (R.bh & 0xfffffu) | 0x100000u;
    const uint32_t y = seed_bits(rcp_seed(as_float(0x3f800000u | ((R.bh & 0xfffffu) << 3) | (R.bl >> 29))));
    // T = 2^76 - B y, exactly: |T| < 2^55, so its low 64 bits are the product's, negated
    const uint64_t P = (uint64_t)R.bl * y + ((uint64_t)(Bh * y) << 32);
    const int64_t T = (int64_t)(0ull - P);
    const uint64_t Y = ((uint64_t)y << 39) + (uint64_t)(((int64_t)(int32_t)(T >> 24) * (int32_t)y) >> 13);
    R.Yh = (uint32_t)(Y >> 32);
    R.Yl = (uint32_t)Y;
    return R;
}

// RN(a / b) for a zero or normal, the reciprocal of an ok b, and a zero or normal quotient
EBB_SOFT_HD double div(double a, const Recip &R)
{
    const uint32_t ah = hi_of(a), al = lo_of(a);
    const uint32_t Ah = (ah & 0xfffffu) | 0x100000u, Bh = (R.bh & 0xfffffu) | 0x100000u;
    const uint32_t s = Ah < Bh || (Ah == Bh && al < R.bl) ? 1u : 0u;  // quotient of the significands below 1
    const uint64_t Q0 = (uint64_t)Ah * R.Yh + mul_hi(Ah, R.Yl) + mul_hi(al, R.Yh);  // scaled by 2^51
    const uint64_t Q = Q0 << (1u + s);
    const uint32_t qh = (uint32_t)(Q >> 32), ql = (uint32_t)Q;
    // remainder A 2^(52+s) - B Q >= 0, its low (and only) 64 bits
    const uint64_t p = (uint64_t)R.bl * ql;
    const uint32_t ph = (uint32_t)(p >> 32) + R.bl * qh + Bh * ql;
    const uint64_t rem = ((uint64_t)(al << (20u + s)) << 32) - (((uint64_t)ph << 32) | (uint32_t)p);
    // whole units missing (one fewer when within 2^-17 of the next), and the remainder
    // they leave: below B, or up to 2^-17 B above it; one unit more when over B / 2
    const uint32_t j = mul_hi((uint32_t)(rem >> 32), R.Yh) >> 19;
    const uint64_t left = rem - ((uint64_t)j * R.bl + ((uint64_t)(j * Bh) << 32));
    const uint32_t up = 2ull * left > (((uint64_t)Bh << 32) | R.bl) ? 1u : 0u;
    const uint64_t N = Q + (j + up);
    const uint32_t h = (uint32_t)(N >> 32) + (ah & kTop) - (R.bh & kTop) + ((1022u - s) << 20);
    const bool zero = (ah & kExp) == 0u;
    return make(zero ? (ah ^ R.bh) & 0x80000000u : h, zero ? 0u : (uint32_t)N);
}

// RN(sqrt(x)) for x zero (the result is +0) or 2^-400 <= x < 2^400
EBB_SOFT_HD double root(double x, bool &bad)
{
    const uint32_t xh = hi_of(x), xl = lo_of(x);
    bad |= (xh - (623u << 20) >= (800u << 20)) && ((xh | xl) != 0u);
    const uint32_t odd = ((xh >> 20) & 1u) ^ 1u;  // biased exponent even: true exponent odd
    const uint32_t m = xh & 0xfffffu;
    // X = significand in [1, 4) scaled by 2^52
    const uint32_t Xh = shl_hi(xl, m | 0x100000u, odd), Xl = xl << odd;
    const uint32_t y = seed_bits(rsqrt_seed(as_float(((127u + odd) << 23) | (m << 3) | (xl >> 29))));
    // Heron from s0 = X y (scaled by 2^30): S = s0 + (X - s0^2) y / 2, never above the root
    const uint32_t x32 = shr_lo(Xl, Xh, 22);
    const uint64_t S0 = (uint64_t)x32 * y;
    const uint32_t s0 = shr_lo((uint32_t)S0, (uint32_t)(S0 >> 32), 24);
    const int64_t d = (int64_t)(((((uint64_t)Xh << 32) | Xl) << 8) - (uint64_t)s0 * s0);
    const int32_t s1 = (int32_t)(((int64_t)(int32_t)(d >> 10) * (int32_t)y) >> 23);  // scaled by 2^52
    const uint64_t S = ((uint64_t)s0 << 22) + (uint64_t)(int64_t)s1 - 1ull;
    // 1/S scaled by 2^31
    const int32_t u = (int32_t)(((int64_t)s1 * (int32_t)y) >> 32);
    const uint32_t Y = (y << 7) + (uint32_t)((int32_t)(((int64_t)u * (int32_t)y) >> 32) >> 5);
    // remainder X 2^52 - S^2 >= 0, its low (and only) 64 bits
    const uint32_t Sh = (uint32_t)(S >> 32), Sl = (uint32_t)S;
    const uint64_t p = (uint64_t)Sl * Sl;
    const uint32_t ph = (uint32_t)(p >> 32) + Sl * (2u * Sh);
    const uint64_t rem = ((uint64_t)(Xl << 20) << 32) - (((uint64_t)ph << 32) | (uint32_t)p);
    // whole units missing (one fewer when within 2^-18 of the next), and the remainder
    // X 2^52 - (S + j)^2 they leave; one unit more when over S + j, i.e. past the half
    const uint32_t j = mul_hi((uint32_t)(rem >> 32), Y) >> 20;
    const uint64_t W = S + j, V = S + W;
    const uint64_t left = rem - ((uint64_t)j * (uint32_t)V + ((uint64_t)(j * (uint32_t)(V >> 32)) << 32));
    const uint64_t N = W + (left > W ? 1u : 0u);
    const uint32_t e = (((xh & kExp) - (odd << 20)) >> 1) & kExp;  // the exponent field halved
    const bool zero = (xh & kExp) == 0u;
    return make(zero ? 0u : (uint32_t)(N >> 32) + e + (511u << 20), zero ? 0u : (uint32_t)N);
}

}  // namespace ebbsoft
