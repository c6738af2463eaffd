// dfpair.cuh -- two double-floats (dfloat.h) side by side in the packed FP32 instructions
// of sm_100 and later: one instruction adds, multiplies or multiply-adds two FP32 pairs.
//
// The double-float flux kernel was bound by issuing and fetching instructions (FMA pipe
// 46% busy at 53% of the issue slots, a quarter of the time waiting for instructions), so
// work that comes in twos -- the two sides of a face, the two directions, two components
// -- takes half the instructions this way.  Now the FMA pipe is 68% busy at 67% of the slots.
// k_flux, with the shorter quotients and square roots of dfloat.h and the registers this
// frees (96 a thread, 20 warps per SM instead of 128 and 16): 400,000 plate cells 93 -> 54
// us, 200,000 triangles (Rusanov) 22 -> 14 us.
//
// Every operation is dfloat.h's, step by step, and gives its bits.  The assembler contracts a
// packed product whose uses all are sums with them, .rn notwithstanding (seen where a root
// ended in such a product), so no operation here leaves one: every product is also used in a
// multiply-add, but for halvings, which are exact.
#pragma once

#include "dfloat.h"

namespace ebbdev {

using ebbdf::df;
typedef unsigned long long f2;  // two FP32 numbers, the first in the low half

__device__ __forceinline__ f2 pack2(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 neg2(f2 a) { return a ^ 0x8000000080000000ull; }

struct dfp {
    f2 hi, lo;
};
__device__ __forceinline__ dfp pair(df a, df b) { return {pack2(a.hi, b.hi), pack2(a.lo, b.lo)}; }
__device__ __forceinline__ dfp both(df a) { return pair(a, a); }
__device__ __forceinline__ void split(dfp v, df &a, df &b)
{
    unpack2(v.hi, a.hi, b.hi);
    unpack2(v.lo, a.lo, b.lo);
}
__device__ __forceinline__ df first(dfp v)
{
    df a, b;
    split(v, a, b);
    return a;
}
__device__ __forceinline__ df second(dfp v)
{
    df a, b;
    split(v, a, b);
    return b;
}
__device__ __forceinline__ dfp swapped(dfp v)
{
    df a, b;
    split(v, a, b);
    return pair(b, a);
}
__device__ __forceinline__ df sum(dfp v)
{
    df a, b;
    split(v, a, b);
    return a + b;
}
__device__ __forceinline__ dfp fast_two_sum2(f2 a, f2 b)
{
    const f2 s = add2(a, b);
    return {s, sub2(b, sub2(s, a))};
}
__device__ __forceinline__ dfp two_sum2(f2 a, f2 b)
{
    const f2 s = add2(a, b), t = sub2(s, a);
    return {s, add2(sub2(a, sub2(s, t)), sub2(b, t))};
}
__device__ __forceinline__ dfp operator+(dfp a, dfp b)
{
    const dfp s = two_sum2(a.hi, b.hi);
    return fast_two_sum2(s.hi, add2(s.lo, add2(a.lo, b.lo)));
}
__device__ __forceinline__ dfp operator-(dfp a, dfp b)
{
    const f2 s = sub2(a.hi, b.hi), t = sub2(s, a.hi);
    const f2 e = sub2(sub2(a.hi, sub2(s, t)), add2(b.hi, t));
    return fast_two_sum2(s, add2(e, sub2(a.lo, b.lo)));
}
__device__ __forceinline__ dfp operator*(dfp a, dfp b)
{
    const f2 p = mul2(a.hi, b.hi);
    return {p, fma2(a.hi, b.lo, fma2(a.lo, b.hi, fma2(a.hi, b.hi, neg2(p))))};
}
__device__ __forceinline__ dfp half(dfp a)
{
    const f2 h = pack2(0.5f, 0.5f);
    return {mul2(h, a.hi), mul2(h, a.lo)};
}
__device__ __forceinline__ dfp operator/(dfp a, dfp b)
{
    float x, y;
    unpack2(b.hi, x, y);
    const f2 r0 = pack2(ebbdf::rcp32(x), ebbdf::rcp32(y)), nh = neg2(b.hi), nl = neg2(b.lo);
    f2 q = mul2(a.hi, r0);
    q = fma2(fma2(q, nh, a.hi), r0, q);
    const dfp r = two_sum2(fma2(q, nh, a.hi), fma2(q, nl, a.lo));
    const f2 l = mul2(r.hi, r0), left = add2(fma2(l, nl, fma2(l, nh, r.hi)), r.lo);
    const dfp s = fast_two_sum2(q, l);
    return fast_two_sum2(s.hi, fma2(left, r0, s.lo));
}
__device__ __forceinline__ dfp recip(dfp b) { return both(df(1.0f)) / b; }
// sqrt of both, which are positive normal numbers (any other element by dfloat.h's sqrt)
__device__ __forceinline__ dfp root(dfp a)
{
    float x, y;
    unpack2(a.hi, x, y);
    if (!(x >= 0x1p-126f && y >= 0x1p-126f)) return pair(sqrt(first(a)), sqrt(second(a)));
    const f2 r = pack2(ebbdf::rsqrt32(x), ebbdf::rsqrt32(y)), h = mul2(pack2(0.5f, 0.5f), r);
    f2 s = mul2(a.hi, r);
    s = fma2(fma2(neg2(s), s, a.hi), h, s);
    const f2 t = add2(fma2(neg2(s), s, a.hi), a.lo);
    f2 c = mul2(t, h);
    c = fma2(fma2(neg2(c), add2(s, s), t), h, c);
    return fast_two_sum2(s, c);
}

}  // namespace ebbdev
