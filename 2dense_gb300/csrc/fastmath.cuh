// fastmath.cuh -- reciprocal, inverse square root and square root of doubles on the integer pipes,
// and the 64-bit integer helpers they share with the reconstructions (weno_fixed.cuh).
//
// GB300's FP64 pipe takes a warp instruction every 16 cycles of an SM, the integer pipes up to two a
// cycle each. From the hardware's double seeds a third-order step costs three (reciprocal) or five
// (inverse square root) FP64 instructions, 51 and 85 cycles; an IEEE divide costs ten. In 64-bit
// integers, from the single-precision seeds, both take some 45 integer instructions, 12 to 15 cycles
// beside the FP64 work of other warps, and round a 58-bit value once (below 0.52 ulp).
//
// The functions compile for the host too, where the tests compare them with long double.
#pragma once
#include <cstdint>
#ifndef __CUDACC__
#include <cmath>
#include <cstring>
#define DENSE_FX inline
#else
#define DENSE_FX __host__ __device__ __forceinline__
#endif

namespace dense {
namespace fx {

typedef uint32_t u32;
typedef uint64_t u64;
typedef int64_t i64;

DENSE_FX u32 hi32(u64 a) { return (u32)(a >> 32); }
DENSE_FX u64 wide(u32 a, u32 b) { return (u64)a * b; }
DENSE_FX int imax(int a, int b) { return a > b ? a : b; }
DENSE_FX int imin(int a, int b) { return a < b ? a : b; }
DENSE_FX u32 umax(u32 a, u32 b) { return a > b ? a : b; }
DENSE_FX u32 umin(u32 a, u32 b) { return a < b ? a : b; }
DENSE_FX u64 abs64(i64 a) {
    const u64 s = (u64)(a >> 63);
    return ((u64)a ^ s) - s;
}
// a >> n with 0 for n > 63, as PTX defines it
DENSE_FX u64 shr(u64 a, u32 n) {
#ifdef __CUDA_ARCH__
    u64 r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(n));
    return r;
#else
    return n > 63 ? 0 : a >> n;
#endif
}
DENSE_FX int clz32(u32 a) {
#ifdef __CUDA_ARCH__
    return __clz((int)a);
#else
    return a ? __builtin_clz(a) : 32;
#endif
}
DENSE_FX int clz64(u64 a) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)a);
#else
    return a ? __builtin_clzll(a) : 64;
#endif
}
DENSE_FX u64 bits(double d) {
#ifdef __CUDA_ARCH__
    return (u64)__double_as_longlong(d);
#else
    u64 r;
    memcpy(&r, &d, 8);
    return r;
#endif
}
DENSE_FX double from_bits(u64 b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double r;
    memcpy(&r, &b, 8);
    return r;
#endif
}
DENSE_FX u32 float_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    u32 r;
    memcpy(&r, &f, 4);
    return r;
#endif
}
DENSE_FX float rcp_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x;
#endif
}

DENSE_FX float rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / sqrtf(x);
#endif
}

// a b / 2^64, at most 2 below its floor: the product of the lower halves is left out
DENSE_FX u64 mulhi(u64 a, u64 b) {
    const u64 m1 = wide(hi32(a), (u32)b), m2 = wide((u32)a, hi32(b));
    return wide(hi32(a), hi32(b)) + hi32(m1) + hi32(m2);
}
// the same for a below 2^63 and b at most 2^63, whose middle products add up within a word
DENSE_FX u64 mulhi63(u64 a, u64 b) {
    const u64 m = wide(hi32(a), (u32)b) + wide((u32)a, hi32(b));
    return wide(hi32(a), hi32(b)) + hi32(m);
}
DENSE_FX u64 sqhi(u64 a) { return wide(hi32(a), hi32(a)) + (wide(hi32(a), (u32)a) >> 31); }

// 2^125 / n for n in [2^62, 2^63), relative error below 2^-59: x0 = 2^61 / (n / 2^32) to 22 bits
// from the hardware's reciprocal, e = 1 - x0 n, and 1/n = x0 (1 + e + e^2 + ...), Householder's third order
DENSE_FX u64 reciprocal(u64 n) {
    const u32 nh = hi32(n);
    // 2^53 (1 - 2^-22) x + 2^23 holds 2^53 x0 in its mantissa, below the next binade
    const float t = fmaf(rcp_seed((float)nh), 9007199254740992.0f * (1.0f - 1.0f / 4194304.0f), 8388608.0f);
    const u32 x0 = (float_bits(t) & 0x7fffffu) << 8;
    const i64 e = (i64)((1ull << 61) - (wide(x0, nh) + hi32(wide(x0, (u32)n))));  // 2^61 (1 - x0 n), below 2^42
    const int es = (int)(e >> 11);
    const i64 f = e + (i64)((u64)((i64)es * es) >> 39);  // 2^61 (e + e^2)
    return ((u64)x0 << 32) + (u64)(((i64)(int)x0 * (int)(f >> 11)) >> 18) + (wide(x0, (u32)f & 0x7ffu) >> 29);
}

// 1/d correctly rounded but for 1 in 50 or so (below 0.51 ulp), without FP64 instructions: the
// mantissa's reciprocal, rounded into a double. d normal and of any sign; results below the
// normal range are 0, and 0, infinities, NaN and denormals give NaN.
DENSE_FX double rcp(double d) {
    const u64 b = bits(d);
    const u32 h = hi32(b), e = (h >> 20) & 0x7ffu;
    const u64 n = ((u64)((((h << 10) | ((u32)b >> 22)) & 0x3fffffffu) | 0x40000000u) << 32) | (u32)((u32)b << 10);
    // 2^125/n = 2^63/1.m: 53 bits of it; their top bit counts into the exponent
    u64 r = ((reciprocal(n) + 0x200) >> 10) + ((u64)(2044u - e) << 52);
    if (e >= 2045u) r = 0;
    if (e - 1u >= 2046u) r = 0x7ff8000000000000ull;
    return from_bits(r | ((u64)(h & 0x80000000u) << 32));
}
// The mantissa and exponent of a positive normal x as v 2^(2 k), v = n/2^62 in [1, 4).
DENSE_FX u64 split_even(u64 b, int& k) {
    const u32 h = hi32(b);
    const int e = (int)(h >> 20) - 1023;
    k = e >> 1;
    const u64 n = ((u64)((((h << 10) | ((u32)b >> 22)) & 0x3fffffffu) | 0x40000000u) << 32) | (u32)((u32)b << 10);
    return n << (e & 1);
}
// 2^63 / sqrt(n/2^62) for n in [2^62, 2^64), relative error below 2^-58: y0 to 22 bits from the
// hardware's inverse square root, e = 1 - v y0^2, and 1/sqrt(v) = y0 (1 + e/2 + 3 e^2/8 + ...)
DENSE_FX u64 rsqrt63(u64 n) {
    // 2^38 (1 - 2^-22) y + 2^23 holds 2^23 y0 in its mantissa (y = 2^-15 / sqrt(v)), below the next binade
    const float t = fmaf(rsqrt_seed((float)hi32(n)), 274877906944.0f * (1.0f - 1.0f / 4194304.0f), 8388608.0f);
    const u32 y0 = (float_bits(t) & 0x7fffffu) << 8;               // 2^31 / sqrt(v)
    const u64 w = wide(y0, y0);                                    // 2^62 / v
    const i64 e = (i64)((1ull << 60) - mulhi(n, w));               // 2^60 e, below 2^41
    const int es = (int)(e >> 10);
    const i64 f = (e >> 1) + (i64)((3 * (u64)((i64)es * es)) >> 43);  // 2^60 (e/2 + 3 e^2/8)
    return ((u64)y0 << 32) + (u64)(((i64)(int)y0 * (int)(f >> 10)) >> 18) + (wide(y0, (u32)f & 0x3ffu) >> 28);
}
// 1/sqrt(x) and sqrt(x), below 0.51 ulp, as rcp; x positive and normal, else NaN.
DENSE_FX double rsqrt(double x) {
    int k;
    const u64 b = bits(x), n = split_even(b, k);
    u64 r = ((rsqrt63(n) + 0x200) >> 10) + ((u64)(u32)(1021 - k) << 52);
    if ((hi32(b) >> 20) - 1u >= 2046u) r = 0x7ff8000000000000ull;
    return from_bits(r);
}
DENSE_FX double sqrt_normal(double x) {
    int k;
    const u64 b = bits(x), n = split_even(b, k);
    const u64 q = mulhi(n, rsqrt63(n));                            // 2^61 sqrt(v)
    u64 r = ((q + 0x100) >> 9) + ((u64)(u32)(1022 + k) << 52);
    if ((hi32(b) >> 20) - 1u >= 2046u) r = 0x7ff8000000000000ull;
    return from_bits(r);
}

}  // namespace fx
}  // namespace dense
