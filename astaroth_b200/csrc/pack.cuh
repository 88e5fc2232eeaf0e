/*
 * The cell values of one thread of the split-stage substep kernel: one double
 * (FP64 meshes), or two floats of two cells with the same x (FP32 compensated
 * meshes) that move through packed FP32x2 instructions, so that both
 * precisions have 64-bit values and one instruction stream.  Multiply-adds are
 * written out (vfma).  A packed product may all the same be fused with a packed sum
 * that follows it; where the rounded product itself is needed (the increment of the
 * RK update), it is formed by scalar products.
 */
#pragma once

#include <stdint.h>

#include "mhd_rhs.cuh"

/* two floats, .x in the low word */
struct F2 {
    unsigned long long v;
};

__host__ __device__ __forceinline__ F2
f2(const float x, const float y)
{
#ifdef __CUDA_ARCH__
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
#else
    union {
        float f[2];
        unsigned long long v;
    } u;
    u.f[0] = x;
    u.f[1] = y;
    return F2{u.v};
#endif
}
__device__ __forceinline__ float
lo_of(const F2 a)
{
    return __uint_as_float((uint32_t)a.v);
}
__device__ __forceinline__ float
hi_of(const F2 a)
{
    return __uint_as_float((uint32_t)(a.v >> 32));
}
__device__ __forceinline__ F2
operator+(const F2 a, const F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2
operator-(const F2 a, const F2 b)
{
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2
operator*(const F2 a, const F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2
vfma(const F2 a, const F2 b, const F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ double
vfma(const double a, const double b, const double c)
{
    return fma(a, b, c);
}
__device__ __forceinline__ F2
operator-(const F2 a)
{
    return F2{a.v ^ 0x8000000080000000ull};
}
__device__ __forceinline__ F2
vabs(const F2 a)
{
    return F2{a.v & 0x7fffffff7fffffffull};
}
__device__ __forceinline__ double
vabs(const double a)
{
    return fabs(a);
}
__device__ __forceinline__ F2
ac_exp(const F2 a)
{
    return f2(ac_exp(lo_of(a)), ac_exp(hi_of(a)));
}
__device__ __forceinline__ F2
ac_rcp(const F2 a)
{
    return f2(ac_rcp(lo_of(a)), ac_rcp(hi_of(a)));
}

template <typename V>
struct Pack;
template <>
struct Pack<double> {
    typedef double T;
    static constexpr int N = 1; /* cells per value */
    static __host__ __device__ __forceinline__ double dup(const double v) { return v; }
};
template <>
struct Pack<F2> {
    typedef float T;
    static constexpr int N = 2;
    static __host__ __device__ __forceinline__ F2 dup(const double v)
    {
        return f2((float)v, (float)v);
    }
};

/* tensor-memory words of a value */
__device__ __forceinline__ void
to_words(const double v, uint32_t* w)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    w[0]                       = (uint32_t)b;
    w[1]                       = (uint32_t)(b >> 32);
}
__device__ __forceinline__ void
to_words(const F2 v, uint32_t* w)
{
    asm("mov.b64 {%0, %1}, %2;" : "=r"(w[0]), "=r"(w[1]) : "l"(v.v));
}
__device__ __forceinline__ void
from_words(const uint32_t* w, double& v)
{
    v = __longlong_as_double(
        (long long)(((unsigned long long)w[1] << 32) | (unsigned long long)w[0]));
}
__device__ __forceinline__ void
from_words(const uint32_t* w, F2& v)
{
    asm("mov.b64 %0, {%1, %2};" : "=l"(v.v) : "r"(w[0]), "r"(w[1]));
}
