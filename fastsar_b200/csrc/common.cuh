// Shared helpers of the ffbp_b200 kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

namespace ffbp {

constexpr float TWO_PI_F = 6.28318530717958647692f;
constexpr double TWO_PI = 6.28318530717958647692;
constexpr double C_LIGHT = 299792458.0;

// exp(2 pi i c) for a phase c in cycles already reduced to [-0.5, 0.5]: the hardware sine and cosine are accurate to
// about 4e-7 absolute on [-pi, pi], which is the whole range they are given here.
__device__ __forceinline__ float2 cis_reduced(float c)
{
    float s, co;
    __sincosf(TWO_PI_F * c, &s, &co);
    return make_float2(co, s);
}

// exp(2 pi i c) for any float32 phase in cycles (reduced first).
__device__ __forceinline__ float2 cis_cycles(float c)
{
    return cis_reduced(c - rintf(c));
}

// exp(2 pi i c) for a float64 phase in cycles: the reduction in float64, the sine and cosine in float32.
__device__ __forceinline__ float2 cis_cycles_d(double c)
{
    return cis_reduced((float)(c - rint(c)));
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// 2^e, e in [-126, 127]
__device__ __forceinline__ float pow2(int e)
{
    return __int_as_float((127 + e) << 23);
}

// ex with 2^(ex - 1) <= m < 2^ex of a largest component m given as its float bits; INT_MIN where m is 0, below the normal
// numbers or not finite, or there is none. On the bits: every thread of the pulse FIR evaluates it.
__device__ __forceinline__ int top_exponent(const int *amax)
{
    const int b = amax ? *amax : 0;
    return b >= 0x00800000 && b < 0x7f800000 ? (b >> 23) - 126 : INT_MIN;
}

// e of the power of two 2^e that a tensor-core level's intermediate is scaled by: values up to 4 m (m the input's largest
// component; the taps' absolute sum is below 4 for the decimators of any plan) come below 2^13, times the window's 2^wexp
// (LevelLaunch::wexp): a float16 intermediate then stays in range and keeps 11 significant bits. 2^e, 2^-e and an eighth of
// either are normal float32 numbers.
__device__ __forceinline__ int level_exponent(const int *amax, int wexp)
{
    const int ex = top_exponent(amax);
    return ex == INT_MIN ? 0 : min(max(11 - ex - wexp, -120), 120);
}

// Two float32 fused multiply-adds in one instruction (sm_100's packed FMA): (a.x b.x + c.x, a.y b.y + c.y), each
// rounded as fmaf rounds it.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c)
{
    float2 d;
    asm("{\n\t.reg .b64 pa, pb, pc, pd;\n\t"
        "mov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\tmov.b64 pc, {%6, %7};\n\t"
        "fma.rn.f32x2 pd, pa, pb, pc;\n\tmov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// Two float32 values in one 64-bit register: the operands of the packed instructions, kept packed so that no moves
// rebuild the pairs.
using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pack2(float x, float y)
{
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}

__device__ __forceinline__ float2 unpack2(f32x2 v)
{
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
}

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

}  // namespace ffbp
