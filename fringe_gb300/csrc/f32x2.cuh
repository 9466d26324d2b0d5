// f32x2.cuh -- packed pairs of floats: one instruction, two IEEE operations
// (sm_100 and later).  A pair is a 64-bit register pair, low half first.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fpl {
// internal linkage: the header is compiled into more than one unit
namespace {

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo2(f32x2 a)
{
    return __uint_as_float((uint32_t)a);
}
__device__ __forceinline__ float hi2(f32x2 a)
{
    return __uint_as_float((uint32_t)(a >> 32));
}
__device__ __forceinline__ f32x2 swap2(f32x2 a) { return pk(hi2(a), lo2(a)); }
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
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

}  // namespace
}  // namespace fpl
