// f32x2.cuh — packed pairs of floats: one instruction, two multiply-adds, each
// rounded to nearest as the scalar instruction rounds.
#pragma once

#include <cuda_runtime.h>

namespace f2x {

using P = unsigned long long;   // (x, y) in one 64-bit register pair
__device__ __forceinline__ P pk(float2 v) {
    P r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
    return r;
}
__device__ __forceinline__ float2 un(P v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ P add(P a, P b) {
    P r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ P sub(P a, P b) {
    P r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ P mul(P a, P b) {
    P r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ P fma(P a, P b, P c) {
    P r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ P both(float k) { return pk(make_float2(k, k)); }

}  // namespace f2x
