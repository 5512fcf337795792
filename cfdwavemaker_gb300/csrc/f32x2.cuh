// Packed FP32x2 arithmetic: two FP32 operations an instruction, each lane
// rounded as the scalar operation.  Values are 64-bit registers.
#pragma once

#include <cuda_runtime.h>

namespace cfdwm {

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 p_pack(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 p_un(f32x2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ float p_hsum(f32x2 a) {
    const float2 r = p_un(a);
    return r.x + r.y;
}
__device__ __forceinline__ f32x2 p_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 p_mul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 p_add(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a packed operand that a long loop keeps: a plain pack is a move that the
// compiler repeats at every use (6 moves a pair in k_pairs_points, velocity
// sums 16 % slower); the result of a packed multiplication (by 1, from a kernel
// argument) is held
__device__ __forceinline__ f32x2 p_hold(float a, float b, f32x2 one2) { return p_mul(p_pack(a, b), one2); }
__device__ __forceinline__ f32x2 p_ex2(f32x2 a) {
    const float2 v = p_un(a);
    return p_pack(ex2(v.x), ex2(v.y));
}

}  // namespace cfdwm
