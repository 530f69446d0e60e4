// Packed FP32 pairs (sm_100): one instruction on two floats, each lane rounding as the scalar
// instruction does. An FP32x2 FMA takes the FMA pipe as long as two scalar ones; what it saves is
// issue slots and dependent-latency bubbles.
#pragma once

namespace us3d {

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void up2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 neg2(f32x2 v) { return v ^ 0x8000000080000000ull; }
__device__ __forceinline__ f32x2 dup2(float v) { return pk2(v, v); }
__device__ __forceinline__ f32x2 lo2(const float4& v) { return pk2(v.x, v.y); }
__device__ __forceinline__ f32x2 hi2(const float4& v) { return pk2(v.z, v.w); }
// 2^x of both lanes
__device__ __forceinline__ f32x2 ex2_2(f32x2 v) {
    float a, b;
    up2(v, a, b);
    return pk2(exp2f(a), exp2f(b));
}
__device__ __forceinline__ float sum2(f32x2 v) {
    float a, b;
    up2(v, a, b);
    return a + b;
}

}  // namespace us3d
