// f32x2.cuh -- the packed single-precision instructions of sm_100 (two IEEE operations per
// instruction, rounded like its scalar form; sum2 for a sum of products) and the float warp reductions.
// Measured on B200: a packed FMA / add / multiply issues every second cycle, so the arithmetic
// rate is that of the scalar forms at half the issue slots.
#pragma once
#include <cuda_runtime.h>

namespace vsdmo {

typedef unsigned long long f32x2;   // (low, high) floats

static __device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
static __device__ __forceinline__ void upk2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
static __device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
static __device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
static __device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// a - b, rounded once like the subtraction
static __device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { return fma2(b, pk2(-1.f, -1.f), a); }
static __device__ __forceinline__ f32x2 dup2(float a) { return pk2(a, a); }
// a + b where a or b is a product and both roundings of the scalar form are needed: ptxas contracts
// mul.rn.f32x2 + add.rn.f32x2 into one rounding where the product has no other use (also with
// --fmad=false, and a factor it can see to be 1 is folded first), so the sum is 1 a + b with a 1 from
// constant memory. The difference above is never contracted. The scalar forms are not affected.
static __constant__ float F32X2_ONE[2] = { 1.f, 1.f };
static __device__ __forceinline__ f32x2 sum2(f32x2 a, f32x2 b) { return fma2(a, pk2(F32X2_ONE[0], F32X2_ONE[1]), b); }
// (ax bx + ay by) + az bz
static __device__ __forceinline__ f32x2 dot2(f32x2 ax, f32x2 ay, f32x2 az, f32x2 bx, f32x2 by, f32x2 bz) {
    return sum2(sum2(mul2(ax, bx), mul2(ay, by)), mul2(az, bz));
}
// min(a, b, c); a NaN operand is ignored like by fminf
static __device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
static __device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// largest value of the full warp, NaNs ignored
static __device__ __forceinline__ float redux_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
static __device__ __forceinline__ float redux_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
static __device__ __forceinline__ float sqrt_approx(float v) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

}  // namespace vsdmo
