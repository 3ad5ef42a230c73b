// Two FP32 values per register pair: sm_100a's packed add, multiply and
// fused multiply-add work on both at once, so a thread that carries two cells
// issues half the arithmetic instructions.  Each half rounds as the scalar
// instruction does.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace lbm {

struct F2 {
    float2 v;
    __device__ __forceinline__ F2() {}
    __device__ __forceinline__ F2(float2 a) : v(a) {}
    __device__ __forceinline__ explicit F2(float s) : v(make_float2(s, s)) {}
    __device__ __forceinline__ F2(float a, float b) : v(make_float2(a, b)) {}
};
__device__ __forceinline__ F2 operator-(F2 a) { return F2(-a.v.x, -a.v.y); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return F2(__fadd2_rn(a.v, make_float2(-b.v.x, -b.v.y))); }
__device__ __forceinline__ F2 xfma(F2 a, F2 b, F2 c) { return F2(__ffma2_rn(a.v, b.v, c.v)); }
__device__ __forceinline__ F2 xmul(F2 a, F2 b) { return F2(__fmul2_rn(a.v, b.v)); }
// a product no sum is fused with: the compiler does fuse a packed product with
// a packed sum where the product has no other use
__device__ __forceinline__ F2 xmul_apart(F2 a, F2 b) { return F2(__fmul_rn(a.v.x, b.v.x), __fmul_rn(a.v.y, b.v.y)); }
__device__ __forceinline__ F2 xadd(F2 a, F2 b) { return F2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ F2 xrcp(F2 a) { return F2(1.0f / a.v.x, 1.0f / a.v.y); }
__device__ __forceinline__ F2 xsqrt(F2 a) { return F2(sqrtf(a.v.x), sqrtf(a.v.y)); }

}  // namespace lbm
