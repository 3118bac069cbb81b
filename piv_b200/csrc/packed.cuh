// Two-component FP32 arithmetic in packed instructions (sm_100).
#pragma once

#include <cuda_runtime.h>

namespace pivb200 {

// Both components in one instruction (FADD2 / FFMA2). The correlation kernels are bound by
// instruction issue (59-67 % of cycles before, FMA pipe 27-37 %), and a packed operation takes one
// issue slot for two results; a - b is written as b * -1 + a, the same single rounding.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 cmul2(float2 a, float2 b) { return __fmul2_rn(a, b); }  // per component
__device__ __forceinline__ float2 cfma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }

// Products that round by themselves before a packed add. The compiler fuses a packed multiplication
// and a packed addition into one FMA2 whatever its -fmad setting and the rounding suffixes (checked on
// random values), so the product is written as an FMA2 with -0, with the -0 made from a value that
// only the launch knows (a count, which is never negative).
struct SeparateProduct {
    float2 nz;
    __device__ __forceinline__ explicit SeparateProduct(int nonnegative) {
        nz.x = nz.y = __int_as_float((nonnegative >> 31) | (int)0x80000000);
    }
    __device__ __forceinline__ float2 operator()(float2 a, float2 b) const { return __ffma2_rn(a, b, nz); }
};

}  // namespace pivb200
