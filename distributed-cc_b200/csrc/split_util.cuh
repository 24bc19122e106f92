// The two-piece splits x = hi + lo of the split-precision GEMM operands.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace dcc {

// x = hi + lo with hi = bf16(x), lo = bf16(x - hi).
__device__ __forceinline__ void split_bf16(double x, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
    hi = __float2bfloat16_rn((float)x);
    lo = __float2bfloat16_rn((float)(x - (double)__bfloat162float(hi)));
}

// The same pieces of an FP32 value without FP64: hi is f rounded to eight bits, so f - hi is exact
// in FP32 (also where it is an infinity or a NaN) and its rounding the one above.  Conversions to and
// from FP64 issue at an eighth of the FP32 rate: at nocc=10, nvir=90 the splits of U and X (5.8 GB
// each) took 1.8-2.1 ms with four of them per element, 1.6-1.8 without.
__device__ __forceinline__ void split_bf16(float f, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
    hi = __float2bfloat16_rn(f);
    lo = __float2bfloat16_rn(f - __bfloat162float(hi));
}

// x = hi + lo with hi, lo rounded to tf32 (10 explicit mantissa bits).
__device__ __forceinline__ float round_tf32(float f) {
    uint32_t u = __float_as_uint(f);
    if ((u & 0x7f800000u) == 0x7f800000u) return f;
    u += 0x1000u;  // round half away from zero on the 13 dropped bits
    u &= 0xffffe000u;
    return __uint_as_float(u);
}
__device__ __forceinline__ void split_tf32(double x, float &hi, float &lo) {
    hi = round_tf32((float)x);
    lo = round_tf32((float)(x - (double)hi));
}

__device__ __forceinline__ void split_tf32(float f, float &hi, float &lo) {
    hi = round_tf32(f);
    lo = round_tf32(f - hi);
}

}  // namespace dcc
