// round_tf32.cuh -- element conversions shared by the contraction kernels' epilogues.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace one {

// Round to the nearest tf32 (10 mantissa bits), ties away from zero, like cvt.rna.tf32.f32 -- but with
// two integer instructions: the conversion instruction runs on the 16-lane special-function pipe and,
// at one per output element, was a measurable share of the epilogue (that pipe 42 % busy on a 3x3
// 64-channel layer).  Adding half an ulp to the magnitude bits and clearing the low 13 carries into the
// exponent correctly.  Infinities and NaNs (exponent all ones) pass through untouched: the add would
// carry a NaN's mantissa into the sign bit and turn it into -0.0, and cvt.rna keeps NaNs too.
__device__ __forceinline__ float round_to_tf32(float v)
{
    const uint32_t u = __float_as_uint(v);
    return ((u & 0x7f800000u) == 0x7f800000u) ? v : __uint_as_float((u + 0x1000u) & 0xffffe000u);
}

// Quantise for an int8 consumer: x * (1/scale), clamp to [-128, 127], roundf
// (device/x86/Conv/conv.c:961-973).
__device__ __forceinline__ int quant_s8(float v, float inv_scale)
{
    float t = __fmul_rn(v, inv_scale);
    t = (t < -128.f) ? -128.f : (t > 127.f) ? 127.f : t;
    return (int)roundf(t);
}

}  // namespace one
