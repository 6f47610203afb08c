// The heads' 1x1 convolutions on the tensor cores in fp32 precision: what the kernels that compute them share.
//
// A channel's fp32 weights (BatchNorm folded) are split into three terms of the tower's storage type; the tower's
// output is in that type, so every product is exact.  With fp16 the channel is scaled by a power of two first, so that
// the third term is still a normal number.  The products with the leading term have an accumulator of their own.
#pragma once
#include <cuda_runtime.h>
#include <cfloat>

namespace ob200 {

// Max(v, 0) that keeps NaN, as torch's relu does (fmaxf would make it 0, and a network that has overflowed would go on
// with plausible numbers).
__device__ __forceinline__ float relu_keep_nan(float v) {
    float r;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(v));
    return r;
}

// The leading products' sum and the rest's.  An infinite factor makes the leading sum what one fp32 product per weight
// would be, but turns the rest into an infinity of either sign or NaN (terms of either sign, or a term of zero): brought
// into fp32's range, the rest changes neither an infinity nor NaN.  (Minimum and maximum rather than a comparison and a
// selection: 0.3 us of an evaluation of 1 to 16 boards.)
__device__ __forceinline__ float join_terms(float leading, float rest) {
    return __fadd_rn(leading, fminf(fmaxf(rest, -FLT_MAX), FLT_MAX));
}

// relu((leading + rest) / 2^e + bias)
__device__ __forceinline__ float head_conv_value(float leading, float rest, float scale, float bias) {
    return relu_keep_nan(__fadd_rn(__fmul_rn(join_terms(leading, rest), scale), bias));
}

}  // namespace ob200
