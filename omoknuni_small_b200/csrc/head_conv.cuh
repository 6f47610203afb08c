// The heads' 1x1 convolutions on the tensor cores in fp32 precision: what the kernels that compute them share.
//
// A channel's fp32 weights (BatchNorm folded) are split into three terms of the tower's storage type; the tower's
// output is in that type, so every product is exact.  With fp16 the channel is scaled by a power of two first, so that
// the third term is still a normal number.  The products with the leading term have an accumulator of their own.
#pragma once
#include <cuda_runtime.h>
#include <cmath>

namespace ob200 {

// Max(v, 0) that keeps NaN, as torch's relu does (fmaxf would make it 0, and a network that has overflowed would go on
// with plausible numbers).
__device__ __forceinline__ float relu_keep_nan(float v) { return v <= 0.0f ? 0.0f : v; }

// The leading products' sum and the rest's.  An infinite factor makes the leading sum what one fp32 product per weight
// would be, but turns the rest into NaN (terms of either sign, or a term of zero): then the leading sum stands alone.
__device__ __forceinline__ float join_terms(float leading, float rest) {
    return fabsf(leading) < INFINITY ? __fadd_rn(leading, rest) : leading;
}

// relu((leading + rest) / 2^e + bias)
__device__ __forceinline__ float head_conv_value(float leading, float rest, float scale, float bias) {
    return relu_keep_nan(__fadd_rn(__fmul_rn(join_terms(leading, rest), scale), bias));
}

}  // namespace ob200
