// The heads' 1x1 convolutions on the tensor cores in fp32 precision: what the kernels that compute them share.
//
// A channel's fp32 weights (BatchNorm folded) are split into three terms of the tower's storage type; the tower's
// output is in that type, so every product is exact.  With fp16 the channel is scaled by a power of two first, so that
// the third term is still a normal number.  The products with the leading term have an accumulator of their own.
#pragma once
#include <cuda_runtime.h>

namespace ob200 {

// relu((leading + rest) / 2^e + bias)
__device__ __forceinline__ float head_conv_value(float leading, float rest, float scale, float bias) {
    return fmaxf(__fadd_rn(__fmul_rn(__fadd_rn(leading, rest), scale), bias), 0.0f);
}

}  // namespace ob200
