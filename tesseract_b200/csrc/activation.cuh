// Activations of gated feed-forwards, in 32-bit: one definition for the kernel that stands behind a product and for the products
// that apply them to their own sums, so that both store the same bits.
#pragma once

#include "common.cuh"

namespace tbact {

enum Activation : int { ACT_SILU = 0, ACT_GELU_TANH = 1, ACT_CLAMPED = 2 };

template <int ACT>
__device__ __forceinline__ float activate(float z) {
    if (ACT == ACT_SILU) return z * (1.0f / (1.0f + expf(-z)));
    const float inner = 0.7978845608028654f * (z + 0.044715f * z * z * z);
    return 0.5f * z * (1.0f + tanhf(inner));
}

// act(gate) * up of a product's 32-bit sums, each first rounded as the product would have stored it
template <int ACT>
__device__ __forceinline__ float gated_rounded(float gate, float up) {
    return activate<ACT>(__bfloat162float(__float2bfloat16_rn(gate))) * __bfloat162float(__float2bfloat16_rn(up));
}

}  // namespace tbact
