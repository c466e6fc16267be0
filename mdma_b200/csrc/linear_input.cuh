// What a token's projections go through before they enter a linear-attention recurrence.
#pragma once
#include "common.cuh"

namespace mdma {

__device__ __forceinline__ float silu_float(float z) { return z / (1.0f + expf(-z)); }

// What happens to a token's projections before they enter the recurrence: SiLU or nothing; the first 2 * half numbers of
// every q and k head turned by the token's position (pairs (i, i + half), or (2i, 2i + 1) if interleaved; half 0: none);
// k times k_scale.
struct LinInput {
    int silu, half, interleaved;
    float k_scale;
    const float* inv_freq;       // [half]
    const int* tok_pos;
};
__device__ __forceinline__ float lin_act(float z, int silu) { return silu ? silu_float(z) : z; }

}  // namespace mdma
