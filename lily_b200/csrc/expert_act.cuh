// The experts' activations, shared by the grouped products and the kernels for a few tokens.
#pragma once

#include "common.cuh"

namespace lily {

// act 0: the clamped gate; 1: silu(g) u
__device__ __forceinline__ float expert_gate(int act, float g, float u, float limit, float alpha) {
    if (act == 1) return (g / (1.f + expf(-g))) * u;
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return (g / (1.f + expf(-alpha * g))) * (u + 1.f);
}

__device__ __forceinline__ float squared_relu(float z) {
    const float r = fmaxf(z, 0.f);
    return r * r;
}

}  // namespace lily
