// What a feed-forward unit computes from the sums of its first product, for the kernels of routed experts.
#pragma once

#include <math.h>

#include "common.cuh"

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }

// The gated product of a unit's two hidden features g (gate) and u (up), by `act`:
//   0: silu(g) * u        1: g' * sigmoid(1.702 g') * (u' + 1), g' = min(g, limit), u' = clamp(u, -limit, limit)
//   2: gelu_tanh(g) * u
__device__ __forceinline__ float gated_value(int act, float limit, float g, float u) {
    if (act == 1) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return g / (1.0f + expf(-1.702f * g)) * (u + 1.0f);
    }
    if (act == 2) return gelu_tanh(g) * u;
    return silu(g) * u;
}

// A unit without a gate: its one hidden feature z, by `act` (0: max(z, 0)^2, 1: gelu_tanh(z), 2: silu(z)).
__device__ __forceinline__ float plain_value(int act, float z) { return act == 0 ? relu_sq(z) : act == 1 ? gelu_tanh(z) : silu(z); }
