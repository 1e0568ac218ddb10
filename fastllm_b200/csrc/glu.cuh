#pragma once
#include "common.cuh"

namespace fl {

__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + expf(-z)); }

// Feed-forward activations (fl_ffn_act), shared by the GEMM epilogue and the stand-alone kernels: 0 = g sigmoid(1.702 g) (u + 1) with
// g <= limit, |u| <= limit; 1 = gelu_tanh(g) u; 2 = relu(g)^2 (no up matrix); 3 = relu(g) u; 4 = silu(g) u.
__device__ __forceinline__ float gelu_tanhf_(float g) { return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))); }
__device__ __forceinline__ float glu_value(float g, float u, int act, float limit) {
    if (act == 2) { g = fmaxf(g, 0.f); return g * g; }
    if (act == 3) return fmaxf(g, 0.f) * u;
    if (act == 4) return g * sigmoidf_(g) * u;
    if (act == 1) return gelu_tanhf_(g) * u;
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g * sigmoidf_(1.702f * g) * (u + 1.f);
}

}  // namespace fl
