// Activations in the epilogues of the projections (linear_packed.cu, linear_tiled.cu, linear_mid.cu, dot_split.cu).
#pragma once
#include "common.cuh"

namespace jsm {

static __device__ __noinline__ float pk_gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752440f)); }
__device__ __forceinline__ float pk_silu(float x) { return __fdividef(x, 1.0f + __expf(-x)); }  // 2 ulp division: short code
// gate/up pair with clamps: min(g, limit) * sigmoid(alpha * min(g, limit)) * (clamp(u, -limit, limit) + 1)
__device__ __forceinline__ float pk_clamped_glu(float g, float u, float alpha, float limit) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return __fdividef(g, 1.0f + __expf(-alpha * g)) * (u + 1.0f);
}

// gate/up pair with the tanh form of GELU: z (1 + tanh(y)) / 2 = z / (1 + e^(-2y)), y = sqrt(2/pi) (z + 0.044715 z^3)
__device__ __forceinline__ float pk_gelu_glu(float z, float u) {
    const float y2 = 1.5957691216057308f * fmaf(0.044715f * z * z, z, z);
    return __fdividef(z, 1.0f + __expf(-y2)) * u;
}

// the same two with exact divisions and functions (f32 models)
__device__ __forceinline__ float clamped_glu_f32(float g, float u, float alpha, float limit) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
}
__device__ __forceinline__ float gelu_glu_f32(float z, float u) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z))) * u;
}

}  // namespace jsm
