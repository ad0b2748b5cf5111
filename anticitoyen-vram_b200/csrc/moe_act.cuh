// Activations of the experts' products.
#pragma once

#include "common.cuh"

// gated activation of an expert (ops.GLU_*)
#define GLU_SWISH_CLAMPED 0  // g = min(a, limit), u = clamp(b, -limit, limit): g * sigmoid(alpha g) * (u + shift), shift 1
// (silu(a) * b is the same unit without limits, alpha 1 and shift 0)
// acv_glu also takes 1, 2, 3: act(a) * b with act the plain activation of that number (gelu_tanh, silu, gelu)

template <typename T> __device__ __forceinline__ float sigmoid_f32(float x);
template <> __device__ __forceinline__ float sigmoid_f32<float>(float x) { return 1.f / (1.f + expf(-x)); }
template <> __device__ __forceinline__ float sigmoid_f32<bf16>(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }

template <typename T>
__device__ __forceinline__ float glu_act(float a, float b, float limit, float alpha, float shift = 1.f) {
    const float g = fminf(a, limit);
    const float u = fminf(fmaxf(b, -limit), limit);
    return g * sigmoid_f32<T>(alpha * g) * (u + shift);
}

// activation of an expert that has no gate: y = act(W_up x), out = W_down y  (ops.ACTIVATIONS)
__device__ __forceinline__ float plain_act(float z, int kind) {
    if (kind == 1) return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
    if (kind == 2) return z / (1.f + expf(-z));
    if (kind == 3) return 0.5f * z * (1.f + erff(z * 0.7071067811865476f));
    return z;
}
