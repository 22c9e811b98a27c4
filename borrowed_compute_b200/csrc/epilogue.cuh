// What a matrix product does with its sums, by number, and the epilogues of the true 32-bit products.
#pragma once

#include "common.cuh"

enum { EPI_STORE = 0, EPI_STORE_F32 = 1, EPI_ADD_F32 = 2, EPI_SWIGLU = 3, EPI_RELU2 = 4, EPI_XIELU = 5, EPI_SILU_F32 = 6 };

// Output (m, n) of a product that is N wide, from its sum v (SwiGLU: gate v, up u).
template <class T, int EPI>
__device__ __forceinline__ void simt_emit(T* out_act, float* out_f32, int m, int n, int N, float v, float u, float act_a, float act_b, int act_cols) {
    const size_t o = (size_t)m * N + n;
    if (EPI == EPI_STORE) out_act[o] = from_f32<T>(v);
    if (EPI == EPI_RELU2) {
        const float z = fmaxf(v, 0.0f);
        out_act[o] = from_f32<T>(z * z);
    }
    if (EPI == EPI_XIELU) out_act[o] = from_f32<T>(fmaf(0.5f, v, v > 0.0f ? act_a * v * v : act_b * (expm1f(v) - v)));
    if (EPI == EPI_SILU_F32) out_f32[o] = n < act_cols ? v / (1.0f + expf(-v)) : v;
    if (EPI == EPI_STORE_F32) out_f32[o] = v;
    if (EPI == EPI_ADD_F32) out_f32[o] += v;
    if (EPI == EPI_SWIGLU) out_act[o] = from_f32<T>(v / (1.0f + expf(-v)) * u);
}
