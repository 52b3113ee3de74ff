// What the kernels of the real-gated linear recurrent unit share.
#pragma once
#include "common.cuh"
#include <math.h>

__device__ __forceinline__ float rg_sigmoid(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float rg_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }
// One output's sum by float32 multiply-adds of the whole inputs: what the three parts of a finite input times an infinite
// weight are not (a part that is zero makes a NaN of it).
static __device__ __noinline__ float rm_plain(const float* u, const bf16* w, int bw) {
    float s = 0.f;
    for (int k = 0; k < bw; ++k) s = fmaf(to_f32(w[(size_t)k * bw]), u[k], s);
    return s;
}
