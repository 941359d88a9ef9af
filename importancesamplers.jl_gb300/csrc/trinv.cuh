// trinv.cuh — FP32 inverse of a lower-triangular factor in shared memory,
// shared by the factor inversion and the moment-fit kernels.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace issm {

// W = L^-1 for d <= 64, both row-major in shared memory with leading dimension
// ld. The 8 x 8 diagonal blocks are inverted one column per thread, then pairs of
// blocks of s = 8, 16, 32 rows are merged, W21 = -W22 (L21 W11): three levels of
// two products each, so six barriers (a forward pass over block rows took seven
// dependent steps: 14,600 cycles at d = 64, now 8,700). L's strict upper triangle is scratch.
// Called by all 256 threads of a CTA.
__device__ __forceinline__ void invert_lower_f32(float *L, float *W, int d, int ld) {
    const int nb = (d + 7) >> 3, t = threadIdx.x;
    for (int e = t; e < d * ld; e += 256) W[e] = 0.f;
    __syncthreads();
    if (t < nb * 8) {
        const int b = t >> 3, c = t & 7, col = 8 * b + c, r0 = 8 * b;
        if (col < d) {
            float w[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const int row = r0 + r;
                float v = 0.f;
                if (row < d && r >= c) {
                    v = (r == c) ? 1.f : 0.f;
#pragma unroll
                    for (int q = 0; q < r; ++q)
                        if (q >= c) v -= L[row * ld + r0 + q] * w[q];
                    v /= L[row * ld + row];
                }
                w[r] = v;
            }
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (r0 + r < d) W[(r0 + r) * ld + col] = w[r];
        }
    }
    __syncthreads();
    auto level = [&](auto size) {
        constexpr int s = decltype(size)::value, U = s / 8;  // rows a0 + 8 u of column b, per thread
        if (s >= d) return;
        const int tp = t & (8 * s - 1), c0 = t / (8 * s) * 2 * s, r0 = c0 + s, b = tp % s, a0 = tp / s;
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = 0.f;
        // T = L21 W11 into L's upper block (c0, r0)
        if (r0 < d) {
#pragma unroll 8
            for (int k = 0; k < s; ++k) {
                const float w = W[(c0 + k) * ld + c0 + b];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int row = min(r0 + a0 + 8 * u, d - 1);
                    v[u] = fmaf(L[row * ld + c0 + k], w, v[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (r0 + a0 + 8 * u < d) L[(c0 + a0 + 8 * u) * ld + r0 + b] = v[u];
        }
        __syncthreads();
        if (r0 < d) {
            const int kn = min(s, d - r0);
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] = 0.f;
#pragma unroll 8
            for (int k = 0; k < kn; ++k) {
                const float x = L[(c0 + k) * ld + r0 + b];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int row = min(r0 + a0 + 8 * u, d - 1);
                    v[u] = fmaf(W[row * ld + r0 + k], x, v[u]);
                }
            }
        }
        __syncthreads();
        if (r0 < d) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (r0 + a0 + 8 * u < d) W[(r0 + a0 + 8 * u) * ld + c0 + b] = -v[u];
        }
        __syncthreads();
    };
    level(std::integral_constant<int, 8>());
    level(std::integral_constant<int, 16>());
    level(std::integral_constant<int, 32>());
}

}  // namespace issm
