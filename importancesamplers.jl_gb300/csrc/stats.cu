// stats.cu — result statistics on the device (src/statistics.jl):
//
//   weighted_sum      sum_i w_i x_i per coordinate with the self-normalised
//                     weights w_i = e^{l_i - m} / S of the result's summary
//                     (Statistics.mean(result) and, on f's values,
//                     Statistics.mean(f, result), :11-33): FP64 sums for FP64
//                     data, compensated FP32 sums merged in FP64 for FP32 data,
//                     per-block partials reduced in a fixed order (bitwise
//                     reproducible).
//
// Samples are n x d row-major (sample i contiguous). Keys order like the
// values (see select.cu); a coordinate holding a NaN returns NaN, as the
// reference does.
#include "issm_device.cuh"
#include "issm_internal.h"

namespace issm {

constexpr int kSumThreads = 256;
constexpr int kSumTile = 64;  // samples per block-iteration staged in shared memory

// per-block partial sums of w_i x_i (d <= 64 per pass over coordinate blocks)
template <typename T>
__global__ void weighted_sum_partial_kernel(const T *__restrict__ x, int d, int64_t n, const T *__restrict__ lw,
                                            const double *__restrict__ summary, double *__restrict__ partial) {
    __shared__ double tile[kSumTile][65];
    __shared__ double ws[kSumTile];
    const double m = summary[0], inv = 1.0 / summary[1];
    const int c0 = blockIdx.y * 64, dc = min(64, d - c0);
    double acc = 0.0;  // thread t < dc owns coordinate c0 + t
    const int64_t tiles = (n + kSumTile - 1) / kSumTile;
    for (int64_t tt = blockIdx.x; tt < tiles; tt += gridDim.x) {
        const int64_t r0 = tt * kSumTile;
        const int rows = (int)min((int64_t)kSumTile, n - r0);
        __syncthreads();
        for (int e = threadIdx.x; e < rows * dc; e += blockDim.x) {
            const int r = e / dc, c = e - r * dc;
            tile[r][c] = (double)x[(r0 + r) * d + c0 + c];
        }
        for (int r = threadIdx.x; r < rows; r += blockDim.x) {
            const double l = (double)lw[r0 + r];
            ws[r] = l == -INFINITY ? 0.0 : exp(l - m) * inv;
        }
        __syncthreads();
        if (threadIdx.x < dc)
            for (int r = 0; r < rows; ++r)
                if (ws[r] != 0.0) acc += ws[r] * tile[r][threadIdx.x];
    }
    if (threadIdx.x < dc) partial[((size_t)blockIdx.x * gridDim.y + blockIdx.y) * 64 + threadIdx.x] = acc;
}

// FP32 samples: per-thread compensated FP32 (Kahan) sums of w x with w in
// FP32 (expf of the FP32 log weight less the summary's max, times 1/S), four
// row groups per coordinate merged in FP64 in a fixed order. In FP64 the pass
// ran on this GPU's narrow FP64 pipe (a conversion and an FMA per element)
// at several times its memory time. Thread t owns coordinate t % 64 of every
// fourth row, so a warp reads consecutive coordinates of one row.
__global__ void __launch_bounds__(kSumThreads) weighted_sum_partial_f32_kernel(const float *__restrict__ x, int d,
                                                                              int64_t n,
                                                                              const float *__restrict__ lw,
                                                                              const double *__restrict__ summary,
                                                                              double *__restrict__ partial) {
    __shared__ float ws[2][kSumTile];
    __shared__ double s4[4][64];
    const float m = (float)summary[0], inv = (float)(1.0 / summary[1]);
    const int c0 = blockIdx.y * 64, dc = min(64, d - c0);
    const int c = threadIdx.x & 63, rg = threadIdx.x >> 6;
    float s = 0.f, k = 0.f;
    const int64_t tiles = (n + kSumTile - 1) / kSumTile;
    constexpr int kRows = kSumTile / 4;  // of a tile, per thread
    int buf = 0;
    for (int64_t tt = blockIdx.x; tt < tiles; tt += gridDim.x, buf ^= 1) {
        const int64_t r0 = tt * kSumTile;
        const int rows = (int)min((int64_t)kSumTile, n - r0);
        // the tile's loads are all in flight before its weights are formed
        float v[kRows];
        const float *xp = x + (r0 + rg) * d + c0 + c;
#pragma unroll
        for (int u = 0; u < kRows; ++u) v[u] = c < dc && rg + 4 * u < rows ? xp[(size_t)(4 * u) * d] : 0.f;
        if (threadIdx.x < kSumTile) {
            const float l = threadIdx.x < rows ? lw[r0 + threadIdx.x] : -INFINITY;
            ws[buf][threadIdx.x] = l == -INFINITY ? 0.f : expf(l - m) * inv;
        }
        __syncthreads();  // two weight buffers: one barrier per tile
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            const float w = ws[buf][rg + 4 * u];
            if (w == 0.f) continue;  // a zero weight contributes nothing (not even a NaN)
            const float y = fmaf(w, v[u], -k);
            const float t = s + y;
            k = (t - s) - y;
            s = t;
        }
    }
    s4[rg][c] = (double)s - (double)k;
    __syncthreads();
    if (threadIdx.x < dc)
        partial[((size_t)blockIdx.x * gridDim.y + blockIdx.y) * 64 + threadIdx.x] =
            ((s4[0][threadIdx.x] + s4[1][threadIdx.x]) + s4[2][threadIdx.x]) + s4[3][threadIdx.x];
}

// Per-block sums in a fixed order: 32 lanes per coordinate, then lane order.
// (One thread walking 1,216 partials took 140 us.)
__global__ void __launch_bounds__(1024) weighted_sum_finish_kernel(const double *__restrict__ partial, int blocks, int d,
                                                                   double *out) {
    __shared__ double red[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, c = blockIdx.x * 32 + tx;
    const int cb = c / 64, cc = c % 64, ncb = (d + 63) / 64;
    double s = 0.0;
    if (c < d)
        for (int b = ty; b < blocks; b += 32) s += partial[((size_t)b * ncb + cb) * 64 + cc];
    red[ty][tx] = s;
    __syncthreads();
    if (ty == 0 && c < d) {
        for (int r = 1; r < 32; ++r) s += red[r][tx];
        out[c] = s;
    }
}

constexpr int kSumBlocksPerSm = 8;  // enough loads in flight to stream the samples

static int sum_blocks(int64_t n) {
    const int64_t t = (n + kSumTile - 1) / kSumTile;
    const int64_t cap = (int64_t)device_sms() * kSumBlocksPerSm;
    return (int)(t < cap ? (t < 1 ? 1 : t) : cap);
}

size_t weighted_sum_workspace_bytes(int64_t n, int d) {
    return sizeof(double) * (size_t)kSMs * kSumBlocksPerSm * (size_t)((d + 63) / 64) * 64;
}

int weighted_sum(const void *x, int d, int64_t n, const void *lw, int dtype, const double *summary, double *out,
                 void *ws, cudaStream_t stream) {
    const int blocks = sum_blocks(n);
    const dim3 grid(blocks, (d + 63) / 64);
    double *partial = (double *)ws;
    if (dtype == ISSM_F32)
        weighted_sum_partial_f32_kernel<<<grid, kSumThreads, 0, stream>>>((const float *)x, d, n,
                                                                         (const float *)lw, summary, partial);
    else
        weighted_sum_partial_kernel<double><<<grid, kSumThreads, 0, stream>>>((const double *)x, d, n,
                                                                             (const double *)lw, summary, partial);
    note_launch();
    weighted_sum_finish_kernel<<<(d + 31) / 32, 1024, 0, stream>>>(partial, blocks, d, out);
    note_launch();
    return (int)cudaGetLastError();
}

}  // namespace issm
