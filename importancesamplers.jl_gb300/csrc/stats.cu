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
    __shared__ float ws[kSumTile];
    __shared__ double s4[4][64];
    const float m = (float)summary[0], inv = (float)(1.0 / summary[1]);
    const int c0 = blockIdx.y * 64, dc = min(64, d - c0);
    const int c = threadIdx.x & 63, rg = threadIdx.x >> 6;
    float s = 0.f, k = 0.f;
    const int64_t tiles = (n + kSumTile - 1) / kSumTile;
    for (int64_t tt = blockIdx.x; tt < tiles; tt += gridDim.x) {
        const int64_t r0 = tt * kSumTile;
        const int rows = (int)min((int64_t)kSumTile, n - r0);
        __syncthreads();
        if (threadIdx.x < rows) {
            const float l = lw[r0 + threadIdx.x];
            ws[threadIdx.x] = l == -INFINITY ? 0.f : expf(l - m) * inv;
        }
        __syncthreads();
        if (c < dc) {
#pragma unroll 4
            for (int r = rg; r < rows; r += 4) {
                const float w = ws[r];
                if (w == 0.f) continue;  // a zero weight contributes nothing (not even a NaN)
                const float y = fmaf(w, x[(r0 + r) * d + c0 + c], -k);
                const float t = s + y;
                k = (t - s) - y;
                s = t;
            }
        }
    }
    s4[rg][c] = (double)s - (double)k;
    __syncthreads();
    if (threadIdx.x < dc)
        partial[((size_t)blockIdx.x * gridDim.y + blockIdx.y) * 64 + threadIdx.x] =
            ((s4[0][threadIdx.x] + s4[1][threadIdx.x]) + s4[2][threadIdx.x]) + s4[3][threadIdx.x];
}

__global__ void weighted_sum_finish_kernel(const double *__restrict__ partial, int blocks, int d, double *out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= d) return;
    const int cb = c / 64, cc = c % 64, ncb = (d + 63) / 64;
    double s = 0.0;
    for (int b = 0; b < blocks; ++b) s += partial[((size_t)b * ncb + cb) * 64 + cc];
    out[c] = s;
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
    weighted_sum_finish_kernel<<<(d + 127) / 128, 128, 0, stream>>>(partial, blocks, d, out);
    note_launch();
    return (int)cudaGetLastError();
}

}  // namespace issm
