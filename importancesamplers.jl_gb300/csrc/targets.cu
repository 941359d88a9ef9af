// targets.cu — built-in batch targets used by the benchmark configurations.
// In the reference the target is user code compiled into the sampling kernel
// or a batch callback (src/batched_targets.jl:54-114); these kernels are the
// native equivalents of the callbacks the benchmark workloads need.
#include "issm_device.cuh"
#include "issm_internal.h"

namespace issm {

constexpr double kLog2Pi = 1.8378770664093454835606594728112;

template <typename T>
__global__ void target_simple_kernel(issm_target t, const T *__restrict__ x, int64_t n, T *__restrict__ out) {
    const int d = t.dim;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const T *a = (const T *)t.a;
    const T *b = (const T *)t.b;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const T *xi = x + i * d;
        T v = T(0);
        if (t.kind == ISSM_TARGET_STD_NORMAL) {
            T r2 = T(0);
            for (int c = 0; c < d; ++c) r2 += xi[c] * xi[c];
            v = T(-0.5 * kLog2Pi) * T(d) - T(0.5) * r2;
        } else if (t.kind == ISSM_TARGET_QUADRATIC) {
            T r2 = T(0);
            for (int c = 0; c < d; ++c) { T z = xi[c] - a[c]; r2 += z * z; }
            v = -r2 / T(t.p0);
        } else if (t.kind == ISSM_TARGET_GAUSS_MIX) {
            LseState<T> lse;
            for (int j = 0; j < t.count; ++j) {
                T r2 = T(0);
                for (int c = 0; c < d; ++c) { T z = xi[c] - a[(size_t)j * d + c]; r2 += z * z; }
                lse.add(T(-0.5) * r2);
            }
            v = lse.value() - dlog(T(t.count)) - T(0.5 * kLog2Pi) * T(d);
        } else if (t.kind == ISSM_TARGET_STUDENT_T) {
            // normalised multivariate t with location a, scale factor b (column-major), nu = p0,
            // log constant p1 (already minus log|L|)
            T z[64];
            T r2 = T(0);
            for (int r = 0; r < d; ++r) {
                T s = xi[r] - a[r];
                for (int c = 0; c < r; ++c) s -= b[r + (size_t)c * d] * z[c];
                s /= b[r + (size_t)r * d];
                z[r] = s;
                r2 += s * s;
            }
            const T nu = T(t.p0);
            v = T(t.p1) - (nu + T(d)) * T(0.5) * dlog1p(r2 / nu);
        }
        out[i] = v;
    }
}

// Regression likelihoods in the target's type. A CTA of 16 x 16 threads takes
// 16 RS samples and walks the observations 64 at a time; a thread holds the
// linear predictors of RS samples x 4 observations while the coordinates pass
// through shared memory (X is nobs x d column-major, so a coordinate's
// observations are contiguous). The logistic terms use
// y eta - max(eta, 0) - log(1 + t), t = e^-|eta|, with the factors (1 + t)
// multiplied into a product, carried less one (P <- P + t + P t) so that small
// terms keep their relative accuracy, whose log1p is taken once per 64.
// Sums of FP32 terms are carried as unevaluated pairs.
//
// Bound by FMA issue with shared operands (FP32) or the FP64 pipe. A warp per
// sample that reread X for every sample took 118 us at 10,007 samples x 500
// observations, d = 33, FP32.
constexpr int kRegObs = 64;   // observations per step
constexpr int kRegDim = 64;   // coordinates staged at a time
constexpr int kRegFlush = 16; // steps between log1ps of the product (4 factors each)

template <typename T> struct RegSum {  // FP64: plain
    T h = T(0);
    __device__ __forceinline__ void add(T x) { h += x; }
    __device__ __forceinline__ void join(int off) { h += __shfl_xor_sync(0xffffffffu, h, off); }
    __device__ __forceinline__ T value() const { return h; }
};
template <> struct RegSum<float> {  // hi + lo, error-free additions
    float h = 0.f, l = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float s = h + x, b = s - h;
        l += (h - (s - b)) + (x - b);
        h = s;
    }
    __device__ __forceinline__ void join(int off) {
        const float oh = __shfl_xor_sync(0xffffffffu, h, off), ol = __shfl_xor_sync(0xffffffffu, l, off);
        add(oh);
        l += ol;
    }
    __device__ __forceinline__ float value() const { return isfinite(h) ? h + l : h; }
};

// N consecutive shared words, 16 bytes at a time where they fill them (aligned by the caller)
template <typename T, int N> __device__ __forceinline__ void reg_load(const T *src, T (&v)[N]) {
    constexpr int V = 16 / sizeof(T);
    if constexpr (N % V == 0) {
#pragma unroll
        for (int k = 0; k < N; k += V) *reinterpret_cast<uint4 *>(v + k) = *reinterpret_cast<const uint4 *>(src + k);
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = src[k];
    }
}

template <typename T, int RS>
__global__ void __launch_bounds__(256) target_regression_kernel(issm_target t, const T *__restrict__ x, int64_t n,
                                                                T constant, T scale, T prior_scale, int dim_tile,
                                                                T *__restrict__ out) {
    constexpr int TS = 16 * RS, LB = TS + 16 / (int)sizeof(T), LX = kRegObs;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *Bs = reinterpret_cast<T *>(smem_raw);  // dim_tile x LB: coordinate c of the CTA's samples
    T *Xs = Bs + (size_t)dim_tile * LB;       // dim_tile x LX: coordinate c of the step's observations
    const int d = t.dim, nobs = t.count, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const T *X = (const T *)t.a;
    const T *y = (const T *)t.b;
    const bool logistic = t.kind == ISSM_TARGET_LOGISTIC;
    const int64_t s0 = (int64_t)blockIdx.x * TS;
    const int rows = (int)min((int64_t)TS, n - s0);
    RegSum<T> acc[RS];
    T prod[RS];  // less one
    T bb[RS];
#pragma unroll
    for (int i = 0; i < RS; ++i) {
        prod[i] = T(0);
        bb[i] = T(0);
    }
    int steps = 0;
    for (int o0 = 0; o0 < max(nobs, 1); o0 += kRegObs) {
        T eta[RS][4];
#pragma unroll
        for (int i = 0; i < RS; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) eta[i][j] = T(0);
        for (int c0 = 0; c0 < d; c0 += dim_tile) {
            const int dc = min(dim_tile, d - c0);
            __syncthreads();
            if (o0 == 0 || dim_tile < d)  // the samples stay when every coordinate fits
                for (int e = tid; e < dc * TS; e += 256) {
                    const int s = e / dc, c = e - s * dc;
                    Bs[c * LB + s] = s < rows ? x[(s0 + s) * d + c0 + c] : T(0);
                }
            for (int e = tid; e < dc * kRegObs; e += 256) {
                const int c = e / kRegObs, o = e - c * kRegObs;
                Xs[c * LX + o] = o0 + o < nobs ? X[(size_t)(c0 + c) * nobs + o0 + o] : T(0);
            }
            __syncthreads();
            if (o0 == 0 && tx == 0)
                for (int c = 0; c < dc; ++c)
#pragma unroll
                    for (int i = 0; i < RS; ++i) {
                        const T b = Bs[c * LB + ty * RS + i];
                        bb[i] += b * b;
                    }
#pragma unroll 4
            for (int c = 0; c < dc; ++c) {
                __align__(16) T b[RS], v[4];
                reg_load(Bs + c * LB + ty * RS, b);
                reg_load(Xs + c * LX + tx * 4, v);
#pragma unroll
                for (int i = 0; i < RS; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) eta[i][j] += v[j] * b[i];
            }
        }
        T yv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) yv[j] = o0 + tx * 4 + j < nobs ? y[o0 + tx * 4 + j] : T(0);
#pragma unroll
        for (int i = 0; i < RS; ++i) {
            T sum = T(0);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (o0 + tx * 4 + j >= nobs) continue;
                const T e = eta[i][j];
                if (logistic) {
                    const T f = dexp(-fabs(e));
                    prod[i] += prod[i] * f + f;
                    sum += yv[j] * e - (e > T(0) ? e : isnan(e) ? e : T(0));
                } else {
                    const T r = yv[j] - e;
                    sum += r * r;
                }
            }
            acc[i].add(sum);
        }
        if (logistic && (++steps % kRegFlush == 0 || o0 + kRegObs >= nobs))
#pragma unroll
            for (int i = 0; i < RS; ++i) {
                acc[i].add(-dlog1p(prod[i]));
                prod[i] = T(0);
            }
    }
#pragma unroll
    for (int i = 0; i < RS; ++i)
        for (int off = 8; off > 0; off >>= 1) acc[i].join(off);
    if (tx == 0)
#pragma unroll
        for (int i = 0; i < RS; ++i)
            if (ty * RS + i < rows) out[s0 + ty * RS + i] = constant + scale * acc[i].value() + prior_scale * bb[i];
}

// Few samples: a warp per sample, four observations per lane in flight, X straight
// from global memory (coalesced; a CTA's four warps share its lines). The tiles above
// put 16 samples on an SM, whose FP64 pipe bounds them: at 1,000 samples x 500
// observations, d = 33, Gaussian, they take 88 us, this 49.
constexpr int kRegRows = 4;  // warps, one per sub-partition
constexpr int kRegFew = 32;  // samples per SM below which FP64 takes them
template <typename T, bool LOGISTIC>
__global__ void __launch_bounds__(32 * kRegRows) target_regression_rows_kernel(issm_target t, const T *__restrict__ x,
                                                                              int64_t n, T constant, T scale,
                                                                              T prior_scale, T *__restrict__ out) {
    constexpr int kAhead = 4;  // coordinates whose loads are in flight together
    const int d = t.dim, nobs = t.count, lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * kRegRows + (threadIdx.x >> 5);
    if (i >= n) return;
    const T *X = (const T *)t.a, *y = (const T *)t.b, *b = x + i * d;
    T acc = T(0), prod = T(0), bb = T(0);
    for (int c = lane; c < d; c += 32) bb += b[c] * b[c];
    int steps = 0;
    for (int o0 = lane; o0 < nobs; o0 += 128) {
        T eta[4] = {T(0), T(0), T(0), T(0)};
        const T *xo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) xo[j] = X + min(o0 + 32 * j, nobs - 1);
        int c = 0;
#pragma unroll 1
        for (; c + kAhead <= d; c += kAhead) {
            T v[kAhead], xv[kAhead][4];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                v[u] = b[c + u];
#pragma unroll
                for (int j = 0; j < 4; ++j) xv[u][j] = xo[j][(size_t)(c + u) * nobs];
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
#pragma unroll
                for (int j = 0; j < 4; ++j) eta[j] += xv[u][j] * v[u];
        }
#pragma unroll 1
        for (; c < d; ++c) {
            const T v = b[c];
#pragma unroll
            for (int j = 0; j < 4; ++j) eta[j] += xo[j][(size_t)c * nobs] * v;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (o0 + 32 * j >= nobs) continue;
            const T yv = y[o0 + 32 * j], e = eta[j];
            if constexpr (LOGISTIC) {
                const T f = dexp(-fabs(e));
                prod += prod * f + f;
                acc += yv * e - (e > T(0) ? e : isnan(e) ? e : T(0));
            } else {
                const T r = yv - e;
                acc += r * r;
            }
        }
        if (LOGISTIC && ++steps % kRegFlush == 0) {
            acc -= dlog1p(prod);
            prod = T(0);
        }
    }
    if (LOGISTIC) acc -= dlog1p(prod);
    for (int off = 16; off > 0; off >>= 1) {
        acc += __shfl_xor_sync(0xffffffffu, acc, off);
        bb += __shfl_xor_sync(0xffffffffu, bb, off);
    }
    if (lane == 0) out[i] = constant + scale * acc + prior_scale * bb;
}

template <typename T, int RS>
static int launch_regression(const issm_target *t, const T *x, int64_t n, T *out, cudaStream_t stream) {
    const double pv = (double)(T)t->p1, sg = (double)(T)t->p0;
    const bool logistic = t->kind == ISSM_TARGET_LOGISTIC;
    const double constant = -0.5 * t->dim * (kLog2Pi + log(pv)) -
                            (logistic ? 0.0 : 0.5 * t->count * (kLog2Pi + 2.0 * log(sg)));
    const double scale = logistic ? 1.0 : -1.0 / (2.0 * sg * sg);
    const int dim_tile = min(t->dim, kRegDim);
    const size_t smem = sizeof(T) * (size_t)dim_tile * (16 * RS + 16 / sizeof(T) + kRegObs);
    if constexpr (sizeof(T) == 8 && RS == 1)
        if (n < kRegFew * (int64_t)device_sms()) {
            const unsigned ctas = (unsigned)((n + kRegRows - 1) / kRegRows);
            auto rows = logistic ? target_regression_rows_kernel<T, true> : target_regression_rows_kernel<T, false>;
            rows<<<ctas, 32 * kRegRows, 0, stream>>>(*t, x, n, (T)constant, (T)scale, (T)(-1.0 / (2.0 * pv)), out);
            note_launch();
            return (int)cudaGetLastError();
        }
    auto kern = target_regression_kernel<T, RS>;
    if (smem > 48 * 1024) {
        const int e = allow_dynamic_smem((const void *)kern);
        if (e) return e;
    }
    const int64_t blocks = (n + 16 * RS - 1) / (16 * RS);
    kern<<<(unsigned)blocks, 256, smem, stream>>>(*t, x, n, (T)constant, (T)scale, (T)(-1.0 / (2.0 * pv)), dim_tile, out);
    note_launch();
    return (int)cudaGetLastError();
}

// The most samples per CTA that still give every SM two CTAs: more FMAs per
// shared load (RS x 4 per RS + 4 words) against idle SMs.
template <typename T>
static int regression_logdensity(const issm_target *t, const T *x, int64_t n, T *out, cudaStream_t stream) {
    const int64_t ctas = 2 * (int64_t)device_sms();
    if (sizeof(T) == 4 && n >= ctas * 128) return launch_regression<T, 8>(t, x, n, out, stream);
    if (n >= ctas * 64) return launch_regression<T, 4>(t, x, n, out, stream);
    if (n >= ctas * 32) return launch_regression<T, 2>(t, x, n, out, stream);
    return launch_regression<T, 1>(t, x, n, out, stream);
}

int target_logdensity(const issm_target *t, const void *x, int64_t n, void *out, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (t->kind == ISSM_TARGET_LINREG || t->kind == ISSM_TARGET_LOGISTIC) {
        if (t->dtype == ISSM_F32) return regression_logdensity<float>(t, (const float *)x, n, (float *)out, stream);
        return regression_logdensity<double>(t, (const double *)x, n, (double *)out, stream);
    } else {
        if (t->kind == ISSM_TARGET_STUDENT_T && t->dim > 64) return ISSM_E_UNSUPPORTED;
        const int blocks = grid_for(n, 128, 8);
        if (t->dtype == ISSM_F32)
            { target_simple_kernel<float><<<blocks, 128, 0, stream>>>(*t, (const float *)x, n, (float *)out); note_launch(); }
        else
            { target_simple_kernel<double><<<blocks, 128, 0, stream>>>(*t, (const double *)x, n, (double *)out); note_launch(); }
    }
    return (int)cudaGetLastError();
}

}  // namespace issm
