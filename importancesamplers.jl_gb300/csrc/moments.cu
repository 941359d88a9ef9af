// moments.cu — weighted mean / covariance of the retained samples and the
// FP64 candidate fit (ridge, Cholesky, Student-t scaling, lognormalizer).
//
// weighted_moments is a two-pass restatement of _weighted_moments!
// (src/adaptive_gaussian_execution.jl:268-273): pass 1 the weighted mean about
// `shift`, pass 2 the weighted covariance about that mean. Weights are
// w_i = exp(l_i - max) / S from the device summary words. Sums run in the data
// type within a thread and in FP64 across blocks. fit_factor runs in one CTA
// with the covariance in shared memory (d <= 64).
#include "issm_device.cuh"
#include "issm_internal.h"
#include "ldlt.cuh"
#include "trinv.cuh"

namespace issm {

constexpr int kMomThreads = 256;
constexpr int kCovThreads = 320;  // most threads of a covariance CTA
constexpr int kMomTile = 64;      // samples staged per step of the covariance pass

// CTAs of either pass: 128 samples each (two staged tiles) until every SM has
// two. With 2048 samples per CTA a 10,000-sample round ran on 5 of 152 SMs.
static int moment_blocks(int64_t n) {
    int64_t b = (n + 127) / 128;
    if (b > kSMs * 2) b = kSMs * 2;
    return b < 1 ? 1 : (int)b;
}

// Register tile of the covariance pass: R x R entries per thread over the
// lower triangle of ceil(d / R) x ceil(d / R) tiles. FP32 takes 8 x 8 above
// d = 16 (64 FMAs per four 16-byte shared loads); smaller d would spend most of an 8 x 8
// tile on padding. FP64 runs at 1.7 FMAs per clock and SM here, whatever the
// loads, so it takes the tile with the least padding.
static int cov_tile(int d, int dtype) { return dtype == ISSM_F32 && d > 16 ? 8 : 4; }
static int cov_tiles(int d, int R) {
    const int nb = (d + R - 1) / R;
    return nb * (nb + 1) / 2;
}

size_t moments_workspace_bytes(int64_t n, int d) {
    const int e4 = cov_tiles(d, 4) * 16, e8 = cov_tiles(d, 8) * 64;
    return sizeof(double) * (size_t)moment_blocks(n) * (size_t)(e4 > e8 ? e4 : e8);
}

// Rows lo .. hi - 1 of this CTA: whole tiles of 64, contiguous.
__device__ __forceinline__ void moment_rows(int64_t n, int64_t &lo, int64_t &hi) {
    const int64_t per = ((n + gridDim.x - 1) / gridDim.x + kMomTile - 1) / kMomTile * kMomTile;
    lo = min(n, (int64_t)blockIdx.x * per);
    hi = min(n, lo + per);
}

// Pass 1: partial[b][c] = sum of w (x_c - c0), c0 the centre rounded to T (the
// finish adds the same rounded value back). Thread t owns coordinate t mod d of
// every (256 / d)-th row, so a warp reads consecutive elements. One read of the
// samples; bound by HBM for FP32 (FP64: a subtraction and an FMA per element).
template <typename T>
__global__ void __launch_bounds__(kMomThreads) mean_partial_kernel(const T *__restrict__ x, int d, int64_t n,
                                                                   const T *__restrict__ lw,
                                                                   const double *__restrict__ summary,
                                                                   const double *__restrict__ center,
                                                                   double *__restrict__ partial) {
    __shared__ T wt[kMomThreads];
    __shared__ double red[kMomThreads];
    const T m = (T)summary[0];
    const T inv = (T)(1.0 / summary[1]);
    const int tid = threadIdx.x, R = kMomThreads / d, c = tid % d, r0 = tid / d;
    const bool own = r0 < R;
    const T c0 = (T)center[c];
    T acc = T(0);
    int64_t lo, hi;
    moment_rows(n, lo, hi);
    for (int64_t t0 = lo; t0 < hi; t0 += kMomThreads) {
        const int cnt = (int)min((int64_t)kMomThreads, hi - t0);
        __syncthreads();
        if (tid < cnt) wt[tid] = dexp(lw[t0 + tid] - m) * inv;
        __syncthreads();
        if (own) {
            const T *xp = x + t0 * d + c;
#pragma unroll 8
            for (int r = r0; r < cnt; r += R) acc += wt[r] * (xp[r * d] - c0);
        }
    }
    // the rows' sums in a fixed tree (256 of them one after the other took 15 us at d = 1)
    red[tid] = own ? (double)acc : 0.0;
    int half = 1;
    while (half < R) half <<= 1;
    for (half >>= 1; half > 0; half >>= 1) {
        __syncthreads();
        if (r0 < half && r0 + half < R) red[tid] += red[tid + half * d];
    }
    if (tid < d) partial[(size_t)blockIdx.x * d + tid] = red[tid];
}

// Pass 2: sums of w z z^T, z = x - (mean rounded to T), over the lower
// triangle. A CTA stages 64 samples at a time (coalesced, one rounding per
// element); thread (h, tile, g) holds one R x R register tile and takes every
// (H G)-th staged sample, so the eight lanes of a 16-byte shared-load phase read
// eight rows of an odd number of 16-byte groups (no bank conflicts). Bound by
// FMA issue with shared-memory operands (FP32) or the FP64 pipe. Single
// entries of the full square per thread (two shared loads per FMA) on few CTAs
// took 3.36 ms over the passes of an 8-round FP32 run of 80,056 samples,
// d = 33, against 0.16 ms; FP64 at n = 100,003, d = 20: 0.72 ms against 0.08.
template <typename T, int R>
__global__ void __launch_bounds__(kCovThreads, 2) cov_partial_kernel(const T *__restrict__ x, int d, int64_t n,
                                                                     const T *__restrict__ lw,
                                                                     const double *__restrict__ summary,
                                                                     const double *__restrict__ mean, int tiles, int G,
                                                                     int H, int LD, double *__restrict__ partial) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *z = reinterpret_cast<T *>(smem_raw);   // kMomTile x LD, columns beyond d zero
    T *wt = z + (size_t)kMomTile * LD;        // kMomTile weights
    T *ctr = wt + kMomTile;                   // d
    const int tid = threadIdx.x, B = blockDim.x;
    const T m = (T)summary[0];
    const T inv = (T)(1.0 / summary[1]);
    for (int c = tid; c < d; c += B) ctr[c] = (T)mean[c];
    for (int e = tid; e < kMomTile * LD; e += B) z[e] = T(0);
    const int g = tid % G, unit = tid / G, tile = unit % tiles, h = unit / tiles;
    int br = 0;
    while ((br + 1) * (br + 2) / 2 <= tile) ++br;
    const int bc = tile - br * (br + 1) / 2;
    T acc[R][R];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[i][j] = T(0);
    const int dq = B / d, dr = B - dq * d;  // (row, column) step of B elements
    int64_t lo, hi;
    moment_rows(n, lo, hi);
    for (int64_t t0 = lo; t0 < hi; t0 += kMomTile) {
        const int cnt = (int)min((int64_t)kMomTile, hi - t0);
        __syncthreads();
        const T *xp = x + t0 * d;
        int s = tid / d, c = tid - s * d;
        for (int e = tid; e < cnt * d;) {
            T v[4];
            int at[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {  // four loads in flight
                at[u] = e < cnt * d ? s * LD + c : -1;
                v[u] = at[u] >= 0 ? xp[e] - ctr[c] : T(0);
                e += B;
                s += dq;
                c += dr;
                if (c >= d) {
                    c -= d;
                    ++s;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (at[u] >= 0) z[at[u]] = v[u];
        }
        for (int r = tid; r < cnt; r += B) wt[r] = dexp(lw[t0 + r] - m) * inv;
        __syncthreads();
        for (int q = h < H ? h * G + g : cnt; q < cnt; q += H * G) {
            const T w = wt[q];
            T a[R], b[R];
            constexpr int V = 16 / sizeof(T);
#pragma unroll
            for (int i = 0; i < R; i += V) {
                *reinterpret_cast<uint4 *>(a + i) = *reinterpret_cast<const uint4 *>(z + q * LD + br * R + i);
                *reinterpret_cast<uint4 *>(b + i) = *reinterpret_cast<const uint4 *>(z + q * LD + bc * R + i);
            }
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const T wa = w * a[i];
#pragma unroll
                for (int j = 0; j < R; ++j) acc[i][j] += wa * b[j];
            }
        }
    }
    // the G sample lanes of a tile (adjacent lanes of one warp), then the H groups in order
    const int entries = tiles * R * R;
    double *red = reinterpret_cast<double *>(smem_raw);
    __syncthreads();
    if ((tid & ~31) < H * tiles * G)  // the other warps only staged samples
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < R; ++j) {
                T v = acc[i][j];
                for (int off = G >> 1; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                if (g == 0 && h < H) red[h * entries + tile * (R * R) + i * R + j] = (double)v;
            }
    __syncthreads();
    for (int e = tid; e < entries; e += B) {
        double s = red[e];
        for (int k = 1; k < H; ++k) s += red[k * entries + e];
        partial[(size_t)blockIdx.x * entries + e] = s;
    }
}

// Block partials summed in FP64: 8 lanes per entry, then in lane order.
constexpr int kFinLanes = 8;
__device__ __forceinline__ double finish_sum(const double *__restrict__ partial, int blocks, int entries, int e,
                                             double (*red)[33]) {
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    double acc = 0.0;
    if (e < entries)
        for (int b = ty; b < blocks; b += kFinLanes) acc += partial[(size_t)b * entries + e];
    red[ty][tx] = acc;
    __syncthreads();
    if (ty == 0)
        for (int r = 1; r < kFinLanes; ++r) acc += red[r][tx];
    return acc;
}

// mean = c0 + S1 (the weights sum to one), c0 the centre as the pass rounded it
template <typename T>
__global__ void __launch_bounds__(32 * kFinLanes) mean_finish_kernel(const double *__restrict__ partial, int blocks,
                                                                     int d, const double *__restrict__ center,
                                                                     double *__restrict__ mean) {
    __shared__ double red[kFinLanes][33];
    const int e = blockIdx.x * 32 + (threadIdx.x & 31);
    const double s = finish_sum(partial, blocks, d, e, red);
    if (threadIdx.x < 32 && e < d) mean[e] = (double)(T)center[e] + s;
}

// cov = S2 - delta delta^T with delta = mean - (mean rounded to T), what the
// pass's centre differs from the mean by (zero in FP64)
template <typename T>
__global__ void __launch_bounds__(32 * kFinLanes) cov_finish_kernel(const double *__restrict__ partial, int blocks,
                                                                    int d, int R, int tiles,
                                                                    const double *__restrict__ mean,
                                                                    double *__restrict__ cov) {
    __shared__ double red[kFinLanes][33];
    const int entries = tiles * R * R, e = blockIdx.x * 32 + (threadIdx.x & 31);
    const double s = finish_sum(partial, blocks, entries, e, red);
    if (threadIdx.x >= 32 || e >= entries) return;
    const int tile = e / (R * R), i = e / R % R, j = e % R;
    int br = 0;
    while ((br + 1) * (br + 2) / 2 <= tile) ++br;
    const int r = br * R + i, c = (tile - br * (br + 1) / 2) * R + j;
    if (r >= d || c > r) return;
    const double v = s - (mean[r] - (double)(T)mean[r]) * (mean[c] - (double)(T)mean[c]);
    cov[r + (size_t)c * d] = v;
    cov[c + (size_t)r * d] = v;
}

template <typename T, int R>
static int moments_t(const T *x, int d, int64_t n, const T *lw, const double *summary, const double *shift,
                     double *mean, double *cov, double *partial, cudaStream_t stream) {
    const int blocks = moment_blocks(n), tiles = cov_tiles(d, R);
    // two samples at least for each of the H G lanes of a tile, whose sums are merged
    // afterwards, and no more lanes than a step's samples
    int G = 32;
    while (G > 1 && (tiles * G > kCovThreads || n < 2 * G)) G >>= 1;
    const int H = (int)max((int64_t)1, min((int64_t)(kCovThreads / (tiles * G)), min(n / 2, (int64_t)kMomTile) / G));
    const int threads = max(128, (H * tiles * G + 31) / 32 * 32);
    constexpr int V = 16 / sizeof(T);
    int LD = (d + R - 1) / R * R;
    if (LD / V % 2 == 0) LD += V;  // an odd number of 16-byte groups per row
    const size_t smem = max(sizeof(T) * ((size_t)kMomTile * LD + kMomTile + d),
                            sizeof(double) * (size_t)H * tiles * R * R);
    mean_partial_kernel<T><<<blocks, kMomThreads, 0, stream>>>(x, d, n, lw, summary, shift, partial);
    note_launch();
    mean_finish_kernel<T><<<(d + 31) / 32, 32 * kFinLanes, 0, stream>>>(partial, blocks, d, shift, mean);
    note_launch();
    cov_partial_kernel<T, R><<<blocks, threads, smem, stream>>>(x, d, n, lw, summary, mean, tiles, G, H, LD, partial);
    note_launch();
    cov_finish_kernel<T><<<(tiles * R * R + 31) / 32, 32 * kFinLanes, 0, stream>>>(partial, blocks, d, R, tiles, mean,
                                                                                   cov);
    note_launch();
    return (int)cudaGetLastError();
}

int weighted_moments(const void *x, int d, int64_t n, const void *lw, int dtype, const double *summary,
                     const double *shift, double *mean, double *cov, void *ws, size_t ws_bytes,
                     cudaStream_t stream) {
    if (d > 64) return ISSM_E_UNSUPPORTED;
    if (ws_bytes < moments_workspace_bytes(n, d)) return ISSM_E_WORKSPACE;
    double *partial = (double *)ws;
    if (dtype == ISSM_F64)
        return moments_t<double, 4>((const double *)x, d, n, (const double *)lw, summary, shift, mean, cov, partial,
                                    stream);
    if (cov_tile(d, dtype) == 8)
        return moments_t<float, 8>((const float *)x, d, n, (const float *)lw, summary, shift, mean, cov, partial,
                                   stream);
    return moments_t<float, 4>((const float *)x, d, n, (const float *)lw, summary, shift, mean, cov, partial, stream);
}

// ---- candidate fit ---------------------------------------------------------------
// ridge = reg * tr(L_prev L_prev^T) * c_nu / d with the overflow fallback of
// _factor_scale_aware_ridge (src/adaptive_gaussian_execution.jl:283-301);
// right-looking Cholesky in FP64; factor *= sqrt(1/c_nu) for Student-t
// (src/proposals.jl:73-80); zero upper triangle; lognormalizer and validity
// (:493-528).
template <typename V> __device__ __forceinline__ V warp_sum_all(V v) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Candidate fit of one moment round (src/adaptive_gaussian_execution.jl:283-528):
// cov + ridge I with ridge = reg tr(L_prev L_prev^T) c_nu / d (reg = sqrt(eps(T)),
// c_nu = nu/(nu-2) for Student-t, 1 for Gaussian; when that product is not
// finite the ridge is summed from the scaled factor, as the reference does),
// an FP64 factorisation, Student-t scaling of the factor by sqrt((nu-2)/nu),
// rounding to T, the validity rule and the lognormalizer, plus (optionally)
// the FP32 inverse of the stored factor for the tensor-core forms.
//
// The factorisation is ldlt_lower's; the Cholesky factor is L diag(sqrt(d)).
// The pivots fail exactly when Cholesky's would (d_j <= 0 or not finite).
template <typename T>
__global__ void __launch_bounds__(256) fit_factor_kernel(const double *__restrict__ mean,
                                                         const double *__restrict__ cov, int d,
                                                         const T *__restrict__ prev, double ridge_scale,
                                                         double ridge_fallback_scale, double lognorm_const,
                                                         double tscale, T *out_loc, T *out_factor, T *out_lognorm,
                                                         uint64_t *failures, int64_t failure_index,
                                                         float *out_inverse, double *out_shift) {
    extern __shared__ __align__(16) double A[];  // d x d column-major
    __shared__ double s_red[8];
    __shared__ double s_ridge;
    __shared__ double s_dg[64];
    __shared__ double s_rinv[8];
    __shared__ double s_w[2][8][64];  // w_c[i] = l_ic d_c of a panel (double-buffered by panel)
    __shared__ double s_scale[64];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dd = d * d;
    // ---- stage the covariance with all loads in flight; trace of the previous factor ----
    T tr = T(0);
    for (int e0 = tid; e0 < dd; e0 += 256 * 8) {
        double v[8];
        T pv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + 256 * u;
            v[u] = e < dd ? cov[e] : 0.0;
            pv[u] = e < dd ? prev[e] : T(0);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + 256 * u;
            if (e < dd) {
                A[e] = v[u];
                if (e % d >= e / d) tr += pv[u] * pv[u];  // lower triangle, in T as the reference sums it
            }
        }
    }
    tr = warp_sum_all(tr);
    if (lane == 0) s_red[warp] = (double)tr;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += s_red[w];
        s_ridge = t * ridge_scale;
    }
    __syncthreads();
    double ridge = s_ridge;
    if (!isfinite(ridge)) {
        // the scaled-factor route of _factor_scale_aware_ridge (rare)
        double acc = 0.0;
        if (ridge_fallback_scale != 0.0)
            for (int e = tid; e < dd; e += 256)
                if (e % d >= e / d) {
                    const double v = (double)prev[e] * ridge_fallback_scale;
                    acc += v * v;
                }
        acc = warp_sum_all(acc);
        __syncthreads();
        if (lane == 0) s_red[warp] = acc;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < 8; ++w) t += s_red[w];
            s_ridge = t;
        }
        __syncthreads();
        ridge = s_ridge;
    }
    for (int c = tid; c < d; c += 256) A[c + c * d] += ridge;
    __syncthreads();

    ldlt_lower(A, d, s_dg, s_rinv, s_w);

    // ---- factor = L diag(sqrt(d)) * Student-t scale, rounded to T ----
    int invalid = 0;
    for (int c = tid; c < d; c += 256) {
        const double dg = s_dg[c];
        invalid |= !(dg > 0.0) || !isfinite(dg);
        s_scale[c] = sqrt(dg) * tscale;
    }
    __syncthreads();
    constexpr int LDI = 65;
    float *Lf = reinterpret_cast<float *>(A + dd);  // FP32 copy of the stored factor for the inverse
    // a warp per column; the FP64 products only where a half of it reaches below the diagonal
    for (int c = warp; c < d; c += 8) {
        const double sc = s_scale[c];
#pragma unroll
        for (int h = 0; h < 64; h += 32) {
            const int r = h + lane;
            T v = T(0);
            if (h + 31 > c && h < d) v = (T)(A[min(r, d - 1) + c * d] * sc);
            if (r <= c) v = r == c ? (T)sc : T(0);
            if (r < d) {
                out_factor[r + (size_t)c * d] = v;
                if (out_inverse != nullptr) Lf[r * LDI + c] = (float)v;
                if (r > c) invalid |= !isfinite(v);
            }
        }
    }
    // log|L_jj| in the factor's own precision, summed across lanes then in FP64
    T lg = T(0);
    for (int c = tid; c < d; c += 256) {
        const T v = (T)s_scale[c];
        invalid |= !isfinite(v) || !(v > T(0));
        lg += dlog(fabs(v));
    }
    for (int c = tid; c < d; c += 256) {
        const T v = (T)mean[c];
        out_loc[c] = v;
        if (out_shift != nullptr) out_shift[c] = (double)v;
        invalid |= !isfinite(v);
    }
    lg = warp_sum_all(lg);
    if (lane == 0) s_red[warp] = (double)lg;
    invalid = __syncthreads_or(invalid);
    if (tid == 0) {
        double logabsdet = 0.0;
        for (int w = 0; w < 8; ++w) logabsdet += s_red[w];
        const double ln = lognorm_const - logabsdet;
        *out_lognorm = (T)ln;
        const bool valid = !invalid && isfinite((T)ln);
        if (!valid) record_failure(failures, failure_index, 0, ISSM_REASON_MOMENT_FIT_INVALID);
    }
    // inverse factor for the tensor-core forms: W = (stored factor)^-1 in
    // FP32, DP x DP row-major zero padded
    if (out_inverse != nullptr) {
        float *Wf = Lf + 64 * LDI;
        __syncthreads();
        invert_lower_f32(Lf, Wf, d, LDI);
        const int DP = d <= 16 ? 16 : d <= 32 ? 32 : 64;
        for (int e = tid; e < DP * DP; e += 256) {
            const int j = e / DP, c = e % DP;
            out_inverse[e] = (j < d && c < d) ? Wf[j * LDI + c] : 0.f;
        }
    }
}

int fit_factor(const double *mean, const double *cov, int d, const void *prev, double dof, double logconst,
               int dtype, void *out_loc, void *out_factor, void *out_lognorm, uint64_t *failures,
               int64_t failure_index, float *out_inverse, double regularization, cudaStream_t stream,
               double *out_shift) {
    if (d > 64) return ISSM_E_UNSUPPORTED;
    size_t smem = sizeof(double) * (size_t)d * d;
    if (out_inverse != nullptr) {
        smem += sizeof(float) * 2 * 64 * 65;
        const int e = allow_dynamic_smem(dtype == ISSM_F32 ? (const void *)fit_factor_kernel<float>
                                                           : (const void *)fit_factor_kernel<double>);
        if (e) return e;
    }
    // scalar constants formed once on the host
    const double mult = dof > 0.0 ? dof / (dof - 2.0) : 1.0;
    // sqrt(eps(T)) of the factor type unless the caller gives the coefficient
    const double reg = regularization >= 0.0 ? regularization
                       : dtype == ISSM_F32 ? sqrt((double)FLT_EPSILON) : sqrt(DBL_EPSILON);
    const double ridge_scale = reg * mult / (double)d;
    const double ridge_fallback = reg != 0.0 ? sqrt(reg) * sqrt(mult / (double)d) : 0.0;
    const double lognorm_const = dof > 0.0 ? logconst : -0.5 * (double)d * log(2.0 * 3.14159265358979323846);
    const double tscale = dof > 0.0 ? sqrt(1.0 / mult) : 1.0;
    if (dtype == ISSM_F32) {
        { fit_factor_kernel<float><<<1, 256, smem, stream>>>(mean, cov, d, (const float *)prev, ridge_scale,
                                                           ridge_fallback, lognorm_const, tscale, (float *)out_loc,
                                                           (float *)out_factor, (float *)out_lognorm, failures,
                                                           failure_index, out_inverse, out_shift); note_launch(); }
    } else {
        { fit_factor_kernel<double><<<1, 256, smem, stream>>>(mean, cov, d, (const double *)prev, ridge_scale,
                                                            ridge_fallback, lognorm_const, tscale,
                                                            (double *)out_loc, (double *)out_factor,
                                                            (double *)out_lognorm, failures, failure_index,
                                                            out_inverse, out_shift); note_launch(); }
    }
    return (int)cudaGetLastError();
}

}  // namespace issm
