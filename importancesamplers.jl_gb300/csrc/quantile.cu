// quantile.cu — component-wise weighted quantiles with the StatsBase generic-
// weight interpolation rule of _weighted_quantile (src/statistics.jl:114-154),
// which the reference evaluates on the host after sorting. Here no sort of the
// samples: for every (coordinate, probability) the element at which the
// cumulative weight of the value-sorted positive-weight samples first exceeds
// the threshold p (W - w_first) + w_first is found by narrowing an interval of
// order-preserving keys (see select.cu) until at most kQCand samples are left,
// which one CTA sorts.
//
//   setup    weights e^{l-m}/S once per sample (FP64), W, and per coordinate the
//            least and greatest key and the first index of the least;
//   level 0  2,048 buckets linear in the value (in FP32, which is monotone:
//            continuous samples spread over hundreds of buckets, where the
//            leading bits of their keys would put most of them in a few),
//            shared by every probability of a coordinate; the chosen bucket's
//            key interval is found by a search over keys;
//   level k  2,048 equal parts of the key interval, for problems that still
//            hold more than kQCand samples (ties, clusters, millions of samples);
//   gather   the samples of the interval and the greatest key below it;
//   finish   sort by (key, index), cumulative weights, the interpolation.
//
// Bound by the column reads (sectors of four coordinates) and FP64 exponentials;
// at n = 100,003, d = 20, three probabilities, FP64 the 8-bit digit passes with
// per-element exponentials, contended shared FP64 atomics and a serial bin
// walk took 7,300 us.
#include "issm_device.cuh"
#include "issm_internal.h"

namespace issm {

template <typename T> struct QKey;
template <> struct QKey<float> {
    static constexpr int kBits = 32;
    __device__ static unsigned long long key(float v) {
        const uint32_t u = __float_as_uint(v);
        return (unsigned long long)((u & 0x80000000u) ? ~u : (u | 0x80000000u));
    }
    __device__ static float value(unsigned long long k) {
        const uint32_t u = (uint32_t)k;
        return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
    }
};
template <> struct QKey<double> {
    static constexpr int kBits = 64;
    __device__ static unsigned long long key(double v) {
        const unsigned long long u = (unsigned long long)__double_as_longlong(v);
        return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
    }
    __device__ static double value(unsigned long long k) {
        return __longlong_as_double((long long)((k & 0x8000000000000000ull) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
    }
};

constexpr int kQThreads = 256;
constexpr int kQBins = 2048;
constexpr int kQPer = kQBins / kQThreads;  // bins per thread of a scan
constexpr int kQCand = 1024;               // samples of an interval that the finish sorts
constexpr int kQCols = 4;                  // coordinates per CTA of level 0 and the gather (a sector of FP64)
constexpr int kQSetupBlocks = 2 * kSMs;
constexpr int64_t kQWeights = 1 << 21;     // weights kept in the workspace; beyond, recomputed by each pass

struct QBins {
    double w[kQBins];
    unsigned n[kQBins];
};
struct QColumn {  // per coordinate
    unsigned long long kmin, kmax;
    double w_first;
    float lo, scale;  // level 0: bucket = (v - lo) scale
    int nan;
};
struct QProblem {  // per (probability, coordinate)
    unsigned long long ka, kb;  // the interval, inclusive
    double thr, below;          // threshold; weight below ka
    unsigned long long klow;    // greatest key below ka (0: none)
    unsigned long long first;   // least index holding ka
    unsigned count, found;      // samples in the interval; candidates gathered
    int ready, beyond;          // no more levels; threshold not exceeded (the largest value)
    unsigned done;              // CTAs of the running level that have added their bins
};
struct QCandidates {
    unsigned long long key[kQCand];
    double w[kQCand];
    long long index[kQCand];
};
struct QPartial {  // setup, per CTA and coordinate
    unsigned long long kmin, kmax;
    long long imin;
    int nan;
};

// One workspace for d coordinates and P = d nprob problems.
struct QWork {
    double *weights, *wsum;  // kQWeights; per setup CTA
    unsigned *counter;
    QColumn *col;
    QProblem *prob;
    QBins *bins0, *bins;
    QCandidates *cand;
    QPartial *part;
};
static size_t q_up(size_t v) { return (v + 255) & ~(size_t)255; }
static size_t q_layout(char *base, int d, int nprob, QWork *w) {
    const size_t P = (size_t)d * (size_t)nprob;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        char *p = base + o;
        o += q_up(bytes);
        return p;
    };
    QWork t;
    t.weights = (double *)take(sizeof(double) * kQWeights);
    t.wsum = (double *)take(sizeof(double) * kQSetupBlocks);
    t.counter = (unsigned *)take(256);
    t.col = (QColumn *)take(sizeof(QColumn) * (size_t)d);
    t.prob = (QProblem *)take(sizeof(QProblem) * P);
    t.bins0 = (QBins *)take(sizeof(QBins) * (size_t)d);
    t.bins = (QBins *)take(sizeof(QBins) * P);
    t.cand = (QCandidates *)take(sizeof(QCandidates) * P);
    t.part = (QPartial *)take(sizeof(QPartial) * (size_t)kQSetupBlocks * (size_t)d);
    if (w) *w = t;
    return o;
}

__device__ __forceinline__ double qweight(double l, double m, double inv) {
    return l == -INFINITY ? 0.0 : exp(l - m) * inv;
}

// exclusive prefix of v over the CTA's threads, in thread order
__device__ __forceinline__ double q_exclusive(double v, double *total) {
    __shared__ double ws[kQThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    __syncthreads();
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    double base = 0.0, all = 0.0;
    for (int k = 0; k < kQThreads / 32; ++k) {
        if (k == warp) base = all;
        all += ws[k];
    }
    *total = all;
    const double ex = __shfl_up_sync(0xffffffffu, inc, 1);
    return base + (lane ? ex : 0.0);
}

// level-0 bucket of a value: monotone in v (every operation is)
template <typename T> __device__ __forceinline__ int q_bucket(T v, float lo, float scale) {
    const float t = ((float)v - lo) * scale;
    return (int)fminf(fmaxf(t, 0.f), (float)(kQBins - 1));
}

// ---- setup -------------------------------------------------------------------
// A warp takes 32 rows: lanes form the rows' weights, then lanes are columns
// (coalesced) and the rows follow one another.
template <typename T>
__global__ void __launch_bounds__(kQThreads) quantile_setup_kernel(const T *__restrict__ x, int d, int64_t n,
                                                                   const T *__restrict__ lw,
                                                                   const double *__restrict__ summary,
                                                                   const double *__restrict__ probs, int nprob,
                                                                   QWork q) {
    using QK = QKey<T>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = kQThreads / 32;
    const double m = summary[0], inv = 1.0 / summary[1];
    __shared__ unsigned long long s_min[kQThreads], s_max[kQThreads];
    __shared__ long long s_idx[kQThreads];
    __shared__ int s_nan[kQThreads];
    __shared__ double s_w[kQThreads / 32];
    __shared__ bool last;
    // bins and states start at zero
    const size_t nb = sizeof(QBins) / 16 * (size_t)d, np = sizeof(QBins) / 16 * (size_t)d * nprob;
    const size_t t0 = (size_t)blockIdx.x * kQThreads + threadIdx.x, ts = (size_t)gridDim.x * kQThreads;
    for (size_t e = t0; e < nb; e += ts) reinterpret_cast<uint4 *>(q.bins0)[e] = make_uint4(0u, 0u, 0u, 0u);
    for (size_t e = t0; e < np; e += ts) reinterpret_cast<uint4 *>(q.bins)[e] = make_uint4(0u, 0u, 0u, 0u);
    double wsum = 0.0;
    const int64_t groups = (n + 31) / 32;
    for (int c0 = 0; c0 < d; c0 += 32) {
        const int c = c0 + lane;
        unsigned long long kmin = ~0ull, kmax = 0ull;
        long long imin = LLONG_MAX;
        int nan = 0;
        for (int64_t g = (int64_t)blockIdx.x * W + warp; g < groups; g += (int64_t)gridDim.x * W) {
            const int64_t i0 = g * 32, i = i0 + lane;
            double w = 0.0;
            if (i < n) {
                if (c0 == 0 || n > kQWeights) w = qweight((double)lw[i], m, inv);
                else w = q.weights[i];
                if (c0 == 0) {
                    if (n <= kQWeights) q.weights[i] = w;
                    wsum += w;
                }
            }
            const unsigned live = __ballot_sync(0xffffffffu, w > 0.0);
            const int rows = (int)min((int64_t)32, n - i0);
            if (c < d) {
#pragma unroll 8
                for (int r = 0; r < rows; ++r) {
                    const T v = x[(i0 + r) * d + c];
                    if (isnan(v)) {
                        nan = 1;
                    } else if (live >> r & 1u) {
                        const unsigned long long k = QK::key(v);
                        if (k < kmin) {  // rows ascend within a thread: the first index stays
                            kmin = k;
                            imin = i0 + r;
                        }
                        kmax = max(kmax, k);
                    }
                }
            }
        }
        __syncthreads();
        s_min[threadIdx.x] = kmin;
        s_max[threadIdx.x] = kmax;
        s_idx[threadIdx.x] = imin;
        s_nan[threadIdx.x] = nan;
        __syncthreads();
        if (warp == 0 && c < d) {
            for (int k = 1; k < W; ++k) {
                const int o = 32 * k + lane;
                if (s_min[o] < kmin || (s_min[o] == kmin && s_idx[o] < imin)) {
                    kmin = s_min[o];
                    imin = s_idx[o];
                }
                kmax = max(kmax, s_max[o]);
                nan |= s_nan[o];
            }
            q.part[(size_t)blockIdx.x * d + c] = QPartial{kmin, kmax, imin, nan};
        }
    }
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if (lane == 0) s_w[warp] = wsum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int k = 0; k < W; ++k) s += s_w[k];
        q.wsum[blockIdx.x] = s;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(q.counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the last CTA: W in block order, the columns' extremes and the problems' thresholds
    double mine = 0.0, total;
    const int per = ((int)gridDim.x + kQThreads - 1) / kQThreads;
    for (int b = threadIdx.x * per; b < min((int)gridDim.x, ((int)threadIdx.x + 1) * per); ++b) mine += __ldcg(q.wsum + b);
    q_exclusive(mine, &total);
    for (int c = warp; c < d; c += W) {  // a warp per column
        unsigned long long kmin = ~0ull, kmax = 0ull;
        long long imin = LLONG_MAX;
        int nan = 0;
        for (int b = lane; b < (int)gridDim.x; b += 32) {
            const QPartial *pp = q.part + (size_t)b * d + c;
            const unsigned long long k = __ldcg(&pp->kmin);
            const long long i = __ldcg(&pp->imin);
            if (k < kmin || (k == kmin && i < imin)) {
                kmin = k;
                imin = i;
            }
            kmax = max(kmax, __ldcg(&pp->kmax));
            nan |= __ldcg(&pp->nan);
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long k = __shfl_xor_sync(0xffffffffu, kmin, o);
            const long long i = __shfl_xor_sync(0xffffffffu, imin, o);
            if (k < kmin || (k == kmin && i < imin)) {
                kmin = k;
                imin = i;
            }
            kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
            nan |= __shfl_xor_sync(0xffffffffu, nan, o);
        }
        if (lane != 0) continue;
        const bool none = imin == LLONG_MAX;  // no positive weight: NaN, as an empty sample gives
        QColumn &col = q.col[c];
        col.kmin = kmin;
        col.kmax = kmax;
        col.nan = nan | (none ? 1 : 0);
        col.w_first = none ? 0.0 : qweight((double)lw[imin], m, inv);
        const float lo = none ? 0.f : fmaxf((float)QK::value(kmin), -3e38f);
        const float hi = none ? 0.f : fminf((float)QK::value(kmax), 3e38f);
        const float scale = (float)kQBins / (hi - lo);
        col.lo = lo;
        col.scale = hi > lo && isfinite(scale) ? scale : 0.f;
        for (int p = 0; p < nprob; ++p) {
            QProblem &s = q.prob[(size_t)p * d + c];
            s.ka = kmin;
            s.kb = kmax;
            s.thr = probs[p] * (total - col.w_first) + col.w_first;
            s.below = 0.0;
            s.klow = 0ull;
            s.first = ~0ull;
            s.count = s.found = s.done = 0u;
            s.ready = s.beyond = 0;
        }
    }
    if (threadIdx.x == 0) *q.counter = 0u;
}

// ---- choosing a bin ------------------------------------------------------------
// The first bin whose cumulative weight (from `below`) exceeds thr; every
// thread returns it (kQBins: none) with the weight below it and its count.
// A thread's starting sum is associated differently from the sum that the thread
// before it ends with, so it may exceed thr by a rounding though no earlier bin
// did: the weight below the bin is then thr itself, as everywhere a sum is chosen.
__device__ __forceinline__ int q_choose(const QBins *bins, double below, double thr, double *under, unsigned *count) {
    __shared__ int s_bin;
    __shared__ double s_under;
    __shared__ unsigned s_count;
    double v[kQPer], sum = 0.0, total;
    for (int k = 0; k < kQPer; ++k) {
        v[k] = __ldcg(&bins->w[threadIdx.x * kQPer + k]);
        sum += v[k];
    }
    double cum = below + q_exclusive(sum, &total);
    __syncthreads();
    if (threadIdx.x == 0) s_bin = kQBins;
    __syncthreads();
    int hit = kQBins;
    double at = 0.0;
    for (int k = 0; k < kQPer; ++k) {
        if (hit == kQBins && v[k] > 0.0 && cum + v[k] > thr) {
            hit = threadIdx.x * kQPer + k;
            at = fmin(cum, thr);
        }
        cum += v[k];
    }
    if (hit < kQBins) atomicMin(&s_bin, hit);
    __syncthreads();
    if (hit == s_bin && hit < kQBins) {
        s_under = at;
        s_count = __ldcg(&bins->n[hit]);
    }
    __syncthreads();
    *under = s_under;
    *count = s_count;
    return s_bin;
}

// least key in [lo, hi] with bucket >= b (hi + 1 if none), by a 32-way search of one warp
template <typename T>
__device__ unsigned long long q_first_key(unsigned long long lo, unsigned long long hi, int b, float clo, float scale) {
    const int lane = threadIdx.x & 31;
    // invariant: keys below lo have smaller buckets; hi + 1 counts as a hit
    unsigned long long end = hi - lo + 1;  // 0 when the interval is the whole 64-bit range (cannot happen: NaNs are out)
    while (end > 0) {
        const unsigned long long step = end / 33 + 1;
        const unsigned long long off = step * (unsigned long long)lane;  // probes lo, lo + step, ...
        const bool in = off < end;
        const bool hit = !in || q_bucket(QKey<T>::value(lo + off), clo, scale) >= b;
        const unsigned ball = __ballot_sync(0xffffffffu, hit);
        if (ball & 1u) return lo;
        const int j = ball ? __ffs(ball) - 1 : 32;  // probe j - 1 misses, probe j (or the end) hits
        const unsigned long long a = step * (unsigned long long)(j - 1) + 1;
        const unsigned long long z = ball ? min(step * (unsigned long long)j, end) : end;
        lo += a;
        end = z - a;
    }
    return lo;
}

__device__ __forceinline__ void q_flush(QBins *dst, const double *w, const unsigned *c) {
    for (int b = threadIdx.x; b < kQBins; b += kQThreads)
        if (c[b]) {
            atomicAdd(&dst->w[b], w[b]);
            atomicAdd(&dst->n[b], c[b]);
        }
}

// ---- level 0: all probabilities of kQCols coordinates -----------------------------
template <typename T>
__global__ void __launch_bounds__(kQThreads) quantile_level0_kernel(const T *__restrict__ x, int d, int64_t n,
                                                                    const T *__restrict__ lw,
                                                                    const double *__restrict__ summary, QWork q) {
    extern __shared__ __align__(16) unsigned char smem[];
    double *bw = reinterpret_cast<double *>(smem);                        // kQCols x kQBins
    unsigned *bn = reinterpret_cast<unsigned *>(bw + kQCols * kQBins);    // kQCols x kQBins
    const int c0 = blockIdx.y * kQCols, nc = min(kQCols, d - c0);
    for (int b = threadIdx.x; b < kQCols * kQBins; b += kQThreads) {
        bw[b] = 0.0;
        bn[b] = 0u;
    }
    float lo[kQCols], scale[kQCols];
#pragma unroll
    for (int j = 0; j < kQCols; ++j) {
        lo[j] = j < nc ? q.col[c0 + j].lo : 0.f;
        scale[j] = j < nc ? q.col[c0 + j].scale : 0.f;
    }
    __syncthreads();
    const double m = summary[0], inv = 1.0 / summary[1];
    const bool kept = n <= kQWeights;
    const int64_t stride = (int64_t)gridDim.x * kQThreads;
    for (int64_t i = (int64_t)blockIdx.x * kQThreads + threadIdx.x; i < n; i += stride) {
        const double w = kept ? q.weights[i] : qweight((double)lw[i], m, inv);
        T v[kQCols];
#pragma unroll
        for (int j = 0; j < kQCols; ++j) v[j] = j < nc ? x[i * d + c0 + j] : T(0);
        if (!(w > 0.0)) continue;
#pragma unroll
        for (int j = 0; j < kQCols; ++j)
            if (j < nc) {
                const int b = j * kQBins + q_bucket(v[j], lo[j], scale[j]);
                atomicAdd(&bw[b], w);
                atomicAdd(&bn[b], 1u);
            }
    }
    __syncthreads();
    for (int j = 0; j < nc; ++j) q_flush(q.bins0 + c0 + j, bw + j * kQBins, bn + j * kQBins);
}

// one CTA per problem: the bucket of level 0 and its key interval
template <typename T> __global__ void __launch_bounds__(kQThreads) quantile_choose0_kernel(int d, QWork q) {
    const int pr = blockIdx.x;
    const QColumn col = q.col[pr % d];
    if (col.nan) return;
    QProblem &s = q.prob[pr];
    double under;
    unsigned count;
    const int b = q_choose(q.bins0 + pr % d, 0.0, s.thr, &under, &count);
    if (threadIdx.x >= 32) return;
    if (b == kQBins) {
        if (threadIdx.x == 0) {
            s.beyond = 1;  // rounding left the threshold at or above W
            s.ready = 1;
        }
        return;
    }
    const unsigned long long ka = q_first_key<T>(col.kmin, col.kmax, b, col.lo, col.scale);
    const unsigned long long kz =
        b + 1 < kQBins ? q_first_key<T>(ka, col.kmax, b + 1, col.lo, col.scale) : col.kmax + 1;
    if (threadIdx.x == 0) {
        s.ka = ka;
        s.kb = kz - 1;
        s.below = under;
        s.count = count;
        s.ready = count <= (unsigned)kQCand || kz - 1 == ka;
    }
}

// ---- further levels: one problem per blockIdx.y ------------------------------------
template <typename T>
__global__ void __launch_bounds__(kQThreads) quantile_level_kernel(const T *__restrict__ x, int d, int64_t n,
                                                                   const T *__restrict__ lw,
                                                                   const double *__restrict__ summary, QWork q) {
    const int pr = blockIdx.y, c = pr % d;
    QProblem &s = q.prob[pr];
    if (s.ready || q.col[c].nan) return;
    __shared__ double bw[kQBins];
    __shared__ unsigned bn[kQBins];
    __shared__ bool last;
    for (int b = threadIdx.x; b < kQBins; b += kQThreads) {
        bw[b] = 0.0;
        bn[b] = 0u;
    }
    const unsigned long long ka = s.ka, kb = s.kb;
    const int shift = max(0, 64 - __clzll((long long)(kb - ka)) - 11);
    __syncthreads();
    const double m = summary[0], inv = 1.0 / summary[1];
    const bool kept = n <= kQWeights;
    const int64_t stride = (int64_t)gridDim.x * kQThreads;
    for (int64_t i = (int64_t)blockIdx.x * kQThreads + threadIdx.x; i < n; i += stride) {
        const unsigned long long k = QKey<T>::key(x[i * d + c]);
        if (k < ka || k > kb) continue;
        const double w = kept ? q.weights[i] : qweight((double)lw[i], m, inv);
        if (!(w > 0.0)) continue;
        const int b = (int)((k - ka) >> shift);
        atomicAdd(&bw[b], w);
        atomicAdd(&bn[b], 1u);
    }
    __syncthreads();
    q_flush(q.bins + pr, bw, bn);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&s.done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    double under;
    unsigned count;
    const int b = q_choose(q.bins + pr, s.below, s.thr, &under, &count);
    for (int e = threadIdx.x; e < kQBins; e += kQThreads) {
        q.bins[pr].w[e] = 0.0;
        q.bins[pr].n[e] = 0u;
    }
    if (threadIdx.x == 0) {
        s.done = 0u;
        if (b == kQBins) {
            // the parts' sums rounded below the whole's: the interval's last key, if anything follows nothing
            s.beyond = 2;
            s.ready = 1;
        } else {
            s.ka = ka + ((unsigned long long)b << shift);
            s.kb = s.ka + min(kb - s.ka, (1ull << shift) - 1ull);  // the sum of the two could pass 2^64
            s.below = under;
            s.count = count;
            s.ready = count <= (unsigned)kQCand || s.kb == s.ka;
        }
    }
}

// ---- the samples of the intervals -----------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kQThreads) quantile_gather_kernel(const T *__restrict__ x, int d, int64_t n,
                                                                    const T *__restrict__ lw,
                                                                    const double *__restrict__ summary, int nprob,
                                                                    QWork q) {
    const int c0 = blockIdx.y * kQCols, nc = min(kQCols, d - c0);
    const double m = summary[0], inv = 1.0 / summary[1];
    const bool kept = n <= kQWeights;
    const int64_t stride = (int64_t)gridDim.x * kQThreads;
    const int lane = threadIdx.x & 31;
    for (int p = 0; p < nprob; ++p) {
        unsigned long long ka[kQCols], kb[kQCols], low[kQCols], first[kQCols];
        bool top[kQCols], tied[kQCols], any = false;
#pragma unroll
        for (int j = 0; j < kQCols; ++j) {
            ka[j] = 1ull;
            kb[j] = 0ull;
            low[j] = 0ull;
            first[j] = ~0ull;
            top[j] = tied[j] = false;
            if (j < nc && !q.col[c0 + j].nan) {
                const QProblem &s = q.prob[(size_t)p * d + c0 + j];
                if (s.beyond == 2) {  // its answer is the greatest key of the interval
                    ka[j] = s.kb + 1ull;
                } else if (s.beyond == 0) {
                    ka[j] = s.ka;
                    kb[j] = s.kb;
                    tied[j] = s.count > (unsigned)kQCand;  // one key: only its first index matters
                    top[j] = !tied[j];
                } else {
                    continue;
                }
                any = true;
            }
        }
        if (!any) continue;
        for (int64_t i = (int64_t)blockIdx.x * kQThreads + threadIdx.x; i < n; i += stride) {
            T v[kQCols];
#pragma unroll
            for (int j = 0; j < kQCols; ++j) v[j] = j < nc ? x[i * d + c0 + j] : T(0);
            const double w = kept ? q.weights[i] : lw[i] == -num<T>::inf() ? 0.0 : qweight((double)lw[i], m, inv);
            if (!(w > 0.0)) continue;
#pragma unroll
            for (int j = 0; j < kQCols; ++j) {
                const unsigned long long k = QKey<T>::key(v[j]);
                if (k < ka[j]) {
                    if (j < nc) low[j] = max(low[j], k);
                } else if (top[j] && k <= kb[j]) {
                    QProblem &s = q.prob[(size_t)p * d + c0 + j];
                    const unsigned at = atomicAdd(&s.found, 1u);
                    if (at < (unsigned)kQCand) {
                        QCandidates &cd = q.cand[(size_t)p * d + c0 + j];
                        cd.key[at] = k;
                        cd.w[at] = w;
                        cd.index[at] = i;
                    }
                } else if (tied[j] && k == ka[j]) {
                    first[j] = min(first[j], (unsigned long long)i);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kQCols; ++j) {
            unsigned long long v = low[j];
            for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (lane == 0 && v != 0ull && j < nc) atomicMax(&q.prob[(size_t)p * d + c0 + j].klow, v);
            unsigned long long f = first[j];
            for (int o = 16; o > 0; o >>= 1) f = min(f, __shfl_xor_sync(0xffffffffu, f, o));
            if (lane == 0 && f != ~0ull && j < nc) atomicMin(&q.prob[(size_t)p * d + c0 + j].first, f);
        }
    }
}

// lower + f (upper - lower) as _weighted_quantile forms it (src/statistics.jl:140-153),
// f = (thr - at) / w with at <= thr < at + w up to the rounding of the sums
__device__ __forceinline__ double q_interpolate(double lo, double up, double thr, double at, double w) {
    const double f = fmin((thr - at) / w, 1.0);
    if (f == 0.0) return lo;
    if (f == 1.0) return up;
    const double diff = up - lo;
    return isfinite(diff) ? fmin(lo + f * diff, up) : (1.0 - f) * lo + f * up;
}

// ---- one CTA per problem: sort the interval's samples, select, interpolate --------------
template <typename T>
__global__ void __launch_bounds__(kQThreads) quantile_finish_kernel(int d, const T *__restrict__ lw,
                                                                    const double *__restrict__ summary,
                                                                    const QWork q, double *__restrict__ out) {
    using QK = QKey<T>;
    const int pr = blockIdx.x, c = pr % d, tid = threadIdx.x;
    const QProblem &s = q.prob[pr];
    if (q.col[c].nan || s.beyond) {
        if (tid == 0)
            out[pr] = q.col[c].nan ? nan("") : (double)(T)QK::value(s.beyond == 2 ? s.klow : q.col[c].kmax);
        return;
    }
    const unsigned long long klow = s.klow;
    if (s.count > (unsigned)kQCand) {
        // more ties of one key than are gathered: only its first index can interpolate from below
        if (tid == 0) {
            const double up = (double)QK::value(s.ka);
            const double w = qweight((double)lw[s.first], summary[0], 1.0 / summary[1]);
            double v = up;
            if (klow != 0ull && s.below + w > s.thr) v = q_interpolate((double)QK::value(klow), up, s.thr, s.below, w);
            out[pr] = (double)(T)v;
        }
        return;
    }
    __shared__ unsigned long long key[kQCand];
    __shared__ long long idx[kQCand];
    __shared__ double w[kQCand];
    __shared__ unsigned short ord[kQCand];
    __shared__ int s_hit;
    const int m = (int)min(s.found, (unsigned)kQCand);
    int size = 1;
    while (size < m) size <<= 1;
    for (int e = tid; e < size; e += kQThreads) {
        const bool in = e < m;
        key[e] = in ? q.cand[pr].key[e] : ~0ull;
        idx[e] = in ? q.cand[pr].index[e] : LLONG_MAX;
        w[e] = in ? q.cand[pr].w[e] : 0.0;
        ord[e] = (unsigned short)e;
    }
    if (tid == 0) s_hit = m;
    __syncthreads();
    for (int k = 2; k <= size; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int e = tid; e < size; e += kQThreads) {
                const int o = e ^ j;
                if (o <= e) continue;
                const int a = ord[e], b = ord[o];
                const bool gt = key[a] > key[b] || (key[a] == key[b] && idx[a] > idx[b]);
                if (gt == ((e & k) == 0)) {
                    ord[e] = (unsigned short)b;
                    ord[o] = (unsigned short)a;
                }
            }
            __syncthreads();
        }
    // cumulative weights in sorted order: kQCand / kQThreads consecutive samples per thread
    constexpr int kPer = kQCand / kQThreads;
    double sum = 0.0, total;
    for (int u = 0; u < kPer; ++u) {
        const int e = tid * kPer + u;
        if (e < m) sum += w[ord[e]];
    }
    double cum = s.below + q_exclusive(sum, &total);
    int hit = m;
    double at = 0.0;
    for (int u = 0; u < kPer; ++u) {
        const int e = tid * kPer + u;
        if (e >= m) break;
        const double we = w[ord[e]];
        if (hit == m && cum + we > s.thr) {
            hit = e;
            at = fmin(cum, s.thr);  // as in q_choose
        }
        cum += we;
    }
    if (hit < m) atomicMin(&s_hit, hit);
    __syncthreads();
    if (s_hit < m) {
        if (hit != s_hit) return;
        const double up = (double)QK::value(key[ord[hit]]);
        double v = up;
        if (hit > 0 || klow != 0ull) {
            const double lo = (double)QK::value(hit > 0 ? key[ord[hit - 1]] : klow);
            v = q_interpolate(lo, up, s.thr, at, w[ord[hit]]);
        }
        out[pr] = (double)(T)v;
    } else if (tid == 0) {  // the sorted sums rounded below the bins': the interval's last sample
        out[pr] = (double)(T)QK::value(m > 0 ? key[ord[m - 1]] : klow);
    }
}

size_t weighted_quantile_workspace_bytes(int d, int nprob) { return q_layout(nullptr, d, nprob, nullptr); }

template <typename T>
static int weighted_quantile_t(const T *x, int d, int64_t n, const T *lw, const double *summary, const double *probs,
                               int nprob, double *out, void *ws, cudaStream_t stream) {
    QWork q;
    q_layout((char *)ws, d, nprob, &q);
    const int P = d * nprob, sms = device_sms(), cg = (d + kQCols - 1) / kQCols;
    cudaError_t e = cudaMemsetAsync(q.counter, 0, sizeof(unsigned), stream);
    if (e != cudaSuccess) return (int)e;
    const int setup = (int)min((int64_t)sms * 2, (n + kQThreads - 1) / kQThreads);
    quantile_setup_kernel<T><<<setup, kQThreads, 0, stream>>>(x, d, n, lw, summary, probs, nprob, q);
    note_launch();
    const size_t smem = (size_t)kQCols * kQBins * (sizeof(double) + sizeof(unsigned));
    const int st = allow_dynamic_smem((const void *)quantile_level0_kernel<T>);
    if (st) return st;
    // row CTAs per column group: two CTAs on every SM, at least 1,024 rows each
    const int rows = (int)max((int64_t)1, min((n + 1023) / 1024, (int64_t)max(1, 2 * sms / cg)));
    quantile_level0_kernel<T><<<dim3(rows, cg), kQThreads, smem, stream>>>(x, d, n, lw, summary, q);
    note_launch();
    quantile_choose0_kernel<T><<<P, kQThreads, 0, stream>>>(d, q);
    note_launch();
    // each level takes 11 bits of the interval; a problem that is ready returns at once
    const int rows_l = (int)max((int64_t)1, min((n + 4095) / 4096, (int64_t)32));
    for (int b = 0; b < QKey<T>::kBits; b += 11) {
        quantile_level_kernel<T><<<dim3(rows_l, P), kQThreads, 0, stream>>>(x, d, n, lw, summary, q);
        note_launch();
    }
    const int rows_g = (int)max((int64_t)1, min((n + 511) / 512, (int64_t)max(1, 4 * sms / cg)));
    quantile_gather_kernel<T><<<dim3(rows_g, cg), kQThreads, 0, stream>>>(x, d, n, lw, summary, nprob, q);
    note_launch();
    quantile_finish_kernel<T><<<P, kQThreads, 0, stream>>>(d, lw, summary, q, out);
    note_launch();
    return (int)cudaGetLastError();
}

int weighted_quantile(const void *x, int d, int64_t n, const void *lw, int dtype, const double *summary,
                      const double *probs, int nprob, double *out, void *ws, cudaStream_t stream) {
    if (dtype == ISSM_F32)
        return weighted_quantile_t<float>((const float *)x, d, n, (const float *)lw, summary, probs, nprob, out, ws,
                                          stream);
    return weighted_quantile_t<double>((const double *)x, d, n, (const double *)lw, summary, probs, nprob, out, ws,
                                       stream);
}

}  // namespace issm
