// group.cu — one launch per phase for every in-flight AMIS run of a serving
// loop: the rounds of many independent posterior runs (uneven dimension,
// sample budget and round) advance together, one round per run per step, so
// the host issues a fixed handful of launches per step whatever the number of
// runs (the per-run sequence is _launch_prefilled_amis_round!,
// src/amis_execution.jl:261-357, then the moment fit,
// src/adaptive_gaussian_execution.jl:348-425).
//
// A step's runs are rows of a descriptor table (GroupRun, device memory).
// Each kernel's blocks are assigned to (run, tile) pairs through per-run
// cumulative block counts (a binary search per block): a run's blocks only
// touch that run's arrays, and every per-run reduction runs in a fixed
// order, so a run's results are bitwise the same alone and in any mix.
//
// Per step, for every run r in its round t:
//   group_draw       x = mu_t + L_t z, z from the counter-based normal stream
//                    (Philox-4x32-10, the run's seed and offset);
//   group_target     the linear-regression log posterior kernel in its exact
//                    mode-centred form log p(y, b) = c0 - |U (b - b_hat)|^2 / 2
//                    (U^T U = X^T X / sigma^2 + I / prior_var, b_hat the mode,
//                    c0 = log p(y, b_hat); formed from X^T X, X^T y, y^T y on
//                    admission) — the same function as the likelihood summed
//                    over the observations;
//   group_mixture    new samples: log sum_{s<=t} n_s q_s(x); retained ones:
//                    logaddexp with n_t q_t(x) (the AMIS recurrence), by
//                    forward substitution in FP32;
//   group_form       log weights log pi - log mixture + log N_t and per-block
//                    (max, S, S2) partials;
//   group_summary    one block per run: the partials merged in order;
//   group_moments    per-block sums of w (x - c) and w (x - c)(x - c)^T about
//                    the previous location c (compensated FP32, stored FP64);
//   group_fit        one block per run: the sums merged in order, mean and
//                    covariance, the ridge sqrt(eps(Float32)) tr(L L^T) / d,
//                    an FP64 Cholesky and the next slot (or the candidate).
#include "issm_device.cuh"
#include "issm_internal.h"
#include "ldlt.cuh"
#include "rng.cuh"

namespace issm {

using GroupRun = issm_group_run;
static_assert(sizeof(GroupRun) == 8 * 31, "issm_group_run is 31 eight-byte fields");

constexpr int kGTile = ISSM_GROUP_TILE;                       // samples per block of the per-sample kernels
constexpr int kGMomTiles = ISSM_GROUP_MOMENT_SAMPLES / kGTile;  // tiles per moment block
constexpr int kMomWords = ISSM_GROUP_MOMENT_WORDS;            // S0, S1, lower S2
static_assert(kMomWords == 1 + 64 + 64 * 65 / 2, "moment partial layout");

__device__ __forceinline__ int find_run(const GroupRun *runs, int nruns, int64_t blk, int which) {
    int lo = 0, hi = nruns - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const int64_t b0 = which == 0 ? runs[mid].blk_new0 : which == 1 ? runs[mid].blk_all0 : runs[mid].blk_mom0;
        if (b0 <= blk) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// ---- per-sample kernels: 128 samples of one run, one per thread ----------------
// The run's d x d matrix sits in shared memory by columns (stride LM, a
// multiple of four, so four consecutive rows of a column are one 16-byte
// broadcast) and the samples in a tile of odd row stride; each thread forms
// four coordinates at a time. Private d-vectors in local memory, reread per
// multiply-add, made these kernels 2.6 ms of a 64-run burst's steps.
struct GroupShared {
    float *M, *mu, *x;
    int LM, LX;
    __device__ GroupShared(float *base, int d) {
        LM = (d + 3) & ~3;
        LX = d | 1;
        M = base;
        mu = M + 64 * 64;
        x = mu + 64;
    }
};
constexpr size_t kGroupSmem = sizeof(float) * (64 * 64 + 64 + kGTile * 65);

__device__ __forceinline__ void group_stage_matrix(const GroupShared &g, const float *m, const float *mu, int d) {
    for (int e = threadIdx.x; e < d * d; e += kGTile) {
        const int c = e / d, r = e - c * d;
        g.M[c * g.LM + r] = m[e];
    }
    for (int c = threadIdx.x; c < d; c += kGTile) g.mu[c] = mu[c];
}
// rows x d contiguous floats <-> the tile
template <bool IN> __device__ __forceinline__ void group_move(const GroupShared &g, float *p, int rows, int d) {
    const int dq = kGTile / d, dr = kGTile - dq * d, total = rows * d;
    int r = threadIdx.x / d, c = threadIdx.x - r * d;
#pragma unroll 4
    for (int e = threadIdx.x; e < total; e += kGTile) {
        if (IN) g.x[r * g.LX + c] = p[e];
        else p[e] = g.x[r * g.LX + c];
        r += dq;
        c += dr;
        if (c >= d) {
            c -= d;
            ++r;
        }
    }
}

// log q of the staged Gaussian factor slot at the thread's row (overwritten by
// its standardised coordinates): lognorm - |L^-1 (x - mu)|^2 / 2
__device__ __forceinline__ float group_logq(const GroupShared &g, float *x, float lognorm, int d) {
    float r2 = 0.f;
    for (int r0 = 0; r0 < d; r0 += 4) {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = r0 + j < d ? x[r0 + j] - g.mu[r0 + j] : 0.f;
#pragma unroll 4
        for (int c = 0; c < r0; ++c) {
            const float4 m = *reinterpret_cast<const float4 *>(g.M + c * g.LM + r0);
            const float z = x[c];
            v[0] = fmaf(-m.x, z, v[0]);
            v[1] = fmaf(-m.y, z, v[1]);
            v[2] = fmaf(-m.z, z, v[2]);
            v[3] = fmaf(-m.w, z, v[3]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (r0 + j < d) {
                const float *col = g.M + (r0 + j) * g.LM + r0;
                v[j] /= col[j];
                r2 = fmaf(v[j], v[j], r2);
                x[r0 + j] = v[j];
#pragma unroll
                for (int i = j + 1; i < 4; ++i) v[i] = fmaf(-col[i], v[j], v[i]);
            }
    }
    return lognorm - 0.5f * r2;
}

__global__ void __launch_bounds__(kGTile) group_draw_kernel(const GroupRun *__restrict__ runs, int nruns) {
    extern __shared__ __align__(16) float smem[];
    const int j = find_run(runs, nruns, blockIdx.x, 0);
    const GroupRun &R = runs[j];
    const int64_t i0 = (int64_t)(blockIdx.x - R.blk_new0) * kGTile;
    const int rows = (int)min((int64_t)kGTile, R.n_round - i0);
    const int d = (int)R.d, t = (int)R.round;
    const GroupShared g(smem, d);
    group_stage_matrix(g, R.fac + (size_t)t * d * d, R.loc + (size_t)t * d, d);
    float *x = g.x + threadIdx.x * g.LX;
    if (threadIdx.x < rows) {
        // elements normal_offset + i d + e of the run's FP32 normal stream
        const uint64_t e0 = R.normal_offset + (uint64_t)(i0 + threadIdx.x) * d;
        for (int e = 0; e < d;) {
            const uint64_t el = e0 + e, blk = el >> 2;
            float v[4];
            NormalBlock<float>::eval(blk, R.seed, v);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q >= (int)(el & 3) && e < d) x[e++] = v[q];
        }
    }
    __syncthreads();
    if (threadIdx.x < rows)
        // from the top down: a group's normals are still there when it is formed
        for (int r0 = (d - 1) & ~3; r0 >= 0; r0 -= 4) {
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = r0 + j < d ? g.mu[r0 + j] : 0.f;
#pragma unroll 4
            for (int c = 0; c < r0; ++c) {
                const float4 m = *reinterpret_cast<const float4 *>(g.M + c * g.LM + r0);
                const float z = x[c];
                v[0] = fmaf(m.x, z, v[0]);
                v[1] = fmaf(m.y, z, v[1]);
                v[2] = fmaf(m.z, z, v[2]);
                v[3] = fmaf(m.w, z, v[3]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (r0 + j < d) {
                    const float *col = g.M + (r0 + j) * g.LM + r0;
                    const float z = x[r0 + j];
#pragma unroll
                    for (int i = j; i < 4; ++i) v[i] = fmaf(col[i], z, v[i]);
                }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (r0 + j < d) x[r0 + j] = v[j];
        }
    __syncthreads();
    group_move<false>(g, R.samples + (size_t)(R.n_old + i0) * d, rows, d);
}

__global__ void __launch_bounds__(kGTile) group_target_kernel(const GroupRun *__restrict__ runs, int nruns) {
    extern __shared__ __align__(16) float smem[];
    const int j = find_run(runs, nruns, blockIdx.x, 0);
    const GroupRun &R = runs[j];
    const int64_t i0 = (int64_t)(blockIdx.x - R.blk_new0) * kGTile, i = i0 + threadIdx.x;
    const int rows = (int)min((int64_t)kGTile, R.n_round - i0);
    const int d = (int)R.d;
    const GroupShared g(smem, d);
    group_stage_matrix(g, R.t_chol, R.t_mode, d);
    group_move<true>(g, R.samples + (size_t)(R.n_old + i0) * d, rows, d);
    __syncthreads();
    if (threadIdx.x >= rows) return;
    float *x = g.x + threadIdx.x * g.LX;
    for (int c = 0; c < d; ++c) x[c] -= g.mu[c];
    // |U (b - b_hat)|^2, U upper: coordinates r0 .. r0 + 3 over columns c >= r
    float q = 0.f;
    for (int r0 = 0; r0 < d; r0 += 4) {
        float u[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (r0 + k < d) {
                const float *col = g.M + (r0 + k) * g.LM + r0;
                const float z = x[r0 + k];
#pragma unroll
                for (int r = 0; r <= k; ++r) u[r] = fmaf(col[r], z, u[r]);
            }
#pragma unroll 4
        for (int c = r0 + 4; c < d; ++c) {
            const float4 m = *reinterpret_cast<const float4 *>(g.M + c * g.LM + r0);
            const float z = x[c];
            u[0] = fmaf(m.x, z, u[0]);
            u[1] = fmaf(m.y, z, u[1]);
            u[2] = fmaf(m.z, z, u[2]);
            u[3] = fmaf(m.w, z, u[3]);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (r0 + r < d) q = fmaf(u[r], u[r], q);
    }
    const float v = (float)R.t_const - 0.5f * q;
    R.logtargets[R.n_old + i] = v;
    if (isnan(v) || v == INFINITY)
        record_failure(R.failures + 3 * R.round, R.n_old + i + 1, 0,
                       isnan(v) ? ISSM_REASON_TARGET_NAN : ISSM_REASON_TARGET_POS_INF);
}

__global__ void __launch_bounds__(kGTile) group_mixture_kernel(const GroupRun *__restrict__ runs, int nruns) {
    extern __shared__ __align__(16) float smem[];
    const int j = find_run(runs, nruns, blockIdx.x, 1);
    const GroupRun &R = runs[j];
    const int64_t i0 = (int64_t)(blockIdx.x - R.blk_all0) * kGTile, i = i0 + threadIdx.x;
    const int64_t ntot = R.n_old + R.n_round;
    const int rows = (int)min((int64_t)kGTile, ntot - i0);
    const int d = (int)R.d, t = (int)R.round;
    const GroupShared g(smem, d);
    const float lc = (float)R.logcount;
    const bool mine = threadIdx.x < rows, fresh = i >= R.n_old;
    // retained samples gain slot t; new ones (the tile's last rows, if any) take every slot so far
    const int first = i0 + rows > R.n_old ? 0 : t;
    LseState<float> lse;
    float lq = 0.f;
    for (int s = first; s <= t; ++s) {
        __syncthreads();
        group_stage_matrix(g, R.fac + (size_t)s * d * d, R.loc + (size_t)s * d, d);
        group_move<true>(g, R.samples + (size_t)i0 * d, rows, d);
        __syncthreads();
        if (mine && (fresh || s == t)) {
            lq = group_logq(g, g.x + threadIdx.x * g.LX, R.lognorm[s], d);
            if (fresh) lse.add(lc + lq);
        }
    }
    if (!mine) return;
    const float out = fresh ? lse.value() : logaddexp(R.lognum[i], lc + lq);
    R.lognum[i] = out;
    if (isnan(out) || out == -INFINITY)
        record_failure(R.failures + 3 * R.round, i + 1, 0, ISSM_REASON_PROPOSAL_INVALID);
}

__global__ void group_form_kernel(const GroupRun *__restrict__ runs, int nruns) {
    const int j = find_run(runs, nruns, blockIdx.x, 1);
    const GroupRun &R = runs[j];
    const int64_t blk = blockIdx.x - R.blk_all0;
    const int64_t i = blk * kGTile + threadIdx.x;
    const int64_t ntot = R.n_old + R.n_round;
    __shared__ double s_logtotal;
    if (threadIdx.x == 0) s_logtotal = log((double)ntot);  // once: an FP64 log is some 34 FP64 operations
    __syncthreads();
    const double logtotal = s_logtotal;
    float l = -INFINITY;
    if (i < ntot) {
        l = (float)((double)R.logtargets[i] - (double)R.lognum[i] + logtotal);
        R.logweights[i] = l;
        if (isnan(l) || l == INFINITY) record_failure(R.failures + 3 * R.round, i + 1, 0, ISSM_REASON_LOGWEIGHT_INVALID);
    }
    // block (max, sum e^{l-m}, sum e^{2(l-m)}) in FP64, merged in a fixed tree order
    __shared__ double sm[kGTile], ss[kGTile], sq[kGTile];
    sm[threadIdx.x] = (double)l;
    __syncthreads();
    for (int o = kGTile / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
        __syncthreads();
    }
    const double m = sm[0];
    const double w = (l == -INFINITY || m == -INFINITY) ? 0.0 : exp((double)l - m);
    ss[threadIdx.x] = w;
    sq[threadIdx.x] = w * w;
    __syncthreads();
    for (int o = kGTile / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            ss[threadIdx.x] += ss[threadIdx.x + o];
            sq[threadIdx.x] += sq[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        R.partial[3 * blk] = m;
        R.partial[3 * blk + 1] = ss[0];
        R.partial[3 * blk + 2] = sq[0];
    }
}

// one CTA per run: the form partials' maximum, then their rescaled sums, each
// thread's share in block order and the threads in a fixed tree
__global__ void __launch_bounds__(256) group_summary_kernel(const GroupRun *__restrict__ runs) {
    const GroupRun &R = runs[blockIdx.x];
    const int64_t nb = (R.n_old + R.n_round + kGTile - 1) / kGTile;
    __shared__ double red[3][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double m = -INFINITY;
    for (int64_t b = threadIdx.x; b < nb; b += 256) m = fmax(m, R.partial[3 * b]);
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[0][warp] = m;
    __syncthreads();
    for (int w = 0; w < 8; ++w) m = fmax(m, red[0][w]);
    double s = 0.0, s2 = 0.0;
    if (m != -INFINITY)
        for (int64_t b = threadIdx.x; b < nb; b += 256) {
            const double bm = R.partial[3 * b];
            if (bm == -INFINITY) continue;
            const double f = exp(bm - m);
            s += R.partial[3 * b + 1] * f;
            s2 += R.partial[3 * b + 2] * f * f;
        }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if (lane == 0) {
        red[1][warp] = s;
        red[2][warp] = s2;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; ++w) {
        s += red[1][w];
        s2 += red[2][w];
    }
    double *o = R.summaries + 3 * R.round;
    o[0] = m;
    o[1] = s;
    o[2] = s2;
}

// per CTA of up to kGMomTiles tiles: S0, S1 = sum w (x - c) and the lower S2 =
// sum w (x - c)(x - c)^T as one Gram matrix of the coordinates and a constant
// 1, each entry a compensated FP32 sum (Kahan, the product inside the FMA)
// stored as FP64 for the fixed-order FP64 merge of the fit. A thread holds a 4 x 4
// tile of the lower triangle and takes every H-th of the 64 staged samples (adjacent
// lanes read other 16-byte groups of the same row). Bound by FP32 issue: four
// operations per entry and sample; single entries with two shared loads and six
// operations each took 5.4 ms over the steps of a 64-run burst.
constexpr int kGMomThreads = 320, kGMomRows = 64;
__global__ void __launch_bounds__(kGMomThreads) group_moments_kernel(const GroupRun *__restrict__ runs, int nruns) {
    __shared__ __align__(16) unsigned char raw[sizeof(double) * kGMomThreads * 16];
    __shared__ float wt[kGMomRows], ctr[64];
    static_assert(sizeof(raw) >= sizeof(float) * kGMomRows * 68, "the staged samples fit");
    float *z = reinterpret_cast<float *>(raw);
    double *red = reinterpret_cast<double *>(raw);
    const int j = find_run(runs, nruns, blockIdx.x, 2);
    const GroupRun &R = runs[j];
    const int64_t mb = blockIdx.x - R.blk_mom0;
    const int d = (int)R.d, t = (int)R.round, tid = threadIdx.x;
    const int64_t ntot = R.n_old + R.n_round;
    const double *sum = R.summaries + 3 * t;
    const double m = sum[0], inv = 1.0 / sum[1];
    const int nb = (d + 4) / 4, tiles = nb * (nb + 1) / 2, LD = nb % 2 ? nb * 4 : nb * 4 + 4;
    const int H = min(kGMomRows, kGMomThreads / tiles), tile = tid % tiles, h = tid / tiles;  // at most 153 tiles
    int br = 0;
    while ((br + 1) * (br + 2) / 2 <= tile) ++br;
    const int bc = tile - br * (br + 1) / 2;
    for (int c = tid; c < d; c += kGMomThreads) ctr[c] = R.loc[(size_t)t * d + c];
    for (int e = tid; e < kGMomRows * LD; e += kGMomThreads) z[e] = e % LD == d ? 1.f : 0.f;
    float s[4][4], k[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) s[a][b] = k[a][b] = 0.f;
    const int dq = kGMomThreads / d, dr = kGMomThreads - dq * d;
    const int64_t i0 = mb * kGMomTiles * kGTile, i1 = min(ntot, i0 + (int64_t)kGMomTiles * kGTile);
    for (int64_t s0 = i0; s0 < i1; s0 += kGMomRows) {
        const int rows = (int)min((int64_t)kGMomRows, i1 - s0);
        __syncthreads();
        const float *xp = R.samples + s0 * d;
        int r = tid / d, c = tid - r * d;
#pragma unroll 4
        for (int e = tid; e < rows * d; e += kGMomThreads) {
            z[r * LD + c] = xp[e] - ctr[c];
            r += dq;
            c += dr;
            if (c >= d) {
                c -= d;
                ++r;
            }
        }
        if (tid < rows) {
            const double l = (double)R.logweights[s0 + tid];
            wt[tid] = l == -INFINITY ? 0.f : (float)(exp(l - m) * inv);
        }
        __syncthreads();
        for (int q = h < H ? h : rows; q < rows; q += H) {
            const float w = wt[q];
            if (w == 0.f) continue;
            const float4 a4 = *reinterpret_cast<const float4 *>(z + q * LD + br * 4);
            const float4 b4 = *reinterpret_cast<const float4 *>(z + q * LD + bc * 4);
            const float a[4] = {w * a4.x, w * a4.y, w * a4.z, w * a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    const float y = fmaf(a[p], b[o], -k[p][o]);
                    const float u = s[p][o] + y;
                    k[p][o] = (u - s[p][o]) - y;
                    s[p][o] = u;
                }
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int o = 0; o < 4; ++o)
            if (h < H) red[(h * tiles + tile) * 16 + p * 4 + o] = (double)s[p][o] - (double)k[p][o];
    __syncthreads();
    double *out = R.mpartial + (size_t)mb * kMomWords;
    for (int e = tid; e < tiles * 16; e += kGMomThreads) {
        double v = red[e];
        for (int u = 1; u < H; ++u) v += red[u * tiles * 16 + e];
        int rb = 0;
        while ((rb + 1) * (rb + 2) / 2 <= e / 16) ++rb;
        const int r = rb * 4 + (e / 4) % 4, c = (e / 16 - rb * (rb + 1) / 2) * 4 + e % 4;
        if (c > r || r > d) continue;
        if (r < d) out[1 + 64 + r * (r + 1) / 2 + c] = v;
        else out[c < d ? 1 + c : 0] = v;
    }
}

// one CTA per run: merge the moment partials, mean and covariance, ridge, FP64
// LDL^T (ldlt_lower), and the next proposal (slot t + 1, or the candidate)
__global__ void __launch_bounds__(256) group_fit_kernel(const GroupRun *__restrict__ runs) {
    const GroupRun &R = runs[blockIdx.x];
    const int d = (int)R.d, t = (int)R.round, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    __shared__ double A[64 * 64];  // d x d column-major
    __shared__ double s1[64], s_dg[64], s_rinv[8], s_w[2][8][64], s_red[8];
    __shared__ double s_s0;
    const int tri = d * (d + 1) / 2;
    const float *c = R.loc + (size_t)t * d;
    auto row_col = [](int e, int &r, int &cc) {
        r = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
        if ((r + 1) * (r + 2) / 2 <= e) ++r;
        if (r * (r + 1) / 2 > e) --r;
        cc = e - r * (r + 1) / 2;
    };
    // merged sums (fixed block order)
    for (int q = tid; q < tri + d + 1; q += 256) {
        const int w = q < 1 ? 0 : q < 1 + d ? q : 1 + 64 + (q - 1 - d);
        double s = 0.0;
#pragma unroll 4
        for (int64_t b = 0; b < R.nmom; ++b) s += R.mpartial[(size_t)b * kMomWords + w];
        if (q == 0) s_s0 = s;
        else if (q < 1 + d) s1[q - 1] = s;
        else {
            int r, cc;
            row_col(q - 1 - d, r, cc);
            A[r + cc * d] = s;
        }
    }
    // ridge: sqrt(eps(Float32)) tr(L_t L_t^T) / d
    double tr = 0.0;
    const float *L = R.fac + (size_t)t * d * d;
    for (int e = tid; e < d * d; e += 256) tr += (double)L[e] * (double)L[e];
    for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
    if (lane == 0) s_red[warp] = tr;
    __syncthreads();
    double ridge = 0.0;
    for (int w = 0; w < 8; ++w) ridge += s_red[w];
    ridge *= 3.4526698300124393e-04 / (double)d;
    const double inv0 = 1.0 / s_s0;
    for (int q = tid; q < d; q += 256) R.mean[q] = (double)c[q] + s1[q] * inv0;
    for (int e = tid; e < tri; e += 256) {
        int r, cc;
        row_col(e, r, cc);
        double v = A[r + cc * d] * inv0 - (s1[r] * inv0) * (s1[cc] * inv0);
        R.cov[r + (size_t)cc * d] = v;
        R.cov[cc + (size_t)r * d] = v;
        if (r == cc) v += ridge;
        A[r + cc * d] = v;
    }
    __syncthreads();
    ldlt_lower(A, d, s_dg, s_rinv, s_w);
    __syncthreads();
    int bad = 0;
    for (int q = tid; q < d; q += 256) {
        const double dg = s_dg[q];
        bad |= !(isfinite(dg) && dg > 0.0);
        s1[q] = sqrt(dg);
    }
    bad = __syncthreads_or(bad);
    const bool last = t + 1 >= R.rounds;
    float *oloc = last ? R.cand_loc : R.loc + (size_t)(t + 1) * d;
    float *ofac = last ? R.cand_fac : R.fac + (size_t)(t + 1) * d * d;
    float *oln = last ? R.cand_lognorm : R.lognorm + (t + 1);
    if (bad) {
        if (tid == 0)
            record_failure(R.failures + 3 * t, R.n_old + R.n_round + 1, 0, ISSM_REASON_MOMENT_FIT_INVALID);
        return;
    }
    for (int q = tid; q < d; q += 256) oloc[q] = (float)R.mean[q];
    for (int e = tid; e < d * d; e += 256) {
        const int cc = e / d, r = e - cc * d;
        ofac[e] = r > cc ? (float)(A[e] * s1[cc]) : r == cc ? (float)s1[cc] : 0.f;
    }
    // Gaussian lognormalizer of the stored FP32 factor
    double ld = tid < d ? log((double)(float)s1[tid]) : 0.0;
    for (int o = 16; o > 0; o >>= 1) ld += __shfl_xor_sync(0xffffffffu, ld, o);
    if (lane == 0) s_red[warp] = ld;
    __syncthreads();
    if (tid == 0) *oln = (float)(-0.5 * (double)d * log(2.0 * 3.14159265358979323846) - (s_red[0] + s_red[1]));
}

int group_step(const void *runs, int nruns, int64_t blocks_new, int64_t blocks_all, int64_t blocks_mom,
               cudaStream_t stream) {
    const GroupRun *R = (const GroupRun *)runs;
    for (const void *k : {(const void *)group_draw_kernel, (const void *)group_target_kernel, (const void *)group_mixture_kernel}) {
        const int e = allow_dynamic_smem(k);
        if (e) return e;
    }
    if (blocks_new > 0) {
        group_draw_kernel<<<(unsigned)blocks_new, kGTile, kGroupSmem, stream>>>(R, nruns);
        note_launch();
        group_target_kernel<<<(unsigned)blocks_new, kGTile, kGroupSmem, stream>>>(R, nruns);
        note_launch();
    }
    group_mixture_kernel<<<(unsigned)blocks_all, kGTile, kGroupSmem, stream>>>(R, nruns);
    note_launch();
    group_form_kernel<<<(unsigned)blocks_all, kGTile, 0, stream>>>(R, nruns);
    note_launch();
    group_summary_kernel<<<nruns, 256, 0, stream>>>(R);
    note_launch();
    group_moments_kernel<<<(unsigned)blocks_mom, kGMomThreads, 0, stream>>>(R, nruns);
    note_launch();
    group_fit_kernel<<<nruns, 256, 0, stream>>>(R);
    note_launch();
    return (int)cudaGetLastError();
}

}  // namespace issm

extern "C" size_t issm_group_run_bytes(void) { return sizeof(issm_group_run); }

extern "C" int issm_group_step(const issm_group_run *runs, int32_t nruns, int64_t blocks_new, int64_t blocks_all,
                               int64_t blocks_mom, issm_stream_t stream) {
    if (nruns < 1 || blocks_all < 1 || blocks_new < 0 || blocks_mom < 1) return ISSM_E_SIZE;
    if (!runs) return ISSM_E_NULL;
    if (blocks_new > 0x7fffffff || blocks_all > 0x7fffffff || blocks_mom > 0x7fffffff) return ISSM_E_SIZE;
    return issm::group_step(runs, nruns, blocks_new, blocks_all, blocks_mom, (cudaStream_t)stream);
}
