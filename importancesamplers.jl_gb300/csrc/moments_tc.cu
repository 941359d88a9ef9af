// moments_tc.cu — tensor-core form of the weighted moments that drive AMIS /
// N-PMC adaptation (_weighted_moments!, src/adaptive_gaussian_execution.jl:268-273).
//
// One streaming pass over the retained samples. For a tile of 128 samples,
// v = sqrt(w) (x - c) (c = previous proposal mean) is split v = vh + vl into
// bf16 parts, and so is sqrt(w) = sh + sl. One MMA per 16-sample K slice
// accumulates, in tensor memory, D = A B^T with A = [vh; vl] (M = 128 rows:
// 64 hi, 64 lo) and B = [vh; vl; sh; sl] (N = 144): all four hi/lo blocks of
// (vh + vl)(vh + vl)^T and the products with sh, sl. The epilogue adds them:
// S2 = sum w z z^T, S1 = sum w z of the split operand, and the converters sum
// S0 = sum (sh + sl)^2 the same way, so [S2 S1; S1^T S0] is the Gram matrix
// of the split operand (about 16 significant bits per element): the
// covariance, its Schur complement, is positive semidefinite up to FP32
// accumulation however few samples carry the weight, and the regularising
// ridge keeps the fit positive definite. Each CTA stores P = S / 2; the
// reduce kernel forms S = P + P^T.
//
// When the new mean lies far from c relative to the spread, S2/S0 and the
// mean's outer product nearly cancel. A second pass centred at the first
// pass's mean runs when the first pass's cancellation error could matter
// against the variance or the fit's ridge (see the reduce kernel); its
// kernels are always launched (graph replays see a fixed sequence) and
// return at once when the flag is clear.
//
// A is stored MN-major: each sample's 8-coordinate groups are 16-byte chunks, so
// a lane converts a group straight from its registers. Warp roles: warp 0 issues
// the MMAs; warps 1..12 read, weight and split the samples, three groups of four
// warps on alternate tiles, each lane's next 64 floats requested as soon as the
// last ones are converted (96 KB on their way per CTA). Per-CTA partials are summed
// across CTAs (compensated FP32) and mean = c + S1/S0, cov = S2/S0 - (S1/S0)
// (S1/S0)^T in FP64.
//
// The pass is bound by reading the samples: 64 us on average over 50,000 ..
// 2,000,000 samples of d = 64, 4.3 TB/s with the launch. Sixteen converter warps
// in lockstep on tiles staged by tensor copies took 66; for d other than 32 and
// 64, where they staged padded rows by cp.async, up to 2.5 times as long (d = 33,
// 100,000 .. 1,000,000 samples: 77 us, now 29). Sixteen warps of this form took
// 71: 17 warps leave 96 registers a thread, and they spill.
#include "issm_device.cuh"
#include "issm_internal.h"
#include "sample_rows.cuh"
#include "tcgen05.cuh"

namespace issm {

constexpr int kMtConvWarps = 12;
constexpr int kMtThreads = 32 * (1 + kMtConvWarps);  // issuer, converters
constexpr int kMtConvGroups = 3;  // groups of four warps, each on its own tile
constexpr int kMtTile = 128;   // samples per tile = MMA K extent per tile
constexpr int kMtCtasPerSm = 1;
constexpr int kMtCols = 80;    // columns of a CTA's partial (64 coordinates, sqrt(w), padding)
constexpr int kMtN = 144;      // MMA N: hi rows, lo rows, sqrt(w) hi and lo, padding
constexpr int kMtABufs = 6;    // operand buffers
// One operand buffer holds 18 row groups of 128 samples x 16 bytes, MN-major:
// groups 0..7 the bf16 hi parts of the 64 coordinates, groups 8..15 their lo
// parts, group 16 (sqrt(w) hi, sqrt(w) lo, zeros) and group 17 zeros. A is
// its first 16 groups (M = 128), B all 18 (N = 144).
constexpr int kMtGroups = 18;
constexpr int kMtBuf = kMtGroups * kMtTile * 16;
constexpr size_t kMtSmem = (size_t)kMtABufs * kMtBuf;
static_assert(kMtSmem <= 232448 - 2048, "dynamic shared memory per CTA");
static_assert(128 * 65 * 4 <= kMtBuf, "the epilogue's row sums fit in one operand buffer");
constexpr int kMtPartial = 65 * kMtCols;  // P = S / 2 of one CTA (the reduce forms S = P + P^T)

__global__ void __launch_bounds__(kMtThreads, kMtCtasPerSm) moments_tc_kernel(const float *__restrict__ x, int d, int64_t n,
                                                                    const float *__restrict__ lw,
                                                                    const double *__restrict__ summary,
                                                                    const double *__restrict__ center,
                                                                    float *__restrict__ partial, int *error,
                                                                    const int *__restrict__ gate) {
    if (gate != nullptr && *gate == 0) return;  // refinement pass not needed
    extern __shared__ __align__(1024) unsigned char s_a[];  // [buf] x kMtBuf
    __shared__ __align__(8) uint64_t a_full[kMtABufs], a_empty[kMtABufs];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    __shared__ float s_s0[kMtConvWarps];
    const int tid = threadIdx.x, warp = tc::uniform_warp(), lane = tid & 31;
    if (warp == 0) tc::tmem_alloc(&tmem_base, 256);
    if (tid == 0) {
        for (int b = 0; b < kMtABufs; ++b) {
            tc::mbar_init(&a_full[b], kMtConvWarps / kMtConvGroups);
            tc::mbar_init(&a_empty[b], 1);
        }
        tc::fence_mbar_init();
        abort_flag = 0;
    }
    // group 17 of every buffer: zeros (B rows 136..143, never read back)
    for (int e = tid; e < kMtABufs * kMtTile; e += kMtThreads)
        *reinterpret_cast<uint4 *>(s_a + (size_t)(e / kMtTile) * kMtBuf + 17 * kMtTile * 16 + (e % kMtTile) * 16) =
            make_uint4(0u, 0u, 0u, 0u);
    if (tid < kMtConvWarps) s_s0[tid] = 0.f;
    const float m = (float)summary[0];
    const float inv_sqrt_s = (float)(1.0 / sqrt(summary[1]));
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = tc::uniform(tmem_base);  // D: 128 lanes x 144 columns
    const int64_t ntiles = (n + kMtTile - 1) / kMtTile;
    const int my_tiles = (int)((ntiles - (int64_t)blockIdx.x + gridDim.x - 1) / gridDim.x);
    auto tile_of = [&](int it) -> int64_t { return (int64_t)blockIdx.x + (int64_t)it * gridDim.x; };
    auto wait = [&](uint64_t *bar, uint32_t parity) -> bool {
        if (abort_flag) return false;
        if (tc::mbar_wait(bar, parity)) return true;
        atomicExch(error, 1);
        abort_flag = 1;
        return false;
    };
    if (warp == 0) {
        // ---- issuer: D += [Ah; Al] [Ah; Al; sqrt(w)]^T, one MMA per K slice ----
        const uint32_t idesc = tc::instr_desc(tc::kBF16, 128, kMtN) | tc::kMajorMN;
        constexpr uint32_t LBO = 128, SBO = kMtTile * 16;  // K-group stride, row-group stride
        for (int it = 0; it < my_tiles; ++it) {
            const int buf = it % kMtABufs;
            {
                const bool ok = __all_sync(0xffffffffu, wait(&a_full[buf], (uint32_t)((it / kMtABufs) & 1)));
                tc::fence_after_sync();
                if (ok) {
                    const uint32_t a0 = tc::smem_u32(s_a + (size_t)buf * kMtBuf);
#pragma unroll
                    for (int s = 0; s < kMtTile / 16; ++s) {
                        const uint64_t da = tc::smem_desc(a0 + s * 256, LBO, SBO);
                        tc::mma_elect(tbase, da, da, idesc, it > 0 || s > 0);
                    }
                }
                tc::commit_elect(&a_empty[buf]);
            }
            __syncwarp();
        }
    } else {
        // ---- converters: groups of four warps take alternate tiles; a warp's 32
        // rows in four passes of 8, lane = row + 8 x group of 8 coordinates ----
        constexpr int RP = 4;
        const int cw = (warp - 1) & 3, cgroup = (warp - 1) >> 2, rl = lane & 7, gl = lane >> 3;
        const int access = row_access(x, d);
        float cc[2][8], v[RP][2][8], l[RP];
#pragma unroll
        for (int gg = 0; gg < 2; ++gg)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int c = (gl + 4 * gg) * 8 + j;
                cc[gg][j] = c < d ? (float)center[c] : 0.f;
            }
        auto load = [&](int it) {
#pragma unroll
            for (int rp = 0; rp < RP; ++rp) {
                const int64_t i = tile_of(it) * kMtTile + 32 * cw + 8 * rp + rl;
                const bool active = it < my_tiles && i < n;
                l[rp] = active ? lw[i] : -INFINITY;
#pragma unroll
                for (int gg = 0; gg < 2; ++gg) load_group(v[rp][gg], x, i, active, d, (gl + 4 * gg) * 8, access);
            }
        };
        load(cgroup);
        float s0 = 0.f;  // sum of (sqrt(w) hi + lo)^2 over this thread's samples: S0 of the split operand
        for (int it = cgroup; it < my_tiles; it += kMtConvGroups) {
            const int buf = it % kMtABufs;
            const bool ok = it < kMtABufs ||
                            __all_sync(0xffffffffu, wait(&a_empty[buf], (uint32_t)(((it / kMtABufs) - 1) & 1)));
            if (ok) {
#pragma unroll
                for (int rp = 0; rp < RP; ++rp) {
                    unsigned char *ab = s_a + (size_t)buf * kMtBuf + (32 * cw + 8 * rp + rl) * 16;
                    const float sw = l[rp] == -INFINITY ? 0.f : expf(0.5f * (l[rp] - m)) * inv_sqrt_s;
#pragma unroll
                    for (int gg = 0; gg < 2; ++gg) {
                        float z[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) z[j] = sw * (v[rp][gg][j] - cc[gg][j]);
                        const uint4 hi = make_uint4(tc::pack_bf16x2(z[0], z[1]), tc::pack_bf16x2(z[2], z[3]),
                                                    tc::pack_bf16x2(z[4], z[5]), tc::pack_bf16x2(z[6], z[7]));
                        auto lo2 = [](float p, float q, uint32_t h) {
                            return tc::pack_bf16x2(p - __uint_as_float(h << 16), q - __uint_as_float(h & 0xffff0000u));
                        };
                        const uint4 lo = make_uint4(lo2(z[0], z[1], hi.x), lo2(z[2], z[3], hi.y),
                                                    lo2(z[4], z[5], hi.z), lo2(z[6], z[7], hi.w));
                        *reinterpret_cast<uint4 *>(ab + (size_t)(gl + 4 * gg) * kMtTile * 16) = hi;
                        *reinterpret_cast<uint4 *>(ab + (size_t)(8 + gl + 4 * gg) * kMtTile * 16) = lo;
                    }
                    if (gl == 0) {
                        // group 16: sqrt(w) hi in row 128, its lo part in row 129
                        const uint32_t h = tc::pack_bf16x2(sw, 0.f);
                        const float swh = __uint_as_float(h << 16);
                        const uint32_t hl = tc::pack_bf16x2(swh, sw - swh);
                        const float swl = __uint_as_float(hl & 0xffff0000u);
                        const float sws = swh + swl;  // exact: swl is a bf16 below swh's last bit
                        s0 = fmaf(sws, sws, s0);
                        *reinterpret_cast<uint4 *>(ab + (size_t)16 * kMtTile * 16) = make_uint4(hl, 0u, 0u, 0u);
                    }
                }
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&a_full[buf]);
            load(it + kMtConvGroups);
        }
        // S0 per warp in a fixed order (lanes by xor tree, warps summed in order below)
        for (int off = 16; off > 0; off >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, off);
        if (lane == 0) s_s0[warp - 1] = s0;
    }
    // ---- the last commit tracks every MMA of the CTA ----
    tc::fence_before_sync();
    __syncthreads();
    if (my_tiles > 0) {
        const int last = my_tiles - 1;
        if (!tc::mbar_wait(&a_empty[last % kMtABufs], (uint32_t)((last / kMtABufs) & 1)) && tid == 0) {
            atomicExch(error, 1);
            abort_flag = 1;
        }
    }
    __syncthreads();
    tc::fence_after_sync();
    float *out = partial + (size_t)blockIdx.x * kMtPartial;
    // row sums T[r][j] = D[r][j] + D[r][64 + j] (j < 64) and T[r][64] =
    // D[r][128] + D[r][129] in the first operand buffer's space (every MMA is done)
    float *T = reinterpret_cast<float *>(s_a);
    // warps 1..4 read TMEM lane quadrants 1, 2, 3, 0 (a warp reads quadrant warp % 4)
    if (!abort_flag && warp >= 1 && warp <= 4) {
        const int q = warp & 3, row = 32 * q + lane;
        const uint32_t lane_base = tbase + ((uint32_t)(32 * q) << 16);
#pragma unroll
        for (int c0 = 0; c0 < 64; c0 += 16) {
            float a[16], b[16];
            if (my_tiles > 0) {
                tc::tmem_ld16(lane_base + (uint32_t)c0, a);
                tc::tmem_ld16(lane_base + (uint32_t)(64 + c0), b);
            } else {
                for (int j = 0; j < 16; ++j) a[j] = b[j] = 0.f;
            }
            for (int j = 0; j < 16; ++j) T[row * 65 + c0 + j] = a[j] + b[j];
        }
        float a[16];
        if (my_tiles > 0) tc::tmem_ld16(lane_base + 128u, a);
        else for (int j = 0; j < 16; ++j) a[j] = 0.f;
        T[row * 65 + 64] = a[0] + a[1];
    }
    __syncthreads();
    // P = S / 2 over 65 x 80: S2 = T[i] + T[64 + i], S1 the sqrt(w) column, S0 from the converters
    if (!abort_flag) {
        float s0_all = 0.f;
        for (int w = 0; w < kMtConvWarps; ++w) s0_all += s_s0[w];
        for (int e = tid; e < kMtPartial; e += kMtThreads) {
            const int r = e / kMtCols, c = e - r * kMtCols;
            float v = 0.f;
            if (r < 64 && c < 65) v = T[r * 65 + c] + T[(64 + r) * 65 + c];
            else if (r == 64 && c < 64) v = T[c * 65 + 64] + T[(64 + c) * 65 + 64];
            else if (r == 64 && c == 64) v = s0_all;
            out[e] = 0.5f * v;
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tbase, 256);
}

// Partials are [block][65][80] FP32 (P = S / 2). Every CTA sums 32 entries
// over the blocks (32 block-strided lanes per entry, coalesced); the last CTA
// to finish (a device-scope counter, reset by that CTA) forms S = P + P^T and
// from it mean = c + S1/S0 and cov = S2/S0 - (S1/S0)(S1/S0)^T in FP64, with c
// the FP32 value the pass subtracted. `center` and `mean` may be the same
// array: each entry is read before it is written. With `refine` given, the
// last CTA sets it when, on some diagonal, the pass's cancellation error
// (2^-16 of the second moment s2 about c) exceeds 2^-8 of the variance v plus
// 2^-4 of R = sqrt(eps(Float32)) tr(L L^T) / d for the previous factor L, the
// scale of the ridge the fit adds (R = 0 without L): s2 > 256 v + 4096 R.
// Low-ESS rounds whose variance is mostly ridge then refine only when the
// mean moved by more than about one previous scale.
constexpr int kMtReduceThreads = 1024;  // 32 entries x 32 block-strided lanes per CTA

// FP64 work here runs on one SM's FP64 pipe (a warp-instruction holds it for
// about 64 cycles on this GPU whatever the active lanes), so the kernel keeps
// FP64 to the Schur complement itself: lanes combine in compensated FP32, the
// ridge scale is FP32, 1/S0 is formed once, and only the lower triangle of the
// covariance is computed (four FP64 operations per element).
__global__ void __launch_bounds__(kMtReduceThreads) moments_tc_reduce_kernel(
    const float *__restrict__ partial, int blocks, double *sums, int d, const double *center, double *mean,
    double *__restrict__ cov, const int *__restrict__ gate, int *refine, const float *__restrict__ prev,
    unsigned *counter) {
    if (gate != nullptr && *gate == 0) return;
    __shared__ float acc_s[32][33], cmp_s[32][33];
    __shared__ double s_m[65];  // S1 / S0 (the mean about c)
    __shared__ double s_inv;
    __shared__ float s_r[32];
    __shared__ int last;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + tx;
    // compensated FP32 over this lane's blocks, then over the 32 lanes
    float s = 0.f, cmp = 0.f;
    if (e < kMtPartial)
        for (int b = ty; b < blocks; b += 32) {
            const float y = partial[(size_t)b * kMtPartial + e] - cmp;
            const float t = s + y;
            cmp = (t - s) - y;
            s = t;
        }
    acc_s[ty][tx] = s;
    cmp_s[ty][tx] = cmp;
    __syncthreads();
    if (ty == 0 && e < kMtPartial) {
        float t = 0.f, c = 0.f;
        for (int r = 0; r < 32; ++r) {
            const float y = acc_s[r][tx] - (cmp_s[r][tx] + c);
            const float u = t + y;
            c = (u - t) - y;
            t = u;
        }
        sums[e] = (double)t - (double)c;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    auto S = [&](int r, int c) { return __ldcg(sums + r * kMtCols + c) + __ldcg(sums + c * kMtCols + r); };
    if (threadIdx.x == 0) s_inv = 1.0 / S(64, 64);
    // R = sqrt(eps(Float32)) tr(L L^T) / d of the previous factor (0 without one), in FP32
    float rr = 0.f;
    if (refine != nullptr && prev != nullptr)
        for (int q = threadIdx.x; q < d * d; q += blockDim.x) rr = fmaf(prev[q], prev[q], rr);
    for (int off = 16; off > 0; off >>= 1) rr += __shfl_xor_sync(0xffffffffu, rr, off);
    if (tx == 0) s_r[ty] = rr;
    __syncthreads();
    if (threadIdx.x < 65) s_m[threadIdx.x] = S(64, threadIdx.x) * s_inv;
    __syncthreads();
    const double inv = s_inv;
    // lower triangle, row-major: q -> (r, c), c <= r
    const int tri = d * (d + 1) / 2;
    for (int q = threadIdx.x; q < tri; q += blockDim.x) {
        int r = (int)((sqrtf(8.f * (float)q + 1.f) - 1.f) * 0.5f);
        if ((r + 1) * (r + 2) / 2 <= q) ++r;
        if (r * (r + 1) / 2 > q) --r;
        const int c = q - r * (r + 1) / 2;
        const double v = fma(S(r, c), inv, -s_m[r] * s_m[c]);
        cov[r + (size_t)c * d] = v;
        cov[c + (size_t)r * d] = v;
    }
    int flag = 0;
    if (refine != nullptr && threadIdx.x < d) {
        float ridge = 0.f;
        for (int w = 0; w < 32; ++w) ridge += s_r[w];
        ridge *= 3.4526698e-4f / (float)d;  // sqrt(FLT_EPSILON)
        const int r = threadIdx.x;
        const double s2 = S(r, r) * inv, v = s2 - s_m[r] * s_m[r];
        // the pass's error (2^-16 of s2) above 2^-8 of v plus 2^-4 of the ridge scale
        flag = !(s2 <= 256.0 * v + 4096.0 * (double)ridge);
    }
    flag = __syncthreads_or(flag);  // also orders the reads of `center` below after every thread's work above
    for (int j = threadIdx.x; j < d; j += blockDim.x) mean[j] = (double)(float)center[j] + s_m[j];
    if (threadIdx.x == 0) {
        if (refine != nullptr) *refine = flag;
        *counter = 0u;
    }
}

constexpr int kMtMaxBlocks = kSMs * kMtCtasPerSm;

static int moments_tc_blocks(int64_t n) {
    const int64_t t = (n + kMtTile - 1) / kMtTile;
    const int64_t cap = (int64_t)device_sms() * kMtCtasPerSm;  // <= kMtMaxBlocks, the scratch bound
    return (int)(t < cap ? (t < 1 ? 1 : t) : cap);
}

size_t moments_tc_workspace_bytes(int64_t n) {
    (void)n;
    return sizeof(float) * (size_t)kMtMaxBlocks * kMtPartial + sizeof(double) * kMtPartial + 256;
}

int moments_tc(const void *x, int d, int64_t n, const void *lw, const double *summary, const double *shift,
               const float *prev_factor, double *mean, double *cov, int precision, void *ws, size_t ws_bytes,
               int *error, cudaStream_t stream) {
    (void)precision;  // both tensor-core forms use the bf16 split contraction
    if (d > 64) return ISSM_E_UNSUPPORTED;
    if (ws_bytes < moments_tc_workspace_bytes(n)) return ISSM_E_WORKSPACE;
    const int blocks = moments_tc_blocks(n);
    float *partial = (float *)ws;
    const int e = allow_dynamic_smem((const void *)moments_tc_kernel);
    if (e) return e;
    double *sums = reinterpret_cast<double *>(partial + (size_t)kMtMaxBlocks * kMtPartial);
    int *refine = reinterpret_cast<int *>(sums + kMtPartial);
    unsigned *counter = reinterpret_cast<unsigned *>(error + 1);  // zero with the workspace; reset by each use
    const int rblocks = (kMtPartial + 31) / 32;
    // pass 1 about `shift`
    { moments_tc_kernel<<<blocks, kMtThreads, kMtSmem, stream>>>((const float *)x, d, n, (const float *)lw,
                                                                       summary, shift, partial, error, nullptr);
      note_launch(); }
    { moments_tc_reduce_kernel<<<rblocks, kMtReduceThreads, 0, stream>>>(partial, blocks, sums, d, shift, mean, cov,
                                                                         nullptr, refine, prev_factor, counter);
      note_launch(); }
    // pass 2 about the new mean (kernels return at once unless pass 1 set `refine`)
    { moments_tc_kernel<<<blocks, kMtThreads, kMtSmem, stream>>>((const float *)x, d, n, (const float *)lw,
                                                                      summary, mean, partial, error, refine);
      note_launch(); }
    { moments_tc_reduce_kernel<<<rblocks, kMtReduceThreads, 0, stream>>>(partial, blocks, sums, d, mean, mean, cov,
                                                                         refine, nullptr, nullptr, counter);
      note_launch(); }
    return (int)cudaGetLastError();
}

}  // namespace issm
