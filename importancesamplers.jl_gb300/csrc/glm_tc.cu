// glm_tc.cu — the regression likelihoods of the batch targets (X beta over
// every observation for every sample; the user batch callback of
// src/batched_targets.jl:54-214, examples/batched_linear_regression.jl:18-37)
// as a tcgen05 GEMM with the log-likelihood reduced in the epilogue.
//
// For a tile of 128 samples (rows, M) and 256 observations (columns, N):
//   D[i, o] = beta_i . x_o         (K = d, padded to DP = 16 / 32 / 64)
// accumulates in tensor memory (FP32), and the epilogue turns each entry into
//   Bernoulli-logit: y_o eta - log(1 + e^eta)
//   Gaussian:        (y_o - eta)^2            (scaled by -1 / (2 sigma^2) at the end)
// summed over the observations in registers: the samples sit on the TMEM
// lanes, so a thread owns one sample and no cross-thread reduction is needed.
// The prior N(0, prior_var I) and the constants are added once per sample.
//
// Precision forms (FP32 accumulation in all):
//   BF16     one kind::f16 MMA per K slice on bf16-rounded operands;
//   BF16x3   operands split v = hi + lo in bf16, D = Bh Xh + Bl Xh + Bh Xl;
//   TF32     one kind::tf32 MMA per K slice, operands rounded to tf32.
//
// The observations' operand form (bf16 hi/lo or tf32, row-contiguous
// canonical K-major layout, 256 observations per tile, zero-padded) is built
// once per target by glm_prepare_kernel. glm_tc_kernel is persistent: a CTA
// walks row tiles of 128 samples, and for each the observation tiles.
//   * warps 1-4 convert the next row tile into the other A buffer (one sample
//     row per thread) and sum its squares for the prior;
//   * warp 0 issues each item's (row tile, observation tile) MMAs into one of
//     two TMEM accumulators; the observation tiles stay in shared memory when
//     all of them fit, else stream through a ring of bulk copies;
//   * warps 5-20, four per TMEM lane quadrant and 64 columns each, reduce the
//     other accumulator.
// The epilogue bounds it, so a pair costs one MUFU and eight FP32 operations: with
// t = e^-|eta|, sum log(1 + t) is log1p of a product of factors 1 + t, carried less
// one, P <- P + t + P t, so that a small t keeps its relative accuracy (the factors
// themselves would round it at 2^-24 of one: at |eta| = 17 all of it), and one log1p
// per 32. A log1p per pair, eight epilogue warps and a cold CTA per row tile took
// 2,384 us at 65,536 samples x 10,000 observations, d = 32 (BF16x3 logistic), now 367
// (512 row tiles leave the fourth wave of 152 a third full), and 103 us at 50,000 x
// 500, d = 64 (Gaussian), now 20. Every wait is bounded; a timeout sets the sticky
// error word.
#include <type_traits>

#include "issm_device.cuh"
#include "issm_internal.h"
#include "tcgen05.cuh"

namespace issm {

constexpr int kGlmRows = 128;      // samples per row tile (MMA M)
constexpr int kGlmCols = 256;      // observations per tile (MMA N)
constexpr int kGlmConvWarps = 4;   // one thread per sample row
constexpr int kGlmEpiWarps = 16;   // four per TMEM lane quadrant
constexpr int kGlmParts = kGlmEpiWarps / 4;           // column parts of an accumulator
constexpr int kGlmPartCols = kGlmCols / kGlmParts;
constexpr int kGlmFirstEpi = 1 + kGlmConvWarps;
constexpr int kGlmThreads = 32 * (1 + kGlmConvWarps + kGlmEpiWarps);
constexpr int kGlmRing = 6;        // observation tiles in shared memory, at most
constexpr size_t kGlmMaxSmem = 232448 - 20 * 1024;    // the static part and the reserved kilobyte
constexpr double kGlmLog2Pi = 1.8378770664093454835606594728112;

template <int KIND> __device__ __forceinline__ uint4 glm_pack(const float *v) {
    if (KIND == tc::kTF32) return make_uint4(tc::tf32_rn(v[0]), tc::tf32_rn(v[1]), tc::tf32_rn(v[2]), tc::tf32_rn(v[3]));
    return make_uint4(tc::pack_bf16x2(v[0], v[1]), tc::pack_bf16x2(v[2], v[3]), tc::pack_bf16x2(v[4], v[5]),
                      tc::pack_bf16x2(v[6], v[7]));
}
__device__ __forceinline__ uint32_t glm_lo_pair(float a, float b, uint32_t hi) {
    return tc::pack_bf16x2(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
}
__device__ __forceinline__ uint4 glm_pack_lo(const float *v, uint4 hi) {
    return make_uint4(glm_lo_pair(v[0], v[1], hi.x), glm_lo_pair(v[2], v[3], hi.y), glm_lo_pair(v[4], v[5], hi.z),
                      glm_lo_pair(v[6], v[7], hi.w));
}

template <int KIND, int SPLIT, int DP> struct GlmShape {
    static constexpr int EB = KIND == tc::kBF16 ? 2 : 4;
    static constexpr int PER = 16 / EB;          // elements per 16-byte K group
    static constexpr int KG = DP / PER;          // K groups
    static constexpr int NPART = SPLIT == 3 ? 2 : 1;
    static constexpr int KSTEPS = KG / 2;        // MMA K slices of 32 bytes
    static constexpr size_t A_PART = (size_t)KG * kGlmRows * 16;
    static constexpr size_t B_PART = (size_t)KG * kGlmCols * 16;
    static constexpr size_t TILE = NPART * B_PART;  // one observation tile of the operand form
};

// Operand form of the observations: tile t, part p, K group q, row j at
//   t * TILE + p * B_PART + q * 256 * 16 + j * 16.
template <int KIND, int SPLIT, int DP>
__global__ void __launch_bounds__(256) glm_prepare_kernel(const float *__restrict__ X, int nobs, int d, int tiles,
                                                          unsigned char *__restrict__ ops) {
    using S = GlmShape<KIND, SPLIT, DP>;
    const int64_t total = (int64_t)tiles * S::KG * kGlmCols;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int j = (int)(e % kGlmCols), q = (int)((e / kGlmCols) % S::KG), t = (int)(e / ((int64_t)kGlmCols * S::KG));
        const int o = t * kGlmCols + j;
        float v[S::PER];
#pragma unroll
        for (int m = 0; m < S::PER; ++m) {
            const int c = q * S::PER + m;
            v[m] = (o < nobs && c < d) ? X[o + (size_t)c * nobs] : 0.f;  // X column-major, nobs x d
        }
        unsigned char *base = ops + (size_t)t * S::TILE + (size_t)q * kGlmCols * 16 + (size_t)j * 16;
        const uint4 hi = glm_pack<KIND>(v);
        *reinterpret_cast<uint4 *>(base) = hi;
        if (S::NPART == 2) *reinterpret_cast<uint4 *>(base + S::B_PART) = glm_pack_lo(v, hi);
    }
}

struct GlmParams {
    int d, nobs, kind, tiles, ring;
    int64_t n;
    const float *x;              // samples, n x d
    const float *y;              // observations' responses, nobs
    const unsigned char *ops;    // operand form of X
    float *out;
    double scale, prior_scale, constant;  // log target = scale * (sum) + prior_scale * |x|^2 + constant
    int *error;
};

// unevaluated hi + lo sums of FP32 terms (error-free additions; about 48 bits)
struct GlmPair {
    float h, l;
    __device__ __forceinline__ void add(float x, float e = 0.f) {
        const float s = h + x, b = s - h;
        l += ((h - (s - b)) + (x - b)) + e;
        h = s;
    }
    __device__ __forceinline__ double value() const { return isfinite(h) ? (double)h + (double)l : (double)h; }
};

// e^-|v| with the rounding of |v| log2(e) put back: 2^p of the product p rounded
// down, times 1 + r with r = -|v| - p ln 2 >= 0 (log2(e) is rounded up for that), so a
// small term keeps its relative accuracy. Saturation makes r 0 for infinite v. The
// largest error is 3.3 units of 2^-24 for |v| up to 30 (5.5 up to 85); without the
// correction 16 at 17 and 63 at 85. expf (2.6) makes the call a quarter slower,
// and the log target's error is the same.
__device__ __forceinline__ float exp_neg(float v) {
    const float a = -fabsf(v), p = __fmul_rd(a, 0x1.715478p+0f);
    float t;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(p));
    const float r = __saturatef(fmaf(p, -0x1.62e43p-1f, a));
    return fmaf(t, r, t);
}
// (1 + p)(1 + t) - 1
__device__ __forceinline__ float join_log1p(float p, float t) { return fmaf(p, t, p + t); }

template <int KIND, int SPLIT, int DP>
__global__ void __launch_bounds__(kGlmThreads, 1) glm_tc_kernel(GlmParams p) {
    using S = GlmShape<KIND, SPLIT, DP>;
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr size_t ABUF = (size_t)S::NPART * S::A_PART;
    unsigned char *s_a = smem;               // two A buffers
    unsigned char *s_b = smem + 2 * ABUF;    // ring x TILE
    __shared__ __align__(8) uint64_t a_full[2], a_empty[2], b_full[kGlmRing], b_empty[kGlmRing], d_full[2], d_empty[2];
    __shared__ __align__(8) uint64_t bb_full[4], part_full[4][4];
    __shared__ GlmPair s_bb[4][kGlmRows], s_part[4][kGlmParts - 1][kGlmRows];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    const int tid = threadIdx.x, warp = tc::uniform_warp(), lane = tid & 31;
    const int R = p.ring, T = p.tiles;
    if (warp == 0) tc::tmem_alloc(&tmem_base, 512);
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&a_full[b], kGlmConvWarps);
            tc::mbar_init(&a_empty[b], 1);
            tc::mbar_init(&d_full[b], 1);
            tc::mbar_init(&d_empty[b], kGlmEpiWarps);
        }
        for (int b = 0; b < kGlmRing; ++b) {
            tc::mbar_init(&b_full[b], 1);
            tc::mbar_init(&b_empty[b], 1);
        }
        for (int b = 0; b < 4; ++b) {
            tc::mbar_init(&bb_full[b], kGlmConvWarps);
            for (int q = 0; q < 4; ++q) tc::mbar_init(&part_full[b][q], kGlmParts - 1);
        }
        tc::fence_mbar_init();
        abort_flag = 0;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = tc::uniform(tmem_base);
    auto wait = [&](uint64_t *bar, uint32_t parity) -> bool {
        if (abort_flag) return false;
        if (tc::mbar_wait(bar, parity)) return true;
        atomicExch(p.error, 1);
        abort_flag = 1;
        return false;
    };
    const int64_t row_tiles = (p.n + kGlmRows - 1) / kGlmRows;
    const int my_tiles = (int)((row_tiles - (int64_t)blockIdx.x + gridDim.x - 1) / gridDim.x);
    const int64_t J = (int64_t)my_tiles * T;  // items: (row tile, observation tile)
    const bool resident = T <= R;             // every observation tile stays in its slot

    if (warp == 0) {
        // ================= issuer: observation tiles in, MMAs out =================
        int64_t issued = 0, waited = 0;
        int t_load = 0;
        auto load = [&]() {  // the next item's observation tile into the next slot
            const int slot = (int)(issued % R);
            if (lane == 0) {
                tc::mbar_arrive_expect_tx(&b_full[slot], (uint32_t)S::TILE);
                tc::bulk_copy_g2s(s_b + (size_t)slot * S::TILE, p.ops + (size_t)t_load * S::TILE, (uint32_t)S::TILE,
                                  &b_full[slot]);
            }
            __syncwarp();
            ++issued;
            if (++t_load == T) t_load = 0;
        };
        for (int q = 0; q < (resident ? T : R) && q < J; ++q) load();
        const uint32_t idesc = tc::instr_desc(KIND, kGlmRows, kGlmCols);
        constexpr uint32_t LBO_A = kGlmRows * 16, LBO_B = kGlmCols * 16;
        int ok = 1, it = 0, t = 0;
        for (int64_t j = 0; j < J && ok; ++j) {
            const int slot = resident ? t : (int)(j % R);
            {
                bool fine = t != 0 || wait(&a_full[it & 1], (uint32_t)((it >> 1) & 1));
                if (fine && (!resident || it == 0)) {
                    fine = wait(&b_full[slot], resident ? 0u : (uint32_t)((j / R) & 1));
                    if (fine) waited = j + 1;
                }
                if (fine && j >= 2) fine = wait(&d_empty[j & 1], (uint32_t)(((j - 2) >> 1) & 1));
                fine = __all_sync(0xffffffffu, fine);
                tc::fence_after_sync();
                if (fine) {
                    const uint32_t dt = tbase + (uint32_t)((j & 1) * kGlmCols);
                    const uint32_t a0 = tc::smem_u32(s_a + (size_t)(it & 1) * ABUF);
                    const uint32_t b0 = tc::smem_u32(s_b + (size_t)slot * S::TILE);
#pragma unroll
                    for (int s = 0; s < S::KSTEPS; ++s) {
                        const uint64_t da = tc::smem_desc(a0 + s * 2 * LBO_A, LBO_A, 128);
                        const uint64_t db = tc::smem_desc(b0 + s * 2 * LBO_B, LBO_B, 128);
                        if (KIND == tc::kTF32) {
                            tc::mma_tf32_elect(dt, da, db, idesc, s > 0);
                        } else {
                            tc::mma_elect(dt, da, db, idesc, s > 0);
                            if (SPLIT == 3) {
                                const uint64_t dal = tc::smem_desc(a0 + (uint32_t)S::A_PART + s * 2 * LBO_A, LBO_A, 128);
                                const uint64_t dbl = tc::smem_desc(b0 + (uint32_t)S::B_PART + s * 2 * LBO_B, LBO_B, 128);
                                tc::mma_elect(dt, dal, db, idesc, true);
                                tc::mma_elect(dt, da, dbl, idesc, true);
                            }
                        }
                    }
                }
                tc::commit_elect(&d_full[j & 1]);  // arrives when this item's MMAs (issued or not) are done
                if (!resident) tc::commit_elect(&b_empty[slot]);
                if (t == T - 1) tc::commit_elect(&a_empty[it & 1]);
                if (!fine) ok = 0;
            }
            // refill the slot the previous item's MMAs have finished with
            if (ok && !resident && j >= 1 && j + R - 1 < J) {
                int fine = 1;
                if (lane == 0) fine = wait(&b_empty[(j - 1) % R], (uint32_t)(((j - 1) / R) & 1));
                if (__shfl_sync(0xffffffffu, fine, 0)) load();
            }
            if (++t == T) {
                t = 0;
                ++it;
            }
        }
        // drain: every requested copy lands before the CTA exits
        if (lane == 0)
            for (int64_t q = waited; q < issued; ++q) tc::mbar_wait(&b_full[q % R], (uint32_t)((q / R) & 1));
    } else if (warp < kGlmFirstEpi) {
        // ================= converters: sample rows -> A operand =================
        const int r = tid - 32;
        const bool vec = p.d % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
        for (int it = 0; it < my_tiles; ++it) {
            const int64_t i = ((int64_t)blockIdx.x + (int64_t)it * gridDim.x) * kGlmRows + r;
            const float *xr = p.x + (i < p.n ? i : 0) * p.d;
            const int dim = i < p.n ? p.d : 0;
            float v[DP];
#pragma unroll
            for (int c = 0; c < DP; c += 4) {
                if (vec && c < dim) {
                    const float4 f = *reinterpret_cast<const float4 *>(xr + c);
                    v[c] = f.x; v[c + 1] = f.y; v[c + 2] = f.z; v[c + 3] = f.w;
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[c + u] = c + u < dim ? xr[c + u] : 0.f;
                }
            }
            if (it >= 2) {
                int ok = 1;
                if (lane == 0) ok = wait(&a_empty[it & 1], (uint32_t)(((it - 2) >> 1) & 1));
                if (!__shfl_sync(0xffffffffu, ok, 0)) break;
            }
            unsigned char *a = s_a + (size_t)(it & 1) * ABUF;
#pragma unroll
            for (int q = 0; q < S::KG; ++q) {
                const uint4 hi = glm_pack<KIND>(v + q * S::PER);
                *reinterpret_cast<uint4 *>(a + (size_t)q * kGlmRows * 16 + r * 16) = hi;
                if (S::NPART == 2)
                    *reinterpret_cast<uint4 *>(a + S::A_PART + (size_t)q * kGlmRows * 16 + r * 16) =
                        glm_pack_lo(v + q * S::PER, hi);
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&a_full[it & 1]);
            // |x|^2 with error-free products; slot it & 3 was read before item (it - 3, 0) was released
            GlmPair bb{0.f, 0.f};
#pragma unroll
            for (int c = 0; c < DP; ++c) {
                const float sq = v[c] * v[c];
                bb.add(sq, fmaf(v[c], v[c], -sq));
            }
            s_bb[it & 3][r] = bb;
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&bb_full[it & 3]);
        }
    } else {
        // ================= epilogue: quadrant warp % 4, 64 columns of the accumulator =================
        const int qd = warp & 3, part = (warp - kGlmFirstEpi) >> 2, row = 32 * qd + lane;
        const bool logistic = p.kind == ISSM_TARGET_LOGISTIC;
        const bool yvec = (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
        GlmPair acc{0.f, 0.f}, bb{0.f, 0.f};
        int it = 0, t = 0;
        for (int64_t j = 0; j < J; ++j) {
            bool ok = __all_sync(0xffffffffu, wait(&d_full[j & 1], (uint32_t)((j >> 1) & 1)));
            tc::fence_after_sync();
            if (!ok) break;
            if (t == 0) {
                acc = GlmPair{0.f, 0.f};
                if (part == 0) {
                    if (!__all_sync(0xffffffffu, wait(&bb_full[it & 3], (uint32_t)((it >> 2) & 1)))) break;
                    bb = s_bb[it & 3][row];
                }
            }
#pragma unroll 1
            for (int c = 0; c < kGlmPartCols; c += 32) {
                const int o0 = t * kGlmCols + part * kGlmPartCols + c;
                if (o0 >= p.nobs) break;
                float v[32], s[4] = {0.f, 0.f, 0.f, 0.f};
                tc::tmem_ld32(tbase + ((uint32_t)(32 * qd) << 16) +
                                  (uint32_t)((int)(j & 1) * kGlmCols + part * kGlmPartCols + c), v);
                // FULL: 32 observations, y read 16 bytes at a time; no test per pair
                auto terms = [&](auto full, auto kind) {
                    constexpr bool FULL = decltype(full)::value, LOGISTIC = decltype(kind)::value;
                    float q[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int u0 = 0; u0 < 32; u0 += 4) {
                        float y[4];
                        if constexpr (FULL) {
                            const float4 f = __ldg(reinterpret_cast<const float4 *>(p.y + o0 + u0));
                            y[0] = f.x; y[1] = f.y; y[2] = f.z; y[3] = f.w;
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e) y[e] = o0 + u0 + e < p.nobs ? __ldg(p.y + o0 + u0 + e) : 0.f;
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const bool in = FULL || o0 + u0 + e < p.nobs;
                            const float eta = v[u0 + e];
                            if constexpr (LOGISTIC) {
                                // y eta - max(eta, 0) - log(1 + t); q, the product of (1 + t)
                                // less one, stays below 2^32
                                q[e] = join_log1p(q[e], in ? exp_neg(eta) : 0.f);
                                const float z = fmaf(y[e], eta, -fmaxf(eta, 0.f));
                                s[e] += in ? z : 0.f;
                            } else {
                                const float r = in ? y[e] - eta : 0.f;
                                s[e] = fmaf(r, r, s[e]);
                            }
                        }
                    }
                    if constexpr (LOGISTIC) s[0] -= log1pf(join_log1p(join_log1p(q[0], q[1]), join_log1p(q[2], q[3])));
                };
                const bool full = o0 + 32 <= p.nobs && yvec;
                if (logistic) {
                    if (full) terms(std::true_type(), std::true_type());
                    else terms(std::false_type(), std::true_type());
                } else {
                    if (full) terms(std::true_type(), std::false_type());
                    else terms(std::false_type(), std::false_type());
                }
                acc.add((s[0] + s[1]) + (s[2] + s[3]));
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&d_empty[j & 1]);
            if (++t < T) continue;
            t = 0;
            // the column parts of a row meet in shared memory; slot it & 3 was
            // read before the items two row tiles back were released
            if (part > 0) {
                s_part[it & 3][part - 1][row] = acc;
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&part_full[it & 3][qd]);
            } else {
                if (!__all_sync(0xffffffffu, wait(&part_full[it & 3][qd], (uint32_t)((it >> 2) & 1)))) break;
#pragma unroll
                for (int q = 0; q < kGlmParts - 1; ++q) {
                    const GlmPair o = s_part[it & 3][q][row];
                    acc.add(o.h, o.l);
                }
                const int64_t i = ((int64_t)blockIdx.x + (int64_t)it * gridDim.x) * kGlmRows + row;
                if (i < p.n)
                    p.out[i] = (float)fma(acc.value(), p.scale, fma(bb.value(), p.prior_scale, p.constant));
            }
            ++it;
        }
    }
    // ---- every role is done; in-flight MMAs have completed before TMEM is freed ----
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0 && abort_flag && J > 0) tc::mbar_wait(&d_full[(J - 1) & 1], (uint32_t)(((J - 1) >> 1) & 1));
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tbase, 512);
}

static int glm_dp(int d) { return d <= 16 ? 16 : d <= 32 ? 32 : 64; }

size_t glm_operand_bytes(int nobs, int d, int precision) {
    const int DP = glm_dp(d);
    const int tiles = (nobs + kGlmCols - 1) / kGlmCols;
    const size_t eb = precision == ISSM_PREC_TF32 ? 4 : 2;
    const size_t parts = precision == ISSM_PREC_BF16 ? 2 : 1;
    return (size_t)tiles * parts * (size_t)DP * eb * kGlmCols;
}

template <int KIND, int SPLIT, int DP>
static int glm_prepare_t(const float *X, int nobs, int d, unsigned char *ops, cudaStream_t stream) {
    using S = GlmShape<KIND, SPLIT, DP>;
    const int tiles = (nobs + kGlmCols - 1) / kGlmCols;
    const int64_t total = (int64_t)tiles * S::KG * kGlmCols;
    glm_prepare_kernel<KIND, SPLIT, DP><<<grid_for(total, 256, 4), 256, 0, stream>>>(X, nobs, d, tiles, ops);
    note_launch();
    return (int)cudaGetLastError();
}

template <int KIND, int SPLIT, int DP>
static int glm_run_t(GlmParams p, cudaStream_t stream) {
    using S = GlmShape<KIND, SPLIT, DP>;
    const size_t base = 2 * S::NPART * S::A_PART;
    const int ring = min(kGlmRing, (int)((kGlmMaxSmem - base) / S::TILE));
    if (ring < 2) return ISSM_E_UNSUPPORTED;
    p.ring = ring;
    // at least half an SM's shared memory, so one CTA (and its 512 TMEM
    // columns) per SM: the allocation never waits for another CTA's columns
    const size_t smem = max((size_t)(120 * 1024), base + (size_t)ring * S::TILE);
    auto kern = glm_tc_kernel<KIND, SPLIT, DP>;
    const int st = allow_dynamic_smem((const void *)kern);
    if (st) return st;
    const int blocks = (int)min((p.n + kGlmRows - 1) / kGlmRows, (int64_t)device_sms());
    if (blocks < 1) return 0;
    { kern<<<blocks, kGlmThreads, smem, stream>>>(p); note_launch(); }
    return (int)cudaGetLastError();
}

#define ISSM_GLM_DISPATCH(FN, ...)                                                           \
    do {                                                                                     \
        const int DP_ = glm_dp(d);                                                           \
        if (precision == ISSM_PREC_TF32) {                                                   \
            if (DP_ == 16) return FN<tc::kTF32, 1, 16>(__VA_ARGS__);                         \
            if (DP_ == 32) return FN<tc::kTF32, 1, 32>(__VA_ARGS__);                         \
            return FN<tc::kTF32, 1, 64>(__VA_ARGS__);                                        \
        }                                                                                    \
        if (precision == ISSM_PREC_BF16) {                                                   \
            if (DP_ == 16) return FN<tc::kBF16, 3, 16>(__VA_ARGS__);                         \
            if (DP_ == 32) return FN<tc::kBF16, 3, 32>(__VA_ARGS__);                         \
            return FN<tc::kBF16, 3, 64>(__VA_ARGS__);                                        \
        }                                                                                    \
        if (DP_ == 16) return FN<tc::kBF16, 1, 16>(__VA_ARGS__);                             \
        if (DP_ == 32) return FN<tc::kBF16, 1, 32>(__VA_ARGS__);                             \
        return FN<tc::kBF16, 1, 64>(__VA_ARGS__);                                            \
    } while (0)

int glm_prepare(const issm_target *t, int precision, void *ops, cudaStream_t stream) {
    const int d = t->dim;
    ISSM_GLM_DISPATCH(glm_prepare_t, (const float *)t->a, t->count, d, (unsigned char *)ops, stream);
}

int glm_logdensity(const issm_target *t, int precision, const void *ops, const float *x, int64_t n, float *out,
                   int *error, cudaStream_t stream) {
    const int d = t->dim;
    GlmParams p{};
    p.d = d;
    p.nobs = t->count;
    p.kind = t->kind;
    p.tiles = (t->count + kGlmCols - 1) / kGlmCols;
    p.n = n;
    p.x = x;
    p.y = (const float *)t->b;
    p.ops = (const unsigned char *)ops;
    p.out = out;
    const double pv = (double)(float)t->p1, sg = (double)(float)t->p0;
    const bool logistic = t->kind == ISSM_TARGET_LOGISTIC;
    p.scale = logistic ? 1.0 : -1.0 / (2.0 * sg * sg);
    p.prior_scale = -1.0 / (2.0 * pv);
    p.constant = -0.5 * d * (kGlmLog2Pi + log(pv)) -
                 (logistic ? 0.0 : 0.5 * t->count * (kGlmLog2Pi + 2.0 * log(sg)));
    p.error = error;
    ISSM_GLM_DISPATCH(glm_run_t, p, stream);
}

}  // namespace issm
