// mixture_pair.cu — the tensor-core mixture density (see mixture_tc.cu for the
// contraction and its precision forms) for more components than one accumulator
// holds: two 128-sample tiles share every chunk of component operands.
//
// With z_k = W_k (x - c) - b_k and W_k = L_k^-1 lower triangular:
//   * a chunk is NC = 128 / DP components, their rows interleaved: operand row
//     n = j NC + kk is row j of component kk, so one MMA of N = 128 covers the
//     chunk and the rows that a K slice touches are its last ones;
//   * the K slice of coordinates 16 s .. (BF16; 8 s .. TF32) has non-zero operand
//     rows j >= 16 s only: its MMA runs over those rows (N shrinks by 16 NC per
//     slice) and only they are kept, the slices packed one after the other so a
//     chunk is one bulk copy: 37% fewer bytes and MMA columns at DP = 64;
//   * the offset -b_k is one K slice of the hi parts alone, two operand columns
//     hi(-b) and lo(-b) against samples extended by (1, 1).
// One CTA per SM walks pairs of tiles (single ones, TILES = 1, where there are no more
// tiles than SMs); an item is a (pair, chunk):
//   warps 1-8   read the next pair's rows into registers, centre, round and
//               split them into the A operand (two tiles, one buffer);
//   warps 0, 17 issue the MMAs of the even and the odd items, each into its own
//               pair of accumulators;
//   warp 18     copies the chunks through a ring of four slots;
//   warps 9-16  reduce the other: four warps (TMEM lane quadrants) per tile,
//               |z|^2 per component, the radial density and an online
//               log-sum-exp that takes a chunk's terms at once.
// One tile at a time, full operand squares and one epilogue warp per quadrant
// ran at 33 bytes of operands per clock and SM out of L2, 1,268 us for
// 1,000,003 samples x 40 components, d = 64 (BF16x3); this form takes 497, 370 of
// them tensor time (1,418 clocks per item). 4,194,304 x 64, d = 16: 3,766 -> 1,095,
// bound by the epilogue's exponentials. Few samples share the tiles out worse
// (pairs, not tiles, per SM), yet 50,000 x 40, d = 64 still gains, 91 -> 58, and
// x 8 35.5 -> 31.4. Every wait is bounded; a timeout sets the sticky error word and
// the CTA unwinds after draining its copies and MMAs.
#include "mixture_tc.cuh"

namespace issm {

constexpr int kPairConvWarps = 8, kPairEpiWarps = 8;
constexpr int kPairFirstEpi = 1 + kPairConvWarps;
constexpr int kPairIssuer2 = kPairFirstEpi + kPairEpiWarps, kPairLoader = kPairIssuer2 + 1;
constexpr int kPairThreads = 32 * (kPairLoader + 1);
constexpr int kPairRing = 4;  // even: a slot's items are one issuer's
constexpr int kPairN = 128;  // accumulator columns of one tile: operand rows of a chunk

template <int KIND, int SPLIT, int DP> struct PairShape {
    static constexpr int EB = KIND == tc::kBF16 ? 2 : 4;
    static constexpr int PER = 16 / EB;             // elements per 16-byte K group
    static constexpr int KG = DP / PER;             // K groups of the coordinates
    static constexpr int KGX = KG + 2;              // hi part: plus the offset slice
    static constexpr int NC = kPairN / DP;          // components per chunk
    static constexpr int KSTEPS = KG / 2;           // K slices of the coordinates
    static constexpr int GROUP = kPairN * 16;       // bytes of one K group, of A (128 samples) and of B
    static constexpr int LO = SPLIT == 3 ? KG : 0;  // lo part groups
    static constexpr size_t TILE = (size_t)(KGX + LO) * GROUP;  // A operand of a tile
    // a chunk: the offset slice, then the hi and the lo part's slices, slice s
    // two K groups of the operand rows n >= first(s)
    static constexpr int PARTS = SPLIT == 3 ? 2 : 1;
    __host__ __device__ static constexpr int first(int s) { return 2 * PER * s * NC; }
    __host__ __device__ static constexpr int slice(int part, int s) {  // its offset
        return 2 * GROUP + part * 32 * (kPairN * KSTEPS - PER * NC * KSTEPS * (KSTEPS - 1)) +
               32 * (kPairN * s - PER * NC * s * (s - 1));
    }
    static constexpr uint32_t CHUNK = slice(PARTS, 0);
};

// Operand form of one slot per CTA: row n = j NC + kk of K group q of a part at
// slice(part, q / 2) + ((q & 1) (128 - first) + n - first) 16 of its chunk.
template <int KIND, int SPLIT, int DP>
__global__ void __launch_bounds__(256) pair_prepare_kernel(const float *__restrict__ w, const float *__restrict__ loc,
                                                           int d, int first, int cslot, unsigned char *__restrict__ ops,
                                                           float *__restrict__ center) {
    using S = PairShape<KIND, SPLIT, DP>;
    constexpr int LD = DP + 1;
    __shared__ float ws[DP * LD], dc[DP], nb[DP];
    const int k = first + blockIdx.x, kk = blockIdx.x % S::NC, tid = threadIdx.x;
    const float *wk = w + (size_t)k * DP * DP;
    for (int e = tid; e < DP * DP; e += 256) ws[(e / DP) * LD + e % DP] = wk[e];
    for (int c = tid; c < DP; c += 256) {
        const float cc = c < d ? loc[(size_t)cslot * d + c] : 0.f;
        dc[c] = c < d ? loc[(size_t)k * d + c] - cc : 0.f;
        if (blockIdx.x == 0) center[c] = cc;
    }
    __syncthreads();
    // -b = -W (mu - c) in FP32, four lanes per row
    if (tid < 4 * DP) {
        const int j = tid >> 2;
        float acc = 0.f;
        for (int c = tid & 3; c < d; c += 4) acc = fmaf(ws[j * LD + c], dc[c], acc);
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        if ((tid & 3) == 0) nb[j] = -acc;
    }
    __syncthreads();
    unsigned char *chunk = ops + (size_t)(blockIdx.x / S::NC) * S::CHUNK;
    for (int e = tid; e < S::KG * DP; e += 256) {
        const int q = e / DP, j = e - q * DP, n = j * S::NC + kk, n0 = S::first(q >> 1);
        if (n < n0) continue;  // above the slice's diagonal: zero, not kept
        float v[S::PER];
#pragma unroll
        for (int m = 0; m < S::PER; ++m) v[m] = ws[j * LD + q * S::PER + m];
        const uint4 hi = pack_hi<KIND>(v);
        const int at = ((q & 1) * (kPairN - n0) + n - n0) * 16;
        *reinterpret_cast<uint4 *>(chunk + S::slice(0, q >> 1) + at) = hi;
        if (S::PARTS == 2) *reinterpret_cast<uint4 *>(chunk + S::slice(1, q >> 1) + at) = pack_lo(v, hi);
    }
    for (int j = tid; j < DP; j += 256) {  // (hi(-b), lo(-b), 0, ..), then zeros
        float v[S::PER];
#pragma unroll
        for (int m = 0; m < S::PER; ++m) v[m] = 0.f;
        v[0] = nb[j];
        uint4 hi = pack_hi<KIND>(v);
        v[1] = KIND == tc::kTF32 ? nb[j] - __uint_as_float(hi.x) : nb[j] - __uint_as_float(hi.x << 16);
        *reinterpret_cast<uint4 *>(chunk + (j * S::NC + kk) * 16) = pack_hi<KIND>(v);
        *reinterpret_cast<uint4 *>(chunk + S::GROUP + (j * S::NC + kk) * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
}

template <int KIND, int SPLIT, int DP, int TILES>
__global__ void __launch_bounds__(kPairThreads, 1) mixture_pair_kernel(TcParams p) {
    using S = PairShape<KIND, SPLIT, DP>;
    constexpr int NC = S::NC;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *s_a = smem;                // two tiles
    unsigned char *s_b = smem + 2 * S::TILE;  // ring of chunks
    __shared__ __align__(8) uint64_t a_full, a_empty, b_full[kPairRing], b_empty[kPairRing], d_full[2], d_empty[2],
        drained[2];
    __shared__ __align__(16) float s_c[DP];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;
    const int tid = threadIdx.x, warp = tc::uniform_warp(), lane = tid & 31;
    if (warp == 0) tc::tmem_alloc(&tmem_base, 512);
    if (tid == 0) {
        tc::mbar_init(&a_full, kPairConvWarps);
        tc::mbar_init(&a_empty, 2);
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&drained[b], 1);
            tc::mbar_init(&d_full[b], 1);
            tc::mbar_init(&d_empty[b], kPairEpiWarps);
        }
        for (int b = 0; b < kPairRing; ++b) {
            tc::mbar_init(&b_full[b], 1);
            tc::mbar_init(&b_empty[b], 1);
        }
        tc::fence_mbar_init();
        abort_flag = 0;
    }
    for (int c = tid; c < DP; c += kPairThreads) s_c[c] = p.center[c];
    // the samples' offset slice: (1, 1, 0, ..)
    for (int e = tid; e < 2 * 2 * kTcTile; e += kPairThreads) {
        const int row = e % kTcTile, g = (e / kTcTile) & 1, tile = e / (2 * kTcTile);
        const uint4 ones = KIND == tc::kTF32 ? make_uint4(0x3F800000u, 0x3F800000u, 0u, 0u)
                                             : make_uint4(0x3F803F80u, 0u, 0u, 0u);
        *reinterpret_cast<uint4 *>(s_a + tile * S::TILE + (size_t)(S::KG + g) * S::GROUP + row * 16) =
            g == 0 ? ones : make_uint4(0u, 0u, 0u, 0u);
    }
    tc::fence_proxy_async();
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
    const int nchunks = (p.nslots + NC - 1) / NC;
    const int npairs = (p.ntiles + TILES - 1) / TILES;
    const int my_pairs = (npairs - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const int J = my_pairs * nchunks;
    auto row0_of = [&](int it) -> int64_t { return ((int64_t)blockIdx.x + (int64_t)it * gridDim.x) * (TILES * kTcTile); };

    if (warp == 0 || warp == kPairIssuer2) {
        // ================= issuers: warp 0 the even items, warp 17 the odd ones =================
        // An issuer's waits before its next item run while the other's MMAs do: one
        // issuer, blocked while its MMAs queue and then waiting on four barriers, took
        // 2,790 clocks per item (764 us in all), two take 1,815 (497). Items alternate accumulator pairs and, the ring being even,
        // slots, so an issuer sees every phase of the barriers it waits on.
        const int mine = warp == 0 ? 0 : 1;
        int it = 0, ch = mine, seen = -1;
        for (int j = mine; j < J; j += 2) {
            const int slot = j % kPairRing;
            bool fine = seen == it || wait(&a_full, (uint32_t)(it & 1));
            seen = it;
            if (fine) fine = wait(&b_full[slot], (uint32_t)((j / kPairRing) & 1));
            if (fine && j >= 2) fine = wait(&d_empty[mine], (uint32_t)(((j - 2) >> 1) & 1));
            fine = __all_sync(0xffffffffu, fine);
            tc::fence_after_sync();
            if (fine) {
                const uint32_t b0 = tc::smem_u32(s_b + (size_t)slot * S::CHUNK);
                const uint32_t full = tc::instr_desc(KIND, kTcTile, kPairN);
                const uint64_t db0 = tc::smem_desc(b0, S::GROUP, 128);
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    if (g >= TILES) break;
                    const uint32_t a0 = tc::smem_u32(s_a + g * S::TILE);
                    const uint32_t dt = tbase + (uint32_t)(mine * 2 * kPairN + g * kPairN);
                    const uint64_t da0 = tc::smem_desc(a0 + S::KG * S::GROUP, S::GROUP, 128);
                    if (KIND == tc::kTF32) tc::mma_tf32_elect(dt, da0, db0, full, false);
                    else tc::mma_elect(dt, da0, db0, full, false);
#pragma unroll
                    for (int s = 0; s < S::KSTEPS; ++s) {
                        // operand rows j >= 2 PER s: the last columns of the accumulator
                        const int n0 = S::first(s);
                        const uint32_t lbo = (uint32_t)(kPairN - n0) * 16;
                        const uint32_t idesc = tc::instr_desc(KIND, kTcTile, kPairN - n0);
                        const uint64_t da = tc::smem_desc(a0 + s * 2 * S::GROUP, S::GROUP, 128);
                        const uint64_t db = tc::smem_desc(b0 + S::slice(0, s), lbo, 128);
                        if (KIND == tc::kTF32) {
                            tc::mma_tf32_elect(dt + n0, da, db, idesc, true);
                        } else {
                            tc::mma_elect(dt + n0, da, db, idesc, true);
                            if (SPLIT == 3) {
                                const uint64_t dal = tc::smem_desc(a0 + (S::KGX + s * 2) * S::GROUP, S::GROUP, 128);
                                const uint64_t dbl = tc::smem_desc(b0 + S::slice(1, s), lbo, 128);
                                tc::mma_elect(dt + n0, dal, db, idesc, true);
                                tc::mma_elect(dt + n0, da, dbl, idesc, true);
                            }
                        }
                    }
                }
            }
            // commits arrive when this issuer's earlier MMAs have completed, issued or not
            tc::commit_elect(&d_full[mine]);
            tc::commit_elect(&b_empty[slot]);
            if (ch + 2 >= nchunks) tc::commit_elect(&a_empty);  // my last item of the pair
            if (!fine) break;
            ch += 2;
            if (ch >= nchunks) {
                ch -= nchunks;
                ++it;
            }
        }
        // drain: my MMAs have completed before the accumulators are freed
        tc::commit_elect(&drained[mine]);
        tc::mbar_wait(&drained[mine], 0u);
    } else if (warp == kPairLoader) {
        // ================= loader: chunks into the ring =================
        int issued = 0, ch = 0;
        for (int j = 0; j < J; ++j) {
            const int slot = j % kPairRing;
            if (j >= kPairRing && !__all_sync(0xffffffffu, wait(&b_empty[slot], (uint32_t)((j / kPairRing - 1) & 1)))) break;
            if (lane == 0) {
                tc::mbar_arrive_expect_tx(&b_full[slot], S::CHUNK);
                tc::bulk_copy_g2s(s_b + (size_t)slot * S::CHUNK, p.ops + (size_t)ch * S::CHUNK, S::CHUNK, &b_full[slot]);
            }
            __syncwarp();
            issued = j + 1;
            if (++ch == nchunks) ch = 0;
        }
        // drain: every requested copy has landed before the CTA exits
        if (lane == 0)
            for (int q = max(0, issued - kPairRing); q < issued; ++q)
                tc::mbar_wait(&b_full[q % kPairRing], (uint32_t)((q / kPairRing) & 1));
    } else if (warp < kPairFirstEpi) {
        // ================= converters: half a row of each tile per thread =================
        const int ctid = tid - 32, row = ctid & (kTcTile - 1), half = ctid >> 7;
        constexpr int HC = DP / 2;
        const bool vec = p.d % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
        for (int it = 0; it < my_pairs; ++it) {
            float v[2][HC];  // loaded before the wait: the previous pair's MMAs hide the latency
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                const int64_t i = row0_of(it) + g * kTcTile + row;
                const bool active = i < p.n && g < TILES;
                const float *xr = p.x + (active ? i : 0) * p.d;
#pragma unroll
                for (int u = 0; u < HC; u += 4) {
                    const int c = half * HC + u;
                    if (vec && active && c < p.d) {
                        const float4 f = *reinterpret_cast<const float4 *>(xr + c);
                        v[g][u] = f.x; v[g][u + 1] = f.y; v[g][u + 2] = f.z; v[g][u + 3] = f.w;
                    } else {
#pragma unroll
                        for (int m = 0; m < 4; ++m) v[g][u + m] = active && c + m < p.d ? xr[c + m] : s_c[c + m];
                    }
                }
            }
            if (it >= 1) {
                int ok = 1;
                if (lane == 0) ok = wait(&a_empty, (uint32_t)((it - 1) & 1));
                if (!__shfl_sync(0xffffffffu, ok, 0)) break;
            }
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                if (g >= TILES) break;
                unsigned char *a = s_a + g * S::TILE;
#pragma unroll
                for (int u = 0; u < HC; u += S::PER) {
                    const int q = (half * HC + u) / S::PER;
                    float z[S::PER];
#pragma unroll
                    for (int m = 0; m < S::PER; ++m) z[m] = v[g][u + m] - s_c[half * HC + u + m];
                    const uint4 hi = pack_hi<KIND>(z);
                    *reinterpret_cast<uint4 *>(a + (size_t)q * S::GROUP + row * 16) = hi;
                    if (S::LO) *reinterpret_cast<uint4 *>(a + (size_t)(S::KGX + q) * S::GROUP + row * 16) = pack_lo(z, hi);
                }
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&a_full);
        }
    } else {
        // ================= epilogue: tile (warp - 9) / 4, lane quadrant warp % 4 =================
        const int qd = warp & 3, g = (warp - kPairFirstEpi) >> 2;
        const int ggen = p.den_kind == ISSM_DENOM_PARTIAL ? p.group[p.fixed_slot] : 0;
        const bool gaussian = p.family == ISSM_GAUSSIAN;
        LseState<float> lse;
        float gen_lq = 0.f;
        int it = 0, ch = 0;
        for (int j = 0; j < J; ++j) {
            const int k0 = p.first_slot + ch * NC, cnt = min(NC, p.last_slot - k0 + 1);
            float ln[NC], cf[NC];
#pragma unroll
            for (int kk = 0; kk < NC; ++kk) {
                ln[kk] = kk < cnt ? p.lognorm[k0 + kk] : 0.f;
                cf[kk] = kk < cnt && p.coef ? p.coef[k0 + kk] : 0.f;
            }
            if (!__all_sync(0xffffffffu, wait(&d_full[j & 1], (uint32_t)((j >> 1) & 1)))) break;
            tc::fence_after_sync();
            if (TILES == 1 && g != 0) {  // no second tile: release the accumulators only
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&d_empty[j & 1]);
                continue;
            }
            constexpr int CH = NC < 4 ? 4 / NC : 1;  // independent chains per component
            float r2[NC * CH];
#pragma unroll
            for (int u = 0; u < NC * CH; ++u) r2[u] = 0.f;
            const uint32_t base = tbase + ((uint32_t)(32 * qd) << 16) + (uint32_t)((j & 1) * 2 * kPairN + g * kPairN);
#pragma unroll
            for (int c = 0; c < kPairN; c += 64) {
                float v[64];
                tc::tmem_ld64(base + (uint32_t)c, v);
#pragma unroll
                for (int u = 0; u < 64; ++u) r2[u % (NC * CH)] = fmaf(v[u], v[u], r2[u % (NC * CH)]);
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&d_empty[j & 1]);
            // the chunk's terms, then one rescaling of the running sum
            float term[NC], top = lse.m;
#pragma unroll
            for (int kk = 0; kk < NC; ++kk) {
                float r = r2[kk];
#pragma unroll
                for (int u = 1; u < CH; ++u) r += r2[kk + u * NC];
                float lq;
                if (gaussian) {
                    lq = ln[kk] - 0.5f * r;
                } else {
                    const float nu = kk < cnt ? p.dofs[k0 + kk] : 1.f;
                    lq = ln[kk] - (nu + (float)p.d) * 0.5f * log1pf(r / nu);
                }
                const int k = k0 + kk;
                bool member = kk < cnt;
                if (p.den_kind == ISSM_DENOM_PARTIAL) member = member && p.group[kk < cnt ? k : k0] == ggen;
                if (kk < cnt && k == p.fixed_slot) gen_lq = lq;
                term[kk] = member ? cf[kk] + lq : -INFINITY;
                if (isnan(term[kk])) {
                    lse.nan = true;
                    term[kk] = -INFINITY;
                }
                top = fmaxf(top, term[kk]);
            }
            if (top > -INFINITY) {
                float s = lse.m == top ? lse.s : lse.s * expf(lse.m - top);
#pragma unroll
                for (int kk = 0; kk < NC; ++kk) s += term[kk] == top ? 1.f : expf(term[kk] - top);
                lse.s = s;
                lse.m = top;
            }
            if (++ch < nchunks) continue;
            ch = 0;
            const int64_t i = row0_of(it) + g * kTcTile + 32 * qd + lane;
            ++it;
            if (i < p.n) {
                float den = lse.value();
                const bool bad = isnan(gen_lq) || gen_lq == -INFINITY || isnan(den) || den == -INFINITY;
                if (bad) {
                    record_failure(p.failures, p.index_base + i + 1, 0, ISSM_REASON_PROPOSAL_INVALID);
                    den = -INFINITY;
                }
                p.out_logden[i] = den;
                if (p.out_generating) p.out_generating[i] = bad ? -INFINITY : gen_lq;
            }
            lse = LseState<float>();
            gen_lq = 0.f;
        }
    }
    // ---- every role is done; in-flight MMAs have completed before TMEM is freed ----
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tbase, 512);
}

template <int KIND, int SPLIT, int DP>
static int launch_pair_t(TcParams p, const float *w, const float *loc, int cslot, unsigned char *ops, float *center,
                         cudaStream_t stream) {
    using S = PairShape<KIND, SPLIT, DP>;
    static_assert(S::CHUNK % 16 == 0 && S::CHUNK <= (size_t)S::NC * DP * (4 * DP + 64),
                  "a chunk is whole 16-byte groups within its slots' share of the workspace");
    // more than half an SM's shared memory: one CTA (and its 512 TMEM columns)
    // per SM, so the allocation never waits
    const size_t smem = max((size_t)(120 * 1024), 2 * S::TILE + kPairRing * (size_t)S::CHUNK);
    p.ntiles = (int)((p.n + kTcTile - 1) / kTcTile);
    // one tile per CTA while every tile can have an SM of its own: half the MMAs before the
    // last (19,000 samples x 40, d = 64: 31.6 -> 28.1 us, x 8 19.1 -> 17.1)
    const int per = p.ntiles <= device_sms() ? 1 : 2;
    const int blocks = min((p.ntiles + per - 1) / per, device_sms());
    if (blocks < 1) return 0;
    pair_prepare_kernel<KIND, SPLIT, DP><<<p.nslots, 256, 0, stream>>>(w, loc, p.d, p.first_slot, cslot, ops, center);
    note_launch();
    auto kern = per == 1 ? mixture_pair_kernel<KIND, SPLIT, DP, 1> : mixture_pair_kernel<KIND, SPLIT, DP, 2>;
    const int st = allow_dynamic_smem((const void *)kern);
    if (st) return st;
    kern<<<blocks, kPairThreads, smem, stream>>>(p);
    note_launch();
    return (int)cudaGetLastError();
}

int launch_pair(int kind, int DP, TcParams p, const float *w, const float *loc, int cslot, unsigned char *ops,
                float *center, cudaStream_t stream) {
#define ISSM_PAIR_DP(D)                                                                                     \
    if (DP == D)                                                                                            \
        return kind == tc::kTF32 ? launch_pair_t<tc::kTF32, 1, D>(p, w, loc, cslot, ops, center, stream)    \
                                 : launch_pair_t<tc::kBF16, 3, D>(p, w, loc, cslot, ops, center, stream);
    ISSM_PAIR_DP(16)
    ISSM_PAIR_DP(32)
    ISSM_PAIR_DP(64)
#undef ISSM_PAIR_DP
    return ISSM_E_UNSUPPORTED;
}

}  // namespace issm
