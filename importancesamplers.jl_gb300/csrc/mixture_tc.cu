// mixture_tc.cu — tensor-core (tcgen05) form of the factor-bank mixture
// density for FP32 samples: the Mahalanobis contraction runs as an MMA and
// the radial density plus the balance-heuristic log-sum-exp run in the
// epilogue straight out of tensor memory.
//
// For every component k the reference solves L_k z = x - mu_k by forward
// substitution (_packed_gaussian_logdensity!, src/native_execution.jl:346-384).
// Here W_k = L_k^-1 (FP32, cached per slot in issm_bank.inverse_factors) and
// the samples are centred on one shift c (the generating / appended slot's
// mean):
//   z_k = W_k (x - c) - b_k,   b_k = W_k (mu_k - c),
// so each 128-sample tile is one GEMM  D[128 x K*DP] = X'[128 x DP] W^T.
// Precision forms (FP32 accumulation in TMEM in both):
//   TF32    one kind::tf32 MMA per K slice, operands rounded to tf32 (RNE);
//   BF16x3  operands split v = hi + lo in bf16, D = Xh Wh + Xl Wh + Xh Wl,
//           about 16 significant bits per product.
//
// Components that fit one 256-column accumulator (and the shared memory beside
// the staged tiles) run here; more of them in mixture_pair.cu. Two kernels per
// launch:
//   tc_prepare_kernel  one CTA per slot: W_k in MMA operand form (bf16 hi/lo
//                      or tf32, row-contiguous canonical layout) and b_k;
//   mixture_tc_kernel  persistent, one 128-sample tile at a time:
//     * warps 1-8 read the samples into registers and centre, round and split
//       them into the A operand, groups of warps on alternate tiles;
//     * warp 0 copies the operands once and issues the MMAs of a tile into one
//       of two TMEM accumulators;
//     * warps 9-16 reduce the accumulators, four (a TMEM lane quadrant each) per
//       accumulator.
// One component of 1,000,003 samples, d = 64: 70 us with the operand kernel (3.8
// TB/s; reading alone is 40), 101 with rows staged by cp.async and one epilogue
// warp per quadrant; four components 310 -> 115; d = 33, one component 173 -> 66;
// d = 63 237 -> 81.
// Every wait is bounded; a timeout sets the sticky error word and the CTA
// unwinds after draining its outstanding copies and MMAs.
#include "mixture_tc.cuh"
#include "trinv.cuh"

namespace issm {

// Operand form of slot k: the DP x (DP + X) matrix [W_k | -b_k | 0], X = 16
// bf16 or 8 tf32 elements (two extra 16-byte K groups), so the MMA yields
// z = W_k (x - c) - b_k directly against samples extended by a constant 1.
// The `chunk` slots of a launch are one block of NPART parts of KGX = KG + 2 K
// groups: part p, K group q, slot kk, row j at
//   p * chunk*B + q * chunk*DP*16 + kk * DP*16 + j * 16
// (B = DP*KGX*16), the block's shared-memory layout.
template <int KIND, int SPLIT, int DP>
__global__ void __launch_bounds__(256) tc_prepare_kernel(const float *__restrict__ w, const float *__restrict__ loc,
                                                         int d, int first, int chunk, int cslot,
                                                         unsigned char *__restrict__ ops, float *__restrict__ center) {
    constexpr int EB = KIND == tc::kBF16 ? 2 : 4;
    constexpr int PER = 16 / EB;
    constexpr int KG = DP / PER;
    constexpr int KGX = KG + 2;
    constexpr int NPART = SPLIT == 3 ? 2 : 1;
    constexpr int LD = DP + 1;
    constexpr int B_COMP = DP * KGX * 16;
    __shared__ float ws[DP * LD];
    __shared__ float dc[DP];
    __shared__ float nb[DP];
    const int k = first + blockIdx.x;
    const float *wk = w + (size_t)k * DP * DP;
    for (int e = threadIdx.x; e < DP * DP; e += blockDim.x) ws[(e / DP) * LD + e % DP] = wk[e];
    for (int c = threadIdx.x; c < DP; c += blockDim.x) {
        const float cc = c < d ? loc[(size_t)cslot * d + c] : 0.f;
        dc[c] = c < d ? loc[(size_t)k * d + c] - cc : 0.f;
        if (blockIdx.x == 0) center[c] = cc;
    }
    __syncthreads();
    // -b_k = -W_k (mu_k - c) in FP32
    for (int j = threadIdx.x; j < DP; j += blockDim.x) {
        float acc = 0.f;
        for (int c = 0; c < d; ++c) acc = fmaf(ws[j * LD + c], dc[c], acc);
        nb[j] = -acc;
    }
    __syncthreads();
    unsigned char *okp = ops + (size_t)blockIdx.x * DP * 16;
    for (int e = threadIdx.x; e < KGX * DP; e += blockDim.x) {
        const int q = e / DP, j = e - q * DP;
        float v[PER];
#pragma unroll
        for (int m = 0; m < PER; ++m)
            v[m] = q < KG ? ws[j * LD + q * PER + m] : (q == KG && m == 0 ? nb[j] : 0.f);
        const uint4 hi = pack_hi<KIND>(v);
        const size_t off = (size_t)q * chunk * DP * 16 + (size_t)j * 16;
        *reinterpret_cast<uint4 *>(okp + off) = hi;
        if (NPART == 2) *reinterpret_cast<uint4 *>(okp + (size_t)chunk * B_COMP + off) = pack_lo(v, hi);
    }
}

// Warp roles of mixture_tc_kernel.
constexpr int kConvWarps = 8;  // read the samples and build the A operand
constexpr int kEpiWarps = 8;   // per accumulator one per TMEM lane quadrant
constexpr int kFirstEpiWarp = 1 + kConvWarps;
constexpr int kTcThreads = 32 * (1 + kConvWarps + kEpiWarps);
// Every converter warp holds 64 floats per lane, whatever DP: groups of warps on
// alternate tiles, 64 KB of samples on their way per CTA. (All eight warps on one
// tile with the next two prefetched was slower: the proxy fence after a tile's
// stores waits for the loads issued before it.)
__host__ __device__ constexpr int conv_groups(int DP) { return 128 / DP; }
__host__ __device__ constexpr int tc_abufs(int DP) { return DP == 64 ? 3 : DP == 32 ? 6 : 10; }  // A operand buffers

// NOB: one component centred at its own location, whose offset column
// -W (mu - c) is therefore zero: the MMAs run over the coordinates' K groups
// only (K = DP instead of DP + 16), and three A buffers fit.
template <int KIND, int SPLIT, int DP, bool NOB>
__global__ void __launch_bounds__(kTcThreads, 1) mixture_tc_kernel(TcParams p) {
    constexpr int EB = KIND == tc::kBF16 ? 2 : 4;
    constexpr int PER = 16 / EB;              // elements per 16-byte K group
    constexpr int KG = DP / PER;              // K groups of the sample coordinates
    constexpr int KGB = KG + 2;               // operand form: plus the offset column and padding
    constexpr int KGX = NOB ? KG : KGB;       // K groups the MMAs read
    constexpr int NPART = SPLIT == 3 ? 2 : 1;
    constexpr int A_PART = kTcTile * KGX * 16;
    constexpr int B_COMP = DP * KGB * 16;
    constexpr int KSTEPS = KGX / 2;           // MMA K slices of 32 bytes
    constexpr uint32_t LBO_A = kTcTile * 16;
    const int chunk = p.nslots;  // components, all in one accumulator
    constexpr int nbufA = tc_abufs(DP), CG = conv_groups(DP);
    const uint32_t LBO_B = (uint32_t)(chunk * DP * 16);
    const uint32_t CHUNK_BYTES = (uint32_t)(NPART * chunk * B_COMP);

    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *s_a = smem;
    unsigned char *s_b = s_a + (size_t)nbufA * NPART * A_PART;
    __shared__ __align__(8) uint64_t a_full[nbufA], a_empty[nbufA], b_full, d_full[2], d_empty[2];
    __shared__ uint32_t tmem_base;
    __shared__ volatile int abort_flag;

    const int tid = threadIdx.x, warp = tc::uniform_warp(), lane = tid & 31;
    const int NW = chunk * DP;  // TMEM columns of one accumulator
    const uint32_t ncols = 2 * NW <= 32 ? 32 : 2 * NW <= 64 ? 64 : 2 * NW <= 128 ? 128 : 2 * NW <= 256 ? 256 : 512;
    if (warp == 0) tc::tmem_alloc(&tmem_base, ncols);
    if (tid == 0) {
        for (int b = 0; b < nbufA; ++b) {
            tc::mbar_init(&a_full[b], kConvWarps / CG);
            tc::mbar_init(&a_empty[b], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&d_full[b], 1);
            tc::mbar_init(&d_empty[b], kEpiWarps / 2);
        }
        tc::mbar_init(&b_full, 1);
        tc::fence_mbar_init();
        abort_flag = 0;
    }
    // constant K groups of the A buffers: a 1 in column DP (hi part), zeros elsewhere
    for (int e = tid; e < (NOB ? 0 : nbufA * NPART * 2 * kTcTile); e += kTcThreads) {
        const int row = e % kTcTile, g = (e / kTcTile) & 1, part = (e / (2 * kTcTile)) % NPART,
                  buf = e / (2 * kTcTile * NPART);
        const uint32_t one = KIND == tc::kTF32 ? 0x3F800000u : 0x3F80u;
        const uint32_t first = (g == 0 && part == 0) ? one : 0u;
        *reinterpret_cast<uint4 *>(s_a + (size_t)(buf * NPART + part) * A_PART + (size_t)(KG + g) * LBO_A +
                                   row * 16) = make_uint4(first, 0u, 0u, 0u);
    }
    tc::fence_proxy_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = tc::uniform(tmem_base);

    const int my_tiles = (p.ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    auto tile_of = [&](int it) -> int64_t { return (int64_t)blockIdx.x + (int64_t)it * gridDim.x; };
    // bounded wait that gives up at once after any role has timed out
    auto wait = [&](uint64_t *bar, uint32_t parity) -> bool {
        if (abort_flag) return false;
        if (tc::mbar_wait(bar, parity)) return true;
        atomicExch(p.error, 1);
        abort_flag = 1;
        return false;
    };

    if (warp == 0) {
        // ================= issuer: component operands and MMAs =================
        // the operands are one contiguous block in the workspace, laid out as
        // in shared memory: one bulk copy
        if (lane == 0 && my_tiles > 0) {
            tc::mbar_arrive_expect_tx(&b_full, CHUNK_BYTES);
            tc::bulk_copy_g2s(s_b, p.ops, CHUNK_BYTES, &b_full);
        }
        __syncwarp();
        for (int it = 0; it < my_tiles; ++it) {
            const int abuf = it % nbufA;
            {
                bool ok = wait(&a_full[abuf], (uint32_t)((it / nbufA) & 1));
                if (it == 0 && !wait(&b_full, 0u)) ok = false;
                if (it >= 2 && !wait(&d_empty[it & 1], (uint32_t)(((it - 2) >> 1) & 1))) ok = false;
                ok = __all_sync(0xffffffffu, ok);
                tc::fence_after_sync();
                if (ok) {
                    const uint32_t d_tmem = tbase + (uint32_t)((it & 1) * NW);
                    const uint32_t idesc = tc::instr_desc(KIND, kTcTile, chunk * DP);
                    const uint32_t a0 = tc::smem_u32(s_a + (size_t)abuf * NPART * A_PART);
                    const uint32_t b0 = tc::smem_u32(s_b);
#pragma unroll
                    for (int s = 0; s < KSTEPS; ++s) {
                        const uint64_t da = tc::smem_desc(a0 + s * 2 * LBO_A, LBO_A, 128);
                        const uint64_t db = tc::smem_desc(b0 + s * 2 * LBO_B, LBO_B, 128);
                        if (KIND == tc::kTF32) {
                            tc::mma_tf32_elect(d_tmem, da, db, idesc, s > 0);
                        } else {
                            tc::mma_elect(d_tmem, da, db, idesc, s > 0);
                            if (SPLIT == 3) {
                                const uint64_t dal = tc::smem_desc(a0 + A_PART + s * 2 * LBO_A, LBO_A, 128);
                                const uint64_t dbl = tc::smem_desc(b0 + chunk * B_COMP + s * 2 * LBO_B, LBO_B, 128);
                                tc::mma_elect(d_tmem, dal, db, idesc, true);
                                tc::mma_elect(d_tmem, da, dbl, idesc, true);
                            }
                        }
                    }
                }
                // commits arrive when every earlier MMA has completed, issued or not
                tc::commit_elect(&d_full[it & 1]);
                tc::commit_elect(&a_empty[abuf]);
            }
            __syncwarp();
        }
        // the copy has landed before the CTA exits, whatever timed out
        if (lane == 0 && my_tiles > 0) tc::mbar_wait(&b_full, 0u);
    } else if (warp < kFirstEpiWarp) {
        // ================= converters: sample tiles -> A operand =================
        // Groups of warps take alternate tiles. A warp converts RL rows x GL groups
        // of 8 coordinates per pass, so a request's lanes read whole 32-byte sectors
        // and eight lanes of a group store 128 contiguous operand bytes; the next
        // tile of the group is requested as soon as this one's registers are free
        constexpr int NG = DP / 8, GL = NG < 4 ? NG : 4, RL = 32 / GL, GP = NG / GL;
        constexpr int WG = kConvWarps / CG, RW = kTcTile / WG, RP = RW / RL;  // warps of a group, rows of a warp
        const int cw = (warp - 1) % WG, cgroup = (warp - 1) / WG, rl = lane % RL, gl = lane / RL;
        const int access = row_access(p.x, p.d);
        float cc[GP][8], v[RP][GP][8];
#pragma unroll
        for (int gp = 0; gp < GP; ++gp)
#pragma unroll
            for (int m = 0; m < 8; ++m) cc[gp][m] = p.center[(gp * GL + gl) * 8 + m];  // zero beyond d
        auto load = [&](int it) {
#pragma unroll
            for (int rp = 0; rp < RP; ++rp) {
                const int64_t i = tile_of(it) * kTcTile + RW * cw + rp * RL + rl;
#pragma unroll
                for (int gp = 0; gp < GP; ++gp)
                    load_group(v[rp][gp], p.x, i, it < my_tiles && i < p.n, p.d, (gp * GL + gl) * 8, access);
            }
        };
        load(cgroup);
        for (int it = cgroup; it < my_tiles; it += CG) {
            const int abuf = it % nbufA;
            const bool ok =
                it < nbufA || __all_sync(0xffffffffu, wait(&a_empty[abuf], (uint32_t)(((it - nbufA) / nbufA) & 1)));
            if (ok) {
                unsigned char *a = s_a + (size_t)abuf * NPART * A_PART;
#pragma unroll
                for (int rp = 0; rp < RP; ++rp) {
                    const int row = RW * cw + rp * RL + rl;
#pragma unroll
                    for (int gp = 0; gp < GP; ++gp) {
                        float z[8];
#pragma unroll
                        for (int m = 0; m < 8; ++m) z[m] = v[rp][gp][m] - cc[gp][m];
#pragma unroll
                        for (int h = 0; h < 8 / PER; ++h) {
                            const int q = (gp * GL + gl) * (8 / PER) + h;
                            const uint4 hi = pack_hi<KIND>(z + h * PER);
                            *reinterpret_cast<uint4 *>(a + (size_t)q * LBO_A + row * 16) = hi;
                            if (NPART == 2)
                                *reinterpret_cast<uint4 *>(a + A_PART + (size_t)q * LBO_A + row * 16) =
                                    pack_lo(z + h * PER, hi);
                        }
                    }
                }
            }
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&a_full[abuf]);
            load(it + CG);
        }
    } else {
        // ================= epilogue: radial densities and the log-sum-exp =================
        const int qd = warp & 3, group = (warp - kFirstEpiWarp) >> 2;
        const int erow = 32 * qd + lane;
        const int ggen = (p.den_kind == ISSM_DENOM_PARTIAL) ? p.group[p.fixed_slot] : 0;
        for (int it = group; it < my_tiles; it += 2) {  // accumulator `group`
            LseState<float> lse;
            float gen_lq = 0.f, last_lq = 0.f, prev_ln = 0.f;
            const int64_t i = tile_of(it) * kTcTile + erow;
            if (p.mode == 1) prev_ln = i < p.n ? p.lognum[i] : 0.f;
            const bool ok = __all_sync(0xffffffffu, wait(&d_full[it & 1], (uint32_t)((it >> 1) & 1)));
            tc::fence_after_sync();
            if (ok) {
                const uint32_t lane_base = tbase + ((uint32_t)(32 * qd) << 16) + (uint32_t)((it & 1) * NW);
                for (int kk = 0; kk < chunk; ++kk) {
                    // a component's DP columns in one round trip (all loads, then one wait)
                    float v[DP];
                    if constexpr (DP == 64) tc::tmem_ld64(lane_base + (uint32_t)(kk * DP), v);
                    else if constexpr (DP == 32) tc::tmem_ld32(lane_base + (uint32_t)(kk * DP), v);
                    else tc::tmem_ld16(lane_base + (uint32_t)(kk * DP), v);
                    float r2a = 0.f, r2b = 0.f;
#pragma unroll
                    for (int q = 0; q < DP; q += 2) {
                        r2a = fmaf(v[q], v[q], r2a);
                        r2b = fmaf(v[q + 1], v[q + 1], r2b);
                    }
                    const float r2 = r2a + r2b;
                    const int k = p.first_slot + kk;
                    float lq;
                    if (p.family == ISSM_GAUSSIAN) {
                        lq = p.lognorm[k] - 0.5f * r2;
                    } else {
                        const float nu = p.dofs[k];
                        lq = p.lognorm[k] - (nu + (float)p.d) * 0.5f * log1pf(r2 / nu);
                    }
                    bool member = true;
                    if (p.den_kind == ISSM_DENOM_GENERATING) member = (k == p.fixed_slot);
                    else if (p.den_kind == ISSM_DENOM_PARTIAL) member = (p.group[k] == ggen);
                    if (k == p.fixed_slot) gen_lq = lq;
                    last_lq = lq;
                    if (member) lse.add((p.coef ? p.coef[k] : 0.f) + lq);
                }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&d_empty[it & 1]);
            if (ok && i < p.n) {
                if (p.mode == 1) {
                    uint16_t reason = isnan(last_lq) ? ISSM_REASON_PROPOSAL_INVALID : 0;
                    if (!reason) {
                        const float v = logaddexp(prev_ln, p.coef[p.first_slot] + last_lq);
                        if (isnan(v) || v == -INFINITY) reason = ISSM_REASON_PROPOSAL_INVALID;
                        else p.lognum[i] = v;
                    }
                    if (reason) record_failure(p.failures, p.index_base + i + 1, 0, reason);
                } else {
                    float den = lse.value();
                    const bool bad = isnan(gen_lq) || gen_lq == -INFINITY || isnan(den) || den == -INFINITY;
                    if (bad) {
                        record_failure(p.failures, p.index_base + i + 1, 0, ISSM_REASON_PROPOSAL_INVALID);
                        den = -INFINITY;
                    }
                    p.out_logden[i] = den;
                    if (p.out_generating) p.out_generating[i] = bad ? -INFINITY : gen_lq;
                }
            }
        }
    }
    // ---- every role is done; in-flight MMAs have completed before TMEM is freed ----
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0 && abort_flag && my_tiles > 0)
        tc::mbar_wait(&d_full[(my_tiles - 1) & 1], (uint32_t)(((my_tiles - 1) >> 1) & 1));
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tbase, ncols);
}

// W_k = L_k^-1 (FP32) for slots first..first+count-1, written DP x DP
// row-major (row j = W_k[j, :]) with zero padding; one CTA of 256 per slot.
template <typename T>
__global__ void __launch_bounds__(256) invert_factors_kernel(const T *__restrict__ L, int d, int DP, int first,
                                                             float *__restrict__ w) {
    constexpr int LD = 65;
    __shared__ float Ls[64 * LD];
    __shared__ float Ws[64 * LD];
    const int k = first + blockIdx.x;
    const T *Lk = L + (size_t)k * d * d;
    // column-major source: element (r, c) at r + c d
    for (int e = threadIdx.x; e < d * d; e += blockDim.x) {
        const int r = e % d, c = e / d;
        Ls[r * LD + c] = (float)Lk[e];
    }
    __syncthreads();
    invert_lower_f32(Ls, Ws, d, LD);
    float *wk = w + (size_t)k * DP * DP;
    for (int e = threadIdx.x; e < DP * DP; e += blockDim.x) {
        const int j = e / DP, c = e % DP;
        wk[e] = (j < d && c < d) ? Ws[j * LD + c] : 0.f;
    }
}

int invert_factors(const issm_bank *bk, int first, int count, float *out, cudaStream_t stream) {
    const int d = bk->dim;
    if (d > 64) return ISSM_E_UNSUPPORTED;
    const int DP = d <= 16 ? 16 : d <= 32 ? 32 : 64;
    if (count <= 0) return 0;
    if (bk->dtype == ISSM_F32) {
        { invert_factors_kernel<float><<<count, 256, 0, stream>>>((const float *)bk->scales, d, DP, first, out);
          note_launch(); }
    } else {
        { invert_factors_kernel<double><<<count, 256, 0, stream>>>((const double *)bk->scales, d, DP, first, out);
          note_launch(); }
    }
    return (int)cudaGetLastError();
}

// Workspace: operand forms (K + 256/DP - 1) x DP * (4 DP + 64) bytes (room
// for the last, partial chunk) | centre (256 bytes) | inverse factors
// K x DP * DP floats (only when the bank has none).
static int dp_of(int d) { return d <= 16 ? 16 : d <= 32 ? 32 : 64; }
static size_t ops_slot_bytes(int DP) { return (size_t)DP * (4 * DP + 64); }
static size_t ops_bytes(int k, int DP) { return (size_t)(k + 256 / DP - 1) * ops_slot_bytes(DP); }

size_t tc_workspace_bytes(int k, int d) {
    const int DP = dp_of(d);
    return ops_bytes(k, DP) + 256 + (size_t)k * DP * DP * 4 + 64;
}

template <int KIND, int SPLIT, int DP>
static int launch_tc(TcParams p, const float *w, const float *loc, int cslot, unsigned char *ops, float *center,
                     cudaStream_t stream) {
    constexpr int EB = KIND == tc::kBF16 ? 2 : 4;
    constexpr int KGX = DP * EB / 16 + 2;
    constexpr int NPART = SPLIT == 3 ? 2 : 1;
    constexpr size_t A_PART = (size_t)kTcTile * KGX * 16;
    constexpr size_t A_PART_NOB = (size_t)kTcTile * (KGX - 2) * 16;
    constexpr size_t B_COMP = (size_t)DP * KGX * 16;
    static_assert(NPART * B_COMP <= (size_t)DP * (4 * DP + 64), "operand form exceeds its workspace slot");
    const int nslots = p.last_slot - p.first_slot + 1;
    // one component centred at its own location: no offset column
    const bool nob = nslots == 1 && cslot == p.first_slot;
    p.nslots = nslots;
    // the A buffers and every component's operands; more components than an
    // accumulator's 256 columns hold go to the paired tiles
    const size_t smem = (size_t)tc_abufs(DP) * NPART * (nob ? A_PART_NOB : A_PART) + (size_t)NPART * nslots * B_COMP;
    static_assert((size_t)tc_abufs(DP) * NPART * A_PART + (size_t)NPART * (256 / DP) * B_COMP <= kTcMaxSmem,
                  "shared memory per CTA");
    if (nslots * DP > 256) return launch_pair(KIND, DP, p, w, loc, cslot, ops, center, stream);
    { tc_prepare_kernel<KIND, SPLIT, DP><<<nslots, 256, 0, stream>>>(w, loc, p.d, p.first_slot, nslots, cslot, ops,
                                                                       center);
      note_launch(); }
    auto kern = nob ? mixture_tc_kernel<KIND, SPLIT, DP, true> : mixture_tc_kernel<KIND, SPLIT, DP, false>;
    const int st = allow_dynamic_smem((const void *)kern);
    if (st) return st;
    int occ = 1;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kTcThreads, smem);
    if (e != cudaSuccess) return (int)e;
    const int nw2 = 2 * nslots * DP;
    const int ncols = nw2 <= 32 ? 32 : nw2 <= 64 ? 64 : nw2 <= 128 ? 128 : nw2 <= 256 ? 256 : 512;
    occ = max(1, min(occ, 512 / ncols));  // TMEM allocations never wait
    p.ntiles = (int)((p.n + kTcTile - 1) / kTcTile);
    const int blocks = min(p.ntiles, device_sms() * occ);
    if (blocks < 1) return 0;
    { kern<<<blocks, kTcThreads, smem, stream>>>(p); note_launch(); }
    return (int)cudaGetLastError();
}

// precision: ISSM_PREC_TF32 or ISSM_PREC_BF16 (split x3)
int tc_mixture(const issm_bank *bk, const issm_denominator *den, int mode, int first, int last,
               const void *x, int64_t n, const int32_t *slots, int fixed_slot, const void *coef,
               void *out_logden, void *out_generating, void *lognum, uint64_t *failures, int64_t index_base,
               int precision, void *ws, size_t ws_bytes, int *error, cudaStream_t stream) {
    const int d = bk->dim;
    if (bk->dtype != ISSM_F32 || bk->scale_kind != ISSM_SCALE_FACTOR || d > 64) return ISSM_E_UNSUPPORTED;
    if (slots != nullptr) return ISSM_E_UNSUPPORTED;  // one centre per launch
    const int DP = dp_of(d);
    const int K = bk->count;
    if (ws_bytes < tc_workspace_bytes(K, d)) return ISSM_E_WORKSPACE;
    unsigned char *ops = (unsigned char *)ws;
    float *center = (float *)(ops + ops_bytes(K, DP));
    float *winv = (float *)((unsigned char *)center + 256);
    const int den_kind = den ? den->kind : ISSM_DENOM_FULL;
    // only the generating slot contributes to a generating-only denominator
    if (mode == 0 && den_kind == ISSM_DENOM_GENERATING) first = last = fixed_slot;
    const float *w = bk->inverse_factors;
    if (!w) {
        const int st = invert_factors(bk, first, last - first + 1, winv, stream);
        if (st) return st;
        w = winv;
    }
    const int cslot = (mode == 1) ? first : fixed_slot;
    TcParams p{};
    p.d = d; p.mode = mode; p.family = bk->family; p.den_kind = den_kind; p.fixed_slot = fixed_slot;
    p.first_slot = first; p.last_slot = last;
    p.n = n; p.x = (const float *)x; p.ops = ops; p.center = center;
    p.lognorm = (const float *)bk->lognormalizers; p.coef = (const float *)coef; p.dofs = (const float *)bk->dofs;
    p.group = den ? den->group_of_slot : nullptr;
    p.out_logden = (float *)out_logden; p.out_generating = (float *)out_generating;
    p.lognum = (float *)lognum; p.failures = failures; p.index_base = index_base; p.error = error;
    const float *loc = (const float *)bk->locations;
    const bool tf32 = precision == ISSM_PREC_TF32;
    if (DP == 16)
        return tf32 ? launch_tc<tc::kTF32, 1, 16>(p, w, loc, cslot, ops, center, stream)
                    : launch_tc<tc::kBF16, 3, 16>(p, w, loc, cslot, ops, center, stream);
    if (DP == 32)
        return tf32 ? launch_tc<tc::kTF32, 1, 32>(p, w, loc, cslot, ops, center, stream)
                    : launch_tc<tc::kBF16, 3, 32>(p, w, loc, cslot, ops, center, stream);
    return tf32 ? launch_tc<tc::kTF32, 1, 64>(p, w, loc, cslot, ops, center, stream)
                : launch_tc<tc::kBF16, 3, 64>(p, w, loc, cslot, ops, center, stream);
}

}  // namespace issm
