// ldlt.cuh — blocked FP64 LDL^T of a symmetric matrix of order d <= 64 in shared
// memory, shared by the moment fit (moments.cu) and the grouped fit (group.cu).
#pragma once

#include "issm_device.cuh"

namespace issm {

// 1 / a in FP64 with few FP64 instructions: an FP32 reciprocal seed refined
// by two Newton-Raphson steps r <- r + r (1 - a r) (about 23 -> 46 -> full
// double bits; the seed is the hardware's approximate FP32 reciprocal). Each
// FP64 instruction occupies a warp's FP64 pipe for about 64 cycles on this
// GPU (and takes as long to complete), so the factorisation's
// sequential chain is built from as few of them as possible. Values outside
// the FP32 seed's range, zero, negative or non-finite values take the exact
// division (and give its NaN / Inf).
__device__ __forceinline__ double rcp_nr(double a) {
    const float af = (float)a;
    if (!(af > 1e-30f && af < 1e30f)) return 1.0 / a;
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(af));  // one MUFU op; Newton makes up the bits
    double r = (double)rf;
    double e = fma(-a, r, 1.0);
    r = fma(r, e, r);
    e = fma(-a, r, 1.0);
    return fma(r, e, r);
}

// The factorisation is a blocked right-looking LDL^T, A = L D L^T with unit
// lower L, in 8-column panels; the Cholesky factor is L diag(sqrt(d)). Each
// FP64 instruction holds a warp's FP64 pipe for about 64 cycles on this GPU
// (and takes as long to complete), so:
//  * the sequential chain per column is only 1/d_j (an FP32 seed and two
//    Newton steps), run by warp 0 on the 8 x 8 diagonal block, which it
//    holds in registers (one element per lane, shuffles between steps);
//  * one thread per row solves its panel row, l_ic = (a_ic - sum_q l_iq d_q
//    l_cq) / d_c;
//  * while warp 0 updates and factors the next diagonal block (lookahead),
//    warps 1-3 and 5-7 apply the rank-8 update to the rest of the trailing
//    lower triangle, each thread holding up to nine independent elements
//    (column pairs (k, m-1-k) balance the work), so the pipe, not latency,
//    bounds it; warp 4 stays out, since it would queue FP64 instructions on
//    warp 0's sub-partition ahead of the pivot chain.
// Every thread of a CTA of 256 calls it; A is d x d column-major (its lower
// triangle is used), synchronised before the call and after it. On return the
// strict lower triangle of A holds L, s_dg[c] the pivots. s_rinv: 8 doubles;
// s_w[panel & 1][c][i] = l_ic d_c of a panel.
__device__ __forceinline__ void ldlt_lower(double *A, int d, double *s_dg, double *s_rinv, double (*s_w)[8][64]) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // warp 0: LDL^T of the nb x nb diagonal block at (kb, kb), in registers.
    // Lane e < 28 holds the strictly-lower element (ei, ec) of the block
    // (row-major lower order, e = ei (ei - 1) / 2 + ec) and lanes 0..nb-1 the
    // diagonal; a column step is a pivot broadcast, the reciprocal chain, one
    // scaling and one update per held element, with the operands exchanged by
    // warp shuffles, so the chain holds no shared-memory round trip
    auto factor_diag = [&](int kb, int nb, double (*w)[64]) {  // warp 0
        int ei = 1, ec = 0;
        {
            int t = lane;
            while (ei < 8 && t >= ei) {
                t -= ei;
                ++ei;
            }
            ec = t;
        }
        const bool hasl = lane < 28 && ei < nb;
        const bool hasd = lane < nb;
        double vl = hasl ? A[(kb + ei) + (kb + ec) * d] : 0.0;
        double vd = hasd ? A[(kb + lane) + (kb + lane) * d] : 0.0;
        double ul = 0.0;  // u = l d of this lane's lower element, once its column is done
        const int lane_d = lane * (lane - 1) / 2;  // lanes of row `lane`'s lower elements start here
        for (int j = 0; j < nb; ++j) {
            const double dj = __shfl_sync(0xffffffffu, vd, j);
            const double rj = rcp_nr(dj);
            if (lane == 0) {
                s_dg[kb + j] = dj;
                s_rinv[j] = rj;
            }
            // column j: element (ei, j) becomes l = u / d_j
            if (hasl && ec == j) {
                ul = vl;
                vl = vl * rj;
                w[j][kb + ei] = ul;
            }
            // (ei, ec), ec > j: -= l(ei, j) u(ec, j); diagonal (c, c), c > j: -= l(c, j) u(c, j)
            const double l_i = __shfl_sync(0xffffffffu, vl, (ei * (ei - 1) / 2 + j) & 31);
            const double u_c = __shfl_sync(0xffffffffu, ul, (ec * (ec - 1) / 2 + j) & 31);
            const double l_d = __shfl_sync(0xffffffffu, vl, (lane_d + j) & 31);
            const double u_d = __shfl_sync(0xffffffffu, ul, (lane_d + j) & 31);
            if (hasl && ec > j) vl = fma(-l_i, u_c, vl);
            if (hasd && lane > j) vd = fma(-l_d, u_d, vd);
        }
        if (hasl) A[(kb + ei) + (kb + ec) * d] = vl;
        if (hasd) A[(kb + lane) + (kb + lane) * d] = vd;  // the pivot d_lane
        __syncwarp();
    };
    if (warp == 0) factor_diag(0, min(8, d), s_w[0]);
    __syncthreads();
    for (int kb = 0; kb < d; kb += 8) {
        const int nb = min(8, d - kb), base = kb + nb, m = d - base;
        if (m <= 0) break;
        double (*wc)[64] = s_w[(kb >> 3) & 1];
        double (*wn)[64] = s_w[((kb >> 3) + 1) & 1];
        // panel: one thread per row i below the diagonal block
        for (int r = tid; r < m; r += 256) {
            const int i = base + r;
            double w[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                if (c < nb) {
                    double v = A[i + (kb + c) * d];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q < c) v = fma(-w[q], A[(kb + c) + (kb + q) * d], v);
                    w[c] = v;                            // l_ic d_c
                    A[i + (kb + c) * d] = v * s_rinv[c];  // l_ic
                    wc[c][i] = v;
                } else {
                    w[c] = 0.0;
                }
            }
        }
        __syncthreads();
        const int nbn = min(8, m);
        if (warp == 0) {
            // lookahead: the next diagonal block gets its rank-nb update first, then is factored
            for (int e = lane; e < nbn * (nbn + 1) / 2; e += 32) {
                int c = 0, t = e;
                while (t >= nbn - c) {
                    t -= nbn - c;
                    ++c;
                }
                const int i = c + t;
                double acc = A[(base + i) + (base + c) * d];
                for (int q = 0; q < nb; ++q) acc = fma(-A[(base + i) + (kb + q) * d], wc[q][base + c], acc);
                A[(base + i) + (base + c) * d] = acc;
            }
            __syncwarp();
            factor_diag(base, nbn, wn);
        } else if (warp != 4) {
            // rank-nb update of the trailing lower triangle outside the next
            // diagonal block, by warps 1-3 and 5-7: warp 4 shares warp 0's
            // sub-partition (warp id mod 4) and so its FP64 pipe, which the
            // pivot chain needs free
            const int wt = (warp < 4 ? warp - 1 : warp - 2) * 32 + lane, half = (m + 1) >> 1,
                      total = half * (m + 1);
            constexpr int kT = 9;  // elements per thread: 192 x 9 >= 28 x 57, the largest trailing triangle
            int ei[kT], ek[kT];
#pragma unroll
            for (int t = 0; t < kT; ++t) {
                ei[t] = -1;
                ek[t] = 0;
                const int e = wt + t * 192;
                if (e < total) {
                    const int c = e / (m + 1), r = e - c * (m + 1);
                    int i = -1, k = 0;
                    if (r < m - c) {
                        k = c;
                        i = c + r;
                    } else {
                        const int k2 = m - 1 - c;
                        if (k2 != c) {
                            k = k2;
                            i = k2 + (r - (m - c));
                        }
                    }
                    if (i >= 0 && !(i < nbn && k < nbn)) {
                        ei[t] = i;
                        ek[t] = k;
                    }
                }
            }
            double acc[kT];
#pragma unroll
            for (int t = 0; t < kT; ++t) acc[t] = ei[t] >= 0 ? A[(base + ei[t]) + (base + ek[t]) * d] : 0.0;
            for (int c = 0; c < nb; ++c) {
#pragma unroll
                for (int t = 0; t < kT; ++t)
                    if (ei[t] >= 0) acc[t] = fma(-A[(base + ei[t]) + (kb + c) * d], wc[c][base + ek[t]], acc[t]);
            }
#pragma unroll
            for (int t = 0; t < kT; ++t)
                if (ei[t] >= 0) A[(base + ei[t]) + (base + ek[t]) * d] = acc[t];
        }
        __syncthreads();
    }
}

}  // namespace issm
