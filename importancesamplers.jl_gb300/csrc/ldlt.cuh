// ldlt.cuh — blocked FP64 LDL^T of a symmetric matrix of order d <= 64 in shared
// memory, shared by the moment fit (moments.cu) and the grouped fit (group.cu).
#pragma once

#include "issm_device.cuh"

namespace issm {

// r0 and t with 1 / a = r0 (1 + t) in full double precision: an approximate FP32
// reciprocal r0 (e = 1 - a r0, |e| < 2^-21) and t = e + e^2 (the next term of the
// geometric series is below 2^-64). x / a is then fma(x r0, t, x r0), x r0 off the
// critical chain. The conversions are integer operations on the exponent and the
// leading mantissa bits, not FP64 instructions. Values outside the seed's range,
// zero, negative or non-finite values take the exact division (and give its NaN /
// Inf).
__device__ __forceinline__ void reciprocal(double a, double &r0, double &t) {
    const uint32_t hi = (uint32_t)__double2hiint(a), lo = (uint32_t)__double2loint(a);
    const uint32_t ex = hi >> 20;  // sign and exponent
    if (ex - (1023u - 100u) <= 200u) {
        const float af = __uint_as_float(((ex - 1023u + 127u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
        float rf;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(af));  // one MUFU op; the series makes up the bits
        const uint32_t rb = __float_as_uint(rf);
        r0 = __hiloint2double((int)((((rb >> 23) + 1023u - 127u) << 20) | ((rb >> 3) & 0xfffffu)), (int)(rb << 29));
        const double e = fma(-a, r0, 1.0);
        t = fma(e, e, e);
    } else {
        r0 = 1.0 / a;
        t = 0.0;
    }
}

// The factorisation is a blocked right-looking LDL^T, A = L D L^T with unit
// lower L, in 8-column panels; the Cholesky factor is L diag(sqrt(d)). An FP64
// instruction holds its sub-partition's pipe for 64 cycles on this GPU and takes
// as long to complete, so the work is counted in instructions per sub-partition
// (warp id mod 4):
//  * warp 0 alone holds the pivot chain: the 8 x 8 diagonal block in registers,
//    one element per lane (the first column in a register of its own, the other 28
//    in lanes 0..27), five FP64 instructions per column (e, t, x r0, l, update);
//    lane 31 carries x = 1, so its l is the pivot's reciprocal. Warp 4, which
//    shares its pipe, stays out;
//  * one thread per row below (warps 1, 2) follows it column by column through
//    named barriers: l_ij = w_ij / d_j, then w_ic -= w_ij l_cj for the block's
//    later columns, so the panel is solved when its diagonal block is;
//  * between panels the rank-8 update is split by who waits for it: the next
//    diagonal block (warp 0, straight into its registers), the rows below it
//    (warps 1-3, 5-7, before the rows are solved), and the rest of the trailing
//    triangle (strips of 64 elements that the warps take from a counter while
//    the next panel is factored).
// d = 64: 60,400 cycles, d = 33 27,100, d = 8 5,200; with the panel solved after
// its diagonal block, an FP64 Newton reciprocal per column and static shares of the
// trailing update 98,400, 51,800 and 7,100. The chain (about 560 cycles per column)
// bounds all but the first panels, where the trailing update does.
// Every thread of a CTA of 256 calls it; A is d x d column-major (its lower
// triangle is used), synchronised before the call and after it. On return the
// strict lower triangle of A holds L, s_dg[c] the pivots. s_rinv: 8 doubles;
// s_w[panel & 1][c][i] = l_ic d_c of a panel. Named barriers 1..9 are used.
__device__ __forceinline__ void ldlt_lower(double *A, int d, double *s_dg, double *s_rinv, double (*s_w)[8][64]) {
    __shared__ int s_next[2];  // next strip of the trailing update, by panel parity
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < 2) s_next[tid] = 0;
    // lane -> element (ei, ec), 1 <= ec <= ei <= 7, of a diagonal block
    int ei = 1, ec = lane + 1;
    while (ei < 7 && ec > ei) {
        ec -= ei;
        ++ei;
    }
    if (lane >= 28) ei = ec = 1;
    __syncthreads();
    for (int kb = 0; kb < d; kb += 8) {
        const int nb = min(8, d - kb), base = kb + nb, m = d - base, par = (kb >> 3) & 1;
        const int solvers = m > 32 ? 2 : m > 0 ? 1 : 0;  // warps of rows below the block
        const bool update = kb > 0;                      // the previous panel's rank-8 update is due
        const int pb = kb - 8;
        double (*wn)[64] = s_w[par], (*wp)[64] = s_w[par ^ 1];
        if (warp == 0) {
            // the block's elements, after the previous panel's update
            const int r0i = kb + min(lane, nb - 1), ri = kb + min(ei, nb - 1), rc = kb + min(ec, nb - 1);
            double v0 = A[r0i + kb * d], v = A[ri + rc * d];
            if (update) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    v0 = fma(-A[r0i + (pb + q) * d], wp[q][kb], v0);
                    v = fma(-A[ri + (pb + q) * d], wp[q][rc], v);
                }
            }
            if (lane == 31) v0 = v = 1.0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j >= nb) break;
                const double x = j == 0 ? v0 : v;
                const double dj = __shfl_sync(0xffffffffu, x, j == 0 ? 0 : j * (j - 1) / 2 + j - 1);
                // rows ei and ec of column j
                const int si = j == 0 ? ei : (ei * (ei - 1) / 2 + j - 1) & 31;
                const int sc = j == 0 ? ec : (ec * (ec - 1) / 2 + j - 1) & 31;
                const double u_c = __shfl_sync(0xffffffffu, x, sc);
                double r0, t;
                reciprocal(dj, r0, t);
                const double xr = x * r0, l = fma(xr, t, xr);
                const int row = j == 0 ? lane : ei;
                if (j == 0 ? (lane > 0 && lane < nb) : (lane < 28 && ec == j && ei > j && ei < nb)) {
                    A[(kb + row) + (kb + j) * d] = l;
                    wn[j][kb + row] = x;
                }
                if (lane == 31) {
                    s_dg[kb + j] = dj;
                    s_rinv[j] = l;
                }
                if (solvers) asm volatile("bar.arrive %0, %1;" ::"r"(2 + j), "r"(32 + 32 * solvers) : "memory");
                if (j < 7) {
                    const double l_i = __shfl_sync(0xffffffffu, l, si);
                    const double vn = fma(-l_i, u_c, v);
                    if (lane < 28 && ec > j) v = vn;
                }
            }
        } else if (warp != 4) {
            const int w6 = warp < 4 ? warp - 1 : warp - 2;  // 0..5
            if (update && m > 0) {
                // the panel's rows below its block
                const int total = m * nb;
                for (int e = w6 * 32 + lane; e < total; e += 192) {
                    const int c = e / m, r = base + e - c * m;
                    double acc = A[r + (kb + c) * d];
#pragma unroll
                    for (int q = 0; q < 8; ++q) acc = fma(-A[r + (pb + q) * d], wp[q][kb + c], acc);
                    A[r + (kb + c) * d] = acc;
                }
                asm volatile("bar.sync 1, 192;" ::: "memory");
            }
            if (warp <= solvers) {
                const int r = (warp - 1) * 32 + lane, i = base + min(r, m - 1);
                const bool mine = r < m;
                double w[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) w[c] = A[i + (kb + c) * d];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    asm volatile("bar.sync %0, %1;" ::"r"(2 + j), "r"(32 + 32 * solvers) : "memory");
#pragma unroll
                    for (int c = j + 1; c < 8; ++c) w[c] = fma(-w[j], A[(kb + c) + (kb + j) * d], w[c]);
                    const double l = w[j] * s_rinv[j];
                    if (mine) {
                        A[i + (kb + j) * d] = l;
                        wn[j][i] = w[j];
                    }
                }
            }
            if (update && m > 0) {
                // the rest of the trailing triangle: columns from base on, strips of
                // 64 entries of the pairing (column c, column m - 1 - c)
                const int half = (m + 1) >> 1, total = half * (m + 1);
                for (;;) {
                    int e0 = 0;
                    if (lane == 0) e0 = atomicAdd(&s_next[par], 64);
                    e0 = __shfl_sync(0xffffffffu, e0, 0);
                    if (e0 >= total) break;
                    int pi[2], pk[2];
                    double acc[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int e = e0 + 32 * u + lane, c = e / (m + 1), r = e - c * (m + 1);
                        pi[u] = -1;
                        pk[u] = 0;
                        if (e < total) {
                            if (r < m - c) {
                                pk[u] = c;
                                pi[u] = c + r;
                            } else if (m - 1 - c != c) {
                                pk[u] = m - 1 - c;
                                pi[u] = m - 1 - c + r - (m - c);
                            }
                        }
                        acc[u] = pi[u] >= 0 ? A[(base + pi[u]) + (base + pk[u]) * d] : 0.0;
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q)
#pragma unroll
                        for (int u = 0; u < 2; ++u)
                            acc[u] = fma(-A[(base + max(pi[u], 0)) + (pb + q) * d], wp[q][base + pk[u]], acc[u]);
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (pi[u] >= 0) A[(base + pi[u]) + (base + pk[u]) * d] = acc[u];
                }
            }
        }
        __syncthreads();
        if (tid == 0) s_next[par] = 0;  // used again two panels on
    }
}

}  // namespace issm
