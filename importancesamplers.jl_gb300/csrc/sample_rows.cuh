// sample_rows.cuh — reading sample rows into the registers of the warps that build
// tensor-core operands from them (mixture_tc.cu, moments_tc.cu).
#pragma once

#include <cstdint>

namespace issm {

// How wide the rows of x can be read: 32, 16 or 4 bytes.
__device__ __forceinline__ int row_access(const float *x, int d) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(x);
    return d % 8 == 0 && (a & 31) == 0 ? 32 : d % 4 == 0 && (a & 15) == 0 ? 16 : 4;
}

// Coordinates c .. c + 7 (c a multiple of 8) of sample i into registers, zeros
// beyond d and for an inactive sample. One 32-byte request per lane: two 16-byte
// ones each ask for half of a lane's sector, and 256 MB read that way came at 4.35
// TB/s against 6.3 for requests of whole sectors. The samples leave L2 first: a run's
// retained rows (512 MB at 2M x 64) pass through it twice a round, and kept out what
// every round rereads, instructions included: 11.06 -> 10.53 ms of device time a run,
// the fit between the passes 47 -> 43 us, an operand preparation 9.9 -> 6.5.
__device__ __forceinline__ void load_group(float (&v)[8], const float *__restrict__ x, int64_t i, bool active, int d,
                                           int c, int access) {
    const float *src = x + i * d + c;
#pragma unroll
    for (int m = 0; m < 8; ++m) v[m] = 0.f;
    if (access == 32) {
        if (active && c < d)
            asm volatile("ld.global.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
                           "=f"(v[7])
                         : "l"(src));
    } else if (access == 16) {
#pragma unroll
        for (int h = 0; h < 8; h += 4)
            if (active && c + h < d) {
                const float4 f = *reinterpret_cast<const float4 *>(src + h);
                v[h] = f.x;
                v[h + 1] = f.y;
                v[h + 2] = f.z;
                v[h + 3] = f.w;
            }
    } else {
#pragma unroll
        for (int m = 0; m < 8; ++m)
            if (active && c + m < d) v[m] = src[m];
    }
}

}  // namespace issm
