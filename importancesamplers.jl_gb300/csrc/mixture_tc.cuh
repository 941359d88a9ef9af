// mixture_tc.cuh — what the tensor-core mixture kernels share: operand packing
// and launch parameters (mixture_tc.cu: components that fit one accumulator;
// mixture_pair.cu: more).
#pragma once

#include "issm_device.cuh"
#include "issm_internal.h"
#include "sample_rows.cuh"
#include "tcgen05.cuh"

namespace issm {

constexpr int kTcTile = 128;
constexpr size_t kTcMaxSmem = 232448 - 1024;  // dynamic shared memory per CTA, static part reserved

// 16 bytes of operand values from v[PER]: 4 tf32 (nearest even), or 8 bf16
// (the hi part; pack_lo gives the lo part bf16(v - hi)).
template <int KIND> __device__ __forceinline__ uint4 pack_hi(const float *v) {
    if (KIND == tc::kTF32) return make_uint4(tc::tf32_rn(v[0]), tc::tf32_rn(v[1]), tc::tf32_rn(v[2]), tc::tf32_rn(v[3]));
    return make_uint4(tc::pack_bf16x2(v[0], v[1]), tc::pack_bf16x2(v[2], v[3]), tc::pack_bf16x2(v[4], v[5]),
                      tc::pack_bf16x2(v[6], v[7]));
}
__device__ __forceinline__ uint32_t lo_pair(float a, float b, uint32_t hi) {
    return tc::pack_bf16x2(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
}
__device__ __forceinline__ uint4 pack_lo(const float *v, uint4 hi) {
    return make_uint4(lo_pair(v[0], v[1], hi.x), lo_pair(v[2], v[3], hi.y), lo_pair(v[4], v[5], hi.z),
                      lo_pair(v[6], v[7], hi.w));
}

struct TcParams {
    int d, mode, family, den_kind, fixed_slot;
    int first_slot, last_slot, nslots, ntiles;
    int64_t n;
    const float *x;
    const unsigned char *ops;
    const float *center;
    const float *lognorm, *coef, *dofs;
    const int32_t *group;
    float *out_logden, *out_generating, *lognum;
    uint64_t *failures;
    int64_t index_base;
    int *error;
};

// mixture_pair.cu. kind / split: tc::kTF32, 1 or tc::kBF16, 3; w: the slots'
// inverse factors (DP x DP); ops and center: workspace.
int launch_pair(int kind, int DP, TcParams p, const float *w, const float *loc, int cslot, unsigned char *ops,
                float *center, cudaStream_t stream);

}  // namespace issm
