// mixture_simt.cu — FP32 instantiation of the SIMT kernels and the host entry
// points of both types (mixture_simt.cuh).
#include "mixture_simt.cuh"

namespace issm {

template int dispatch_simt<float>(const MixParams<float> &, cudaStream_t);
extern template int dispatch_simt<double>(const MixParams<double> &, cudaStream_t);  // mixture_simt_f64.cu

template <typename T>
static MixParams<T> params_from(const issm_bank *b, const issm_denominator *den) {
    MixParams<T> p{};
    p.d = b->dim;
    p.k = b->count;
    p.family = b->family;
    p.scale_kind = b->scale_kind;
    p.loc = (const T *)b->locations;
    p.scales = (const T *)b->scales;
    p.lognorm = (const T *)b->lognormalizers;
    p.dofs = (const T *)b->dofs;
    p.range_risk = b->range_risk;
    p.first_slot = 0;
    p.last_slot = b->count - 1;
    if (den) {
        p.den_kind = den->kind;
        p.terms = den->terms;
        p.coef = (const T *)den->logcoefficients;
        p.group = den->group_of_slot;
        if (den->kind == ISSM_DENOM_PREFIX) p.last_slot = den->terms - 1;
    } else {
        p.den_kind = ISSM_DENOM_GENERATING;
    }
    return p;
}

int simt_mixture(const issm_bank *b, const issm_denominator *den, const void *x, int64_t n,
                 const int32_t *slots, int32_t fixed_slot, void *out_logden, void *out_generating,
                 uint64_t *failures, int64_t index_base, cudaStream_t stream) {
    if (b->dtype == ISSM_F32) {
        auto p = params_from<float>(b, den);
        p.n = n; p.x = (const float *)x; p.slots = slots; p.fixed_slot = fixed_slot;
        p.out_logden = (float *)out_logden; p.out_generating = (float *)out_generating;
        p.failures = failures; p.index_base = index_base; p.mode = kModeDenominator;
        return dispatch_simt(p, stream);
    }
    auto p = params_from<double>(b, den);
    p.n = n; p.x = (const double *)x; p.slots = slots; p.fixed_slot = fixed_slot;
    p.out_logden = (double *)out_logden; p.out_generating = (double *)out_generating;
    p.failures = failures; p.index_base = index_base; p.mode = kModeDenominator;
    return dispatch_simt(p, stream);
}

template <typename T>
static int simt_round_t(const issm_bank *b, const issm_denominator *den, const int32_t *slots, int fixed_slot,
                        const void *normals, const void *rn, int rn_stride, const void *ru, int ru_stride,
                        const void *logtargets, int64_t n, void *samples, void *logweights,
                        const int64_t *proposal_ids, int64_t *proposal_ids_out, uint64_t *failures,
                        int64_t index_base, int mode, cudaStream_t stream) {
    auto p = params_from<T>(b, den);
    p.n = n; p.slots = slots; p.fixed_slot = fixed_slot;
    p.normals = (const T *)normals; p.rnormals = (const T *)rn; p.rn_stride = rn_stride;
    p.runiforms = (const T *)ru; p.ru_stride = ru_stride;
    p.logtargets = (const T *)logtargets; p.samples_out = (T *)samples; p.logweights = (T *)logweights;
    p.proposal_ids = proposal_ids; p.proposal_ids_out = proposal_ids_out;
    p.failures = failures; p.index_base = index_base; p.mode = mode;
    return dispatch_simt(p, stream);
}

int simt_round(const issm_bank *b, const issm_denominator *den, const int32_t *slots, const void *normals,
               const void *rn, int rn_stride, const void *ru, int ru_stride, const void *logtargets,
               int64_t n, void *samples, void *logweights, const int64_t *proposal_ids,
               int64_t *proposal_ids_out, uint64_t *failures, cudaStream_t stream) {
    if (b->dtype == ISSM_F32)
        return simt_round_t<float>(b, den, slots, 0, normals, rn, rn_stride, ru, ru_stride, logtargets, n,
                                   samples, logweights, proposal_ids, proposal_ids_out, failures, 0,
                                   kModeRound, stream);
    return simt_round_t<double>(b, den, slots, 0, normals, rn, rn_stride, ru, ru_stride, logtargets, n,
                                samples, logweights, proposal_ids, proposal_ids_out, failures, 0,
                                kModeRound, stream);
}

int simt_draw(const issm_bank *b, const int32_t *slots, int32_t fixed_slot, const void *normals,
              const void *rn, int rn_stride, const void *ru, int ru_stride, int64_t n, void *samples,
              uint64_t *failures, int64_t index_base, cudaStream_t stream) {
    if (b->dtype == ISSM_F32)
        return simt_round_t<float>(b, nullptr, slots, fixed_slot, normals, rn, rn_stride, ru, ru_stride,
                                   nullptr, n, samples, nullptr, nullptr, nullptr, failures, index_base,
                                   kModeDraw, stream);
    return simt_round_t<double>(b, nullptr, slots, fixed_slot, normals, rn, rn_stride, ru, ru_stride,
                                nullptr, n, samples, nullptr, nullptr, nullptr, failures, index_base,
                                kModeDraw, stream);
}

template <typename T>
static int simt_draw_fused_t(const issm_bank *b, int fixed_slot, uint64_t seed, const uint64_t *counter,
                             uint64_t offset, const void *rn, int rn_stride, const void *ru, int ru_stride,
                             int64_t n, void *samples, uint64_t *failures, int64_t index_base,
                             cudaStream_t stream) {
    auto p = params_from<T>(b, nullptr);
    p.n = n; p.slots = nullptr; p.fixed_slot = fixed_slot;
    p.rnormals = (const T *)rn; p.rn_stride = rn_stride;
    p.runiforms = (const T *)ru; p.ru_stride = ru_stride;
    p.samples_out = (T *)samples;
    p.failures = failures; p.index_base = index_base; p.mode = kModeDraw;
    p.fused = 1; p.nseed = seed; p.nbase = counter; p.noffset = offset;
    return dispatch_simt(p, stream);
}

int simt_draw_fused(const issm_bank *b, int32_t fixed_slot, uint64_t seed, const uint64_t *counter,
                    uint64_t offset, const void *rn, int rn_stride, const void *ru, int ru_stride, int64_t n,
                    void *samples, uint64_t *failures, int64_t index_base, cudaStream_t stream) {
    if (b->scale_kind != ISSM_SCALE_FACTOR) return ISSM_E_UNSUPPORTED;
    if (b->dtype == ISSM_F32)
        return simt_draw_fused_t<float>(b, fixed_slot, seed, counter, offset, rn, rn_stride, ru, ru_stride, n,
                                        samples, failures, index_base, stream);
    return simt_draw_fused_t<double>(b, fixed_slot, seed, counter, offset, rn, rn_stride, ru, ru_stride, n,
                                     samples, failures, index_base, stream);
}

template <typename T>
static int simt_append_t(const issm_bank *b, int slot, const void *logcounts, const void *x, int64_t n,
                         void *lognum, uint64_t *failures, cudaStream_t stream) {
    auto p = params_from<T>(b, nullptr);
    p.den_kind = ISSM_DENOM_FULL;
    p.coef = (const T *)logcounts;
    p.first_slot = slot;
    p.last_slot = slot;
    p.n = n; p.x = (const T *)x; p.fixed_slot = slot;
    p.lognum = (T *)lognum; p.failures = failures; p.mode = kModeAppend;
    return dispatch_simt(p, stream);
}

int simt_append(const issm_bank *b, int slot, const void *logcounts, const void *x, int64_t n, void *lognum,
                uint64_t *failures, cudaStream_t stream) {
    if (b->dtype == ISSM_F32) return simt_append_t<float>(b, slot, logcounts, x, n, lognum, failures, stream);
    return simt_append_t<double>(b, slot, logcounts, x, n, lognum, failures, stream);
}

}  // namespace issm
