// mixture_simt.cuh — SIMT (CUDA-core) kernels of the radial proposal banks in
// the bank's own precision, instantiated per type (mixture_simt.cu: FP32 and
// the host entry points, mixture_simt_f64.cu: FP64).
//
// Every (sample, component) pair runs the reference's forward substitution
// (_packed_gaussian_logdensity!, src/native_execution.jl:346-384) followed by
// the radial density (src/proposals.jl:24-70). The balance-heuristic sum is an
// online log-sum-exp (one exp per pair) instead of the reference's chained
// logaddexp (src/mis_execution.jl:30-65): same value, two fewer
// transcendentals per term, same NaN / -Inf semantics.
//
// Non-finite radii, subnormal Student-t radii and range-risk Student-t slots
// leave the fast path for `slow_component_logdensity`, a restatement of the
// reference's exponent-extended solves (src/student_t_range.jl:82-153).
#pragma once

#include "issm_device.cuh"
#include "issm_internal.h"
#include "rng.cuh"
#include "tcgen05.cuh"

namespace issm {

enum Mode { kModeDenominator = 0, kModeRound = 1, kModeAppend = 2, kModeDraw = 3 };

template <typename T> struct MixParams {
    // bank
    int d, k, family, scale_kind;
    const T *loc, *scales, *lognorm, *dofs;
    const uint8_t *range_risk;
    // denominator
    int den_kind, terms;
    const T *coef;
    const int32_t *group;
    // samples / slots
    int64_t n;
    const T *x;            // input samples (DENOM / APPEND)
    const int32_t *slots;  // generating slots or NULL
    int fixed_slot;
    // draw inputs (ROUND)
    const T *normals, *rnormals, *runiforms;
    // fused normals (fixed-slot factor draws): element e of row i is element
    // noffset (+ *nbase) + i d + e of the (nseed) normal stream
    int fused;
    uint64_t nseed, noffset;
    const uint64_t *nbase;
    int rn_stride, ru_stride;
    T *samples_out;
    // outputs
    T *out_logden, *out_generating;
    const T *logtargets;
    T *logweights;
    const int64_t *proposal_ids;
    int64_t *proposal_ids_out;
    T *lognum;             // APPEND in/out
    uint64_t *failures;
    int64_t index_base;
    int mode;
    int first_slot, last_slot;
    int chunk, resident;   // components staged at a time; whether that is all of them, once per CTA
    int whole;             // resident, and all of the bank
    int nslots, nchunks;   // components evaluated; their chunks
    int ksplit;            // thread groups of a CTA that share its samples and split the components
    int prefetch;          // two sample tiles: the next one loads while one is evaluated
};

// ---- slow path ----------------------------------------------------------
template <typename T> struct Rng { T m; int e; };
template <typename T> __device__ Rng<T> rfrexp(T v) { Rng<T> r; r.m = dfrexp(v, &r.e); return r; }
template <typename T> __device__ Rng<T> range_subtract(Rng<T> l, Rng<T> r) {
    if (l.m == T(0)) return Rng<T>{-r.m, r.e};
    if (r.m == T(0)) return l;
    int e = l.e > r.e ? l.e : r.e;
    int s;
    T m = dfrexp(dldexp(l.m, l.e - e) - dldexp(r.m, r.e - e), &s);
    return Rng<T>{m, m == T(0) ? 0 : e + s};
}
template <typename T> __device__ Rng<T> range_multiply(Rng<T> v, T f) {
    int fe, s;
    T fm = dfrexp(f, &fe);
    T p = dfrexp(v.m * fm, &s);
    return Rng<T>{p, p == T(0) ? 0 : v.e + fe + s};
}
template <typename T> __device__ Rng<T> range_divide(Rng<T> v, T dv) {
    int de, s;
    T dm = dfrexp(dv, &de);
    T q = dfrexp(v.m / dm, &s);
    return Rng<T>{q, q == T(0) ? 0 : v.e - de + s};
}
template <typename T> __device__ T logabsdiff(T l, T r) {
    T diff = l - r;
    if (isfinite(diff) || !isfinite(l) || !isfinite(r)) return dlog(fabs(diff));
    T al = fabs(l), ar = fabs(r);
    T big = al > ar ? al : ar, small = al > ar ? ar : al;
    return dlog(big) + dlog1p(small / big);
}

// Full reference semantics for one pair, reading the component from its
// global (reference-layout) arrays. Only taken for exceptional radii.
template <typename T>
__device__ __noinline__ T slow_component_logdensity(const MixParams<T> &p, int slot, const T *x) {
    const int d = p.d;
    T z[64];
    int ex[64];
    const T *mu = p.loc + (size_t)slot * d;
    T lognorm = p.lognorm[slot];
    T r2 = T(0);
    const bool factor = p.scale_kind == ISSM_SCALE_FACTOR;
    const T *L = factor ? p.scales + (size_t)slot * d * d : nullptr;
    const T *sc = p.scale_kind == ISSM_SCALE_SPHERICAL ? p.scales + slot : p.scales + (size_t)slot * d;
    auto scale_at = [&](int c) { return p.scale_kind == ISSM_SCALE_SPHERICAL ? sc[0] : sc[c]; };
    if (factor) {
        for (int r = 0; r < d; ++r) {
            T v = x[r] - mu[r];
            for (int c = 0; c < r; ++c) v -= L[r + (size_t)c * d] * z[c];
            v /= L[r + (size_t)r * d];
            z[r] = v;
            r2 += v * v;
        }
        if (!isfinite(r2)) {
            bool all_finite = true;
            for (int c = 0; c < d; ++c) all_finite &= (bool)isfinite(z[c]);
            if (!all_finite) {
                r2 = T(0);
                for (int r = 0; r < d; ++r) {
                    // _factor_standardized_coordinate (src/student_t_range.jl:89-109)
                    T v = x[r] - mu[r];
                    for (int c = 0; c < r; ++c) v -= L[r + (size_t)c * d] * z[c];
                    T dg = L[r + (size_t)r * d];
                    v /= dg;
                    if (!(isfinite(v) || !isfinite(x[r]) || !isfinite(mu[r]))) {
                        Rng<T> val = range_subtract(rfrexp(x[r]), rfrexp(mu[r]));
                        bool done = false;
                        for (int c = 0; c < r && !done; ++c) {
                            if (!isfinite(z[c])) { v = z[c]; done = true; break; }
                            val = range_subtract(val, range_multiply(rfrexp(z[c]), L[r + (size_t)c * d]));
                        }
                        if (!done) {
                            Rng<T> q = range_divide(val, dg);
                            v = dldexp(q.m, q.e);
                        }
                    }
                    z[r] = v;
                    r2 += v * v;
                }
            }
        }
    } else {
        for (int c = 0; c < d; ++c) {
            T v = (x[c] - mu[c]) / scale_at(c);
            r2 += v * v;
        }
        for (int c = 0; c < d; ++c) {
            T diff = x[c] - mu[c];
            z[c] = (isfinite(diff) || !isfinite(x[c]) || !isfinite(mu[c])) ? diff / scale_at(c)
                                                                           : x[c] / scale_at(c) - mu[c] / scale_at(c);
        }
    }
    auto logradius = [&]() -> T {
        T total = -num<T>::inf();
        if (factor) {
            for (int r = 0; r < d; ++r) {
                Rng<T> val = range_subtract(rfrexp(x[r]), rfrexp(mu[r]));
                for (int c = 0; c < r; ++c)
                    val = range_subtract(val, range_multiply(Rng<T>{z[c], ex[c]}, L[r + (size_t)c * d]));
                Rng<T> q = range_divide(val, L[r + (size_t)r * d]);
                z[r] = q.m;
                ex[r] = q.e;
                T la = dlog(fabs(q.m)) + T(q.e) * dlog(T(2));
                total = logaddexp(total, T(2) * la);
            }
        } else {
            for (int c = 0; c < d; ++c) {
                T v = logabsdiff(x[c], mu[c]) - dlog(scale_at(c));
                total = logaddexp(total, T(2) * v);
            }
        }
        return total;
    };
    if (p.family == ISSM_GAUSSIAN) {
        T half = T(0.5) * r2;
        if (!isfinite(r2)) {
            half = T(0);
            for (int c = 0; c < d; ++c) half += (T(0.5) * z[c]) * z[c];
        }
        return lognorm - half;
    }
    const T dof = p.dofs[slot];
    const bool risk = factor && p.range_risk != nullptr && p.range_risk[slot];
    const T ratio = r2 / dof;
    T radial;
    if (risk) {
        radial = log1pexp(logradius() - dlog(dof));
    } else if (r2 < num<T>::fmin()) {
        T s = dsqrt(dof), acc = T(0);
        for (int c = 0; c < d; ++c) { T v = z[c] / s; acc += v * v; }
        radial = dlog1p(acc);
    } else if (isfinite(ratio)) {
        radial = dlog1p(ratio);
    } else if (isfinite(r2)) {
        radial = dlog(r2) - dlog(dof);
    } else {
        T scale = T(0);
        for (int c = 0; c < d; ++c) scale = fmax(scale, fabs(z[c]));
        if (!isfinite(scale)) {
            radial = log1pexp(logradius() - dlog(dof));
        } else {
            T acc = T(0);
            for (int c = 0; c < d; ++c) { T v = z[c] / scale; acc += v * v; }
            radial = log1pexp(T(2) * dlog(scale) + dlog(acc) - dlog(dof));
        }
    }
    return lognorm - (dof + T(d)) / T(2) * radial;
}

// ---- shared-memory layout of one staged component (units of T) ------------------
//   [0] lognormalizer  [1] coefficient  [2] dof  [3] range-risk flag
//   [4] 1 / dof  [5] (dof + d) / 2
//   mu[D]  inv[D] (1 / diagonal or 1 / scale)
//   factor: column q from row q rounded down to a 16-byte group, columns packed
//   (compile-time offsets; the zero-padded rows beyond d are read, never used)
//   diagonal and spherical: scale[D]
template <typename T, int D, bool FACTOR> struct Layout {
    static constexpr int V = 16 / sizeof(T);
    static constexpr int kMu = 8, kInv = kMu + D, kBody = kInv + D;
    __host__ __device__ static constexpr int off(int q) {
        return V * D * (q / V) - V * V * (q / V) * (q / V - 1) / 2 + (q % V) * (D - V * (q / V));
    }
    static constexpr int kVecs = off(D) / V;  // 16-byte groups of the packed factor
    static constexpr int kStride = kBody + (FACTOR ? off(D) : D);
    static_assert(D % V == 0 && kStride % V == 0, "16-byte groups");
};

constexpr int kSimtThreads = 128;

__device__ __forceinline__ void cp_async_elem(float *dst, const float *src) { tc::cp_async4(dst, src); }
__device__ __forceinline__ void cp_async_elem(double *dst, const double *src) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(src) : "memory");
}

// Request components [k0, k0 + count) of the bank into shared memory with
// asynchronous copies (one commit group); stage_finish after their arrival.
template <typename T, int D, bool FACTOR>
__device__ __forceinline__ void stage_request(T *sm, const MixParams<T> &p, int k0, int count) {
    using Ly = Layout<T, D, FACTOR>;
    constexpr int V = Ly::V, NV = Ly::kVecs, kB = kSimtThreads;
    const int d = p.d, tid = threadIdx.x;
    for (int kk = tid; kk < count; kk += kB) {
        const int k = k0 + kk;
        T *c = sm + (size_t)kk * Ly::kStride;
        const T dof = p.dofs ? p.dofs[k] : T(0);
        c[0] = p.lognorm[k];
        c[1] = (p.den_kind == ISSM_DENOM_GENERATING || p.coef == nullptr) ? T(0) : p.coef[k];
        c[2] = dof;
        c[3] = (p.range_risk && p.scale_kind == ISSM_SCALE_FACTOR && p.family == ISSM_STUDENT_T) ? T(p.range_risk[k])
                                                                                                : T(0);
        c[4] = T(1) / dof;
        c[5] = (dof + T(d)) * T(0.5);
    }
    for (int e = tid; e < count * D; e += kB) {
        const int kk = e / D, r = e - kk * D;
        T *dst = sm + (size_t)kk * Ly::kStride + Ly::kMu + r;
        if (r < d) cp_async_elem(dst, p.loc + (size_t)(k0 + kk) * d + r);
        else *dst = T(0);
    }
    if constexpr (FACTOR) {
        // a thread keeps its 16-byte groups (column q, rows r0 ..) over the components
        constexpr int kSide = NV >= kB ? 1 : kB / NV;  // components side by side
        const bool vec = d % V == 0 && (reinterpret_cast<uintptr_t>(p.scales) & 15) == 0;
        const int kk0 = NV >= kB ? 0 : tid / NV;
        if (kk0 < kSide)
            for (int id = NV >= kB ? tid : tid % NV; id < NV; id += kB) {
                int b = 0, rest = id;  // V columns of D / V - b groups each
                while (rest >= V * (D / V - b)) {
                    rest -= V * (D / V - b);
                    ++b;
                }
                const int q = V * b + rest / (D / V - b), r0 = V * (b + rest % (D / V - b));
                const T *src = p.scales + (size_t)k0 * d * d + (size_t)q * d + r0;
                for (int kk = kk0; kk < count; kk += kSide) {
                    T *dst = sm + (size_t)kk * Ly::kStride + Ly::kBody + id * V;
                    const T *s = src + (size_t)kk * d * d;
                    if (vec && q < d && r0 < d) {
                        tc::cp_async16(dst, s);
                    } else {
#pragma unroll
                        for (int v = 0; v < V; ++v) {
                            if (q < d && r0 + v < d) cp_async_elem(dst + v, s + v);
                            else dst[v] = T(0);
                        }
                    }
                }
            }
    } else {
        for (int e = tid; e < count * D; e += kB) {
            const int kk = e / D, r = e - kk * D, k = k0 + kk;
            T *dst = sm + (size_t)kk * Ly::kStride + Ly::kBody + r;
            if (r < d) *dst = p.scale_kind == ISSM_SCALE_SPHERICAL ? p.scales[k] : p.scales[(size_t)k * d + r];
            else *dst = T(0);
        }
    }
    tc::cp_async_commit();
}

// the reciprocals of the staged diagonals or scales (zero beyond d)
template <typename T, int D, bool FACTOR> __device__ __forceinline__ void stage_finish(T *sm, int d, int count) {
    using Ly = Layout<T, D, FACTOR>;
    for (int e = threadIdx.x; e < count * D; e += kSimtThreads) {
        const int kk = e / D, r = e - kk * D;
        T *c = sm + (size_t)kk * Ly::kStride;
        c[Ly::kInv + r] = r < d ? T(1) / c[Ly::kBody + (FACTOR ? Ly::off(r) + r % Ly::V : r)] : T(0);
    }
}

// a / b given inv = 1 / b rounded: one Newton correction of the quotient with
// its exact remainder, three FP64 operations where the division takes nine of
// this GPU's narrow FP64 pipe. A quotient that overflows becomes NaN and takes
// the slow path's division.
template <typename T> __device__ __forceinline__ T quotient(T a, T b, T inv) {
    const T q = a * inv;
    return fma(fma(-q, b, a), inv, q);
}

template <typename T> __device__ __forceinline__ void load16(const T *src, T (&v)[16 / sizeof(T)]) {
    *reinterpret_cast<uint4 *>(v) = *reinterpret_cast<const uint4 *>(src);
}

// |L^-1 (x - mu)|^2 of S samples against one staged factor component: forward
// substitution by columns, v_r -= L_rq z_q, so each row's sum runs over q in
// ascending order and the updates of one column are independent. A 16-byte
// broadcast load serves V S FMAs. XREG: the samples are in registers; else in
// the shared tile (row s at xt + s * step).
template <typename T, int D, int S, bool XREG>
__device__ __forceinline__ void factor_radius(const T *__restrict__ c, const T (&x)[S][XREG ? D : 1],
                                              const T *__restrict__ xt, int step, int d, T (&r2)[S]) {
    using Ly = Layout<T, D, true>;
    constexpr int V = Ly::V;
    constexpr bool kSkip = sizeof(T) == 8;  // FP64 work beyond d costs more than its test
    T v[S][D];
#pragma unroll
    for (int r0 = 0; r0 < D; r0 += V) {
        T mu[V];
        load16(c + Ly::kMu + r0, mu);
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int j = 0; j < V; ++j) {
                if constexpr (XREG) v[s][r0 + j] = !kSkip || r0 < d ? x[s][r0 + j] - mu[j] : T(0);
                else v[s][r0 + j] = !kSkip || r0 < d ? xt[s * step + r0 + j] - mu[j] : T(0);
            }
    }
#pragma unroll
    for (int s = 0; s < S; ++s) r2[s] = T(0);
#pragma unroll
    for (int q = 0; q < D; ++q) {
        if (kSkip && q >= d) break;
        constexpr int M = V - 1;
        const int r1 = q & ~M;
        T col[V], z[S];
        load16(c + Ly::kBody + Ly::off(q), col);
        const T inv = c[Ly::kInv + q];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            z[s] = sizeof(T) == 4 ? v[s][q] * inv : quotient(v[s][q], col[q & M], inv);
            r2[s] += z[s] * z[s];
#pragma unroll
            for (int j = 0; j < V; ++j)
                if (r1 + j > q) v[s][r1 + j] -= col[j] * z[s];
        }
#pragma unroll
        for (int r0 = r1 + V; r0 < D; r0 += V) {
            if (kSkip && r0 >= d) break;
            load16(c + Ly::kBody + Ly::off(q) + (r0 - r1), col);
#pragma unroll
            for (int s = 0; s < S; ++s)
#pragma unroll
                for (int j = 0; j < V; ++j) v[s][r0 + j] -= col[j] * z[s];
        }
    }
}

template <typename T>
__device__ __forceinline__ T radial_logdensity(const T *__restrict__ c, T r2, int family, bool *slow) {
    if (family == ISSM_GAUSSIAN) {
        bool finite;
        if constexpr (sizeof(T) == 8) finite = (__double2hiint(r2) & 0x7ff00000) != 0x7ff00000;  // no FP64 instruction
        else finite = isfinite(r2);
        if (!finite) { *slow = true; return T(0); }
        return c[0] - T(0.5) * r2;
    }
    const T ratio = quotient(r2, c[2], c[4]);
    if constexpr (sizeof(T) == 8) {
        // c[3] is 0 or 1; r2 >= 0 or NaN: its order is its bits'
        const uint32_t b = (uint32_t)__double2hiint(r2), q = (uint32_t)__double2hiint(ratio);
        if (__double2hiint(c[3]) != 0 || b < 0x00100000u || b >= 0x7ff00000u || q >= 0x7ff00000u) {
            *slow = true;
            return T(0);
        }
        return c[0] - c[5] * table_log1p(ratio);
    }
    if (c[3] != T(0) || r2 < num<T>::fmin() || !isfinite(ratio)) { *slow = true; return T(0); }
    return c[0] - c[5] * dlog1p(ratio);
}

// Student-t radial multiplier from buffered draws (src/native_execution.jl:153-180).
template <typename T>
__device__ T radial_multiplier(T dof, const T *rn, const T *ru, bool has_u, uint16_t *reason) {
    *reason = 0;
    if (!has_u || dof == T(1)) {
        T den = fabs(rn[0]);
        if (!(isfinite(den) && den > T(0))) { *reason = ISSM_REASON_DRAW_EXHAUSTED; return T(0); }
        return T(1) / den;
    }
    const T shape = dof / T(2);
    const T adjusted = shape < T(1) ? shape + T(1) : shape;
    const T offset = adjusted - T(1) / T(3);
    const T coefm = T(1) / dsqrt(offset) / T(3);
    for (int a = 0; a < 8; ++a) {
        const T normal = rn[a], uniform = ru[a];
        const T root = T(1) + coefm * normal;
        if (!(root > T(0))) continue;
        const T cube = root * root * root;
        const T n2 = normal * normal;
        const bool acc = uniform < T(1) - T(0.0331) * (n2 * n2) ||
                         dlog(uniform) < T(0.5) * n2 + offset * (T(1) - cube + dlog(cube));
        if (!acc) continue;
        T g = offset * cube;
        if (shape < T(1)) g *= dpow(ru[8], T(1) / shape);
        if (!(isfinite(g) && g > T(0))) break;
        return dsqrt(dof / (T(2) * g));
    }
    *reason = ISSM_REASON_DRAW_EXHAUSTED;
    return T(0);
}

// The Student-t radial multiplier of sample i (1 for Gaussians; NaN with the
// failure recorded when the draws are exhausted).
template <typename T>
__device__ __forceinline__ T draw_multiplier(const MixParams<T> &p, int64_t i, int slot, bool record = true) {
    if (p.family != ISSM_STUDENT_T) return T(1);
    uint16_t r;
    const T m = radial_multiplier(p.dofs[slot], p.rnormals + (size_t)i * p.rn_stride,
                                  p.runiforms ? p.runiforms + (size_t)i * p.ru_stride : nullptr,
                                  p.runiforms != nullptr && p.ru_stride > 0, &r);
    if (!r) return m;
    if (record) record_failure(p.failures, p.index_base + i + 1, 0, r);
    return qnan<T>();
}

// x = mu_s + L_s (m n) of one row with the packed-bank summation order
// (_native_proposal_coordinate, src/native_execution.jl:238-264), for every
// `step`-th group of four coordinates from group g on, from the top down (so
// out may be in when step is 1: every normal a group needs is still there). c:
// the staged component, or null (then the bank's global arrays). Returns
// whether the coordinates formed are finite.
template <typename T, int D, bool FACTOR>
__device__ __forceinline__ bool draw_row(const MixParams<T> &p, int slot, const T *c, T m, int g, int step, const T *in,
                                         T *out) {
    using Ly = Layout<T, D, FACTOR>;
    const int d = p.d;
    const T *mu = c ? c + Ly::kMu : p.loc + (size_t)slot * d;
    bool valid = true;
    if constexpr (FACTOR) {
        const T *L = p.scales + (size_t)slot * d * d;
        const int top = (d - 1) >> 2;
        for (int r0 = 4 * (top - (top - g % step + step) % step); r0 >= 0; r0 -= 4 * step) {
            T acc[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = r0 + j < d ? mu[r0 + j] : T(0);
            // columns before the group's diagonal block, then its (up to four) columns
            if (c) {
#pragma unroll 4
                for (int q = 0; q < r0; ++q) {
                    const T z = in[q] * m;
                    T col[4];
                    const T *cq = c + Ly::kBody + Ly::off(q) - (q & ~(Ly::V - 1)) + r0;
                    *reinterpret_cast<uint4 *>(col) = *reinterpret_cast<const uint4 *>(cq);
                    if constexpr (sizeof(T) == 8)
                        *reinterpret_cast<uint4 *>(col + 2) = *reinterpret_cast<const uint4 *>(cq + 2);
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[j] += col[j] * z;
                }
            } else {
#pragma unroll 4
                for (int q = 0; q < r0; ++q) {
                    const T z = in[q] * m;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (r0 + j < d) acc[j] += L[(size_t)q * d + r0 + j] * z;
                }
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int q = r0 + t;
                if (q < d) {
                    const T z = in[q] * m;
                    const T *cq = c ? c + Ly::kBody + Ly::off(q) - (q & ~(Ly::V - 1)) : L + (size_t)q * d;
#pragma unroll
                    for (int j = t; j < 4; ++j)
                        if (r0 + j < d) acc[j] += cq[r0 + j] * z;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (r0 + j < d) {
                    out[r0 + j] = acc[j];
                    valid &= (bool)isfinite(acc[j]);
                }
        }
    } else {
        for (int r = g; r < d; r += step) {
            const T sc = p.scale_kind == ISSM_SCALE_SPHERICAL ? p.scales[slot] : p.scales[(size_t)slot * d + r];
            const T v = mu[r] + sc * (in[r] * m);
            out[r] = v;
            valid &= (bool)isfinite(v);
        }
    }
    return valid;
}

// One short row (d <= D <= 16) between global memory and registers: a thread's
// whole row is a sector or two, so a shared tile would add only its barriers.
template <typename T, int D> __device__ __forceinline__ void load_row(const T *g, int d, bool vec, T (&x)[D]) {
    constexpr int V = 16 / sizeof(T);
#pragma unroll
    for (int r0 = 0; r0 < D; r0 += V) {
        T v[V];
#pragma unroll
        for (int j = 0; j < V; ++j) v[j] = T(0);
        if (vec && r0 < d) load16(g + r0, v);
        else
#pragma unroll
            for (int j = 0; j < V; ++j)
                if (r0 + j < d) v[j] = g[r0 + j];
#pragma unroll
        for (int j = 0; j < V; ++j) x[r0 + j] = v[j];
    }
}
template <typename T, int D> __device__ __forceinline__ void store_row(T *g, int d, bool vec, const T (&x)[D]) {
    constexpr int V = 16 / sizeof(T);
#pragma unroll
    for (int r0 = 0; r0 < D; r0 += V) {
        if (vec && r0 < d) *reinterpret_cast<uint4 *>(g + r0) = *reinterpret_cast<const uint4 *>(&x[r0]);
        else
#pragma unroll
            for (int j = 0; j < V; ++j)
                if (r0 + j < d) g[r0 + j] = x[r0 + j];
    }
}

// draw_row in registers: x holds the normals, then the sample
template <typename T, int D, bool FACTOR>
__device__ __forceinline__ bool draw_registers(const MixParams<T> &p, int slot, const T *c, T m, T (&x)[D]) {
    using Ly = Layout<T, D, FACTOR>;
    constexpr int V = Ly::V;
    const int d = p.d;
    const T *mu = c ? c + Ly::kMu : p.loc + (size_t)slot * d;
    if constexpr (!FACTOR) {
        const bool one = p.scale_kind == ISSM_SCALE_SPHERICAL;
        const T *sc = c ? c + Ly::kBody : one ? p.scales + slot : p.scales + (size_t)slot * d;
        bool valid = true;
#pragma unroll
        for (int r = 0; r < D; ++r)
            if (r < d) {
                x[r] = mu[r] + sc[c || !one ? r : 0] * (x[r] * m);
                valid &= (bool)isfinite(x[r]);
            }
        return valid;
    }
    const T *L = p.scales + (size_t)slot * d * d;
    T y[D];
#pragma unroll
    for (int r = 0; r < D; ++r) y[r] = r < d ? mu[r] : T(0);
#pragma unroll
    for (int q = 0; q < D; ++q) {
        const T z = x[q] * m;
#pragma unroll
        for (int r0 = q & ~(V - 1); r0 < D; r0 += V) {
            T col[V];
            if (c) {
                load16(c + Ly::kBody + Ly::off(q) + r0 - (q & ~(V - 1)), col);
            } else {
#pragma unroll
                for (int j = 0; j < V; ++j) col[j] = q < d && r0 + j >= q && r0 + j < d ? L[q * d + r0 + j] : T(0);
            }
#pragma unroll
            for (int j = 0; j < V; ++j)
                if (r0 + j >= q) y[r0 + j] += col[j] * z;
        }
    }
    bool valid = true;
#pragma unroll
    for (int r = 0; r < D; ++r) {
        x[r] = y[r];
        if (r < d) valid &= (bool)isfinite(y[r]);
    }
    return valid;
}

// rows x d contiguous elements between global memory and the padded tile,
// coalesced, four in flight per thread
template <typename T, int LX, bool IN>
__device__ __forceinline__ void move_tile(T *tile, T *g, int rows, int d) {
    constexpr int kB = kSimtThreads;
    const int dq = kB / d, dr = kB - dq * d, total = rows * d;
    int r = threadIdx.x / d, c = threadIdx.x - r * d;
    for (int e = threadIdx.x; e < total;) {
        T v[4];
        int at[4];
        const int e0 = e;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            at[u] = e < total ? r * LX + c : -1;
            if (at[u] >= 0) v[u] = IN ? g[e] : tile[at[u]];
            e += kB;
            r += dq;
            c += dr;
            if (c >= d) {
                c -= d;
                ++r;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (at[u] >= 0) {
                if (IN) tile[at[u]] = v[u];
                else g[e0 + u * kB] = v[u];
            }
    }
}

// the same into the tile with asynchronous copies (one commit group)
template <typename T, int LX> __device__ __forceinline__ void request_tile(T *tile, const T *g, int rows, int d) {
    constexpr int kB = kSimtThreads;
    const int dq = kB / d, dr = kB - dq * d, total = rows * d;
    int r = threadIdx.x / d, c = threadIdx.x - r * d;
    for (int e = threadIdx.x; e < total; e += kB) {
        cp_async_elem(tile + r * LX + c, g + e);
        r += dq;
        c += dr;
        if (c >= d) {
            c -= d;
            ++r;
        }
    }
    tc::cp_async_commit();
}

// rows go between global memory and registers, without a tile
template <typename T, int D> __host__ __device__ constexpr bool simt_direct() { return sizeof(T) == 4 && D <= 16; }

// Mixture densities, static-MIS rounds and appends. CTAs of 128 threads
// walk tiles of samples; the bank is staged in shared memory, whole and once
// per CTA when it fits (`resident`), else in double-buffered chunks prefetched
// with asynchronous copies while the previous chunk is evaluated. Each thread
// owns S samples; with ksplit > 1 the CTA's thread groups share the samples
// and take every ksplit-th component, and their log-sum-exp states merge at the
// end (few samples would otherwise leave most warps idle).
//
// Bound by FP32 FMA issue with shared-memory operands (one 16-byte broadcast
// load costs about 2.4 clocks of an SM; two samples per load is where FMAs
// overtake loads) or by the FP64 pipe. One thread per sample, one CTA per 128
// samples and the bank restaged element by element by each took 11.9 ms for a
// static-MIS call of 4,194,304 samples, d = 16, 64 components (now 2.9 ms, 2.6 of
// them this kernel: 263 issue slots per sample and component, 190 on the FMA pipe, 136
// of those the substitution's), and 1.33 ms in the kernel for a population round of
// 16,384 samples, d = 32, 256 components (0.25).
template <typename T, int D, bool FACTOR, int S, int MINB, bool DIRECT>
__global__ void __launch_bounds__(kSimtThreads, MINB) mixture_simt_kernel(MixParams<T> p) {
    using Ly = Layout<T, D, FACTOR>;
    constexpr bool XREG = DIRECT || (FACTOR && sizeof(T) == 4 && D <= 32);  // beyond, x and v together exceed the registers
    constexpr int LX = D + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *comps = reinterpret_cast<T *>(smem_raw);
    const int d = p.d, tid = threadIdx.x, KS = p.ksplit, GT = kSimtThreads / KS, TR = GT * S;
    T *tiles = comps + (size_t)(p.resident ? 1 : 2) * p.chunk * Ly::kStride;
    T *merge = tiles + (DIRECT ? 0 : (size_t)(p.prefetch ? 2 : 1) * TR * LX);  // ksplit > 1: per thread (max, sum, generating, flags),
    T *mult = merge + 4 * kSimtThreads;          // per sample the radial multiplier,
    T *drawn_tile = mult + kSimtThreads;         // and the drawn samples
    __shared__ int s_bad[kSimtThreads], s_lo, s_hi;
    const int grp = tid / GT, si = tid - grp * GT;
    const int nslots = p.nslots, nchunks = p.nchunks;
    const int64_t ntiles = (p.n + TR - 1) / TR;
    const int my_tiles = (int)((ntiles - (int64_t)blockIdx.x + gridDim.x - 1) / gridDim.x);
    const bool only_own = p.den_kind == ISSM_DENOM_GENERATING;  // a tile needs its own samples' slots only
    auto request = [&](int ch, int buf) {
        const int k0 = ch * p.chunk;
        stage_request<T, D, FACTOR>(comps + (size_t)buf * p.chunk * Ly::kStride, p, p.first_slot + k0,
                                    min(p.chunk, nslots - k0));
    };
    // a draw's component: staged where the whole bank is, else null (a prefix may stop
    // before a drawn slot)
    auto staged = [&](int slot) -> const T * { return p.whole ? comps + (size_t)slot * Ly::kStride : nullptr; };
    const bool drawn = p.mode == kModeRound;
    const T *rows_in = drawn ? p.normals : p.x;
    auto tile_row = [&](int it) -> int64_t { return ((int64_t)blockIdx.x + (int64_t)it * gridDim.x) * TR; };
    auto request_rows = [&](int it) {
        const int64_t r0 = tile_row(it);
        request_tile<T, LX>(tiles + (size_t)(it & 1) * TR * LX, rows_in + (size_t)r0 * d, (int)min((int64_t)TR, p.n - r0), d);
    };
    // coordinates beyond d are read as zeros
    for (int e = DIRECT ? TR * LX : tid; e < TR * LX; e += kSimtThreads) {
        tiles[e] = T(0);
        if (p.prefetch) tiles[TR * LX + e] = T(0);
        if (KS > 1) drawn_tile[e] = T(0);
    }
    if (!DIRECT && p.prefetch) {
        __syncthreads();
        request_rows(0);
    }
    const bool vec = DIRECT && d % Ly::V == 0 &&
                     ((reinterpret_cast<uintptr_t>(rows_in) | reinterpret_cast<uintptr_t>(p.samples_out)) & 15) == 0;
    if (p.resident || !only_own) request(0, 0);
    if (p.resident) {
        tc::cp_async_wait_all();
        __syncthreads();
        stage_finish<T, D, FACTOR>(comps, d, nslots);
    }
    int item = 0;  // chunks evaluated so far: the buffer in use alternates
    for (int it = 0; it < my_tiles; ++it) {
        const int64_t row0 = tile_row(it);
        const int rows = (int)min((int64_t)TR, p.n - row0);
        T *tile = tiles;
        if (DIRECT) {
            if (it == 0 || KS > 1) __syncthreads();  // the staged bank; the merge buffer
        } else if (p.prefetch) {
            tile += (size_t)(it & 1) * TR * LX;
            tc::cp_async_wait_all();
            __syncthreads();
            if (it + 1 < my_tiles) request_rows(it + 1);
        } else {
            __syncthreads();
            move_tile<T, LX, true>(tile, const_cast<T *>(rows_in + (size_t)row0 * d), rows, d);
            __syncthreads();
        }
        bool ok[S];
        int gen[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int64_t i = row0 + si + s * GT;
            ok[s] = i < p.n;
            gen[s] = ok[s] ? (p.slots ? p.slots[i] : p.fixed_slot) : 0;
        }
        T *xs = tile;
        T x[S][XREG ? D : 1];
        if constexpr (DIRECT) {
            auto put = [&](int s) {
                const int64_t i = row0 + si + s * GT;
                if (i >= p.n) return;
                if (!ok[s]) record_failure(p.failures, p.index_base + i + 1, 0, ISSM_REASON_GENERATED_NONFINITE);
                if (p.samples_out) store_row<T, D>(p.samples_out + (size_t)i * d, d, vec, x[s]);
            };
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int64_t i = row0 + si + s * GT;
                load_row<T, D>(rows_in + (size_t)(ok[s] ? i : 0) * d, d, vec, x[s]);
                if (drawn && ok[s])
                    ok[s] = draw_registers<T, D, FACTOR>(p, gen[s], staged(gen[s]), draw_multiplier(p, i, gen[s], grp == 0), x[s]);
                if (drawn && KS == 1) put(s);
            }
            if (S == 1 && drawn && KS > 1) {
                __syncthreads();  // every group has its normals: the samples may take their place
                if (grp == 0) put(0);
            }
            if (drawn && KS > 1) __syncthreads();  // the slow path reads the stored samples
        } else if (drawn) {
            if (KS == 1) {
#pragma unroll
                for (int s = 0; s < S; ++s)
                    if (ok[s]) {
                        const int64_t i = row0 + si + s * GT;
                        const T *c = staged(gen[s]);
                        T *row = tile + (size_t)(si + s * GT) * LX;
                        if (!draw_row<T, D, FACTOR>(p, gen[s], c, draw_multiplier(p, i, gen[s]), 0, 1, row, row)) {
                            record_failure(p.failures, p.index_base + i + 1, 0, ISSM_REASON_GENERATED_NONFINITE);
                            ok[s] = false;
                        }
                    }
            } else {
                // every group draws: the samples' multipliers, then the rows' coordinates, are dealt out
                const int64_t i = row0 + si;
                if (ok[0] && si % KS == grp) mult[si] = draw_multiplier(p, i, gen[0]);
                if (grp == 0) s_bad[si] = 0;
                __syncthreads();
                if (ok[0]) {
                    const T *c = staged(gen[0]);
                    if (!draw_row<T, D, FACTOR>(p, gen[0], c, mult[si], grp, KS, tile + (size_t)si * LX,
                                                drawn_tile + (size_t)si * LX))
                        s_bad[si] = 1;
                }
                xs = drawn_tile;
            }
            __syncthreads();
            if (KS > 1 && ok[0] && s_bad[si]) {
                ok[0] = false;
                if (grp == 0)
                    record_failure(p.failures, p.index_base + row0 + si + 1, 0, ISSM_REASON_GENERATED_NONFINITE);
            }
            if (p.samples_out) move_tile<T, LX, false>(xs, p.samples_out + (size_t)row0 * d, rows, d);
            __syncthreads();  // the slow path reads the stored samples
        }
        const T *xt = xs + (size_t)si * LX;
        if constexpr (XREG && !DIRECT) {
#pragma unroll
            for (int s = 0; s < S; ++s)
#pragma unroll
                for (int r = 0; r < D; ++r) x[s][r] = xt[s * GT * LX + r];
        }
        LseState<T> lse[S];
        T gen_lq[S], last_lq[S];
        int g_gen[S];
        bool has_gen[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            gen_lq[s] = last_lq[s] = T(0);
            has_gen[s] = false;
            g_gen[s] = (p.den_kind == ISSM_DENOM_PARTIAL && ok[s]) ? p.group[gen[s]] : 0;
        }
        int ch0 = 0, ch1 = nchunks - 1;
        if (only_own && !p.resident) {
            // the chunks that hold the tile's slots (neighbours for a stratified assignment)
            if (tid == 0) {
                s_lo = 0x7fffffff;
                s_hi = -1;
            }
            __syncthreads();
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (ok[s]) {
                    atomicMin(&s_lo, gen[s]);
                    atomicMax(&s_hi, gen[s]);
                }
            __syncthreads();
            ch0 = max(0, s_lo - p.first_slot) / p.chunk;
            ch1 = s_hi < 0 ? ch0 - 1 : min(nchunks - 1, (s_hi - p.first_slot) / p.chunk);
            if (ch0 <= ch1) request(ch0, item & 1);
        }
        for (int ch = ch0; ch <= ch1; ++ch, ++item) {
            const T *buf = comps;
            const int k0 = p.first_slot + ch * p.chunk, count = min(p.chunk, p.last_slot - k0 + 1);
            if (!p.resident) {
                T *b = comps + (size_t)(item & 1) * p.chunk * Ly::kStride;
                tc::cp_async_wait_all();
                __syncthreads();  // the chunk has landed and the other buffer is free
                stage_finish<T, D, FACTOR>(b, d, count);
                if (ch < ch1) request(ch + 1, (item + 1) & 1);
                else if (!only_own && it + 1 < my_tiles) request(0, (item + 1) & 1);
                __syncthreads();
                buf = b;
            }
            for (int kk = grp; kk < count; kk += KS) {
                const int k = k0 + kk;
                bool need[S], any = false;
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    need[s] = ok[s];
                    if (p.den_kind == ISSM_DENOM_GENERATING) need[s] = ok[s] && k == gen[s];
                    else if (p.den_kind == ISSM_DENOM_PARTIAL) need[s] = ok[s] && p.group[k] == g_gen[s];
                    any |= need[s];
                }
                if (!__any_sync(0xffffffffu, any)) continue;
                const T *c = buf + (size_t)kk * Ly::kStride;
                T r2[S];
                if constexpr (FACTOR) {
                    factor_radius<T, D, S, XREG>(c, x, xt, GT * LX, d, r2);
                } else {
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        r2[s] = T(0);
                        auto add = [&](T xr, int r) {
                            const T dv = xr - c[Ly::kMu + r];
                            const T v = sizeof(T) == 4 ? dv * c[Ly::kInv + r]
                                                       : quotient(dv, c[Ly::kBody + r], c[Ly::kInv + r]);
                            r2[s] += v * v;
                        };
                        if constexpr (XREG) {
#pragma unroll
                            for (int r = 0; r < D; ++r)
                                if (r < d) add(x[s][r], r);
                        } else {
                            for (int r = 0; r < d; ++r) add(xt[s * GT * LX + r], r);
                        }
                    }
                }
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    if (!need[s]) continue;
                    bool slow = false;
                    T lq = radial_logdensity<T>(c, r2[s], p.family, &slow);
                    if (slow) {
                        const int64_t i = row0 + si + s * GT;
                        lq = slow_component_logdensity<T>(p, k, (drawn ? p.samples_out : p.x) + (size_t)i * d);
                    }
                    if (k == gen[s]) {
                        gen_lq[s] = lq;
                        has_gen[s] = true;
                    }
                    last_lq[s] = lq;
                    lse[s].add(c[1] + lq);
                }
            }
        }
        if (KS > 1) {
            // merge the groups' states in group order (S == 1 here)
            T *mine = merge + (size_t)tid * 4;
            mine[0] = lse[0].m;
            mine[1] = lse[0].s;
            mine[2] = gen_lq[0];
            mine[3] = T((has_gen[0] ? 1 : 0) + (lse[0].nan ? 2 : 0));
            __syncthreads();
            if (grp == 0)
                for (int g = 1; g < KS; ++g) {
                    const T *o = merge + (size_t)(g * GT + si) * 4;
                    const int flags = (int)o[3];
                    if (flags & 1) gen_lq[0] = o[2];
                    lse[0].merge(o[0], o[1], (flags & 2) != 0);
                }
        }
        if (grp != 0) continue;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int64_t i = row0 + si + s * GT;
            if (i >= p.n) continue;
            if (p.mode == kModeAppend) {
                uint16_t reason = isnan(last_lq[s]) ? ISSM_REASON_PROPOSAL_INVALID : 0;
                if (!reason) {
                    const T v = logaddexp(p.lognum[i], p.coef[p.first_slot] + last_lq[s]);
                    if (isnan(v) || v == -num<T>::inf()) reason = ISSM_REASON_PROPOSAL_INVALID;
                    else p.lognum[i] = v;
                }
                if (reason) record_failure(p.failures, p.index_base + i + 1, 0, reason);
                continue;
            }
            T den = -num<T>::inf();
            if (ok[s]) {
                den = lse[s].value();
                if (isnan(gen_lq[s]) || gen_lq[s] == -num<T>::inf() || isnan(den) || den == -num<T>::inf()) {
                    record_failure(p.failures, p.index_base + i + 1, 0, ISSM_REASON_PROPOSAL_INVALID);
                    ok[s] = false;
                    den = -num<T>::inf();
                }
            }
            if (p.mode == kModeDenominator) {
                p.out_logden[i] = den;
                if (p.out_generating) p.out_generating[i] = ok[s] ? gen_lq[s] : -num<T>::inf();
                continue;
            }
            // kModeRound: _mis_round_launch_kernel! (src/mis_execution.jl:674-720)
            T lw = -num<T>::inf();
            int64_t pid = 0;
            if (ok[s]) {
                const T target = p.logtargets ? p.logtargets[i] : T(0);
                const uint16_t tr = p.logtargets ? target_reason(target) : 0;
                if (tr) {
                    record_failure(p.failures, p.index_base + i + 1, 0, tr);
                } else {
                    T w;
                    const uint16_t r = subtract_logweight(target, den, &w);
                    if (r) record_failure(p.failures, p.index_base + i + 1, 0, r);
                    else {
                        lw = w;
                        pid = p.proposal_ids ? p.proposal_ids[gen[s]] : (int64_t)gen[s] + 1;
                    }
                }
            }
            p.logweights[i] = lw;
            if (p.proposal_ids_out) p.proposal_ids_out[i] = pid;
            if (p.out_logden) p.out_logden[i] = den;
            if (p.out_generating) p.out_generating[i] = gen_lq[s];
        }
    }
}

// Draws from given slots: a thread per sample, its row in registers, the components
// from global memory (L1: the bank is small against the samples). Longer rows pass
// through a shared tile, so that they are read and written whole lines at a time (FP32,
// 100,000 x 64: 142 -> 112 us), except in FP64 beyond 32 coordinates, whose tile
// leaves too few warps (d = 33, up to 10,000 samples: 47 -> 58). In the kernel above,
// without registers to unroll into, FP64 draws of 100,000 x 33 took 268 us, here 172.
template <typename T, int D> constexpr bool draw_slots_tile() { return D > 4 && D * sizeof(T) <= 256; }
template <typename T, int D, bool FACTOR>
__global__ void __launch_bounds__(kSimtThreads) draw_slots_kernel(MixParams<T> p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr bool TILE = draw_slots_tile<T, D>();
    constexpr int LX = D + 1;
    const int d = p.d;
    const int64_t row0 = (int64_t)blockIdx.x * kSimtThreads, i = row0 + threadIdx.x;
    const int rows = (int)min((int64_t)kSimtThreads, p.n - row0);
    T *tile = reinterpret_cast<T *>(smem_raw);
    if (TILE) {
        move_tile<T, LX, true>(tile, const_cast<T *>(p.normals + (size_t)row0 * d), rows, d);
        __syncthreads();
    }
    if (i < p.n) {
        const int slot = p.slots ? p.slots[i] : p.fixed_slot;
        const T m = draw_multiplier(p, i, slot);
        const T *mu = p.loc + (size_t)slot * d, *in = TILE ? tile + threadIdx.x * LX : p.normals + (size_t)i * d;
        T *out = TILE ? tile + threadIdx.x * LX : p.samples_out + (size_t)i * d;
        T z[D];
#pragma unroll
        for (int c = 0; c < D; ++c) z[c] = c < d ? in[c] * m : T(0);
        const T *L = p.scales + (size_t)slot * (p.scale_kind == ISSM_SCALE_SPHERICAL ? 1 : FACTOR ? d * d : d);
        bool valid = true;
#pragma unroll
        for (int r = 0; r < D; ++r) {
            if (r >= d) continue;
            T v = mu[r];
            if constexpr (FACTOR) {
#pragma unroll
                for (int c = 0; c <= r; ++c) v += L[r + (size_t)c * d] * z[c];
            } else {
                v += L[p.scale_kind == ISSM_SCALE_SPHERICAL ? 0 : r] * z[r];
            }
            out[r] = v;
            valid &= (bool)isfinite(v);
        }
        if (!valid) record_failure(p.failures, p.index_base + i + 1, 0, ISSM_REASON_GENERATED_NONFINITE);
    }
    if (TILE) {
        __syncthreads();
        move_tile<T, LX, false>(tile, p.samples_out + (size_t)row0 * d, rows, d);
    }
}

template <typename T, int D, bool FACTOR> static int launch_draw_slots(const MixParams<T> &p, cudaStream_t stream) {
    if (p.n < 1) return 0;
    auto kern = draw_slots_kernel<T, D, FACTOR>;
    const size_t smem = draw_slots_tile<T, D>() ? (size_t)kSimtThreads * (D + 1) * sizeof(T) : 0;  // 34 KB at most
    kern<<<(unsigned)((p.n + kSimtThreads - 1) / kSimtThreads), kSimtThreads, smem, stream>>>(p);
    note_launch();
    return (int)cudaGetLastError();
}

// Fixed-slot draws from one factor component, x = mu + L (m z) with the
// reference's summation order (mu first, then q = 0..r). A CTA of 256 threads
// takes a tile of 64 rows:
//  * the factor is staged once per CTA, column-major (column q holds L[., q],
//    so 4 consecutive rows of a column are one 16-byte broadcast load), with
//    its upper triangle zeroed;
//  * the tile's normals are staged transposed, zT[q][row], from coalesced
//    loads or, with fused normals, generated there from the counter-based
//    stream (the tile's elements are contiguous in the stream, so the threads
//    take its Philox blocks in turn and no normal touches HBM);
//  * four threads share a row and split its output coordinates where the
//    triangular work quarters; each forms 4 coordinates at a time as
//    independent FMA chains over q = 0..r0+3 (the zero upper triangle makes
//    the extra terms exact no-ops), reading z[q] of 32 consecutive rows from
//    32 banks, so the loops stay compact (a fully unrolled triangle overflows
//    the instruction cache);
//  * x goes to a row-major staging tile and is stored coalesced.
constexpr int kDrawRows = 64;     // rows per tile
constexpr int kDrawParts = 4;     // threads per row
template <int D> struct DrawSplit {
    // first output coordinate of part i: 4 * ceil(D sqrt(i / 4) / 4), the triangle's quarters
    static constexpr int at(int i) {
        return i == 0 ? 0 : i >= 4 ? D : D == 64 ? (i == 1 ? 32 : i == 2 ? 44 : 56)
                                       : D == 32 ? (i == 1 ? 16 : i == 2 ? 24 : 28)
                                       : D == 16 ? (i == 1 ? 8 : i == 2 ? 12 : 16)
                                                 : D;
    }
};

template <typename T, int D>
__global__ void __launch_bounds__(kDrawRows * kDrawParts) draw_fixed_kernel(MixParams<T> p) {
    constexpr int LC = D + 4;          // column stride of the staged factor (16-byte aligned columns)
    constexpr int LR = kDrawRows + 4;  // row stride of zT (per coordinate)
    constexpr int LX = D + 4;          // row stride of the x tile
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *Lc = reinterpret_cast<T *>(smem_raw);  // D columns of LC
    T *mus = Lc + D * LC;                      // D
    T *zT = mus + D;                           // D x LR
    T *xs = zT + D * LR;                       // kDrawRows x LX
    __shared__ T s_mult[kDrawRows];
    __shared__ int s_bad[kDrawRows];
    const int d = p.d, k = p.fixed_slot, tid = threadIdx.x;
    const int row = tid % kDrawRows, part = tid / kDrawRows;  // warp-uniform parts
    const T *Lk = p.scales + (size_t)k * d * d;
    // rows of whole 16-byte vectors, both buffers 16-byte aligned
    const bool vec = (d * sizeof(T)) % 16 == 0 && (p.fused || (reinterpret_cast<uintptr_t>(p.normals) & 15) == 0) &&
                     (reinterpret_cast<uintptr_t>(p.samples_out) & 15) == 0;
    if (d == D && (reinterpret_cast<uintptr_t>(Lk) & 15) == 0) {
        // every column in flight at once (16-byte asynchronous copies; the padding is never read)
        constexpr int V = 16 / sizeof(T), CV = D / V;
        for (int e = tid; e < D * CV; e += blockDim.x) {
            const int q = e / CV, c = e - q * CV;
            tc::cp_async16(Lc + q * LC + c * V, Lk + (size_t)q * D + c * V);
        }
        tc::cp_async_commit();
        tc::cp_async_wait_all();
        __syncthreads();
        for (int e = tid; e < D * D; e += blockDim.x) {
            const int q = e / D, r = e - q * D;
            if (r < q) Lc[q * LC + r] = T(0);
        }
    } else {
        for (int e = tid; e < D * LC; e += blockDim.x) {
            const int q = e / LC, r = e - q * LC;
            Lc[e] = (q < d && r < d && r >= q) ? Lk[(size_t)q * d + r] : T(0);
        }
    }
    for (int r = tid; r < D; r += blockDim.x) mus[r] = r < d ? p.loc[(size_t)k * d + r] : T(0);
    const T dof = p.family == ISSM_STUDENT_T ? p.dofs[k] : T(0);
    const uint64_t noff = p.fused ? p.noffset + (p.nbase ? *p.nbase : 0ull) : 0ull;
    // coordinates d..D-1 of z stay zero
    for (int e = tid; e < (D - d) * LR; e += blockDim.x) zT[d * LR + e] = T(0);
    __syncthreads();
    const int lo = DrawSplit<D>::at(part), hi = DrawSplit<D>::at(part + 1);
    const int64_t ntiles = (p.n + kDrawRows - 1) / kDrawRows;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t row0 = tile * kDrawRows;
        const int rows = (int)min((int64_t)kDrawRows, p.n - row0);
        if (p.fused) {
            using NB = NormalBlock<T>;
            const uint64_t first = noff + (uint64_t)row0 * d;
            const int count = rows * d;
            const uint64_t b0 = first >> NB::kShift;
            if (d == D && (first & (NB::kPer - 1)) == 0) {
                // every Philox block is kPer consecutive coordinates of one row;
                // consecutive lanes take consecutive rows (conflict-free stores into zT)
                constexpr int BPR = D / NB::kPer;
                for (int j = tid; j < kDrawRows * BPR; j += blockDim.x) {
                    const int r = j % kDrawRows, cb = j / kDrawRows;
                    if (r >= rows) continue;
                    T v[NB::kPer];
                    NB::eval(b0 + (uint64_t)(r * BPR + cb), p.nseed, v);
#pragma unroll
                    for (int l = 0; l < NB::kPer; ++l) zT[(cb * NB::kPer + l) * LR + r] = v[l];
                }
            } else {
                const int nb = (int)(((first + (uint64_t)count - 1) >> NB::kShift) - b0 + 1);
                for (int j = tid; j < nb; j += blockDim.x) {
                    const uint64_t blk = b0 + (uint64_t)j;
                    T v[NB::kPer];
                    NB::eval(blk, p.nseed, v);
                    const int q0 = (int)(int64_t)((blk << NB::kShift) - first);  // negative in a split first block
                    int r = q0 >= 0 ? q0 / d : -1;
                    int c = q0 - r * d;
#pragma unroll
                    for (int l = 0; l < NB::kPer; ++l) {
                        if (c >= d) { c -= d; ++r; }
                        if (q0 + l >= 0 && q0 + l < count) zT[c * LR + r] = v[l];
                        ++c;
                    }
                }
            }
        } else {
            const T *nz = p.normals + row0 * d;
            for (int e = tid; e < rows * d; e += blockDim.x) {
                const int r = e / d, c = e - r * d;
                zT[c * LR + r] = nz[e];
            }
        }
        // the radial multiplier of each row (Student-t), once per row
        if (part == 0 && row < rows) {
            T m = T(1);
            if (p.family == ISSM_STUDENT_T) {
                const int64_t i = row0 + row;
                uint16_t rr;
                m = radial_multiplier(dof, p.rnormals + (size_t)i * p.rn_stride,
                                      p.runiforms ? p.runiforms + (size_t)i * p.ru_stride : nullptr,
                                      p.runiforms != nullptr && p.ru_stride > 0, &rr);
                if (rr) {
                    record_failure(p.failures, p.index_base + i + 1, 0, rr);
                    m = qnan<T>();
                }
            }
            s_mult[row] = m;
            s_bad[row] = 0;
        }
        __syncthreads();
        if (row < rows) {
            const T m = s_mult[row];
            const bool scaled = p.family == ISSM_STUDENT_T;
            bool valid = true;
            for (int r0 = lo; r0 < hi; r0 += 4) {
                T v0 = mus[r0], v1 = mus[r0 + 1], v2 = mus[r0 + 2], v3 = mus[r0 + 3];
                for (int q0 = 0; q0 <= r0; q0 += 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int q = q0 + u;
                        const T z = scaled ? zT[q * LR + row] * m : zT[q * LR + row];
                        const T *col = Lc + q * LC + r0;
                        v0 += col[0] * z;
                        v1 += col[1] * z;
                        v2 += col[2] * z;
                        v3 += col[3] * z;
                    }
                }
                T *xr = xs + row * LX + r0;
                xr[0] = v0; xr[1] = v1; xr[2] = v2; xr[3] = v3;
                if (r0 < d) valid &= (bool)isfinite(v0);
                if (r0 + 1 < d) valid &= (bool)isfinite(v1);
                if (r0 + 2 < d) valid &= (bool)isfinite(v2);
                if (r0 + 3 < d) valid &= (bool)isfinite(v3);
            }
            if (!valid) s_bad[row] = 1;
        }
        __syncthreads();
        if (part == 0 && row < rows && s_bad[row])
            record_failure(p.failures, p.index_base + row0 + row + 1, 0, ISSM_REASON_GENERATED_NONFINITE);
        T *out = p.samples_out + row0 * d;
        if (vec) {
            constexpr int V = 16 / sizeof(T);
            const int dv = d / V;
            for (int e = tid; e < rows * dv; e += blockDim.x) {
                const int r = e / dv, c = e - r * dv;
                *reinterpret_cast<uint4 *>(out + (size_t)e * V) = *reinterpret_cast<const uint4 *>(xs + r * LX + c * V);
            }
        } else {
            for (int e = tid; e < rows * d; e += blockDim.x) {
                const int r = e / d, c = e - r * d;
                out[e] = xs[r * LX + c];
            }
        }
        __syncthreads();
    }
}

template <typename T, int D> static int launch_draw_fixed(const MixParams<T> &p, cudaStream_t stream) {
    const size_t smem = sizeof(T) * ((size_t)D * (D + 4) + D + (size_t)D * (kDrawRows + 4) +
                                     (size_t)kDrawRows * (D + 4));
    auto kern = draw_fixed_kernel<T, D>;
    if (smem > 48 * 1024) {
        const int e = allow_dynamic_smem((const void *)kern);
        if (e) return e;
    }
    const int64_t tiles = (p.n + kDrawRows - 1) / kDrawRows;
    const int blocks = (int)min(tiles, (int64_t)device_sms() * 64);
    if (blocks < 1) return 0;
    kern<<<blocks, kDrawRows * kDrawParts, smem, stream>>>(p);
    note_launch();
    return (int)cudaGetLastError();
}

constexpr size_t kSimtSmem = 227 * 1024;  // shared memory of an SM that CTAs can take (1 KB each reserved)

template <typename T, int D, bool FACTOR, int S, int MINB, bool DIRECT = simt_direct<T, D>()>
static int launch_simt(MixParams<T> p, cudaStream_t stream) {
    using Ly = Layout<T, D, FACTOR>;
    if (p.n < 1) return 0;
    const int nslots = p.last_slot - p.first_slot + 1;
    const int sms = device_sms();
    auto tiles_of = [&](int ks) { return (p.n + kSimtThreads / ks * S - 1) / (kSimtThreads / ks * S); };
    // Components are split over thread groups while there are fewer than four
    // CTAs per SM, FP64 from eight components per group on than eight waves of them:
    // it runs at the pipe's rate from one warp per scheduler on, so finer tiles only
    // even out the last wave, for the price of the merge's exponentials. A
    // generating-only denominator has one component per sample to split.
    int ks = 1;
    if (S == 1 && nslots > 1 && p.den_kind != ISSM_DENOM_GENERATING)
        while (ks < 4 && nslots >= 2 * ks &&
               tiles_of(ks) < (int64_t)sms * min(MINB, 4) * (sizeof(T) == 8 && nslots >= 16 * ks ? 8 : 1))
            ks *= 2;
    p.ksplit = ks;
    const int64_t tiles = tiles_of(ks);
    const size_t per = (size_t)Ly::kStride * sizeof(T);
    const size_t rows_bytes = DIRECT ? 0 : (size_t)(kSimtThreads / ks) * S * (D + 1) * sizeof(T);
    const size_t fixed = rows_bytes + (ks > 1 ? (size_t)kSimtThreads * 5 * sizeof(T) + rows_bytes : 0);
    // the bank's share of shared memory with as many CTAs on an SM as the
    // registers allow, or as there are; one fewer where the bank then stays
    int want = (int)max((int64_t)1, min((int64_t)MINB, (tiles + sms - 1) / sms));
    if (want > 2 && nslots * per > kSimtSmem / want - 1024 - fixed && nslots * per <= kSimtSmem / (want - 1) - 1024 - fixed)
        --want;
    const size_t budget = kSimtSmem / want - 1024 - fixed;
    p.resident = nslots * per <= budget;
    p.whole = p.resident && nslots == p.k;
    // A second tile where it costs no CTA of the bank's: with few components the
    // tile's loads are most of a CTA's time.
    p.prefetch = p.resident && tiles > (int64_t)sms * want && nslots * per + rows_bytes <= budget;
    p.chunk = p.resident ? nslots : max(1, (int)(budget / 2 / per));
    p.nslots = nslots;
    p.nchunks = (nslots + p.chunk - 1) / p.chunk;
    const size_t smem = fixed + (p.prefetch ? rows_bytes : 0) + (p.resident ? 1 : 2) * (size_t)p.chunk * per;
    auto kern = mixture_simt_kernel<T, D, FACTOR, S, MINB, DIRECT>;
    if (smem > 46 * 1024) {  // the limit without opting in, less the static part
        const int e = allow_dynamic_smem((const void *)kern);
        if (e) return e;
    }
    const int64_t fit = max((int64_t)1, min((int64_t)16, (int64_t)(kSimtSmem / (smem + 1024))));
    const int blocks = (int)min(tiles, sms * fit);
    kern<<<blocks, kSimtThreads, smem, stream>>>(p);
    note_launch();
    return (int)cudaGetLastError();
}

// FP32 substitution does the padded work beyond d (branches would keep the
// next column's loads from being issued early), so the dimensions come in
// steps of at most a quarter; two samples per thread (half the loads per FMA)
// from the size on where every SM still has two tiles per resident CTA.
template <typename T> static int dispatch_factor(const MixParams<T> &p, cudaStream_t stream) {
    const int d = p.d;
    if constexpr (sizeof(T) == 4) {
        const bool two = p.n >= (int64_t)device_sms() * 4 * 2 * 2 * kSimtThreads;
#define ISSM_PAIR(DD, MIN2, MIN1)                                      \
    if (d <= DD)                                                       \
        return two ? launch_simt<T, DD, true, 2, MIN2>(p, stream)      \
                   : launch_simt<T, DD, true, 1, MIN1>(p, stream);
        ISSM_PAIR(4, 6, 8)
        ISSM_PAIR(8, 5, 6)
        ISSM_PAIR(12, 5, 6)
        ISSM_PAIR(16, 4, 5)
        ISSM_PAIR(24, 3, 4)
        ISSM_PAIR(32, 3, 4)
#undef ISSM_PAIR
        if (d <= 40) return launch_simt<T, 40, true, 1, 4>(p, stream);
        if (d <= 48) return launch_simt<T, 48, true, 1, 3>(p, stream);
        return launch_simt<T, 64, true, 1, 3>(p, stream);
    } else {
        // short FP64 rows straight into registers, but not for draws, which thread groups share
        if (d <= 4)
            return p.mode == kModeDenominator || p.mode == kModeAppend ? launch_simt<T, 4, true, 1, 4, true>(p, stream)
                                                                       : launch_simt<T, 4, true, 1, 4>(p, stream);
        if (d <= 8) return launch_simt<T, 8, true, 1, 4>(p, stream);
        if (d <= 16) return launch_simt<T, 16, true, 1, 4>(p, stream);
        if (d <= 32) return launch_simt<T, 32, true, 1, 4>(p, stream);
        return launch_simt<T, 64, true, 1, 2>(p, stream);
    }
}

template <typename T> int dispatch_simt(const MixParams<T> &p0, cudaStream_t stream) {
    MixParams<T> p = p0;
    const int d = p.d;
    if (d > 64) return ISSM_E_UNSUPPORTED;
    // with one generating slot for every sample only that component counts
    if (p.mode == kModeDenominator && p.den_kind == ISSM_DENOM_GENERATING && p.slots == nullptr)
        p.first_slot = p.last_slot = p.fixed_slot;
    if (p.mode == kModeDraw && (p.scale_kind != ISSM_SCALE_FACTOR || p.slots != nullptr)) {
        const bool factor = p.scale_kind == ISSM_SCALE_FACTOR;
#define ISSM_DRAW(DD) \
    if (d <= DD) return factor ? launch_draw_slots<T, DD, true>(p, stream) : launch_draw_slots<T, DD, false>(p, stream);
        ISSM_DRAW(4)
        ISSM_DRAW(16)
        ISSM_DRAW(32)
        ISSM_DRAW(64)
#undef ISSM_DRAW
    }
    if (p.scale_kind != ISSM_SCALE_FACTOR) {
        constexpr int kMinB = sizeof(T) == 4 ? 8 : 4;
        if (d <= 4) return launch_simt<T, 4, false, 1, kMinB>(p, stream);
        if (d <= 8) return launch_simt<T, 8, false, 1, kMinB>(p, stream);
        if (d <= 16) return launch_simt<T, 16, false, 1, kMinB>(p, stream);
        return launch_simt<T, 64, false, 1, 2>(p, stream);
    }
    if (p.mode == kModeDraw) {
        if (d <= 4) return launch_draw_fixed<T, 4>(p, stream);
        if (d <= 16) return launch_draw_fixed<T, 16>(p, stream);
        if (d <= 32) return launch_draw_fixed<T, 32>(p, stream);
        return launch_draw_fixed<T, 64>(p, stream);
    }
    return dispatch_factor(p, stream);
}

}  // namespace issm
