// What the rows of a Sampler step go through before a token is selected, for CTAs of THREADS threads: the log-partition of the raw
// row, the grammar bitmask and the penalties (src/cpp/src/sampling/logit_processor.hpp:28-112 fixes the order).
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "../../include/sampler_b200.h"
#include "sampler_kernels.h"

namespace sampler {
namespace {

template <class T>
__device__ __forceinline__ T shfl_xor_any(T v, int o) {
    static_assert(sizeof(T) % 4 == 0, "word-sized types only");
    union { T t; uint32_t w[sizeof(T) / 4]; } in, out;
    in.t = v;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 4); ++i) out.w[i] = __shfl_xor_sync(0xffffffffu, in.w[i], o);
    return out.t;
}

template <int THREADS, class T, class Op>
__device__ T block_reduce_n(T v, T identity, Op op, T* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, shfl_xor_any(v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    v = lane < (THREADS / 32) ? sh[lane] : identity;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, shfl_xor_any(v, o));
    return v;
}

// Calls fn(value, index) once for every element of a row, in no particular order. 16-byte loads,
// four of them in flight per thread: with one 4-byte load per iteration a pass over the row is bound
// by the latency of that load, not by bandwidth.
template <int THREADS, class F>
__device__ __forceinline__ void for_row(const float* row, long long V, int tid, F&& fn) {
    if ((reinterpret_cast<uintptr_t>(row) & 15) != 0) {
        for (long long i = tid; i < V; i += THREADS) fn(row[i], i);
        return;
    }
    const float4* r4 = reinterpret_cast<const float4*>(row);
    const long long n4 = V >> 2;
    long long i = tid;
    for (; i + 3 * THREADS < n4; i += 4 * THREADS) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = r4[i + u * THREADS];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long e = 4 * (i + u * THREADS);
            fn(v[u].x, e); fn(v[u].y, e + 1); fn(v[u].z, e + 2); fn(v[u].w, e + 3);
        }
    }
    for (; i < n4; i += THREADS) {
        const float4 v = r4[i];
        fn(v.x, 4 * i); fn(v.y, 4 * i + 1); fn(v.z, 4 * i + 2); fn(v.w, 4 * i + 3);
    }
    for (long long j = 4 * n4 + tid; j < V; j += THREADS) fn(row[j], j);
}

__device__ void apply_history(float* row, long long V, const sampler_row_params& p, const int32_t* ids, const uint32_t* meta,
                              long long n, uint32_t* status, float* raw_out) {
    const double rep = (double)p.repetition_penalty, pres = (double)p.presence_penalty, freq = (double)p.frequency_penalty;
    for (long long i = threadIdx.x; i < n; i += blockDim.x) {
        const int id = ids[i];
        const uint32_t m = meta[i];
        if (id < 0 || id >= V) {
            atomicOr(status, 1u);
            continue;
        }
        float v = row[id];
        if (raw_out) raw_out[i] = v;   // the raw logit, for rows that report raw log-probabilities
        if (m & SAMPLER_HIST_STOP_MASK) v = -CUDART_INF_F;
        if (p.repetition_penalty != 1.0f && (m & (SAMPLER_HIST_IN_PROMPT | SAMPLER_HIST_GENERATED)))
            v = v >= 0 ? (float)__ddiv_rn((double)v, rep) : (float)__dmul_rn((double)v, rep);
        if (m & SAMPLER_HIST_GENERATED) {
            if (p.presence_penalty != 0.0f) v = v >= 0 ? (float)__dsub_rn((double)v, pres) : (float)__dadd_rn((double)v, pres);
            if (p.frequency_penalty != 0.0f) {
                const double t = __dmul_rn(freq, (double)(m >> 3));
                v = v >= 0 ? (float)__dsub_rn((double)v, t) : (float)__dadd_rn((double)v, t);
            }
        }
        row[id] = v;
    }
}

// History entries of row r.
struct RowHistory {
    long long begin, end;
};
__device__ __forceinline__ RowHistory row_history(const StepArgs& a, int r) {
    return a.hist_offsets ? RowHistory{a.hist_offsets[r], a.hist_offsets[r + 1]} : RowHistory{0, 0};
}

// Log-partition of the raw row (FullVocabLogSumExpTransform, logit_transformers.hpp:264-277).  The reference adds the exponentials in
// single precision in index order; here they are added in double precision in parallel and rounded once, which is within an ulp
// or two of any float order.  *ok: the raw logits of the history entries can be kept (else status bit 2).
template <int THREADS>
__device__ float raw_log_partition(const StepArgs& a, const float* row, RowHistory h, float* buf_f, double* buf_d, bool* ok) {
    const int tid = threadIdx.x;
    float mx = -CUDART_INF_F;
    for_row<THREADS>(row, a.vocab, tid, [&](float x, long long) { mx = fmaxf(mx, x); });
    mx = block_reduce_n<THREADS>(mx, -CUDART_INF_F, [](float x, float y) { return fmaxf(x, y); }, buf_f);
    double s = 0.0;
    for_row<THREADS>(row, a.vocab, tid, [&](float x, long long) { s += (double)expf(x - mx); });
    s = block_reduce_n<THREADS>(s, 0.0, [](double x, double y) { return x + y; }, buf_d);
    *ok = !(h.end > h.begin && !a.hist_raw);
    if (!*ok && tid == 0) atomicOr(a.status, 4u);
    return logf((float)s) + mx;
}
// The raw log-probability of the selected token: its logit before the penalties minus the log-partition.
__device__ __forceinline__ float raw_log_prob(const StepArgs& a, const float* row, RowHistory h, long long idx, float raw_lse, bool ok) {
    if (!ok) return CUDART_NAN_F;
    float raw = row[idx];
    for (long long i = h.begin; i < h.end; ++i)
        if (a.hist_ids[i] == idx) { raw = a.hist_raw[i]; break; }
    return raw - raw_lse;
}

// Grammar bitmask (logit_processor.hpp:52-57: after the stop-token mask, before the penalties; both only write -inf, so their order
// does not show), then the penalties, in place.
template <int THREADS>
__device__ void mask_and_penalise(const StepArgs& a, float* row, const sampler_row_params& p, int r, RowHistory h, bool keep_raw) {
    const long long V = a.vocab;
    const int mi = a.bitmask_index ? a.bitmask_index[r] : -1;
    if (mi >= 0) {
        const uint32_t* mask = reinterpret_cast<const uint32_t*>(a.token_bitmasks) + (long long)mi * a.bitmask_words;
        for (long long w = threadIdx.x; w < a.bitmask_words; w += THREADS) {
            uint32_t denied = ~mask[w];
            if (w == a.bitmask_words - 1 && (V & 31)) denied &= (1u << (V & 31)) - 1u;   // bits beyond the vocabulary
            while (denied) {
                const int b = __ffs(denied) - 1;
                denied &= denied - 1;
                row[32 * w + b] = -CUDART_INF_F;
            }
        }
        __syncthreads();
    }
    if (h.end > h.begin)
        apply_history(row, V, p, a.hist_ids + h.begin, a.hist_meta + h.begin, h.end - h.begin, a.status, keep_raw ? a.hist_raw + h.begin : nullptr);
    __syncthreads();
}

// Multinomial over the whole vocabulary: the rows of sampler_exact_kernel.
__device__ __forceinline__ bool whole_vocabulary_row(const sampler_row_params& p, long long V) {
    return (p.do_sample & SAMPLER_ROW_MULTINOMIAL) && !(p.top_k > 0 && p.top_k < 0x7fffffffffffffffLL && p.top_k < V);
}

}  // namespace
}  // namespace sampler
