// Cache maintenance kernels of the PagedAttention operator: writing a chunk's new keys / values
// into their paged slots (with by-token u8 quantisation), re-rotating the keys of listed blocks,
// and block copies for copy-on-write.  All three are byte movers; one warp, or eight lanes where chunks
// are written in groups of tokens, own one (token, kv head) row, so the min/max for the quantiser is a
// handful of shuffles.
#include <algorithm>

#include "pa_common.cuh"
#include "pa_kernels.h"

namespace pa {

namespace {

// Locates the sequence that owns flattened token `t` by binary search in subsequence_begins.
__device__ __forceinline__ int find_sequence(const int32_t* begins, int num_seq, int t) {
    int lo = 0, hi = num_seq;  // begins[lo] <= t < begins[hi]
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (begins[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}

// Number of 32-token context tiles of one decode row (0 for rows that are not decode rows), plus the phantom tiles
// of the slicing sequence where the decode kernel asks for them.
__device__ __forceinline__ int seq_tiles(const KernelArgs& a, int s) {
    SeqView v;
    if (!seq_view(a, s, v) || v.n != 1) return 0;
    return (v.past + 1 + 31) / 32 + a.decode_phantom;
}

// Builds the decode plan with one block of 256 threads: the exclusive prefix sum of the per-row
// tile counts (workers slice the global tile sequence through it) and zeroed per-stream counters.
__device__ void build_decode_plan(const KernelArgs& a) {
    __shared__ int sh_warp[8];
    __shared__ int sh_run;
    __shared__ int sh_warp_p[8];
    __shared__ int sh_run_p;
    constexpr int kPrefixCap = 2048;           // rows whose prefix sums are also kept in shared memory
    __shared__ int sh_prefix[kPrefixCap + 1];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int B = a.num_sequences;
    const int G = a.g.Hq / a.g.Hkv, HK = a.g.Hkv * ((G + 15) / 16);
    if (tid == 0) { sh_run = 0; sh_run_p = 0; }
    __syncthreads();
    for (int base = 0; base < B; base += 256) {
        const int s = base + tid;
        const int n = s < B ? seq_tiles(a, s) : 0;
        // prefill chunks: q tiles of kPrefillItemRows (new token, q head of one group) pairs
        int np = 0;
        if (s < B) {
            SeqView sv;
            if (n == 0 && seq_view(a, s, sv) && sv.n > 1) np = (sv.n * G + kPrefillItemRows - 1) / kPrefillItemRows;
        }
        int v = n, vp = np;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o), up = __shfl_up_sync(0xffffffffu, vp, o);
            if (lane >= o) { v += u; vp += up; }
        }
        if (lane == 31) { sh_warp[wid] = v; sh_warp_p[wid] = vp; }
        __syncthreads();
        int off = sh_run, offp = sh_run_p;
        for (int w = 0; w < wid; ++w) { off += sh_warp[w]; offp += sh_warp_p[w]; }
        if (s < B) {
            a.tile_prefix[s] = off + v - n;
            a.ptile_prefix[s] = offp + vp - np;
            if (s <= kPrefixCap) sh_prefix[s] = off + v - n;
        }
        __syncthreads();
        if (tid == 255) { sh_run = off + v; sh_run_p = offp + vp; }
        __syncthreads();
    }
    for (int i = tid; i < B * HK; i += 256) a.stream_done[i] = 0;
    // start records of the decode workers: the row that holds each slice's first tile
    if (a.worker_start && a.decode_all_workers > 0) {
        const int total_tiles = sh_run * HK;
        if (B <= kPrefixCap) {
            if (tid == 0) sh_prefix[B] = sh_run;
            __syncthreads();
            const DecodeSlices sl = decode_slices(total_tiles, a.decode_all_workers);
            for (int w = tid; w < a.decode_all_workers; w += 256) {
                WorkerStart ws{-1, 0, 0, total_tiles, 0, 0, 0, 0};
                const long long g_tile = sl.begin(w);
                if (w < sl.workers1 && g_tile < sl.end(w)) {
                    const int key = (int)(g_tile / HK);
                    int lo = 0, hi = B;   // sh_prefix[lo] <= key < sh_prefix[hi]
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (sh_prefix[mid] <= key) lo = mid; else hi = mid;
                    }
                    const int tb = a.block_indices_begins[lo];
                    ws = WorkerStart{lo, sh_prefix[lo], sh_prefix[lo + 1] - sh_prefix[lo], total_tiles, a.past_lens[lo] + 1, tb,
                                     a.block_indices_begins[lo + 1] - tb, a.subsequence_begins[lo]};
                } else {
                    ws.s = -2;   // no tiles for this worker
                }
                a.worker_start[w] = ws;
            }
        } else {
            for (int w = tid; w < a.decode_all_workers; w += 256) a.worker_start[w] = WorkerStart{-1, 0, 0, total_tiles, 0, 0, 0, 0};
        }
    }
    // The prefill kernel hands out (q tile, kv head) items from a counter.  Longest context first keeps the last items
    // short, so the CTAs finish together; sequence order leaves a long item for the end.
    const int total_p = sh_run_p;
    const bool sort_items = a.pitem_order != nullptr && total_p > 1 && total_p <= kPrefillSortCap;
    if (sort_items) {
        __shared__ int sh_cost[kPrefillSortCap];
        const bool in_shared = B <= kPrefixCap;
        if (tid == 0) a.ptile_prefix[B] = total_p;
        __syncthreads();   // the prefix sums written above are visible to the whole block
        if (in_shared)
            for (int s = tid; s <= B; s += 256) sh_prefix[s] = a.ptile_prefix[s];   // (the decode prefix there is no longer needed)
        __syncthreads();
        for (int t = tid; t < total_p; t += 256) {
            int lo = 0, hi = B;   // ptile_prefix[lo] <= t < ptile_prefix[hi]
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if ((in_shared ? sh_prefix[mid] : a.ptile_prefix[mid]) <= t) lo = mid; else hi = mid;
            }
            const int p0 = in_shared ? sh_prefix[lo] : a.ptile_prefix[lo], np = (in_shared ? sh_prefix[lo + 1] : a.ptile_prefix[lo + 1]) - p0;
            const int qt = np - 1 - (t - p0);   // the kernel's mapping: late (heavy) q tiles first
            const int n_new = a.subsequence_begins[lo + 1] - a.subsequence_begins[lo];
            const int r_hi = min(n_new * G, (qt + 1) * kPrefillItemRows) - 1;
            sh_cost[t] = a.past_lens[lo] + r_hi / G + 1;   // context of the q tile's last row
        }
        __syncthreads();
        for (int t = tid; t < total_p; t += 256) {
            const int c = sh_cost[t];
            int rank = 0;
            for (int u = 0; u < total_p; ++u) {
                const int cu = sh_cost[u];
                rank += (cu > c || (cu == c && u < t)) ? 1 : 0;
            }
            a.pitem_order[rank] = t;
        }
    }
    if (tid == 0) {
        a.tile_prefix[B] = sh_run;
        a.plan->total_tiles = sh_run * HK;
        a.ptile_prefix[B] = sh_run_p;
        a.plan->total_ptiles = sh_run_p;
        a.plan->next_pitem = 0;
        a.plan->pitems_sorted = sort_items ? 1 : 0;
    }
}

// Eight consecutive activations as they lie in memory, and their values.  The loads are apart from the conversions so that
// those of several pieces are in flight together: with the branch on the type around each load they were not.
template <bool F32>
struct RawAct8 {
    uint4 w[F32 ? 2 : 1];
    __device__ __forceinline__ void load(const void* p, long long i) {   // 16-byte aligned
        const uint4* q = reinterpret_cast<const uint4*>((const uint8_t*)p + i * (F32 ? 4 : 2));
#pragma unroll
        for (int k = 0; k < (F32 ? 2 : 1); ++k) w[k] = q[k];
    }
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int k = 0; k < (F32 ? 2 : 1); ++k) w[k] = make_uint4(0u, 0u, 0u, 0u);
    }
    __device__ __forceinline__ void values(int act, float (&out)[8]) const {
        if constexpr (F32) {
            const uint32_t u[8] = {w[0].x, w[0].y, w[0].z, w[0].w, w[1].x, w[1].y, w[1].z, w[1].w};
#pragma unroll
            for (int e = 0; e < 8; ++e) out[e] = __uint_as_float(u[e]);
        } else {
            const uint32_t u[4] = {w[0].x, w[0].y, w[0].z, w[0].w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const unsigned short b = (unsigned short)(u[e / 2] >> (16 * (e & 1)));
                out[e] = act == PA_DTYPE_F16 ? __half2float(__ushort_as_half(b)) : __bfloat162float(__ushort_as_bfloat16(b));
            }
        }
    }
};

// Cache record (byte offset of (block, head 0)) and slot of flattened token t, or false with the status bit set.
__device__ __forceinline__ bool locate_token(const KernelArgs& a, int t, bool report, long long& rec, int& slot) {
    const int s = find_sequence(a.subsequence_begins, a.num_sequences, t);
    SeqView sv;
    if (!seq_view(a, s, sv)) return false;
    if (t < sv.t0 || t >= sv.t0 + sv.n) {   // prefix sums that are not monotone, or that leave tokens uncovered
        if (report) atomicOr(a.status, PA_DEV_BAD_BEGINS);
        return false;
    }
    const int pos = sv.past + (t - sv.t0);
    const int block = a.block_indices[sv.tb + pos / a.g.bs];
    if (block < 0 || block >= a.num_blocks) {
        if (report) atomicOr(a.status, PA_DEV_BAD_BLOCK_INDEX);
        return false;
    }
    slot = pos % a.g.bs;
    rec = (long long)block * a.g.block_bytes;
    return true;
}

// Chunks: one CTA writes kWriteTokens consecutive tokens of one kv head, eight lanes per token.  A token is located once per
// CTA (a chain of about eight dependent loads) instead of once per head and warp, activations come in 16-byte pieces that
// are all in flight together, the quantiser's divisions are shared by sixteen elements per lane, and the token-minor value
// bytes of the u8 cache are turned around in shared memory and leave as words instead of single bytes.  Bound by the chain
// locate -> load -> quantise -> store and, from some 30 k rows on, by the bytes: 65536 rows (bf16 in, u8 out) 55 -> 26 us.
constexpr int kWriteTokens = 32;
constexpr long long kWriteLightRows = 2048, kWriteChunkRows = 3072;
template <int D, bool F32>
__device__ __forceinline__ void write_group(const KernelArgs& a, int group, int h) {
    constexpr int NP = D / 64;                      // pieces of eight dims per lane: dims 8 l + 64 p
    constexpr int kCols = kWriteTokens + 4, kColWords = kCols / 4;
    __shared__ long long sh_rec[kWriteTokens];      // record of (block, head) or -1
    __shared__ int sh_slot[kWriteTokens];
    __shared__ long long sh_word[kColWords];        // where a word of four columns goes in its record's value data, or -1
    __shared__ __align__(4) uint8_t sh_v[D][kCols]; // value bytes, column = token + slot of the first token mod 4
    const int tid = threadIdx.x;
    const int t0 = group * kWriteTokens, n = min(kWriteTokens, a.num_tokens - t0);
    if (tid < kWriteTokens) {
        long long rec = -1;
        int slot = 0;
        if (tid < n && locate_token(a, t0 + tid, h == 0, rec, slot)) rec += (long long)h * a.g.head_bytes;
        else rec = -1;
        sh_rec[tid] = rec;
        sh_slot[tid] = slot;
    }
    const int i = tid >> 3, l = tid & 7;            // token, lane of the token
    RawAct8<F32> kraw[NP], vraw[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const long long src = ((long long)(t0 + i) * a.g.Hkv + h) * D + 8 * l + 64 * p;
        if (i < n) { kraw[p].load(a.key, src); vraw[p].load(a.value, src); }
        else { kraw[p].zero(); vraw[p].zero(); }
    }
    __syncthreads();
    const long long rec = sh_rec[i];
    const int slot = sh_slot[i];
    if (a.g.cache != PA_DTYPE_U8) {
        if (rec < 0) return;
        const bool same = !F32 && a.g.act == a.g.cache;   // 16-bit activations of the cache's type go in as they are
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
            uint8_t* dst = (uint8_t*)(kv ? a.value_cache : a.key_cache) + rec + (long long)slot * D * 2;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const RawAct8<F32>& raw = kv ? vraw[p] : kraw[p];
                uint4 w = raw.w[0];
                if (!same) {
                    float x[8];
                    raw.values(a.g.act, x);
                    uint32_t o[4];
#pragma unroll
                    for (int e = 0; e < 8; e += 2)
                        o[e / 2] = a.g.cache == PA_DTYPE_F16
                                       ? __half_as_ushort(__float2half_rn(x[e])) | (uint32_t)__half_as_ushort(__float2half_rn(x[e + 1])) << 16
                                       : __bfloat16_as_ushort(__float2bfloat16_rn(x[e])) | (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x[e + 1])) << 16;
                    w = make_uint4(o[0], o[1], o[2], o[3]);
                }
                *reinterpret_cast<uint4*>(dst + (8 * l + 64 * p) * 2) = w;
            }
        }
        return;
    }
    const int shift = sh_slot[0] & 3;
    if (tid < kColWords) {   // a word whose tokens are neighbours in one record is stored as one
        const int i0 = 4 * tid - shift;
        bool whole = i0 >= 0 && i0 + 3 < kWriteTokens;
        if (whole) {
            whole = sh_rec[i0] >= 0 && (sh_slot[i0] & 3) == 0;
            for (int u = 1; u < 4; ++u) whole = whole && sh_rec[i0 + u] == sh_rec[i0] && sh_slot[i0 + u] == sh_slot[i0] + u;
        }
        sh_word[tid] = whole ? sh_rec[i0] + sh_slot[i0] : -1;
    }
#pragma unroll
    for (int kv = 0; kv < 2; ++kv) {
        float x[NP][8];
        float mn = 0.f, mx = 0.f;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            (kv ? vraw[p] : kraw[p]).values(a.g.act, x[p]);
            if (p == 0) { mn = x[0][0]; mx = x[0][0]; }
#pragma unroll
            for (int e = 0; e < 8; ++e) { mn = fminf(mn, x[p][e]); mx = fmaxf(mx, x[p][e]); }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {   // over the token's lanes
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        float sc, zp, inv;
        quant_params(mn, mx, sc, zp, inv);
        uint8_t* data = (uint8_t*)(kv ? a.value_cache : a.key_cache) + (rec < 0 ? 0 : rec);
        if (rec >= 0 && l == 0) {
            float* par = (float*)(data + (long long)a.g.bs * D);
            par[slot] = sc; par[a.g.bs + slot] = zp;
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            if (kv) {
#pragma unroll
                for (int e = 0; e < 8; ++e) sh_v[8 * l + 64 * p + e][i + shift] = (uint8_t)quant_one(x[p][e], inv, zp);
            } else if (rec >= 0) {   // key data [bs][D]
                *reinterpret_cast<uint2*>(data + (long long)slot * D + 8 * l + 64 * p) =
                    make_uint2(quant_four(x[p][0], x[p][1], x[p][2], x[p][3], inv, zp), quant_four(x[p][4], x[p][5], x[p][6], x[p][7], inv, zp));
            }
        }
    }
    __syncthreads();
    uint8_t* vc = (uint8_t*)a.value_cache;   // value data [D][bs]
    for (int w = tid; w < D * kColWords; w += 256) {
        const int d = w / kColWords, g = w % kColWords;
        const long long at = sh_word[g];
        if (at >= 0) {
            *reinterpret_cast<uint32_t*>(vc + at + (long long)d * a.g.bs) = *reinterpret_cast<const uint32_t*>(&sh_v[d][4 * g]);
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = 4 * g + u - shift;
                if (j >= 0 && j < kWriteTokens && sh_rec[j] >= 0) vc[sh_rec[j] + (long long)d * a.g.bs + sh_slot[j]] = sh_v[d][4 * g + u];
            }
        }
    }
}

// One warp per (token, kv head).  Lane l owns dims {l + 32*i}.  With PLAN set, the first block of
// the grid builds the decode plan instead.
template <int D, bool PLAN, bool GROUPS>
__global__ void __launch_bounds__(256) write_kv_kernel(KernelArgs a) {
    constexpr int PER = D / 32;
    grid_wait();
    if (a.release_early) grid_release();
    // The plan blocks come first, so that they run beside the writes of a long chunk and not behind them.
    int first_block = 0;
    if constexpr (PLAN) {
        if (blockIdx.x == 0) {
            build_decode_plan(a);
            return;
        }
        first_block = 1;
        if (a.scores && a.score_aggregation_window) {   // with a score output the second block prepares the score offsets and work list
            if (blockIdx.x == 1) {
                if (threadIdx.x < 32) build_score_plan(a);
                return;
            }
            first_block = 2;
        }
    }
    if constexpr (GROUPS) {
        const int i = blockIdx.x - first_block;
        if (a.g.act == PA_DTYPE_F32) write_group<D, true>(a, i / a.g.Hkv, i % a.g.Hkv);
        else write_group<D, false>(a, i / a.g.Hkv, i % a.g.Hkv);
        return;
    }
    const int warp = ((blockIdx.x - first_block) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int total = a.num_tokens * a.g.Hkv;
    if (warp >= total) return;
    const int t = warp / a.g.Hkv, h = warp % a.g.Hkv;
    long long rec;
    int slot;
    if (!locate_token(a, t, lane == 0, rec, slot)) return;
    rec += (long long)h * a.g.head_bytes;
    const long long src = ((long long)t * a.g.Hkv + h) * D;
    float k[PER], v[PER];
    if (a.g.act == PA_DTYPE_F32) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            k[i] = ((const float*)a.key)[src + lane + 32 * i];
            v[i] = ((const float*)a.value)[src + lane + 32 * i];
        }
    } else {   // all loads in flight before the first conversion
        unsigned short kr[PER], vr[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            kr[i] = ((const unsigned short*)a.key)[src + lane + 32 * i];
            vr[i] = ((const unsigned short*)a.value)[src + lane + 32 * i];
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            k[i] = a.g.act == PA_DTYPE_F16 ? __half2float(__ushort_as_half(kr[i])) : __bfloat162float(__ushort_as_bfloat16(kr[i]));
            v[i] = a.g.act == PA_DTYPE_F16 ? __half2float(__ushort_as_half(vr[i])) : __bfloat162float(__ushort_as_bfloat16(vr[i]));
        }
    }
    if (a.g.cache == PA_DTYPE_U8) {
        uint8_t* kr = (uint8_t*)a.key_cache + rec;
        uint8_t* vr = (uint8_t*)a.value_cache + rec;
        float kmn = k[0], kmx = k[0], vmn = v[0], vmx = v[0];
#pragma unroll
        for (int i = 1; i < PER; ++i) {
            kmn = fminf(kmn, k[i]); kmx = fmaxf(kmx, k[i]);
            vmn = fminf(vmn, v[i]); vmx = fmaxf(vmx, v[i]);
        }
        kmn = warp_min(kmn); kmx = warp_max(kmx); vmn = warp_min(vmn); vmx = warp_max(vmx);
        float ks, kz, ki, vs, vz, vi;
        quant_params(kmn, kmx, ks, kz, ki);
        quant_params(vmn, vmx, vs, vz, vi);
        float* kp = (float*)(kr + (long long)a.g.bs * D);
        float* vp = (float*)(vr + (long long)a.g.bs * D);
        if (lane == 0) {
            kp[slot] = ks; kp[a.g.bs + slot] = kz;
            vp[slot] = vs; vp[a.g.bs + slot] = vz;
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int d = lane + 32 * i;
            kr[(long long)slot * D + d] = (uint8_t)quant_one(k[i], ki, kz);   // key data   [bs][D]
            vr[(long long)d * a.g.bs + slot] = (uint8_t)quant_one(v[i], vi, vz);  // value data [D][bs]
        }
    } else {
        uint16_t* kr = (uint16_t*)((uint8_t*)a.key_cache + rec) + (long long)slot * D;
        uint16_t* vr = (uint16_t*)((uint8_t*)a.value_cache + rec) + (long long)slot * D;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int d = lane + 32 * i;
            if (a.g.cache == PA_DTYPE_F16) {
                kr[d] = __half_as_ushort(__float2half_rn(k[i]));
                vr[d] = __half_as_ushort(__float2half_rn(v[i]));
            } else {
                kr[d] = __bfloat16_as_ushort(__float2bfloat16_rn(k[i]));
                vr[d] = __bfloat16_as_ushort(__float2bfloat16_rn(v[i]));
            }
        }
    }
}

// HALF / EL lanes per (rotated block, kv head, token).  Lane l owns the pairs (j, j + D/2) for
// j in EL*l .. EL*l + EL-1.  k'[j] = fma(-k[j+D/2], s, k[j]*c);  k'[j+D/2] = fma(k[j], s, k[j+D/2]*c)
// with c = lut[row][j], s = lut[row][D/2 + j].  EL = 8: the three divisions of a token's new scale and
// zero-point (every lane of the token computes them) are spread over sixteen elements per lane.
// One CTA per rotated block, 256 / LPT of its (kv head, token) units at a time; a pass's loads are issued before the pass
// before it is worked on.  Bound by instruction issue (81 % of the slots, 332 instructions per warp and pass): 6200 blocks of
// 4 heads x 32 tokens (u8) 115 us, 95 without conversion instructions (quant_bits), 78 with the loads ahead, shifts for the
// divisions by the block size and three-way minima; the keys' bytes, once in and once out, take 33.
__device__ __forceinline__ float min3(float a, float b, float c) {
    float y;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
template <bool U8>
struct RotateRaw {   // a lane's EL elements of both halves, as they lie in memory
    uint2 l, h;
    float sc, zp;
};
template <>
struct RotateRaw<false> {
    uint4 l, h;
};
template <int D, bool U8>
__global__ void __launch_bounds__(256, 4) rotate_kernel(KernelArgs a) {
    constexpr int HALF = D / 2;
    constexpr int EL = 8;                  // pairs per lane: an 8-byte (u8) or 16-byte (f16 / bf16) vector per half
    constexpr int LPT = HALF / EL;         // lanes per token: 8 (D = 128) or 4 (D = 64)
    constexpr int UPP = 256 / LPT;         // units per pass
    grid_wait();
    grid_release();
    const int l = threadIdx.x % LPT;
    const int r = blockIdx.x;
    const int units = a.g.Hkv * a.g.bs;
    const int block = a.rotated_block_indices[r];
    const int row = a.rotation_deltas[r];
    if (block < 0 || block >= a.num_blocks || row < 0 || row >= a.rotation_lut_rows) {   // the same for the whole CTA
        if (threadIdx.x == 0) atomicOr(a.status, PA_DEV_BAD_ROTATION);
        return;
    }
    uint8_t* const base = (uint8_t*)a.key_cache + (long long)block * a.g.block_bytes;
    const int bs_log2 = 31 - __clz(a.g.bs);   // 16 or 32 tokens
    auto record = [&](int unit, int& tok) {
        tok = unit & (a.g.bs - 1);
        return base + (unsigned)(unit >> bs_log2) * (unsigned)a.g.head_bytes;   // (inside one block: 32 bits)
    };
    auto load = [&](int unit) {
        RotateRaw<U8> x;
        int tok;
        const uint8_t* rec = record(min(unit, units - 1), tok);
        if constexpr (U8) {
            const float* params = (const float*)(rec + (long long)a.g.bs * D);
            x.sc = params[tok]; x.zp = params[a.g.bs + tok];
            x.l = *reinterpret_cast<const uint2*>(rec + (long long)tok * D + EL * l);
            x.h = *reinterpret_cast<const uint2*>(rec + (long long)tok * D + HALF + EL * l);
        } else {
            const uint16_t* p = (const uint16_t*)rec + (long long)tok * D;
            x.l = *reinterpret_cast<const uint4*>(p + EL * l);
            x.h = *reinterpret_cast<const uint4*>(p + HALF + EL * l);
        }
        return x;
    };
    RotateRaw<U8> next = load(threadIdx.x / LPT);
    const float* lut = a.rotation_trig_lut + (long long)row * D;
    float cv[EL], sv[EL];
#pragma unroll
    for (int i = 0; i < EL; i += 4) {
        const float4 c4 = *reinterpret_cast<const float4*>(lut + EL * l + i), s4 = *reinterpret_cast<const float4*>(lut + HALF + EL * l + i);
        cv[i] = c4.x; cv[i + 1] = c4.y; cv[i + 2] = c4.z; cv[i + 3] = c4.w;
        sv[i] = s4.x; sv[i + 1] = s4.y; sv[i + 2] = s4.z; sv[i + 3] = s4.w;
    }
    for (int unit = threadIdx.x / LPT; unit - (int)(threadIdx.x / LPT) < units; unit += UPP) {   // the same number of passes for every thread
        const RotateRaw<U8> x = next;
        if (unit - (int)(threadIdx.x / LPT) + UPP < units) next = load(unit + UPP);
        const bool live = unit < units;
        int tok;
        uint8_t* rec = record(min(unit, units - 1), tok);
        float lo[EL], hi[EL], nlo[EL], nhi[EL];
        if constexpr (U8) {
            const uint32_t wl[2] = {x.l.x, x.l.y}, wh[2] = {x.h.x, x.h.y};
#pragma unroll
            for (int i = 0; i < EL; ++i) {
                lo[i] = dequant_byte(wl[i >> 2], i & 3, x.sc, x.zp);
                hi[i] = dequant_byte(wh[i >> 2], i & 3, x.sc, x.zp);
            }
        } else {
            const uint32_t wl[4] = {x.l.x, x.l.y, x.l.z, x.l.w}, wh[4] = {x.h.x, x.h.y, x.h.z, x.h.w};
#pragma unroll
            for (int i = 0; i < EL; ++i) {
                const unsigned short el = (unsigned short)(wl[i >> 1] >> (16 * (i & 1))), eh = (unsigned short)(wh[i >> 1] >> (16 * (i & 1)));
                lo[i] = a.g.cache == PA_DTYPE_F16 ? __half2float(__ushort_as_half(el)) : __bfloat162float(__ushort_as_bfloat16(el));
                hi[i] = a.g.cache == PA_DTYPE_F16 ? __half2float(__ushort_as_half(eh)) : __bfloat162float(__ushort_as_bfloat16(eh));
            }
        }
#pragma unroll
        for (int i = 0; i < EL; ++i) {
            nlo[i] = __fmaf_rn(-hi[i], sv[i], __fmul_rn(lo[i], cv[i]));
            nhi[i] = __fmaf_rn(lo[i], sv[i], __fmul_rn(hi[i], cv[i]));
        }
        if constexpr (U8) {
            float mn = fminf(nlo[0], nhi[0]), mx = fmaxf(nlo[0], nhi[0]);
#pragma unroll
            for (int i = 1; i < EL; ++i) {
                mn = min3(mn, nlo[i], nhi[i]);
                mx = max3(mx, nlo[i], nhi[i]);
            }
#pragma unroll
            for (int o = LPT / 2; o > 0; o >>= 1) {   // over the token's lanes (every lane of the warp takes part)
                mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            float sc, zp, inv;
            quant_params(mn, mx, sc, zp, inv);
            if (live) {
                if (l == 0) {   // (the token's lanes read its parameters one pass ago at the latest)
                    float* params = (float*)(rec + (long long)a.g.bs * D);
                    params[tok] = sc; params[a.g.bs + tok] = zp;
                }
                uint32_t wl[2], wh[2];
#pragma unroll
                for (int i = 0; i < EL; i += 4) {
                    wl[i >> 2] = quant_four(nlo[i], nlo[i + 1], nlo[i + 2], nlo[i + 3], inv, zp);
                    wh[i >> 2] = quant_four(nhi[i], nhi[i + 1], nhi[i + 2], nhi[i + 3], inv, zp);
                }
                *reinterpret_cast<uint2*>(rec + (long long)tok * D + EL * l) = make_uint2(wl[0], wl[1]);
                *reinterpret_cast<uint2*>(rec + (long long)tok * D + HALF + EL * l) = make_uint2(wh[0], wh[1]);
            }
        } else if (live) {
            uint16_t* p = (uint16_t*)rec + (long long)tok * D;
            uint32_t wl[4] = {0, 0, 0, 0}, wh[4] = {0, 0, 0, 0};
#pragma unroll
            for (int i = 0; i < EL; ++i) {
                const bool f16 = a.g.cache == PA_DTYPE_F16;
                const unsigned short el = f16 ? __half_as_ushort(__float2half_rn(nlo[i])) : __bfloat16_as_ushort(__float2bfloat16_rn(nlo[i]));
                const unsigned short eh = f16 ? __half_as_ushort(__float2half_rn(nhi[i])) : __bfloat16_as_ushort(__float2bfloat16_rn(nhi[i]));
                wl[i >> 1] |= (uint32_t)el << (16 * (i & 1));
                wh[i >> 1] |= (uint32_t)eh << (16 * (i & 1));
            }
            *reinterpret_cast<uint4*>(p + EL * l) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
            *reinterpret_cast<uint4*>(p + HALF + EL * l) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
        }
    }
}

// Block copies: grid.x = pair, grid.y = slice of the block.  16-byte vectors.
__global__ void __launch_bounds__(256) copy_blocks_kernel(uint8_t* key_cache, uint8_t* value_cache, long long block_bytes,
                                                          int num_blocks, const int32_t* pairs, uint32_t* status) {
    const int src = pairs[2 * blockIdx.x], dst = pairs[2 * blockIdx.x + 1];
    if (src < 0 || src >= num_blocks || dst < 0 || dst >= num_blocks) {
        if (threadIdx.x == 0 && blockIdx.y == 0) atomicOr(status, PA_DEV_BAD_BLOCK_INDEX);
        return;
    }
    if (src == dst) return;
    const long long vecs = block_bytes / 16;
    const uint4* ks = (const uint4*)(key_cache + (long long)src * block_bytes);
    uint4* kd = (uint4*)(key_cache + (long long)dst * block_bytes);
    const uint4* vs = (const uint4*)(value_cache + (long long)src * block_bytes);
    uint4* vd = (uint4*)(value_cache + (long long)dst * block_bytes);
    for (long long i = (long long)blockIdx.y * blockDim.x + threadIdx.x; i < vecs; i += (long long)gridDim.y * blockDim.x) {
        kd[i] = ks[i];
        vd[i] = vs[i];
    }
}

}  // namespace

cudaError_t launch_write_kv(const KernelArgs& a, cudaStream_t stream, bool with_plan) {
    if (a.num_tokens <= 0 && !with_plan) return cudaSuccess;
    const long long warps = (long long)a.num_tokens * a.g.Hkv;
    const int plan_blocks = (with_plan ? 1 : 0) + (with_plan && a.scores && a.score_aggregation_window ? 1 : 0);
    // Chunks go in groups of 32 tokens once they have enough rows (tokens x kv heads) to give every SM a few.  Decode rows, each in a
    // block of its own, are better off with a warp per row: their u8 value bytes are scattered one by one, 4096 of them by one CTA
    // instead of four.  The line lies where the chunks' gain pays for that (us, warp per row | groups; a 600-token chunk is "600"):
    // u8, 8 kv heads x 128: 2048 18.5 | 10.2, 512 8.4 | 6.2, 250 decode + 1100 16.5 | 12.4, 1000 + 1010 20.6 | 18.6, but 500 + 520
    // 12.4 | 12.8 and 128 + 130 6.6 | 8.3; 4 x 64: 64 + 4 x 256 8.3 | 7.3, but 256 + 280 6.3 | 8.3 and 120 + 2 x 300 6.3 | 7.3.  f32 activations,
    // which every cache type converts, lie the same way (f16 cache, 8 x 128: 250 + 1100 8.3 | 6.3, 128 + 130 4.5 | 5.3).  16-bit
    // activations into 16-bit caches gain from 2048 rows on, decode rows or not (bf16, 8 x 128: 128 + 130 4.9 | 4.5, 1000 + 1010
    // 10.4 | 6.3).
    // The groups' wider loads and stores need activations and caches on 16-byte boundaries.
    const long long chunk_rows = std::max(0LL, (long long)a.num_tokens - a.num_sequences) * a.g.Hkv, decode_rows = (long long)a.num_sequences * a.g.Hkv;
    const bool light = a.g.cache != PA_DTYPE_U8 && a.g.act != PA_DTYPE_F32;
    const bool groups = a.num_tokens >= 2LL * a.num_sequences && (light ? warps >= kWriteLightRows : chunk_rows >= kWriteChunkRows + decode_rows / 2) &&
                        ((reinterpret_cast<uintptr_t>(a.key) | reinterpret_cast<uintptr_t>(a.value) | reinterpret_cast<uintptr_t>(a.key_cache) |
                          reinterpret_cast<uintptr_t>(a.value_cache)) & 15) == 0;
    const long long blocks = groups ? (long long)((a.num_tokens + kWriteTokens - 1) / kWriteTokens) * a.g.Hkv : (warps * 32 + 255) / 256;
    const int grid = (int)blocks + plan_blocks;
    auto launch = [&](auto kernel) { return launch_dependent(kernel, dim3(grid), dim3(256), 0, stream, a); };
    if (a.g.D == 128) {
        if (with_plan) return groups ? launch(write_kv_kernel<128, true, true>) : launch(write_kv_kernel<128, true, false>);
        return groups ? launch(write_kv_kernel<128, false, true>) : launch(write_kv_kernel<128, false, false>);
    }
    if (with_plan) return groups ? launch(write_kv_kernel<64, true, true>) : launch(write_kv_kernel<64, true, false>);
    return groups ? launch(write_kv_kernel<64, false, true>) : launch(write_kv_kernel<64, false, false>);
}

cudaError_t launch_rotate(const KernelArgs& a, cudaStream_t stream) {
    if (a.num_rotated_blocks <= 0) return cudaSuccess;
    const int grid = a.num_rotated_blocks;
    const bool u8 = a.g.cache == PA_DTYPE_U8;
    auto launch = [&](auto kernel) { return launch_dependent(kernel, dim3(grid), dim3(256), 0, stream, a); };
    if (a.g.D == 128) return u8 ? launch(rotate_kernel<128, true>) : launch(rotate_kernel<128, false>);
    return u8 ? launch(rotate_kernel<64, true>) : launch(rotate_kernel<64, false>);
}

cudaError_t launch_copy_blocks(void* key_cache, void* value_cache, long long block_bytes, int num_blocks,
                               const int32_t* pairs, int num_pairs, uint32_t* status, cudaStream_t stream) {
    if (num_pairs <= 0) return cudaSuccess;
    dim3 grid(num_pairs, 8);
    copy_blocks_kernel<<<grid, 256, 0, stream>>>((uint8_t*)key_cache, (uint8_t*)value_cache, block_bytes, num_blocks, pairs, status);
    return cudaGetLastError();
}

}  // namespace pa
