// Multinomial rows over the full vocabulary (no active top-k), bit for bit as the reference computes
// them on the host:
//   TemperatureLogitTransform   src/cpp/src/sampling/logit_transformers.hpp:299-362
//       p_i = expf((x_i - max) * (1 / T)), sum in index order in single precision, p_i /= sum
//   MinPFilter                  logit_transformers.hpp:157-190   (keep p_i >= float(min_p) * p_max)
//   TopPFilter                  logit_transformers.hpp:94-139    (sort descending, add until the float sum > top_p)
//   Sampler::_multinomial_sample  src/cpp/src/sampling/sampler.cpp:1036-1089
//       total = sum of the kept probabilities in their order, r = total * u, first running sum > r
// Every float the reference produces on the way is reproduced: expf with the host libm's bits and the
// sequential float sums through the step algebra of fsum_exact.cuh, so token ids agree with the
// reference except where several kept elements have exactly the same probability and the draw falls
// among them (their relative order after std::sort is not defined; the lowest index comes first here).
//
// One CTA of 1024 threads per SM works on one row at a time:
//   1. maximum, and the mass of every 256 elements from approximate exponentials;
//   2. exponentials into a scratch row, the amounts that ordered_sum adds and, for top-p, the counts of 2048 bins of their
//      bit patterns (128 per binade);
//   3. the rest of the index-order sum of the exponentials (ordered_sum);
//   4. without top-p the same for the probabilities, the exact sum before every 256 elements kept for the draws;
//      with top-p the elements of the highest bins are brought into shared memory bin by bin (one atomic gives a place)
//      and ordered_sum runs over them in segments of whole bins until the sum exceeds top_p;
//   5. a draw looks its segment up in the recorded sums and adds that segment's elements one by one; with top-p a pass over the row, or the
//      list that a row with several draws makes, gives the element's index.
//
// ordered_sum: while a float sum s stays in one binade, adding x to it is adding a whole number of ulps that depends on s
// through its parity only, and not even on that unless x lies half-way between two.  So a lane adds its eight elements with
// real float additions to the two sums 2^e and 2^e + ulp, which gives its amounts for an even and an odd s for two
// additions per element; without a half-way case the amounts of a segment add up as integers in any order - the
// elements of a bin need not be sorted -, with one the segment is sorted and its lanes' amounts are composed in order.  The
// binade of every segment is guessed from the masses (near a change of binade: both) and checked by the walk of one warp over
// the segments.  Where the sum changes binade the lanes' amounts tell the lane, whose elements are added one by one; a segment
// whose guess was wrong, or in which the sum goes through binades, is added one by one.  (The rules: segment_sum.cuh.)
//
// 128 rows x 128256 of N(0, 4), top-p 0.95 (46 k kept): 417 - 436 -> 195 - 222 us a step (by box); 200 rows x 151936, a quarter each greedy, top-k, top-p and
// plain: 495 -> 160.  Before, one thread walked the bins and lists of sorted elements (most of the 400 - 500 k cycles of a top-p row's
// sorted part), and the CTA rescanned spans with half-way cases (100 k of the index-order sum).  A top-p row's cycles now: 1. 38 k (HBM);
// 2. 72 k (instruction issue); 3. 30 k (the walk, latency); 4. 130 k (ranks of the bins 8, gather 39, probabilities 12, amounts 40, walk 30);
// 5. 27 k (a pass over the row to find the element's index 21).  Some registers spill (64 for each of 1024 threads: 1.1 % of the instructions
// are loads from local memory).
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/sampler_b200.h"
#include "sampler_kernels.h"
#include "sampler_rows.cuh"
#include "segment_sum.cuh"

namespace sampler {

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kBlock = 256;           // consecutive elements a warp takes at a time, eight per lane
constexpr int kMaxSegs = 640;         // segments of a row in index order; longer rows have segments of several blocks
constexpr int kFusedBlocks = 4;       // segments of more (rows of more than 655360 elements) are summed in passes of their own
constexpr int kBigSegs = 4;           // a bin of so many segments' elements is a segment by itself
constexpr int kSegCap = kMaxSegs + 2 * kMaxSegs / kBigSegs + 192;   // in descending order: those, two boundaries per such bin, some per level
constexpr int kBins = 2048;
constexpr int kBinsPerThread = kBins / kThreads;
constexpr int kTopShift = 16;         // first level: 2^16 bit patterns per bin, 128 bins per binade, 16 binades
constexpr int kFinerBy = 5;           // bits a level is cut finer by where a bin is too full to be sorted
constexpr int kCap = 46592;           // elements of a chunk in shared memory
constexpr int kListed = 4096;         // elements that a row with several draws lists with their indices
constexpr int kSlots = 32;            // segments with the amounts of their lanes at hand, for those in which the sum may change binade
constexpr int kTwice = 220;           // further ones whose amounts are taken for two binades (of a chunk; of a row in memory: all)
constexpr uint8_t kInKeys = 255;
static_assert(kSlots + kTwice < kInKeys, "slot numbers");
constexpr int kMaxMisses = 10;        // segments with a wrong guess before the guesses of those behind are made anew (each is added one by one, 3 k
                                      // cycles; a new pass over a row takes 35 k)
using fsx::kEmpty, fsx::kMargin, fsx::kNoGuess;
constexpr float kDrawMargin = 1.0f / 256;   // relative margin around the approximate sums within which an element may be drawn
constexpr uint32_t kOneBits = 0x3f800000u;

// -DSAMPLER_EXACT_PROF: cycles per part of a row, printed by some of the CTAs
enum { kProfMax, kProfExp, kProfGuess, kProfSteps, kProfWalk, kProfMisses, kProfRank, kProfGather, kProfSame, kProfPlace, kProfFind, kProfIndex, kProfIndex2, kProfOther, kProfTile, kProfTiles, kProfSlot, kProfSlots, kProfSerial, kProfN };
#ifdef SAMPLER_EXACT_PROF
#define PROF_BEGIN long long prof_t0 = clock64()
#define PROF_END(slot) do { if (threadIdx.x == 0) sh.prof[slot] += clock64() - prof_t0; prof_t0 = clock64(); } while (0)
#define PROF_COUNT(slot) do { if (threadIdx.x == 0) ++sh.prof[slot]; } while (0)
#else
#define PROF_BEGIN
#define PROF_END(slot)
#define PROF_COUNT(slot)
#endif

struct ExactShared {
    alignas(16) float keys[kCap];        // a chunk's probabilities, bin by bin
    alignas(16) uint32_t bins[kBins];    // counts, then the rank of a bin's first element in its level, then (taken bins) of its end
    uint32_t start[kSegCap + 1];         // first element of a segment; the next one's start is its end
    float cum[kSegCap + 1];              // approximate sum before a segment
    float state[kSegCap];                // exact sum before a segment
    uint32_t step[kSegCap];              // amounts of a segment's elements for an even and an odd sum (pack_amounts)
    uint8_t E[kSegCap];                  // binade the sum is taken to lie in
    uint8_t sorted[kSegCap];             // 1: the elements are in descending order, 2: they are to be brought into it
    uint8_t slot[kSegCap];               // 1 + its place in `upto` and `from`, or 1 + kSlots + its place in step_up; kInKeys; 0: none
    uint32_t step_up[kTwice];            // amounts of such segments under E + 1
    uint16_t bin[kSegCap + 1];           // the segment's first bin
    uint16_t tile[kSegCap / 2];          // runs of segments that the walk took as a whole: the first, and 2^11 times the others' number
    int tiles;
    uint32_t upto[kSlots][32];           // amounts of the segment's lanes up to this one under E (pack_amounts)
    uint32_t from[kSlots][32];           // ... from this one on under E + 1
    alignas(16) float serial[kBlock];    // elements the walking warp adds one by one
    uint32_t queue[kWarps];              // rows of this CTA among the kThreads rows looked at, a bit each
    int stop;                            // first segment of a chunk that is too large to be sorted
    int count;
    uint32_t scan_u[kWarps];
    float scan_f[kWarps];
    double scan_d[kWarps];
    int red_i[kWarps];
    // results of the walking warp
    float bc_s;
    int bc_seg;
    long long bc_hit;
    float bc_p;
#ifdef SAMPLER_EXACT_PROF
    long long prof[kProfN];
#endif
};
static_assert(sizeof(ExactShared) <= 232448, "shared memory of a CTA");
static_assert(kSlots * kBlock + kSegCap <= kCap && 3 * kListed <= kCap, "room in keys");
extern __shared__ __align__(16) uint8_t sx_smem[];
// (by its name and not by an argument: the compiler then knows that it is shared memory)
__device__ __forceinline__ ExactShared& shared_memory() { return *reinterpret_cast<ExactShared*>(sx_smem); }

// ---- reductions and scans over the CTA ------------------------------------------------------------------
template <class T, class Op>
__device__ T block_reduce(T v, Op op, T* buf) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) buf[w] = v;
    __syncthreads();
    v = buf[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <class T>
__device__ T block_sum(T v, T* buf) { return block_reduce(v, [](T a, T b) { return a + b; }, buf); }

// combination of the earlier threads' values (of the identity T(0) for the first); *total: of all
template <class T, class Op>
__device__ T block_scan_exclusive(T v, T* buf, T* total, Op op) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl = op(up, incl);
    }
    __syncthreads();
    if (lane == 31) buf[w] = incl;
    __syncthreads();
    T t = buf[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T up = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t = op(up, t);
    }
    if (total) *total = __shfl_sync(0xffffffffu, t, 31);
    const T before = __shfl_sync(0xffffffffu, t, w > 0 ? w - 1 : 0);
    const T own = __shfl_up_sync(0xffffffffu, incl, 1);
    return op(w > 0 ? before : T(0), lane > 0 ? own : T(0));
}
template <class T>
__device__ T block_scan_exclusive(T v, T* buf, T* total) { return block_scan_exclusive(v, buf, total, [](T a, T b) { return a + b; }); }

// ---- sums in a fixed order ---------------------------------------------------------------------------------
struct Segs {
    int shift;   // 2^shift elements per segment, kBlock at least
    int count;   // segments of the row in index order
    __device__ uint32_t len() const { return 1u << shift; }
};
__device__ __forceinline__ Segs segments_of(uint32_t end) {
    int shift = 8;
    while (((end - 1) >> shift) >= (uint32_t)kMaxSegs) ++shift;
    return Segs{shift, (int)((end + (1u << shift) - 1) >> shift)};
}

// Eight elements from i on (a multiple of eight), those outside lo .. hi - 1 as zero, which leaves a sum as it is.
__device__ __forceinline__ void load8(const float* v, uint32_t i, uint32_t lo, uint32_t hi, float (&x)[8]) {
    if (i >= lo && i + 8 <= hi) {
        const float4 a = *reinterpret_cast<const float4*>(v + i), b = *reinterpret_cast<const float4*>(v + i + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = i + e >= lo && i + e < hi ? v[i + e] : 0.f;
    }
}

// The probability of an exponential (norm > 0): logit_transformers.hpp:357-359
__device__ __forceinline__ float probability(float e, float norm, float inv_norm) { return e == 0.f ? 0.f : fsx::div_shared(e, norm, inv_norm); }

// What is added: element `i` of the row is v[i - off]; elements that are not in the sum count as zero.
struct Exponentials {
    const float* v;
    uint32_t off;
    static constexpr bool kSortable = false, kThreshold = false;
    __device__ __forceinline__ const float* data() const { return v; }
    __device__ __forceinline__ void prepare(float (&x)[8]) const {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = fmaxf(x[e], 0.f);   // NaN: not in the sum
    }
};
struct Probabilities {
    const float* v;
    uint32_t off;
    float norm, inv_norm, min_thr;
    static constexpr bool kSortable = false, kThreshold = true;   // some elements may count as zero
    __device__ __forceinline__ const float* data() const { return v; }
    __device__ __forceinline__ void prepare(float (&x)[8]) const {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float p = probability(x[e], norm, inv_norm);
            x[e] = p >= min_thr ? p : 0.f;
        }
    }
};
struct Chunk {   // probabilities in shared memory (keys), and the row that they also are in
    uint32_t off;
    float* out;
    static constexpr bool kSortable = true, kThreshold = false;
    __device__ __forceinline__ const float* data() const { return shared_memory().keys; }
    __device__ __forceinline__ void prepare(float (&)[8]) const {}
};
struct Sorted {
    const float* v;
    uint32_t off;
    static constexpr bool kSortable = false, kThreshold = false;
    __device__ __forceinline__ const float* data() const { return v; }
    __device__ __forceinline__ void prepare(float (&)[8]) const {}
};

// Masses in cum[0 .. n - 1] -> sums before the segments.
__device__ void masses_to_sums(int n) {
    ExactShared& sh = shared_memory();
    constexpr int kPer = (kMaxSegs + kThreads - 1) / kThreads;
    const int j0 = (int)threadIdx.x * kPer;
    __syncthreads();
    float m[kPer], sum = 0.f;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        m[k] = j0 + k < n ? sh.cum[j0 + k] : 0.f;
        sum += m[k];
    }
    float all, before = block_scan_exclusive(sum, sh.scan_f, &all);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        if (j0 + k < n) sh.cum[j0 + k] = before;
        before += m[k];
    }
    if (threadIdx.x == 0) sh.cum[n] = all;
    __syncthreads();
}

// Sorts a[0 .. n) in descending order (one warp; no value is negative): bitonic merges in the form whose comparators all point the
// same way.  Up to 512 values lie in registers, sixteen consecutive ones per lane; longer segments are sorted in place, entries
// beyond n left out.
__device__ __forceinline__ void order(float& x, float& y) {
    const float a = x, b = y;
    x = fmaxf(a, b);
    y = fminf(a, b);
}
__device__ __noinline__ void sort_segment(float* a, int n) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if (n <= 512) {
        float v[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = 16 * lane + r < n ? a[16 * lane + r] : -1.f;
#pragma unroll
        for (int k = 1; k <= 4; ++k) {   // within a lane
#pragma unroll
            for (int r = 0; r < 16; ++r)
                if ((r ^ ((1 << k) - 1)) > r) order(v[r], v[r ^ ((1 << k) - 1)]);
#pragma unroll
            for (int j = k - 2; j >= 0; --j)
#pragma unroll
                for (int r = 0; r < 16; ++r)
                    if ((r ^ (1 << j)) > r) order(v[r], v[r ^ (1 << j)]);
        }
#pragma unroll 1
        for (int k = 5; k <= 9; ++k) {
            const int mask = (1 << (k - 4)) - 1;
            bool upper = (lane >> (k - 5)) & 1;
            float w[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) w[r] = __shfl_xor_sync(0xffffffffu, v[15 - r], mask);
#pragma unroll
            for (int r = 0; r < 16; ++r) v[r] = upper ? fminf(v[r], w[r]) : fmaxf(v[r], w[r]);
#pragma unroll 1
            for (int j = k - 6; j >= 0; --j) {
                upper = (lane >> j) & 1;
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    const float u = __shfl_xor_sync(0xffffffffu, v[r], 1 << j);
                    v[r] = upper ? fminf(v[r], u) : fmaxf(v[r], u);
                }
            }
#pragma unroll
            for (int j = 3; j >= 0; --j)
#pragma unroll
                for (int r = 0; r < 16; ++r)
                    if ((r ^ (1 << j)) > r) order(v[r], v[r ^ (1 << j)]);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 16; ++r)
            if (16 * lane + r < n) a[16 * lane + r] = v[r];
        __syncwarp();
        return;
    }
    int bits = 1;
    while ((1 << bits) < n) ++bits;
    const int half = 1 << (bits - 1);
    auto exchange = [&](int i, int l) {
        if (l >= n) return;
        const float x = a[i], y = a[l];
        if (x < y) { a[i] = y; a[l] = x; }
    };
    for (int k = 1; k <= bits; ++k) {
        for (int t = lane; t < half; t += 32) {
            const int block = (t >> (k - 1)) << k, at = t & ((1 << (k - 1)) - 1);
            exchange(block + at, block + (1 << k) - 1 - at);
        }
        __syncwarp();
        for (int j = k - 2; j >= 0; --j) {
            for (int t = lane; t < half; t += 32) {
                const int i = ((t >> j) << (j + 1)) + (t & ((1 << j) - 1));
                exchange(i, i + (1 << j));
            }
            __syncwarp();
        }
    }
}
// Segment j of a chunk in shared memory, there and in the row in descending order (one warp).
__device__ __forceinline__ void sort_in_chunk(Chunk src, int j) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31;
    const uint32_t lo = sh.start[j] - src.off, hi = sh.start[j + 1] - src.off;
    sort_segment(sh.keys + lo, (int)(hi - lo));
    for (uint32_t i = lo + lane; i < hi; i += 32) src.out[src.off + i] = sh.keys[i];
    __syncwarp();
    if (lane == 0) sh.sorted[j] = 1;
    __syncwarp();
}

// Guesses the binade of the sum at the segments c .. c1 - 1 from the approximate sums and the exact one, s, before c.  Where the sum may
// change binade, or may have, the amounts are taken for two; the first of the former also get a slot each.  Segments of
// unsorted elements in which the order will matter are marked: those, and where the sum may pass one of two thresholds.
// `rows`: the elements are a row's in memory, and `keys` has room for every segment's second amounts.
__device__ void guess_binades(int c, int c1, float s, float thr, float thr2, bool rows) {
    ExactShared& sh = shared_memory();
    __syncthreads();
    const float shift = s - sh.cum[c];
    uint32_t slots = 0, twice = 0;
    for (int base = c; base < c1; base += kThreads) {
        const int j = base + (int)threadIdx.x;
        bool edge = false, twofold = false;
        uint32_t alone = 0;
        if (j < c1) {
            const float lo = j == c ? s : sh.cum[j] + shift, hi = sh.cum[j + 1] + shift;
            const fsx::Guess g = fsx::guess_binade(lo, hi, sh.start[j] == sh.start[j + 1]);
            edge = g.edge;
            twofold = g.two;
            alone = g.alone;
            sh.E[j] = (uint8_t)g.E;
            if (sh.sorted[j] == 0 && (j == 0 || g.changes || (lo * (1.f - kMargin) <= thr && thr <= hi * (1.f + kMargin)) ||
                                      (lo * (1.f - kDrawMargin) <= thr2 && thr2 <= hi * (1.f + kDrawMargin))))
                sh.sorted[j] = 2;
        }
        uint32_t n;
        const uint32_t before = block_scan_exclusive((edge ? 1u : 0u) | (twofold ? 65536u : 0u), sh.scan_u, &n);
        if (j < c1) {
            const uint32_t at = slots + (before & 0xffffu), at2 = twice + (before >> 16);
            const bool lanes = edge && at < (uint32_t)kSlots, two = twofold && (rows || at2 < (uint32_t)kTwice);
            sh.slot[j] = lanes ? (uint8_t)(at + 1) : !two ? 0 : rows ? kInKeys : (uint8_t)(at2 + 1 + kSlots);
            if (twofold && !lanes && !two) sh.E[j] = (uint8_t)alone;
        }
        slots += n & 0xffffu;
        twice += n >> 16;
    }
    __syncthreads();
}
// Where a segment's amounts under E + 1 are (its slot holds none for the lanes).
__device__ __forceinline__ uint32_t& step_up(int slot, int j) {
    ExactShared& sh = shared_memory();
    return slot == kInKeys ? reinterpret_cast<uint32_t*>(sh.keys)[kSlots * kBlock + j] : sh.step_up[slot - 1 - kSlots];
}

using fsx::pack_amounts, fsx::unpack_amounts;

// The amounts of a warp's 256 elements under binade E, the same on all lanes; *tie (the same too): they depend on the order, and only lane 0
// has those of all elements.
__device__ __forceinline__ fsx::Step block_step(const float (&x)[8], uint32_t E, bool in_order, bool* tie) {
    fsx::Sums sums = fsx::sums_begin(E);
#pragma unroll
    for (int e = 0; e < 8; ++e) fsx::sums_add(sums, x[e]);
    fsx::Step st = fsx::sums_amounts(sums, E);
    *tie = __any_sync(0xffffffffu, st.a != st.b);
    if (!*tie) {
        st.a = st.b = min(__reduce_add_sync(0xffffffffu, st.a), fsx::kSat);   // 32 x kSat at most
    } else if (in_order) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {   // lane 0: all lanes in order
            const fsx::Step next{__shfl_down_sync(0xffffffffu, st.a, o), __shfl_down_sync(0xffffffffu, st.b, o)};
            st = fsx::then(st, next);
        }
    }
    return st;
}

// Does the slot hold the amounts of the segment's lanes (else: those of the whole segment under the next binade)?
__device__ __forceinline__ bool lanes_at_hand(int slot) { return slot != 0 && slot <= kSlots; }

// A segment with a slot: the amounts of its lanes, each of which takes m * 8 consecutive elements, under E up to every lane and under
// E + 1 from every lane on.  Elements of rows in memory stay at hand in `keys`, which nothing else uses then (m = 1).  Out of line: a few segments
// of a row come here, and without its instructions the passes are 2 - 3 us shorter.
template <class Src>
__device__ __noinline__ void lane_steps(Src src, int j) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31, slot = sh.slot[j] - 1;
    const uint32_t lo = sh.start[j] - src.off, hi = sh.start[j + 1] - src.off, lo8 = lo & ~7u, m = (hi - lo8 + kBlock - 1) / kBlock;
    const uint32_t E = sh.E[j];
    fsx::Sums here = fsx::sums_begin(E), above = fsx::sums_begin(E + 1u);
    for (uint32_t t = 0; t < m; ++t) {
        float x[8];
        load8(src.data(), lo8 + 8 * (lane * m + t), lo, hi, x);
        src.prepare(x);
        if (!Src::kSortable && m == 1) {
            *reinterpret_cast<float4*>(sh.keys + slot * kBlock + 8 * lane) = make_float4(x[0], x[1], x[2], x[3]);
            *reinterpret_cast<float4*>(sh.keys + slot * kBlock + 8 * lane + 4) = make_float4(x[4], x[5], x[6], x[7]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            fsx::sums_add(here, x[e]);
            fsx::sums_add(above, x[e]);
        }
    }
    fsx::Step p = fsx::sums_amounts(here, E), q = fsx::sums_amounts(above, E + 1u);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const fsx::Step pu{__shfl_up_sync(0xffffffffu, p.a, o), __shfl_up_sync(0xffffffffu, p.b, o)};
        const fsx::Step qd{__shfl_down_sync(0xffffffffu, q.a, o), __shfl_down_sync(0xffffffffu, q.b, o)};
        if (lane >= o) p = fsx::then(pu, p);
        if (lane + o < 32) q = fsx::then(q, qd);
    }
    sh.upto[slot][lane] = pack_amounts(p);
    sh.from[slot][lane] = pack_amounts(q);
    if (lane == 31) sh.step[j] = pack_amounts(p);
    __syncwarp();
}

// Amounts of the segments' elements under the guesses: rows in memory, a block of each of two segments at a time (a warp's loads are
// what it waits for: one block at a time 23 k cycles for 152 k elements).
template <class Src>
__device__ __forceinline__ void segment_steps(Src src, int c, int c1) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kAtOnce = 2;
    for (int j = c + warp; j < c1; j += kAtOnce * kWarps) {
        uint32_t lo[kAtOnce], hi[kAtOnce];
        fsx::Step total[kAtOnce];
        bool more = false;
#pragma unroll
        for (int u = 0; u < kAtOnce; ++u) {
            const bool in = j + u * kWarps < c1;
            lo[u] = in ? sh.start[j + u * kWarps] - src.off : 0u;
            hi[u] = in ? sh.start[j + u * kWarps + 1] - src.off : 0u;
            total[u] = fsx::step_identity();
            more |= lo[u] < hi[u];
        }
        for (uint32_t at = 0; more; at += kBlock) {
            float x[kAtOnce][8];
            more = false;
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u) {
                const uint32_t i = (lo[u] & ~7u) + at;
                load8(src.data(), i + 8 * lane, lo[u], hi[u], x[u]);
                more |= i + kBlock < hi[u];
            }
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u) {
                const uint32_t E = j + u * kWarps < c1 ? sh.E[j + u * kWarps] : kNoGuess;
                if (E == kNoGuess || E == kEmpty) continue;
                src.prepare(x[u]);
                bool tie;
                total[u] = fsx::then(total[u], block_step(x[u], E, true, &tie));
                const int slot = sh.slot[j + u * kWarps];
                if (slot > kSlots) {
                    const fsx::Step up = block_step(x[u], E + 1u, true, &tie);
                    if (lane == 0) step_up(slot, j + u * kWarps) = pack_amounts(at ? fsx::then(unpack_amounts(step_up(slot, j + u * kWarps)), up) : up);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kAtOnce; ++u)
            if (j + u * kWarps < c1) {
                if (lane == 0) sh.step[j + u * kWarps] = pack_amounts(total[u]);
                if (lanes_at_hand(sh.slot[j + u * kWarps])) lane_steps(src, j + u * kWarps);
            }
    }
    __syncthreads();
}
// A chunk in shared memory: a segment is sorted only where the order matters.
__device__ void segment_steps(Chunk src, int c, int c1) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int j = c + warp; j < c1; j += kWarps) {
        const uint32_t E = sh.E[j];
        if (sh.sorted[j] == 2) sort_in_chunk(src, j);
        if (E == kNoGuess || E == kEmpty) continue;
        const int slot = sh.slot[j];
        if (lanes_at_hand(slot)) { lane_steps(src, j); continue; }   // (sorted now)
        const uint32_t lo = sh.start[j] - src.off, hi = sh.start[j + 1] - src.off;
        for (bool again = true; again;) {
            const bool in_order = sh.sorted[j] == 1;
            fsx::Step total = fsx::step_identity(), total_up = fsx::step_identity();
            again = false;
            for (uint32_t i = lo & ~7u; i < hi && !again; i += kBlock) {
                float x[8];
                load8(src.data(), i + 8 * lane, lo, hi, x);
                bool tie, tie_up = false;
                total = fsx::then(total, block_step(x, E, in_order, &tie));
                if (slot) total_up = fsx::then(total_up, block_step(x, E + 1u, in_order, &tie_up));
                again = (tie || tie_up) && !in_order;
            }
            if (!again && slot && lane == 0) step_up(slot, j) = pack_amounts(total_up);
            if (again) sort_in_chunk(src, j);
            else if (lane == 0) sh.step[j] = pack_amounts(total);
        }
    }
    __syncthreads();
}

// Adds segment j to s element by element (one warp).  It stops at the first running sum above thr and returns that
// element (its value in p), else -1.
template <class Src>
__device__ __forceinline__ long long add_segment(Src src, int j, float& s, float thr, float& p) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31;
    const uint32_t lo = sh.start[j] - src.off, hi = sh.start[j + 1] - src.off;
    float4* buf = reinterpret_cast<float4*>(sh.serial);
    for (uint32_t i = lo & ~7u; i < hi; i += kBlock) {
        float x[8];
        load8(src.data(), i + 8 * lane, lo, hi, x);
        src.prepare(x);
        __syncwarp();
        buf[2 * lane] = make_float4(x[0], x[1], x[2], x[3]);
        buf[2 * lane + 1] = make_float4(x[4], x[5], x[6], x[7]);
        __syncwarp();
        float4 v[4], w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = buf[u];
        for (int q = 0; q < kBlock / 4; q += 16) {   // every lane adds the same, sixteen elements ahead of the additions
            const float before = s;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                float4 (&now)[4] = h & 1 ? w : v;
                float4 (&next)[4] = h & 1 ? v : w;
#pragma unroll
                for (int u = 0; u < 4; ++u) next[u] = buf[(q + 4 * h + 4 + u) & (kBlock / 4 - 1)];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    s = __fadd_rn(s, now[u].x);
                    s = __fadd_rn(s, now[u].y);
                    s = __fadd_rn(s, now[u].z);
                    s = __fadd_rn(s, now[u].w);
                }
            }
            if (s > thr) {   // sums only grow: the end of the 64 tells
                s = before;
                for (int h = q;; h += 2) {
                    const float4 a = buf[h], b = buf[h + 1];
                    float t = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, a.x), a.y), a.z), a.w);
                    t = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(t, b.x), b.y), b.z), b.w);
                    if (!(t > thr)) { s = t; continue; }
                    for (int e = 4 * h;; ++e) {
                        p = sh.serial[e];
                        s = __fadd_rn(s, p);
                        if (s > thr) return (long long)src.off + i + e;
                    }
                }
            }
        }
    }
    return -1;
}

// Walks the segments from c on (warp 0): whole ones while the guesses hold, one by one elsewhere.  Leaves the sum, the segment
// it came to and the element whose running sum is the first above thr (-1: none) in shared memory.
template <class Src>
__device__ void walk_segments(Src src, int c, int c1, float s, float thr) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31;
    uint32_t E = fsx::state_exp(s), S = fsx::state_sig(s);
    int misses = 0, tiles = 0;
    long long hit = -1;
    PROF_BEGIN;
    while (c < c1) {
        PROF_END(kProfOther);
        PROF_COUNT(kProfTiles);
        const int n = min(32, c1 - c), my = c + lane;
        const uint32_t Eg = lane < n ? sh.E[my] : kEmpty;
        uint32_t word = lane < n ? sh.step[my] : 1u;
        const int own_slot = lane < n ? sh.slot[my] : 0;
        const bool above = own_slot != 0 && Eg + 1u == E;   // the sum has changed binade before this one
        if (above) word = own_slot <= kSlots ? sh.from[own_slot - 1][0] : step_up(own_slot, my);
        const uint32_t wrong = __ballot_sync(0xffffffffu, !fsx::guess_holds(Eg, above, E));
        const int most = wrong ? __ffs(wrong) - 1 : n;   // as far as the guesses hold
        if (lane == 0) sh.state[c] = fsx::state_float(E, S);
        if (most > 0) {
            fsx::Step st = lane < most && Eg != kEmpty ? unpack_amounts(word) : fsx::step_identity();
            int taken = 0;
            if (!__any_sync(0xffffffffu, st.a != st.b)) {
                const uint32_t after = S + __reduce_add_sync(0xffffffffu, st.a);   // 32 x kSat at most
                if (after < fsx::kOne24 && !(fsx::state_float(E, after) > thr)) {
                    if (most > 1) {
                        if (lane == 0) sh.tile[tiles] = (uint16_t)(c | (most - 1) << 11);
                        ++tiles;
                        if (lane < most && Eg != kEmpty) sh.step[my] = word;   // (what the sums before them are filled in from)
                    }
                    S = after;
                    taken = most;
                }
            }
            if (taken == 0) {   // a half-way case, or the sum leaves the binade or passes the threshold: one segment after the other
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const fsx::Step up{__shfl_up_sync(0xffffffffu, st.a, o), __shfl_up_sync(0xffffffffu, st.b, o)};
                    if (lane >= o) st = fsx::then(up, st);
                }
                const uint32_t after = fsx::apply(st, S);
                const uint32_t up = __shfl_up_sync(0xffffffffu, after, 1);
                const uint32_t before = lane > 0 ? up : S;
                const uint32_t mask = __ballot_sync(0xffffffffu, lane < most && (after >= fsx::kOne24 || fsx::state_float(E, after) > thr));
                taken = mask ? __ffs(mask) - 1 : most;
                if (lane < n && lane <= taken) sh.state[my] = fsx::state_float(E, before);   // (from `most` on nothing is added)
                S = taken < 32 ? __shfl_sync(0xffffffffu, before, taken & 31) : __shfl_sync(0xffffffffu, after, 31);
            }
            c += taken;
            PROF_END(kProfTile);
            if (taken == n) continue;
            if (lane == 0) sh.state[c] = fsx::state_float(E, S);
        }
        if (lanes_at_hand(sh.slot[c])) {   // the sum may change binade in this one: its lanes' amounts are at hand
            const int slot = sh.slot[c] - 1;
            const uint32_t Eg = sh.E[c];
            uint32_t E2 = E, S2 = fsx::kOne24;
            if (E == Eg + 1u) {
                S2 = fsx::apply(unpack_amounts(sh.from[slot][0]), S);
            } else if (E == Eg) {
                const uint32_t upto = fsx::apply(unpack_amounts(sh.upto[slot][lane]), S);
                const uint32_t over = __ballot_sync(0xffffffffu, upto >= fsx::kOne24);
                if (!over) {
                    S2 = __shfl_sync(0xffffffffu, upto, 31);
                } else {
                    const int l = __ffs(over) - 1;   // this lane's elements take it into the next binade
                    const uint32_t below = __shfl_sync(0xffffffffu, upto, l > 0 ? l - 1 : 0);
                    float t = fsx::state_float(E, l > 0 ? below : S);
                    const uint32_t lo = sh.start[c] - src.off, hi = sh.start[c + 1] - src.off, lo8 = lo & ~7u, m = (hi - lo8 + kBlock - 1) / kBlock;
                    for (uint32_t q = 0; q < m; ++q) {
                        float x[8];
                        if (!Src::kSortable && m == 1) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) x[e] = sh.keys[slot * kBlock + 8 * l + e];
                        } else {
                            load8(src.data(), lo8 + 8 * (l * m + q), lo, hi, x);
                            src.prepare(x);
                        }
#pragma unroll
                        for (int e = 0; e < 8; ++e) t = __fadd_rn(t, x[e]);
                    }
                    E2 = fsx::state_exp(t);
                    if (E2 == E + 1u && !(t > thr)) S2 = l < 31 ? fsx::apply(unpack_amounts(sh.from[slot][l < 31 ? l + 1 : 31]), fsx::state_sig(t)) : fsx::state_sig(t);
                }
            }
            if (S2 < fsx::kOne24 && !(fsx::state_float(E2, S2) > thr)) {
                E = E2; S = S2;
                ++c;
                PROF_END(kProfSlot);
                PROF_COUNT(kProfSlots);
                continue;
            }
        }
        const uint32_t guessed = sh.E[c];   // (none or a right one: another would not help)
        if (guessed != kNoGuess && guessed != E && ++misses > kMaxMisses && c1 - c > 32) break;
        PROF_COUNT(kProfMisses);
        if constexpr (Src::kSortable) {
            if (sh.sorted[c] != 1) sort_in_chunk(src, c);
        }
        s = fsx::state_float(E, S);
        float p;
        hit = add_segment(src, c, s, thr, p);
        E = fsx::state_exp(s); S = fsx::state_sig(s);
        PROF_END(kProfSerial);
        if (hit >= 0) break;
        ++c;
    }
    if (lane == 0) { sh.bc_s = fsx::state_float(E, S); sh.bc_seg = c; sh.bc_hit = hit; sh.tiles = tiles; }
}
// The sums before the segments of the runs that the walk took as a whole.
__device__ void fill_states() {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = warp; t < sh.tiles; t += kWarps) {
        const int c = sh.tile[t] & 2047, n = (sh.tile[t] >> 11) + 1;
        const float s = sh.state[c];
        uint32_t sum = lane < n && sh.E[c + lane] != kEmpty ? sh.step[c + lane] >> 2 : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
        }
        const uint32_t before = __shfl_up_sync(0xffffffffu, sum, 1);
        if (lane > 0 && lane < n) sh.state[c + lane] = fsx::state_float(fsx::state_exp(s), fsx::state_sig(s) + before);
    }
}

// Sums before the segments of a row from its elements as they are prepared, for rows of which min-p may drop so much that the sums at hand are of
// no use.  (A pass of 12 us over 128256 elements; with the sums of all elements most guesses are wrong and a step takes 960 us instead of 145.)
template <class Src>
__device__ __noinline__ void sums_of(Src src, int n) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kAtOnce = 2;
    __syncthreads();
    for (int j = warp; j < n; j += kAtOnce * kWarps) {
        uint32_t lo[kAtOnce], hi[kAtOnce];
        float mass[kAtOnce];
#pragma unroll
        for (int u = 0; u < kAtOnce; ++u) {
            const int k = min(j + u * kWarps, n);   // (n: nothing)
            lo[u] = sh.start[k] - src.off;
            hi[u] = sh.start[min(k + 1, n)] - src.off;
            mass[u] = 0.f;
        }
        bool more = true;
        for (uint32_t at = 0; more; at += kBlock) {
            float x[kAtOnce][8];
            more = false;
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u) {
                const uint32_t i = (lo[u] & ~7u) + at;
                load8(src.data(), i + 8 * lane, lo[u], hi[u], x[u]);
                more |= i + kBlock < hi[u];
            }
#pragma unroll
            for (int u = 0; u < kAtOnce; ++u) {
                src.prepare(x[u]);
#pragma unroll
                for (int e = 0; e < 8; ++e) mass[u] += x[u][e];
            }
        }
#pragma unroll
        for (int u = 0; u < kAtOnce; ++u) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mass[u] += __shfl_xor_sync(0xffffffffu, mass[u], o);
            if (lane == 0 && j + u * kWarps < n) sh.cum[j + u * kWarps] = mass[u];
        }
    }
    masses_to_sums(n);
}
// Adds the segments c .. c1 - 1 to s in order, exactly as `s += x[i]` does, from the approximate sums in sh.cum (have_steps: the guesses
// are made and the amounts known).  It stops at the first running sum above thr and returns that element, else -1.  sh.state: the sum before every segment it came to.
template <class Src>
__device__ __noinline__ long long ordered_sum(Src src, int c, int c1, float& s, float thr, float thr2, bool have_steps = false) {
    ExactShared& sh = shared_memory();
    PROF_BEGIN;
    if constexpr (Src::kThreshold) {
        // What is dropped is below min_thr each, and all probabilities together are one: a 256th less is within the guesses' wide margin.
        if (src.min_thr * (float)(sh.start[c1] - sh.start[c]) > 1.f / 256) sums_of(src, c1);
    }
    for (;; have_steps = false) {
        if (!have_steps) {
            guess_binades(c, c1, s, thr, thr2, !Src::kSortable);
            PROF_END(kProfGuess);
            segment_steps(src, c, c1);
            PROF_END(kProfSteps);
        }
        if (threadIdx.x < 32) walk_segments(src, c, c1, s, thr);
        __syncthreads();
        fill_states();
        PROF_END(kProfWalk);
        s = sh.bc_s; c = sh.bc_seg;
        const long long hit = sh.bc_hit;
        __syncthreads();
        if (hit >= 0 || c >= c1) return hit;
    }
}
// The segments of a row in index order: elements lo .. hi - 1.
__device__ void index_order_segments(Segs g, uint32_t lo, uint32_t hi) {
    ExactShared& sh = shared_memory();
    for (int j = threadIdx.x; j <= g.count; j += kThreads) {
        sh.start[j] = max(lo, min(hi, (uint32_t)j << g.shift));
        if (j < g.count) sh.sorted[j] = 1;
    }
}

// ---- descending order --------------------------------------------------------------------------------------
// Keys are the bit patterns of the exponentials.  A level cuts the keys below F into bins of 2^shift, highest first; what lies
// below the last bin is the level's rest.
struct Level {
    uint32_t F;
    int shift;
    uint32_t total;   // elements in its bins
    bool rest;
};
__device__ __forceinline__ uint32_t bin_of(const Level& L, uint32_t key) { return (L.F - 1u - key) >> L.shift; }

// Adds one to a word of shared memory where x < end, without a branch; take_below returns what was there, put_below stores.
__device__ __forceinline__ void count_below(uint32_t addr, uint32_t x, uint32_t end) {
    asm volatile("{ .reg .pred p; setp.lt.u32 p, %1, %2; @p red.shared.add.u32 [%0], 1; }" ::"r"(addr), "r"(x), "r"(end) : "memory");
}
__device__ __forceinline__ uint32_t take_below(uint32_t addr, uint32_t x, uint32_t end) {
    uint32_t old = 0;
    asm volatile("{ .reg .pred p; setp.lt.u32 p, %2, %3; @p atom.shared.add.u32 %0, [%1], 1; }" : "+r"(old) : "r"(addr), "r"(x), "r"(end) : "memory");
    return old;
}
__device__ __forceinline__ void put_below(uint32_t addr, float v, uint32_t x, uint32_t end) {
    asm volatile("{ .reg .pred p; setp.lt.u32 p, %2, %3; @p st.shared.f32 [%0], %1; }" ::"r"(addr), "f"(v), "r"(x), "r"(end) : "memory");
}

// Calls fn(four elements) for the exponentials, 16-byte loads, four in flight per thread.  The row begins on a 16-byte boundary, its
// elements are those from lo to hi - 1, and what the first and the last load bring along are zeros.
template <class F>
__device__ __forceinline__ void for_exponentials(const float* ex, uint32_t hi, F&& fn) {
    const float4* e4 = reinterpret_cast<const float4*>(ex);
    const uint32_t n4 = (hi + 3) >> 2;
    for (uint32_t i = threadIdx.x; i < n4; i += 4 * kThreads) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = i + u * kThreads < n4 ? e4[i + u * kThreads] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 4; ++u) fn(v[u]);
    }
}

__device__ __noinline__ void count_level(Level& L, const float* ex, uint32_t hi) {
    ExactShared& sh = shared_memory();
    __syncthreads();
    for (int j = threadIdx.x; j < kBins; j += kThreads) sh.bins[j] = 0;
    __syncthreads();
    bool rest = false;
    const uint32_t bins = (uint32_t)__cvta_generic_to_shared(sh.bins);
    for_exponentials(ex, hi, [&](float4 v) {
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t key = __float_as_uint(e[u]), b = bin_of(L, key);
            const bool in = key - 1u < L.F - 1u;   // zeros are left to the end; NaN and what an earlier level has taken
            count_below(bins + 4 * b, in ? b : 0xffffffffu, (uint32_t)kBins);
            rest |= in && b >= (uint32_t)kBins;
        }
    });
    L.rest = __syncthreads_or(rest) != 0;
}

struct Row {
    const float* ex;    // exponentials in index order: elements lo .. hi - 1
    float* sorted;      // the largest probabilities, as far as they were needed: segment by segment in descending order, those within
                        // a segment only where it mattered
    uint32_t lo, hi;
    float norm, inv_norm, min_thr;
};

// Segments that n elements in descending order may take, two boundaries per bin of its own included
__device__ __forceinline__ uint32_t most_segments(uint32_t n, int shift) { return (n >> shift) + 2 * ((n >> shift) / kBigSegs) + 4; }

// Counts -> ranks of the bins' first elements, and the level's segments from number c on: whole bins, one beginning with the first
// bin at or after every multiple of the segment length, bins of kBigSegs times that by themselves.  The segments are as short as the table has
// room for (g: their length; the row's own at most): up to 512 elements are sorted in a warp's registers, and with the 512 to 1024 of a
// row of 200064 bf16 logits a step took 306 us where it takes 238.  `placed` elements come
// before the level, `sum` is their sum.  Bins of nothing but probabilities below the min-p threshold are left out, and with them what
// lies below the level.  Returns the number after the level's last segment; *reach: the first segment that begins
// above target as far as the bins tell (that number: none).
__device__ __noinline__ int rank_bins(Level& L, Row row, Segs& g, int c, uint32_t placed, float sum, float target, int* reach) {
    ExactShared& sh = shared_memory();
    const int tid = threadIdx.x, j0 = tid * kBinsPerThread;
    __syncthreads();
    uint32_t n[kBinsPerThread];
#pragma unroll
    for (int k = 0; k < kBinsPerThread; ++k) n[k] = sh.bins[j0 + k];
    int bins = kBins;   // those that count: the bins' largest keys fall
    if (row.min_thr > 0.f) {
        int dropped = kBins;
#pragma unroll
        for (int k = 0; k < kBinsPerThread; ++k) {
            const unsigned long long down = ((unsigned long long)(j0 + k) << L.shift) + 1u;
            if (down >= L.F || !(probability(__uint_as_float(L.F - (uint32_t)down), row.norm, row.inv_norm) >= row.min_thr)) {
                n[k] = 0;
                dropped = min(dropped, j0 + k);
            }
        }
        bins = block_reduce(dropped, [](int a, int b) { return min(a, b); }, sh.red_i);
        if (bins < kBins) L.rest = false;
    }
    float value[kBinsPerThread], mass = 0.f;
    uint32_t count = 0, own_last = 0;
#pragma unroll
    for (int k = 0; k < kBinsPerThread; ++k) {   // the middle of the bin
        const uint32_t down = ((uint32_t)(j0 + k) << L.shift) + ((1u << L.shift) >> 1) + 1u;
        value[k] = n[k] && down < L.F ? (float)n[k] * (__uint_as_float(L.F - down) * row.inv_norm) : 0.f;
        mass += value[k];
        count += n[k];
        own_last = n[k] ? n[k] : own_last;
    }
    const uint32_t first = block_scan_exclusive(count, sh.scan_u, &L.total);
    int shift = 8;
    while (shift < g.shift && (uint32_t)c + most_segments(L.total, shift) > (uint32_t)kSegCap) ++shift;
    g.shift = shift;
    const uint32_t big = (uint32_t)kBigSegs << shift;
    float cum = sum + block_scan_exclusive(mass, sh.scan_f, (float*)nullptr);
    // does a segment begin with the bin?  The last bin before that is not empty tells
    const uint32_t n_before = block_scan_exclusive(own_last, sh.scan_u, (uint32_t*)nullptr, [](uint32_t a, uint32_t b) { return b ? b : a; });
    bool begins[kBinsPerThread];
    uint32_t at = first, before = n_before, marks = 0;
#pragma unroll
    for (int k = 0; k < kBinsPerThread; ++k) {
        begins[k] = n[k] && (at == 0 || (at >> shift) != ((at - before) >> shift) || n[k] >= big || before >= big);
        marks += begins[k] ? 1u : 0u;
        at += n[k];
        if (n[k]) before = n[k];
    }
    uint32_t total;
    uint32_t no = c + block_scan_exclusive(marks, sh.scan_u, &total);
    at = first;
    int far = 0x7fffffff;
#pragma unroll
    for (int k = 0; k < kBinsPerThread; ++k) {
        sh.bins[j0 + k] = at;
        if (begins[k]) {
            if (no < (uint32_t)kSegCap) {
                sh.start[no] = placed + at; sh.bin[no] = (uint16_t)(j0 + k); sh.cum[no] = cum;
                sh.sorted[no] = L.shift == 0 ? 1 : 0;   // bins of one value
                if (cum > target) far = min(far, (int)no);
            }
            ++no;
        }
        at += n[k];
        cum += value[k];
    }
    const int end = min(c + (int)total, kSegCap);
    if (tid == kThreads - 1) { sh.start[end] = placed + L.total; sh.bin[end] = (uint16_t)bins; sh.cum[end] = cum; }
    far = block_reduce(far, [](int a, int b) { return min(a, b); }, sh.red_i);   // (its barriers cover the tables)
    *reach = min(far, end);
    return end;
}

// Brings the segments c .. c1 - 1 (whole bins, at most kCap elements) into shared memory and the row, up to sh.stop, the first one that is
// too large to be sorted and not all the same; elements below the min-p threshold as zeros.  Returns how many are not.
__device__ __noinline__ uint32_t place_chunk(Row row, Level L, Segs g, int c, int c1, uint32_t placed) {
    ExactShared& sh = shared_memory();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    PROF_BEGIN;
    const int j0 = sh.bin[c], j1 = sh.bin[c1];
    const uint32_t off = sh.start[c];
    if (tid == 0) sh.stop = c1;
    __syncthreads();
    const uint32_t high = L.F - ((uint32_t)j0 << L.shift);   // keys from low to high - 1
    const long long below = (long long)L.F - ((long long)j1 << L.shift);
    const uint32_t low = below > 1 ? (uint32_t)below : 1u;
    const uint32_t bins = (uint32_t)__cvta_generic_to_shared(sh.bins), keys = (uint32_t)__cvta_generic_to_shared(sh.keys) - 4 * (off - placed);
    for_exponentials(row.ex, row.hi, [&](float4 v) {
        const float e[4] = {v.x, v.y, v.z, v.w};
        uint32_t pos[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {   // (as many as were counted: a place is within the chunk)
            const uint32_t key = __float_as_uint(e[u]);
            pos[u] = take_below(bins + 4 * bin_of(L, key), key - low, high - low);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) put_below(keys + 4 * pos[u], e[u], __float_as_uint(e[u]) - low, high - low);
    });
    __syncthreads();
    PROF_END(kProfGather);
    const uint32_t big = (uint32_t)kBigSegs << g.shift;
    for (int j = c + warp; j < c1; j += kWarps) {
        const uint32_t a = sh.start[j] - off, z = sh.start[j + 1] - off;
        if (z - a < big || sh.sorted[j] == 1) continue;
        bool same = true;
        const float first = sh.keys[a];
        for (uint32_t i = a + lane; i < z; i += 32) same &= sh.keys[i] == first;
        same = __all_sync(0xffffffffu, same);
        if (lane == 0) {
            if (same) sh.sorted[j] = 1;
            else if (z - a >= 2 * big) atomicMin(&sh.stop, j);
        }
    }
    __syncthreads();
    PROF_END(kProfSame);
    uint32_t valid = 0;
    float* out = row.sorted + off;
    const uint32_t n = sh.start[sh.stop] - off;
    for (uint32_t i = tid; i < n; i += 4 * kThreads) {
        float p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = i + u * kThreads < n ? sh.keys[i + u * kThreads] : 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            p[u] = probability(p[u], row.norm, row.inv_norm);
            const bool in = i + u * kThreads < n, keep = p[u] >= row.min_thr;
            valid += in && keep ? 1u : 0u;
            if (in) {
                sh.keys[i + u * kThreads] = keep ? p[u] : 0.f;
                out[i + u * kThreads] = keep ? p[u] : 0.f;
            }
        }
    }
    valid = block_sum(valid, sh.scan_u);
    PROF_END(kProfPlace);
    return valid;
}

struct Kept {
    uint32_t n;        // elements kept, zeros included
    uint32_t placed;   // of them in row.sorted
    int segs;          // segments with a recorded sum
    float total;
};

// Makes one of every two of the segments 0 .. c - 1.
__device__ __noinline__ int merge_segments(int c) {
    ExactShared& sh = shared_memory();
    constexpr int kPer = (kSegCap / 2 + kThreads - 1) / kThreads + 1;
    const int half = (c + 1) / 2;
    uint32_t start[kPer];
    float state[kPer];
    uint8_t sorted[kPer];
    __syncthreads();
    const uint32_t end = sh.start[c];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int j = 2 * ((int)threadIdx.x + k * kThreads);
        if (j >= c) continue;
        start[k] = sh.start[j];
        state[k] = sh.state[j];
        sorted[k] = sh.sorted[j] == 1 && (j + 1 >= c || sh.sorted[j + 1] == 1) ? 1 : 0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int j = (int)threadIdx.x + k * kThreads;
        if (2 * j >= c) continue;
        sh.start[j] = start[k]; sh.state[j] = state[k]; sh.sorted[j] = sorted[k];
    }
    if (threadIdx.x == 0) sh.start[half] = end;
    __syncthreads();
    return half;
}

// TopPFilter: descending order, until the float sum exceeds top_p.  The first level's bins are counted already.  `u`: the number of
// the row's own draw.
__device__ __noinline__ Kept keep_top_p(Row row, Segs longest, Level L, float top_p, float u) {
    ExactShared& sh = shared_memory();
    const int tid = threadIdx.x;
    uint32_t placed = 0;       // elements before segment c, and their sum
    int c = 0;
    float s = 0.f;
    int next_shift = kTopShift;
    bool last = false;
    while (!last) {
        PROF_BEGIN;
        // room for the segments of all that is left (a row of many levels: one or two extra for each)
        while (c > 1 && (uint32_t)c + most_segments(row.hi - placed, longest.shift) > (uint32_t)kSegCap) c = merge_segments(c);
        int reach;
        Segs g = longest;
        const int end = rank_bins(L, row, g, c, placed, s, top_p * (1.0f + 1.0f / 1024), &reach);
        PROF_END(kProfRank);
        const uint32_t level_at = placed;
        bool again = false;    // another level takes over before this one's end
        while (c < end && !last && !again) {
            // the most segments that fit and may be needed
            int c1 = c, hi = c < reach ? reach : end;
            while (c1 < hi) {
                const int mid = (c1 + hi + 1) >> 1;
                if (sh.start[mid] - sh.start[c] <= (uint32_t)kCap) c1 = mid; else hi = mid - 1;
            }
            const uint32_t key_below = L.F - ((uint32_t)sh.bin[c] << L.shift);   // keys of this segment and those behind are below
            long long hit = -1;
            if (c1 > c) {
                const uint32_t valid = place_chunk(row, L, g, c, c1, level_at);
                const int stop = sh.stop;
                const uint32_t n = sh.start[stop] - placed;
                hit = ordered_sum(Chunk{placed, row.sorted}, c, stop, s, top_p, top_p * u);
                if (hit >= 0) return Kept{(uint32_t)hit + 1, sh.start[sh.bc_seg + 1], sh.bc_seg + 1, s};
                last = valid < n;   // below the min-p threshold from here on
                placed += valid;
                c = stop;
                if (stop < c1 && !last) {
                    L = Level{L.F - ((uint32_t)sh.bin[stop] << L.shift), max(0, L.shift - kFinerBy), 0, false};
                    next_shift = L.shift;
                    again = true;
                }
            } else if (L.shift > 0) {   // one bin with more than fits
                L = Level{key_below, max(0, L.shift - kFinerBy), 0, false};
                next_shift = L.shift;
                again = true;
            } else {                    // one value: its segments are made here, those of the level are made anew behind it
                const uint32_t n = sh.start[c + 1] - sh.start[c];
                const float p = probability(__uint_as_float(key_below - 1u), row.norm, row.inv_norm);
                __syncthreads();
                if (p >= row.min_thr) {
                    for (uint32_t i = tid; i < n; i += kThreads) row.sorted[placed + i] = p;
                    const int segs = min((int)((n + g.len() - 1) >> g.shift), kSegCap - c);
                    for (int j = tid; j <= segs; j += kThreads) {
                        sh.start[c + j] = placed + min(n, (uint32_t)j << g.shift);
                        sh.cum[c + j] = s + p * (float)min(n, (uint32_t)j << g.shift);
                        if (j < segs) sh.sorted[c + j] = 1;
                    }
                    __syncthreads();
                    hit = ordered_sum(Sorted{row.sorted, 0}, c, c + segs, s, top_p, -1.f);
                    if (hit >= 0) return Kept{(uint32_t)hit + 1, placed + n, sh.bc_seg + 1, s};
                    placed += n;
                    c += segs;
                    L = Level{key_below - 1u, next_shift, 0, true};
                    again = true;
                } else {
                    last = true;
                }
            }
            if (c >= reach) reach = end;
        }
        if (last) break;
        if (!again) {
            const unsigned long long span = (unsigned long long)kBins << L.shift;
            if (!L.rest || span >= L.F) break;
            if (L.total < 4096u) next_shift = min(kTopShift, next_shift + kFinerBy);
            L = Level{(uint32_t)(L.F - span), next_shift, 0, false};
        }
        if (L.F <= 1u) break;
        count_level(L, row.ex, row.hi);
    }
    // every candidate is in the sum; without a min-p threshold the zeros are candidates too
    uint32_t zeros = 0;
    if (!last && 0.f >= row.min_thr) {
        for (uint32_t i = row.lo + tid; i < row.hi; i += kThreads) zeros += row.ex[i] == 0.f ? 1u : 0u;
        zeros = block_sum(zeros, sh.scan_u);
    }
    while (c > 0 && sh.start[c - 1] >= placed) --c;   // segments of nothing but zeros
    return Kept{placed + zeros, placed, c, s};
}

// The vocabulary index of the element of rank `rank` in descending order, whose probability is p: among equal ones, however many, the
// lowest index comes first.
__device__ __noinline__ long long index_of_rank(Row row, uint32_t rank, float p) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    PROF_BEGIN;
    // the exponentials with this probability are neighbours: a look around p * norm finds the first and the last of them
    uint32_t key_lo = 0, key_hi = 0;   // zero: they are compared by their probabilities
    {
        const int mid = (int)__float_as_uint(p * row.norm), cand = mid - 16 + lane;
        const bool in = p > 0.f && cand > 0 && cand <= (int)kOneBits && probability(__uint_as_float((uint32_t)cand), row.norm, row.inv_norm) == p;
        const uint32_t m = __ballot_sync(0xffffffffu, in);
        if (m && !(m & 0x80000001u)) {
            key_lo = (uint32_t)(mid - 16 + __ffs(m) - 1);
            key_hi = (uint32_t)(mid - 16 + 31 - __clz(m));
        }
    }
    auto equal = [&](float e) {
        if (key_lo) return __float_as_uint(e) - key_lo <= key_hi - key_lo;
        return probability(e, row.norm, row.inv_norm) == p;
    };
    auto above = [&](float e) { return key_lo ? e > __uint_as_float(key_hi) : probability(e, row.norm, row.inv_norm) > p; };
    uint32_t same = 0, lowest = 0xffffffffu;
    const float4* e4 = reinterpret_cast<const float4*>(row.ex);
    const uint32_t n4 = (row.hi + 3) >> 2;
    const uint32_t span = key_lo ? key_hi - key_lo : 0xffffffffu;
    for (uint32_t i0 = threadIdx.x; i0 < n4; i0 += 4 * kThreads) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = i0 + u * kThreads < n4 ? e4[i0 + u * kThreads] : make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F);
        uint32_t nearest = 0xffffffffu;   // two instructions for an element that is not one of them
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            nearest = min(nearest, min(__float_as_uint(v[u].x) - key_lo, __float_as_uint(v[u].y) - key_lo));
            nearest = min(nearest, min(__float_as_uint(v[u].z) - key_lo, __float_as_uint(v[u].w) - key_lo));
        }
        if (nearest > span) continue;
#pragma unroll 1
        for (int u = 0; u < 16; ++u) {
            const uint32_t i = 4 * (i0 + (u >> 2) * kThreads) + (u & 3);
            if (i >= row.lo && i < row.hi && equal(row.ex[i])) { ++same; lowest = min(lowest, i); }
        }
    }
    __syncthreads();
    same = block_sum(same, sh.scan_u);
    lowest = block_reduce(lowest, [](uint32_t a, uint32_t b) { return min(a, b); }, sh.scan_u);
    PROF_END(kProfIndex);
    if (same <= 1) return lowest == 0xffffffffu ? row.lo : (long long)lowest;
    // several: the rank among them
    const uint32_t blocks = (row.hi + kBlock - 1) / kBlock, per = (blocks + kWarps - 1) / kWarps;
    const uint32_t b0 = min(blocks, warp * per), b1 = min(blocks, b0 + per);
    uint32_t greater = 0;
    same = 0;
    for (uint32_t b = b0; b < b1; ++b) {
        const uint32_t i = b * kBlock + 8 * lane;
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (i + e >= row.lo && i + e < row.hi) {
                const float q = row.ex[i + e];
                same += equal(q) ? 1u : 0u;
                greater += above(q) ? 1u : 0u;
            }
    }
    same = __reduce_add_sync(0xffffffffu, same);
    greater = block_sum(greater, sh.scan_u);
    const uint32_t scanned = block_scan_exclusive(lane == 0 ? same : 0u, sh.scan_u, (uint32_t*)nullptr);
    const uint32_t before = __shfl_sync(0xffffffffu, scanned, 0);
    const uint32_t want = rank < greater ? 0u : rank - greater;
    if (threadIdx.x == 0) sh.bc_hit = lowest;
    __syncthreads();
    if (want >= before && want < before + same) {   // one warp
        uint32_t seen = before;
        for (uint32_t b = b0; b < b1 && seen <= want; ++b) {
            const uint32_t i = b * kBlock + 8 * lane;
            uint32_t mine = 0;   // a bit per element
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (i + e >= row.lo && i + e < row.hi && equal(row.ex[i + e])) mine |= 1u << e;
            uint32_t incl = __popc(mine);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            uint32_t at = seen + incl - __popc(mine);
            for (; mine; mine &= mine - 1, ++at)
                if (at == want) sh.bc_hit = (long long)i + __ffs(mine) - 1;
            seen += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
    const long long idx = sh.bc_hit;
    __syncthreads();
    PROF_END(kProfIndex2);
    return idx;
}

// A row with several draws and few elements kept: their probabilities and indices are listed in one pass, at the end of `keys` (what a draw may
// sort there has room before it).  Without the list every draw takes a pass of its own: a row of three to eight kept elements with 16 further
// draws 352 us a step, with it 205.  False: more elements than fit.
__device__ __forceinline__ uint2* listed() { return reinterpret_cast<uint2*>(shared_memory().keys + kCap - 2 * kListed); }
__device__ __forceinline__ bool list_kept(Row row, uint32_t placed) {
    ExactShared& sh = shared_memory();
    if (placed > (uint32_t)kListed) return false;
    float least = CUDART_INF_F;   // (zeros are below the min-p threshold)
    for (uint32_t i = threadIdx.x; i < placed; i += kThreads) {
        const float p = row.sorted[i];
        if (p > 0.f) least = fminf(least, p);
    }
    least = block_reduce(least, [](float a, float b) { return fminf(a, b); }, sh.scan_f);
    if (!(least >= 0x1p-100f)) return false;   // (too few bits for `about`)
    if (threadIdx.x == 0) sh.count = 0;
    __syncthreads();
    const float about = least * row.norm * (1.f - 1.f / 1048576);   // (a little below the least exponential: the division tells)
    const float4* e4 = reinterpret_cast<const float4*>(row.ex);
    const uint32_t n4 = (row.hi + 3) >> 2;
    for (uint32_t i0 = threadIdx.x; i0 < n4; i0 += 4 * kThreads) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = i0 + u * kThreads < n4 ? e4[i0 + u * kThreads] : make_float4(0.f, 0.f, 0.f, 0.f);
        float most = 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) most = fmaxf(most, fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w)));
        if (!(most >= about)) continue;
#pragma unroll 1
        for (int u = 0; u < 16; ++u) {
            const uint32_t i = 4 * (i0 + (u >> 2) * kThreads) + (u & 3);
            if (i < row.lo || i >= row.hi || !(row.ex[i] >= about)) continue;
            const float p = probability(row.ex[i], row.norm, row.inv_norm);
            if (!(p >= least)) continue;
            const int at = atomicAdd(&sh.count, 1);
            if (at < kListed) listed()[at] = make_uint2(__float_as_uint(p), i);
        }
    }
    __syncthreads();
    return sh.count <= kListed;
}
// index_of_rank from the list (-1: not there, or too many of one value).
__device__ __noinline__ long long listed_index(uint32_t rank, float p) {
    ExactShared& sh = shared_memory();
    const int n = sh.count, tid = threadIdx.x;
    uint32_t* equal = reinterpret_cast<uint32_t*>(sh.serial);   // the indices of those with this probability
    if (tid == 0) { sh.stop = 0; sh.bc_hit = -1; }
    __syncthreads();
    uint32_t greater = 0;
    for (int i = tid; i < n; i += kThreads) {
        const uint2 e = listed()[i];
        const float q = __uint_as_float(e.x);
        greater += q > p ? 1u : 0u;
        if (q == p) {
            const int at = atomicAdd(&sh.stop, 1);
            if (at < kBlock) equal[at] = e.y;
        }
    }
    greater = block_sum(greater, sh.scan_u);   // (its barriers cover the list)
    const int same = sh.stop;
    if (same <= kBlock && tid < same) {
        uint32_t before = 0;
        for (int k = 0; k < same; ++k) before += equal[k] < equal[tid] ? 1u : 0u;
        if (before == (rank < greater ? 0u : rank - greater)) sh.bc_hit = equal[tid];
    }
    __syncthreads();
    const long long at = sh.bc_hit;
    __syncthreads();
    return at;
}

// First element of src, of those below n, whose running sum exceeds r (-1: none), from the sums recorded before the segments
// 0 .. segs - 1.  `unsorted`: the row in memory whose segment may have to be sorted first.
template <class Src>
__device__ __noinline__ long long find_draw(Src src, int segs, uint32_t n, float* unsorted, float r, float& p) {
    ExactShared& sh = shared_memory();
    PROF_BEGIN;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int lo = 0, hi = segs - 1;   // the last segment with a sum not above r (the first has none)
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (!(sh.state[mid] > r)) lo = mid; else hi = mid - 1;
        }
        float s = segs > 0 ? sh.state[lo] : 0.f, q = 0.f;
        long long hit = -1;
        for (int j = lo; j < segs && hit < 0; ++j) {
            if (unsorted && sh.sorted[j] != 1) {
                const uint32_t a = sh.start[j], len = sh.start[j + 1] - a;
                if (len <= (uint32_t)kCap) {
                    for (uint32_t i = lane; i < len; i += 32) sh.keys[i] = unsorted[a + i];
                    sort_segment(sh.keys, (int)len);
                    for (uint32_t i = lane; i < len; i += 32) unsorted[a + i] = sh.keys[i];
                } else {
                    sort_segment(unsorted + a, (int)len);   // (merged segments of a very long row)
                }
                __syncwarp();
                if (lane == 0) sh.sorted[j] = 1;
                __syncwarp();
            }
            hit = add_segment(src, j, s, r, q);
        }
        if (hit >= (long long)n) hit = -1;
        if (lane == 0) { sh.bc_hit = hit; sh.bc_p = q; }
    }
    __syncthreads();
    const long long hit = sh.bc_hit;
    p = sh.bc_p;
    __syncthreads();
    PROF_END(kProfFind);
    return hit;
}

// The table of 2^(i / 32) in the lanes' registers: in shared memory, 32 different entries of eight bytes cost a warp six to seven
// passes, two shuffles cost two.
struct LaneTable {
    uint32_t lo, hi;
    __device__ explicit LaneTable(int lane) {
        const uint64_t entry = fsx::kExp2TabDev[lane];
        lo = (uint32_t)entry;
        hi = (uint32_t)(entry >> 32);
    }
    __device__ __forceinline__ double operator()(uint64_t ki) const {   // (lane ki mod 32)
        const uint32_t k = (uint32_t)ki, l = __shfl_sync(0xffffffffu, lo, (int)k), h = __shfl_sync(0xffffffffu, hi, (int)k);
        return __hiloint2double((int)(h + (k << 15)), (int)l);
    }
};

// expf with the host libm's bits (fsx::expf_libm), one argument per lane
__device__ __forceinline__ float expf_lanes(float x, LaneTable tab) {
    const bool in = x >= -103.972076f && !(x > 88.72283f);
    const float f = fsx::expf_scaled((double)(in ? x : 0.f), tab);
    return in ? f : x > 0.f ? CUDART_INF_F : x != x ? x : 0.f;
}
// The same for arguments from -inf to 0, without the selections.
__device__ __forceinline__ float expf_lanes_nonpositive(float x, LaneTable tab) { return fsx::expf_scaled(fsx::nonpositive_as_double(x), tab); }

// The elements of a logits row from an address on a 16-byte boundary on: lo .. hi - 1 of `base`.
struct Logits {
    const float* base;
    uint32_t lo, hi;
    // i: a multiple of four; -inf beyond the elements.  kLast: the row is not read again, its place in L2 is the exponentials'
    template <bool kLast = false>
    __device__ __forceinline__ void load4(uint32_t i, float (&x)[4]) const {
        if (i >= lo && i + 4 <= hi) {
            const float4* at = reinterpret_cast<const float4*>(base + i);
            const float4 q = kLast ? __ldcs(at) : *at;
            x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = i + e >= lo && i + e < hi ? base[i + e] : -CUDART_INF_F;
        }
    }
};

// Maximum of the row and, for `masses`, the approximate sums of the exponentials before its segments (of one block each; kLong: of up to
// kFusedBlocks), from the maxima and masses of 1024 elements at a time; *odd: the row holds NaN or +inf.  Bound by HBM.
template <bool kLong>
__device__ __noinline__ float survey(Logits row, Segs g, float inv_T, bool masses, bool* odd) {
    ExactShared& sh = shared_memory();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr float kLog2e = 1.442695040888963f;
    const float scale = inv_T * kLog2e;
    const uint32_t blocks = (row.hi + kBlock - 1) / kBlock;
    float mx = -CUDART_INF_F;
    bool bad = false;
    for (uint32_t b = 4 * warp; b < blocks; b += 4 * kWarps) {
        float x[8][4];
#pragma unroll
        for (int u = 0; u < 8; ++u) row.load4(b * kBlock + u * 128 + 4 * lane, x[u]);
        float top = -CUDART_INF_F;
#pragma unroll
        for (int u = 0; u < 8; ++u) top = fmaxf(top, fmaxf(fmaxf(x[u][0], x[u][1]), fmaxf(x[u][2], x[u][3])));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        mx = fmaxf(mx, top);
        const float ref = top == -CUDART_INF_F ? 0.f : -top * scale;
        float whole = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float m = 0.f;
#pragma unroll
            for (int u = 2 * k; u < 2 * k + 2; ++u)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float y;
                    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaf(x[u][e], scale, ref)));
                    m += y;   // NaN where the row or the temperature is odd
                }
            bad |= !(m < CUDART_INF_F);
            if (masses) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
                if (kLong) {   // (b is a multiple of four)
                    const int per = g.shift - 8;
                    const uint32_t j = (b + k) >> per;
                    whole += m;
                    if (((k + 1) & ((1 << per) - 1)) == 0) {
                        if (lane == 0 && j < (uint32_t)g.count) { sh.cum[j] = whole; sh.state[j] = top; }
                        whole = 0.f;
                    }
                } else if (lane == 0 && b + k < blocks) { sh.cum[b + k] = m; sh.state[b + k] = top; }
            }
        }
    }
    *odd = __syncthreads_or(bad) != 0;
    mx = block_reduce(mx, [](float a, float b) { return fmaxf(a, b); }, sh.scan_f);
    if (masses && !*odd) {
        for (int j = threadIdx.x; j < g.count; j += kThreads) sh.cum[j] *= exp2f((sh.state[j] - mx) * scale);   // (-inf: 0)
        masses_to_sums(g.count);
    }
    return mx;
}

// Exponentials of the row into ex[], with kCount the counts of the first level's bins, and the amounts of the segments (of one block
// each) under the guesses made.  For rows and temperatures that make every exponential a number from 0 to 1.
// Bound by instruction issue (some 35 per element, eight of them in double precision).
template <bool kCount>
__device__ __noinline__ void exponentials(Logits row, float mx, float inv_T, float* ex, Level& level) {
    ExactShared& sh = shared_memory();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const LaneTable tab(lane);
    const uint32_t bins = (uint32_t)__cvta_generic_to_shared(sh.bins);
    if (kCount)
        for (int j = tid; j < kBins; j += kThreads) sh.bins[j] = 0;
    __syncthreads();
    bool rest = false;
    const uint32_t blocks = (row.hi + kBlock - 1) / kBlock;
    for (uint32_t b = warp; b < blocks; b += 2 * kWarps) {   // two blocks: four 16-byte loads in flight per lane
        float x[2][2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int u = 0; u < 2; ++u) row.load4<true>((b + h * kWarps) * kBlock + 8 * lane + 4 * u, x[h][u]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t j = b + h * kWarps;
            if (j >= blocks) break;
            float y[8];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int e = 0; e < 4; ++e) y[4 * u + e] = expf_lanes_nonpositive(__fmul_rn(__fsub_rn(x[h][u][e], mx), inv_T), tab);   // (inv_T 1: as it is)
                if (kCount) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const uint32_t bin = (kOneBits - __float_as_uint(y[4 * u + e])) >> kTopShift;
                        count_below(bins + 4 * bin, bin, (uint32_t)kBins);
                        rest |= bin >= (uint32_t)kBins;   // (zeros too: the next level's counts tell)
                    }
                }
                *reinterpret_cast<float4*>(ex + j * kBlock + 8 * lane + 4 * u) = make_float4(y[4 * u], y[4 * u + 1], y[4 * u + 2], y[4 * u + 3]);
            }
            const uint32_t E = sh.E[j];
            const int slot = sh.slot[j];
            if (lanes_at_hand(slot)) {
                __syncwarp();   // the block's exponentials are in memory
                lane_steps(Exponentials{ex, 0}, (int)j);
            } else if (E != kNoGuess && E != kEmpty) {
                bool tie;
                const fsx::Step st = block_step(y, E, true, &tie);
                if (lane == 0) sh.step[j] = pack_amounts(st);
                if (slot) {
                    const fsx::Step up = block_step(y, E + 1u, true, &tie);
                    if (lane == 0) step_up(slot, (int)j) = pack_amounts(up);
                }
            }
        }
    }
    rest = __syncthreads_or(rest) != 0;
    level = Level{kOneBits + 1u, kTopShift, 0, rest};
}
// The same for segments of two or four blocks.
template <bool kCount>
__device__ __noinline__ void exponentials_long(Logits row, Segs g, float mx, float inv_T, float* ex, Level& level) {
    ExactShared& sh = shared_memory();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const LaneTable tab(lane);
    const uint32_t bins = (uint32_t)__cvta_generic_to_shared(sh.bins);
    if (kCount)
        for (int j = tid; j < kBins; j += kThreads) sh.bins[j] = 0;
    __syncthreads();
    bool rest = false;
    const uint32_t blocks = (row.hi + kBlock - 1) / kBlock, per = 1u << (g.shift - 8);
    for (int j = warp; j < g.count; j += kWarps) {
        const uint32_t E = sh.E[j];
        const int slot = sh.slot[j];
        const bool lanes = lanes_at_hand(slot), amounts = !lanes && E != kNoGuess && E != kEmpty;
        fsx::Step total = fsx::step_identity(), total_up = fsx::step_identity();
        for (uint32_t b = j * per; b < min(blocks, (j + 1) * per); b += 2) {
            float x[2][2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int u = 0; u < 2; ++u) row.load4<true>((b + h) * kBlock + 8 * lane + 4 * u, x[h][u]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (b + h >= blocks) break;
                float y[8];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) y[4 * u + e] = expf_lanes_nonpositive(__fmul_rn(__fsub_rn(x[h][u][e], mx), inv_T), tab);
                    if (kCount) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint32_t bin = (kOneBits - __float_as_uint(y[4 * u + e])) >> kTopShift;
                            count_below(bins + 4 * bin, bin, (uint32_t)kBins);
                            rest |= bin >= (uint32_t)kBins;
                        }
                    }
                    *reinterpret_cast<float4*>(ex + (b + h) * kBlock + 8 * lane + 4 * u) = make_float4(y[4 * u], y[4 * u + 1], y[4 * u + 2], y[4 * u + 3]);
                }
                if (!amounts) continue;
                bool tie;
                total = fsx::then(total, block_step(y, E, true, &tie));
                if (slot) total_up = fsx::then(total_up, block_step(y, E + 1u, true, &tie));
            }
        }
        if (lanes) {
            __syncwarp();   // the segment's exponentials are in memory
            lane_steps(Exponentials{ex, 0}, j);
        } else if (amounts && lane == 0) {
            sh.step[j] = pack_amounts(total);
            if (slot) step_up(slot, j) = pack_amounts(total_up);
        }
    }
    rest = __syncthreads_or(rest) != 0;
    level = Level{kOneBits + 1u, kTopShift, 0, rest};
}
// The same for any row and temperature, and the sums before the segments.
__device__ __noinline__ void exponentials_any(Logits row, Segs g, float mx, float inv_T, float* ex) {
    ExactShared& sh = shared_memory();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const LaneTable tab(lane);
    for (int j = tid; j < g.count; j += kThreads) sh.cum[j] = 0.f;
    __syncthreads();
    const uint32_t blocks = (row.hi + kBlock - 1) / kBlock;
    for (uint32_t b = warp; b < blocks; b += kWarps) {
        float mass = 0.f;
        for (int u = 0; u < 2; ++u) {
            const uint32_t i = b * kBlock + u * 128 + 4 * lane;
            float x[4];
            row.load4(i, x);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float y = expf_lanes(__fmul_rn(__fsub_rn(x[e], mx), inv_T), tab);
                x[e] = i + e >= row.lo && i + e < row.hi ? y : 0.f;
                if (x[e] >= 0.f) mass += x[e];
            }
            *reinterpret_cast<float4*>(ex + i) = make_float4(x[0], x[1], x[2], x[3]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
        if (lane == 0) atomicAdd(&sh.cum[(b * kBlock) >> g.shift], mass);
    }
    masses_to_sums(g.count);
}

__device__ void sample_row(const StepArgs& a, float* scratch, int r) {
    ExactShared& sh = shared_memory();
    const int tid = threadIdx.x;
    const sampler_row_params p = a.rows[r];
    const uint32_t V = (uint32_t)a.vocab;
    float* logits = a.logits + p.logits_row * a.vocab;
    const bool raw_lp = (p.do_sample & SAMPLER_ROW_RAW_LOG_PROB) != 0;
    const RowHistory hist = row_history(a, r);
    __syncthreads();
    float raw_lse = 0.f;
    bool raw_ok = true;
    if (raw_lp) raw_lse = raw_log_partition<kThreads>(a, logits, hist, sh.scan_f, sh.scan_d, &raw_ok);
    mask_and_penalise<kThreads>(a, logits, p, r, hist, raw_lp && raw_ok);
    const bool top_p_active = p.top_p != 1.0f;
    const uint32_t lo = (uint32_t)(reinterpret_cast<uintptr_t>(logits) & 15) / 4, hi = lo + V;   // (a row may begin anywhere)
    const Logits in{logits - lo, lo, hi};
    const Segs g = segments_of(hi);
    float* ex = scratch;
    float* sorted = scratch + sampler_exact_pitch(a.vocab);
    const float inv_T = __fdiv_rn(1.0f, p.temperature);
#ifdef SAMPLER_EXACT_PROF
    __syncthreads();
    if (tid < kProfN) sh.prof[tid] = 0;
#endif
    __syncthreads();
    PROF_BEGIN;
    bool odd;
    const bool one_block = g.shift == 8;
    const bool fused = g.len() <= (uint32_t)(kFusedBlocks * kBlock);
    const float mx = one_block ? survey<false>(in, g, inv_T, true, &odd) : survey<true>(in, g, inv_T, fused, &odd);
    PROF_END(kProfMax);
    const bool plain = !odd && fabsf(mx) < CUDART_INF_F && inv_T > 0.f && inv_T < CUDART_INF_F;   // every exponential is between 0 and 1
    index_order_segments(g, lo, hi);
    Level level{kOneBits + 1u, kTopShift, 0, false};
    float norm = 0.f;
    if (plain && fused) {
        guess_binades(0, g.count, 0.f, CUDART_INF_F, -1.f, true);
        if (!one_block) top_p_active ? exponentials_long<true>(in, g, mx, inv_T, ex, level) : exponentials_long<false>(in, g, mx, inv_T, ex, level);
        else if (top_p_active) exponentials<true>(in, mx, inv_T, ex, level);
        else exponentials<false>(in, mx, inv_T, ex, level);
        PROF_END(kProfExp);
        ordered_sum(Exponentials{ex, 0}, 0, g.count, norm, CUDART_INF_F, -1.f, true);
    } else {
        exponentials_any(in, g, mx, inv_T, ex);
        if (top_p_active) count_level(level, ex, hi);
        PROF_END(kProfExp);
        ordered_sum(Exponentials{ex, 0}, 0, g.count, norm, CUDART_INF_F, -1.f);
    }
    const float inv_norm = __fdiv_rn(1.0f, norm);   // the largest probability, that of the maximum, and the shared reciprocal of the divisions
    const bool any = norm > 0.0f;                   // else every probability is NaN: none is kept
    const float min_thr = p.min_p > 0.0f ? __fmul_rn((float)(double)p.min_p, inv_norm) : 0.0f;
    const Row row{ex, sorted, lo, hi, norm, inv_norm, min_thr};
    const Probabilities probs{ex, 0, norm, inv_norm, min_thr};
    Kept kept{0, 0, 0, 0.f};
    float total = 0.0f;
    if (any && top_p_active) {
        kept = keep_top_p(row, g, level, p.top_p, p.rand_u);
        total = kept.total;
    } else if (any) {
        // approximate sums: those of the exponentials over the norm (with min-p they are taken anew)
        __syncthreads();
        for (int j = tid; j <= g.count; j += kThreads) sh.cum[j] *= inv_norm;
        ordered_sum(probs, 0, g.count, total, CUDART_INF_F, -1.f);
    }
    const bool uniform_fallback = !(total > 0.0f && isfinite(total)) || (top_p_active && kept.n == 0);
    long long kept_count = kept.n, last_kept = -1;
    bool looked = top_p_active;   // kept_count and, without top-p, last_kept are known
    auto look = [&] {
        if (looked) return;
        looked = true;
        uint32_t n = 0;
        int last = -1;
        for (uint32_t i = lo + tid; any && i < hi; i += kThreads)
            if (probability(ex[i], norm, inv_norm) >= min_thr) { ++n; last = (int)i; }
        kept_count = block_sum(n, sh.scan_u);
        last_kept = block_reduce(last, [](int x, int y) { return max(x, y); }, sh.red_i);
    };
    const long long x0 = a.extra_offsets ? a.extra_offsets[r] : 0, x1 = a.extra_offsets ? a.extra_offsets[r + 1] : 0;
    const bool list = x1 > x0 && top_p_active && !uniform_fallback && list_kept(row, kept.placed);
    for (long long k = -1; k < x1 - x0; ++k) {   // the row's own draw, then the further ones (sampler.cpp:1065)
        const float u = k < 0 ? p.rand_u : a.extra_rand_u[x0 + k];
        long long pick = -1;
        float pick_p = 0.f;
        if (uniform_fallback) look();
        else {
            const float rr = __fmul_rn(total, u);
            if (!top_p_active) {
                pick = find_draw(probs, g.count, hi, nullptr, rr, pick_p);
                if (pick < 0) {   // rounding left r at or beyond the total: the last kept element
                    look();
                    pick = last_kept;
                    pick_p = probability(ex[pick < 0 ? lo : pick], norm, inv_norm);
                }
                pick -= lo;
            } else {
                long long rank = find_draw(Sorted{sorted, 0}, kept.segs, kept.n, sorted, rr, pick_p);
                if (rank < 0) {   // the last of the kept ones
                    rank = (long long)kept.n - 1;
                    pick_p = rank < (long long)kept.placed ? sorted[rank] : 0.f;
                }
                pick = list && pick_p > 0.f ? listed_index((uint32_t)rank, pick_p) : -1;
                if (pick < 0) pick = index_of_rank(row, (uint32_t)rank, pick_p);
                pick -= lo;
            }
        }
        if (tid == 0) {
            float lp;
            if (uniform_fallback) {
                // non-finite or empty mass: the reference draws an index uniformly (sampler.cpp:1047-1059)
                const long long n = kept_count > 0 ? kept_count : (long long)V;
                long long q = (long long)(u * (float)n);
                if (q > n - 1) q = n - 1;
                pick = q < (long long)V ? q : (long long)V - 1;
                lp = logf(1.0f / (float)n);
            } else {
                lp = logf(pick_p) - logf(total);
                if (raw_lp) lp = raw_log_prob(a, logits, hist, pick, raw_lse, raw_ok);
            }
            if (k < 0) { a.out_token[r] = pick; a.out_log_prob[r] = lp; }
            else { a.extra_out_token[x0 + k] = pick; a.extra_out_log_prob[x0 + k] = lp; }
        }
    }
#ifdef SAMPLER_EXACT_PROF
    if (tid == 0 && blockIdx.x % 37 == 0)
        printf("row %d kept %u: max %lld exp %lld | guesses %lld steps %lld walk %lld (misses %lld) | ranks %lld gather %lld same %lld place %lld | find %lld index %lld + %lld cycles; walk: tiles %lld in %lld, slots %lld in %lld, serial %lld\n", r, kept.n, sh.prof[kProfMax],
               sh.prof[kProfExp], sh.prof[kProfGuess], sh.prof[kProfSteps], sh.prof[kProfWalk], sh.prof[kProfMisses], sh.prof[kProfRank], sh.prof[kProfGather], sh.prof[kProfSame],
               sh.prof[kProfPlace], sh.prof[kProfFind], sh.prof[kProfIndex], sh.prof[kProfIndex2], sh.prof[kProfTiles], sh.prof[kProfTile], sh.prof[kProfSlots], sh.prof[kProfSlot], sh.prof[kProfSerial]);
#endif
}

__global__ void __launch_bounds__(kThreads, 1) sampler_exact_kernel(StepArgs a, float* scratch) {
    ExactShared& sh = shared_memory();
    const int tid = threadIdx.x;
    float* own = scratch + (size_t)blockIdx.x * 2 * sampler_exact_pitch(a.vocab);
    uint32_t seen = 0;   // rows of this kernel among those looked at: they are dealt to the CTAs in turn
    for (int base = 0; base < a.num_rows; base += kThreads) {
        bool take = false;
        if (base + tid < a.num_rows) {
            const sampler_row_params& p = a.rows[base + tid];
            take = whole_vocabulary_row(p, a.vocab) && p.logits_row >= 0 && p.logits_row < a.num_logit_rows;   // (else reported by the first kernel)
        }
        if (!__syncthreads_or(take)) continue;
        uint32_t n;
        const uint32_t at = seen + block_scan_exclusive(take ? 1u : 0u, sh.scan_u, &n);
        const uint32_t mine = __ballot_sync(0xffffffffu, take && at % gridDim.x == blockIdx.x);
        if ((tid & 31) == 0) sh.queue[tid >> 5] = mine;
        __syncthreads();
        for (int w = 0; w < kWarps; ++w)
            for (uint32_t rows = sh.queue[w]; rows; rows &= rows - 1) sample_row(a, own, base + 32 * w + __ffs(rows) - 1);
        seen += n;
        __syncthreads();
    }
    // The step's first kernel has its rows done: what follows in the stream waits for this one only.
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Both forms; NaN where they differ.
__global__ void expf_selftest_kernel(const float* in, float* out, long long n) {
    const int lane = threadIdx.x & 31;
    const LaneTable tab(lane);
    for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x - lane; i0 < n; i0 += (long long)gridDim.x * blockDim.x) {
        const long long i = i0 + lane;
        const float x = i < n ? in[i] : 0.f;
        const float y = expf_lanes(x, tab), z = expf_lanes_nonpositive(fminf(x, 0.f), tab);
        if (i < n) out[i] = x <= 0.f && __float_as_uint(y) != __float_as_uint(z) ? CUDART_NAN_F : y;
    }
}

}  // namespace

cudaError_t launch_expf_selftest(const float* in, float* out, long long n, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    expf_selftest_kernel<<<592, 256, 0, stream>>>(in, out, n);
    return cudaGetLastError();
}

size_t sampler_exact_scratch_bytes(int ctas, long long vocab) { return (size_t)ctas * 2 * sampler_exact_pitch(vocab) * sizeof(float); }

cudaError_t launch_sampler_exact(const StepArgs& a, float* scratch, int ctas, cudaStream_t stream) {
    if (a.num_rows <= 0 || ctas <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(sampler_exact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ExactShared));
    if (e != cudaSuccess) return e;
    // Programmatic dependent launch: the rows of the two kernels of a step have nothing to do with one another, so the CTAs of this one
    // start where the first one's leave room.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.num_rows < ctas ? a.num_rows : ctas));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = sizeof(ExactShared);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, sampler_exact_kernel, a, scratch);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace sampler
