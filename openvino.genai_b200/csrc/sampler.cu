// Sampler step for sm_100a: one kernel launch for the whole batch, one CTA per sampled row.
//
// Phases of a row (src/cpp/src/sampling/logit_processor.hpp:28-112 fixes the order):
//   1. penalties, in place on the logits row, one thread per distinct history id, in the
//      reference's float (+) double -> float arithmetic with every step individually rounded;
//   2. greedy rows: strict-> argmax with lowest-index ties over the row (one HBM pass);
//   3. multinomial rows with an active top-k: the reference keeps a K-element min-heap whose final
//      ARRAY ORDER feeds every later float sum and the draw itself, so the order is reproduced
//      exactly: 15 producer warps stream the row with 16-byte loads, keep only elements above a
//      conservative lower bound of the heap minimum, and append them in index order to a ring;
//      warp 0 replays libstdc++'s pop_heap / push_heap on the few hundred that really enter, with
//      the heap spread over its registers (K <= 64) or by one lane over shared memory.  Softmax,
//      min-p, top-p and the draw then run over <= K elements in the same warp, in the reference's
//      order of operations.  A step (both launches, no penalties, logits in place) of 256 rows x
//      151936, K 50: 301 -> 91 us (the serial replay, about 400 replacements of 250 cycles with two
//      rows per SM, is what a row waits for; reading the rows takes 24 us); 5 rows x 32000: 215 -> 50 us;
//   4. multinomial rows over the full vocabulary are left to sampler_exact_kernel (sampler_exact.cu), which reproduces the
//      reference's index-order and sorted-order float sums exactly and runs beside this kernel where there is room.
// Greedy rows are bound by reading the row once (HBM from some 100 rows on, latency below); top-k rows by the serial replay;
// what the whole-vocabulary rows wait for is said in sampler_exact.cu.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "../../include/sampler_b200.h"
#include "sampler_kernels.h"
#include "sampler_rows.cuh"

namespace sampler {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kProducerWarps = kWarps - 1;            // warps 1..15 filter, warp 0 replays the heap
constexpr int kProducerThreads = 32 * kProducerWarps;
constexpr int kPerThread = 8;                         // elements a producer thread filters per round
constexpr int kChunk = kProducerThreads * kPerThread; // elements per filter round
constexpr int kMaxTopK = 1024;                        // heap capacity in shared memory
constexpr int kRegTopK = 64;                          // heaps up to here live in the registers of warp 0
constexpr int kRing = 4096;                           // candidates between producers and consumer; a power of two, at least kChunk:
                                                      // 8192 gave top-k rows nothing (90.7 | 90.6 us) and cost the others their L1
                                                      // (256 greedy rows 31.9 -> 31.5 us a step)
static_assert(kRing >= kChunk && (kRing & (kRing - 1)) == 0, "a round must fit the ring");

struct __align__(8) Cand {
    float v;
    int idx;
};

// The aligned forms of the barrier instructions ask for a converged warp; the callers come from loops and branches whose
// trip counts and conditions differ between lanes, so the warp is brought together first.
__device__ __forceinline__ void named_sync(int id, int count) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ int named_count(int id, int count, bool pred) {   // barrier that returns how many threads' pred holds
    int n;
    __syncwarp();
    asm volatile("{ .reg .pred p; setp.ne.s32 p, %3, 0; barrier.cta.red.popc.aligned.u32 %0, %1, %2, p; }" : "=r"(n) : "r"(id), "r"(count), "r"((int)pred) : "memory");
    return n;
}

// expf as "exp in double, rounded once to float": within an ulp of glibc's expf and equal to it
// except where glibc's own result is not the correctly rounded one.
__device__ __forceinline__ float exp_as_float(float x) { return (float)exp((double)x); }

// ---- libstdc++ heap primitives on (value, index) pairs with comp(a, b) = a.v > b.v (min-heap) ----
__device__ void push_heap_from(Cand* h, int hole, int top, Cand value) {
    int parent = (hole - 1) / 2;
    while (hole > top && h[parent].v > value.v) {
        h[hole] = h[parent];
        hole = parent;
        parent = (hole - 1) / 2;
    }
    h[hole] = value;
}

__device__ void adjust_heap(Cand* h, int hole, int len, Cand value) {
    const int top = hole;
    int child = hole;
    while (child < (len - 1) / 2) {
        child = 2 * (child + 1);
        const Cand right = h[child], left = h[child - 1];   // both children in flight together
        const bool take_left = right.v > left.v;
        if (take_left) --child;
        h[hole] = take_left ? left : right;
        hole = child;
    }
    if ((len & 1) == 0 && child == (len - 2) / 2) {
        child = 2 * (child + 1);
        h[hole] = h[child - 1];
        hole = child - 1;
    }
    push_heap_from(h, hole, top, value);
}

__device__ void make_heap(Cand* h, int len) {
    if (len < 2) return;
    for (int parent = (len - 2) / 2;; --parent) {
        adjust_heap(h, parent, len, h[parent]);
        if (parent == 0) return;
    }
}

// make_heap by one warp: the parents of one level own disjoint subtrees, so a level's sift-downs run side by side and
// leave the same array as the library's loop from the last parent to the first.
__device__ void make_heap_warp(Cand* h, int len, int lane) {
    if (len < 2) return;
    const int last = (len - 2) / 2;
    for (int lvl = 31 - __clz(last + 1); lvl >= 0; --lvl) {
        const int first = (1 << lvl) - 1, end = min(last, 2 * first);   // parents first .. end
        for (int p = first + lane; p <= end; p += 32) adjust_heap(h, p, len, h[p]);
        __syncwarp();
    }
}

// Order of the floats as signed integers; both zeros get the key of +0, so equal floats have equal keys (NaN apart).
__device__ __forceinline__ int order_key(float x) {
    const int b = __float_as_int(__fadd_rn(x, 0.0f));
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float order_value(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// A heap of K <= 64 entries in the registers of one warp, for the replay of the top-k path: pop_heap, back() = x, push_heap
// (src/cpp/src/sampling/logit_transformers.hpp:240-246) without a walk through memory.
//
// Lane j holds the children of node j, so the comparison of two siblings is local; the root is in every lane.  pop_heap
// takes the hole down the smaller-child path to a leaf and the last entry up the same path again: along the path the values
// ascend, so the last entry ends at the depth where they begin to exceed it, and every entry above moves one step up.  A
// lane tells from one vote over all sibling comparisons whether its node is on the path (its ancestors' bits are constants
// of the lane) and from its own and its chosen child's value what the slot receives.  push_heap does the same along the
// constant path from entry K - 1 to the root; slot `a` is the child on that path (the left one elsewhere), so that its
// shuffle needs no selection first.  Equal values go right and stay below, as the library's comparisons have it.
//
// Bound by latency: about ten dependent steps of a comparison and a selection (11 cycles) or a shuffle (26).  145 cycles per
// replacement back to back, 208 with the search for the next candidate (250 with a second row on the SM), against 750 for one
// lane over shared memory.
struct RegHeap {
    int a, b, ai, bi;   // children of node `lane`: order keys and vocabulary indices
    int root, root_i;
};
struct RegHeapLane {    // constants of the lane
    uint32_t anc_mask, anc_bits;   // ancestors of node `lane`, and those of them whose slot a is on the way to it
    int flip;                      // 1: slot a is the right child
    int a_min, b_min;              // raises a slot that is not in the popped heap to the largest key
    int a_src, b_src;              // the lanes that hold the children of the slots (lane 31 has none in a popped heap)
    int chain_src, last_lane;      // the lane that holds this lane's own node; the one that holds entry K - 1
    bool on_chain, is_root;        // slot a is on the way from entry K - 1 to the root
    int K, lane;

    __device__ RegHeapLane(int K_, int lane_) : K(K_), lane(lane_) {
        flip = 0;
        on_chain = false;
        is_root = lane == 0;
        for (int n = K - 1; n > 0; n = (n - 1) / 2)
            if ((n - 1) / 2 == lane) { on_chain = true; flip = (n & 1) ? 0 : 1; }
        anc_mask = anc_bits = 0;
        for (int n = lane; n > 0;) {
            const int up = (n - 1) / 2;
            bool up_flip = false;   // of lane `up`, as above
            for (int m = K - 1; m > 0; m = (m - 1) / 2)
                if ((m - 1) / 2 == up) up_flip = !(m & 1);
            anc_mask |= 1u << up;
            if (up_flip == !(n & 1)) anc_bits |= 1u << up;
            n = up;
        }
        a_min = a_node() < K - 1 ? (int)0x80000000 : 0x7fffffff;
        b_min = b_node() < K - 1 ? (int)0x80000000 : 0x7fffffff;
        a_src = min(a_node(), 31);
        b_src = min(b_node(), 31);
        chain_src = lane > 0 ? (lane - 1) / 2 : 0;
        last_lane = K > 1 ? (K - 2) / 2 : 0;
    }
    __device__ __forceinline__ int a_node() const { return 2 * lane + 1 + flip; }
    __device__ __forceinline__ int b_node() const { return 2 * lane + 2 - flip; }

    __device__ RegHeap load(const Cand* h) const {
        const int an = a_node(), bn = b_node();
        const Cand x = h[an < K ? an : 0], y = h[bn < K ? bn : 0], z = h[0];
        return RegHeap{an < K ? order_key(x.v) : 0x7fffffff, bn < K ? order_key(y.v) : 0x7fffffff, x.idx, y.idx, order_key(z.v), z.idx};
    }
    __device__ void store(const RegHeap& h, Cand* out) const {
        if (a_node() < K) out[a_node()] = Cand{order_value(h.a), h.ai};
        if (b_node() < K) out[b_node()] = Cand{order_value(h.b), h.bi};
        if (lane == 0) out[0] = Cand{order_value(h.root), h.root_i};
    }

    // The heap after pop_heap; entry K - 1 is left open.  Slots outside the popped heap count as the largest key (which no
    // float has): they are chosen by nobody, never "at or below" the last entry, and the open one takes any value.
    __device__ __forceinline__ RegHeap popped(const RegHeap& h) const {
        RegHeap n;
        const int av = max(h.a, a_min), bv = max(h.b, b_min);
        const bool pick_a = bv > max(h.a - flip, a_min);   // the smaller child, the right one of equals
        const int cv = pick_a ? av : bv, ci = pick_a ? h.ai : h.bi, src = pick_a ? a_src : b_src;
        const uint32_t bits = __ballot_sync(0xffffffffu, pick_a);
        const int gv = __shfl_sync(0xffffffffu, cv, src), gi = __shfl_sync(0xffffffffu, ci, src);   // the chosen child's own choice
        const int last_v = __shfl_sync(0xffffffffu, h.a, last_lane), last_i = __shfl_sync(0xffffffffu, h.ai, last_lane);
        const int top_v = __shfl_sync(0xffffffffu, cv, 0), top_i = __shfl_sync(0xffffffffu, ci, 0);
        const bool move = (bits & anc_mask) == anc_bits && cv <= last_v;   // on the path, and passed by the last entry
        const bool wa = move && pick_a, wb = move && !pick_a;
        const bool deeper = gv <= last_v;
        const int nv = deeper ? gv : last_v, ni = deeper ? gi : last_i;
        n.a = wa ? nv : av; n.ai = wa ? ni : h.ai;
        n.b = wb ? nv : bv; n.bi = wb ? ni : h.bi;
        const bool up = top_v <= last_v;
        n.root = up ? top_v : last_v;
        n.root_i = up ? top_i : last_i;
        return n;
    }

    // push_heap of x into the open entry K - 1 of a popped heap
    __device__ __forceinline__ void push(RegHeap& h, int x, int xi) const {
        int pv = __shfl_sync(0xffffffffu, h.a, chain_src), pi = __shfl_sync(0xffffffffu, h.ai, chain_src);
        if (is_root) { pv = h.root; pi = h.root_i; }
        const bool here = on_chain && h.a > x, down = on_chain && pv > x;
        const int sv = here ? x : h.a, si = here ? xi : h.ai;
        h.a = down ? pv : sv;
        h.ai = down ? pi : si;
        const bool top = h.root > x;
        h.root = top ? x : h.root;
        h.root_i = top ? xi : h.root_i;
    }
};

// The same replacement (pop_heap, back() = x, push_heap) for heaps of more than kRegTopK entries, by one lane over shared
// memory: written with 32-bit shared-memory addresses and paired 8-byte accesses so that one level of the heap costs
// one shared-memory round trip.  The writes of the popped minimum and of x into slot k - 1 that
// libstdc++ performs in between are dead (the slot is not read before it is overwritten).
__device__ __forceinline__ void lds_cand(uint32_t addr, float& v, int& i) {
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=f"(v), "=r"(i) : "r"(addr));
}
__device__ __forceinline__ void sts_cand(uint32_t addr, float v, int i) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "f"(v), "r"(i) : "memory");
}
__device__ __forceinline__ void replace_min_shared(uint32_t base, int k, float xv, int xi) {
    if (k > 1) {
        const int len = k - 1;
        float lastv;
        int lasti;
        lds_cand(base + 8u * len, lastv, lasti);
        // __adjust_heap(first, 0, len, last)
        int hole = 0, child = 0;
        const int half = (len - 1) / 2;
        while (child < half) {
            child = 2 * (child + 1);
            float rv, lv;
            int ri, li;
            lds_cand(base + 8u * child, rv, ri);
            lds_cand(base + 8u * (child - 1), lv, li);
            const bool take_left = rv > lv;
            if (take_left) --child;
            sts_cand(base + 8u * hole, take_left ? lv : rv, take_left ? li : ri);
            hole = child;
        }
        if ((len & 1) == 0 && child == (len - 2) / 2) {
            child = 2 * (child + 1);
            float v;
            int i;
            lds_cand(base + 8u * (child - 1), v, i);
            sts_cand(base + 8u * hole, v, i);
            hole = child - 1;
        }
        // __push_heap(first, hole, 0, last)
        while (hole > 0) {
            const int parent = (hole - 1) / 2;
            float pv;
            int pi;
            lds_cand(base + 8u * parent, pv, pi);
            if (!(pv > lastv)) break;
            sts_cand(base + 8u * hole, pv, pi);
            hole = parent;
        }
        sts_cand(base + 8u * hole, lastv, lasti);
    }
    // push_heap(first, first + k) with x in the last slot
    int hole = k - 1;
    while (hole > 0) {
        const int parent = (hole - 1) / 2;
        float pv;
        int pi;
        lds_cand(base + 8u * parent, pv, pi);
        if (!(pv > xv)) break;
        sts_cand(base + 8u * hole, pv, pi);
        hole = parent;
    }
    sts_cand(base + 8u * hole, xv, xi);
}

// ---- libstdc++ partial_sort / sort on (value, index) pairs with comp(a, b) = a.v > b.v --------------
// TopPFilter sorts candidates with std::partial_sort and std::sort; neither is stable, so to scan
// equal probabilities in the reference's order the algorithms themselves are restated:
// heap-select + sort-heap, and introsort (median-of-three, threshold 16, depth 2*floor(log2 n))
// with the final guarded / unguarded insertion pass.
__device__ __forceinline__ bool desc(const Cand& a, const Cand& b) { return a.v > b.v; }
__device__ __forceinline__ void swap_cand(Cand& a, Cand& b) { const Cand t = a; a = b; b = t; }

__device__ void pop_heap_into(Cand* first, int len, Cand* result) {  // __pop_heap(first, first + len, result)
    const Cand value = *result;
    *result = first[0];
    adjust_heap(first, 0, len, value);
}

__device__ void std_partial_sort(Cand* v, int middle, int n) {
    make_heap(v, middle);
    for (int i = middle; i < n; ++i)
        if (desc(v[i], v[0])) pop_heap_into(v, middle, &v[i]);
    for (int last = middle; last > 1;) {
        --last;
        pop_heap_into(v, last, &v[last]);
    }
}

__device__ void unguarded_linear_insert(Cand* v, int last) {
    const Cand val = v[last];
    int next = last - 1;
    while (desc(val, v[next])) {
        v[last] = v[next];
        last = next;
        --next;
    }
    v[last] = val;
}

__device__ void insertion_sort(Cand* v, int first, int last) {
    if (first == last) return;
    for (int i = first + 1; i != last; ++i) {
        if (desc(v[i], v[first])) {
            const Cand val = v[i];
            for (int j = i; j > first; --j) v[j] = v[j - 1];
            v[first] = val;
        } else {
            unguarded_linear_insert(v, i);
        }
    }
}

__device__ void move_median_to_first(Cand* v, int result, int a, int b, int c) {
    if (desc(v[a], v[b])) {
        if (desc(v[b], v[c])) swap_cand(v[result], v[b]);
        else if (desc(v[a], v[c])) swap_cand(v[result], v[c]);
        else swap_cand(v[result], v[a]);
    } else if (desc(v[a], v[c])) swap_cand(v[result], v[a]);
    else if (desc(v[b], v[c])) swap_cand(v[result], v[c]);
    else swap_cand(v[result], v[b]);
}

__device__ int unguarded_partition(Cand* v, int first, int last, int pivot) {
    for (;;) {
        while (desc(v[first], v[pivot])) ++first;
        --last;
        while (desc(v[pivot], v[last])) --last;
        if (!(first < last)) return first;
        swap_cand(v[first], v[last]);
        ++first;
    }
}

__device__ void std_sort(Cand* v, int n) {
    if (n == 0) return;
    int lg = 0;
    for (int t = n; t > 1; t >>= 1) ++lg;
    // explicit stack instead of the recursive call on [cut, last): the two halves are independent
    int stack_first[48], stack_last[48], stack_depth[48];
    int sp = 0;
    stack_first[sp] = 0; stack_last[sp] = n; stack_depth[sp] = 2 * lg; ++sp;
    while (sp > 0) {
        --sp;
        int first = stack_first[sp], last = stack_last[sp], depth = stack_depth[sp];
        while (last - first > 16) {
            if (depth == 0) {
                std_partial_sort(v + first, last - first, last - first);
                break;
            }
            --depth;
            const int mid = first + (last - first) / 2;
            move_median_to_first(v, first, first + 1, mid, last - 1);
            const int cut = unguarded_partition(v, first + 1, last, first);
            stack_first[sp] = cut; stack_last[sp] = last; stack_depth[sp] = depth; ++sp;
            last = cut;
        }
    }
    if (n > 16) {
        insertion_sort(v, 0, 16);
        for (int i = 16; i < n; ++i) unguarded_linear_insert(v, i);
    } else {
        insertion_sort(v, 0, n);
    }
}

// ---- block reductions -------------------------------------------------------------------------------
struct ArgMax {
    float v;
    int i;
};
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
    // strict '>' with the lowest index among equals; NaN never wins (sampler.cpp:952-961)
    if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
    return a;
}

// Order-preserving 32-bit key of a float: larger float <=> larger unsigned key.
__device__ __forceinline__ uint32_t float_key(float x) {
    const uint32_t b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

constexpr int kSortWarp = 128;   // candidates one warp ranks by counting
struct Shared {
    Cand heap[kMaxTopK];
    Cand ring[kRing];          // survivors of the filter, in index order
    int head, tail;            // entries published / taken (running counts)
    int idle;                  // the consumer's empty polls since the producers' last step
    int done;                  // every round is published
    int give_up;               // a wait ran out
    float tau;                 // consumer's heap minimum as the producers see it (may lag, never leads)
    int warp_cnt[2][kProducerWarps];
    float prob[kMaxTopK];      // exponentials of the heap entries
    Cand sorted[kSortWarp];
    float red_f[kWarps];
    double red_d[kWarps];
    int red_i[kWarps];
    unsigned long long red_u[kWarps];
    ArgMax red_a[kWarps];
};

// ---- phase 3 tail: softmax / min-p / top-p over the K heap entries, then the draws, one thread -------
// Mirrors TemperatureLogitTransform, MinPFilter, TopPFilter (logit_transformers.hpp:90-362) and
// Sampler::_multinomial_sample (sampler.cpp:979-1095) statement by statement.  The distribution is
// built once; a request with num_return_sequences > 1 draws from it several times (sampler.cpp:1065).
struct TopKDist {
    int n;          // kept candidates, v[0 .. n)
    bool defer;     // expf deferred into the draw (top-k without top-p / min-p): v holds scaled logits
    bool uniform;   // non-finite or empty mass: uniform draws
    float mx, sum;  // deferred form: maximum and float sum of the exponentials
    float total;    // normal form: float sum of the kept probabilities
};

// TopPFilter::apply: partial sorts of the top 16, 32, ... 1024 until the running float sum exceeds top_p, else a full
// sort (logit_transformers.hpp:94-139).  Returns the number of kept candidates, v[0 .. n).
__device__ int top_p_serial(Cand* v, int n, float top_p) {
    const double tp = (double)top_p;
    for (int step = 16; step <= 1024; step *= 2) {
        if (n <= step) break;
        std_partial_sort(v, step, n);
        float sum = 0.0f;
        for (int i = 0; i < step; ++i) {
            sum += v[i].v;
            if ((double)sum > tp) return i + 1;
        }
    }
    std_sort(v, n);
    float sum = 0.0f;
    int keep = 0;
    for (int i = 0; i < n; ++i) {
        sum += v[i].v;
        ++keep;
        if ((double)sum > tp) break;
    }
    return keep;
}

__device__ TopKDist build_top_k_dist(Cand* v, float* ex, int n, const sampler_row_params& p) {
    TopKDist d{n, false, false, 0.f, 0.f, 0.f};
    const bool min_p_active = p.min_p > 0.0f;
    d.defer = p.top_p == 1.0f && !min_p_active;
    const float T = p.temperature;
    if (d.defer) {
        if (T != 1.0f) {
            const float f = 1.0f / T;
            for (int i = 0; i < n; ++i) v[i].v *= f;
        }
        float mx = v[0].v;
        for (int i = 1; i < n; ++i) if (v[i].v > mx) mx = v[i].v;
        float sum = 0.0f;
        for (int i = 0; i < n; ++i) { ex[i] = exp_as_float(v[i].v - mx); sum += ex[i]; }
        d.uniform = !(sum > 0.0f && isfinite(sum));
        if (d.uniform) sum = (float)n;
        d.mx = mx; d.sum = sum;
        return d;
    }
    {   // softmax(logits / T) over the heap array, in array order
        float mx = v[0].v;
        for (int i = 1; i < n; ++i) if (v[i].v > mx) mx = v[i].v;
        float sum = 0.0f;
        if (T == 1.0f) {
            for (int i = 0; i < n; ++i) { v[i].v = exp_as_float(v[i].v - mx); sum += v[i].v; }
        } else {
            const float f = 1.0f / T;
            for (int i = 0; i < n; ++i) { v[i].v = exp_as_float((v[i].v - mx) * f); sum += v[i].v; }
        }
        for (int i = 0; i < n; ++i) v[i].v = __fdiv_rn(v[i].v, sum);
    }
    if (min_p_active) {
        float mx = 0.0f;
        int arg = 0;
        for (int i = 0; i < n; ++i) if (v[i].v > mx) { mx = v[i].v; arg = i; }
        const float thr = (float)(double)p.min_p * mx;
        int m = 0;
        for (int i = 0; i < n; ++i) if (v[i].v >= thr) v[m++] = v[i];
        if (m == 0) { v[0] = v[arg]; m = 1; }
        n = m;
    }
    if (p.top_p != 1.0f) n = top_p_serial(v, n, p.top_p);
    float total = 0.0f;
    for (int i = 0; i < n; ++i) total += v[i].v;
    d.n = n;
    d.total = total;
    d.uniform = !(total > 0.0f && isfinite(total));
    return d;
}

// The same distribution built by one warp: every element's own arithmetic in parallel, the float sums in array order as
// above.  The sort of top-p is a rank by counting when all values differ - the sorted order is then unique, and the
// running sum stops at the same element whichever of the partial sorts finds it - and the library's algorithms otherwise.
// One thread took 40k cycles for K = 50, a warp takes about 4k.  Returns the array that holds the kept candidates.
__device__ const Cand* build_top_k_dist_warp(Shared& sh, int n, const sampler_row_params& p, int lane, TopKDist& d) {
    Cand* v = sh.heap;
    const bool min_p_active = p.min_p > 0.0f;
    d = TopKDist{n, p.top_p == 1.0f && !min_p_active, false, 0.f, 0.f, 0.f};
    const float T = p.temperature, f = 1.0f / T;
    if (d.defer && T != 1.0f)
        for (int i = lane; i < n; i += 32) v[i].v *= f;
    __syncwarp();
    float mx = -CUDART_INF_F;
    for (int i = lane; i < n; i += 32) mx = fmaxf(mx, v[i].v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    for (int i = lane; i < n; i += 32) sh.prob[i] = exp_as_float(d.defer || T == 1.0f ? v[i].v - mx : (v[i].v - mx) * f);
    __syncwarp();
    float sum = 0.0f;
#pragma unroll 8
    for (int i = 0; i < n; ++i) sum += sh.prob[i];
    if (d.defer) {
        d.uniform = !(sum > 0.0f && isfinite(sum));
        if (d.uniform) sum = (float)n;
        d.mx = mx; d.sum = sum;
        return v;
    }
    for (int i = lane; i < n; i += 32) v[i].v = __fdiv_rn(sh.prob[i], sum);
    __syncwarp();
    if (min_p_active) {
        float top = 0.0f;
        for (int i = lane; i < n; i += 32) top = fmaxf(top, v[i].v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float thr = (float)(double)p.min_p * top;
        int m = 0;
        unsigned arg = 0xffffffffu;
        for (int base = 0; base < n; base += 32) {   // in place: an entry moves down, past the reads of its own group at most
            const int i = base + lane;
            const Cand c = i < n ? v[i] : Cand{0.f, 0};
            if (i < n && top > 0.0f && c.v == top) arg = min(arg, (unsigned)i);
            const bool keep = i < n && c.v >= thr;
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (keep) v[m + __popc(mask & ((1u << lane) - 1u))] = c;
            m += __popc(mask);
            __syncwarp();
        }
        arg = __reduce_min_sync(0xffffffffu, arg);
        if (m == 0) {   // nothing was moved
            const Cand c = v[arg == 0xffffffffu ? 0 : arg];
            __syncwarp();
            if (lane == 0) v[0] = c;
            m = 1;
            __syncwarp();
        }
        n = m;
    }
    if (p.top_p != 1.0f) {
        bool ranked = n <= kSortWarp;
        if (ranked) {
            bool same = false;
            for (int i = lane; i < n; i += 32) {
                const Cand c = v[i];
                int rank = 0, other = 0;
#pragma unroll 4
                for (int j = 0; j < n; ++j) {
                    const float w = v[j].v;
                    rank += w > c.v ? 1 : 0;
                    other += w > c.v || w < c.v ? 0 : 1;   // equal or unordered: the element itself only
                }
                same |= other != 1;
                sh.sorted[rank] = c;
            }
            ranked = !__any_sync(0xffffffffu, same);
            __syncwarp();
        }
        if (ranked) {
            v = sh.sorted;
            const double tp = (double)p.top_p;
            float run = 0.0f;
            int keep = 0;
            while (keep < n) {
                run += v[keep].v;
                ++keep;
                if ((double)run > tp) break;
            }
            n = keep;
        } else {
            if (lane == 0) n = top_p_serial(v, n, p.top_p);
            n = __shfl_sync(0xffffffffu, n, 0);
            __syncwarp();
        }
    }
    float total = 0.0f;
#pragma unroll 8
    for (int i = 0; i < n; ++i) total += v[i].v;
    d.n = n;
    d.total = total;
    d.uniform = !(total > 0.0f && isfinite(total));
    return v;
}

// One draw with the uniform number u: the candidate's vocabulary index and its log-probability.  `ex`: the exponentials of
// the deferred form.
__device__ void draw_top_k(const Cand* v, const TopKDist& d, const float* ex, float u, float* out_p, long long* out_idx) {
    const int n = d.n;
    if (d.defer) {
        const float log_sum = logf(d.sum) + (d.uniform ? 0.0f : d.mx);
        const float r = d.sum * u;
        float run = 0.0f;
        int pick = n - 1;
        for (int i = 0; i < n; ++i) {
            run += d.uniform ? 1.0f : ex[i];
            if (run > r) { pick = i; break; }
        }
        *out_p = d.uniform ? logf(1.0f / (float)n) : v[pick].v - log_sum;
        *out_idx = v[pick].idx;
        return;
    }
    if (d.uniform) {
        int pick = (int)(u * (float)n);
        if (pick > n - 1) pick = n - 1;
        *out_p = logf(1.0f / (float)n);
        *out_idx = v[pick].idx;
        return;
    }
    const float log_total = logf(d.total);
    const float r = d.total * u;
    float run = 0.0f;
    int pick = n - 1;
    for (int i = 0; i < n; ++i) {
        run += v[i].v;
        if (run > r) { pick = i; break; }
    }
    *out_p = logf(v[pick].v) - log_total;
    *out_idx = v[pick].idx;
}

// The ring's counts in shared memory: what a thread wrote before it stored a count is visible to whoever loads that count.
__device__ __forceinline__ int load_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
    return v;
}
__device__ __forceinline__ void store_release(int* p, int v) {
    asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}

// ---- the filter and the ring between it and the replay ------------------------------------------------------
// Warps 1..15 read the row in rounds of kChunk elements, keep what exceeds a lower bound of the heap minimum, and append it
// in index order to a ring in shared memory that warp 0 empties.  The bound is the consumer's minimum as last published or
// the K-th largest of the threads' own maxima so far (K distinct elements of the prefix; taken after every round whose
// number is a power of two), whichever is larger; so the filter does not wait for the replay, only for room.  The first
// round is filtered in three parts of 60, 180 and 240 threads with a bound after each: 4 k candidates of a 150 k row
// became about 1 k, 400 of which enter.  A part with T threads bounds heaps of up to T entries (its K-th largest maximum
// exists): 60 threads serve the usual K of 20 to 50 after their 480 elements, which all pass; heaps of 61 to 240 entries
// take their first bound from the second part, larger ones from the third.  One barrier among the producers per step: passing
// it, all entries of the steps before are written, and the count is published.
template <class Load>
__device__ __forceinline__ void produce_candidates(Shared& sh, int K, long long V, long long start, int rounds, float (&x)[kPerThread],
                                                   float (&xn)[kPerThread], Load&& load_round, int wait_polls, int ptid, int pwarp, int lane) {
    volatile int* v_give_up = &sh.give_up;
    float bound = -CUDART_INF_F, top = -CUDART_INF_F;   // top: the thread's maximum so far
    int head = 0;
    for (int step = rounds > 0 ? 0 : 3; step < rounds + 2; ++step) {
        const int c = step < 2 ? 0 : step - 2;   // the round; steps 0, 1, 2 are the parts of round 0
        const int t_lo = step == 1 ? 60 : step == 2 ? 240 : 0, t_hi = step == 0 ? 60 : step == 1 ? 240 : kProducerThreads;
        if ((step == 0 || step > 2) && c + 1 < rounds) load_round(c + 1, xn);  // in flight while this round is compacted
        const bool active = ptid >= t_lo && ptid < t_hi;
        const float tau = fmaxf(bound, *reinterpret_cast<volatile float*>(&sh.tau));
        int mine = 0;
#pragma unroll
        for (int e = 0; e < kPerThread; ++e) {
            mine += active && x[e] > tau ? 1 : 0;
            if (active) top = fmaxf(top, x[e]);   // ignores NaN
        }
        int incl = mine;
        if (__any_sync(0xffffffffu, mine != 0)) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
        }
        if (lane == 31) sh.warp_cnt[step & 1][pwarp] = incl;
        named_sync(5, kProducerThreads);
        if (ptid == 0) *reinterpret_cast<volatile int*>(&sh.idle) = 0;
        if (step > 0 && ptid == 0) store_release(&sh.head, head);   // the entries of the steps before this one
        const int cnt = lane < kProducerWarps ? sh.warp_cnt[step & 1][lane] : 0;
        const int total = __reduce_add_sync(0xffffffffu, cnt), before = __reduce_add_sync(0xffffffffu, lane < pwarp ? cnt : 0);
        if (total > 0) {
            for (int polls = 0, tail, seen = 0; head + total - (tail = load_acquire(&sh.tail)) > kRing && *v_give_up == 0; seen = tail) {
                polls = tail == seen ? polls + 1 : 0;   // polls without progress of the consumer
                if (polls > wait_polls) *v_give_up = 1;
            }
            const long long base = start + (long long)c * kChunk + (long long)ptid * kPerThread;
            int pos = head + before + incl - mine;
            if (mine) {
#pragma unroll
                for (int e = 0; e < kPerThread; ++e)
                    if (x[e] > tau) sh.ring[pos++ & (kRing - 1)] = Cand{x[e], (int)(base + e)};
            }
            head += total;
        }
        if (((c + 1) & c) == 0 && K <= t_hi && (step < 2 || c + 1 < rounds)) {
            // bisection over the keys: at least K of the maxima are at or above `lo`; 16 steps leave it within a percent
            const uint32_t key = float_key(top);
            uint32_t lo = float_key(-CUDART_INF_F), span = 0x80000000u;
            for (int it = 0; it < 16; ++it, span >>= 1) {
                const uint32_t mid = lo + span;
                const int n = named_count(6, kProducerThreads, mid > lo && key >= mid);
                if (n >= K) lo = mid;
                if (it == 0 && ptid == 0) store_release(&sh.head, head);
            }
            bound = __uint_as_float((lo & 0x80000000u) ? lo & 0x7fffffffu : ~lo);   // float_key's inverse
        }
        if (step >= 2) {
#pragma unroll
            for (int e = 0; e < kPerThread; ++e) x[e] = xn[e];
        }
    }
    if (rounds > 0) named_sync(5, kProducerThreads);
    if (ptid == 0) {
        store_release(&sh.head, head);
        store_release(&sh.done, 1);
    }
}

// Warp 0: hands the ring's entries to `take` (32 at a time in index order, the first in the highest lane) until the
// producers are done; `take` returns the heap minimum.  False when a wait ran out.
template <class Take>
__device__ __forceinline__ bool consume_candidates(Shared& sh, int wait_polls, int lane, Take&& take) {
    int tail = 0;
    for (;;) {
        int head = 0, done = 0;
        if (lane == 0) {
            done = load_acquire(&sh.done);   // before the head: no entry is published after it
            head = load_acquire(&sh.head);
        }
        __syncwarp();   // what lane 0 has acquired, the whole warp may read
        head = __shfl_sync(0xffffffffu, head, 0);
        done = __shfl_sync(0xffffffffu, done, 0);
        if (head == tail) {
            if (done) break;
            int polls = 0;
            if (lane == 0) {   // (counted where the producers reset it: no register of the replay's)
                polls = *reinterpret_cast<volatile int*>(&sh.idle) + 1;
                *reinterpret_cast<volatile int*>(&sh.idle) = polls;
            }
            if (__shfl_sync(0xffffffffu, polls, 0) > wait_polls) {
                *reinterpret_cast<volatile int*>(&sh.give_up) = 1;
                break;
            }
            continue;
        }
        while (tail < head) {
            const int i = tail + 31 - lane;
            const bool valid = i < head;
            const Cand c = sh.ring[i & (kRing - 1)];
            const float heap_min = take(c.v, c.idx, valid);
            tail = min(head, tail + 32);
            __syncwarp();
            if (lane == 0) {
                *reinterpret_cast<volatile float*>(&sh.tau) = heap_min;
                store_release(&sh.tail, tail);   // the warp has read these entries: their places may be written again
            }
        }
    }
    __syncwarp();
    return *reinterpret_cast<volatile int*>(&sh.give_up) == 0;
}

// A heap with NaN among its first K elements: the comparisons are those of no order, its root may fall as well as rise, and no
// bound holds.  Warps 1..15 bring the row into the ring's place, kFeed elements at a time, the next ones in flight while warp 0
// takes them one by one.  64 rows x 151936, K 50: 312 us; 473 with warp 0 reading the row by itself, 278 through a filter with
// bounds.  Out of line: these registers are not the filter's.
constexpr int kFeedLoads = 16, kFeed = kFeedLoads * kProducerThreads;
static_assert(kRing * sizeof(Cand) >= kFeed * sizeof(float), "the elements take the ring's place");
__device__ __noinline__ void feed_unordered(Shared& sh, const float* row, long long V, int K) {
    const int ptid = threadIdx.x - 32;
    float* const buf = reinterpret_cast<float*>(sh.ring);
    float v[kFeedLoads];
    auto load = [&](long long base) {
#pragma unroll
        for (int u = 0; u < kFeedLoads; ++u) { const long long i = base + kProducerThreads * u + ptid; v[u] = i < V ? row[i] : CUDART_NAN_F; }
    };
    load(K);
    for (long long base = K; base < V; base += kFeed) {
        named_sync(7, kThreads);   // warp 0 is done with the elements before these
#pragma unroll
        for (int u = 0; u < kFeedLoads; ++u) buf[kProducerThreads * u + ptid] = v[u];
        named_sync(7, kThreads);
        load(base + kFeed);
    }
}
__device__ __noinline__ void replay_unordered(Shared& sh, long long V, int K) {
    const int lane = threadIdx.x & 31;
    const uint32_t heap_addr = (uint32_t)__cvta_generic_to_shared(sh.heap);
    const float* const buf = reinterpret_cast<const float*>(sh.ring);
    if (lane == 0) make_heap(sh.heap, K);
    for (long long base = K; base < V; base += kFeed) {
        named_sync(7, kThreads);
        named_sync(7, kThreads);
        for (int at = 0; at < kFeed; at += 8 * 32) {
            float w[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) w[u] = buf[at + 32 * u + lane];
            // the first element after the last one that entered, of those the root lets in now
            for (int last = -1;;) {
                const float root = sh.heap[0].v;
                int first = 8 * 32;
#pragma unroll
                for (int u = 7; u >= 0; --u)
                    if (w[u] > root && 32 * u + lane > last) first = 32 * u + lane;   // (nothing is greater than NaN, nor NaN than anything)
                first = __reduce_min_sync(0xffffffffu, first);
                if (first == 8 * 32) break;
                if (lane == 0) replace_min_shared(heap_addr, K, buf[at + first], (int)(base + at + first));
                __syncwarp();
                last = first;
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads, 2) sampler_kernel(StepArgs a) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    Shared& sh = *reinterpret_cast<Shared*>(smem_raw);
    // the next kernel's CTAs may come as soon as every CTA of this one is there (they wait for its end before they leave)
    asm volatile("griddepcontrol.launch_dependents;");
    const int r = blockIdx.x;
    const sampler_row_params p = a.rows[r];
    const long long V = a.vocab;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (p.logits_row < 0 || p.logits_row >= a.num_logit_rows) {
        if (tid == 0) { atomicOr(a.status, 2u); a.out_token[r] = -1; a.out_log_prob[r] = 0.f; }
        return;
    }
    float* row = a.logits + p.logits_row * V;

    const bool multinomial = (p.do_sample & SAMPLER_ROW_MULTINOMIAL) != 0;
    const bool raw_lp = (p.do_sample & SAMPLER_ROW_RAW_LOG_PROB) != 0;
    const RowHistory hist = row_history(a, r);

    // Whole-vocabulary rows are the next kernel's from the beginning on: it may run beside this one.
    if (whole_vocabulary_row(p, V)) return;

    // ---- 0. log-partition of the raw row -----------------------------------------------------------
    float raw_lse = 0.f;
    bool raw_ok = true;
    if (raw_lp) raw_lse = raw_log_partition<kThreads>(a, row, hist, sh.red_f, sh.red_d, &raw_ok);
    auto raw_log_prob_of = [&](long long idx) { return raw_log_prob(a, row, hist, idx, raw_lse, raw_ok); };

    // ---- 1. grammar bitmask, penalties -------------------------------------------------------------
    mask_and_penalise<kThreads>(a, row, p, r, hist, raw_lp && raw_ok);

    // ---- 2. greedy ----------------------------------------------------------------------------------
    if (!multinomial) {
        ArgMax best{-CUDART_INF_F, 0x7fffffff};
        long long done = 0;
        if ((V & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
            // 16-byte loads, four in flight per thread; indices ascend per thread so the first maximum is kept.  The last, partial
            // four too: one behind the other they were up to three more round trips, most of what a row of 32 k waits for
            // (1 row 10.4 -> 10.2 us a step, 256 rows x 151936 32.9 -> 31.9).
            const float4* row4 = reinterpret_cast<const float4*>(row);
            const long long n4 = V >> 2;
            for (long long i = tid; i < n4; i += 4 * kThreads) {
                float4 q[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {   // beyond the row: above nothing
                    q[u] = make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
                    if (i + u * kThreads < n4) q[u] = __ldcs(row4 + i + u * kThreads);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int b = (int)((i + u * kThreads) << 2);
                    if (q[u].x > best.v) { best.v = q[u].x; best.i = b; }
                    if (q[u].y > best.v) { best.v = q[u].y; best.i = b + 1; }
                    if (q[u].z > best.v) { best.v = q[u].z; best.i = b + 2; }
                    if (q[u].w > best.v) { best.v = q[u].w; best.i = b + 3; }
                }
            }
            done = V;
        }
        for (long long i = done + tid; i < V; i += kThreads) {
            const float x = row[i];
            if (x > best.v) { best.v = x; best.i = (int)i; }
        }
        best = block_reduce_n<kThreads>(best, ArgMax{-CUDART_INF_F, 0x7fffffff}, better, sh.red_a);
        if (tid == 0) {
            const int chosen = best.i == 0x7fffffff ? 0 : best.i;  // all -inf / NaN: the reference returns index 0
            a.out_token[r] = chosen;
            a.out_log_prob[r] = raw_lp ? raw_log_prob_of(chosen) : 0.f;   // sampler.cpp:965-974
        }
        return;
    }

    const bool top_k_active = p.top_k > 0 && p.top_k < 0x7fffffffffffffffLL;
    if (top_k_active && p.top_k < V && p.top_k <= kMaxTopK) {
        // ---- 3. exact top-k heap replay --------------------------------------------------------------
        const int K = (int)p.top_k;
        // the producers start at the first 16-byte boundary at or after element K; warp 0 feeds the (at most 3) elements in
        // between to the heap itself
        const long long start = min(V, K + (long long)((16 - ((reinterpret_cast<uintptr_t>(row + K)) & 15)) & 15) / 4);
        const int rounds = (int)((V - start + kChunk - 1) / kChunk);
        const int ptid = tid - 32, pwarp = warp - 1;
        float x[kPerThread], xn[kPerThread];
        auto load_round = [&](int c, float (&dst)[kPerThread]) {
            const long long base = start + (long long)c * kChunk + (long long)ptid * kPerThread;
            if (base + kPerThread <= V) {
                const float4 q0 = __ldcs(reinterpret_cast<const float4*>(row + base));
                const float4 q1 = __ldcs(reinterpret_cast<const float4*>(row + base + 4));
                dst[0] = q0.x; dst[1] = q0.y; dst[2] = q0.z; dst[3] = q0.w;
                dst[4] = q1.x; dst[5] = q1.y; dst[6] = q1.z; dst[7] = q1.w;
            } else {
#pragma unroll
                for (int e = 0; e < kPerThread; ++e) dst[e] = base + e < V ? row[base + e] : CUDART_NAN_F;  // NaN never passes '>'
            }
        };
        if (warp > 0 && rounds > 0) load_round(0, x);
        bool nan_here = false;
        for (int i = tid; i < K; i += kThreads) {
            const float h = row[i];
            sh.heap[i] = Cand{h, i};
            nan_here |= h != h;
        }
        if (tid == 0) { sh.head = 0; sh.tail = 0; sh.idle = 0; sh.done = 0; sh.give_up = 0; sh.tau = -CUDART_INF_F; }
        // NaN among the first K: the heap's comparisons are then those of no order, and the elements are taken one by one
        const bool nan_heap = __syncthreads_or(nan_here) != 0;
        if (warp > 0) {
            if (nan_heap) {
                feed_unordered(sh, row, V, K);
                return;
            }
            produce_candidates(sh, K, V, start, rounds, x, xn, load_round, a.wait_polls, ptid, pwarp, lane);
            return;
        }
        const uint32_t heap_addr = (uint32_t)__cvta_generic_to_shared(sh.heap);
        // takes up to 32 elements in index order - the highest lane holds the first - into the heap in shared memory
        auto take_shared = [&](float v, int idx, bool valid) {
            float heap_min = sh.heap[0].v;
            unsigned mask = __ballot_sync(0xffffffffu, valid && v > heap_min);
            while (mask) {
                const int src = 31 - __clz(mask);
                const float xv = __shfl_sync(0xffffffffu, v, src);
                const int xi = __shfl_sync(0xffffffffu, idx, src);
                if (lane == 0) replace_min_shared(heap_addr, K, xv, xi);
                __syncwarp();
                heap_min = sh.heap[0].v;
                mask = __ballot_sync(0xffffffffu, valid && lane < src && v > heap_min);   // those the new minimum has not overtaken
            }
            return heap_min;
        };
        const Cand* kept = sh.heap;
        TopKDist dist;
        if (nan_heap) {
            replay_unordered(sh, V, K);
            if (lane == 0) dist = build_top_k_dist(sh.heap, sh.prob, K, p);
        } else {
            make_heap_warp(sh.heap, K, lane);
            const int l0 = 31 - lane;   // lanes hold elements last to first
            const float x0 = l0 < start - K ? row[K + l0] : CUDART_NAN_F;
            bool ok;
            if (K <= kRegTopK) {
                const RegHeapLane lh(K, lane);
                RegHeap heap = lh.load(sh.heap);
                RegHeap next = lh.popped(heap);   // the pop does not depend on the entering value: it is taken ahead
                auto take = [&](float v, int idx, bool valid) {
                    const int key = valid && v == v ? order_key(v) : (int)0x80000000;   // below every heap entry
                    unsigned mask = __ballot_sync(0xffffffffu, key > heap.root);
                    while (mask) {
                        const int src = 31 - __clz(mask);   // the highest lane holds the earliest element
                        const int xv = __shfl_sync(0xffffffffu, key, src), xi = __shfl_sync(0xffffffffu, idx, src);
                        const unsigned rest = mask & ~(1u << src);
                        lh.push(next, xv, xi);
                        heap = next;
                        mask = __ballot_sync(0xffffffffu, key > heap.root) & rest;   // those the new minimum has not overtaken
                        next = lh.popped(heap);
                    }
                    return order_value(heap.root);
                };
                take(x0, K + l0, true);
                ok = consume_candidates(sh, a.wait_polls, lane, take);
                lh.store(heap, sh.heap);
            } else {
                take_shared(x0, K + l0, true);
                ok = consume_candidates(sh, a.wait_polls, lane, take_shared);
            }
            __syncwarp();
            if (!ok) {   // a wait between the warps ran out
                if (lane == 0) {
                    atomicOr(a.status, 32u); a.out_token[r] = -1; a.out_log_prob[r] = 0.f;
                    if (a.extra_offsets)
                        for (long long k = a.extra_offsets[r]; k < a.extra_offsets[r + 1]; ++k) { a.extra_out_token[k] = -1; a.extra_out_log_prob[k] = 0.f; }
                }
                return;
            }
            kept = build_top_k_dist_warp(sh, K, p, lane, dist);
        }
        if (lane == 0) {
            const long long x0 = a.extra_offsets ? a.extra_offsets[r] : 0, x1 = a.extra_offsets ? a.extra_offsets[r + 1] : 0;
            for (long long k = -1; k < x1 - x0; ++k) {   // the row's own draw, then the further ones
                float lp;
                long long idx;
                draw_top_k(kept, dist, sh.prob, k < 0 ? p.rand_u : a.extra_rand_u[x0 + k], &lp, &idx);
                if (raw_lp && !dist.uniform) lp = raw_log_prob_of(idx);   // sampler.cpp:1022-1029, 1076-1081
                if (k < 0) { a.out_token[r] = idx; a.out_log_prob[r] = lp; }
                else { a.extra_out_token[x0 + k] = idx; a.extra_out_log_prob[x0 + k] = lp; }
            }
        }
        return;
    }

    // a heap larger than the shared-memory capacity: not supported, and said so (status bit 3, token -1)
    if (tid == 0) {
        atomicOr(a.status, 8u); a.out_token[r] = -1; a.out_log_prob[r] = 0.f;
        if (a.extra_offsets)
            for (long long k = a.extra_offsets[r]; k < a.extra_offsets[r + 1]; ++k) { a.extra_out_token[k] = -1; a.extra_out_log_prob[k] = 0.f; }
    }
}

}  // namespace

size_t sampler_smem_bytes() { return sizeof(Shared); }

cudaError_t launch_sampler(const StepArgs& a, cudaStream_t stream) {
    if (a.num_rows <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(sampler_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared));
    if (e != cudaSuccess) return e;
    sampler_kernel<<<a.num_rows, kThreads, sizeof(Shared), stream>>>(a);
    return cudaGetLastError();
}

}  // namespace sampler
