// What the CPU tests of this folder know as fsum_exact.cuh: the header of that name that the CUDA kernel is compiled from, and a sequential
// statement of sums over sorted probabilities by bins and lists on top of its step algebra (topp_model.hpp runs it against a plain loop).
// The kernel takes the same sums from segments (segment_sum.cuh).
#pragma once

#include "../../openvino.genai_b200/csrc/fsum_exact.cuh"

namespace fsx {

// The step of adding x (finite, >= 0) to a sum whose biased exponent is E.  `tie` is set when the
// amount depends on the parity of the sum.
FSX_HD Step step_of(float x, uint32_t E, bool* tie) {
    const uint32_t bx = float_bits(x);
    uint32_t ex = bx >> 23, m = bx & 0x7fffffu;
    if (ex) m |= 0x800000u; else ex = 1u;
    *tie = false;
    const int d = (int)E - (int)ex;
    if (d <= 0) {
        const uint32_t k = d < -2 ? kSat : (m << (-d));
        const uint32_t c = k > kSat ? kSat : k;
        return Step{c, c};
    }
    if (d >= 25) return Step{0u, 0u};
    const uint32_t q = m >> d, rem = m & ((1u << d) - 1u), half = 1u << (d - 1);
    if (rem == half) {
        *tie = true;
        return Step{q + (q & 1u), q + 1u - (q & 1u)};
    }
    const uint32_t c = q + (rem > half ? 1u : 0u);
    return Step{c, c};
}
FSX_HD Step step_of(float x, uint32_t E) { bool t; return step_of(x, E, &t); }

// The amount of a term that is not a tie, in five float operations, for the passes that add whole spans
// or bins.  scale = 2^(150 - E) turns x into units of the sum's ulp exactly (a power of two); rintf
// rounds to nearest, and the distance to the rounded value tells a tie (exactly one half).  `defer` is
// set for a tie and for a term of 2^24 ulps or more, which the callers add element by element.
FSX_HD float amount_scale(uint32_t E) {   // 0 where the scale is not a normal float: such sums go element by element
    return (E >= 24u && E <= 254u) ? bits_float((277u - E) << 23) : 0.0f;
}
FSX_HD uint32_t plain_amount(float x, float scale, bool* defer) {
    const float t = x * scale;
#if defined(__CUDA_ARCH__)
    const float r = rintf(t);
    *defer = fabsf(t - r) == 0.5f || !(t < 16777216.0f);
    return __float2uint_rz(r);
#else
    const float r = std::nearbyint(t);   // round half to even in the default rounding mode
    *defer = std::fabs(t - r) == 0.5f || !(t < 16777216.0f);
    return t < 4294967040.0f ? (uint32_t)r : 0xffffffffu;
#endif
}

// ---- sums over probabilities sorted in descending order --------------------------------------------
// TopPFilter adds the sorted probabilities one by one until the running float sum exceeds top_p
// (logit_transformers.hpp:105-125) and the draw walks the same running sums (sampler.cpp:1065-1074).
// Keys are the bit patterns of the probabilities (non-negative floats: larger key <=> larger value).
// A level cuts the keys below `F` into kBins bins of 2^sh consecutive keys, highest keys first; what
// lies below the last bin is the level's rest.  A bin whose elements cannot meet a tie, a change of
// binade, the threshold or the element limit is added as one translation: the sum of its elements'
// amounts under the hypothesised exponent E[j] of the running sum, which does not depend on their
// order.  Every other bin is listed element by element, sorted, and added with real float additions.
// Hypotheses come from approximate masses and are checked by the walk itself: a bin whose hypothesis
// does not hold is never taken as a whole, so a wrong guess costs another pass, not a wrong sum.

constexpr int kBins = 2048;
constexpr int kTopSh = 16;          // first level: 128 bins per binade of the probabilities, 16 binades
constexpr int kSubBits = 11;        // a bin that has to be cut further becomes a level of its own

enum : uint8_t {
    kBinListed = 1,    // the bin's elements are in the list
    kBinTie = 2,       // an element of the bin is a tie under E[j]
    kBinValid = 4,     // A[j] holds the sum of amounts under E[j]
    kBinDirty = 8,     // A[j] is to be accumulated by the next pass
    kBinCollect = 16,  // the next pass appends the bin's elements to the list
    kBinStep = 32,     // listed bin: A[j] holds the composition of its elements' steps under E[j], in list order (pack_step)
};

struct Level {
    uint32_t F;   // keys < F belong to this level
    int sh;
};
FSX_HD uint32_t bin_of(Level L, uint32_t key) {   // key < L.F; kBins and above = the level's rest
    return (L.F - 1u - key) >> L.sh;
}

struct Bins {
    uint32_t* A;      // [kBins] sum of amounts (valid bins)
    uint32_t* C;      // [kBins] element counts
    float* R;         // [kBins] approximate masses, for the hypotheses only
    uint32_t* PA;     // [kBins] sum of A over the plain bins from the last stop up to and including j (saturating)
    uint32_t* PC;     // [kBins] the same for C
    uint16_t* next;   // [kBins + 1] next[j] = first stop bin at or after j (kBins if none)
    uint8_t* E;       // [kBins] hypothesised exponent
    uint8_t* flag;    // [kBins]
};

// A step whose even-state amount is below 2^24 and whose two amounts differ by less than 128, in one word.
FSX_HD bool step_packs(Step st) {
    const long long d = (long long)st.b - (long long)st.a;
    return st.a < kOne24 && st.b < kSat && d >= -128 && d <= 127;
}
FSX_HD uint32_t pack_step(Step st) { return st.a | ((uint32_t)(uint8_t)(int8_t)((int)st.b - (int)st.a) << 24); }
FSX_HD Step unpack_step(uint32_t w) {
    const uint32_t a = w & 0xffffffu;
    return Step{a, (uint32_t)((int)a + (int)(int8_t)(uint8_t)(w >> 24))};
}

// plain: non-empty, summed as a whole
FSX_HD bool bin_plain(const Bins& b, int j) {
    return b.C[j] != 0 && (b.flag[j] & (kBinListed | kBinTie | kBinValid)) == kBinValid;
}
// A stop is a non-empty bin at which the walk has to look: listed, unresolved, or the first bin of a
// run of plain bins (after a bin that is not plain, or where the hypothesis changes).
// prev_plain_E: E of the nearest non-empty bin before j if that bin is plain, else -1.
FSX_HD bool bin_is_stop(const Bins& b, int j, int prev_plain_E) {
    if (b.C[j] == 0) return false;
    if (!bin_plain(b, j)) return true;
    return (int)b.E[j] != prev_plain_E;
}

struct Walk {
    float s;          // running sum so far
    uint32_t cnt;     // elements added so far
    int j;            // next bin
    int li;           // next list entry
    int status;       // kWalk*
    uint32_t hit_key; // found: the element at which the sum exceeded the threshold or the limit was reached
    uint32_t hit_idx;
    bool by_limit;    // found by the element limit, not by the threshold
};
enum { kWalkFound = 0, kWalkUnresolved = 1, kWalkEnd = 2 };

FSX_HD uint32_t entry_key(uint64_t e) { return (uint32_t)(e >> 32); }
FSX_HD uint32_t entry_idx(uint64_t e) { return 0xffffffffu - (uint32_t)e; }
FSX_HD uint64_t make_entry(uint32_t key, uint32_t idx) { return ((uint64_t)key << 32) | (0xffffffffu - idx); }

// Where a walk stood when it came to a bin: the exact sum and count of everything before the bin, and its place in the list.
// A later walk of the same row with a lower threshold may start from the last such record that is still below its threshold
// instead of from the top (the sums are the same additions in the same order).
// One record per group of kCkGroup bins (the last bin of the group the walk came to).
constexpr int kCkGroup = 4;
struct Checkpoints {
    float* s;
    uint32_t* cnt;
    uint16_t* j;
    uint16_t* li;
};

// Continues the walk from (w.s, w.cnt, w.j, w.li) until the running sum exceeds `thr`, `limit`
// elements have been added (limit 0: no limit), a bin cannot be taken, or the level ends.
// `list` is sorted in descending order (key, then ascending index).  One thread runs this.
FSX_HD void walk_level(Walk& w, Level L, const Bins& b, const uint64_t* list, int list_n, float thr, uint32_t limit, const Checkpoints* ck = nullptr) {
    for (;;) {
        if (w.j >= kBins) { w.status = kWalkEnd; return; }
        const int j = w.j;
        if (ck) { const int g = j / kCkGroup; ck->s[g] = w.s; ck->cnt[g] = w.cnt; ck->j[g] = (uint16_t)j; ck->li[g] = (uint16_t)w.li; }
        if (b.C[j] == 0) { w.j = (int)b.next[j]; continue; }     // only empty bins up to the next stop
        const uint8_t f = b.flag[j];
        if (f & kBinListed) {
            if ((f & kBinStep) && w.s != 0.0f && (uint32_t)b.E[j] == state_exp(w.s)) {
                // The bin's elements as one step: while the sum stays in the binade of the hypothesis (it only grows, so the end
                // tells), below the threshold and short of the element limit, the composition of the elements' two-state steps
                // in list order is what adding them one by one gives.
                const uint32_t E = state_exp(w.s), S = state_sig(w.s);
                const Step st = unpack_step(b.A[j]);
                const uint32_t S2 = apply(st, S), n = b.C[j];
                if (S2 < kOne24 && !(state_float(E, S2) > thr) && !(limit && w.cnt + n >= limit)) {
                    while (w.li < list_n) {   // entries added earlier
                        const uint32_t key = entry_key(list[w.li]);
                        if (key >= L.F || bin_of(L, key) < (uint32_t)j) ++w.li; else break;
                    }
                    w.li += (int)n;
                    w.s = state_float(E, S2);
                    w.cnt += n;
                    ++w.j;
                    continue;
                }
            }
            while (w.li < list_n) {   // entries of this bin, one real addition each
                const uint64_t e = list[w.li];
                const uint32_t key = entry_key(e);
                const uint32_t bj = key < L.F ? bin_of(L, key) : 0u;
                if (key >= L.F || bj < (uint32_t)j) { ++w.li; continue; }   // added earlier
                if (bj != (uint32_t)j) break;
                w.s = fadd_rn(w.s, bits_float(key));
                ++w.cnt;
                ++w.li;
                const bool over = w.s > thr;
                if (over || (limit && w.cnt >= limit)) {
                    w.status = kWalkFound; w.hit_key = key; w.hit_idx = entry_idx(e); w.by_limit = !over;
                    return;
                }
            }
            ++w.j;
            continue;
        }
        if ((f & kBinTie) || !(f & kBinValid)) { w.status = kWalkUnresolved; return; }
        // a run of plain (and empty) bins: from the stop j up to the next stop
        const uint32_t E = state_exp(w.s), S = state_sig(w.s);
        if (w.s == 0.0f || (uint32_t)b.E[j] != E || (int)b.next[j] != j) { w.status = kWalkUnresolved; return; }
        const int k = (int)b.next[j + 1];
        int lo = j, hi = k;      // bins j .. lo - 1 can be taken as a whole
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            const uint32_t add = b.PA[mid - 1], n = b.PC[mid - 1];
            const bool ok = add < kOne24 && S + add < kOne24 && !(state_float(E, S + add) > thr) && !(limit && w.cnt + n >= limit);
            if (ok) lo = mid; else hi = mid - 1;
        }
        if (lo > j) {
            w.s = state_float(E, S + b.PA[lo - 1]);
            w.cnt += b.PC[lo - 1];
        }
        w.j = lo;
        if (lo < k) { w.status = kWalkUnresolved; return; }
    }
}

// The exponent hypothesised for a float sum whose real-valued counterpart runs from lo to hi, and
// whether the range widened by the relative margin stays inside one binade.
FSX_HD bool hyp_exponent(double lo, double hi, double margin, uint32_t* E) {
    const float flo = (float)(lo * (1.0 - margin)), fhi = (float)(hi * (1.0 + margin));
    *E = state_exp(flo);
    return lo > 0.0 && state_exp(flo) == state_exp(fhi);
}

// Adds `c` copies of x to the sum s (real additions where the binade changes, powers of the step
// otherwise) until the sum exceeds thr or `limit` elements have been added.  Returns the number of
// copies added; *found tells whether it stopped for the threshold or the limit.
FSX_HD uint32_t add_repeated(float& s, uint32_t& cnt, float x, uint32_t c, float thr, uint32_t limit, bool* found, bool* by_limit) {
    uint32_t done = 0;
    *found = false;
    while (done < c) {
        const uint32_t E = state_exp(s);
        uint32_t S = state_sig(s);
        if (s != 0.0f) {
            Step pw[32];
            pw[0] = step_of(x, E);
            int top = 0;
            while ((1u << (top + 1)) <= c - done && top < 30) { pw[top + 1] = then(pw[top], pw[top]); ++top; }
            uint32_t n = 0;
            for (int k = top; k >= 0; --k) {
                const uint32_t m = 1u << k;
                if (n + m > c - done) continue;
                const uint32_t S2 = apply(pw[k], S);
                if (S2 >= kOne24 || state_float(E, S2) > thr || (limit && cnt + n + m >= limit)) continue;
                S = S2; n += m;
            }
            s = state_float(E, S);
            cnt += n; done += n;
            if (done == c) break;
        }
        s = fadd_rn(s, x);   // the copy that changes the binade, meets the threshold or the limit
        ++cnt; ++done;
        const bool over = s > thr;
        if (over || (limit && cnt >= limit)) { *found = true; *by_limit = !over; return done; }
    }
    return done;
}

}  // namespace fsx
