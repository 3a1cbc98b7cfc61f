// The rules of segment_sum.cuh on the CPU: amounts of single terms and of runs against float additions, their packing, and a walk over
// segments with guessed binades - 32 lanes of eight elements each, as the kernel has them - against `s += x[i]`.
//
// usage: segment_sum_test sums SEEDS        every sum before a segment and every crossing of a threshold is the plain loop's
//        segment_sum_test late SEEDS        rows whose sum begins late or grows in jumps: the walk goes by the amounts, except where the sum
//                                           changes binade
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <random>
#include <string>
#include <vector>

#include "segment_sum.cuh"

static long failures = 0;
#define CHECK(cond, ...) do { if (!(cond) && ++failures < 20) { std::printf("%s:%d: ", __FILE__, __LINE__); std::printf(__VA_ARGS__); std::printf("\n"); } } while (0)

constexpr int kBlock = 256, kLanes = 32, kPer = 8;

static fsx::Step amounts(const float* x, int n, uint32_t E) {
    fsx::Sums s = fsx::sums_begin(E);
    for (int i = 0; i < n; ++i) fsx::sums_add(s, x[i]);
    return fsx::sums_amounts(s, E);
}

// A segment's amounts as a warp takes them: the lanes' added up where they do not depend on the order, else composed.
static uint32_t segment_word(const float* x, uint32_t E) {
    fsx::Step lanes[kLanes], st = fsx::step_identity();
    bool tie = false;
    uint64_t sum = 0;
    for (int l = 0; l < kLanes; ++l) {
        lanes[l] = amounts(x + kPer * l, kPer, E);
        tie |= lanes[l].a != lanes[l].b;
        sum += lanes[l].a;
    }
    if (!tie) st.a = st.b = (uint32_t)std::min<uint64_t>(sum, fsx::kSat);
    else for (const fsx::Step& l : lanes) st = fsx::then(st, l);
    CHECK((int64_t)st.b - (int64_t)st.a <= 1 && (int64_t)st.a - (int64_t)st.b <= 1, "amounts %u and %u", st.a, st.b);
    const fsx::Step back = fsx::unpack_amounts(fsx::pack_amounts(st));
    CHECK(back.a == st.a && back.b == st.b, "packing of %u, %u", st.a, st.b);
    return fsx::pack_amounts(st);
}

// The elements of a segment without amounts made before: all lanes' at once as far as the sum stays in its binade.
static int add_by_lanes(const float* x, uint32_t& E, uint32_t& S, float thr) {
    for (int from = 0; from < kLanes; ++from) {
        if (E < 252u) {
            fsx::Step st = fsx::step_identity();
            uint32_t before = S;
            int l = from;
            for (; l < kLanes; ++l) {
                st = fsx::then(st, amounts(x + kPer * l, kPer, E));
                const uint32_t after = fsx::apply(st, S);
                if (after >= fsx::kOne24 || fsx::state_float(E, after) > thr) break;
                before = after;
            }
            S = before;
            if (l == kLanes) break;
            from = l;
        }
        float s = fsx::state_float(E, S);
        for (int e = 0; e < kPer; ++e) {
            s += x[kPer * from + e];
            if (s > thr) { E = fsx::state_exp(s); S = fsx::state_sig(s); return kPer * from + e; }
        }
        E = fsx::state_exp(s);
        S = fsx::state_sig(s);
    }
    return -1;
}

struct Walk {
    std::vector<float> before;   // sum before every segment
    float s = 0.f;
    long long hit = -1;
    int misses = 0;              // segments that were not taken by their amounts,
    int wrong = 0;               // of them those whose guess did not hold
};

static Walk walk(const std::vector<float>& x, const std::vector<float>& cum, float thr) {
    Walk w;
    const size_t segs = x.size() / kBlock;
    uint32_t E = fsx::state_exp(0.f), S = fsx::state_sig(0.f);
    for (size_t j = 0; j < segs; ++j) {
        const float* at = x.data() + j * kBlock;
        const fsx::Guess g = fsx::guess_binade(cum[j], cum[j + 1], false);
        const bool holds = g.E != fsx::kNoGuess && fsx::guess_holds(g.E, g.two, E);
        w.before.push_back(fsx::state_float(E, S));
        if (holds) {
            const uint32_t after = g.E == fsx::kEmpty ? S : fsx::apply(fsx::unpack_amounts(segment_word(at, E)), S);
            if (after < fsx::kOne24 && !(fsx::state_float(E, after) > thr)) {
                S = after;
                continue;
            }
        }
        ++w.misses;
        w.wrong += holds || g.E == fsx::kNoGuess ? 0 : 1;
        const int e = add_by_lanes(at, E, S, thr);
        if (e >= 0) {
            w.hit = (long long)(j * kBlock) + e;
            break;
        }
    }
    w.s = fsx::state_float(E, S);
    return w;
}

// ---- rows: exponentials of logits of several kinds ----------------------------------------------------------
static std::vector<float> exponentials(const std::string& kind, std::mt19937& rng, int n) {
    std::normal_distribution<float> N(0.f, 2.f);
    std::vector<float> x(n);
    for (float& v : x) v = N(rng);
    float T = 1.f;
    if (kind == "spikes" || kind == "cold_spikes") {
        for (int k = 0; k < 8; ++k) x[rng() % n] += 15.f;
    }
    if (kind == "cold" || kind == "cold_spikes") T = 0.1f;
    if (kind == "freezing") T = 0.01f;
    if (kind == "quantised") for (float& v : x) v = std::nearbyint(4.f * v) / 4.f;
    if (kind == "equal") for (float& v : x) v = 1.5f;
    if (kind == "late") x[n - n / 8] = 60.f;
    if (kind == "last_ids") for (int i = 0; i < n - 200; ++i) x[i] = -std::numeric_limits<float>::infinity();
    if (kind == "few_ids") {
        std::vector<float> y(n, -std::numeric_limits<float>::infinity());
        for (int k = 0; k < 20; ++k) { const int i = (int)(rng() % n); y[i] = x[i]; }
        x = y;
    }
    if (kind == "upper_half") for (int i = 0; i < n / 2; ++i) x[i] = -std::numeric_limits<float>::infinity();
    const float mx = *std::max_element(x.begin(), x.end());
    for (float& v : x) v = fsx::expf_libm((v - mx) * (1.f / T));
    if (kind == "tiny") for (float& v : x) v = fsx::bits_float((uint32_t)(rng() % 0x01800000u));   // denormals and the lowest binades
    x.resize((n + kBlock - 1) / kBlock * kBlock, 0.f);
    return x;
}
// Sums before the segments as the kernel has them: float masses with an error of some 2^-20, nothing below the normal range.
static std::vector<float> approximate_sums(const std::vector<float>& x, std::mt19937& rng) {
    std::vector<float> cum{0.f};
    std::uniform_real_distribution<double> U(-1e-6, 1e-6);
    for (size_t j = 0; j < x.size() / kBlock; ++j) {
        double mass = 0;
        for (int i = 0; i < kBlock; ++i) mass += x[j * kBlock + i];
        const float m = (float)(mass * (1 + U(rng)));
        cum.push_back(cum.back() + (m < 0x1p-126f ? 0.f : m));
    }
    return cum;
}

static void check_walk(const std::string& kind, const std::vector<float>& x, const std::vector<float>& cum, float thr) {
    const Walk w = walk(x, cum, thr);
    volatile float s = 0.f;
    long long hit = -1;
    for (size_t i = 0; i < x.size() && hit < 0; ++i) {
        if (i % kBlock == 0) CHECK(fsx::float_bits(w.before[i / kBlock]) == fsx::float_bits(s), "%s: sum before segment %zu: %a, not %a", kind.c_str(), i / kBlock, w.before[i / kBlock], s);
        s = s + x[i];
        if (s > thr) hit = (long long)i;
    }
    CHECK(w.hit == hit, "%s: threshold %a passed at %lld, not %lld", kind.c_str(), thr, w.hit, hit);
    CHECK(fsx::float_bits(w.s) == fsx::float_bits(s), "%s: sum %a, not %a", kind.c_str(), w.s, s);
}

static const char* kKinds[] = {"normal", "spikes", "cold", "cold_spikes", "freezing", "quantised", "equal", "late", "last_ids", "few_ids", "upper_half", "tiny"};

int main(int argc, char** argv) {
    const std::string mode = argc > 1 ? argv[1] : "sums";
    const int seeds = argc > 2 ? std::atoi(argv[2]) : 2;
    if (mode == "sums") {
        // single terms: half-way cases, terms far below an ulp, terms that leave the binade, either parity, every kind of binade
        std::mt19937 rng(1);
        for (int k = 0; k < 400000; ++k) {
            const uint32_t E = k % 5 == 0 ? 1u + rng() % 4u : 1u + rng() % 250u;
            const uint32_t S = 0x800000u + (k % 3 == 0 ? rng() % 4u : rng() % 0x800000u);
            float x[kPer], s = fsx::state_float(E, S);
            for (float& v : x) {
                const int e = (int)E - (int)(rng() % 30u);
                uint32_t m = rng() & 0x7fffffu;
                if (rng() % 2) m &= 0x7fffffu << (rng() % 24u);   // few bits: half-way cases
                v = fsx::bits_float((uint32_t)std::max(e, 0) << 23 | m);
            }
            const int n = 1 + (int)(rng() % kPer);
            for (int i = 0; i < n; ++i) s = s + x[i];
            const fsx::Step st = amounts(x, n, E);
            const uint32_t after = fsx::apply(st, S);
            if (fsx::state_exp(s) == E) CHECK(after < fsx::kOne24 && fsx::float_bits(fsx::state_float(E, after)) == fsx::float_bits(s), "E %u S %u: %u, not %a", E, S, after, s);
            else CHECK(after >= fsx::kOne24, "E %u S %u: the sum leaves the binade (%a), the amounts do not (%u)", E, S, s, after);
        }
        for (int seed = 0; seed < seeds; ++seed)
            for (const char* kind : kKinds)
                for (int n : {1, 255, 256, 257, 8193, 40000}) {
                    std::mt19937 r(977u * seed + n);
                    const std::vector<float> x = exponentials(kind, r, n), cum = approximate_sums(x, r);
                    const float total = cum.back();
                    for (float thr : {std::numeric_limits<float>::infinity(), 0.f, 0.37f * total, 0.95f * total, total}) check_walk(kind, x, cum, thr);
                    std::vector<float> off = cum;   // guesses that do not hold cost time only
                    for (float& c : off) c *= std::exp2((float)(int)(r() % 7u) - 3.f);
                    check_walk(kind, x, off, 0.6f * total);
                }
    }
    if (mode == "late") {
        for (int seed = 0; seed < seeds; ++seed)
            for (const char* kind : {"cold_spikes", "freezing", "late", "last_ids", "few_ids", "upper_half"}) {
                std::mt19937 r(31u + seed);
                const std::vector<float> x = exponentials(kind, r, 128256), cum = approximate_sums(x, r);
                const Walk w = walk(x, cum, std::numeric_limits<float>::infinity());
                int changes = 0;   // segments in which the sum changes binade: those the walk has to open
                for (size_t j = 0; j < w.before.size(); ++j)
                    changes += fsx::state_exp(w.before[j]) != fsx::state_exp(j + 1 < w.before.size() ? w.before[j + 1] : w.s);
                std::printf("%s: %d changes of binade, %d segments not taken by their amounts, %d of them guessed wrong\n", kind, changes, w.misses, w.wrong);
                CHECK(w.misses <= changes + 4 && w.wrong <= 4, "%s: %d segments are not taken by their amounts, %d wrong guesses", kind, w.misses, w.wrong);
            }
    }
    std::printf("%ld failures\n", failures);
    return failures != 0;
}
