// The rules by which sampler_exact.cu takes a sequential float sum in segments (host + device: tests/cpp/segment_sum_test.cpp runs a walk
// over them on the CPU against a plain loop).
//
// While a float sum stays in the binade [2^e, 2^(e+1)) it is S * ulp with S from 2^23 to 2^24 - 1, and adding x >= 0 adds a whole number
// of ulps that depends on S through its parity only (fsum_exact.cuh).  So the amounts of elements added in order are what the two
// sums 2^e and 2^e + ulp, one with an even and one with an odd S, gain by real float additions.  Below the lowest binade (zero and
// denormal sums: E = 1, S < 2^23) the ulp is that binade's and every addition is exact: its amounts hold there too.
#pragma once

#include "fsum_exact.cuh"

namespace fsx {

constexpr uint32_t kNoGuess = 0, kEmpty = 255;   // in place of a binade: no amounts are taken; the segment adds nothing
// Relative margins around the approximate sums: where the sum may change binade (the second one: or may not have yet, since what
// rounding took from a sum of small terms adds up)
constexpr float kMargin = 1.0f / 1024, kWideMargin = 1.0f / 64;

struct Sums {
    float even, odd;
};
FSX_HD Sums sums_begin(uint32_t E) { return Sums{bits_float(E << 23), bits_float((E << 23) + 1u)}; }
FSX_HD void sums_add(Sums& s, float x) {
    s.even = fadd_rn(s.even, x);
    s.odd = fadd_rn(s.odd, x);
}
// What was added since sums_begin(E); saturated where a sum has left the binade.
FSX_HD Step sums_amounts(const Sums& s, uint32_t E) {
    const uint32_t base = E << 23, even = float_bits(s.even), odd = float_bits(s.odd);
    Step st{even - base, odd - (base + 1u)};
    if (odd >= base + (1u << 23)) st = Step{kSat, kSat};
    return st;
}

// The amounts for an even and an odd sum differ by one at most: without a half-way case they are the same; at the first x = q + 1/2
// ulps both sums become even - S and S + 1 come to S + q and S + q + 2 where S and q are even, to one sum where q is odd -, and sums of
// one parity go on by the same amounts.
FSX_HD uint32_t pack_amounts(Step st) { return st.a << 2 | (st.b - st.a + 1u); }
FSX_HD Step unpack_amounts(uint32_t w) { return Step{w >> 2, (w >> 2) + (w & 3u) - 1u}; }

// Where the sum is taken to lie in a segment before which it is about lo and behind which about hi.
struct Guess {
    uint32_t E;       // binade, kNoGuess (near infinity, and where the sum goes through binades: its first segment) or kEmpty
    uint32_t alone;   // the one to take where amounts for two are not kept
    bool two;         // it may be in the binade above E as well: amounts are taken for both
    bool edge;        // ... and may go from one to the other in this segment
    bool changes;     // the sum may change binade in it
};
FSX_HD Guess guess_binade(float lo, float hi, bool empty) {
    const uint32_t El = state_exp(lo * (1.f - kMargin)), Eh = state_exp(hi * (1.f + kMargin));
    const uint32_t Ew = state_exp(lo * (1.f - kWideMargin)), Ev = state_exp(hi * (1.f + kWideMargin));
    const bool usable = lo >= 0.f && Ev < 252u && Eh <= El + 2u, two = !empty && usable && Ev == Ew + 1u;
    return Guess{empty ? kEmpty : !usable ? kNoGuess : two ? Ew : state_exp(lo), El, two, two && El != Eh, El != Eh};
}

// Do the amounts of a segment guessed to lie in Eg (two: and Eg + 1) hold for a sum in binade E?
FSX_HD bool guess_holds(uint32_t Eg, bool two, uint32_t E) { return Eg == kEmpty || Eg == E || (two && Eg + 1u == E); }

}  // namespace fsx
