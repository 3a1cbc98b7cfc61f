// The conversion of non-positive arguments in integers (fsx::nonpositive_as_double) in front of the shared sum (fsx::expf_scaled) against
// this host's expf: every `stride`-th float from -0 to -inf, and the edges.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "fsum_exact.cuh"

static float nonpositive(float x) {
    return fsx::expf_scaled(fsx::nonpositive_as_double(x), [](uint64_t ki) { return fsx::u64_as_double(fsx::kExp2TabHost[ki & 31] + (ki << 47)); });
}

int main(int argc, char** argv) {
    const uint32_t stride = argc > 1 ? (uint32_t)std::atoi(argv[1]) : 61u;
    long bad = 0, n = 0;
    auto check = [&](uint32_t bits) {
        const float x = fsx::bits_float(bits), want = expf(x), got = nonpositive(x);
        ++n;
        if (fsx::float_bits(got) != fsx::float_bits(want) && ++bad < 10) std::printf("expf(%a): %a, not %a\n", x, got, want);
    };
    for (uint64_t b = 0x80000000u; b <= 0xff800000u; b += stride) check((uint32_t)b);
    for (uint32_t edge : {0u, 0x80000000u, 0x80000001u, 0x80800000u, 0xff800000u, fsx::float_bits(-104.5f), fsx::float_bits(-103.972076f), fsx::float_bits(-103.27893f), fsx::float_bits(-87.33655f)})
        for (int d = -40; d <= 40; ++d) {
            const uint32_t b = edge + (uint32_t)d;
            if (b == 0u || (b >= 0x80000000u && b <= 0xff800000u)) check(b);
        }
    std::printf("%ld arguments, %ld differ\n", n, bad);
    return bad != 0;
}
