// Host check of narrow64 and widen32 (shamrock_gb300/csrc/split64.cuh) against the plain
// conversions, and of how often the roots, reciprocals and quotients of lean64.cuh fail
// their proof on normal operands of ordinary size.
#include "../../shamrock_gb300/csrc/lean64.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace gbsph;

static long wrong = 0, checks = 0;

static uint32_t bits32(float f) {
    uint32_t b;
    std::memcpy(&b, &f, 4);
    return b;
}
static void narrow(uint64_t b) {
    const double v = from64(b);
    const float got = narrow64(v), want = (float) v;
    checks++;
    if (bits32(got) != bits32(want) && !(got != got && want != want)) {
        if (wrong < 5) std::printf("narrow64(%a) = %a, not %a\n", v, (double) got, (double) want);
        wrong++;
    }
}
static void widen(uint32_t b) {
    const float f = split64_bits_to_float(b);
    const double got = widen32(f), want = (double) f;
    checks++;
    if (bits64(got) != bits64(want) && !(got != got && want != want)) {
        if (wrong < 5) std::printf("widen32(%a) = %a\n", (double) f, got);
        wrong++;
    }
}

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 4000000;
    std::mt19937_64 g(11);
    // every exponent of the double range, with random significands, those at and beside the
    // ties of 24 bits, all ones and zero; both signs
    for (uint64_t e = 0; e < 2048; e++)
        for (long k = 0; k < n / 2048; k++) {
            uint64_t m = g() & 0xFFFFFFFFFFFFFull;
            if (k % 8 == 1) m = (m & ~0x1FFFFFFFull) | 0x10000000ull;
            if (k % 8 == 2) m = (m & ~0x1FFFFFFFull) | 0x10000001ull;
            if (k % 8 == 3) m = (m & ~0x1FFFFFFFull) | 0x0FFFFFFFull;
            if (k % 8 == 4) m = 0xFFFFFFFFFFFFFull - (g() & 3) * 0x10000000ull;
            if (k % 8 == 5) m = k % 16 == 5 ? 0 : (m & ~0x1FFFFFFFull);
            narrow((g() << 63) | (e << 52) | m);
        }
    // all float exponents with random significands, and every 4,099th float
    for (uint32_t e = 0; e < 256; e++)
        for (long k = 0; k < n / 256; k++) widen((uint32_t) (g() << 31) | (e << 23) | (k < 2 ? (uint32_t) k : (uint32_t) g() & 0x7FFFFFu));
    for (uint64_t b = 0; b < (1ull << 32); b += 4099) widen((uint32_t) b);
    // shares of unproven roots, reciprocals of roots, and quotients
    long bad[4] = {0, 0, 0, 0};
    std::uniform_real_distribution<double> u(-20, 20);
    for (long i = 0; i < n; i++) {
        const double a = std::exp2(u(g)), b = std::exp2(u(g));
        bool x = false, y = false, z = false, w = false;
        const Root r = root64(a, x);
        root_reciprocal(r, y);
        quotient64(a, b, z);
        divide_by(a, denominator(b), w);
        bad[0] += x, bad[1] += y, bad[2] += z, bad[3] += w;
    }
    std::printf("checks %ld wrong %ld unproven root %.2e reciprocal %.2e quotient %.2e by %.2e\n", checks, wrong,
                bad[0] / (double) n, bad[1] / (double) n, bad[2] / (double) n, bad[3] / (double) n);
    for (long k : bad)
        if (k > n / 10000) return 1;
    return wrong == 0 ? 0 : 1;
}
