// Host check of shamrock_gb300/csrc/lean64.cuh against the operators: every value that is
// not reported `bad` equals the operator's bit for bit, few are reported, and the operands
// at the edges of the ranges (zeros, subnormals, infinities, NaN, powers of two and their
// neighbours, all-ones mantissas) are either right or reported.
#include "../../shamrock_gb300/csrc/lean64.cuh"

#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>
#include <vector>

using namespace gbsph;

static long wrong = 0, reported = 0, checks = 0;

static void expect(double got, double want, bool bad) {
    checks++;
    if (bad) {
        reported++;
        return;
    }
    if (bits64(got) != bits64(want) && !(got != got && want != want)) {
        if (wrong < 5) std::printf("got %a want %a\n", got, want);
        wrong++;
    }
}

static void all(double a, double b) {
    bool bad = false;
    if (a > 0) {
        const Root r = root64(a, bad);
        expect(root_value(r), std::sqrt(a), bad);
        if (!bad) {
            bool bad2 = false;
            const double y = root_reciprocal(r, bad2);
            expect(y, 1.0 / std::sqrt(a), bad2);
        }
    }
    bad = false;
    if (a > 0 && b > 0) {
        const double q = quotient64(a, b, bad);
        expect(q, a / b, bad);
    }
    bad = false;
    const double q = divide_by(a, denominator(b), bad);
    expect(q, a / b, bad);
    expect(mul64i(a, b), a * b, false);
    expect(mul64i(-a, b), -a * b, false);
    const float c = cut32(a);
    if (std::fabs(a) >= 1.2e-38 && std::fabs(a) < 3.4e38) {
        checks++;
        if (!(std::fabs((double) c) <= std::fabs(a) && std::fabs((double) c) >= std::fabs(a) * (1 - 1.2e-7))) wrong++;
    }
}

// the cell equals the clamped division's, and half the coordinates sit on cell faces or next
// to them, on the box's faces or beyond
static void cells(std::mt19937_64 &g, long n) {
    std::uniform_real_distribution<double> u(-0.1, 1.1);
    for (const uint32_t count : {1024u, 2097152u})
        for (long b = 0; b < 64; b++) {
            const double lo   = b % 8 == 0 ? 0.0 : (b % 8 == 1 ? -0.5 : std::ldexp(u(g) - 0.5, (int) (b % 40) - 20));
            const double size = b % 16 < 2 ? 1.0 : (b == 17 ? 0.0 : (b == 18 ? 1e-320 : std::ldexp(1 + std::fabs(u(g)), (int) (b * 5 % 61) - 30)));
            const double hi = lo + size, step = (hi - lo) / (double) count;
            const double inv = step > 1e-300 && step < 1e300 ? 1.0 / step : 0.0;
            std::vector<double> ps = {lo, hi, std::nextafter(lo, -1e308), std::nextafter(hi, 1e308), -0.0, 1e308, -1e308,
                                      std::numeric_limits<double>::infinity(), -std::numeric_limits<double>::infinity(),
                                      std::numeric_limits<double>::quiet_NaN(), lo + 1e6 * size, hi - 1e9 * size};
            for (long i = 0; i < n / 128; i++) {
                double p = lo + u(g) * (hi - lo);
                if (i % 2) p = lo + (double) (g() % count) * step;
                if (i % 4 == 3) p = std::nextafter(p, i % 8 == 3 ? 1e308 : -1e308);
                ps.push_back(p);
            }
            for (double p : ps) {
                const double r = std::fmin(std::fmax(p, lo), hi), q = (r - lo) / step;
                const uint32_t want = !(q > 0) ? 0u : (q >= (double) (count - 1) ? count - 1 : (uint32_t) q);
                checks++;
                if (grid_cell(p, lo, hi, step, inv, count - 1) != want) {
                    if (wrong < 5) std::printf("cell of %a in [%a, %a], %u\n", p, lo, hi, count);
                    wrong++;
                }
            }
        }
}

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
    std::mt19937_64 g(7);
    std::uniform_int_distribution<int> ex(-40, 40), wide(-1000, 1000);
    std::vector<double> edge = {0.0, -0.0, 1.0, 2.0, 4.0, 0.5, 3.0, 1.0 / 3, 5e-324, 2.2250738585072014e-308,
                                1.7976931348623157e308, std::numeric_limits<double>::infinity(),
                                std::numeric_limits<double>::quiet_NaN(), 1e-300, 1e300, -1.0, -3e-7};
    const size_t plain = edge.size();
    for (size_t i = 0; i < plain; i++)
        for (double to : {0.0, 1e308}) edge.push_back(std::nextafter(edge[i], to));
    for (double a : edge)
        for (double b : edge) all(a, b);
    const long edges_reported = reported;
    reported = 0;
    const long before = checks;
    for (long i = 0; i < n; i++) {
        const uint64_t m = g(), m2 = g();
        double a = from64((m & 0xFFFFFFFFFFFFFull) | (1023ull << 52));
        double b = from64((m2 & 0xFFFFFFFFFFFFFull) | (1023ull << 52));
        if (i % 7 == 0) a = from64((0xFFFFFFFFFFFFFull - (m & 15)) | (1023ull << 52));
        if (i % 11 == 0) b = from64((m2 & 15) | (1023ull << 52));
        if (i % 13 == 0) b = from64((0xFFFFFFFFFFFFFull - (m2 & 15)) | (1023ull << 52));
        const int ea = i % 5 ? ex(g) : wide(g), eb = i % 5 ? ex(g) : wide(g);
        all(std::ldexp(a, ea), std::ldexp(b, eb));
    }
    const double share = (double) reported / (double) (checks - before);
    cells(g, n);
    std::printf("checks %ld wrong %ld reported %.3g edges reported %ld\n", checks, wrong, share, edges_reported);
    return wrong == 0 && share < 0.05 ? 0 : 1;
}
