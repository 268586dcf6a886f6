// Host check of csrc/exact_int.h's quotients and square roots (div_int_with,
// sqrt_int_from) against the host's IEEE binary64 division and square root,
// bit for bit, wherever they do not flag the operands.  The seeds that the
// device takes from its FP32 approximation instructions are the host's rounded
// values here, moved by up to 4 units in the last place either way: more than
// the error that the instructions' documentation allows (1 ulp for the
// reciprocal, a relative 2^-22.9 for the reciprocal root).  Operands: random bit
// patterns, significands of few bits, leading or trailing ones, quotients and
// squares next to a rounding boundary, exponents at the ends of the range and
// special values.
#include "../1dsweptcuda_gb300/csrc/exact_int.h"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

using namespace sw;

static long n_checked = 0, n_fast = 0, n_bad = 0;

static bool same(double a, double b) { return f64_bits(a) == f64_bits(b) || (std::isnan(a) && std::isnan(b)); }

static float moved(float y, int ulps) {
    for (int i = 0; i < std::abs(ulps); ++i) y = std::nextafterf(y, ulps > 0 ? 4.0f : 0.0f);
    return y;
}

static void check(double a, double b) {
    for (int u = -4; u <= 4; ++u) {
        uint32_t bad = 0;
        const double q = div_int_with(a, rcp_int_from(b, moved(f32_rcp_seed(rcp_int_arg(b)), u)), bad);
        ++n_checked;
        n_fast += !bad;
        if (!bad && !same(q, a / b) && n_bad++ < 8) std::printf("%a / %a = %a, not %a (seed %d)\n", a, b, a / b, q, u);
        bad = 0;
        const double r = sqrt_int_from(b, bad, moved(f32_rsqrt_seed(sqrt_int_arg(b)), u));
        ++n_checked;
        n_fast += !bad;
        if (!bad && !same(r, std::sqrt(b)) && n_bad++ < 8) std::printf("sqrt(%a) = %a, not %a (seed %d)\n", b, std::sqrt(b), r, u);
    }
}

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 100000;
    std::mt19937_64 g(20261205);
    const uint64_t all = 0x000fffffffffffffull;
    auto value = [&](uint64_t m, int e) { return f64_from_bits(((g() & 1) << 63) | ((uint64_t)e << 52) | (m & all)); };
    const int ends[] = {1, 2, 3, 1022, 1023, 1024, 2044, 2045, 2046};
    for (long i = 0; i < n; ++i) {
        check(f64_from_bits(g()), f64_from_bits(g()));
        uint64_t a = g(), b = g();
        switch (i % 4) {
        case 1: a |= all >> (g() % 40); break;                                          // trailing ones
        case 2: b |= all >> (g() % 44); a &= ~(all >> (g() % 52)); break;                // ... and zeros
        case 3: a &= 0xfull << (g() % 49); b &= ~(all >> (g() % 52)); break;             // few bits
        }
        check(value(a, 1000 + (int)(g() % 40)), std::fabs(value(b, 1000 + (int)(g() % 40))));
        const double d = std::fabs(value(g(), 1023)), q = std::fabs(value(g(), 1023));   // next to a boundary
        check(q * d, d);
        check(std::nextafter(q * d, 9.0), d);
        check(q * q, q * q);
        check(1.0, std::nextafter(q * q, 0.0));
        check(q, std::nextafter(q * q, 9.0));
        check(value(g(), ends[g() % 9]), value(g(), ends[g() % 9]));
    }
    const double special[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 4.9e-324, 2.2250738585072014e-308, 1.7976931348623157e308,
                              1.0, -1.0, 0.5, 0.25, 2.0, 3.0, 4.0, 4.0 - 0x1p-51, 2.0 - 0x1p-52, 1.0 + 0x1p-52, 0x1p-1022};
    for (double a : special)
        for (double b : special) check(a, b);
    std::printf("checked %ld (%ld unflagged), differ %ld\n", n_checked, n_fast, n_bad);
    return n_bad != 0;
}
