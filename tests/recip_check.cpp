// Division by a known divisor with the two-term reciprocal (csrc/bfb_recip.h)
// against IEEE division: argv[1] divisors of the Thomas factors' range, each
// with random numerators, the numerators nearest to the midpoints (listed here
// by walking the quotients' midpoints, not by the header's own search) and
// powers of two. Prints "<accepted> <refused> <mismatches>".
#include <cstdio>
#include <cstdlib>
#include <random>

#include "bfb_recip.h"

int main(int argc, char **argv) {
    const int n = argc > 1 ? std::atoi(argv[1]) : 1000;
    std::mt19937_64 g(20240);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    long accepted = 0, refused = 0, bad = 0;
    for (int i = 0; i < n; ++i) {
        double b;
        if (i % 8 == 7) b = 1.0 + (double)(g() % 64) / (double)(1ull << (g() % 7));  // few mantissa bits
        else b = 1.0 + std::exp(std::log(1e-4) + u(g) * std::log(1e8)) * (1.0 + u(g));
        const double hi = 1.0 / b;
        double lo;
        if (!bfb::two_term_reciprocal(b, hi, &lo)) {
            ++refused;
            continue;
        }
        ++accepted;
        auto check = [&](double t) {
            if (std::fma(t, hi, t * lo) != t / b) ++bad;
        };
        for (int q = 0; q < 400; ++q) check((u(g) - 0.5) * std::ldexp(1.0, (int)(g() % 200) - 100));
        for (int q = -100; q <= 100; ++q) check(std::ldexp(1.0, q));
        // numerators next to the product of b with a midpoint between two doubles
        for (int q = 0; q < 400; ++q) {
            const double x = 1.0 + u(g), h = std::ldexp(1.0, -53);  // midpoint x + h
            const double p = std::fma(h, b, x * b);
            for (double t : {p, std::nextafter(p, 0.0), std::nextafter(p, 1e300)}) check(t);
        }
    }
    std::printf("%ld %ld %ld\n", accepted, refused, bad);
    return 0;
}
