// The two-term reciprocal (csrc/bfb_recip.h) on numerators and mantissa widths
// given by tests/test_recip_hard_cpu.py.
//   recip_hard divide      stdin: lines "b n X1 .. Xn" (b as %a, X integers in
//                          [2^52, 2^53)); prints per line "accepted wrong nearest
//                          least": quotients X/b that differ from IEEE division
//                          with the header's low term, with the nearest low term,
//                          and the least over all low terms that the header tries
//   recip_hard search P    for every P-bit mantissa Y (P 10 or 12) a line "Y X1 X2 ..."
//                          of the numerators that the header's search visits (residues to 4)
//   recip_hard axes n..    per axis length "proofs alone, proofs after the axes before, same result"
#include "bfb_recip.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

template <int P>
static void search() {
    for (uint64_t Y = 1ull << (P - 1); Y < 1ull << P; ++Y) {
        std::printf("%llu", (unsigned long long)Y);
        bfb::recip_candidates<P>(Y, 4, [](uint64_t X) {
            std::printf(" %llu", (unsigned long long)X);
            return true;
        });
        std::printf("\n");
    }
}

// Divisors as the axes of an nx x ny x nz mesh have them: "proofs" tried per axis,
// and whether each axis' states and low terms are those of a proof on its own.
static int axes(int argc, char **argv) {
    const int S = 3;
    bfb::RecipTable shared;
    for (int a = 2; a < argc; ++a) {
        const int n = std::atoi(argv[a]);
        std::vector<double> den((size_t)n * S), hi(den.size());
        for (int d = 0; d < S; ++d) {
            const double c1 = 0.3 * std::pow(7.0, d), c3a = 1.0 + 0.001 + c1, c3 = c3a + c1;
            double c = 0;
            for (int m = 0; m < n; ++m) {
                const double b = (m == 0 || m == n - 1 ? c3a : c3) - (m ? c1 * c : 0.0);
                den[(size_t)m * S + d] = b;
                c = c1 / b;
            }
        }
        for (size_t q = 0; q < den.size(); ++q) hi[q] = 1.0 / den[q];
        bfb::RecipTable alone;
        bfb::prove_rows(den, hi, S, n - 1, shared);
        bfb::prove_rows(den, hi, S, n - 1, alone);
        std::printf("%ld %ld %d\n", alone.proofs, shared.proofs, shared.state == alone.state && shared.lo == alone.lo);
    }
    return 0;
}

int main(int argc, char **argv) {
    if (argc > 2 && !std::strcmp(argv[1], "axes")) return axes(argc, argv);
    if (argc > 2 && !std::strcmp(argv[1], "search")) {
        if (std::atoi(argv[2]) == 10) search<10>();
        else search<12>();
        return 0;
    }
    double b;
    int n;
    while (std::scanf("%la %d", &b, &n) == 2) {
        std::vector<double> t(n);
        for (double &v : t)
            if (std::scanf("%lf", &v) != 1) return 1;
        const double hi = 1.0 / b;
        auto wrong = [&](double lo) {
            int bad = 0;
            for (double v : t) bad += std::fma(v, hi, v * lo) != v / b;
            return bad;
        };
        double lo = 0;
        const bool ok = bfb::two_term_reciprocal(b, hi, &lo);
        const double nearest = std::fma(-hi, b, 1.0) / b;
        int least = wrong(nearest);
        for (double to : {1.0, -1.0}) {
            double l = nearest;
            for (int j = 0; j < 2; ++j) least = std::min(least, wrong(l = std::nextafter(l, to)));
        }
        std::printf("%d %d %d %d\n", ok ? 1 : 0, ok ? wrong(lo) : 0, wrong(nearest), least);
    }
    return 0;
}
