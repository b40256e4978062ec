// bfb_recip.h -- two-term reciprocals for division by a known divisor (host).
//
// With hi = RN(1/b) and lo close to 1/b - hi, the two operations
//     w = RN(t * lo),  q = RN(t * hi + w)        (one multiply, one FMA)
// give t/b correctly rounded for every t unless t/b lies very close to the
// midpoint of two doubles (N. Brisebarre, J.-M. Muller, S. K. Raina,
// "Accelerating correctly rounded floating-point division when the divisor is
// known in advance", IEEE Trans. Computers 53(8), 2004). The numerators for
// which it does are few and can be listed for a given b, so each divisor is
// either proven, by trying them all, or refused.
//
// The list. Let t = X 2^e and b = Y 2^f with X, Y integers in [2^52, 2^53).
// The value before the last rounding is t/b (1 + d) with
// |d| <= (1/2 + j) 2^-105 + 2^-106 when lo is the double nearest to 1/b - hi
// moved by at most j of its own ulps. A wrong rounding needs a midpoint within
// |d| t/b of t/b: with k = 53 (X >= Y, quotient in [1, 2)) or k = 54 (X < Y),
// |X 2^k - (2M + 1) Y| <= |d| X 2^k, which is below 4.01 (1 + j). So X solves
// X 2^k = r (mod Y) for some |r| <= recip_window(j) (r = 0 would make t/b a
// midpoint, which no quotient is). The argument is free of scale as long as
// nothing underflows: |t| above 2^-968 or 0, and finite. Below that quotients
// can be off by one unit in the last place (from about 2^-994 down, most often,
// one in ten, near 2^-1022; the residual form's are from 2^-1002 down).
#pragma once
#include <cmath>
#include <cstdint>
#include <initializer_list>
#include <utility>
#include <vector>

namespace bfb {

constexpr int recip_window(int j) { return 4 * (1 + j) + 2; }

// Calls f(X) for every candidate numerator of divisor mantissa Y (P-bit
// mantissas, residues up to W); stops when f returns false.
template <int P = 53, typename F>
inline bool recip_candidates(uint64_t Y, int W, F f) {
    constexpr uint64_t lo = 1ull << (P - 1), hi = 1ull << P;
    int s = 0;  // Y = 2^s Yo: X 2^k = r (mod Y) needs 2^s | r, and then X = r 2^-k (mod Yo)
    uint64_t Yo = Y;
    while (!(Yo & 1)) {
        Yo >>= 1;
        ++s;
    }
    if ((W >> s) == 0) return true;  // every |r| <= W but 0 is ruled out (and for Yo = 1 the reciprocal is exact)
    // 2^-P mod Yo = (1 + Yo m) / 2^P with m = -1/Yo mod 2^P (Newton's iteration
    // doubles the 3 bits that Yo is its own inverse to)
    uint64_t m = Yo;
    for (int it = 0; it < 5; ++it) m *= 2 - Yo * m;
    m = (0 - m) & (hi - 1);
    uint64_t inv = (uint64_t)(((unsigned __int128)Yo * m + 1) >> P);
    for (int k = P; k <= P + 1; ++k) {
        if (k > P) inv = (inv & 1) ? (inv + Yo) >> 1 : inv >> 1;
        uint64_t x = 0;
        for (int r = 1; r <= W; ++r) {
            x += inv;  // r 2^-k mod Yo
            if (x >= Yo) x -= Yo;
            if (s && (r & ((1 << s) - 1))) continue;
            for (int sign = 0; sign < 2; ++sign) {
                uint64_t X = sign ? Yo - x : x;
                if (X < lo) X += (lo - X + Yo - 1) / Yo * Yo;
                for (; X < hi; X += Yo)
                    if ((k == P) == (X >= Y) && !f(X)) return false;
            }
        }
    }
    return true;
}

// lo for divisor b with hi = RN(1/b), or false when b is not a normal positive
// number or no lo within two ulps is right for every numerator (about one
// divisor in 1600). The nearest lo does for all but one in 120, and its window
// is the smallest.
inline bool two_term_reciprocal(double b, double hi, double *lo_out) {
    if (!std::isnormal(b) || !std::isnormal(hi) || b <= 0) return false;
    int e;
    const double m = std::frexp(b, &e);  // [1/2, 1)
    const uint64_t Y = (uint64_t)std::ldexp(m, 53);
    const double h1 = std::ldexp(hi, e - 53);  // RN(1/Y), exactly hi scaled
    const double y = (double)Y;
    const double l1 = std::fma(-h1, y, 1.0) / y;
    if (l1 != 0.0 && !std::isnormal(l1)) return false;
    double up = l1, down = l1;
    for (int j = 0; j <= 2; ++j) {
        for (const double l : {up, down}) {
            if (recip_candidates(Y, recip_window(j), [&](uint64_t X) {
                    const double t = (double)X;
                    return std::fma(t, h1, t * l) == t / y;
                })) {
                *lo_out = std::ldexp(l, 53 - e);
                return std::isnormal(*lo_out) || *lo_out == 0.0;
            }
        }
        up = std::nextafter(up, 1.0);
        down = std::nextafter(down, -1.0);
    }
    return false;
}

// The low terms of a factor table's divisors, [row][substrate].
struct RecipTable {
    std::vector<double> den, lo;  // lo 0 where not proven
    std::vector<char> state;      // kNotTried, kProven, kRefused
    int S = 0;
    long proofs = 0;              // divisors tried by prove_rows
    static constexpr char kNotTried = 0, kProven = 1, kRefused = 2;
};

// Proves rows 1 .. last of `den` ([row][S], hi = RN(1/den)) into t. t holds
// another axis' table or nothing: the axes of a uniform mesh have the same
// divisors but for their last rows, so each is tried once.
inline void prove_rows(const std::vector<double> &den, const std::vector<double> &hi, int S, int last, RecipTable &t) {
    const RecipTable old = std::move(t);
    t = RecipTable();
    t.den = den;
    t.lo.assign(den.size(), 0.0);
    t.state.assign(den.size(), RecipTable::kNotTried);
    t.S = S;
    for (size_t q = S; q < (size_t)(last + 1) * S; ++q) {
        if (old.S == S && q < old.den.size() && old.state[q] && old.den[q] == den[q]) {
            t.state[q] = old.state[q];
            t.lo[q] = old.lo[q];
            continue;
        }
        double lo = 0.0;
        ++t.proofs;
        if (two_term_reciprocal(den[q], hi[q], &lo)) {
            t.state[q] = RecipTable::kProven;
            t.lo[q] = lo;
        } else {
            t.state[q] = RecipTable::kRefused;
        }
    }
}

}  // namespace bfb
