// pearl_division.hpp — host side of the kernels' division by a constant.
//
// A divisor b known in advance is replaced by two constants, zh = RN(1/b) and
// zl close to 1/b - zh, and a/b by RN(a*zh + RN(a*zl)): one multiplication and
// one fused multiply-add (Brisebarre, Muller, Raina, "Accelerating correctly
// rounded floating-point division when the divisor is known in advance", IEEE
// Trans. Comput. 53(8), 2004).  The result is the correctly rounded quotient
// for every normal a with a normal quotient unless a/b lies closer to the
// midpoint of two neighbouring doubles than the method's error, and for one b
// only a handful of significands a come that close: they solve
// a 2^s = m b + n with m odd and |n| small.  exact_reciprocal() solves for them
// and tries each, so a pair that it returns is right for all a.
#pragma once

#include <cmath>
#include <cstdint>
#include <initializer_list>

namespace pearl_gpu {

namespace division_detail {

inline uint64_t mul_mod(uint64_t a, uint64_t b, uint64_t m) { return (uint64_t)((unsigned __int128)a * b % m); }

// Significands A in [2^52, 2^53) with A 2^s = M B + n, M odd, |n| < 8, where
// s = 53 for A >= B and 54 for A < B (so that M / 2 is the scaled quotient's
// midpoint).  Calls f(A) for each until it returns false.
//
// The bound on |n|: with zl at most 1.5 units in its last place from 1/b - zh,
// |zh + zl - 1/b| <= 3 2^-106 / b and the rounding of a*zl adds 2^-106 |a/b|, so
// the value before the last rounding is within 2^-51 units in the last place of
// the quotient; a distance of |n| / (2B) >= |n| 2^-54 units below that means
// |n| < 8.
template <class F>
bool near_midpoints(uint64_t B, F&& f) {
    int t = 0;
    while (!((B >> t) & 1)) ++t;
    const uint64_t Bo = B >> t, lo = 1ull << 52, hi = 1ull << 53;
    if (Bo == 1) return true;  // a power of two divides exactly
    const uint64_t half = (Bo + 1) / 2;  // 1/2 modulo Bo
    for (int s = 53; s <= 54; ++s) {
        uint64_t inv = 1;  // 2^-(s - t) modulo Bo
        for (int k = 0; k < s - t; ++k) inv = mul_mod(inv, half, Bo);
        for (int n = -7; n <= 7; ++n) {
            if (n == 0 || n % (1 << (t < 5 ? t : 5)) != 0) continue;  // 2^t has to divide n
            const int no = n / (1 << (t < 5 ? t : 5));
            const uint64_t residue = no > 0 ? (uint64_t)no % Bo : (Bo - (uint64_t)(-no) % Bo) % Bo;
            uint64_t A = mul_mod(residue, inv, Bo);
            if (A < lo) A += (lo - A + Bo - 1) / Bo * Bo;
            for (; A < hi; A += Bo) {
                if ((s == 53) != (A >= B)) continue;
                const __int128 x = ((__int128)A << s) - n;
                if (x % B != 0 || !((x / B) & 1)) continue;
                if (!f(A)) return false;
            }
        }
    }
    return true;
}

}  // namespace division_detail

// Constants (zh, zl) for the divisor b, true when they give a/b for all normal
// a with a normal quotient.  zl is 1/b - zh rounded, or a neighbour of it where
// that one misses a quotient (about one divisor in 160); for one divisor in a
// thousand none of the three does, and the kernels divide with div_exact.
inline bool exact_reciprocal(double b, double& zh, double& zl) {
    zh = 1.0 / b;
    zl = std::fma(-b, zh, 1.0) / b;  // the residual is exact
    if (std::fpclassify(b) != FP_NORMAL || std::fpclassify(zh) != FP_NORMAL) return false;
    if (zl != 0 && std::fpclassify(zl) != FP_NORMAL) return false;
    int e = 0;
    const double m = std::ldexp(std::frexp(std::fabs(b), &e), 53);  // scaling by powers of two changes no rounding
    const double mh = 1.0 / m, ml = std::fma(-m, mh, 1.0) / m;
    for (double l : {ml, std::nextafter(ml, INFINITY), std::nextafter(ml, -INFINITY)}) {
        const bool ok = division_detail::near_midpoints((uint64_t)m, [&](uint64_t A) {
            const double a = (double)A;
            return std::fma(a, mh, a * l) == a / m;
        });
        if (ok) {
            zl = std::copysign(1.0, b) * std::ldexp(l, 53 - e);
            return true;
        }
    }
    return false;
}

}  // namespace pearl_gpu
