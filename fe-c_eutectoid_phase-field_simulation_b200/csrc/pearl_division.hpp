// pearl_division.hpp — host side of the kernels' division by a constant.
//
// A divisor b known in advance is replaced by two constants, zh = RN(1/b) and
// zl close to 1/b - zh, and a/b by RN(a*zh + RN(a*zl)): one multiplication and
// one fused multiply-add (Brisebarre, Muller, Raina, "Accelerating correctly
// rounded floating-point division when the divisor is known in advance", IEEE
// Trans. Comput. 53(8), 2004).  As long as a*zl is a normal number, the result is
// the correctly rounded quotient unless a/b lies closer to the
// midpoint of two neighbouring doubles than the method's error, and for one b
// only a handful of significands a come that close: they solve
// a 2^s = m b + n with m odd and |n| small.  exact_reciprocal() solves for them
// and tries each, so a pair that it returns is right for all a of that range.
//
// The range: 1 - b zh is a multiple of 2^-105, so |a*zl| is at least about
// 2^-105 |a/b| (or zl is 0 and a*zh exact), and every quotient from kExactFrom up
// to the largest double is in it.  Below, a*zl loses bits to underflow, and a normal
// quotient may be one unit in the last place off (1 of 300 numerators between
// 2^-1000 and 2^-980 at b = 9.4e6).  No result hangs on that unit: a force's
// quotient is added to obstacle terms of some 1e7, a face weight to a
// susceptibility, a gradient's energy is its square, and what a chemical energy or
// a phase's composition divides is 0 or a difference of numbers far above that range.
#pragma once

#include <cmath>
#include <cstdint>
#include <initializer_list>

namespace pearl_gpu {

// The smallest |a/b| whose rounding exact_reciprocal answers for.
constexpr double kExactFrom = 0x1p-916;

namespace division_detail {

// Calls f(A) until it returns false for the significands A in [2^52, 2^53) with
// A 2^s = M B + n, |n| < 8, where s = 53 (for A >= B) or 54 (for A < B): with M
// odd, M / 2 is a midpoint of the scaled quotient.  (An even M is a quotient
// next to a double, which f finds right as well: M is not looked at.)
//
// The bound on |n|: with zl at most 1.5 units in its last place from 1/b - zh,
// |zh + zl - 1/b| <= 3 2^-106 / b and the rounding of a*zl adds 2^-106 |a/b|, so
// the value before the last rounding is within 2^-51 units in the last place of
// the quotient; a distance of |n| / (2B) >= |n| 2^-54 units below that means
// |n| < 8.
//
// A few hundred nanoseconds: a single step on a small domain pays for nine.
template <class F>
bool near_midpoints(uint64_t B, F&& f) {
    int t = 0;
    while (!((B >> t) & 1)) ++t;
    if (t > 2) return true;  // 2^t divides n
    const uint64_t Bo = B >> t, lo = 1ull << 52, hi = 1ull << 53;
    uint64_t inv64 = Bo;  // 1/Bo modulo 2^64 by Newton's iteration (right to 3 bits at first)
    for (int k = 0; k < 5; ++k) inv64 *= 2 - Bo * inv64;
    for (int s = 53; s <= 54; ++s) {
        // 2^-(s - t) modulo Bo: (1 + Bo m) / 2^(s - t) with m = -1/Bo modulo 2^(s - t)
        const int k = s - t;
        const uint64_t m = (0 - inv64) & ((1ull << k) - 1);
        const uint64_t inv = (uint64_t)(((unsigned __int128)Bo * m + 1) >> k);
        uint64_t r = 0;
        for (int n = 1; n << t < 8; ++n) {
            r += inv;
            if (r >= Bo) r -= Bo;
            for (uint64_t A : {r, Bo - r})
                for (A += A < lo ? (lo - A + Bo - 1) / Bo * Bo : 0; A < hi; A += Bo)
                    if (!f(A)) return false;
        }
    }
    return true;
}

}  // namespace division_detail

// Constants (zh, zl) for the divisor b, true when they give a/b for all a with
// |a/b| from kExactFrom to the largest double.  zl is 1/b - zh rounded, or a neighbour of it where
// that one misses a quotient (about one divisor in 160); for one divisor in a
// thousand none of the three does, and the kernels of the general division run.
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
