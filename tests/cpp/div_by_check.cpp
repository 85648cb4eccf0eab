// div_by (csrc/ae_div.h) against a / d: the rounded quotient, or the other neighbour where the quotient lies
// within 2^-47 units in the last place of the middle of two numbers.  Random mantissas and exponents, every
// exponent around the edges of the guard, reciprocals up to four units of 2^-53 off, zeros, subnormals,
// infinities and NaN.  Exit status 0 when every case holds.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <limits>
#include <random>

#include "ae_div.h"

static std::mt19937_64 rng(12345);

static double make(int exponent_field, uint64_t mantissa, bool negative) {
    const uint64_t b = (uint64_t)negative << 63 | (uint64_t)exponent_field << 52 | (mantissa & 0xfffffffffffffull);
    double v;
    std::memcpy(&v, &b, sizeof v);
    return v;
}
static uint64_t mantissa() {
    switch (rng() % 8) {
        case 0: return 0;
        case 1: return ~0ull;
        case 2: return rng() % 16;
        case 3: return ~(uint64_t)(rng() % 16);
        default: return rng();
    }
}
static long long differ = 0, total = 0;

static bool check(double a, double d, double inv) {
    const double c = ae::div_by(a, d, inv), w = a / d;
    ++total;
    if (c == w || (std::isnan(c) && std::isnan(w))) return true;
    ++differ;
    // the neighbour of w, and a / d near their middle: |a - d c| against |d| ulp / 2
    const bool up = c == std::nextafter(w, INFINITY), down = c == std::nextafter(w, -INFINITY);
    const double half = 0.5 * std::fabs(c - w) * std::fabs(d), r = std::fabs(std::fma(-d, c, a));
    if ((up || down) && std::isfinite(c) && std::fabs(r - half) <= std::ldexp(half, -46)) return true;
    std::printf("a %a d %a inv %a: %a, not %a\n", a, d, inv, c, w);
    return false;
}

// the reciprocals the callers pass: 1 / d rounded, and that off by up to three units more
static bool with_reciprocals(double a, double d) {
    const double inv = 1.0 / d;
    if (!check(a, d, inv)) return false;
    if (!std::isfinite(inv) || inv == 0.0) return true;
    for (int s : {-3, -1, 1, 3})
        if (!check(a, d, inv * (1.0 + s * std::ldexp(1.0, -53) * 0.999))) return false;
    return true;
}

int main() {
    for (int n = 0; n < 4000000; ++n) {  // exponents as weights and Krylov sums have them
        const double a = make(1023 - 40 + (int)(rng() % 80), mantissa(), rng() & 1);
        const double d = make(1023 - 40 + (int)(rng() % 80), mantissa(), rng() & 1);
        if (!with_reciprocals(a, d)) return 1;
    }
    for (int n = 0; n < 2000000; ++n) {  // the whole range
        const double a = make((int)(rng() % 2048), mantissa(), rng() & 1);
        const double d = make((int)(rng() % 2048), mantissa(), rng() & 1);
        if (!with_reciprocals(a, d)) return 1;
    }
    const int edge[] = {0, 1, 2, 62, 63, 64, 65, 66, 1022, 1023, 1024, 1981, 1982, 1983, 1984, 1985, 2045, 2046, 2047};
    for (int ea : edge)
        for (int ed : edge)
            for (int n = 0; n < 2000; ++n)
                if (!with_reciprocals(make(ea, mantissa(), rng() & 1), make(ed, mantissa(), rng() & 1))) return 1;
    // results at the edges: a from the exponent of the quotient and of d
    for (int eq : edge)
        for (int n = 0; n < 20000; ++n) {
            const int ed = 66 + (int)(rng() % 1900), ea = eq + ed - 1023 - (int)(rng() % 2);
            if (ea < 0 || ea > 2046) continue;
            if (!with_reciprocals(make(ea, mantissa(), rng() & 1), make(ed, mantissa(), rng() & 1))) return 1;
        }
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    const double den = std::numeric_limits<double>::denorm_min(), big = std::numeric_limits<double>::max();
    const double special[] = {0.0, -0.0, den, -den, 3 * den, 1e-310, 1.0, -1.0, 1.5, big, -big, inf, -inf, nan};
    for (double a : special)
        for (double d : special)
            if (!check(a, d, 1.0 / d)) return 1;
    std::printf("ok: %lld quotients, %lld at the middle of two numbers\n", total, differ);
    return 0;
}
