// Compares unb::quotient with the division it replaces, bit for bit where the
// quotient is a normal number, over random and awkward operands. Prints the number of differences.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "quotient.hpp"

static uint64_t state = 0x9E3779B97F4A7C15ull;
static uint64_t next() {
    state ^= state << 13; state ^= state >> 7; state ^= state << 17;
    return state;
}
static double make(uint64_t mantissa, int exponent) {
    const uint64_t u = (uint64_t(exponent + 1023) << 52) | (mantissa & 0xFFFFFFFFFFFFFull);
    double d;
    std::memcpy(&d, &u, 8);
    return d;
}

int main() {
    long differ = 0, tried = 0;
    auto check = [&](double a, double b) {
        ++tried;
        const double q = unb::quotient(a, b, 1.0 / b), e = a / b;
        // A subnormal quotient may be off by its last bit.
        if (std::fabs(e) < 0x1p-1022 ? std::fabs(q - e) > 0x1p-1074 : q != e) ++differ;
    };
    // Significands: all ones, all ones but the last bits, one, one and the last bits, random.
    auto significand = [&](int k) -> uint64_t {
        switch (k) {
        case 0: return 0xFFFFFFFFFFFFFull;
        case 1: return 0xFFFFFFFFFFFFFull - next() % 64;
        case 2: return 0;
        case 3: return next() % 64;
        default: return next();
        }
    };
    for (int i = 0; i < 4000000; ++i) {
        const double b = make(significand(int(next() % 8)), int(next() % 280) - 39);
        const double a = make(significand(int(next() % 8)), int(next() % 1500) - 900);
        check(a, b);
        check(-a, b);
    }
    // Composite alphas: near one, where an opaque stack's rounding leaves them.
    for (int i = 0; i < 4000000; ++i) {
        const double al = make(next(), -int(next() % 40) - 1), dd = 1.0 - double(next() % 3) * 0x1p-53;
        const double b = dd * (1.0 - al) + (al * dd + al * (1.0 - dd));
        check(make(significand(int(next() % 8)), int(next() % 80) - 78), b);
    }
    check(0.0, 0.75);
    // The reciprocal from approximations good to 2^-20 (either side).
    for (int i = 0; i < 4000000; ++i) {
        const double b = make(significand(int(next() % 8)), int(next() % 280) - 39);
        uint64_t u;
        std::memcpy(&u, &b, 8);
        if ((u & 0xFFFFFFFFFFFFFull) == 0xFFFFFFFFFFFFFull) continue;   // (all ones: set by its bits)
        const double r = 1.0 / b, y = unb::refine_reciprocal(b, r * (1.0 + (double(next() % 2001) - 1000.0) * 0x1p-30));
        ++tried;
        if (y != r) ++differ;
    }
    std::printf("%ld of %ld\n", differ, tried);
    return differ ? 1 : 0;
}
