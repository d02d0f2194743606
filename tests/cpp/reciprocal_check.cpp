// unb::refine_reciprocal from starts as far off as it allows (a relative error
// of 2^-16 either way), over random and awkward significands: 1 / b exactly;
// for a significand of all ones, one of the two numbers that `reciprocal`
// decides between by its bits, the second of which is 1 / b. Prints the number
// of differences.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>

#include "quotient.hpp"

static uint64_t state = 0x9E3779B97F4A7C15ull;
static uint64_t next() {
    state ^= state << 13; state ^= state >> 7; state ^= state << 17;
    return state;
}
static double make(uint64_t significand, int exponent) {
    const uint64_t u = (uint64_t(exponent + 1023) << 52) | (significand & 0xFFFFFFFFFFFFFull);
    double d;
    std::memcpy(&d, &u, 8);
    return d;
}

int main() {
    const uint64_t ones = 0xFFFFFFFFFFFFFull;
    long differ = 0;
    for (int i = 0; i < 4000000; ++i) {
        const uint64_t pick = next() % 8;
        const uint64_t sig = pick == 0 ? ones - 1 - next() % 64 : pick == 1 ? next() % 64 : next() % ones;   // (not all ones)
        const double b = make(sig, int(next() % 281) - 40), r = 1.0 / b;
        for (double e : {0x1p-16, -0x1p-16, (double(next() % 20001) - 10000.0) / 10000.0 * 0x1p-16})
            if (unb::refine_reciprocal(b, r * (1.0 + e)) != r) ++differ;
    }
    for (int k = -40; k <= 240; ++k) {
        const double b = make(ones, k), r = 1.0 / b;
        if (r != std::nextafter(std::ldexp(1.0, -k - 1), 1e300)) ++differ;   // the number above a power of two
        for (int i = 0; i < 1000; ++i) {
            const double y = unb::refine_reciprocal(b, r * (1.0 + (double(next() % 20001) - 10000.0) / 10000.0 * 0x1p-16));
            if (y != r && y != std::ldexp(1.0, -k - 1)) ++differ;
        }
    }
    std::printf("%ld\n", differ);
    return differ ? 1 : 0;
}
