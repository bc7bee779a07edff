// Quotients of fast_div against the division, for the divisors of argv: every
// numerator around each multiple that a lattice of 2^27 nodes reaches near its
// ends, powers of two, and random ones, all below 2^31.  A divisor below 2
// prints "refused".
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <stdexcept>

#include "fast_div.h"

int main(int argc, char** argv) {
    std::mt19937 random(7);
    for (int a = 1; a < argc; ++a) {
        const auto d = static_cast<uint32_t>(std::strtoul(argv[a], nullptr, 10));
        orr::FastDiv f;
        try {
            f = orr::fast_div(d);
        } catch (const std::domain_error&) {
            std::printf("%u refused\n", d);
            continue;
        }
        uint64_t wrong = 0;
        const auto check = [&](uint64_t n) {
            if (n < (uint64_t{1} << 31)) {
                wrong += orr::divide(static_cast<uint32_t>(n), f) != n / d;
            }
        };
        const uint64_t top = ((uint64_t{1} << 31) - 1) / d;
        for (uint64_t k = 0; k < 4096; ++k) {
            for (const uint64_t multiple : {k, top - (k < top ? k : top), random() % (top + 1)}) {
                check(multiple * d);
                check(multiple * d + d - 1);
                check(multiple * d + 1);
            }
            check(random() >> 1);
        }
        for (int b = 0; b < 31; ++b) {
            check(uint64_t{1} << b);
            check((uint64_t{1} << b) - 1);
        }
        check((uint64_t{1} << 31) - 1);
        std::printf("%u %llu\n", d, static_cast<unsigned long long>(wrong));
    }
}
