// Quotients of 32-bit numbers by a divisor known before the launch, by one
// multiplication (the node coordinates of the linear-order steps).
#pragma once

#include <cstdint>
#include <stdexcept>

#if defined(__CUDACC__)
#define ORR_FAST_DIV_HD __host__ __device__ __forceinline__
#else
#define ORR_FAST_DIV_HD inline
#endif

namespace orr {

struct FastDiv {
    uint32_t mul = 0, shift = 0;
};

// For d >= 2 and quotients of n < 2^31 (n / 1 is not of the form below, and
// a lattice has at least 3 nodes along each axis).
inline FastDiv fast_div(uint32_t d) {
    if (d < 2u) {
        throw std::domain_error("fast_div: the divisor must be at least 2");
    }
    // mul = ceil(2^(32 + shift) / d) with 2^shift <= d < 2^(shift + 1): mul d
    // exceeds 2^(32 + shift) by less than d, so n mul / 2^(32 + shift) is below
    // n / d + 1 / d while n < 2^31.  A power of two takes half of both.
    FastDiv f;
    while ((d >> f.shift) > 1u) ++f.shift;
    if ((d & (d - 1u)) == 0u) {
        f.mul = 1u << 31;
        --f.shift;
    } else {
        f.mul = static_cast<uint32_t>(((uint64_t{1} << (32 + f.shift)) + d - 1u) / d);
    }
    return f;
}

ORR_FAST_DIV_HD uint32_t divide(uint32_t n, FastDiv f) {
#if defined(__CUDA_ARCH__)
    return __umulhi(n, f.mul) >> f.shift;
#else
    return static_cast<uint32_t>((static_cast<uint64_t>(n) * f.mul) >> 32) >> f.shift;
#endif
}

} // namespace orr
