// croma_bits.cuh -- arithmetic on the exponent field of doubles, the same on
// the host and the device.  No other header of this library, and nothing of
// CUDA, is needed to compile it.
#pragma once

#include <cstring>

#ifndef CROMA_HD
#ifdef __CUDACC__
#define CROMA_HD __host__ __device__ __forceinline__
#else
#define CROMA_HD inline
#endif
#endif

namespace croma {

// sign, exponent and the upper twenty bits of the fraction
CROMA_HD unsigned high_word(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(x);
#else
    unsigned long long u;
    std::memcpy(&u, &x, sizeof u);
    return (unsigned)(u >> 32);
#endif
}

// A pivot n / th counts as zero (the reference's |d| <= 1e-300): |n| below |th|
// by a factor of 2^996, compared in the exponent fields.  Unsigned: the sum
// passes 2^31 from |n| = 2^29 on, which continuants reach within eight rows; it
// stays below 2^32 for every n.
CROMA_HD bool continuant_singular(double n, double th)
{
    return (high_word(n) & 0x7fffffffu) + (996u << 20) < (high_word(th) & 0x7fffffffu);
}

}  // namespace croma
