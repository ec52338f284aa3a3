// icp_quot.cuh -- quotients by one divisor.  Host and device code alike (the host test compiles it
// with g++).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define ICP_QUOT_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define ICP_QUOT_HD inline
#endif
#ifndef __CUDA_ARCH__
#include <cstring>
#endif

namespace icp {

// Quotients by one divisor, rounded as the division operator rounds them.  The reciprocal is
// evaluated once (correctly rounded), and each quotient is refined twice with the exact FMA
// remainder: Markstein's theorem (IBM J. Res. Dev. 34, 1990) gives the correctly rounded quotient
// from a correctly rounded reciprocal and a faithful quotient, away from overflow and underflow.
// Numerators or divisors outside 2^-450 .. 2^450 take the operator (zeros keep their sign): inside,
// quotients lie within 2^-901 .. 2^901 and remainders above 2^-560.  The operator costs the FP64 trace
// kernels a divergent call for every zero component and the same reciprocal again for every
// component of a vector.
struct DivBy {
    double b, y;
    bool ok;
};
ICP_QUOT_HD bool mid_range(double x)
{
#ifdef __CUDA_ARCH__
    const uint32_t high = (uint32_t)__double2hiint(x);
#else
    uint64_t bits;
    std::memcpy(&bits, &x, sizeof bits);
    const uint32_t high = (uint32_t)(bits >> 32);
#endif
    return (high & 0x7fffffffu) - 0x23d00000u < 0x38400000u; // exponents -450 .. 449
}
ICP_QUOT_HD DivBy div_by(double b)
{
#ifdef __CUDA_ARCH__
    return {b, __drcp_rn(b), mid_range(b)};
#else
    return {b, 1.0 / b, mid_range(b)};
#endif
}
ICP_QUOT_HD double quot(double a, const DivBy& d)
{
    const double q0 = a * d.y;
    const double q1 = fma(fma(-d.b, q0, a), d.y, q0);
    double q = fma(fma(-d.b, q1, a), d.y, q1);
    if (!(mid_range(a) && d.ok)) {
        q = q0;
        if (!(a == 0 && d.ok)) q = a / d.b;
    }
    return q;
}

} // namespace icp
