// icp_outward.cuh -- the neighbours of a number, for outward-rounded enclosures.  Host and device code
// alike (the host test compiles it with g++ -frounding-math).
#pragma once

#ifdef __CUDACC__
#define ICP_OUTWARD_HD __host__ __device__ __forceinline__
#else
#define ICP_OUTWARD_HD inline
#endif
#ifndef __CUDA_ARCH__
#include <cfenv>
#endif

namespace icp {

#ifndef __CUDA_ARCH__
template <class T> inline T add_rounded(T x, T y, int mode)
{
    const int before = std::fegetround();
    std::fesetround(mode);
    const volatile T a = x, b = y;
    const volatile T sum = a + b;
    std::fesetround(before);
    return sum;
}
#endif

// nextUp: the least representable number above x (+inf and NaN unchanged, either zero to the
// least positive subnormal); nextDown(x) = -nextUp(-x).  x plus the least subnormal, rounded up, is
// that number for every x but -inf, which stays, the sign of a zero apart: one addition where the step
// on the bits takes six operations.  An enclosure whose finite end has overflowed stays infinite, on the side
// that excludes it already.
ICP_OUTWARD_HD float next_up(float x)
{
#ifdef __CUDA_ARCH__
    return __fadd_ru(x, 0x1p-149f);
#else
    return add_rounded(x, 0x1p-149f, FE_UPWARD);
#endif
}
ICP_OUTWARD_HD double next_up(double x)
{
#ifdef __CUDA_ARCH__
    return __dadd_ru(x, 0x1p-1074);
#else
    return add_rounded(x, 0x1p-1074, FE_UPWARD);
#endif
}
ICP_OUTWARD_HD float next_down(float x)
{
#ifdef __CUDA_ARCH__
    return __fadd_rd(x, -0x1p-149f);
#else
    return add_rounded(x, -0x1p-149f, FE_DOWNWARD);
#endif
}
ICP_OUTWARD_HD double next_down(double x)
{
#ifdef __CUDA_ARCH__
    return __dadd_rd(x, -0x1p-1074);
#else
    return add_rounded(x, -0x1p-1074, FE_DOWNWARD);
#endif
}

} // namespace icp
