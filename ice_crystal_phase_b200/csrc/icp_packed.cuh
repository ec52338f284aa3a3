// icp_packed.cuh -- packed binary32 pairs (sm_100a) and the activation's derivative in pairs, for the
// surrogate's epilogues and streaming kernels.
#pragma once
#include <cstdint>

namespace icp::mlp {

// Packed FP32 pairs (sm_100 add / mul / fma .f32x2: one instruction for two lanes of work).
__device__ __forceinline__ uint64_t pk2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk2(uint64_t r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// 2^x on the special-function unit with subnormal results flushed (one instruction; the
// exponential here is only ever added to 1).
__device__ __forceinline__ float ex2_ftz(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_ftz(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Logistic function s and derivative of z s(z) of a pair (the training kernels: both special functions on
// their unit, ~1e-7 relative; z clamped at -80).
__device__ __forceinline__ void silu_grad_pair(uint64_t z, uint64_t& s, uint64_t& grad)
{
    constexpr float kNegLog2e = -1.44269504088896341f;
    const uint64_t one = pk2(1.0f, 1.0f), m1 = pk2(-1.0f, -1.0f);
    float a, b;
    upk2(z, a, b);
    upk2(mul2(pk2(fmaxf(a, -80.0f), fmaxf(b, -80.0f)), pk2(kNegLog2e, kNegLog2e)), a, b);
    upk2(add2(pk2(ex2_ftz(a), ex2_ftz(b)), one), a, b);
    s = pk2(rcp_ftz(a), rcp_ftz(b));
    grad = mul2(s, fma2(z, fma2(s, m1, one), one));
}

} // namespace icp::mlp
