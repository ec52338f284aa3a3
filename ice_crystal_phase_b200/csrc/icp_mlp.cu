// icp_mlp.cu -- the surrogate's kernels around the tensor-core GEMMs: input rows, the per-record
// softmax loss, the head's backward pass, Adam with the BF16 weight copies, and cell probabilities
// of stored CDF records (the training targets).  All are bandwidth-bound streaming kernels:
// 16-byte loads / stores along the contiguous dimension, one block per 128-1024 rows.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "icp_mlp.h"
#include "icp_mlp_features.cuh"
#include "icp_packed.cuh"

namespace icp::mlp {

namespace {

// X rows: thread per 8 BF16 (one uint4) of a row.  A warp takes two neighbouring chunks of 16 rows (whole
// 32-byte sectors), so that it copies record features, copies cell features or evaluates harmonics; a warp
// of two rows ran all three, with half its lanes idle (0.26 ms for 16 records of 131072 rows; 0.15 ms so).
__global__ void features_kernel(const uint4* __restrict__ rec16, const uint4* __restrict__ cells, uint32_t C,
                                uint32_t q_row, uint32_t q_axis, uint32_t warps, const double* __restrict__ recgeo,
                                const double* __restrict__ cellgeo, uint4* __restrict__ X)
{
    const uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (w >= warps) return;
    const uint32_t pairs = q_row / 2u, tile = w / pairs;
    const uint32_t q = 2u * (w - tile * pairs) + (lane & 1u);
    const uint32_t m = 16u * tile + (lane >> 1);
    const uint32_t r = m / C, c = m - r * C;
    const uint64_t t = (uint64_t)m * q_row + q;
    if (q < 2) {
        X[t] = rec16[2u * r + q];
    } else if (q < q_axis) {
        X[t] = cells[(uint64_t)c * (q_row - 2) + (q - 2)];
    } else {
        __align__(16) __nv_bfloat16 h[8];
        axis_harmonics8(cos_psi(recgeo, cellgeo, r, c), 1u + 8u * (q - q_axis), h);
        X[t] = *reinterpret_cast<const uint4*>(h);
    }
}

__device__ __forceinline__ double block_sum(double v, double* sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const uint32_t w = threadIdx.x >> 5, l = threadIdx.x & 31u, nw = blockDim.x >> 5;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double s = 0;
    for (uint32_t i = 0; i < nw; ++i) s += sh[i];
    return s;
}
__device__ __forceinline__ float block_max(float v, float* sh)
{
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const uint32_t w = threadIdx.x >> 5, l = threadIdx.x & 31u, nw = blockDim.x >> 5;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    float s = sh[0];
    for (uint32_t i = 1; i < nw; ++i) s = fmaxf(s, sh[i]);
    return s;
}

// One block per record: max, log-sum-exp (FP64 sums), KL loss and dy.
__global__ void __launch_bounds__(1024) softmax_loss_kernel(const float* __restrict__ y, const float* __restrict__ p,
                                                            uint32_t C, float scale, float* __restrict__ dy,
                                                            double* __restrict__ loss)
{
    __shared__ double shd[32];
    __shared__ float shf[32];
    const uint64_t base = (uint64_t)blockIdx.x * C;
    const float4* y4 = reinterpret_cast<const float4*>(y + base);
    const float4* p4 = reinterpret_cast<const float4*>(p + base);
    const uint32_t n4 = C / 4u;
    float mx = -INFINITY;
    for (uint32_t i = threadIdx.x; i < n4; i += blockDim.x) {
        const float4 v = y4[i];
        mx = fmaxf(mx, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
    }
    mx = block_max(mx, shf);
    double se = 0, py = 0, plp = 0;
    for (uint32_t i = threadIdx.x; i < n4; i += blockDim.x) {
        const float4 v = y4[i], q = p4[i];
        const float ys[4] = {v.x, v.y, v.z, v.w}, ps[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            se += (double)__expf(ys[j] - mx);
            if (ps[j] > 0.0f) {
                py += (double)ps[j] * (double)(ys[j] - mx);
                plp += (double)ps[j] * log((double)ps[j]);
            }
        }
    }
    se = block_sum(se, shd);
    py = block_sum(py, shd);
    plp = block_sum(plp, shd);
    const double lse = log(se); // relative to mx
    if (threadIdx.x == 0) loss[blockIdx.x] = plp - py + lse; // sum p = 1
    const float lsef = (float)lse + mx;
    float4* d4 = reinterpret_cast<float4*>(dy + base);
    for (uint32_t i = threadIdx.x; i < n4; i += blockDim.x) {
        const float4 v = y4[i], q = p4[i];
        d4[i] = make_float4((__expf(v.x - lsef) - q.x) * scale, (__expf(v.y - lsef) - q.y) * scale,
                            (__expf(v.z - lsef) - q.z) * scale, (__expf(v.w - lsef) - q.w) * scale);
    }
}

// One block of 256 threads per tile of kHeadRows = 64 rows x H columns (H <= 256, a multiple of
// 64): thread t owns the 8 columns 8 (t mod H/8) .. and the rows t / (H/8) + k (256 / (H/8)), reading
// z3 and writing dz3 as 16-byte vectors (coalesced rows); the loads of eight rows are issued together.
// Column sums of dy h3 (dw4) and of dz3 (db3) are reduced in registers and shared memory, one
// atomic per column per block.
// Issue-bound (0.33 ms of traffic for 16 records of 131072 rows): packed pairs 0.61 -> 0.55 ms.
constexpr uint32_t kHeadRows = 64;
__global__ void __launch_bounds__(256) head_backward_kernel(const __nv_bfloat16* __restrict__ z3,
                                                            const float* __restrict__ dy, const float* __restrict__ w4,
                                                            uint32_t M, uint32_t H, __nv_bfloat16* __restrict__ dz3,
                                                            float* __restrict__ dw4, float* __restrict__ db3)
{
    // partial column sums of each row group r0 (rstep groups x H columns = 2048 values for every
    // H): written once per thread, summed in order by one thread per column (no atomics)
    __shared__ float pw[2048], pb[2048];
    const uint32_t t = threadIdx.x, groups = H / 8u, rstep = 256u / groups;
    const uint32_t g = t % groups, r0 = t / groups, c = 8u * g;
    const uint64_t m0 = (uint64_t)blockIdx.x * kHeadRows;
    uint64_t w[4], aw[4], ab[4]; // pairs of columns
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        w[q] = pk2(w4[c + 2 * q], w4[c + 2 * q + 1]);
        aw[q] = ab[q] = pk2(0.0f, 0.0f);
    }
    // H = 256: one pass of eight rows; smaller H: fewer rows per thread, a pass of the same kind
    for (uint32_t rb = r0; rb < kHeadRows; rb += 8u * rstep) {
        uint4 zz[8];
        float dd[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t r = rb + i * rstep;
            if (r < kHeadRows) {
                zz[i] = __ldg(reinterpret_cast<const uint4*>(z3 + (m0 + r) * H + c));
                dd[i] = __ldg(dy + m0 + r);
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t r = rb + i * rstep;
            if (r >= kHeadRows) break;
            const uint64_t d = pk2(dd[i], dd[i]);
            const uint32_t zw[4] = {zz[i].x, zz[i].y, zz[i].z, zz[i].w};
            uint32_t ow[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 z = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&zw[q]));
                const uint64_t zp = pk2(z.x, z.y);
                uint64_t sg, grad;
                silu_grad_pair(zp, sg, grad);
                const uint64_t g2 = mul2(mul2(d, w[q]), grad);
                aw[q] = fma2(d, mul2(zp, sg), aw[q]);
                ab[q] = add2(ab[q], g2);
                float g0, g1;
                upk2(g2, g0, g1);
                const __nv_bfloat162 p = __floats2bfloat162_rn(g0, g1);
                ow[q] = *reinterpret_cast<const uint32_t*>(&p);
            }
            *reinterpret_cast<uint4*>(dz3 + (m0 + r) * H + c) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        upk2(aw[q], pw[r0 * H + c + 2 * q], pw[r0 * H + c + 2 * q + 1]);
        upk2(ab[q], pb[r0 * H + c + 2 * q], pb[r0 * H + c + 2 * q + 1]);
    }
    __syncthreads();
    if (t < H) {
        float sw = 0.0f, sb = 0.0f;
        for (uint32_t k = 0; k < rstep; ++k) {
            sw += pw[k * H + t];
            sb += pb[k * H + t];
        }
        atomicAdd(&dw4[t], sw);
        atomicAdd(&db3[t], sb);
    }
}

__global__ void adam_kernel(AdamArgs a)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const float g = a.g[i];
    const float m = a.beta1 * a.m[i] + (1.0f - a.beta1) * g;
    const float v = a.beta2 * a.v[i] + (1.0f - a.beta2) * g * g;
    a.m[i] = m;
    a.v[i] = v;
    const float mh = m / a.bias1, vh = v / a.bias2;
    a.p[i] -= a.lr * (mh / (sqrtf(vh) + a.eps) + a.weight_decay * a.p[i]);
}

__global__ void weight_copies_kernel(WeightViews w)
{
    const uint32_t H = w.H, K0 = w.K0;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n1 = H * K0, n2 = H * H;
    if (i < n1) {
        w.w1b[i] = __float2bfloat16_rn(w.w1[i]);
    } else if (i < n1 + n2) {
        const uint32_t j = i - n1, r = j / H, c = j - r * H;
        const __nv_bfloat16 b = __float2bfloat16_rn(w.w2[j]);
        w.w2b[j] = b;
        w.w2t[c * H + r] = b;
    } else if (i < n1 + 2 * n2) {
        const uint32_t j = i - n1 - n2, r = j / H, c = j - r * H;
        const __nv_bfloat16 b = __float2bfloat16_rn(w.w3[j]);
        w.w3b[j] = b;
        w.w3t[c * H + r] = b;
    }
}

__global__ void scale_rows_kernel(const double* __restrict__ frac, const double* __restrict__ sums, uint32_t nt,
                                  uint32_t total, double* __restrict__ rows)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < total) rows[t] = sums[t / nt] * frac[t];
}

__global__ void cdf_cells_kernel(const double* __restrict__ phi, const double* __restrict__ theta, uint32_t ct,
                                 uint32_t cp, uint64_t total, float* __restrict__ p)
{
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const uint64_t cells = (uint64_t)ct * cp;
    const uint32_t r = (uint32_t)(t / cells);
    const uint32_t k = (uint32_t)(t - (uint64_t)r * cells);
    const uint32_t i = k / cp, j = k - i * cp;
    const double* a = phi + (uint64_t)r * (cp + 1);
    const double* T = theta + ((uint64_t)r * cp + j) * (ct + 1);
    p[t] = (float)((a[j + 1] - a[j]) * (T[i + 1] - T[i]));
}

unsigned blocks_of(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

} // namespace

int launch_features(const __nv_bfloat16* rec16, const __nv_bfloat16* cells, uint32_t records, uint32_t C, uint32_t K0,
                    uint32_t P, const double* recgeo, const double* cellgeo, __nv_bfloat16* X, cudaStream_t st)
{
    if (K0 % 64 || C % 128 || !records || P % 8 || P + 16 > K0) return -1;
    const uint32_t q_row = K0 / 8u;
    if ((uint64_t)records * C > 0xffffffffull) return -1;
    const uint64_t warps = (uint64_t)records * C / 16u * (q_row / 2u); // C is a multiple of 128, q_row of 8
    if (warps > 0xffffffffull) return -1;
    features_kernel<<<blocks_of(warps * 32u, 256), 256, 0, st>>>(reinterpret_cast<const uint4*>(rec16),
                                                                 reinterpret_cast<const uint4*>(cells), C, q_row,
                                                                 q_row - P / 8u, (uint32_t)warps, recgeo, cellgeo,
                                                                 reinterpret_cast<uint4*>(X));
    return (int)cudaGetLastError();
}

int launch_softmax_loss(const float* y, const float* p, uint32_t records, uint32_t C, float scale, float* dy,
                        double* loss, cudaStream_t st)
{
    if (C % 4 || !records) return -1;
    softmax_loss_kernel<<<records, 1024, 0, st>>>(y, p, C, scale, dy, loss);
    return (int)cudaGetLastError();
}

int launch_head_backward(const __nv_bfloat16* z3, const float* dy, const float* w4, uint32_t M, uint32_t H,
                         __nv_bfloat16* dz3, float* dw4, float* db3, cudaStream_t st)
{
    if (M % kHeadRows || H > 256 || H % 64) return -1;
    head_backward_kernel<<<M / kHeadRows, 256, 0, st>>>(z3, dy, w4, M, H, dz3, dw4, db3);
    return (int)cudaGetLastError();
}

int launch_adam(const AdamArgs& a, cudaStream_t st)
{
    adam_kernel<<<blocks_of(a.n, 256), 256, 0, st>>>(a);
    return (int)cudaGetLastError();
}

int launch_weight_copies(const WeightViews& w, cudaStream_t st)
{
    const uint64_t n = (uint64_t)w.H * w.K0 + 2ull * w.H * w.H;
    weight_copies_kernel<<<blocks_of(n, 256), 256, 0, st>>>(w);
    return (int)cudaGetLastError();
}

int launch_scale_rows(const double* frac, const double* sums, uint32_t records, uint32_t nt, double* rows,
                      cudaStream_t st)
{
    const uint32_t total = records * nt;
    scale_rows_kernel<<<blocks_of(total, 256), 256, 0, st>>>(frac, sums, nt, total, rows);
    return (int)cudaGetLastError();
}

int launch_cdf_cells(const double* phi, const double* theta, uint32_t records, uint32_t ct, uint32_t cp, float* p,
                     cudaStream_t st)
{
    const uint64_t total = (uint64_t)records * ct * cp;
    cdf_cells_kernel<<<blocks_of(total, 256), 256, 0, st>>>(phi, theta, ct, cp, total, p);
    return (int)cudaGetLastError();
}

} // namespace icp::mlp
