// icp_rainbow.cu -- Table-II rainbow diffraction on the query grid (sm_100a) and its C ABI
// (include/icp_b200.h, "Table-II rainbow diffraction").  Built with -fmad=false: every
// binary64 product and sum rounds on its own, and the explicit fma calls stay fused, as in
// the reference's host build of include/rainbow/rainbow_diffraction.hpp.
//
// The model (RainbowDiffraction, rainbow_diffraction.hpp:40-139): an edge between query
// rows r and r + 1 at one phi is a primary transition when the TRT family starts there and
// a secondary one when the TRRT family ends there, provided the total intensity jumps by
// the contrast; every direction within support x sigma of its nearest labelled edge is
// replaced by a solid-angle weighted spherical Gaussian of its neighbourhood (secondary
// sigma = 2 x primary), blended out between inner_blend and support sigmas.
//
// Kernels (one thread per query direction unless said otherwise):
//   rainbow_detect_kernel  edge labels; also packs each sample to (s, p) -- NaN when the
//                          sample is unavailable -- and marks the rows that carry a label.
//                          A thread walks kDetectRows rows of one column, so that each focal
//                          record is read once and not again as the row below.
//   rainbow_prepare_kernel the packing and row marks for caller-supplied labels.
//   Both also fill the table sin^2(m dphi / 2).
//   rainbow_filter_kernel  one block per kFilterThreads columns of one row.  The nearest-edge
//                          search keeps the labels of its window as bit masks in shared memory
//                          and takes, per labelled row and kind, the nearest column by bit scans
//                          (the angular distance along a row grows with it); the haversine terms
//                          that do not depend on phi are in shared memory too.  The Gaussian's
//                          weight of (row, sampled row, column offset) does not depend on the
//                          column, so a block evaluates the asin and exp once per table entry and
//                          its threads only multiply and add, in the reference's compensated
//                          sums.  Directions that no labelled edge reaches leave with their
//                          input, written coalesced.
// Device libm (sin, asin, acos, exp, sqrt) is CUDA's; its last-ulp differences from the
// host's are the only source of difference from the reference's host results.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstddef>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "../../include/icp_b200.h"
#include "icp_internal.h"

using namespace icp;

namespace {

thread_local char g_msg[512];

int fail(int status, const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_msg, sizeof g_msg, fmt, ap);
    va_end(ap);
    set_last_error(g_msg);
    return status;
}
int ok()
{
    set_last_error("");
    return ICP_OK;
}
#define ICP_CUDA(call)                                                                                  \
    do {                                                                                                \
        const cudaError_t e_ = (call);                                                                  \
        if (e_ != cudaSuccess) return fail(ICP_ERR_DEVICE, "%s failed: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

constexpr double kPi = 3.141592653589793238462643383279502884;
constexpr double kCapSlack = 0x1p-44; // closed-cap cutoff slack (rainbow_diffraction.hpp:14)
constexpr unsigned kThreads = 256;
constexpr uint32_t kMaxAxis = 32767u;

enum Counter { kPrimary, kSecondary, kUnknown, kFiltered, kUnavailable, kUnderresolved, kCounters };
constexpr uint32_t kUnavailableMask = ICP_DIFFRACTION_INPUT_UNAVAILABLE | ICP_DIFFRACTION_STENCIL_UNAVAILABLE |
                                      ICP_DIFFRACTION_DETECTION_UNAVAILABLE | ICP_DIFFRACTION_INVALID_DATA;

struct Grid {
    double sigma, support, contrast, inner;
    uint32_t nt, np;
    int reach; // rows within the search distance of a direction's row, rounded up
};

bool config_ok(uint32_t nt, uint32_t np, const icp_diffraction_config& c)
{
    auto fin = [](double x) { return x >= -DBL_MAX && x <= DBL_MAX; };
    return nt >= 2u && np >= 1u && nt <= kMaxAxis && np <= kMaxAxis && c.primary_sigma_rad > 0 &&
           fin(c.primary_sigma_rad) && c.support_sigma >= 2 && c.support_sigma <= 8 && c.inner_blend_sigma >= 0 &&
           c.inner_blend_sigma < c.support_sigma && 2 * c.primary_sigma_rad * c.support_sigma < kPi &&
           c.transition_contrast >= 0 && c.transition_contrast < 1;
}

__device__ __forceinline__ bool finite64(double x) { return x >= -DBL_MAX && x <= DBL_MAX; }
__device__ __forceinline__ double nan64() { return __longlong_as_double(0x7ff8000000000000ll); }

// (s, p) of a focal record, or NaN when the record is unavailable (flags, sign, finiteness).
// kWide: the grid starts on 16 bytes, and with it every pair (a record asks for 8 only; two loads cost the
// pass at 1800 x 3600 0.3 %).
template <bool kWide> __device__ __forceinline__ double2 load_sample(const icp_focal_sample* f, uint64_t i)
{
    double s, p;
    if constexpr (kWide) {
        const double2 sp = __ldg(reinterpret_cast<const double2*>(&f[i].intensity_s));
        s = sp.x;
        p = sp.y;
    } else {
        s = __ldg(&f[i].intensity_s);
        p = __ldg(&f[i].intensity_p);
    }
    const bool good = __ldg(&f[i].flags) == 0u && s >= 0 && p >= 0 && finite64(s + p);
    return good ? make_double2(s, p) : make_double2(nan64(), nan64());
}
static_assert(offsetof(icp_focal_sample, intensity_s) % 16 == 0 && sizeof(icp_focal_sample) % 16 == 0, "pairs follow the grid");
bool wide_pairs(const icp_focal_sample* f) { return reinterpret_cast<uintptr_t>(f) % 16u == 0; }
__device__ __forceinline__ bool available(double2 v) { return v.x == v.x; }

__device__ __forceinline__ void warp_count(uint32_t* counters, int which, bool pred)
{
    const unsigned mask = __ballot_sync(0xffffffffu, pred);
    if ((threadIdx.x & 31u) == 0 && mask) atomicAdd(&counters[which], (unsigned)__popc(mask));
}

// vv[m] = sin^2(m dphi / 2), m <= np / 2: the part of the haversine that varies along a row.
__device__ __forceinline__ void fill_vv(const Grid& g, uint64_t m, double* vv)
{
    if (m > g.np / 2u) return;
    const double v = sin(0.5 * (double(m) * (2 * kPi / double(g.np))));
    vv[m] = v * v;
}

// Bound by DRAM: the fields it needs touch nearly every 64-byte block of the 144-byte records (933 MB
// at 1800 x 3600, 0.17 ms; one thread per direction, reading each record twice: 0.21 ms).
// Rows a thread of the detect kernel walks: eight where that leaves eight blocks per SM, else
// fewer, so that small grids still cover the chip.
constexpr unsigned kDetectRows = 8;

template <bool kWide>
__global__ void __launch_bounds__(kThreads) rainbow_detect_kernel(const icp_focal_sample* __restrict__ f, Grid g,
                                                                  uint32_t rows,
                                                                  uint32_t* __restrict__ edges,
                                                                  double2* __restrict__ packed,
                                                                  uint32_t* __restrict__ row_marks,
                                                                  double* __restrict__ vv,
                                                                  uint32_t* __restrict__ counters)
{
    const uint32_t col = blockIdx.x * kThreads + threadIdx.x;
    const uint32_t r0 = blockIdx.y * rows, r1 = min(g.nt, r0 + rows);
    const bool in = col < g.np;
    if (blockIdx.y == 0 && in) fill_vv(g, col, vv);
    unsigned primary = 0, secondary = 0, unknown = 0; // of this warp
    double2 a = in ? load_sample<kWide>(f, uint64_t(r0) * g.np + col) : make_double2(0.0, 0.0);
    for (uint32_t base = r0; base < r1; base += 4u) {
        double2 below[4]; // the next four rows' samples, in flight together
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u) {
            const uint32_t r = base + u;
            below[u] = in && r < r1 && r + 1u < g.nt ? load_sample<kWide>(f, uint64_t(r + 1u) * g.np + col) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u) {
            const uint32_t r = base + u;
            if (r >= r1) break;
            uint32_t e = 0;
            if (in) {
                const uint64_t i = uint64_t(r) * g.np + col;
                packed[i] = a;
                if (r + 1u != g.nt) {
                    const double2 b = below[u];
                    if (!available(a) || !available(b))
                        e = ICP_TRANSITION_UNKNOWN;
                    else {
                        const double x = a.x + a.y, y = b.x + b.y, peak = fmax(x, y);
                        if (peak > 0 && finite64(peak) && !(fabs(y - x) / peak < g.contrast)) {
                            if (__ldg(&f[i].family_hits[2]) == 0u && __ldg(&f[i + g.np].family_hits[2]) > 0u &&
                                __ldg(&f[i + g.np].family_incoherent[2]) > 0)
                                e |= ICP_TRANSITION_PRIMARY;
                            if (__ldg(&f[i].family_hits[3]) > 0u && __ldg(&f[i + g.np].family_hits[3]) == 0u &&
                                __ldg(&f[i].family_incoherent[3]) > 0)
                                e |= ICP_TRANSITION_SECONDARY;
                        }
                    }
                    a = b;
                }
                edges[i] = e;
            }
            const unsigned any = __ballot_sync(0xffffffffu, e != 0u);
            if (any) {
                if ((threadIdx.x & 31u) == 0) row_marks[r] = 1u;
                primary += __popc(__ballot_sync(0xffffffffu, (e & ICP_TRANSITION_PRIMARY) != 0));
                secondary += __popc(__ballot_sync(0xffffffffu, (e & ICP_TRANSITION_SECONDARY) != 0));
                unknown += __popc(__ballot_sync(0xffffffffu, (e & ICP_TRANSITION_UNKNOWN) != 0));
            }
        }
    }
    if ((threadIdx.x & 31u) == 0) {
        if (primary) atomicAdd(&counters[kPrimary], primary);
        if (secondary) atomicAdd(&counters[kSecondary], secondary);
        if (unknown) atomicAdd(&counters[kUnknown], unknown);
    }
}

template <bool kWide>
__global__ void __launch_bounds__(kThreads) rainbow_prepare_kernel(const icp_focal_sample* __restrict__ f,
                                                                   const uint32_t* __restrict__ edges, Grid g,
                                                                   double2* __restrict__ packed,
                                                                   uint32_t* __restrict__ row_marks,
                                                                   double* __restrict__ vv)
{
    const uint64_t n = uint64_t(g.nt) * g.np, stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        packed[i] = load_sample<kWide>(f, i);
        fill_vv(g, i, vv);
        if (__ldg(&edges[i])) atomicOr(&row_marks[i / g.np], 1u);
    }
}

// Terms of the haversine distance between colatitude t and row colatitude tr
// (RainbowDiffraction::angular_distance): h = ss sin^2(phi / 2) + uu, only phi varies along a row.
struct RowTerms {
    double uu, ss; // sin((t - tr) / 2)^2, sin(t) sin(tr)
};
__device__ __forceinline__ RowTerms row_terms(double t, double st, double tr)
{
    const double u = sin(0.5 * (t - tr));
    return {u * u, st * sin(tr)};
}
__device__ __forceinline__ double haversine_distance(double h) { return 2 * asin(sqrt(fmin(1.0, fmax(0.0, h)))); }
// Half-width in columns of the cap's longitude window on row colatitude r, -1 when the row
// misses the cap, nc when the cap wraps it (RainbowDiffraction::phi_radius).
__device__ __forceinline__ int cap_window(double t, double st, double ct, double r, double radius, double cos_radius,
                                          double dp, int nc)
{
    if (fabs(t - r) > radius + kCapSlack) return -1;
    const double a = st * sin(r), b = ct * cos(r);
    if (!(a > 0)) return nc;
    const double x = (cos_radius - b) / a;
    if (x <= -1) return nc;
    if (x >= 1) return 1;
    const int w = int(ceil(acos(x) / dp)) + 1;
    return nc < w ? nc : w;
}

struct Compensated {
    double s = 0, c = 0;
    // Knuth's two-sum: the same exact error term as the reference's branch on the larger
    // magnitude, without the comparison and the selects
    __device__ __forceinline__ void add(double x)
    {
        const double n = s + x, y = n - s;
        c += (s - (n - y)) + (x - y);
        s = n;
    }
    __device__ __forceinline__ double value() const { return s + c; }
};

// Columns to the nearest set bit on either side of bit p (p < 32 n) of a row's label mask: on a
// full circle of nc columns (32 n >= nc) around it, else within the mask; -1 when there is none.
__device__ __forceinline__ int nearest_label(const uint32_t* mask, int n, int p, bool full, int nc)
{
    const int at = p >> 5, b = p & 31;
    int best = INT_MAX;
    uint32_t x = mask[at] & (0xffffffffu >> (31 - b));
    int k = at;
    while (!x && k > 0) x = mask[--k];
    if (x) best = p - (k * 32 + 31 - __clz(int(x)));
    else if (full) { // wraps: the row's last label
        k = n;
        while (!x && k > at) x = mask[--k];
        if (x) best = p + nc - (k * 32 + 31 - __clz(int(x)));
    }
    x = mask[at] & (0xffffffffu << b);
    k = at;
    while (!x && k + 1 < n) x = mask[++k];
    if (x) best = min(best, k * 32 + __ffs(int(x)) - 1 - p);
    else if (full) { // the row's first label
        k = -1;
        while (!x && k < at) x = mask[++k];
        if (x) best = min(best, k * 32 + __ffs(int(x)) - 1 + nc - p);
    }
    return best == INT_MAX ? -1 : best;
}

constexpr unsigned kFilterThreads = 256;
constexpr int kTileRows = 32;    // sampled rows whose windows are evaluated together
constexpr int kTableSize = 2048; // weights of one tile: several rows, or a part of one wide row
constexpr int kMaskWords = 2 * kTableSize; // the label masks use the table's memory before it is filled
static_assert(kMaskWords >= 3 * ((int(kMaxAxis) + 31) / 32), "the masks of one full row fit");

// What bounds it: FP64 issue in the band (about a dozen additions and multiplications per tap of
// the two compensated sums; 0.18 ms of FP64 pipe time at 1800 x 3600, r = 0.5 mm), the result stores
// elsewhere.  Measured there on one B200: 3.86 ms with asin and exp evaluated per tap and every edge
// of the search window visited; 0.48 ms now, the whole pass 4.2 -> 0.68 ms.  256 columns per block
// share a row's table and masks (128: 0.60 ms); four blocks per SM at 64 registers with small
// spills beat two at 126 (0.56 ms) and three at 80 (0.53 ms).
__global__ void __launch_bounds__(kFilterThreads, 4) rainbow_filter_kernel(const double2* __restrict__ packed,
                                                                        const uint32_t* __restrict__ edges,
                                                                        const uint32_t* __restrict__ row_marks,
                                                                        const double* __restrict__ vv, Grid g,
                                                                        icp_diffraction_result* __restrict__ results,
                                                                        double* __restrict__ density,
                                                                        uint32_t* __restrict__ counters)
{
    __shared__ double s_uu[kFilterThreads], s_ss[kFilterThreads];
    __shared__ int s_row[kFilterThreads], s_half[kFilterThreads];
    __shared__ uint32_t s_kinds[kFilterThreads];
    __shared__ double s_table[kTableSize];
    __shared__ double s_area[kTileRows];
    __shared__ int s_width[kTileRows];
    __shared__ unsigned s_count[kFilterThreads / 32];
    static_assert(kTableSize * sizeof(double) >= kFilterThreads * sizeof(icp_diffraction_result), "result staging");
    const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
    const int nr = int(g.nt), nc = int(g.np), row = int(blockIdx.y), col0 = int(blockIdx.x * kFilterThreads),
              col = col0 + tid;
    const double dt = kPi / double(nr), dp = 2 * kPi / double(nc), t = (row + 0.5) * dt;
    const double support = g.support, search = 2 * g.sigma * support;
    // rows that an edge within the search distance can have, and a few more: the windows below decide
    const int lo = max(0, row - g.reach), hi = min(nr - 2, row + g.reach);
    uint32_t marked = 0;
    for (int rr = lo + tid; rr <= hi; rr += int(kFilterThreads)) marked |= row_marks[rr];

    icp_diffraction_result out{};
    const bool in = col < nc;
    const double2 center = in ? packed[uint64_t(row) * g.np + uint32_t(col)] : make_double2(0.0, 0.0);
    out.intensity_s = center.x;
    out.intensity_p = center.y;
    const bool usable = in && available(center);
    if (in && !usable) {
        out.flags = ICP_DIFFRACTION_INPUT_UNAVAILABLE;
        out.intensity_s = out.intensity_p = nan64();
    }

    if (__syncthreads_or(marked)) {
        // Nearest labelled edge within twice the primary support, in units of its own sigma: per
        // row and kind the nearest column is the nearest edge.
        const double st = sin(t), ct = cos(t), cos_search = cos(search);
        double near_h[3] = {4.0, 4.0, 4.0}; // smallest haversine of each kind (a real one is <= 1)
        for (int base = lo; base <= hi; base += int(kFilterThreads)) {
            const int rr = base + tid;
            const double tr = (rr + 1.0) * dt;
            int half = -1; // columns on each side of the direction, nc for the whole circle
            if (rr <= hi && row_marks[rr]) half = cap_window(t, st, ct, tr, search, cos_search, dp, nc);
            const bool keep = half >= 0;
            const unsigned vote = __ballot_sync(0xffffffffu, keep);
            __syncthreads(); // the previous tile's rows are no longer read
            if (lane == 0) s_count[warp] = unsigned(__popc(vote));
            __syncthreads();
            int at = __popc(vote & ((1u << lane) - 1u)), count = 0;
            for (int w = 0; w < int(kFilterThreads / 32); ++w) {
                if (w < warp) at += int(s_count[w]);
                count += int(s_count[w]);
            }
            if (keep) {
                const RowTerms r = row_terms(t, st, tr);
                s_uu[at] = r.uu;
                s_ss[at] = r.ss;
                s_row[at] = rr;
                // the mask covers the block's columns and the window on both sides
                s_half[at] = 2 * half + int(kFilterThreads) >= nc ? nc : half;
            }
            __syncthreads();
            uint32_t* masks = reinterpret_cast<uint32_t*>(s_table); // [row][kind][words]
            for (int k0 = 0; k0 < count;) {
                int rows = 0, words = 1;
                for (; k0 + rows < count; ++rows) {
                    const int h = s_half[k0 + rows];
                    const int n = max(words, h == nc ? (nc + 31) / 32 : (2 * h + int(kFilterThreads) + 31) / 32);
                    if (rows && 3 * n * (rows + 1) > kMaskWords) break;
                    words = n;
                }
                if (tid < rows) s_kinds[tid] = 0u;
                __syncthreads();
                for (int q = warp; q < rows * words; q += int(kFilterThreads / 32)) {
                    const int k = q / words, h = s_half[k0 + k], bit = (q % words) * 32 + lane;
                    uint32_t e = 0;
                    if (h == nc) {
                        if (bit < nc) e = __ldg(&edges[uint64_t(s_row[k0 + k]) * g.np + uint32_t(bit)]);
                    } else if (bit < 2 * h + int(kFilterThreads)) {
                        int c = col0 - h + bit; // within one turn: 2 h + kFilterThreads < nc
                        c += c < 0 ? nc : (c >= nc ? -nc : 0);
                        e = __ldg(&edges[uint64_t(s_row[k0 + k]) * g.np + uint32_t(c)]);
                    }
#pragma unroll
                    for (int kind = 0; kind < 3; ++kind) {
                        const unsigned bits = __ballot_sync(0xffffffffu, (e >> kind) & 1u);
                        if (lane == 0) {
                            masks[(k * 3 + kind) * words + q % words] = bits;
                            if (bits) atomicOr(&s_kinds[k], 1u << kind);
                        }
                    }
                }
                __syncthreads();
                if (usable)
                    for (int k = 0; k < rows; ++k) {
                        const int h = s_half[k0 + k];
                        const double uu = s_uu[k0 + k], ss = s_ss[k0 + k];
                        const uint32_t kinds = s_kinds[k];
#pragma unroll
                        for (int kind = 0; kind < 3; ++kind) {
                            if (!((kinds >> kind) & 1u)) continue;
                            const int m = nearest_label(masks + (k * 3 + kind) * words, words, h == nc ? col : tid + h,
                                                        h == nc, nc);
                            if (m >= 0) near_h[kind] = fmin(near_h[kind], fma(ss, __ldg(&vv[min(m, nc / 2)]), uu));
                        }
                    }
                __syncthreads();
                k0 += rows;
            }
        }
        uint32_t need = 0;
        double best = support + 1;
        if (usable) {
            if (near_h[2] <= 3.0 && !(haversine_distance(near_h[2]) > search + kCapSlack)) {
                out.flags |= ICP_DIFFRACTION_DETECTION_UNAVAILABLE;
                out.intensity_s = out.intensity_p = nan64();
            }
            // a primary edge wins ties within 1e-12, as in the reference's edge order
#pragma unroll
            for (uint32_t kind = ICP_TRANSITION_PRIMARY; kind <= ICP_TRANSITION_SECONDARY; kind *= 2u) {
                if (near_h[kind - 1] > 3.0) continue;
                const double d = haversine_distance(near_h[kind - 1]);
                if (d > search + kCapSlack) continue;
                const double sigma = g.sigma * (kind == ICP_TRANSITION_SECONDARY ? 2 : 1);
                const double distance = d / sigma;
                if (distance < support && distance < best - 1e-12) {
                    best = distance;
                    out.sigma_rad = sigma;
                    out.transition_kind = kind;
                }
            }
            // no kind: unchanged, no global blur
            if (out.transition_kind && !(out.flags & ICP_DIFFRACTION_DETECTION_UNAVAILABLE)) {
                need = out.transition_kind;
                const double sigma = out.sigma_rad;
                if (dt > 0.5 * sigma || st * dp > 0.5 * sigma) out.flags |= ICP_DIFFRACTION_UNDERRESOLVED;
                out.blend = 1;
                if (best > g.inner) {
                    const double x = (best - g.inner) / (support - g.inner);
                    out.blend = 1 - x * x * (3 - 2 * x);
                }
            }
        }

        const double half_dt = sin(0.5 * dt);
        for (uint32_t kind = ICP_TRANSITION_PRIMARY; kind <= ICP_TRANSITION_SECONDARY; kind *= 2u) {
            if (!__syncthreads_or(need == kind)) continue;
            const double sigma = g.sigma * (kind == ICP_TRANSITION_SECONDARY ? 2 : 1);
            const double radius = support * sigma, cos_radius = cos(radius);
            const int lower = max(0, int(floor((t - radius) / dt)) - 1);
            const int upper = min(nr - 1, int(ceil((t + radius) / dt)));
            Compensated sum_s, sum_p, weights; // weights: of the table entries this thread evaluates
            bool holes = false;
            for (int rr0 = lower; rr0 <= upper;) {
                __syncthreads(); // the previous tile's table is no longer read
                if (tid < kTileRows) {
                    int width = -1; // columns on each side of the direction
                    if (rr0 + tid <= upper) {
                        const double tr = (rr0 + tid + 0.5) * dt;
                        const int w = cap_window(t, st, ct, tr, radius, cos_radius, dp, nc);
                        if (w >= 0) {
                            const RowTerms r = row_terms(t, st, tr);
                            s_uu[tid] = r.uu;
                            s_ss[tid] = r.ss;
                            s_area[tid] = 2 * sin(tr) * half_dt * dp;
                            width = 2 * w + 1 >= nc ? nc / 2 : w;
                            // down to the last column inside the cap (the window has one or two to spare)
                            while (width >= 0 &&
                                   haversine_distance(fma(r.ss, __ldg(&vv[width]), r.uu)) > radius + kCapSlack)
                                --width;
                        }
                    }
                    s_width[tid] = width;
                }
                __syncthreads();
                int rows = 0, wide = 1; // rows of this tile and its widest window
                for (; rows < kTileRows && rr0 + rows <= upper; ++rows) {
                    const int w = max(wide, s_width[rows] + 1);
                    if (rows && w * (rows + 1) > kTableSize) break;
                    wide = w;
                }
                const int part = min(wide, kTableSize);
                for (int m0 = 0; m0 < wide; m0 += part) {
                    if (m0) __syncthreads();
                    for (int q = tid; q < rows * part; q += int(kFilterThreads)) {
                        const int k = q / part, m = m0 + q % part;
                        if (m > s_width[k]) continue;
                        const double d = haversine_distance(fma(s_ss[k], __ldg(&vv[m]), s_uu[k]));
                        const double weight = exp(-0.5 * (d / sigma) * (d / sigma)) * s_area[k];
                        s_table[q] = weight;
                        // both sides of the direction, once at its own and at the opposite column
                        weights.add(m == 0 || 2 * m == nc ? weight : 2 * weight);
                    }
                    __syncthreads();
                    if (need != kind) continue;
                    auto tap = [&](double weight, double2 q) {
                        // packed marks an unavailable sample by this NaN; the sums are not used then
                        holes |= __double2hiint(q.x) == 0x7ff80000;
                        sum_s.add(weight * q.x);
                        sum_p.add(weight * q.y);
                    };
                    const bool inner = col0 >= wide && col0 + int(kFilterThreads) + wide <= nc; // no seam
                    for (int k = 0; k < rows; ++k) {
                        const int m1 = min(s_width[k], m0 + part - 1), mb = max(m0, 1);
                        const double* table = s_table + k * part - m0;
                        const double2* sample_row = packed + uint64_t(rr0 + k) * g.np;
                        if (inner) {
                            const double2* here = sample_row + col;
#pragma unroll 4
                            for (int m = m1; m >= mb; --m) tap(table[m], __ldg(&here[-m]));
#pragma unroll 4
                            for (int m = m0; m <= m1; ++m) tap(table[m], __ldg(&here[m]));
                        } else {
                            for (int m = 2 * m1 == nc ? m1 - 1 : m1; m >= mb; --m)
                                tap(table[m], __ldg(&sample_row[col >= m ? col - m : col - m + nc]));
                            for (int m = m0; m <= m1; ++m)
                                tap(table[m], __ldg(&sample_row[col + m < nc ? col + m : col + m - nc]));
                        }
                    }
                }
                rr0 += rows;
            }
            // the weight total is the row's: the threads' partial sums added by one of them
            __syncthreads();
            s_uu[tid] = weights.s;
            s_ss[tid] = weights.c;
            __syncthreads();
            if (tid == 0) {
                Compensated total;
                for (unsigned k = 0; k < kFilterThreads; ++k) {
                    total.add(s_uu[k]);
                    total.c += s_ss[k];
                }
                s_area[0] = total.value();
            }
            __syncthreads();
            if (need != kind) continue;
            const double total = s_area[0];
            if (holes) { // no hole filling: an unavailable neighbour makes the direction unavailable
                out.flags |= ICP_DIFFRACTION_STENCIL_UNAVAILABLE;
                out.intensity_s = out.intensity_p = nan64();
            } else if (!(total > 0) || !finite64(total)) {
                out.flags |= ICP_DIFFRACTION_INVALID_DATA;
                out.intensity_s = out.intensity_p = nan64();
            } else {
                // Constant-preserving local normalisation, blended toward the unfiltered value.
                out.intensity_s = fma(out.blend, sum_s.value() / total - center.x, center.x);
                out.intensity_p = fma(out.blend, sum_p.value() / total - center.y, center.y);
                if (!(out.intensity_s >= 0 && out.intensity_p >= 0) || !finite64(out.intensity_s + out.intensity_p)) {
                    out.flags |= ICP_DIFFRACTION_INVALID_DATA;
                    out.intensity_s = out.intensity_p = nan64();
                } else
                    out.flags |= ICP_DIFFRACTION_FILTERED;
            }
        }
    }

    warp_count(counters, kFiltered, in && (out.flags & ICP_DIFFRACTION_FILTERED) != 0);
    warp_count(counters, kUnavailable, in && (out.flags & kUnavailableMask) != 0u);
    warp_count(counters, kUnderresolved, in && (out.flags & ICP_DIFFRACTION_UNDERRESOLVED) != 0);
    if (in && density) density[uint64_t(row) * g.np + uint32_t(col)] = out.intensity_s + out.intensity_p;
    // the 40-byte results through shared memory, so that the stores are contiguous
    __syncthreads();
    reinterpret_cast<icp_diffraction_result*>(s_table)[tid] = out;
    __syncthreads();
    const int words = min(int(kFilterThreads), nc - col0) * int(sizeof(icp_diffraction_result) / 8);
    uint64_t* dst = reinterpret_cast<uint64_t*>(results + uint64_t(row) * g.np + uint32_t(col0));
    for (int q = tid; q < words; q += int(kFilterThreads)) dst[q] = reinterpret_cast<const uint64_t*>(s_table)[q];
}

// Scratch of one call: packed samples (16 B per direction), the sin^2 table, row marks, counters.
struct Buffers {
    double2* packed;
    double* vv;
    uint32_t* rows;
    uint32_t* counters;
};

int prepare(icp_context* ctx, const icp_focal_sample* d_focal, uint32_t nt, uint32_t np,
            const icp_diffraction_config* config, Grid& g, Buffers& b)
{
    if (!ctx || !d_focal || !config) return fail(ICP_ERR_INVALID_ARGUMENT, "icp_rainbow: null argument");
    if (!config_ok(nt, np, *config)) return fail(ICP_ERR_INVALID_ARGUMENT, "Invalid diffraction/grid configuration.");
    g = {config->primary_sigma_rad, config->support_sigma, config->transition_contrast, config->inner_blend_sigma, nt, np,
         int(std::ceil(2 * config->primary_sigma_rad * config->support_sigma / (kPi / nt))) + 2};
    const uint64_t n = uint64_t(nt) * np;
    const size_t packed = n * sizeof(double2), vv = (size_t(np) / 2 + 1) * sizeof(double),
                 rows = (size_t(nt) + 1) & ~size_t(1);
    ICP_CUDA(cudaSetDevice(ctx->device));
    ICP_CUDA(ctx->rainbow.ensure(packed + vv + (rows + kCounters + 2) * sizeof(uint32_t)));
    char* base = static_cast<char*>(ctx->rainbow.ptr);
    b.packed = reinterpret_cast<double2*>(base);
    b.vv = reinterpret_cast<double*>(base + packed);
    b.rows = reinterpret_cast<uint32_t*>(base + packed + vv);
    b.counters = b.rows + rows;
    ICP_CUDA(cudaMemsetAsync(b.rows, 0, (rows + kCounters) * sizeof(uint32_t), ctx->stream));
    return ICP_OK;
}

int launch_detect(icp_context* ctx, const icp_focal_sample* f, const Grid& g, const Buffers& b, uint32_t* edges)
{
    const uint32_t across = (g.np + kThreads - 1) / kThreads, sms = uint32_t(ctx->sms > 0 ? ctx->sms : 148);
    const uint32_t rows = std::max(1u, std::min(kDetectRows, uint32_t(uint64_t(across) * g.nt / (8u * sms))));
    const dim3 grid(across, (g.nt + rows - 1) / rows);
    const auto kernel = wide_pairs(f) ? rainbow_detect_kernel<true> : rainbow_detect_kernel<false>;
    kernel<<<grid, kThreads, 0, ctx->stream>>>(f, g, rows, edges, b.packed, b.rows, b.vv, b.counters);
    ICP_CUDA(cudaGetLastError());
    count_launch();
    return ICP_OK;
}

int launch_filter(icp_context* ctx, const uint32_t* edges, const Grid& g, const Buffers& b,
                  icp_diffraction_result* results, double* density)
{
    const dim3 grid((g.np + kFilterThreads - 1) / kFilterThreads, g.nt);
    rainbow_filter_kernel<<<grid, kFilterThreads, 0, ctx->stream>>>(b.packed, edges, b.rows, b.vv, g, results,
                                                                    density, b.counters);
    ICP_CUDA(cudaGetLastError());
    count_launch();
    return ICP_OK;
}

int finish(icp_context* ctx, const Buffers& b, icp_diffraction_stats* stats)
{
    if (stats) {
        uint32_t c[kCounters];
        ICP_CUDA(cudaMemcpyAsync(c, b.counters, sizeof c, cudaMemcpyDeviceToHost, ctx->stream));
        ICP_CUDA(cudaStreamSynchronize(ctx->stream));
        *stats = {c[kPrimary], c[kSecondary], c[kUnknown], c[kFiltered], c[kUnavailable], c[kUnderresolved]};
    } else
        ICP_CUDA(cudaStreamSynchronize(ctx->stream));
    return ok();
}

} // namespace

extern "C" {

int icp_rainbow_table_sigma(float radius_mm, double* primary_sigma_deg)
{
    // Sadeghi et al. (2012) Table II: primary-bow width (degrees) at radii 0.1 .. 1.0 mm,
    // linear between the tabulated radii, no extrapolation.
    static const float radii[10] = {0.1f, 0.2f, 0.3f, 0.4f, 0.5f, 0.6f, 0.7f, 0.8f, 0.9f, 1.0f};
    static const double widths[10] = {0.70, 0.45, 0.30, 0.25, 0.22, 0.20, 0.18, 0.17, 0.16, 0.15};
    if (!primary_sigma_deg) return fail(ICP_ERR_INVALID_ARGUMENT, "icp_rainbow_table_sigma: null argument");
    if (!(radius_mm >= radii[0] && radius_mm <= radii[9]))
        return fail(ICP_ERR_INVALID_ARGUMENT, "Table II covers radius 0.1..1.0 mm only.");
    for (unsigned j = 0; j < 10; ++j) {
        if (radius_mm == radii[j]) {
            *primary_sigma_deg = widths[j];
            return ok();
        }
        if (j > 0 && radius_mm < radii[j]) {
            const double f = (double(radius_mm) - radii[j - 1]) / (double(radii[j]) - radii[j - 1]);
            *primary_sigma_deg = std::fma(f, widths[j] - widths[j - 1], widths[j - 1]);
            return ok();
        }
    }
    return fail(ICP_ERR_INVALID_ARGUMENT, "Table II covers radius 0.1..1.0 mm only.");
}

int icp_rainbow_detect(icp_context* ctx, const icp_focal_sample* d_focal, uint32_t nt, uint32_t np,
                       const icp_diffraction_config* config, uint32_t* d_transitions)
{
    if (!d_transitions) return fail(ICP_ERR_INVALID_ARGUMENT, "icp_rainbow_detect: null argument");
    Grid g;
    Buffers b;
    if (const int st = prepare(ctx, d_focal, nt, np, config, g, b)) return st;
    if (const int st = launch_detect(ctx, d_focal, g, b, d_transitions)) return st;
    return finish(ctx, b, nullptr);
}

int icp_rainbow_filter(icp_context* ctx, const icp_focal_sample* d_focal, const uint32_t* d_transitions, uint32_t nt,
                       uint32_t np, const icp_diffraction_config* config, icp_diffraction_result* d_results,
                       double* d_density, icp_diffraction_stats* stats)
{
    if (!d_transitions || !d_results) return fail(ICP_ERR_INVALID_ARGUMENT, "icp_rainbow_filter: null argument");
    Grid g;
    Buffers b;
    if (const int st = prepare(ctx, d_focal, nt, np, config, g, b)) return st;
    const uint64_t need = (uint64_t(nt) * np + kThreads - 1) / kThreads;
    const unsigned blocks = unsigned(std::min<uint64_t>(need, uint64_t(ctx->sms > 0 ? ctx->sms : 148) * 8u));
    const auto kernel = wide_pairs(d_focal) ? rainbow_prepare_kernel<true> : rainbow_prepare_kernel<false>;
    kernel<<<blocks, kThreads, 0, ctx->stream>>>(d_focal, d_transitions, g, b.packed, b.rows, b.vv);
    ICP_CUDA(cudaGetLastError());
    count_launch();
    if (const int st = launch_filter(ctx, d_transitions, g, b, d_results, d_density)) return st;
    return finish(ctx, b, stats);
}

int icp_rainbow_diffraction(icp_context* ctx, const icp_focal_sample* d_focal, uint32_t nt, uint32_t np,
                            const icp_diffraction_config* config, uint32_t* d_transitions,
                            icp_diffraction_result* d_results, double* d_density, icp_diffraction_stats* stats)
{
    if (!d_transitions || !d_results) return fail(ICP_ERR_INVALID_ARGUMENT, "icp_rainbow_diffraction: null argument");
    Grid g;
    Buffers b;
    if (const int st = prepare(ctx, d_focal, nt, np, config, g, b)) return st;
    if (const int st = launch_detect(ctx, d_focal, g, b, d_transitions)) return st;
    if (const int st = launch_filter(ctx, d_transitions, g, b, d_results, d_density)) return st;
    return finish(ctx, b, stats);
}

} // extern "C"
