// icp_hex_kernel.cuh -- fused single-particle trace + (u,phi) binning kernel (sm_100a), with
// two geometries: the hexagonal prism (HexGeo) and the axisymmetric drop (DropGeo).
//
// One launch traces one orientation node's ray range [first, first+count) and adds every
// exit into the FP64 cell-mass histogram.  It replaces the reference's count kernel, serial
// prefix, replay kernel, 200-byte CSR round trip and FP64 atomic accumulate
// (hex_trace/device/hex_trace.cu:12-48, hex_phase/device/phase_accumulate.cu:10-28):
//   * persistent warps, each owning a contiguous slice of ray ids; a lane whose ray ends
//     takes the next id of its warp's slice in the next step (no warp idles on long rays);
//   * one event per lane per step: the entry split, or one internal boundary + split; each
//     event emits at most one exit;
//   * prism exits go to a shared-memory table in 2^-44 fixed point, flushed to FP64 once per
//     block; drop exits straight to the FP64 histogram.
// Ray algorithm: hex_trace/include/ice_crystal/hex_trace_core.hpp:190-259 (linear R/T chain),
// hex_prism.hpp:64-175 (entry sampling, nearest exit plane), flux_interface.hpp:26-88.
#pragma once
#include <type_traits>
#include "icp_bin.cuh"
#include "icp_device.cuh"
#include "icp_drop.cuh"

namespace icp {

// Accumulators shared by all blocks of one launch (device memory, zeroed by the host).
// Power sums are exact 128-bit fixed-point integers (lo, hi words) in units of 2^-44.
struct DevStats {
    unsigned long long esc[2], unres[2], fwd[2], bwd[2];
    double axial;
    unsigned long long max_bal_bits, max_iface_bits; // bit patterns of non-negative doubles
    unsigned long long rays, outputs, status[8], rejected, snapped, near_edge, fallback, invalid;
    unsigned long long encounters, missed, gauge_evals;
};

__device__ __forceinline__ void add128(unsigned long long* p, unsigned long long t)
{
    if (!t) return;
    const unsigned long long old = atomicAdd(p, t);
    if (old + t < old) atomicAdd(p + 1, 1ull);
}

// Hexagonal prism in units of its circumradius, body frame (long axis +y).
template <class R> struct HexGeo {
    R half_len;
    R cum[8];           // cumulative projected face weights (plain adds in face order)
    uint32_t face_mask; // faces with positive projected weight
    R area;             // total projected weight (Kahan sum, as the reference's projected_area)
};
// Axisymmetric drop in units of its equal-volume radius; rays start on a disk of radius
// `disk` around the axis through the centre, a distance `back` before the centre.
template <class R> struct DropGeo {
    DropShape<R> shape;
    R disk, back;
    V3<R> e1;           // second transverse axis (k x ke0)
};

template <class R, class G> struct TraceParams {
    G geo;
    V3<R> k, ke0;    // incident direction and its frame vector
    R tail, bal_tol;
    unsigned long long tail_fx; // floor(tail * 2^44): the tail test of the fixed-point path
    Media<R> enter, leave; // n_ext -> n_int at entry, n_int -> n_ext inside
    uint64_t seed, total, first, count;
    uint32_t max_hits;
    uint32_t batch_size;
    uint32_t* batch_out;   // per-batch exit counters or nullptr
    // binning
    BinGridF gf;
    BinGridD gd;
    const double* edges_d; // nt+1 (global)
    const float* edges_f;  // nt+1 (global)
    double* mass;          // nt*np FP64 histogram (global)
    double to_mass;        // area weight * 2^-44
    DevStats* stats;
    uint32_t hash_slots;   // power of two, 0 = no shared table
    uint32_t smem_edges;   // 1 = stage edges in shared memory
};

// Normal of face f by selects (a switch diverges by face).
template <class R> __device__ __forceinline__ V3<R> face_normal(unsigned f)
{
    const R h = R(0.5), s = R(kSqrt3 / 2);
    const unsigned k = f >= 3u ? f - 3u : f; // axis of a side face; f < 3 points along it
    const R x = k == 0u ? R(1) : (k == 1u ? h : -h), z = k == 0u ? R(0) : s;
    const bool side = f < 6u, neg = f >= 3u;
    return v3(side ? (neg ? -x : x) : R(0), side ? R(0) : (f == 6u ? R(1) : R(-1)), side && k ? (neg ? -z : z) : R(0));
}
// The same by cases: the binary32 entry point's products contract around these constants, and the
// entry points keep their bits this way.
__device__ __forceinline__ V3<float> entry_normal(unsigned f)
{
    const float h = 0.5f, s = float(kSqrt3 / 2);
    switch (f) {
    case 0: return v3(1.f, 0.f, 0.f);
    case 1: return v3(h, 0.f, s);
    case 2: return v3(-h, 0.f, s);
    case 3: return v3(-1.f, 0.f, 0.f);
    case 4: return v3(-h, 0.f, -s);
    case 5: return v3(h, 0.f, -s);
    case 6: return v3(0.f, 1.f, 0.f);
    default: return v3(0.f, -1.f, 0.f);
    }
}
template <class R> __device__ __forceinline__ V3<R> hex_vertex(unsigned f)
{
    const R s = R(kSqrt3 / 2);
    switch (f % 6u) {
    case 0: return v3(s, R(0), R(0.5));
    case 1: return v3(R(0), R(0), R(1));
    case 2: return v3(-s, R(0), R(0.5));
    case 3: return v3(-s, R(0), R(-0.5));
    case 4: return v3(R(0), R(0), R(-1));
    default: return v3(s, R(0), R(-0.5));
    }
}
template <class R> __device__ __forceinline__ R face_offset(const HexGeo<R>& P, unsigned f)
{
    return f < 6u ? R(kSqrt3 / 2) : P.half_len;
}

// Products of v with the prism's four face axes (faces 0, 1, 2 and 6; the opposite faces have the
// exact negatives).  Equal to the dot products with the normals: a zero component adds nothing, and
// in binary32 the last product is fused into the sum (h v.x is exact).
template <class R> struct Axes {
    R a[4];
};
template <class R> __device__ __forceinline__ Axes<R> prism_axes(V3<R> v)
{
    const R h = R(0.5), s = R(kSqrt3 / 2);
    if constexpr (sizeof(R) == 4) return {{v.x, fmaf(s, v.z, h * v.x), fmaf(s, v.z, -h * v.x), v.y}};
    else return {{v.x, h * v.x + s * v.z, -h * v.x + s * v.z, v.y}};
}
template <class R> __device__ __forceinline__ R axis_of(const Axes<R>& A, unsigned f) // product with face f's normal
{
    const unsigned k = f < 6u ? (f >= 3u ? f - 3u : f) : 3u;
    const R x = k == 0u ? A.a[0] : (k == 1u ? A.a[1] : (k == 2u ? A.a[2] : A.a[3]));
    return f == 7u || (f >= 3u && f < 6u) ? -x : x;
}

// hex_prism.hpp:54-57 / 108-120 (FP64 path only): every other face strictly outside tolerance.
__device__ __forceinline__ bool strict_face_point(const HexGeo<double>& P, V3<double> p, unsigned face)
{
    const double tol = 128 * Eps<double>::eps * fmax(1.0, fmax(P.half_len, fmax(fabs(p.x), fmax(fabs(p.y), fabs(p.z)))));
    const Axes<double> A = prism_axes(p);
    unsigned inside = 1u << face; // faces that p is inside of by more than the tolerance
#pragma unroll
    for (unsigned k = 0; k < 4; ++k) {
        const double off = k < 3 ? kSqrt3 / 2 : P.half_len;
        inside |= off - A.a[k] > tol ? 1u << (k < 3 ? k : 6u) : 0u;
        inside |= off + A.a[k] > tol ? 1u << (k < 3 ? k + 3u : 7u) : 0u;
    }
    const double gap = face_offset(P, face) - axis_of(A, face);
    return inside == 0xffu && fabs(gap) <= tol;
}

struct Boundary {
    unsigned face;
    int status; // 0 regular, 3 ambiguous, 5 numerical
    bool near_edge;
};

// Nearest exit plane of the convex prism from a point on `start` (hex_prism.hpp:123-147).
// FP32: exit t = min over forward-facing planes (no positivity filter, so a point rounded
// just outside a neighbouring plane exits there at t = 0); near ties are counted only.
// FP64 (below): the reference rules, ties within geometry tolerance are ambiguous.
// Of each pair of opposite faces one at most faces forward: four quotients instead of eight; on
// equal distances the lower face number wins, as it does in face order.
__device__ __forceinline__ Boundary next_boundary(const HexGeo<float>& P, V3<float>& p, V3<float> d, unsigned start,
                                                  float& t_out)
{
    Boundary out{8u, 0, false};
    const Axes<float> D = prism_axes(d), A = prism_axes(p);
    float best = 3.0e38f, second = 3.0e38f;
#pragma unroll
    for (unsigned k = 0; k < 4; ++k) {
        const bool fwd = D.a[k] > 0.f;
        const unsigned f = k < 3 ? (fwd ? k : k + 3u) : (fwd ? 6u : 7u);
        const float off = k < 3 ? float(kSqrt3 / 2) : P.half_len;
        const float q = (off - (fwd ? A.a[k] : -A.a[k])) / rabs(D.a[k]);
        const float t = D.a[k] != 0.f && f != start ? q : 3.0e38f;
        const bool less = t < best || (t == best && f < out.face);
        second = less ? best : (t < second ? t : second);
        out.face = t < 3.0e38f && less ? f : out.face;
        best = less ? t : best;
    }
    if (out.face == 8u) { out.status = 5; return out; }
    const float t = rmax(best, 0.f);
    p = p + d * t;
    out.near_edge = (second - best) <= 64.f * Eps<float>::eps * rmax(1.f, P.half_len);
    t_out = t;
    return out;
}

// Reciprocal to about 20 bits, for choosing between candidates only.
__device__ __forceinline__ double rcp_rough(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// FP64.  Of each pair of opposite faces one at most faces forward, so there are four candidates; a
// rough reciprocal finds the nearest, whose distance is then divided out exactly.  Only when the
// runner-up is within the rough quotients' error does every candidate get its exact distance (the
// reference's tie rule needs both).  The point itself was checked against `start` when it
// was reached (strict_face_point below and at the entry), so it is not checked again here.
// In two parts: the plane and the point on it (nearest_plane; status 5 without one), and whether they are
// certain (boundary_status).
__device__ __forceinline__ Boundary nearest_plane(const HexGeo<double>& P, V3<double>& p, V3<double> d, unsigned start,
                                                  double& best, double& second)
{
    Boundary out{8u, 0, false};
    const Axes<double> D = prism_axes(d), A = prism_axes(p);
    if (axis_of(D, start) > 128 * Eps<double>::eps) { out.status = 5; return out; }
    const double none = 1.7976931348623157e308;
    best = second = none;
    double gap = 0, slope = 1;
    double num[4];
    bool valid[4];
#pragma unroll
    for (unsigned k = 0; k < 4; ++k) {
        const bool fwd = D.a[k] > 0;
        const unsigned f = k < 3 ? (fwd ? k : k + 3u) : (fwd ? 6u : 7u);
        const double off = k < 3 ? kSqrt3 / 2 : P.half_len;
        num[k] = off - (fwd ? A.a[k] : -A.a[k]);
        valid[k] = D.a[k] != 0 && f != start && num[k] > 0;
        const double t = valid[k] ? num[k] * rcp_rough(fabs(D.a[k])) : none;
        const bool less = t < best;
        second = less ? best : (t < second ? t : second);
        best = less ? t : best;
        gap = less ? num[k] : gap;
        slope = less ? fabs(D.a[k]) : slope;
        out.face = less ? f : out.face;
    }
    const double span = fmax(1.0, P.half_len);
    if (!(second - best > 0x1p-16 * (best + second) + 0x1p-30 * span) || !(best < 0x1p900)) {
        best = second = none;
        out.face = 8u;
#pragma unroll 1
        for (unsigned f = 0; f < 8; ++f) { // in face order, as the reference
            const unsigned k = f < 6u ? f % 3u : 3u;
            const bool fwd = f < 3u || f == 6u;
            if (f == start) continue;
            const double ck = k == 0u ? D.a[0] : (k == 1u ? D.a[1] : (k == 2u ? D.a[2] : D.a[3]));
            const double ak = k == 0u ? A.a[0] : (k == 1u ? A.a[1] : (k == 2u ? A.a[2] : A.a[3]));
            const double c = fwd ? ck : -ck;
            if (!(c > 0)) continue;
            const double t = ((k < 3u ? kSqrt3 / 2 : P.half_len) - (fwd ? ak : -ak)) / c;
            if (!(t > 0) || !finite_r(t)) continue;
            if (t < best) { second = best; best = t; out.face = f; }
            else if (t < second) second = t;
        }
        if (out.face == 8u) { out.status = 5; return out; }
    } else {
        best = quot(gap, div_by(slope));
        second = none; // further than the tolerance below
    }
    p = p + d * best;
    return out;
}
__device__ __forceinline__ int boundary_status(const HexGeo<double>& P, V3<double> p, unsigned face, double best, double second)
{
    const double tol = 128 * Eps<double>::eps * fmax(1.0, fmax(P.half_len, fmax(fmax(fabs(p.x), fmax(fabs(p.y), fabs(p.z))), fabs(best))));
    return second - best <= tol || !strict_face_point(P, p, face) ? 3 : 0;
}
__device__ __forceinline__ Boundary next_boundary(const HexGeo<double>& P, V3<double>& p, V3<double> d, unsigned start,
                                                  double& t_out)
{
    double second;
    Boundary out = nearest_plane(P, p, d, start, t_out, second);
    if (!out.status) out.status = boundary_status(P, p, out.face, t_out, second);
    return out;
}

// Entry of a fresh ray: point on the particle and the outward normal there.
// Returns 0, ICP_RAY_AMBIGUOUS (3), or -1 when the sampled ray misses the particle.
template <class R>
__device__ __forceinline__ int geo_entry(const HexGeo<R>& G, uint64_t seed, uint64_t id, V3<R>& pos, V3<R>& n,
                                         unsigned& face)
{
    // face in proportion to projected area, point on the face (hex_prism.hpp:64-98)
    const R u0 = uniform<R>(rng_bits(seed, id, 0));
    const R u1 = uniform<R>(rng_bits(seed, id, 1));
    const R u2 = uniform<R>(rng_bits(seed, id, 2));
    const R target = u0 * G.area;
    unsigned f8 = 8u, last = 8u;
#pragma unroll
    for (unsigned f = 0; f < 8; ++f) {
        if ((G.face_mask >> f) & 1u) {
            last = f;
            if (f8 == 8u && target < G.cum[f]) f8 = f;
        }
    }
    if (f8 == 8u) f8 = last;
    face = f8;
    if constexpr (sizeof(R) == 4) n = entry_normal(f8);
    else n = face_normal<R>(f8);
    if (f8 < 6u) {
        const V3<R> tangent = v3(-n.z, R(0), n.x);
        pos = (n * R(kSqrt3 / 2) + tangent * (u1 - R(0.5))) + v3(R(0), (R(2) * u2 - R(1)) * G.half_len, R(0));
    } else {
        const R sector = R(6) * u1;
        const unsigned j = (unsigned)sector;
        const R r = sqrt_r(sector - (R)j);
        pos = (hex_vertex<R>(j) * (R(1) - u2) + hex_vertex<R>(j + 1u) * u2) * r;
        pos.y = (f8 == 6u ? R(1) : R(-1)) * G.half_len;
    }
    if constexpr (sizeof(R) == 8) {
        if (!strict_face_point(G, pos, f8)) return 3;
    }
    return 0;
}
// Next exit point of an interior ray: advances p, returns 0 / 3 / 5 and the outward normal.
template <class R>
__device__ __forceinline__ int geo_next(const HexGeo<R>& G, V3<R>& p, V3<R> d, unsigned& face, V3<R>& n, bool& near_edge)
{
    R t;
    const Boundary hit = next_boundary(G, p, d, face, t);
    near_edge = hit.near_edge;
    if (hit.status) return hit.status;
    face = hit.face;
    n = face_normal<R>(hit.face);
    return 0;
}

// Drop: uniform point on the sampling disk (radius^2 uniform, angle uniform) a distance `back`
// before the centre; the reference's drops use a deterministic vertex grid instead
// (raindrop_paths.hpp:52-58), so the counter RNG of the prism path is reused here.
template <class R>
__device__ __forceinline__ V3<R> drop_origin(const DropGeo<R>& G, const V3<R>& k, const V3<R>& e0, uint64_t seed,
                                             uint64_t id)
{
    const R u0 = uniform<R>(rng_bits(seed, id, 0));
    const R u1 = uniform<R>(rng_bits(seed, id, 1));
    const R rad = G.disk * sqrt_r(u0);
    R sn, cs;
    if constexpr (sizeof(R) == 4) sincospif(R(2) * u1, &sn, &cs);
    else sincospi(R(2) * u1, &sn, &cs);
    return (e0 * (rad * cs) + G.e1 * (rad * sn)) - k * G.back;
}

template <class R> struct LaneRay {
    V3<R> p, d, e;
    Stokes<R> S;
    uint64_t id;
    R esc;                       // binary64 path: escaped power of this ray
    unsigned long long pfx, escfx; // binary32 path: power of the continuing branch and escaped
                                   // power, exact integers in units of 2^-44 of one ray
    uint32_t face, hits;
    bool live;
};

// Per-lane accumulators of what changes every step or every ray, summed per warp when a block (or
// a batch chunk) ends.  The power sums are exact 64-bit fixed-point integers; the counts are
// 32-bit: a
// lane traces at most lane_rays_max(max_hits) rays between flushes (the launchers cut launches
// and chunks to that), so that none of them can wrap.
template <class R> struct LaneAcc {
    unsigned long long esc_fx, unres_fx, fwd_fx, bwd_fx;
    uint32_t outputs, fallback, encounters, gauge_evals, snapped, near_edge;
    double axial;
    R max_iface;
    uint64_t cur_batch;
    uint32_t cur_batch_out;
};

// Per-warp tally in shared memory of what changes once per ray or more rarely (the rays per
// status, misses, rejections, invalid exits, the largest energy residual and, for the drop, the
// unresolved and pole powers), added with shared atomics.  Kept out of the lanes' registers, which
// the FP32 kernels need for the ray state at 64 registers; without them the drop kernel's spills
// halve and its DRAM traffic falls from 130 MB to 17 MB per 1e8-ray launch.  The warp's ray count
// is the status counts plus the misses; its power sums stay below 2^60 (lane_rays_max).  The
// prism keeps snapped exits, near-edge hits and the power sums per lane: its symmetric directions
// make them frequent (forward exits through parallel faces), and contended 64-bit shared atomics
// cost it 7 %.
struct Tally {
    unsigned status[8];
    unsigned missed, rejected, invalid, pad;
    unsigned long long unres_fx, fwd_fx, bwd_fx, max_bal_bits;
};
constexpr uint32_t kTallyWarps = 8; // blocks of 64..256 threads
constexpr size_t kTallyBytes = 80;
// whether a trace's power sums go to the tally (the drop) or stay per lane (the prism)
template <class P_> __host__ __device__ constexpr bool power_in_tally()
{
    return !std::is_same_v<std::remove_cv_t<decltype(P_::geo)>, HexGeo<std::remove_cv_t<decltype(P_::tail)>>>;
}
static_assert(sizeof(Tally) == kTallyBytes, "tally layout");
// Byte offset of the tallies in the trace kernel's shared memory (after the histogram table's
// values and keys, 16-byte aligned); the u edges follow the kTallyWarps tallies.
__host__ __device__ constexpr size_t trace_tally_offset(uint32_t hash_slots)
{
    return ((size_t)hash_slots * 12u + 15u) / 16u * 16u;
}

template <class R, class P_>
__device__ __forceinline__ void finish_ray(const P_& P, LaneRay<R>& L, LaneAcc<R>& A, Tally* T, int status,
                                           unsigned long long residual_fx, R residual)
{
    L.live = false;
    double bal;
    if constexpr (sizeof(R) == 4) {
        // escaped + residual is one ray's power exactly unless a branch was lost
        constexpr unsigned long long one = 1ull << kFixBits;
        const unsigned long long total = L.escfx + residual_fx;
        bal = (total >= one ? (double)(total - one) : (double)(one - total)) * kFixUnit;
    } else {
        bal = fabs((double)L.esc + (double)residual - 1.0);
    }
    if constexpr (power_in_tally<P_>()) {
        if (residual_fx) atomicAdd(&T->unres_fx, residual_fx);
    } else {
        A.unres_fx += residual_fx;
    }
    if (bal > 0.0) atomicMax(&T->max_bal_bits, (unsigned long long)__double_as_longlong(bal));
    atomicAdd(&T->status[status], 1u);
    const bool ok = (status == 0 || status == 1) && bal <= P.bal_tol;
    if (!ok) atomicAdd(&T->rejected, 1u);
}

// Ends the ray if the continuing branch is exhausted / below the tail / out of encounters
// (the top-of-loop and after-loop tests of hex_trace_core.hpp:217-251, applied eagerly).
template <class R, class P_>
__device__ __forceinline__ void settle(const P_& P, LaneRay<R>& L, LaneAcc<R>& A, Tally* T)
{
    if constexpr (sizeof(R) == 4) {
        const unsigned long long p = L.pfx;
        if (p == 0ull) finish_ray<R>(P, L, A, T, 0, 0ull, R(0));
        else if (p <= P.tail_fx) finish_ray<R>(P, L, A, T, 1, p, R(0));
        else if (L.hits >= P.max_hits) finish_ray<R>(P, L, A, T, 2, p, R(0));
    } else {
        // (one place that ends rays: 5 % of the prism's time)
        const R power = L.S.I;
        const int status = power == R(0) ? 0 : power <= P.tail ? 1 : L.hits >= P.max_hits ? 2 : -1;
        if (status >= 0) finish_ray<R>(P, L, A, T, status, to_fix(power), power);
    }
}

// Per-block shared state: the privatised histogram table, this warp's tally and (optionally) the
// u edges.
template <class R> struct BlockShared {
    SmemHist H;
    Tally* T;
    const R* edges;
};

template <class R, class P_>
__device__ __forceinline__ BlockShared<R> block_setup(const P_& P, unsigned char* smem)
{
    BlockShared<R> B;
    unsigned long long* s_vals = reinterpret_cast<unsigned long long*>(smem);
    uint32_t* s_keys = reinterpret_cast<uint32_t*>(s_vals + P.hash_slots);
    Tally* tallies = reinterpret_cast<Tally*>(smem + trace_tally_offset(P.hash_slots));
    B.T = tallies + (threadIdx.x >> 5);
    R* s_edges = reinterpret_cast<R*>(tallies + kTallyWarps);
    const uint32_t nt = P.gf.nt;
    for (uint32_t s = threadIdx.x; s < P.hash_slots; s += blockDim.x) { s_keys[s] = 0u; s_vals[s] = 0ull; }
    for (uint32_t i = threadIdx.x; i < kTallyWarps * kTallyBytes / 4; i += blockDim.x)
        reinterpret_cast<unsigned*>(tallies)[i] = 0u;
    if (P.smem_edges) {
        for (uint32_t i = threadIdx.x; i <= nt; i += blockDim.x) {
            if constexpr (sizeof(R) == 4) s_edges[i] = P.edges_f[i];
            else s_edges[i] = P.edges_d[i];
        }
        B.edges = s_edges;
    } else {
        if constexpr (sizeof(R) == 4) B.edges = P.edges_f;
        else B.edges = P.edges_d;
    }
    B.H = SmemHist{s_keys, s_vals, P.hash_slots ? P.hash_slots - 1u : 0u};
    return B;
}

template <class R> __device__ __forceinline__ void lane_acc_clear(LaneAcc<R>& A)
{
    A.esc_fx = A.unres_fx = A.fwd_fx = A.bwd_fx = 0ull;
    A.outputs = A.fallback = A.encounters = A.gauge_evals = A.snapped = A.near_edge = 0u;
    A.axial = 0.0;
    A.max_iface = R(0);
    A.cur_batch = ~0ull;
    A.cur_batch_out = 0u;
}

// Idle lanes at which a warp of the prism takes new rays: 1.6e7 rays over eight orientations, FP32,
// 12.4 / 11.7 / 12.1 / 12.4 / 13.2 ms at 1 / 4 / 8 / 12 / 16.
constexpr int kRefill = 4;

// Whether idle lanes take their next rays in this step.  The prism waits for several: its entry
// is a divergent path of its own, which a step would otherwise run for two or three lanes; the
// drop enters through the code that its live lanes run anyway.
template <class R, class G> __device__ __forceinline__ bool refill_now(unsigned idle)
{
    if constexpr (std::is_same_v<G, HexGeo<R>>) return __popc(idle) >= kRefill;
    else return idle != 0u;
}

// The rays [wnext, wend) of one warp: persistent lanes, one event per lane per step, every
// exit binned where it is made (hex_trace_core.hpp:190-259 per ray).
template <class R, class G, class P_>
__device__ __forceinline__ void trace_slice(const P_& P, const BlockShared<R>& B, uint64_t wnext, const uint64_t wend,
                                            LaneAcc<R>& A)
{
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    Tally* T = B.T;
    LaneRay<R> L;
    L.live = false;
    while (true) {
        // ---- refill idle lanes from the warp's slice
        const unsigned idle = __ballot_sync(kFull, !L.live);
        bool fresh = false;
        if (refill_now<R, G>(idle)) {
            if (!L.live) {
                const uint64_t id = wnext + __popc(idle & lt_mask);
                if (id < wend) { L.id = id; fresh = true; }
            }
            wnext += __popc(idle);
        }
        if (!__any_sync(kFull, L.live || fresh)) break;

        bool has = false;
        V3<R> od;
        R opow = R(0);
        unsigned long long efx = 0ull; // fixed-point power of this step's exit
        // ---- gather the inputs of this step's interface: the entry face of a fresh ray,
        // or the next exit plane of a live one (one shared split per lane per step)
        bool do_split = false;
        V3<R> sd, se, sn;
        Stokes<R> sS;
        const Media<R>* media = &P.enter;
        if constexpr (!std::is_same_v<G, HexGeo<R>>) {
            // drop: every active lane runs one intersection -- entering from its sampling-disk
            // origin (fresh) or leaving from its current surface point (live)
            V3<R> q, w, n;
            if (fresh) {
                q = drop_origin(P.geo, P.k, P.ke0, P.seed, L.id);
                w = P.k;
            } else {
                q = L.p;
                w = L.d;
            }
            bool hit = false;
            if (fresh || L.live) {
                R t;
                hit = drop_intersect(P.geo.shape, q, w, fresh, t, A.gauge_evals);
                q = q + w * t;
                if (hit) n = drop_normal(P.geo.shape, q);
            }
            if (fresh) {
                if (!hit) {
                    // a sampled ray that misses the particle carries no incident power
                    atomicAdd(&T->missed, 1u);
                } else {
                    L.live = true;
                    L.esc = R(0);
                    L.pfx = 1ull << kFixBits;
                    L.escfx = 0ull;
                    L.hits = 0u;
                    L.p = q;
                    L.face = 0u;
                    do_split = true;
                    sd = P.k;
                    se = P.ke0;
                    sS = Stokes<R>{R(1), R(0), R(0), R(0)};
                    sn = n;
                    media = &P.enter;
                }
            } else if (L.live) {
                // one internal encounter (hex_trace_core.hpp:217-246)
                L.p = q;
                ++L.hits;
                ++A.encounters;
                do_split = true;
                sd = L.d;
                se = L.e;
                sS = L.S;
                sn = -n;
                media = &P.leave;
            }
        } else if (fresh) {
            V3<R> pos, n;
            unsigned face = 8u;
            const int es = geo_entry(P.geo, P.seed, L.id, pos, n, face);
            if (es < 0) {
                // a sampled ray that misses the particle carries no incident power
                atomicAdd(&T->missed, 1u);
            } else {
                L.live = true;
                L.esc = R(0);
                L.pfx = 1ull << kFixBits;
                L.escfx = 0ull;
                L.hits = 0u;
                L.p = pos;
                L.face = face;
                do_split = true;
                if (es) {
                    finish_ray<R>(P, L, A, T, es, 1ull << kFixBits, R(1));
                    do_split = false;
                }
                sd = P.k;
                se = P.ke0;
                sS = Stokes<R>{R(1), R(0), R(0), R(0)};
                sn = n;
                media = &P.enter;
            }
        } else if (L.live) {
            // one internal encounter (hex_trace_core.hpp:217-246)
            V3<R> n;
            bool near_edge = false;
            const int hs = geo_next(P.geo, L.p, L.d, L.face, n, near_edge);
            if (hs) {
                finish_ray<R>(P, L, A, T, hs, sizeof(R) == 4 ? L.pfx : to_fix(L.S.I), L.S.I);
            } else {
                A.near_edge += near_edge ? 1u : 0u;
                ++L.hits;
                ++A.encounters;
                do_split = true;
                sd = L.d;
                se = L.e;
                sS = L.S;
                sn = -n;
                media = &P.leave;
            }
        }
        if (do_split) {
            const Interface<R> sp = split(sd, se, sS, sn, *media);
            A.max_iface = rmax(A.max_iface, sp.balance);
            // entry: exterior reflection exits, transmission continues;
            // internal: transmission exits, reflection continues
            unsigned long long cont_fx = 0ull;
            if constexpr (sizeof(R) == 4) {
                // the reflected share is rounded once, the transmitted share is the exact rest
                const unsigned long long rq = to_fix(sp.r.I);
                const unsigned long long rfx = (sp.tir || rq > L.pfx) ? L.pfx : rq;
                const unsigned long long tfx = L.pfx - rfx;
                efx = fresh ? rfx : tfx;
                cont_fx = fresh ? tfx : rfx;
                if (efx) {
                    has = true;
                    od = fresh ? sp.dr : sp.dt;
                    opow = (R)efx * R(kFixUnit);
                    L.escfx += efx;
                }
            } else {
                const R epow = fresh ? sp.r.I : (sp.has_t ? sp.t.I : R(0));
                if (epow > R(0)) {
                    has = true;
                    od = fresh ? sp.dr : sp.dt;
                    opow = epow;
                    efx = to_fix(epow);
                    L.esc += opow;
                }
            }
            if (sizeof(R) == 4 && fresh && !sp.has_t) { // binary64: settle ends it, its power is 0
                finish_ray<R>(P, L, A, T, 0, 0ull, R(0));
            } else {
                L.d = fresh ? sp.dt : sp.dr;
                L.e = sp.s;
                L.S = fresh ? sp.t : sp.r;
                if constexpr (sizeof(R) == 4) {
                    L.pfx = cont_fx;
                    L.S.I = (R)cont_fx * R(kFixUnit);
                }
                settle<R>(P, L, A, T);
            }
        }

        // ---- bin this step's exits
        if (has) {
            BinResult b;
            if constexpr (sizeof(R) == 4) b = bin_f32(P.gf, B.edges, od);
            else b = bin_f64(P.gd, B.edges, od);
            if (!b.valid) {
                atomicAdd(&T->invalid, 1u);
            } else {
                const uint64_t v = efx;
                A.esc_fx += v;
                A.outputs += 1;
                A.snapped += b.snapped ? 1u : 0u;
                A.axial += (double)opow * b.mu;
                if (b.pole > 0) {
                    if constexpr (power_in_tally<P_>()) atomicAdd(&T->fwd_fx, (unsigned long long)v);
                    else A.fwd_fx += v;
                } else if (b.pole < 0) {
                    if constexpr (power_in_tally<P_>()) atomicAdd(&T->bwd_fx, (unsigned long long)v);
                    else A.bwd_fx += v;
                } else {
                    hist_add(B.H, P.mass, P.to_mass, b.cell, v, A.fallback);
                }
            }
        }

        // ---- per-batch exit counts (the prism's capacity audit), flushed when the lane's batch
        // changes
        if constexpr (std::is_same_v<G, HexGeo<R>>) {
            if (P.batch_out && (has || fresh)) {
                const uint64_t bidx = L.id / P.batch_size;
                if (bidx != A.cur_batch) {
                    if (A.cur_batch != ~0ull && A.cur_batch_out) atomicAdd(&P.batch_out[A.cur_batch], A.cur_batch_out);
                    A.cur_batch = bidx;
                    A.cur_batch_out = 0u;
                }
                A.cur_batch_out += has ? 1u : 0u;
            }
        }
    }
    if constexpr (std::is_same_v<G, HexGeo<R>>)
        if (P.batch_out && A.cur_batch != ~0ull && A.cur_batch_out) atomicAdd(&P.batch_out[A.cur_batch], A.cur_batch_out);
}

// The warp's sums into the record's statistics: its lanes' accumulators (shuffled) and its tally
// (lane 0 adds, then clears the tally).  Called by whole warps after the lanes' last update.
template <class R>
__device__ __forceinline__ void warp_stats_flush(DevStats* Gs, const LaneAcc<R>& A, Tally* T)
{
    unsigned long long w[10] = {A.esc_fx, A.outputs, A.fallback, A.encounters, A.gauge_evals, A.snapped, A.near_edge,
                                A.unres_fx, A.fwd_fx, A.bwd_fx};
#pragma unroll
    for (int q = 0; q < 10; ++q)
        for (int o = 16; o; o >>= 1) w[q] += __shfl_xor_sync(kFull, w[q], o);
    double ax = A.axial, mi = (double)A.max_iface;
    for (int o = 16; o; o >>= 1) {
        ax += __shfl_xor_sync(kFull, ax, o);
        mi = fmax(mi, __shfl_xor_sync(kFull, mi, o));
    }
    __syncwarp();
    if ((threadIdx.x & 31u) == 0) {
        add128(Gs->esc, w[0]);
        // one of each pair is zero: the sums sit per lane (the prism) or in the tally (the drop)
        add128(Gs->unres, w[7] + T->unres_fx);
        add128(Gs->fwd, w[8] + T->fwd_fx);
        add128(Gs->bwd, w[9] + T->bwd_fx);
        unsigned long long rays = T->missed;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            rays += T->status[s];
            if (T->status[s]) atomicAdd(&Gs->status[s], (unsigned long long)T->status[s]);
        }
        const unsigned long long c[10] = {rays, w[1], T->rejected, w[5], w[6], w[2], T->invalid, w[3], T->missed, w[4]};
        unsigned long long* counters[10] = {&Gs->rays, &Gs->outputs, &Gs->rejected, &Gs->snapped, &Gs->near_edge,
                                            &Gs->fallback, &Gs->invalid, &Gs->encounters, &Gs->missed, &Gs->gauge_evals};
#pragma unroll
        for (int q = 0; q < 10; ++q)
            if (c[q]) atomicAdd(counters[q], c[q]);
        if (ax != 0.0) atomicAdd(&Gs->axial, ax);
        atomicMax(&Gs->max_bal_bits, T->max_bal_bits);
        atomicMax(&Gs->max_iface_bits, (unsigned long long)__double_as_longlong(mi));
        *T = Tally{};
    }
    __syncwarp();
}

// Block epilogue (all threads): flush the table into P.mass and every warp's sums into P.stats;
// leaves the table and the tallies cleared.
template <class R, class P_>
__device__ __forceinline__ void block_flush(const P_& P, const BlockShared<R>& B, const LaneAcc<R>& A)
{
    __syncthreads();
    hist_flush(B.H, P.mass, P.to_mass);
    warp_stats_flush<R>(P.stats, A, B.T);
}

// Block shape of the single-record trace: the FP32 drop runs 128-thread blocks, seven per SM at
// 72 registers (fewer spills than four 256-thread blocks at 64 registers: 1 % faster); the FP32
// prism keeps four 256-thread blocks (its 48 KB shared histogram table per block).  The FP64 kernels
// wait on chains of dependent operations: the prism runs two 256-thread blocks at 128 registers (1e6
// rays over two orientations 3.87 ms with one block at 162, 3.04 with two, 3.44 with three at 80 and
// their spills), the drop three 128-thread blocks at 162 registers (fewer registers lengthen the
// long chains that small records wait for).
template <class R, class G> struct TraceShape {
    static constexpr bool hex = std::is_same_v<G, HexGeo<R>>;
    static constexpr bool drop32 = sizeof(R) == 4 && !hex;
    static constexpr unsigned threads = drop32 ? 128u : 256u; // the largest block
    static constexpr unsigned min_blocks = sizeof(R) == 4 ? (drop32 ? 7u : 4u) : (hex ? 2u : 1u);
};

// One record: the ray range [first, first+count) split into contiguous per-warp slices.
template <class R, class G>
__global__ void __launch_bounds__(TraceShape<R, G>::threads, TraceShape<R, G>::min_blocks)
    trace_bin_kernel(const TraceParams<R, G> P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const BlockShared<R> B = block_setup<R>(P, smem);
    __syncthreads();
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    const uint64_t warp = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint64_t per = (P.count + warps - 1) / warps;
    const uint64_t wnext = P.first + warp * per;
    const uint64_t wend = min(P.first + P.count, wnext + per);
    LaneAcc<R> A;
    lane_acc_clear(A);
    trace_slice<R, G>(P, B, wnext, wend, A);
    block_flush<R>(P, B, A);
}

} // namespace icp
