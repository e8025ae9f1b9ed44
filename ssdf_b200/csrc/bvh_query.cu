// bvh_query.cu -- closest-triangle queries over the device BVH.
//
// Stands in for the reference's device query (serial/bvh/bvh.cu:60-76 + cuBQL CPAT) and its CPU
// grid samplers (serial/bvh/bvh.cpp:1574-1798). Three arithmetics (SSDF_PREC_*):
//   F64   the reference's exact double expression per triangle; lexicographic
//         (d^2, triangle index) minimum: bitwise the reference's double value;
//   F32   the same over float triangles with the reference's float expression (its
//         edf<float> value);
//   F32X  float traversal with fused multiply-adds keeps the K smallest float d^2 inside a
//         window (sqrt(best) + tau)^2; the window's members are re-evaluated in double and the
//         lexicographic minimum taken. tau bounds twice the float error of one distance, so the
//         double winner is always in the window; a query whose window overflowed the K slots is
//         walked again with the window fixed, re-evaluating every member in double (k_window, a
//         warp per query).
//         Result: bitwise the F64 result.
// Traversal: nearest child first, the farther one pushed with its box distance on a per-lane stack
// and culled on pop against the current thresholds. All three walk the same float tree of oriented boxes
// (DeviceMesh::obb), whose distances are lower bounds in every arithmetic: on the torus-knot 256^3 grid
// a 32-query packet visits 86 nodes and 59 triangles where it met 140 and 197 with axis-aligned boxes
// (16.6 -> 10.1 ms; plain double 31.1 -> 11.4 ms). Each lane answers kQ queries (a build option;
// 1 by default, 2 measured no faster: it shares each node and triangle load between two chains of
// arithmetic but costs the registers of the second). Grid queries map a
// warp to a 4 x 4 x 2kQ brick of nodes, so the warp's traversals stay coherent; by default a grid
// warp walks the tree as one packet.
// Outputs (SSDF_OUT_*): in/out distance (edf), in/out squared distance (sqedf), signed distance
// with the pseudo-normal rule of serial/bvh/bvh.cpp:1751-1792, closest point + triangle
// (closest_point_bvh, serial/bvh/bvh.cpp:178-194).
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>

#include "box_margin.h"
#include "device_geom.cuh"
#include "internal.h"

namespace ssdf_b200 {

namespace {

constexpr int kThreads = 128;
// F32X window slots: candidates kept per query in shared memory. A window that overflows them sends
// its query to the second stage (k_window). Torus-knot 256^3 grid: 11.1 ms with 8 slots, 10.8 with 10, 10.0 with
// 12, which overflow on 0.01 % of the queries. (16, with none there and a longer insertion, were slower on an
// earlier kernel and not measured again.)
#ifndef SSDF_B200_WINDOW_SLOTS
#define SSDF_B200_WINDOW_SLOTS 12
#endif
constexpr int kCand = SSDF_B200_WINDOW_SLOTS;

// Minimum resident blocks per SM the float query kernels are compiled for: 7 blocks of 128 (72
// registers). A node visit loads 128 bytes into registers, so the kernels want more of them than with
// 64-byte axis-aligned nodes (whose best was 10 blocks at 48). Torus-knot 256^3 grid, fix-up: 10.15 ms
// at 7, 10.33 at 8, 10.68 at 9, 11.47 at 10; 4M points on the beam lattice, float: 5.34 / 5.45 / 5.38 /
// 5.63 ms.
#ifndef SSDF_B200_QUERY_MIN_BLOCKS
#define SSDF_B200_QUERY_MIN_BLOCKS 7
#endif

// The double kernel keeps 5 resident blocks per SM (at most 102 registers), chosen when it walked double boxes and
// not measured again since.
constexpr int kF64MinBlocks = 5;

struct Counters {
    unsigned long long tri = 0, box = 0, fix = 0;
};

__device__ __forceinline__ double dinf() { return __longlong_as_double(0x7ff0000000000000ll); }
__device__ __forceinline__ float finf() { return __int_as_float(0x7f800000); }

// ---- query mapping ------------------------------------------------------------------------------

// Each lane answers kQ queries. Grid: a block covers an 8 (x) x 4 (y) column of nodes and, at step
// `step`, the 4 kQ z-planes from (column * grid_steps + step) * 4 kQ on; a warp takes a 4 x 4 x 2kQ
// brick of them, lane (lx, ly, lz) kQ consecutive z nodes. Point lists: query
// (block * kQ + s) * 128 + thread, so each of a lane's queries is a coalesced load.
__device__ __forceinline__ bool map_query(const QueryArgs &a, long long b, int step, int s, long long &q,
                                          long long &i, long long &j, long long &k) {
    if (!a.is_grid) {
        const long long slot = (b * kQ + s) * kThreads + threadIdx.x;
        if (slot >= a.npoints) return false;
        q = a.order ? (long long)__ldg(a.order + slot) : slot;
        return true;
    }
    // fewer than 2^31 blocks: 32-bit divisions
    const unsigned bxn = unsigned(grid_blocks_x(a.nx)), byn = unsigned(grid_blocks_y(a.ny));
    const unsigned r = unsigned(b) / bxn;
    const long long bx = unsigned(b) - r * bxn;
    const unsigned bz = r / byn;
    const long long by = r - bz * byn;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    i = bx * 8 + (warp & 1) * 4 + (lane & 3);
    j = by * 4 + ((lane >> 2) & 3);
    k = ((((long long)bz * a.grid_steps + step) * 4 + (warp >> 1) * 2) + (lane >> 4)) * kQ + s;
    q = i + a.nx * (j + a.ny * k);
    return i < a.nx && j < a.ny && k < a.nz;
}

__device__ __forceinline__ void grid_ijk(const QueryArgs &a, long long q, long long &i, long long &j, long long &k) {
    i = q % a.nx;
    const long long r = q / a.nx;
    j = r % a.ny;
    k = r / a.ny;
}

__device__ __forceinline__ void query_point(const QueryArgs &a, long long q, long long i, long long j, long long k,
                                            double &x, double &y, double &z) {
    if (a.is_grid) {
        if (a.coord_f64) {
            x = grid_coord<double>(a.lo64[0], a.h64[0], i);
            y = grid_coord<double>(a.lo64[1], a.h64[1], j);
            z = grid_coord<double>(a.lo64[2], a.h64[2], k + a.z0);
        } else {
            x = grid_coord<float>(a.lo32[0], a.h32[0], i);
            y = grid_coord<float>(a.lo32[1], a.h32[1], j);
            z = grid_coord<float>(a.lo32[2], a.h32[2], k + a.z0);
        }
    } else if (a.coord_f64) {
        x = __ldg((const double *)a.x + q);
        y = __ldg((const double *)a.y + q);
        z = __ldg((const double *)a.z + q);
    } else {
        x = double(__ldg((const float *)a.x + q));
        y = double(__ldg((const float *)a.y + q));
        z = double(__ldg((const float *)a.z + q));
    }
}

__device__ __forceinline__ double load_out(const QueryArgs &a, long long q) {
    return a.out_f64 ? ((const double *)a.out)[q] : double(((const float *)a.out)[q]);
}
__device__ __forceinline__ void store_out(const QueryArgs &a, long long q, double v) {
    if (a.out_f64)
        ((double *)a.out)[q] = v;
    else
        ((float *)a.out)[q] = float(v);
}

// ---- node and triangle loads ----------------------------------------------------------------------

struct Tri32 {
    float ax, ay, az, bx, by, bz, cx, cy, cz;
    int id;
};

// The fix-up filter's record of leaf position p (DeviceMesh::filt32, 3 x float4): the precomputed
// triangle (or proxy, the sign bit of its ab.ab set).
__device__ __forceinline__ FiltRec load_filt(const float4 *__restrict__ f, int p) {
    const float4 u = __ldg(f + 3 * p), v = __ldg(f + 3 * p + 1), w = __ldg(f + 3 * p + 2);
    const float pen = (__float_as_uint(u.w) >> 31) ? __int_as_float(0x7f800000) : 0.f;
    return FiltRec{u.x, u.y, u.z, v.x, v.y, v.z, w.x, w.y, w.z, fabsf(u.w), v.w, w.w, pen};
}
__device__ __forceinline__ Tri32 load_tri32(const float4 *__restrict__ t, int p) {
    const float4 u = __ldg(t + 3 * p), v = __ldg(t + 3 * p + 1), w = __ldg(t + 3 * p + 2);
    return Tri32{u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w, w.x, __float_as_int(w.y)};
}

struct Tri64 {
    double ax, ay, az, bx, by, bz, cx, cy, cz;
    int id;
};
__device__ __forceinline__ Tri64 load_tri64(const double2 *__restrict__ t, int p) {
    const double2 *r = t + 5 * p;
    const double2 u = __ldg(r), v = __ldg(r + 1), w = __ldg(r + 2), x = __ldg(r + 3), y = __ldg(r + 4);
    return Tri64{u.x, u.y, v.x, v.y, w.x, w.y, x.x, x.y, y.x, int(y.y)};
}

// ---- traversal policies ---------------------------------------------------------------------------
//
// A policy owns a lane's kQ queries (points, incumbents, prune thresholds `thr`) and knows how to
// test a node's child boxes and a leaf's triangles in its arithmetic. A node or leaf is wanted by a
// lane when any of its queries wants it (`want` returns the per-query mask); a pushed node keeps the
// smallest of its queries' box distances and is entered on pop while that is below the largest
// threshold (conservative for every query of the lane).

template <typename T>
struct ExactData;
template <>
struct ExactData<double> {
    using Tri = Tri64;
    // squared margin added to the prune threshold
    static __device__ __forceinline__ double margin(const DeviceMesh &m) {
        const double s = double(m.coord_scale) * 0x1p-40;
        return s * s;
    }
    // the float threshold of the boxes (in the box frame's scale), rounded up
    static __device__ __forceinline__ float box_thr(double best, double margin, const DeviceMesh &m) {
        const double t = (best * (1.0 + 1.0 / 65536.0) + margin) * (m.box_scale * m.box_scale);
        return fmaxf(__double2float_ru(t), FLT_MIN);  // a box at distance 0 is always wanted
    }
    static __device__ __forceinline__ float start_thr(double init, double margin, const DeviceMesh &m) {
        return box_thr(init, margin, m);
    }
    static __device__ __forceinline__ float box_coord(double p, int d, const DeviceMesh &m) {
        return float((p - double(m.box_c[d])) * m.box_scale);
    }
    // a coordinate from here on has no finite squared distance to the mesh (in a mesh within float's range)
    static __device__ __forceinline__ double beyond(const DeviceMesh &m) {
        return m.coord_scale < __int_as_float(0x7f800000) ? 0x1p520 : dinf();
    }
    // a threshold beyond float's range is +inf: a box distance that overflowed still counts as inside
    static __device__ __forceinline__ float box_key(float d) { return fminf(d, FLT_MAX); }
    static __device__ __forceinline__ Tri tri(const DeviceMesh &m, int pos) { return load_tri64(m.tris64, pos); }
};
template <>
struct ExactData<float> {
    using Tri = Tri32;
    // the prune threshold's margins (box_margin.h)
    static __device__ __forceinline__ float margin(const DeviceMesh &m) { return float_box_margin(m.coord_scale); }
    static __device__ __forceinline__ float box_thr(float best, float margin, const DeviceMesh &m) {
        return fmaxf(float_box_reach(best, margin) * m.box_scale_f * m.box_scale_f, FLT_MIN);
    }
    // the threshold a walk starts with, from an incoming bound that may be infinite
    static __device__ __forceinline__ float start_thr(float init, float margin, const DeviceMesh &m) {
        return init > FLT_MAX ? fmaxf(float_box_limit(margin, m.box_scale_f), FLT_MIN) : box_thr(init, margin, m);
    }
    static __device__ __forceinline__ float box_coord(float p, int d, const DeviceMesh &m) {
        return (p - m.box_c[d]) * m.box_scale_f;
    }
    // a coordinate from here on has no finite squared distance to the mesh
    static __device__ __forceinline__ float beyond(const DeviceMesh &) { return __int_as_float(0x7f800000); }
    static __device__ __forceinline__ float box_key(float d) { return d; }
    static __device__ __forceinline__ Tri tri(const DeviceMesh &m, int pos) { return load_tri32(m.tris32, pos); }
};

__device__ __forceinline__ float2 twice(float v) { return make_float2(v, v); }
// Box coordinate of a lane without a query: farther from every box than any query's.
constexpr float kNowhere = 0x1p62f;

// Lexicographic (d^2, id) minimum over all triangles, starting from (best, -1): a triangle replaces
// the incumbent if strictly closer, or equally close with a lower index (never the initial bound on
// a tie). The walk is float in either arithmetic: oriented boxes whose float distance is a lower bound
// of their triangles' are kept while it is below best * (1 + 2^-16) + margin, so neither rounding in box
// distances nor the conversion drops a tie. (Walking float boxes instead of double ones took the
// plain double kernel's nodes off its FP64 pipe, which was 52 % busy.) A point with a NaN or infinite
// coordinate has no finite distance to anything: it keeps its incoming bound without a walk.
template <typename T, int Q>
struct ExactPolicy {
    using R = float;
    static constexpr int kQn = Q;
    static constexpr bool kVote = sizeof(T) == sizeof(float), kRestarts = false;
    const DeviceMesh &m;
    T px[Q], py[Q], pz[Q], best[Q];
    float2 bx[Q], by[Q], bz[Q];  // the point in the box frame, each coordinate twice (two-wide FP32)
    float thr[Q];
    int bid[Q], bpos[Q];
    bool gone = false;  // the packet handed its queries to the second stage
    T margin;
    __device__ explicit ExactPolicy(const DeviceMesh &mesh) : m(mesh) { margin = ExactData<T>::margin(m); }
    __device__ __forceinline__ void set(int q, T x, T y, T z, T init) {
        px[q] = x, py[q] = y, pz[q] = z, best[q] = init, bid[q] = -1, bpos[q] = -1;
        bx[q] = twice(ExactData<T>::box_coord(x, 0, m));
        by[q] = twice(ExactData<T>::box_coord(y, 1, m));
        bz[q] = twice(ExactData<T>::box_coord(z, 2, m));
        const T lim = ExactData<T>::beyond(m);
        const bool finite = fabs(x) < lim && fabs(y) < lim && fabs(z) < lim;
        thr[q] = finite ? ExactData<T>::start_thr(init, margin, m) : -1.f;
    }
    __device__ __forceinline__ void disable(int q) {
        px[q] = py[q] = pz[q] = T(0), best[q] = T(0), bid[q] = -1, bpos[q] = -1;
        bx[q] = by[q] = bz[q] = twice(kNowhere);
        thr[q] = -1.f;
    }
    __device__ __forceinline__ void abandon() { gone = true; }
    // Starts query q from the triangle at leaf position pos, as if the walk had tested it first (it
    // replaces the incoming bound only when strictly closer; the walk meets it again without effect).
    __device__ __forceinline__ void seed(int q, int pos) {
        const auto t = ExactData<T>::tri(m, pos);
        const T d2 = tri_dist_sq_exact<T>(px[q], py[q], pz[q], t.ax, t.ay, t.az, t.bx, t.by, t.bz, t.cx, t.cy, t.cz);
        if (d2 < best[q]) {
            best[q] = d2;
            bid[q] = t.id;
            bpos[q] = pos;
            thr[q] = ExactData<T>::box_thr(best[q], margin, m);
        }
    }
    __device__ __forceinline__ void boxes(int node, float (&d0)[Q], float (&d1)[Q], int &r0, int &r1) const {
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const float2 d = obb_dist_sq_pair(bx[q], by[q], bz[q], m.obb + 8 * node, r0, r1);
            d0[q] = ExactData<T>::box_key(d.x);
            d1[q] = ExactData<T>::box_key(d.y);
        }
    }
    __device__ __forceinline__ float max_thr() const {
        float t = thr[0];
#pragma unroll
        for (int q = 1; q < Q; q++) t = t > thr[q] ? t : thr[q];
        return t;
    }
    template <bool COUNT>
    __device__ __forceinline__ void leaf(int first, int n, unsigned mask, Counters &cnt) {
        for (int k = 0; k < n; k++) {
            const auto t = ExactData<T>::tri(m, first + k);
#pragma unroll
            for (int q = 0; q < Q; q++) {
                if (!((mask >> q) & 1u)) continue;
                const T d2 = tri_dist_sq_exact<T>(px[q], py[q], pz[q], t.ax, t.ay, t.az, t.bx, t.by, t.bz, t.cx,
                                                  t.cy, t.cz);
                if (COUNT) cnt.tri++;
                if (d2 < best[q] || (d2 == best[q] && bid[q] >= 0 && t.id < bid[q])) {
                    best[q] = d2;
                    bid[q] = t.id;
                    bpos[q] = first + k;
                    thr[q] = ExactData<T>::box_thr(best[q], margin, m);
                }
            }
        }
    }
};

// F32X: float filter. Per query, the kCand smallest float d^2 inside the window
// (sqrt(best) + tau)^2 are kept, unordered, in shared memory (slot (q, s) of thread t at
// [(q * kCand + s) * kThreads + t]: consecutive threads, consecutive banks), with the smallest d^2
// pushed out of the slots. A candidate is appended to the used slots; only when they are full are
// the entries the shrinking window has left behind dropped (their d^2 is at or above the final
// window, so dropping them loses nothing), and if every slot is still inside the window the largest
// of the kCand + 1 is pushed out. The slots hold the same inside-the-window set as a sorted list
// would, for an append instead of a sorted insertion.
//
// The float filter's error is second order in its error along the triangle's plane, which stays
// small unless the triangle is ill-conditioned (a needle or a
// sliver: the face-region solve divides by its area). Such a triangle is filtered through a
// well-conditioned proxy that contains it (DeviceMesh::filt32): a lower bound of its distance,
// within the float filter's error, which may enter the window but, with its +inf penalty, never
// moves its centre; the member is re-evaluated in double like any other, so the double winner,
// whose key is at most its distance plus that error, stays inside the window.
__device__ __forceinline__ float window_thr(float best, float tau_rel, float scale) {
    if (!(best < finf())) return finf();
    const float d = sqrtf(best);
    const float w = d + tau_rel * (scale + d);
    return w * w * (1.0f + 1.0f / 65536.0f);
}

// A query coordinate as the filter and its boxes take it: less the mesh's middle, rounded once.
__device__ __forceinline__ float filter_coord(double p, int d, const DeviceMesh &m) {
    return float(p - double(m.box_c[d]));
}

template <int Q>
struct FastPolicy {
    using R = float;
    static constexpr int kQn = Q;
    static constexpr bool kVote = true, kRestarts = true;
    const DeviceMesh &m;
    float2 bx[Q], by[Q], bz[Q];  // the point in the box frame (the filter records' too), each coordinate twice
    float best[Q], thr[Q], evicted[Q];
    int used[Q];  // window slots in use
    float tau_rel;
    float *wd;
    int *wp;
    __device__ FastPolicy(const DeviceMesh &mesh, float tau, float *sd, int *sp)
        : m(mesh), tau_rel(tau), wd(sd + threadIdx.x), wp(sp + threadIdx.x) {}
    __device__ __forceinline__ int slot(int q, int s) const { return (q * kCand + s) * kThreads; }
    __device__ __forceinline__ void set(int q, float x, float y, float z, float init) {
        bx[q] = twice(x), by[q] = twice(y), bz[q] = twice(z), best[q] = init, evicted[q] = finf(), used[q] = 0;
        // a NaN or infinite coordinate: no finite distance, nothing to walk for
        const bool finite = isfinite(x) && isfinite(y) && isfinite(z);
        thr[q] = finite && !(init < 0.f) ? window_thr(init, tau_rel, m.coord_scale) : -1.f;  // no distance is below 0
    }
    __device__ __forceinline__ void disable(int q) {
        set(q, kNowhere, kNowhere, kNowhere, finf());
        thr[q] = -1.f;
    }
    // Starts query q's window from the key of the triangle at leaf position pos (not a proxy), as the
    // walk would on meeting it: best is then still the key of a tested triangle, and the walk inserts
    // the triangle when it meets it.
    __device__ __forceinline__ void seed(int q, int pos) {
        const FiltRec t = load_filt(m.filt32, pos);
        const float d2 = tri_dist_sq_filter(bx[q].x, by[q].x, bz[q].x, t);
        if (t.pen == 0.f && d2 < best[q]) {
            best[q] = d2;
            thr[q] = window_thr(best[q], tau_rel, m.coord_scale);
        }
    }
    // the walk starts over with the windows it has
    __device__ __forceinline__ void restart() {
#pragma unroll
        for (int q = 0; q < Q; q++) used[q] = 0, evicted[q] = finf();
    }
    // the walk stops early: every live query goes to the second stage with its current window
    __device__ __forceinline__ void abandon() {
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (thr[q] > 0.f) evicted[q] = 0.f;
    }
    __device__ __forceinline__ void boxes(int node, float (&d0)[Q], float (&d1)[Q], int &r0, int &r1) const {
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const float2 d = obb_dist_sq_pair(bx[q], by[q], bz[q], m.obb + 8 * node, r0, r1);
            d0[q] = d.x;
            d1[q] = d.y;
        }
    }
    __device__ __forceinline__ float max_thr() const {
        float t = thr[0];
#pragma unroll
        for (int q = 1; q < Q; q++) t = fmaxf(t, thr[q]);
        return t;
    }
    __device__ __forceinline__ void insert(int q, float d, int p) {
        if (used[q] < kCand) {
            wd[slot(q, used[q])] = d;
            wp[slot(q, used[q])] = p;
            used[q]++;
            return;
        }
        // full: keep the entries still inside the window, in place
        int w = 0, imax = 0;
        float vmax = -1.f;
        for (int s = 0; s < kCand; s++) {
            const float cur = wd[slot(q, s)];
            if (cur < thr[q]) {
                const int cp = wp[slot(q, s)];
                wd[slot(q, w)] = cur;
                wp[slot(q, w)] = cp;
                if (cur > vmax) vmax = cur, imax = w;
                w++;
            }
        }
        if (w < kCand) {
            wd[slot(q, w)] = d;
            wp[slot(q, w)] = p;
            used[q] = w + 1;
        } else if (d < vmax) {  // every slot inside the window: the largest of the kCand + 1 goes
            evicted[q] = fminf(evicted[q], vmax);
            wd[slot(q, imax)] = d;
            wp[slot(q, imax)] = p;
        } else {
            evicted[q] = fminf(evicted[q], d);
        }
    }
    template <bool COUNT>
    __device__ __forceinline__ void leaf(int first, int n, unsigned mask, Counters &cnt) {
        for (int k = 0; k < n; k++) {
            const FiltRec t = load_filt(m.filt32, first + k);
            const float pen = t.pen;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                if (!((mask >> q) & 1u)) continue;
                const float d2 = tri_dist_sq_filter(bx[q].x, by[q].x, bz[q].x, t);
                if (COUNT) cnt.tri++;
                if (d2 < thr[q]) {
                    insert(q, d2, first + k);
                    if (d2 + pen < best[q]) {
                        best[q] = d2;
                        thr[q] = window_thr(best[q], tau_rel, m.coord_scale);
                    }
                }
            }
        }
    }
};

template <class P, int Q = P::kQn>
__device__ __forceinline__ unsigned want_mask(const P &p, const typename P::R (&d)[Q]) {
    unsigned m = 0;
#pragma unroll
    for (int q = 0; q < Q; q++) m |= (d[q] < p.thr[q]) ? (1u << q) : 0u;
    return m;
}

template <typename R, int Q>
__device__ __forceinline__ R min_of(const R (&d)[Q]) {
    R v = d[0];
#pragma unroll
    for (int q = 1; q < Q; q++) v = d[q] < v ? d[q] : v;
    return v;
}

// Lanes that rank two children for their packet, of those that hold a query: a lane without one sits far
// outside, where the children's order says nothing (asked all the same, at (1, 1, 1) of the 4 x 4 x 2 brick, a
// 145^3 grid of the torus knot, whose last bricks have one column each, took 5,900 us against 2,900 for 144^3).
// All of them vote: 500,003 points near the knot 862 -> 829 us, the beams' points 5,280 -> 5,235, 64^3 grid on
// 5,120 triangles 226 -> 221. The double kernel follows one lane, (1, 1, 1) clamped to the brick's part inside
// the grid (of a list's last packet: its last lane); counting the votes cost it 2 % (1,167 -> 1,195).
template <class P>
__device__ __forceinline__ unsigned packet_rankers(unsigned active) {
    if (P::kVote) return active;
    int lane = 21;
    if (!(active & 0xeeeeeeeeu)) lane -= 1;   // one column of x
    if (!(active & 0xfff0fff0u)) lane -= 4;   // one row of y
    if (!(active & 0xffff0000u)) lane -= 16;  // one plane of z
    if (!((active >> lane) & 1u)) lane = 31 - __clz(int(active | 1u));
    return 1u << lane;
}

// Warp minimum / maximum of floats that order like their bits: distances (not negative) and thresholds (not
// negative, or -1). Through the intrinsics, which the compiler keeps where the whole warp is: the results
// feed divergent code, and an inline redux on floats could be sunk into it.
__device__ __forceinline__ float warp_min(float v) {
    return __int_as_float(__reduce_min_sync(0xffffffffu, __float_as_int(v)));
}
__device__ __forceinline__ float warp_max(float v) {
    return __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(v)));
}

// The next node of the packet's stack that some lane still wants (-1: none). An entry: node, key bits.
template <class P>
__device__ __forceinline__ int next_entry(const P &p, const int2 *const entry, int &sp) {
    const float tmax = warp_max(p.max_thr());
    while (sp > 0) {
        sp--;
        const int2 e = entry[sp];
        if (__int_as_float(e.y) < tmax) return e.x;
    }
    return -1;
}

// Packet walk (a grid warp as one packet): the node ids on the stack are the same in every lane, so
// the warp keeps one stack in shared memory instead of 32 copies in local memory. An entry keeps
// the smallest box distance over the warp's lanes and is entered on pop while that is below the
// largest lane threshold: a superset of "some lane's distance below its own threshold", so never a
// miss. Lanes without a query sit far from the mesh (P::disable), so they take no part in the keys.
// Of two wanted children the one the packet's lanes (packet_rankers) rank first is the nearer; a
// wanted leaf is tested at once, and when it was the nearer one the other child is asked for again, its lanes'
// thresholds having shrunk.
//
// Walks from `node` with sp nodes on the stack. Past its budget (checked where a path ends) the walk stops and returns
// how many nodes the stack still holds, else -1.
template <bool COUNT, class P>
__device__ __forceinline__ int traverse_packet(P &p, Counters &cnt, int budget, int2 *const entry, int node, int sp) {
    constexpr int Q = P::kQn;
    constexpr unsigned kAll = 0xffffffffu;
    int work = 0;  // triangle records the packet has tested (the same in every lane)
    if (budget <= 0) budget = 0x7fffffff;
    const unsigned rankers = packet_rankers<P>(__ballot_sync(kAll, p.max_thr() > 0.f));
    const int half = __popc(rankers) / 2;
    auto test_leaf = [&](int ref, unsigned m) {
        p.template leaf<COUNT>(leaf_first(ref), leaf_count(ref), m, cnt);
        work += leaf_count(ref);
    };
    while (true) {
        float d0[Q], d1[Q];
        int r0, r1;
        p.boxes(node, d0, d1, r0, r1);
        if (COUNT) cnt.box += 2 * Q;
        const unsigned m0 = want_mask(p, d0), m1 = r1 == kEmptyRef ? 0u : want_mask(p, d1);
        const bool any0 = __any_sync(kAll, m0 != 0u), any1 = __any_sync(kAll, m1 != 0u);
        int next = -1;
        if (any0 && any1) {
            const float k0 = min_of<float, Q>(d0), k1 = min_of<float, Q>(d1);
            const unsigned votes = __ballot_sync(kAll, k1 < k0) & rankers;
            const bool swap = P::kVote ? __popc(votes) > half : votes != 0;
            const int rn = swap ? r1 : r0, rf = swap ? r0 : r1;
            if (rf >= 0 && rn >= 0) {
                if (sp < kStackSize) {
                    entry[sp] = make_int2(rf, __float_as_int(warp_min(swap ? k0 : k1)));  // every lane stores the same
                    sp++;
                }
                next = rn;
            } else if (rn >= 0) {
                test_leaf(rf, swap ? m0 : m1);
                next = rn;
            } else {
                test_leaf(rn, swap ? m1 : m0);
                float df[Q];
#pragma unroll
                for (int q = 0; q < Q; q++) df[q] = swap ? d0[q] : d1[q];
                const unsigned mf = want_mask(p, df);
                if (__any_sync(kAll, mf != 0u)) {
                    if (rf < 0) test_leaf(rf, mf);
                    else next = rf;
                }
            }
        } else if (any0 || any1) {
            const int r = any0 ? r0 : r1;
            if (r < 0) test_leaf(r, any0 ? m0 : m1);
            else next = r;
        }
        if (next < 0) {
            if (work > budget) return sp;  // warp-uniform
            next = next_entry(p, entry, sp);
            if (next < 0) return -1;
        }
        node = next;
    }
}

// Nearest-child-first traversal of every thread for its own queries, with a stack of (node, smallest box
// distance) culled on pop.
template <bool COUNT, class P>
__device__ __forceinline__ void traverse_thread(P &p, Counters &cnt) {
    using R = typename P::R;
    constexpr int Q = P::kQn;
    int snode[kStackSize];
    R sdist[kStackSize];
    int sp = 0;
    int node = 0;
    while (true) {
        R d0[Q], d1[Q];
        int r0, r1;
        p.boxes(node, d0, d1, r0, r1);
        if (COUNT) cnt.box += 2 * Q;
        R k0 = min_of<R, Q>(d0), k1 = min_of<R, Q>(d1);
        if (k1 < k0) {
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const R t = d0[q];
                d0[q] = d1[q];
                d1[q] = t;
            }
            const R tk = k0;
            k0 = k1;
            k1 = tk;
            const int tr = r0;
            r0 = r1;
            r1 = tr;
        }
        int next = -1;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int rc = h ? r1 : r0;
            const unsigned m = rc == kEmptyRef ? 0u : (h ? want_mask(p, d1) : want_mask(p, d0));
            if (m == 0u) continue;
            if (rc < 0) {
                p.template leaf<COUNT>(leaf_first(rc), leaf_count(rc), m, cnt);
            } else if (next < 0) {
                next = rc;
            } else if (sp < kStackSize) {
                snode[sp] = rc;
                sdist[sp] = h ? k1 : k0;
                sp++;
            }
        }
        if (next < 0) {
            const R tmax = p.max_thr();
            while (sp > 0) {
                sp--;
                if (sdist[sp] < tmax) {
                    next = snode[sp];
                    break;
                }
            }
            if (next < 0) break;
        }
        node = next;
    }
}

// WARP: the 32 lanes of a warp walk one path together (every lane must call it), so node and triangle loads are
// broadcasts and leaf work does not diverge; else every thread walks by itself. A packet past its budget hands
// over while the list is short (QueryArgs::hand_most). Else it walks on without one; the fix-up's packets
// from the root again, with the windows they have: they seldom do, and a walk that can be entered anywhere cost
// every packet 2.5 % (knot 256^3 9,887 -> 10,143 us, spheres' 160^3 7 %).
template <bool WARP, bool COUNT, class P>
__device__ __forceinline__ void traverse(P &p, Counters &cnt, const QueryArgs &a) {
    if constexpr (WARP) {
        __shared__ int2 s_entry[kThreads / 32][kStackSize];
        int2 *const entry = s_entry[threadIdx.x >> 5];
        int node = 0, sp = 0, budget = a.warp_budget;
        while ((sp = traverse_packet<COUNT>(p, cnt, budget, entry, node, P::kRestarts ? 0 : sp)) >= 0) {
            if (__any_sync(0xffffffffu, *(volatile int *)a.fallback_count < a.hand_most)) {
                p.abandon();
                break;
            }
            budget = 0;
            if constexpr (P::kRestarts) {
                p.restart();
            } else {
                node = next_entry(p, entry, sp);
                if (node < 0) break;
            }
        }
    } else {
        traverse_thread<COUNT>(p, cnt);
    }
}

// ---- outputs ----------------------------------------------------------------------------------------

// Signed distance from the closest triangle (caller's index t, leaf position pos) and d^2, in
// double: the closest point, its barycentric coordinates, the pseudo-normal they select and the
// sign of (q - c) . n (serial/bvh/bvh.cpp:1751-1792, tolerance 1e-4 from bvh.cpp:1738).
__device__ double signed_distance(const DeviceMesh &m, int pos, int t, double qx, double qy, double qz, double d2,
                                  double &cx, double &cy, double &cz) {
    const Tri64 tr = load_tri64(m.tris64, pos);
    tri_closest_point_exact<double>(qx, qy, qz, tr.ax, tr.ay, tr.az, tr.bx, tr.by, tr.bz, tr.cx, tr.cy, tr.cz, cx, cy,
                                    cz);
    const double e1[3] = {tr.bx - tr.ax, tr.by - tr.ay, tr.bz - tr.az};
    const double e2[3] = {tr.cx - tr.ax, tr.cy - tr.ay, tr.cz - tr.az};
    const double r[3] = {cx - tr.ax, cy - tr.ay, cz - tr.az};
    const double d11 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
    const double d12 = e1[0] * e2[0] + e1[1] * e2[1] + e1[2] * e2[2];
    const double d22 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
    const double r1 = r[0] * e1[0] + r[1] * e1[1] + r[2] * e1[2];
    const double r2 = r[0] * e2[0] + r[1] * e2[1] + r[2] * e2[2];
    const double det = d11 * d22 - d12 * d12;
    const double l1 = det > 0 ? (d22 * r1 - d12 * r2) / det : 0;
    const double l2 = det > 0 ? (d11 * r2 - d12 * r1) / det : 0;
    const double l[3] = {1 - l1 - l2, l1, l2};
    const double tol = 1e-4;
    int small = 0, last_small = -1, last_large = -1;
#pragma unroll
    for (int v = 0; v < 3; v++) {
        if (l[v] < tol) {
            small++;
            last_small = v;
        } else {
            last_large = v;
        }
    }
    const double *n;
    if (small == 0) {
        n = m.face_n + 3 * (size_t)t;
    } else if (small == 1) {
        n = m.edge_n + 9 * (size_t)t + 3 * ((last_small + 1) % 3);
    } else {
        const int *s = last_large == 0 ? m.s0 : (last_large == 1 ? m.s1 : m.s2);
        n = m.vertex_n + 3 * (size_t)__ldg(s + t);
    }
    const double dot = (qx - cx) * __ldg(n) + (qy - cy) * __ldg(n + 1) + (qz - cz) * __ldg(n + 2);
    const double dist = sqrt(d2);
    return dot < 0 ? -dist : dist;
}

// Writes one query's outputs from its double result (best, bid, bpos); `init` is the bound the
// search started from (incoming value for the in/out outputs).
__device__ void write_result(const QueryArgs &a, long long q, double qx, double qy, double qz, double best, int bid,
                             int bpos) {
    switch (a.output) {
        case SSDF_OUT_EDF:
            store_out(a, q, sqrt(best));
            if (a.outtri && bid >= 0) a.outtri[q] = bid;
            break;
        case SSDF_OUT_SQEDF:
            store_out(a, q, best);
            break;
        case SSDF_OUT_SDF: {
            double cx, cy, cz;
            const double v = bid >= 0 ? signed_distance(a.m, bpos, bid, qx, qy, qz, best, cx, cy, cz) : sqrt(best);
            store_out(a, q, v);
            if (a.outtri) a.outtri[q] = bid;
            break;
        }
        case SSDF_OUT_CLOSEST: {
            if (bid < 0) break;
            const double dist = sqrt(best);
            const double din = load_out(a, q);
            const double dist_t = a.out_f64 ? dist : double(float(dist));
            if (din > dist_t) {
                const Tri64 tr = load_tri64(a.m.tris64, bpos);
                double cx, cy, cz;
                tri_closest_point_exact<double>(qx, qy, qz, tr.ax, tr.ay, tr.az, tr.bx, tr.by, tr.bz, tr.cx, tr.cy,
                                                tr.cz, cx, cy, cz);
                store_out(a, q, dist);
                if (a.coord_f64) {
                    ((double *)a.outx)[q] = cx, ((double *)a.outy)[q] = cy, ((double *)a.outz)[q] = cz;
                } else {
                    ((float *)a.outx)[q] = float(cx), ((float *)a.outy)[q] = float(cy), ((float *)a.outz)[q] = float(cz);
                }
                a.outtri[q] = bid;
            }
            break;
        }
        default:
            break;
    }
}

// Incoming bound of the search, as a squared distance in double.
__device__ __forceinline__ double initial_bound(const QueryArgs &a, long long q) {
    switch (a.output) {
        case SSDF_OUT_EDF:
        case SSDF_OUT_CLOSEST: {
            const double o = load_out(a, q);
            return o * o;
        }
        case SSDF_OUT_SQEDF:
            return load_out(a, q);
        default:
            return dinf();
    }
}

__device__ __forceinline__ void flush_counters(const QueryArgs &a, const Counters &c) {
    unsigned long long t = c.tri, b = c.box, f = c.fix;
    for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(0xffffffffu, t, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
        f += __shfl_xor_sync(0xffffffffu, f, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(a.counters + 0, t);
        atomicAdd(a.counters + 1, b);
        atomicAdd(a.counters + 2, f);
    }
}

// ---- kernels ----------------------------------------------------------------------------------------

// Streamed download: the block's results are stored; the last block of its chunk to finish tells the
// host, which copies the chunk out while the launch goes on. Every thread fences its own stores
// before the block counts itself, and the last block fences at system scope before the flag.
__device__ __forceinline__ void signal_chunk(const QueryArgs &a) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned c = blockIdx.x / unsigned(a.chunk_blocks);
        const unsigned members = min(unsigned(a.chunk_blocks), gridDim.x - c * unsigned(a.chunk_blocks));
        if (atomicAdd(a.chunk_counts + c, 1) == int(members) - 1) {
            __threadfence_system();
            *(volatile int *)(a.chunk_flags + c) = 1;
        }
    }
}

// Lists query q for the second stage, with its threshold (q < 2^31 is checked on the host).
__device__ __forceinline__ void hand_over(const QueryArgs &a, long long q, float thr) {
    const int slot = atomicAdd(a.fallback_count, 1);
    a.fallback_ids[slot] = int(q);
    a.fallback_thr[slot] = thr;
}

// One block of 128 lanes x kQ queries: a point-list block, or one step of a grid block's column.
// Lanes without a query (the edge of a grid brick, the tail of a point list) take part in warp-mode
// traversal with a negative threshold, so they never ask for a node. seed[s] is the leaf position of
// the closest triangle the lane's query s found one step below (-1: none); it is updated here.
template <int PREC, bool WARP, bool COUNT>
__device__ __forceinline__ void query_step(const QueryArgs &a, int step, const bool (&valid)[kQ],
                                           const long long (&qid)[kQ], const long long (&gi)[kQ],
                                           const long long (&gj)[kQ], const long long (&gk)[kQ], bool any,
                                           int (&seed)[kQ], Counters &cnt) {
    constexpr int Q = kQ;
    const bool seeded = a.seed != 0 && step > 0;
    if (PREC == SSDF_PREC_F64) {
        ExactPolicy<double, Q> p(a.m);
#pragma unroll
        for (int s = 0; s < Q; s++) {
            if (valid[s]) {
                double x, y, z;
                query_point(a, qid[s], gi[s], gj[s], gk[s], x, y, z);
                p.set(s, x, y, z, initial_bound(a, qid[s]));
                if (seeded && seed[s] >= 0) p.seed(s, seed[s]);
            } else {
                p.disable(s);
            }
        }
        if (WARP || any) traverse<WARP, COUNT>(p, cnt, a);
#pragma unroll
        for (int s = 0; s < Q; s++) {
            if (!valid[s]) continue;
            if (WARP && p.gone && p.thr[s] > 0.f) {
                hand_over(a, qid[s], p.thr[s]);
                continue;
            }
            write_result(a, qid[s], p.px[s], p.py[s], p.pz[s], p.best[s], p.bid[s], p.bpos[s]);
            if (p.bpos[s] >= 0) seed[s] = p.bpos[s];
        }
    } else if (PREC == SSDF_PREC_F32) {
        // the reference's float arithmetic end to end (edf<float>'s value); edf and sqedf outputs
        ExactPolicy<float, Q> p(a.m);
#pragma unroll
        for (int s = 0; s < Q; s++) {
            if (valid[s]) {
                double x, y, z;
                query_point(a, qid[s], gi[s], gj[s], gk[s], x, y, z);
                const long long q = qid[s];
                const float o = a.out_f64 ? float(((const double *)a.out)[q]) : ((const float *)a.out)[q];
                p.set(s, float(x), float(y), float(z), a.output == SSDF_OUT_SQEDF ? o : o * o);
                if (seeded && seed[s] >= 0) p.seed(s, seed[s]);
            } else {
                p.disable(s);
            }
        }
        if (WARP || any) traverse<WARP, COUNT>(p, cnt, a);
#pragma unroll
        for (int s = 0; s < Q; s++) {
            if (!valid[s]) continue;
            const long long q = qid[s];
            if (WARP && p.gone && p.thr[s] > 0.f) {
                hand_over(a, q, p.thr[s]);
                continue;
            }
            if (a.output == SSDF_OUT_SQEDF) {
                store_out(a, q, double(p.best[s]));
            } else {
                store_out(a, q, double(sqrtf(p.best[s])));
                if (a.outtri && p.bid[s] >= 0) a.outtri[q] = p.bid[s];
            }
            if (p.bpos[s] >= 0) seed[s] = p.bpos[s];
        }
    } else {
        __shared__ float s_wd[kQ * kCand * kThreads];
        __shared__ int s_wp[kQ * kCand * kThreads];
        FastPolicy<Q> p(a.m, a.tau_rel, s_wd, s_wp);
        bool exact[Q];  // a finite point beyond the float filter's range: the second stage, exactly
#pragma unroll
        for (int s = 0; s < Q; s++) {
            exact[s] = false;
            if (valid[s]) {
                double x, y, z;
                query_point(a, qid[s], gi[s], gj[s], gk[s], x, y, z);
                const double ax = fabs(x), ay = fabs(y), az = fabs(z);
                exact[s] = (ax > kFilterMaxCoord || ay > kFilterMaxCoord || az > kFilterMaxCoord) &&
                           ax < dinf() && ay < dinf() && az < dinf();
                const double init = initial_bound(a, qid[s]);
                // float start bound rounded up, so no triangle closer in double is cut off
                if (exact[s]) {
                    p.disable(s);
                } else {
                    p.set(s, filter_coord(x, 0, a.m), filter_coord(y, 1, a.m), filter_coord(z, 2, a.m),
                          init < dinf() ? __double2float_ru(init) : finf());
                    if (seeded && seed[s] >= 0) p.seed(s, seed[s]);
                }
            } else {
                p.disable(s);
            }
        }
        if (WARP || any) traverse<WARP, COUNT>(p, cnt, a);
#pragma unroll
        for (int s = 0; s < Q; s++) {
            if (!valid[s]) continue;
            const long long q = qid[s];
            if (exact[s] || p.evicted[s] < p.thr[s]) {
                hand_over(a, q, exact[s] ? finf() : p.thr[s]);
                continue;
            }
            // the double point and bound are recomputed here rather than kept live through the walk
            double rx, ry, rz;
            query_point(a, q, gi[s], gj[s], gk[s], rx, ry, rz);
            double b = initial_bound(a, q);
            int bid = -1, bpos = -1;
            for (int c = 0; c < p.used[s]; c++) {
                const int ix = p.slot(s, c);
                if (p.wd[ix] < p.thr[s]) {
                    const int pos = p.wp[ix];
                    const Tri64 t = load_tri64(a.m.tris64, pos);
                    const double d2 =
                        tri_dist_sq_exact<double>(rx, ry, rz, t.ax, t.ay, t.az, t.bx, t.by, t.bz, t.cx, t.cy, t.cz);
                    if (COUNT) cnt.fix++;
                    if (d2 < b || (d2 == b && bid >= 0 && t.id < bid)) {
                        b = d2;
                        bid = t.id;
                        bpos = pos;
                    }
                }
            }
            write_result(a, q, rx, ry, rz, b, bid, bpos);
            if (bpos >= 0) seed[s] = bpos;
        }
    }
}

// A point-list block, or a grid block's column step by step (each step seeded from the one below).
template <int PREC, bool WARP, bool COUNT>
__device__ __forceinline__ void query_block(const QueryArgs &a, long long block, Counters &cnt) {
    constexpr int Q = kQ;
    int seed[Q];
#pragma unroll
    for (int s = 0; s < Q; s++) seed[s] = -1;
    const int steps = a.is_grid ? a.grid_steps : 1;
    for (int step = 0; step < steps; step++) {
        long long qid[Q], gi[Q], gj[Q], gk[Q];
        bool valid[Q];
        bool any = false;
#pragma unroll
        for (int s = 0; s < Q; s++) {
            gi[s] = gj[s] = gk[s] = 0;
            valid[s] = map_query(a, block, step, s, qid[s], gi[s], gj[s], gk[s]);
            any |= valid[s];
        }
        // this warp's part of the column has left the grid (higher steps have no node either); a warp
        // decision, not a block one: the warps share nothing, and a block barrier per step made every
        // warp wait for the block's slowest (17 % on the torus knot)
        if (step > 0 && !__any_sync(0xffffffffu, any)) break;
        query_step<PREC, WARP, COUNT>(a, step, valid, qid, gi, gj, gk, any, seed, cnt);
    }
}

// SIGNAL: the streamed grid download's instantiation, whose blocks count themselves done per chunk
// (a separate instantiation: the dormant signal code cost the fix-up kernel 3 % where it was merely
// compiled in). The arguments are __grid_constant__: their address is passed on (to query_step,
// map_query, write_result), and without it each thread first copies them to its local memory (64^3 grid on
// 5,120 triangles 239 -> 224 us, 500,003 points near the knot 915 -> 889, 1,000 points 48 -> 43).
template <int PREC, bool WARP, bool COUNT, bool SIGNAL = false>
__global__ void __launch_bounds__(kThreads, PREC == SSDF_PREC_F64 ? kF64MinBlocks : SSDF_B200_QUERY_MIN_BLOCKS)
    k_query(const __grid_constant__ QueryArgs a) {
    Counters cnt;
    query_block<PREC, WARP, COUNT>(a, blockIdx.x, cnt);
    if (COUNT) flush_counters(a, cnt);
    if constexpr (SIGNAL) signal_chunk(a);
}

// ---- second fix-up stage: one warp per overflowed query --------------------------------------------
//
// A query whose window overflowed its slots is walked again from its final window, and a query whose
// packet ran out of budget from the window it had then: every triangle whose float distance is
// inside the window is re-evaluated in double. The window only shrinks: after each step, by the first stage's
// rule, to what the warp's smallest non-proxy key allows, or the smallest double distance found where that is
// nearer (it bounds the winner's distance as a key does, without a key's error; beside needles, whose proxies'
// keys count for nothing, it is all there is: 24^3 nodes at 2,000 needles 3,251 -> 303 us). So the visiting
// order is free, and the warp walks the tree breadth-parallel: each step
// the 32 lanes take up to 32 nodes from the warp's shared stack, test their children, run the
// wanted leaves, and push the wanted internal children (ballot-compacted). A lane keeps the
// lexicographic (d^2, index) minimum of the triangles it evaluated (the incoming bound ranks -1, so
// it wins ties, as in the sequential rule) and a warp reduction takes the minimum of those: the
// same value as the sequential walk, since each triangle's double distance does not depend on the
// order. The boxes and the float test are the first stage's: the double winner
// lies inside the window by the margin tau, so its boxes pass.
constexpr int kWinStack = 512;  // node slots of a warp's shared stack
// Blocks per SM of the second stage's grid. Its kernel keeps its registers (capping them for 5, 6 or 8
// resident blocks: 64^3 icosphere grid 233 -> 234 / 238 / 255 us); a grid of 12 per SM queues the rest
// behind the resident blocks, so a warp takes one query where a smaller grid had each take two or three,
// and blocks that finish early make room.
#ifndef SSDF_B200_WINDOW_BLOCKS_PER_SM
#define SSDF_B200_WINDOW_BLOCKS_PER_SM 12
#endif
constexpr int kWindowBlocksPerSm = SSDF_B200_WINDOW_BLOCKS_PER_SM;

// A window of +inf takes every node and triangle, whatever its float key (a query point beyond the
// float filter's range, whose keys may have overflowed, is answered this way: exactly, in double).
__device__ __forceinline__ bool in_window(float key, float thr) { return key < thr || thr == finf(); }

// A finite point beyond the fix-up filter's range: everything is evaluated, exactly, in double.
template <int PREC>
__device__ __forceinline__ bool beyond_filter(double x, double y, double z) {
    return PREC == SSDF_PREC_F32_FIXUP && fmax(fmax(fabs(x), fabs(y)), fabs(z)) > double(kFilterMaxCoord);
}

// What a lane of a warp-per-query walk knows: the query in the arithmetic's own terms, the lexicographic
// minimum of the triangles the lane evaluated, and the box threshold its finds allow. PREC as the query
// kernels'.
template <int PREC>
struct LaneWalk {
    using T = typename std::conditional<PREC == SSDF_PREC_F32, float, double>::type;
    const DeviceMesh &m;
    T qx, qy, qz;
    float2 bx, by, bz;  // the point in the box frame, each coordinate twice
    T d2;               // the minimum, its triangle and leaf position (-1: the incoming bound)
    int id = -1, pos = -1;
    float kbest = finf();  // fix-up: the smallest key of a non-proxy triangle met
    float tau_rel;
    T margin;
    __device__ LaneWalk(const QueryArgs &a, double x, double y, double z, T init)
        : m(a.m), qx(T(x)), qy(T(y)), qz(T(z)), d2(init), tau_rel(a.tau_rel), margin(ExactData<T>::margin(a.m)) {
        if constexpr (PREC == SSDF_PREC_F32_FIXUP) {
            bx = twice(filter_coord(x, 0, m)), by = twice(filter_coord(y, 1, m)), bz = twice(filter_coord(z, 2, m));
        } else {
            bx = twice(ExactData<T>::box_coord(qx, 0, m));
            by = twice(ExactData<T>::box_coord(qy, 1, m));
            bz = twice(ExactData<T>::box_coord(qz, 2, m));
        }
    }
    __device__ __forceinline__ bool finite() const {
        const T lim = ExactData<T>::beyond(m);
        return fabs(qx) < lim && fabs(qy) < lim && fabs(qz) < lim;
    }
    // the threshold the incoming bound allows
    __device__ __forceinline__ float start_thr() const {
        if constexpr (PREC == SSDF_PREC_F32_FIXUP)
            return d2 < T(0) ? -1.f : window_thr(d2 < T(dinf()) ? __double2float_ru(d2) : finf(), tau_rel, m.coord_scale);
        else
            return ExactData<T>::start_thr(d2, margin, m);
    }
    // the threshold the whole warp's finds allow (warp-wide)
    __device__ __forceinline__ float found_thr() const {
        if constexpr (PREC == SSDF_PREC_F32_FIXUP)
            return window_thr(warp_min(fminf(kbest, __double2float_ru(d2))), tau_rel, m.coord_scale);
        else
            return warp_min(ExactData<T>::box_thr(d2, margin, m));
    }
    // the threshold a squared distance (in the box frame) that some triangle does not exceed allows, and
    // whether the minimum found bears it out
    __device__ __forceinline__ float cut_thr(float cut) const {
        if constexpr (PREC == SSDF_PREC_F32_FIXUP) return window_thr(cut, tau_rel, m.coord_scale);
        return cut;
    }
    __device__ __forceinline__ bool confirms(float cut) const {
        if constexpr (PREC == SSDF_PREC_F32_FIXUP) return d2 <= double(cut);
        return ExactData<T>::box_thr(d2, margin, m) <= cut;
    }
    __device__ __forceinline__ bool wants(float key, float thr) const {
        if constexpr (PREC == SSDF_PREC_F32_FIXUP) return in_window(key, thr);
        return ExactData<T>::box_key(key) < thr;
    }
    __device__ __forceinline__ void take(T e2, int t, int p) {
        if (e2 < d2 || (e2 == d2 && t < id)) d2 = e2, id = t, pos = p;
    }
    // tests the triangle at leaf position k
    __device__ __forceinline__ void triangle(int k, float thr, bool count, Counters &cnt) {
        if (count) cnt.tri++;
        if constexpr (PREC == SSDF_PREC_F32_FIXUP) {
            const FiltRec r = load_filt(m.filt32, k);
            const float f = tri_dist_sq_filter(bx.x, by.x, bz.x, r);  // the packets' key
            if (r.pen == 0.f && f < kbest) kbest = f;
            if (!in_window(f, thr)) return;
            if (count) cnt.fix++;
        }
        const auto u = ExactData<T>::tri(m, k);
        take(tri_dist_sq_exact<T>(qx, qy, qz, u.ax, u.ay, u.az, u.bx, u.by, u.bz, u.cx, u.cy, u.cz), u.id, k);
    }
};

// A lane's own depth-first walk of the subtree under `root` (when the warp's stack is full). Depth
// below kStackSize is checked when the mesh is built, and a depth-first walk that pushes both
// children holds at most depth + 1 entries.
template <int PREC>
__device__ __noinline__ void lane_subtree(LaneWalk<PREC> &w, int root, float thr, bool count, Counters &cnt) {
    int st[kStackSize];
    int sp = 0;
    st[sp++] = root;
    while (sp > 0) {
        int r[2];
        const float2 d = obb_dist_sq_pair(w.bx, w.by, w.bz, w.m.obb + 8 * st[--sp], r[0], r[1]);
        if (count) cnt.box += 2;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (r[h] == kEmptyRef || !w.wants(h ? d.y : d.x, thr)) continue;
            if (r[h] < 0)
                for (int k = 0; k < leaf_count(r[h]); k++) w.triangle(leaf_first(r[h]) + k, thr, count, cnt);
            else if (sp < kStackSize)
                st[sp++] = r[h];
        }
    }
}

// A warp's shared memory: its node stack, the nodes of a step, and the leaves they found.
struct WarpShared {
    int stack[kWinStack];
    float4 node[32][9];  // 8 per node, rows of 144 bytes: a lane reads its own without bank conflicts
    int leaf[64];
};

// The whole warp walks the tree for one query from threshold thr; w then holds the minimum in every lane.
// Each step takes up to 32 nodes from the warp's stack, a lane each. The loads are the bound (a lane
// reading its own 128-byte node touches a line per lane and load): eight lanes fetch a node together
// and each lane reads its node back from shared memory, and the leaves' triangles go four lanes to a leaf,
// neighbours reading neighbouring records. 130,000 points near the 131,072-triangle knot, a warp each:
// 1,862 -> 1,604 us, from the root; with the copy below 1,460.
// shrink: the threshold follows the finds (false: it stays +inf, everything is evaluated). upper: no close
// bound is known yet, so the boxes' own upper bounds (the farthest a triangle inside can be) cut the walk
// before the first triangle is met. Such a cut assumes that a triangle's computed distance is not above
// its box's bound (with 5 % to spare), which a needle's rounding can break: the walk returns false when
// the minimum found does not confirm the smallest cut it used, and is then repeated without them.
template <int PREC, bool COUNT>
__device__ bool warp_walk(LaneWalk<PREC> &w, float thr, bool shrink, bool upper, WarpShared &sh, int cap,
                          Counters &cnt) {
    const unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    using T = typename LaneWalk<PREC>::T;
    float cut = finf();  // the smallest box upper bound used
    int *const stack = sh.stack;
    // the walk starts from the tree's first nodes with internal children only, at most 32 (k_box_frame)
    int sp = 1;  // warp-uniform
    if (cap >= 32) {
        sp = __ldg(w.m.entry);
        if (lane < sp) stack[lane] = __ldg(w.m.entry + 1 + lane);
    } else if (lane == 0) {
        stack[0] = 0;
    }
    __syncwarp();
    while (sp > 0) {
        const int take = sp < 32 ? sp : 32, base = sp - take;
        sp = base;
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int row = 4 * r + (lane >> 3);
            if (row < take) sh.node[row][lane & 7] = __ldg(w.m.obb + 8 * stack[base + row] + (lane & 7));
        }
        __syncwarp();
        int c0 = kEmptyRef, c1 = kEmptyRef;
        float2 d = make_float2(0.f, 0.f), far = make_float2(finf(), finf());
        if (lane < take) {
            d = obb_dist_sq_bounds(w.bx, w.by, w.bz, sh.node[lane], c0, c1, far);
            if (COUNT) cnt.box += 2;
        }
        if (upper) {
            const float u = warp_min(fminf(c0 == kEmptyRef ? finf() : far.x, c1 == kEmptyRef ? finf() : far.y));
            cut = fminf(cut, u < finf() ? fmaxf(u * 1.05f, FLT_MIN) : finf());  // an overflow or a NaN cuts nothing
            thr = fminf(thr, w.cut_thr(cut));
        }
        const bool w0 = c0 != kEmptyRef && w.wants(d.x, thr), w1 = c1 != kEmptyRef && w.wants(d.y, thr);
        // leaves: listed, then tested eight at a time, four lanes to each
        const unsigned l0 = __ballot_sync(kAll, w0 && c0 < 0), l1 = __ballot_sync(kAll, w1 && c1 < 0);
        const int nl0 = __popc(l0), nl = nl0 + __popc(l1);
        if (nl > 0) {
            if (w0 && c0 < 0) sh.leaf[__popc(l0 & below)] = c0;
            if (w1 && c1 < 0) sh.leaf[nl0 + __popc(l1 & below)] = c1;
            __syncwarp();
            for (int f = 0; f < nl; f += 8) {
                const int at = f + (lane >> 2);
                if (at < nl) {
                    const int ref = sh.leaf[at], first = leaf_first(ref), n = leaf_count(ref);
                    for (int k = lane & 3; k < n; k += 4) w.triangle(first + k, thr, COUNT, cnt);
                }
                __syncwarp();
                if (shrink) thr = fminf(thr, w.found_thr());
            }
        }
        const bool p0 = w0 && c0 >= 0, p1 = w1 && c1 >= 0;
        const unsigned m0 = __ballot_sync(kAll, p0), m1 = __ballot_sync(kAll, p1);
        const int n0 = __popc(m0), total = n0 + __popc(m1);
        if (sp + total <= cap) {
            if (p0) stack[sp + __popc(m0 & below)] = c0;
            if (p1) stack[sp + n0 + __popc(m1 & below)] = c1;
            sp += total;
        } else {
            LaneWalk<PREC> own = w;  // a copy goes by reference, so that w stays in registers
            if (p0) lane_subtree(own, c0, thr, COUNT, cnt);
            if (p1) lane_subtree(own, c1, thr, COUNT, cnt);
            w.d2 = own.d2, w.id = own.id, w.pos = own.pos, w.kbest = own.kbest;
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const T od = __shfl_xor_sync(kAll, w.d2, o);
        const int oid = __shfl_xor_sync(kAll, w.id, o), opos = __shfl_xor_sync(kAll, w.pos, o);
        if (od < w.d2 || (od == w.d2 && oid < w.id)) w.d2 = od, w.id = oid, w.pos = opos;
    }
    return !(cut < finf()) || w.confirms(cut);  // whatever the cuts left out lies above the minimum
}

// The incoming bound of a query in the arithmetic's own terms, and its result.
template <int PREC>
__device__ __forceinline__ typename LaneWalk<PREC>::T lane_bound(const QueryArgs &a, long long q) {
    if constexpr (PREC == SSDF_PREC_F32) {
        const float o = a.out_f64 ? float(((const double *)a.out)[q]) : ((const float *)a.out)[q];
        return a.output == SSDF_OUT_SQEDF ? o : o * o;
    } else {
        return initial_bound(a, q);
    }
}
template <int PREC>
__device__ __forceinline__ void lane_result(const QueryArgs &a, long long q, double x, double y, double z,
                                            const LaneWalk<PREC> &w) {
    if constexpr (PREC == SSDF_PREC_F32) {
        if (a.output == SSDF_OUT_SQEDF) {
            store_out(a, q, double(w.d2));
        } else {
            store_out(a, q, double(sqrtf(w.d2)));
            if (a.outtri && w.id >= 0) a.outtri[q] = w.id;
        }
    } else {
        write_result(a, q, x, y, z, w.d2, w.id, w.pos);
    }
}

// The whole warp answers handed-over query `idx` of job `a`; lane 0 writes the result.
template <int PREC, bool COUNT>
__device__ void window_warp(const QueryArgs &a, int idx, WarpShared &sh, int cap, Counters &cnt) {
    const long long q = a.fallback_ids[idx];
    long long i = 0, j = 0, k = 0;
    if (a.is_grid) grid_ijk(a, q, i, j, k);
    double qx, qy, qz;
    query_point(a, q, i, j, k, qx, qy, qz);
    const float thr = a.fallback_thr[idx];
    LaneWalk<PREC> w(a, qx, qy, qz, lane_bound<PREC>(a, q));
    // The infinite window of a point beyond the filter's range stays; a packet that met only proxies before
    // its budget ran out hands over an infinite one too, which shrinks like any other.
    warp_walk<PREC, COUNT>(w, thr, !beyond_filter<PREC>(qx, qy, qz), false, sh, cap, cnt);
    if ((threadIdx.x & 31) == 0) lane_result(a, q, qx, qy, qz, w);
}

// Handed-over queries of one launch, a warp each. `cap` (<= kWinStack) is the shared stack's usable
// depth: kWinStack, lowered only to test the per-lane subtree walk.
template <int PREC, bool COUNT>
__global__ void __launch_bounds__(kThreads) k_window(const __grid_constant__ QueryArgs a, int cap) {
    __shared__ WarpShared s_warp[kThreads / 32];
    const int n = *a.fallback_count;
    const int w = (blockIdx.x * kThreads + threadIdx.x) >> 5, nw = (gridDim.x * kThreads) >> 5;
    Counters cnt;
    for (int idx = w; idx < n; idx += nw) window_warp<PREC, COUNT>(a, idx, s_warp[threadIdx.x >> 5], cap, cnt);
    if (COUNT) flush_counters(a, cnt);
}

// ---- small point lists: one warp per query ------------------------------------------------------------
//
// A list too short to fill the GPU with 32-query packets is bound by one walk's serial chain. Here the 32
// lanes share it: up to 32 nodes a step, so a walk takes about as many steps as the tree is deep, in one
// launch without ordering the points, an overflow list or a second stage. It is bound by the latency of its
// dependent loads (1,000 points on the sphere: 2,419 instructions a query, 13 % of issue slots busy). us against packets (fix-up, points
// near the surface; 131,072-triangle knot, 1,280-triangle sphere): 100 points 57 / 244 and 44 / 106; 1,000
// 59 / 320 and 46 / 98; 16,000 242 / 577 and 162 / 215; 65,536 836 / 620 and 508 / 214.
template <int PREC, bool COUNT>
__global__ void __launch_bounds__(kThreads, 6) k_query_warp(const __grid_constant__ QueryArgs a, int cap) {
    __shared__ WarpShared s_warp[kThreads / 32];
    const long long q = (blockIdx.x * (long long)kThreads + threadIdx.x) >> 5;
    if (q >= a.npoints) return;  // a whole warp
    WarpShared &sh = s_warp[threadIdx.x >> 5];
    Counters cnt;
    double x, y, z;
    query_point(a, q, 0, 0, 0, x, y, z);
    LaneWalk<PREC> w(a, x, y, z, lane_bound<PREC>(a, q));
    if (w.finite()) {
        const bool beyond = beyond_filter<PREC>(x, y, z);
        bool upper = !beyond;
        while (!warp_walk<PREC, COUNT>(w, beyond ? finf() : w.start_thr(), !beyond, upper, sh, cap, cnt)) upper = false;
    }
    if ((threadIdx.x & 31) == 0) lane_result(a, q, x, y, z, w);
    if (COUNT) flush_counters(a, cnt);
}

// ---- batches: many (mesh, query set) jobs in one persistent launch -----------------------------------
//
// The job table lives in device memory (BatchHeader + QueryArgs[] + first block of each job), so a
// captured CUDA graph of these two kernels replays for any batch composition without being
// re-instantiated: only the table is rewritten before each replay. Blocks pull work items (one
// 128-query block of one job) from an atomic counter, largest jobs first (the host orders them).

template <int PREC, bool WARP, bool COUNT>
__global__ void __launch_bounds__(kThreads, PREC == SSDF_PREC_F64 ? kF64MinBlocks : SSDF_B200_QUERY_MIN_BLOCKS)
    k_query_batch(const BatchHeader *__restrict__ hdr, const QueryArgs *__restrict__ jobs,
                  const long long *__restrict__ first_block, unsigned long long *__restrict__ next_item) {
    __shared__ long long s_item;
    const int njobs = hdr->njobs;
    const long long total = hdr->total_blocks;
    Counters cnt;
    while (true) {
        if (threadIdx.x == 0) s_item = (long long)atomicAdd(next_item, 1ull);
        __syncthreads();
        const long long it = s_item;
        __syncthreads();
        if (it >= total) break;
        int lo = 0, hi = njobs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(first_block + mid) <= it) lo = mid; else hi = mid - 1;
        }
        query_block<PREC, WARP, COUNT>(jobs[lo], it - __ldg(first_block + lo), cnt);
    }
    if (COUNT && njobs > 0) flush_counters(jobs[0], cnt);
}

// Overflowed queries of every job: the jobs' lists laid end to end and dealt to the warps in turn,
// so no warp takes the same position of every list.
template <int PREC, bool COUNT>
__global__ void __launch_bounds__(kThreads) k_window_batch(const BatchHeader *__restrict__ hdr,
                                                           const QueryArgs *__restrict__ jobs, int cap) {
    __shared__ WarpShared s_warp[kThreads / 32];
    const int njobs = hdr->njobs;
    const long long w = (blockIdx.x * kThreads + threadIdx.x) >> 5, nw = (gridDim.x * kThreads) >> 5;
    Counters cnt;
    long long base = 0;  // overflowed queries of the jobs before jb
    for (int jb = 0; jb < njobs; jb++) {
        const QueryArgs &a = jobs[jb];
        if (!a.fallback_count) continue;
        const int n = *a.fallback_count;
        for (long long idx = ((w - base) % nw + nw) % nw; idx < n; idx += nw)
            window_warp<PREC, COUNT>(a, int(idx), s_warp[threadIdx.x >> 5], cap, cnt);
        base += n;
    }
    if (COUNT && njobs > 0) flush_counters(jobs[0], cnt);
}

// Usable depth of the second stage's shared stack: kWinStack, or SSDF_B200_WINDOW_STACK (1 ..
// kWinStack) to exercise the per-lane subtree walk in tests.
int window_stack_cap() {
    const int v = env_int("SSDF_B200_WINDOW_STACK", kWinStack);
    return v < 1 ? 1 : (v > kWinStack ? kWinStack : v);
}

// Blocks of the second fix-up stage (kWindowBlocksPerSm per SM, four warps each; more than fit at
// once). The warps stride over the overflow count, which is only known on the device.
unsigned window_grid() {
    static int cached[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    int &g = cached[dev & 63];
    if (g == 0) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        g = kWindowBlocksPerSm * std::max(1, sms);
    }
    return unsigned(g);
}

template <int PREC, bool WARP>
cudaError_t launch_batch_main(const BatchLaunch &b, bool count, cudaStream_t stream) {
    if (count)
        k_query_batch<PREC, WARP, true><<<b.grid, kThreads, 0, stream>>>(b.hdr, b.jobs, b.first_block, b.next_item);
    else
        k_query_batch<PREC, WARP, false><<<b.grid, kThreads, 0, stream>>>(b.hdr, b.jobs, b.first_block, b.next_item);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (count)
        k_window_batch<PREC, true><<<kWindowBlocksPerSm * b.sms, kThreads, 0, stream>>>(b.hdr, b.jobs, window_stack_cap());
    else
        k_window_batch<PREC, false><<<kWindowBlocksPerSm * b.sms, kThreads, 0, stream>>>(b.hdr, b.jobs, window_stack_cap());
    return cudaGetLastError();
}

template <int PREC>
cudaError_t launch_batch_prec(const BatchLaunch &b, bool count, cudaStream_t stream) {
    return b.warp ? launch_batch_main<PREC, true>(b, count, stream) : launch_batch_main<PREC, false>(b, count, stream);
}

template <int PREC, bool WARP>
int batch_occupancy() {
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_query_batch<PREC, WARP, false>, kThreads, 0);
    return nb > 0 ? nb : 1;
}

thread_local unsigned long long t_last_counts[4] = {0, 0, 0, 0};

template <int PREC>
cudaError_t launch_query_warp(const QueryArgs &a, bool count, cudaStream_t stream) {
    const unsigned blocks = unsigned((a.npoints * 32 + kThreads - 1) / kThreads);
    const int cap = window_stack_cap();
    count ? k_query_warp<PREC, true><<<blocks, kThreads, 0, stream>>>(a, cap)
          : k_query_warp<PREC, false><<<blocks, kThreads, 0, stream>>>(a, cap);
    return cudaGetLastError();
}

template <int PREC, bool WARP>
cudaError_t launch_main(const QueryArgs &a, bool count, unsigned nblocks, cudaStream_t stream) {
    // a counting launch raises no chunk flags: its streamed download copies every chunk once the launch
    // has ended
    if (count)
        k_query<PREC, WARP, true><<<nblocks, kThreads, 0, stream>>>(a);
    else if (a.chunk_flags)
        k_query<PREC, WARP, false, true><<<nblocks, kThreads, 0, stream>>>(a);
    else
        k_query<PREC, WARP, false><<<nblocks, kThreads, 0, stream>>>(a);
    return cudaGetLastError();
}

template <int PREC>
cudaError_t launch_prec(const QueryArgs &a, bool warp, bool count, unsigned nblocks, cudaStream_t stream) {
    return warp ? launch_main<PREC, true>(a, count, nblocks, stream) : launch_main<PREC, false>(a, count, nblocks, stream);
}

// The query kernel and, with a hand-over list, the second stage.
template <int PREC>
cudaError_t launch_two_stages(const QueryArgs &a, bool warp, bool count, unsigned nblocks, cudaStream_t stream,
                              int cap = 0) {
    const cudaError_t e = launch_prec<PREC>(a, warp, count, nblocks, stream);
    if (e != cudaSuccess || !a.fallback_count) return e;
    if (cap == 0) cap = window_stack_cap();
    count ? k_window<PREC, true><<<window_grid(), kThreads, 0, stream>>>(a, cap)
          : k_window<PREC, false><<<window_grid(), kThreads, 0, stream>>>(a, cap);
    return cudaGetLastError();
}

}  // namespace

void set_last_counts(unsigned long long tri, unsigned long long box, unsigned long long fix,
                     unsigned long long fallback) {
    t_last_counts[0] = tri, t_last_counts[1] = box, t_last_counts[2] = fix, t_last_counts[3] = fallback;
}

int query_counts(int64_t *tri, int64_t *box, int64_t *fix, int64_t *fallback) {
    if (tri) *tri = (int64_t)t_last_counts[0];
    if (box) *box = (int64_t)t_last_counts[1];
    if (fix) *fix = (int64_t)t_last_counts[2];
    if (fallback) *fallback = (int64_t)t_last_counts[3];
    return SSDF_OK;
}

// Traversal mode: SSDF_B200_TRAVERSAL=warp|thread overrides; by default grids (coherent bricks) walk
// in warp packets and point lists thread by thread.
static bool use_warp(const QueryArgs &a) {
    if (a.force_traversal) return a.force_traversal == 1;
    const char *v = env_str("SSDF_B200_TRAVERSAL");
    if (v && !strcmp(v, "warp")) return true;
    if (v && !strcmp(v, "thread")) return false;
    return a.is_grid != 0 || a.order != nullptr;  // sorted point lists are coherent enough for packets
}

// Point lists in Morton order: a warp's 32 slots then hold neighbouring points, which the packet walk
// needs (in input order a warp of scattered queries keeps about 5 of its lanes busy). Keys are 30-bit
// Morton codes of the points in the mesh's bounding box (the union of the root's two child boxes),
// points outside it clamped to its faces; the stable radix sort makes the order deterministic.
__global__ void k_point_keys(long long n, const void *__restrict__ x, const void *__restrict__ y,
                             const void *__restrict__ z, int f64, const float4 *__restrict__ root,
                             uint32_t *__restrict__ keys, int *__restrict__ vals) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 c0 = __ldg(root), c1 = __ldg(root + 1), c2 = __ldg(root + 2);
    // child boxes: (lox, hix, loy, hiy) of each, then (loz, hiz) of both; an empty child is inverted
    const float lo[3] = {fminf(c0.x, c1.x), fminf(c0.z, c1.z), fminf(c2.x, c2.z)};
    const float hi[3] = {fmaxf(c0.y, c1.y), fmaxf(c0.w, c1.w), fmaxf(c2.y, c2.w)};
    const float p[3] = {f64 ? float(((const double *)x)[i]) : ((const float *)x)[i],
                        f64 ? float(((const double *)y)[i]) : ((const float *)y)[i],
                        f64 ? float(((const double *)z)[i]) : ((const float *)z)[i]};
    uint32_t key = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const float ext = hi[d] - lo[d];
        float u = ext > 0.f ? (p[d] - lo[d]) / ext : 0.5f;
        u = fminf(fmaxf(u, 0.f), 1.f);  // NaN -> 0
        uint32_t v = uint32_t(fminf(u * 1024.f, 1023.f));
        v = (v * 0x00010001u) & 0xFF0000FFu;
        v = (v * 0x00000101u) & 0x0F00F00Fu;
        v = (v * 0x00000011u) & 0xC30C30C3u;
        v = (v * 0x00000005u) & 0x49249249u;
        key |= v << (2 - d);
    }
    keys[i] = key;
    vals[i] = int(i);
}

// Seeded steps save box and triangle tests, but a column is one serial chain, and its last wave is as long
// as its steps. Ten waves of resident blocks is where one pays for the other. us at 1 / 2 / 4 / 8 steps,
// fix-up: 110^3 on 81,920 triangles (10 waves at one step) 1,824 / 2,113 / 2,823 / 3,567; 145^3 (23 waves)
// 4,109 / 4,013 / 4,947; 200^3 (60) 6,476 / 6,128 / 6,195 / 7,214; torus knot 115^3 (11) 1,982 / 1,924 /
// 2,329, 145^3 (23) 3,192 / 2,922 / 2,954, 180^3 (44) 5,160 / 4,699 / 4,481, 200^3 (60) 6,574 / 5,945 /
// 5,563 / 5,575, 256^3 (127) 12,111 / 10,864 / 10,190 / 9,910, 400^3 (483) 38,789 / 34,249 / 31,691 / 30,203;
// 41,006-triangle torus 150^3 (25) 2,417 / 2,625 / 2,994, 256^3 7,658 / 7,461 / 7,430 / 7,618.
// The double kernel takes the same steps, by the float kernels' blocks per SM, without sweeps of its own; the knot's
// 128^3 grid in double loses by it (2,582 us with the rule of four waves, 2,753 with this one).
constexpr long long kGridWaves = 10;

int grid_steps_for(long long one_step_blocks) {
    const int forced = env_int("SSDF_B200_GRID_STEPS", 0);
    if (forced > 0) return forced < kMaxGridSteps ? forced : kMaxGridSteps;
    static int slots[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    int &r = slots[dev & 63];
    if (r == 0) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        r = std::max(1, sms) * SSDF_B200_QUERY_MIN_BLOCKS;
    }
    int steps = kMaxGridSteps;
    while (steps > 1 && one_step_blocks / steps < kGridWaves * r) steps >>= 1;
    return steps;
}

void set_grid_steps(QueryArgs *a) {
    if (!a->is_grid) return;
    a->grid_steps = grid_steps_for(grid_blocks_x(a->nx) * grid_blocks_y(a->ny) * grid_blocks_z(a->nz, 1));
}

// Measured on B200 over axis-aligned boxes: the torus knot with 29 % of its triangles slivers still ran 1.4x
// faster on the fix-up path than on FP64; the beam lattice (64 % slivers, in parallel bundles) ran 5x slower. Not
// measured again over oriented boxes, with which the two kernels are closer.
constexpr double kIllMaxFraction = 0.5;

// The fix-up path hands a mesh to the FP64 kernel when more than this fraction of its triangles are
// ill-conditioned (SSDF_B200_ILL_MAX overrides; above 1 never).
bool sliver_heavy(const DeviceMesh &m) {
    const char *v = env_str("SSDF_B200_ILL_MAX");
    const double f = v ? atof(v) : kIllMaxFraction;
    return m.nt > 0 && double(m.nill) > f * double(m.nt);
}

// A fix-up request on this mesh runs the FP64 kernel (the same bits): a mesh made mostly of slivers,
// or one outside the float filter's preconditions (coordinates beyond 2^28, a record that rounding to
// float made degenerate or too small, or a window wider than 2^-8).
bool fixup_runs_f64(const DeviceMesh &m) { return sliver_heavy(m) || !m.filter_ok; }


int morton_point_order(long long n, const void *x, const void *y, const void *z, int f64, const float4 *nodes32,
                       int **order, cudaStream_t stream) {
    *order = nullptr;
    if (n <= 0 || n >= 0x7fffffffll) return fail(SSDF_ERR_INVALID_ARGUMENT, "point count out of range for sorting");
    uint32_t *keys = nullptr;
    SSDF_CUDA(cudaMallocAsync(&keys, sizeof(uint32_t) * size_t(n), stream));
    cudaError_t e = cudaMallocAsync(order, sizeof(int) * size_t(n), stream);
    int st = e == cudaSuccess ? SSDF_OK : cuda_fail(e, "sort order", __FILE__, __LINE__);
    if (st == SSDF_OK) {
        k_point_keys<<<unsigned((n + 255) / 256), 256, 0, stream>>>(n, x, y, z, f64, nodes32, keys, *order);
        e = cudaGetLastError();
        st = e == cudaSuccess ? radix_sort_pairs_u32(keys, *order, int(n), 30, stream)
                              : cuda_fail(e, "point keys", __FILE__, __LINE__);
    }
    cudaFreeAsync(keys, stream);
    if (st != SSDF_OK && *order) {
        cudaFreeAsync(*order, stream);
        *order = nullptr;
    }
    return st;
}

// A captured double or float launch stays a single kernel node: a list would put an allocation into the
// caller's graph, which then cannot be a child graph or run twice at once.
static bool capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) == cudaSuccess) return status != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

int launch_query(const QueryArgs &args_in, int precision, cudaStream_t stream) {
    return launch_query_keep(args_in, precision, stream, nullptr);
}

int launch_query_keep(const QueryArgs &args_in, int precision, cudaStream_t stream, int **fallback_list) {
    if (fallback_list) *fallback_list = nullptr;
    retain_pool_memory();
    QueryArgs a = args_in;
    const long long n = a.is_grid ? a.nx * a.ny * a.nz : a.npoints;
    if (n <= 0) return SSDF_OK;
    if (precision == SSDF_PREC_F64 && !a.m.tris64)
        return fail(SSDF_ERR_INVALID_ARGUMENT, "mesh built without double data (keep_fp64=0)");
    if (precision == SSDF_PREC_F32_FIXUP && (!a.m.tris64 || !a.m.filt32))
        return fail(SSDF_ERR_INVALID_ARGUMENT, "fix-up queries need the double triangles and BVH (keep_fp64=1)");
    if (a.output == SSDF_OUT_SDF && !a.m.face_n)
        return fail(SSDF_ERR_INVALID_ARGUMENT, "signed queries need a mesh built with normals=1");
    if (a.output == SSDF_OUT_SDF && !a.m.tris64)
        return fail(SSDF_ERR_INVALID_ARGUMENT, "signed queries need the double triangles (keep_fp64=1)");
    // A mesh made mostly of ill-conditioned triangles (needles, slivers) is answered faster by the
    // plain FP64 kernel: the fix-up filter sees each such triangle through a wide proxy, whose keys
    // crowd the window. Both give the same bits.
    if (precision == SSDF_PREC_F32_FIXUP && fixup_runs_f64(a.m)) precision = SSDF_PREC_F64;
    const bool forced_budget = a.warp_budget >= 0;
    resolve_hand_over(&a, precision == SSDF_PREC_F32_FIXUP, n);
    if (a.output == SSDF_OUT_CLOSEST && (!a.m.tris64 || !a.outx || !a.outy || !a.outz || !a.outtri))
        return fail(SSDF_ERR_INVALID_ARGUMENT, "closest-point queries need outx/outy/outz/outtri and double data");
    if (precision == SSDF_PREC_F32 && (a.output == SSDF_OUT_SDF || a.output == SSDF_OUT_CLOSEST))
        return fail(SSDF_ERR_INVALID_ARGUMENT, "SSDF_PREC_F32 serves the edf and sqedf outputs");
    const bool count = env_int("SSDF_B200_COUNT", 0) != 0;
    // large point lists: visit them in Morton order, as warp packets (results are per query, so the
    // order changes nothing but the time); the order array is freed behind the launches
    struct StreamFree {  // stream-ordered free when the launch returns, on every path
        int *p;
        cudaStream_t s;
        ~StreamFree() {
            if (p) cudaFreeAsync(p, s);
        }
    } sorted{nullptr, stream};
    const bool short_list = !a.is_grid && !a.force_traversal && !env_str("SSDF_B200_TRAVERSAL") &&
                            n <= env_int("SSDF_B200_WARP_POINTS", kWarpPoints);
    if (!a.is_grid && !short_list && !a.force_traversal && n >= kSortMinPoints && n < 0x7fffffffll &&
        env_int("SSDF_B200_SORT_POINTS", 1) != 0) {
        SSDF_CHECK(morton_point_order(n, a.x, a.y, a.z, a.coord_f64, a.m.nodes32, &sorted.p, stream));
        a.order = sorted.p;
    }
    const bool warp = use_warp(a);
    const long long nblocks = query_blocks(a);
    if (nblocks > 0x7fffffffll) return fail(SSDF_ERR_NOT_SUPPORTED, "too many queries in one launch");
    unsigned long long *counters = nullptr;
    int *fb = nullptr;
    int st = SSDF_OK;
    if (count) {
        SSDF_CUDA(cudaMallocAsync(&counters, 4 * sizeof(unsigned long long), stream));
        SSDF_CUDA(cudaMemsetAsync(counters, 0, 4 * sizeof(unsigned long long), stream));
    }
    a.counters = counters;
    cudaError_t e = cudaSuccess;
    if (short_list) {
        e = precision == SSDF_PREC_F64   ? launch_query_warp<SSDF_PREC_F64>(a, count, stream)
            : precision == SSDF_PREC_F32 ? launch_query_warp<SSDF_PREC_F32>(a, count, stream)
                                         : launch_query_warp<SSDF_PREC_F32_FIXUP>(a, count, stream);
    } else {
        const bool fixup = precision == SSDF_PREC_F32_FIXUP;
        if (fixup && n >= 0x7fffffffll) {
            st = fail(SSDF_ERR_NOT_SUPPORTED, "more than 2^31 - 1 queries in one fix-up launch");
        } else if (fixup || (warp && a.warp_budget > 0 && (forced_budget || budget_reachable(a)) &&
                             n <= kHandOverMaxQueries && !capturing(stream))) {
            if (cudaMallocAsync(&fb, sizeof(int) * size_t(2 * n + 1), stream) != cudaSuccess) {
                fb = nullptr;
                if (fixup) st = fail(SSDF_ERR_OUT_OF_MEMORY, "fix-up overflow list");
                else cudaGetLastError();  // the plain arithmetics only walk on without a budget
            }
        }
        if (fb) {
            a.fallback_count = fb;
            a.fallback_ids = fb + 1;
            a.fallback_thr = reinterpret_cast<float *>(fb + 1 + n);
            e = cudaMemsetAsync(fb, 0, sizeof(int), stream);
        } else {
            a.warp_budget = 0;
        }
        if (st == SSDF_OK && e == cudaSuccess)
            e = precision == SSDF_PREC_F64   ? launch_two_stages<SSDF_PREC_F64>(a, warp, count, unsigned(nblocks), stream)
                : precision == SSDF_PREC_F32 ? launch_two_stages<SSDF_PREC_F32>(a, warp, count, unsigned(nblocks), stream)
                                             : launch_two_stages<SSDF_PREC_F32_FIXUP>(a, warp, count, unsigned(nblocks), stream);
    }
    if (e != cudaSuccess && st == SSDF_OK) st = cuda_fail(e, "query launch", __FILE__, __LINE__);
    if (count && st == SSDF_OK) {
        unsigned long long h[4] = {0, 0, 0, 0};
        int nfb = 0;
        cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, stream);
        if (fb) cudaMemcpyAsync(&nfb, fb, sizeof(int), cudaMemcpyDeviceToHost, stream);
        e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) st = cuda_fail(e, "query counters", __FILE__, __LINE__);
        h[3] = (unsigned long long)nfb;
        memcpy(t_last_counts, h, sizeof(h));
    }
    if (fb && fallback_list && st == SSDF_OK)
        *fallback_list = fb;  // [count, ids...]; the caller frees it (stream-ordered)
    else if (fb)
        cudaFreeAsync(fb, stream);
    if (counters) cudaFreeAsync(counters, stream);
    return st;
}

// Resident blocks per SM of the batch kernel for this arithmetic / traversal.
int batch_blocks_per_sm(int precision, bool warp) {
    if (precision == SSDF_PREC_F64)
        return warp ? batch_occupancy<SSDF_PREC_F64, true>() : batch_occupancy<SSDF_PREC_F64, false>();
    if (precision == SSDF_PREC_F32)
        return warp ? batch_occupancy<SSDF_PREC_F32, true>() : batch_occupancy<SSDF_PREC_F32, false>();
    return warp ? batch_occupancy<SSDF_PREC_F32_FIXUP, true>() : batch_occupancy<SSDF_PREC_F32_FIXUP, false>();
}

// Enqueues the persistent batch kernel (and the fix-up window stage) on `stream`; the job table and
// counters in `b` must already be in device memory. Capturable in a CUDA graph. Batch jobs carry no
// counter buffer (QueryArgs::counters is null), so batch launches never take the counting
// instantiations, whatever SSDF_B200_COUNT says.
int launch_batch(const BatchLaunch &b, int precision, cudaStream_t stream) {
    const bool count = false;
    cudaError_t e;
    if (precision == SSDF_PREC_F64)
        e = launch_batch_prec<SSDF_PREC_F64>(b, count, stream);
    else if (precision == SSDF_PREC_F32)
        e = launch_batch_prec<SSDF_PREC_F32>(b, count, stream);
    else
        e = launch_batch_prec<SSDF_PREC_F32_FIXUP>(b, count, stream);
    if (e != cudaSuccess) return cuda_fail(e, "batch launch", __FILE__, __LINE__);
    return SSDF_OK;
}

bool default_warp(int is_grid) {
    const char *v = env_str("SSDF_B200_TRAVERSAL");
    if (v && !strcmp(v, "warp")) return true;
    if (v && !strcmp(v, "thread")) return false;
    return is_grid != 0;
}

// ---- allocation-free variant of the fix-up grid query ------------------------------------------------
//
// For callers that cannot allocate device memory while they query (a real-time loop whose memory is
// reserved up front, an application that runs under a custom allocator and forbids the CUDA one, a
// plugin host that owns all allocations): the FP32 + FP64 fix-up query keeps its overflow list
// (count, query ids, window thresholds) in this fixed array instead of stream-ordered scratch. The
// array is part of the library image, so every GPU that loads the library holds it (8 MiB) until
// the process exits. All calls share it: each call clears the count it starts from, and two calls
// whose kernels overlap on the GPU (different streams, no ordering between them) race on it.
constexpr long long kNoAllocMaxQueries = 1ll << 20;  // queries per call
static __device__ __align__(256) int g_noalloc_scratch[2 * kNoAllocMaxQueries + 1];

static std::mutex g_noalloc_mutex;
static int *g_noalloc_ptr[256];

// Device address of g_noalloc_scratch on the current device, looked up once per device (the host
// symbol is only a stand-in for it). The address belongs to the device's context: a process that calls
// cudaDeviceReset on a device must not use the allocation-free query on that device afterwards.
static int noalloc_scratch(int **ptr) {
    int dev = 0;
    SSDF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) return fail(SSDF_ERR_NOT_SUPPORTED, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
        g_noalloc_ptr[dev] = static_cast<int *>(p);
    }
    *ptr = g_noalloc_ptr[dev];
    return SSDF_OK;
}

long long noalloc_max_queries() { return kNoAllocMaxQueries; }

// The fix-up query of `args` with its overflow list in g_noalloc_scratch: no allocation. It takes the
// same launch decisions as launch_query_keep: the packet work budget of a launch this size, and the
// FP64 kernel (which needs no scratch) for a mesh made mostly of ill-conditioned triangles.
int launch_query_noalloc(const QueryArgs &args_in, cudaStream_t stream) {
    QueryArgs a = args_in;
    const long long n = a.is_grid ? a.nx * a.ny * a.nz : a.npoints;
    if (n <= 0) return SSDF_OK;
    if (n > kNoAllocMaxQueries)
        return fail(SSDF_ERR_NOT_SUPPORTED, "the allocation-free query takes at most " +
                                                std::to_string(kNoAllocMaxQueries) + " queries per call, got " +
                                                std::to_string(n) + ": split the grid into slabs");
    if (!a.m.tris64 || !a.m.filt32)
        return fail(SSDF_ERR_INVALID_ARGUMENT, "fix-up queries need the double triangles and BVH (keep_fp64=1)");
    if (a.output == SSDF_OUT_SDF && !a.m.face_n)
        return fail(SSDF_ERR_INVALID_ARGUMENT, "signed queries need a mesh built with normals=1");
    a.counters = nullptr;
    const bool warp = use_warp(a);
    const long long nblocks = query_blocks(a);
    cudaError_t e;
    if (fixup_runs_f64(a.m)) {
        // the same bits from the double kernel, without a budget: it hands nothing over, so these calls share
        // nothing and may overlap
        a.warp_budget = 0;
        e = launch_prec<SSDF_PREC_F64>(a, warp, false, unsigned(nblocks), stream);
    } else {
        resolve_hand_over(&a, true, n);
        int *scratch = nullptr;
        SSDF_CHECK(noalloc_scratch(&scratch));
        a.fallback_count = scratch;
        a.fallback_ids = scratch + 1;
        a.fallback_thr = reinterpret_cast<float *>(scratch + 1 + n);
        e = cudaMemsetAsync(scratch, 0, sizeof(int), stream);  // the count starts at zero
        if (e == cudaSuccess)
            e = launch_two_stages<SSDF_PREC_F32_FIXUP>(a, warp, false, unsigned(nblocks), stream, kWinStack);
    }
    if (e != cudaSuccess) return cuda_fail(e, "allocation-free query launch", __FILE__, __LINE__);
    return SSDF_OK;
}

}  // namespace ssdf_b200

