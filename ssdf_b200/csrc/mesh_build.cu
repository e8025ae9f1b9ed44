// mesh_build.cu -- device-resident mesh: triangle records, LBVH, refit, pseudo-normals.
//
// Replaces the reference's per-call host packing + cuBQL build (serial/bvh/bvh.cu:108-130,
// serial/bvh/bvh.cpp:155-165) with a device pipeline that runs once per mesh:
//   1. validate indices, gather vertices, triangle boxes (FP32 and FP64), scene box of centroids;
//   2. 30-bit Morton codes of the centroids, stable radix sort (radix_sort.cu);
//   3. Karras LBVH topology over the sorted primitives (index tie-break for equal codes);
//   4. node boxes as unions of leaf ranges (k_boxes_inside, k_boxes_across);
//   5. optional SAH treelet refinement (treelet_opt.cu);
//   6. node records in the child-box layout, subtrees of <= leaf_size triangles collapsed into
//      leaves, triangle records in leaf order, oriented boxes of the same children (internal.h documents the
//      layouts);
//   7. optional angle-weighted pseudo-normals (serial/bvh/bvh.cpp:1669-1721), summed in the
//      reference's order so they are bitwise its values up to the last bit of acos.
#include <cuda_runtime.h>

#include <cfloat>
#include <cstring>
#include <vector>

#include "internal.h"

namespace ssdf_b200 {

// SAH treelet refinement (treelet_opt.cu): restructures the topology in place, refits the boxes and
// re-derives the leaf order (ids, leaf references, first_of) and the counts, so subtrees stay contiguous ranges.
int treelet_optimize(int n, int *child_l, int *child_r, int *parent_int, int *parent_leaf, int *first_of, int *count,
                     float *nbox32, double *nbox64, const float *pbox32, const double *pbox64, int *sorted_ids,
                     cudaStream_t stream);

struct MeshStorage {
    std::vector<void *> blocks;
    size_t bytes = 0;
};

namespace {

template <typename T>
int dalloc(MeshStorage *s, T **p, size_t count, cudaStream_t stream) {
    void *ptr = nullptr;
    const size_t b = sizeof(T) * (count ? count : 1);
    cudaError_t e = cudaMallocAsync(&ptr, b, stream);
    if (e != cudaSuccess) return fail(SSDF_ERR_OUT_OF_MEMORY, "device allocation of " + std::to_string(b) + " bytes");
    s->blocks.push_back(ptr);
    s->bytes += b;
    *p = reinterpret_cast<T *>(ptr);
    return SSDF_OK;
}

// Monotone float <-> int for atomicMin/atomicMax on floats.
__device__ __forceinline__ int f2o(float f) {
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

__global__ void k_validate(int nt, int nv, const int *__restrict__ s0, const int *__restrict__ s1,
                           const int *__restrict__ s2, int *__restrict__ bad) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const int a = s0[t], b = s1[t], c = s2[t];
    if (a < 0 || a >= nv || b < 0 || b >= nv || c < 0 || c >= nv) atomicMin(bad, t);
}

template <typename G>
__global__ void k_widen(int nv, const G *__restrict__ sx, const G *__restrict__ sy, const G *__restrict__ sz,
                        double *__restrict__ vx, double *__restrict__ vy, double *__restrict__ vz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    vx[i] = double(sx[i]);
    vy[i] = double(sy[i]);
    vz[i] = double(sz[i]);
}

// Per triangle: FP32 / FP64 boxes, FP32 centroid; scene centroid bounds and coordinate scale.
__global__ void k_prep(int nt, const int *__restrict__ s0, const int *__restrict__ s1, const int *__restrict__ s2,
                       const double *__restrict__ vx, const double *__restrict__ vy, const double *__restrict__ vz,
                       float *__restrict__ box32, double *__restrict__ box64, float *__restrict__ cen,
                       int *__restrict__ scene /* 6 ordered ints: lo xyz, hi xyz */, int *__restrict__ scale) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    float c[3] = {0.f, 0.f, 0.f};
    float amax = 0.f;
    const bool ok = t < nt;
    if (ok) {
        const int id[3] = {s0[t], s1[t], s2[t]};
        double p[3][3];
        for (int v = 0; v < 3; v++) p[v][0] = vx[id[v]], p[v][1] = vy[id[v]], p[v][2] = vz[id[v]];
        for (int d = 0; d < 3; d++) {
            const double lo = fmin(fmin(p[0][d], p[1][d]), p[2][d]);
            const double hi = fmax(fmax(p[0][d], p[1][d]), p[2][d]);
            box64[6 * t + 2 * d] = lo;
            box64[6 * t + 2 * d + 1] = hi;
            const float f0 = float(p[0][d]), f1 = float(p[1][d]), f2 = float(p[2][d]);
            const float flo = fminf(fminf(f0, f1), f2), fhi = fmaxf(fmaxf(f0, f1), f2);
            box32[6 * t + 2 * d] = flo;
            box32[6 * t + 2 * d + 1] = fhi;
            c[d] = 0.5f * (flo + fhi);
            cen[3 * t + d] = c[d];
            amax = fmaxf(amax, fmaxf(fabsf(flo), fabsf(fhi)));
        }
    }
    // warp-level reduction then one atomic per warp
    float lo[3], hi[3];
    for (int d = 0; d < 3; d++) lo[d] = ok ? c[d] : FLT_MAX, hi[d] = ok ? c[d] : -FLT_MAX;
    for (int o = 16; o > 0; o >>= 1) {
        for (int d = 0; d < 3; d++) {
            lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    }
    if ((threadIdx.x & 31) == 0) {
        for (int d = 0; d < 3; d++) {
            atomicMin(&scene[d], f2o(lo[d]));
            atomicMax(&scene[3 + d], f2o(hi[d]));
        }
        atomicMax(scale, __float_as_int(amax));
    }
}

__device__ __forceinline__ uint32_t expand_bits(uint32_t v) {
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

__global__ void k_morton(int nt, const float *__restrict__ cen, const int *__restrict__ scene,
                         uint32_t *__restrict__ keys, int *__restrict__ vals) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    uint32_t q[3];
    for (int d = 0; d < 3; d++) {
        const float lo = o2f(scene[d]), hi = o2f(scene[3 + d]);
        const float ext = hi - lo;
        float u = ext > 0.f ? (cen[3 * t + d] - lo) / ext : 0.5f;
        u = fminf(fmaxf(u, 0.f), 1.f);
        q[d] = uint32_t(fminf(u * 1024.f, 1023.f));
    }
    keys[t] = (expand_bits(q[0]) << 2) | (expand_bits(q[1]) << 1) | expand_bits(q[2]);
    vals[t] = t;
}

__device__ __forceinline__ int karras_delta(const uint32_t *__restrict__ k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = k[i], b = k[j];
    if (a == b) return 32 + __clz(i ^ j);
    return __clz(a ^ b);
}

// Internal node i of the n-1: children (>= 0 internal, < 0 leaf -(pos + 1)), range (first leaf, count), parents.
__global__ void k_karras(int n, const uint32_t *__restrict__ k, int *__restrict__ child_l, int *__restrict__ child_r,
                         int *__restrict__ first_of, int *__restrict__ count, int *__restrict__ parent_int,
                         int *__restrict__ parent_leaf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (karras_delta(k, n, i, i + 1) - karras_delta(k, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = karras_delta(k, n, i, i - d);
    int lmax = 2;
    while (karras_delta(k, n, i, i + lmax * d) > dmin) lmax *= 2;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (karras_delta(k, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = karras_delta(k, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (karras_delta(k, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int first = min(i, j), last = max(i, j);
    const int left = (first == gamma) ? -(gamma + 1) : gamma;
    const int right = (last == gamma + 1) ? -(gamma + 2) : gamma + 1;
    child_l[i] = left;
    child_r[i] = right;
    first_of[i] = first;
    count[i] = last - first + 1;
    if (left < 0) parent_leaf[gamma] = i; else parent_int[gamma] = i;
    if (right < 0) parent_leaf[gamma + 1] = i; else parent_int[gamma + 1] = i;
    if (i == 0) parent_int[0] = -1;
}

// Node boxes. Every box is a union of leaves' boxes, and minima and maxima come out the same in any order, so
// nothing has to climb the tree through L2 (with one thread a leaf that did, an arrival counter and a box
// load a level, the deepest path took 40 to 75 us). A block of k_boxes_inside has the subtrees inside its
// kRefitBlock leaves to itself and climbs them in shared memory (a node's index lies in its range of
// leaves); it also unites its leaves by 32 and all together. k_boxes_across gives each of the remaining nodes,
// whose leaves lie in several blocks, a warp: the leaves at the range's ends one by one, then by 32, the
// blocks between them whole. Bound by latency: three dependent loads and a union over the warp, a node at a
// time; a warp looks through kAcrossNodes nodes (131,072 triangles: 27 us with 32, 14 with 8, 19 with 2).
// Together 16 / 20 / 27 / 33 us instead of 40 / 55 / 63 / 75 at 5,120 / 41,006 / 81,920 / 131,072 triangles.
constexpr int kRefitBlock = 256, kRuns = kRefitBlock / 32, kAcrossNodes = 8;

// A box as three (min, max) pairs, 24 and 48 bytes: aligned for two-element loads.
struct Boxes {
    float2 f[3];
    double2 d[3];
};
__device__ __forceinline__ void clear_box(Boxes &b) {
#pragma unroll
    for (int k = 0; k < 3; k++) b.f[k] = make_float2(FLT_MAX, -FLT_MAX), b.d[k] = make_double2(DBL_MAX, -DBL_MAX);
}
__device__ __forceinline__ void add_pair(Boxes &b, int k, float2 x, double2 y) {
    b.f[k] = make_float2(fminf(b.f[k].x, x.x), fmaxf(b.f[k].y, x.y));
    b.d[k] = make_double2(fmin(b.d[k].x, y.x), fmax(b.d[k].y, y.y));
}
__device__ __forceinline__ void add_box(Boxes &b, const Boxes &o) {
#pragma unroll
    for (int k = 0; k < 3; k++) add_pair(b, k, o.f[k], o.d[k]);
}
__device__ __forceinline__ void add_box(Boxes &b, const float *f, const double *d, size_t i) {
#pragma unroll
    for (int k = 0; k < 3; k++)
        add_pair(b, k, __ldg(reinterpret_cast<const float2 *>(f + 6 * i) + k),
                 __ldg(reinterpret_cast<const double2 *>(d + 6 * i) + k));
}
__device__ __forceinline__ void store_box(const Boxes &b, float *f, double *d, size_t i) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        reinterpret_cast<float2 *>(f + 6 * i)[k] = b.f[k];
        reinterpret_cast<double2 *>(d + 6 * i)[k] = b.d[k];
    }
}
// Union over the warp, in every lane.
__device__ __forceinline__ void warp_union(Boxes &b) {
    constexpr unsigned kAll = 0xffffffffu;
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float2 x = make_float2(__shfl_xor_sync(kAll, b.f[k].x, o), __shfl_xor_sync(kAll, b.f[k].y, o));
            const double2 y = make_double2(__shfl_xor_sync(kAll, b.d[k].x, o), __shfl_xor_sync(kAll, b.d[k].y, o));
            add_pair(b, k, x, y);
        }
    }
}

__global__ void __launch_bounds__(kRefitBlock)
    k_boxes_inside(int n, const int *__restrict__ sorted_ids, const int *__restrict__ child_l,
                   const int *__restrict__ child_r, const int *__restrict__ parent_int,
                   const int *__restrict__ parent_leaf, const int *__restrict__ first_of,
                   const int *__restrict__ count, const float *__restrict__ pbox32,
                   const double *__restrict__ pbox64, float *__restrict__ nbox32, double *__restrict__ nbox64,
                   float *__restrict__ run32, double *__restrict__ run64, float *__restrict__ block32,
                   double *__restrict__ block64) {
    __shared__ int s_arrivals[kRefitBlock], s_left[kRefitBlock], s_right[kRefitBlock], s_parent[kRefitBlock];
    __shared__ Boxes s_leaf[kRefitBlock], s_box[kRefitBlock];
    constexpr int kElsewhere = 1 << 30;  // arrivals of a node with leaves in other blocks
    const int base = blockIdx.x * kRefitBlock, tid = threadIdx.x, p = base + tid;
    bool mine = false;  // node p has all its leaves in this block
    if (p < n - 1) {
        s_left[tid] = child_l[p], s_right[tid] = child_r[p], s_parent[tid] = parent_int[p];
        const int first = first_of[p] - base;
        mine = first >= 0 && first + count[p] <= kRefitBlock;
    }
    s_arrivals[tid] = mine ? 0 : kElsewhere;
    Boxes own, all;
    clear_box(own);
    if (p < n) add_box(own, pbox32, pbox64, sorted_ids[p]);
    s_leaf[tid] = own;
    all = own;
    warp_union(all);
    if ((tid & 31) == 0 && p < n) store_box(all, run32, run64, p >> 5);
    __syncthreads();
    int node = p < n ? parent_leaf[p] : -1, self = -p - 1;
    while (node >= 0) {
        const int at = node - base;
        if (at < 0 || at >= kRefitBlock || s_arrivals[at] >= kElsewhere) break;
        const int l = s_left[at], r = s_right[at], other = l == self ? r : l;
        __threadfence_block();
        if (atomicAdd(&s_arrivals[at], 1) == 0) break;  // the second child to arrive goes on
        __threadfence_block();
        add_box(own, other < 0 ? s_leaf[-other - 1 - base] : s_box[other - base]);
        s_box[at] = own;
        self = node;
        node = s_parent[at];
    }
    __syncthreads();
    if (mine) store_box(s_box[tid], nbox32, nbox64, p);
    __syncthreads();
    if ((tid & 31) == 0) s_box[tid >> 5] = all;
    __syncthreads();
    if (tid < 32) {
        clear_box(all);
        if (tid < kRefitBlock / 32) add_box(all, s_box[tid]);
        warp_union(all);
        if (tid == 0) store_box(all, block32, block64, blockIdx.x);
    }
}

__global__ void __launch_bounds__(128)
    k_boxes_across(int n, const int *__restrict__ sorted_ids, const int *__restrict__ first_of,
                   const int *__restrict__ count, const float *__restrict__ pbox32,
                   const double *__restrict__ pbox64, const float *__restrict__ run32,
                   const double *__restrict__ run64, const float *__restrict__ block32,
                   const double *__restrict__ block64, float *__restrict__ nbox32, double *__restrict__ nbox64) {
    // nodes a warp count apart: such nodes' indices cluster at the blocks' edges
    const int lane = threadIdx.x & 31, warps = int(gridDim.x * 4);
    const int i = lane < kAcrossNodes ? lane * warps + int(blockIdx.x * 4 + (threadIdx.x >> 5)) : n;
    int first = 0, end = 0;
    if (i < n - 1) first = first_of[i], end = first + count[i];
    unsigned todo = __ballot_sync(0xffffffffu, i < n - 1 && first / kRefitBlock != (end - 1) / kRefitBlock);
    for (; todo; todo &= todo - 1) {  // warp-uniform
        const int from = __ffs(int(todo)) - 1;
        const int f = __shfl_sync(0xffffffffu, first, from), e = __shfl_sync(0xffffffffu, end, from);
        const int b0 = (f + kRefitBlock - 1) / kRefitBlock, b1 = e / kRefitBlock;  // whole blocks [b0, b1)
        Boxes b;
        clear_box(b);
        const int r0 = (f + 31) / 32, r1 = e / 32;  // whole runs of 32 leaves [r0, r1)
        if (f + lane < r0 * 32) add_box(b, pbox32, pbox64, sorted_ids[f + lane]);
        if (r1 * 32 + lane < e) add_box(b, pbox32, pbox64, sorted_ids[r1 * 32 + lane]);
        if (r0 + lane < b0 * kRuns) add_box(b, run32, run64, r0 + lane);
        if (b1 * kRuns + lane < r1) add_box(b, run32, run64, b1 * kRuns + lane);
#pragma unroll 4
        for (int q = b0 + lane; q < b1; q += 32) add_box(b, block32, block64, q);
        warp_union(b);
        if (lane == from) store_box(b, nbox32, nbox64, i);
    }
}

// Node records. A child with <= L triangles in its subtree becomes a leaf over its range.
__global__ void k_write_nodes(int n, int L, const int *__restrict__ child_l, const int *__restrict__ child_r,
                              const int *__restrict__ first_of, const int *__restrict__ count,
                              const int *__restrict__ sorted_ids, const float *__restrict__ pbox32,
                              const float *__restrict__ nbox32, float4 *__restrict__ nodes32) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int ref[2];
    const float *b32[2];
    const int c[2] = {child_l[i], child_r[i]};
    for (int h = 0; h < 2; h++) {
        if (c[h] < 0) {
            const int pos = -c[h] - 1;
            ref[h] = leaf_ref(pos, 1);
            b32[h] = pbox32 + 6 * sorted_ids[pos];
        } else {
            ref[h] = count[c[h]] <= L ? leaf_ref(first_of[c[h]], count[c[h]]) : c[h];
            b32[h] = nbox32 + 6 * c[h];
        }
    }
    nodes32[4 * i + 0] = make_float4(b32[0][0], b32[0][1], b32[0][2], b32[0][3]);
    nodes32[4 * i + 1] = make_float4(b32[1][0], b32[1][1], b32[1][2], b32[1][3]);
    nodes32[4 * i + 2] = make_float4(b32[0][4], b32[0][5], b32[1][4], b32[1][5]);
    nodes32[4 * i + 3] = make_float4(__int_as_float(ref[0]), __int_as_float(ref[1]), 0.f, 0.f);
}

// A single root holding one leaf over all n <= L triangles (child 1 empty, inverted box).
__global__ void k_write_small_root(int n, const float *__restrict__ box32, float4 *__restrict__ nodes32) {
    float b[6] = {FLT_MAX, -FLT_MAX, FLT_MAX, -FLT_MAX, FLT_MAX, -FLT_MAX};
    for (int t = 0; t < n; t++)
        for (int k = 0; k < 6; k += 2)
            b[k] = fminf(b[k], box32[6 * t + k]), b[k + 1] = fmaxf(b[k + 1], box32[6 * t + k + 1]);
    const float inf = __int_as_float(0x7f800000);
    nodes32[0] = make_float4(b[0], b[1], b[2], b[3]);
    nodes32[1] = make_float4(inf, -inf, inf, -inf);
    nodes32[2] = make_float4(b[4], b[5], inf, -inf);
    nodes32[3] = make_float4(__int_as_float(leaf_ref(0, n)), __int_as_float(kEmptyRef), 0.f, 0.f);
}

// The flag words of the build: [0] the first bad triangle (none: INT_MAX), [1..6] the scene's box as
// ordered ints (min seeded with +FLT_MAX, max with -FLT_MAX), the rest zero.
__global__ void k_init_flags(int *__restrict__ flags) {
    const int k = threadIdx.x;
    if (k >= 16) return;
    int v = 0;
    if (k == 0) v = 0x7fffffff;
    if (k >= 1 && k <= 3) v = 0x7f7fffff;
    if (k >= 4 && k <= 6) v = int(0xff7fffffu ^ 0x7fffffffu);
    flags[k] = v;
}

// Depth and leaf count of the collapsed tree: a node is kept iff its subtree has > L triangles
// (its ancestors then have more), so walk parents from every kept node.
__global__ void k_depth(int n, int L, const int *__restrict__ count, const int *__restrict__ parent_int,
                        const int *__restrict__ child_l, const int *__restrict__ child_r, int *__restrict__ stats) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    if (i != 0 && count[i] <= L) return;
    int depth = 1;
    for (int p = parent_int[i]; p >= 0 && depth < 1 << 20; p = parent_int[p]) depth++;
    atomicMax(&stats[0], depth);
    int leaves = 0;
    const int c[2] = {child_l[i], child_r[i]};
    for (int h = 0; h < 2; h++) leaves += (c[h] < 0 || count[c[h]] <= L) ? 1 : 0;
    atomicAdd(&stats[1], leaves);
}

// Whether the float filter sees a triangle through a proxy: height below 1/8 of the longest edge.
__device__ bool ill_conditioned(double ax, double ay, double az, double bx, double by, double bz, double cx, double cy,
                                double cz) {
    const double abx = bx - ax, aby = by - ay, abz = bz - az, acx = cx - ax, acy = cy - ay, acz = cz - az;
    const double bcx = cx - bx, bcy = cy - by, bcz = cz - bz;
    const double lab = abx * abx + aby * aby + abz * abz, lac = acx * acx + acy * acy + acz * acz;
    const double lbc = bcx * bcx + bcy * bcy + bcz * bcz;
    const double l2 = fmax(fmax(lab, lac), lbc);
    const double nx = aby * acz - abz * acy, ny = abz * acx - abx * acz, nz = abx * acy - aby * acx;
    return l2 > 0.0 && !(64.0 * (nx * nx + ny * ny + nz * nz) >= l2 * l2);
}

// The fix-up path's FP32 filter record of one triangle: the triangle itself, or, when it is
// ill-conditioned (height below 1/8 of its longest edge PQ, third corner R), a proxy triangle that
// contains it: PQ widened by L/4 at both ends (L = |PQ|) and an apex L/2 off its middle, towards R in
// the triangle's plane. R projects inside PQ (PQ is the longest edge) at height below L/8, and the
// proxy is at least L/6 high over all of PQ, so it contains P, Q and R; its distance is a lower
// bound of the triangle's, and its height (1/3 of its base) keeps the float test accurate. A proxy's
// record has the sign bit of its ab.ab set: its key may enter the window but never moves its centre.
__device__ void filter_record(double ax, double ay, double az, double bx, double by, double bz, double cx,
                              double cy, double cz, bool ill, float4 *__restrict__ out) {
    const double abx = bx - ax, aby = by - ay, abz = bz - az, acx = cx - ax, acy = cy - ay, acz = cz - az;
    const double bcx = cx - bx, bcy = cy - by, bcz = cz - bz;
    const double lab = abx * abx + aby * aby + abz * abz, lac = acx * acx + acy * acy + acz * acz;
    const double lbc = bcx * bcx + bcy * bcy + bcz * bcz;
    const double l2 = fmax(fmax(lab, lac), lbc);
    double v[3][3] = {{ax, ay, az}, {bx, by, bz}, {cx, cy, cz}};
    if (ill) {
        // P, Q: the longest edge; R: the third corner
        int ip = 0, iq = 1, ir = 2;
        if (lac >= lab && lac >= lbc) ip = 0, iq = 2, ir = 1;
        else if (lbc >= lab && lbc >= lac) ip = 1, iq = 2, ir = 0;
        const double *P = v[ip], *Q = v[iq], *R = v[ir];
        const double L = sqrt(l2);
        double e[3] = {(Q[0] - P[0]) / L, (Q[1] - P[1]) / L, (Q[2] - P[2]) / L};
        const double rp[3] = {R[0] - P[0], R[1] - P[1], R[2] - P[2]};
        const double x = rp[0] * e[0] + rp[1] * e[1] + rp[2] * e[2];
        double u[3] = {rp[0] - x * e[0], rp[1] - x * e[1], rp[2] - x * e[2]};  // R's offset off PQ
        double lu = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
        if (!(lu > 1e-9 * L)) {  // collinear to rounding: any direction across PQ
            const double w[3] = {fabs(e[0]) < 0.9 ? 1.0 : 0.0, fabs(e[0]) < 0.9 ? 0.0 : 1.0, 0.0};
            u[0] = e[1] * w[2] - e[2] * w[1], u[1] = e[2] * w[0] - e[0] * w[2], u[2] = e[0] * w[1] - e[1] * w[0];
        }
        const double ue = u[0] * e[0] + u[1] * e[1] + u[2] * e[2];  // re-orthogonalised against PQ
        for (int d = 0; d < 3; d++) u[d] -= ue * e[d];
        lu = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
        for (int d = 0; d < 3; d++) u[d] /= lu;
        double pr[3][3];
        for (int d = 0; d < 3; d++) {
            pr[0][d] = P[d] - 0.25 * L * e[d];
            pr[1][d] = Q[d] + 0.25 * L * e[d];
            pr[2][d] = 0.5 * (P[d] + Q[d]) + 0.5 * L * u[d];
        }
        for (int a = 0; a < 3; a++)
            for (int d = 0; d < 3; d++) v[a][d] = pr[a][d];
    }
    // a, ab = b - a, ac = c - a and the products ab.ab, ac.ac, ab.ac, from the rounded corners (so the
    // record is the triangle the float corners describe), in double and then rounded once
    float f[3][3];
    for (int k = 0; k < 3; k++)
        for (int d = 0; d < 3; d++) f[k][d] = float(v[k][d]);
    double eb[3], ec[3];
    for (int d = 0; d < 3; d++) eb[d] = double(f[1][d]) - double(f[0][d]), ec[d] = double(f[2][d]) - double(f[0][d]);
    const double bb = eb[0] * eb[0] + eb[1] * eb[1] + eb[2] * eb[2];
    const double cc = ec[0] * ec[0] + ec[1] * ec[1] + ec[2] * ec[2];
    const double bc = eb[0] * ec[0] + eb[1] * ec[1] + eb[2] * ec[2];
    // a proxy is marked by the sign bit of ab.ab (never negative otherwise)
    const float fbb = float(bb);
    out[0] = make_float4(f[0][0], f[0][1], f[0][2], ill ? __int_as_float(__float_as_int(fbb) | 0x80000000) : fbb);
    out[1] = make_float4(float(eb[0]), float(eb[1]), float(eb[2]), float(cc));
    out[2] = make_float4(float(ec[0]), float(ec[1]), float(ec[2]), float(bc));
}

// The fix-up window's bound term of one filter record (the triangle the float corners describe, or its
// proxy): the FP32 filter's error at a query p is at most u (8 R + 7.7 alpha L) + min(D, 2 D^2 / d) with D
// = 90 u alpha R (device_geom.cuh, tri_dist_sq_filter, states the terms it bounds: input rounding, each
// fmaf, the quotient and reciprocal, the region decisions), u = 2^-24, L the record's longest edge, alpha =
// L^2 / |ab x ac| and R the largest distance from p to a corner. That is at most u (17 d + (16 + 188 alpha)
// L) at any distance d (near the record R <= 2L; far from it the D^2 term is below u d); with the input
// rounding of p and of the corners it stays below u (18.1 d + 2 sqrt(3) M) + u (20 + 188 alpha) L, M the
// largest coordinate magnitude. This returns the record's term (20 + 188 alpha) L, and false when the
// record is not safe for the float filter: an edge shorter than 2^-23 (its products underflow), a record
// that rounding to float made degenerate or needle-like (alpha > 16), or a non-finite value.
__device__ bool filter_bound(const float4 *__restrict__ rec, float *term) {
    const double e1[3] = {rec[1].x, rec[1].y, rec[1].z}, e2[3] = {rec[2].x, rec[2].y, rec[2].z};
    const double e3[3] = {e2[0] - e1[0], e2[1] - e1[1], e2[2] - e1[2]};
    const double l1 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
    const double l2 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
    const double l3 = e3[0] * e3[0] + e3[1] * e3[1] + e3[2] * e3[2];
    const double ll = fmax(fmax(l1, l2), l3);
    *term = 0.f;
    if (ll == 0.0) return true;  // all corners equal: only the corner test runs, exactly
    const double nx = e1[1] * e2[2] - e1[2] * e2[1], ny = e1[2] * e2[0] - e1[0] * e2[2];
    const double nz = e1[0] * e2[1] - e1[1] * e2[0];
    const double n = sqrt(nx * nx + ny * ny + nz * nz);
    const double shortest = fmin(fmin(l1, l2), l3);
    const double alpha = ll / n;
    if (!(shortest >= 0x1p-46) || !(alpha <= 16.0) || !(ll < 0x1p120)) return false;
    *term = __double2float_ru((20.0 + 188.0 * alpha) * sqrt(ll));
    return true;
}

}  // namespace

// The window (sqrt(best) + tau)^2 (1 + 2^-16), tau = tau_rel (M + sqrt(best)), keeps the double
// winner whenever tau exceeds the sum of its key's error above its distance and the error below of
// the key that set best. With the bound above both are at most u (18.1 d + 2 sqrt(3) M + term), so
// tau_rel >= u (6.93 + 2 term / M) and tau_rel >= 36.2 u suffice (2^-9 added for best lying below
// the winner's distance; the (1 + 2^-16) factor covers the rounding of the window itself). The
// default 2^-16 = 256 u holds them whenever term / M <= 124: the torus-knot tube's largest term is 27.7 M (a triangle of aspect 7.2),
// a 320-triangle sphere's 94 M; a mesh of a few large triangles gets a wider window. A mesh whose
// window would pass 2^-8, or with a record the float filter cannot take, is answered by the FP64
// kernel.
void set_filter_window(DeviceMesh *m, float largest_term, bool records_safe) {
    const double u = 0x1p-24, M = double(m->coord_scale);
    double tau = 1.0 / 65536.0;
    if (largest_term > 0.f) {
        if (!(M > 0.0)) {
            m->tau_rel_min = 1.0f;
            m->filter_ok = 0;
            return;
        }
        tau = fmax(tau, u * (6.93 + 2.0 * double(largest_term) / M) * (1.0 + 0x1p-9));
    }
    m->tau_rel_min = float(tau) < tau ? nextafterf(float(tau), INFINITY) : float(tau);
    // (a safe record that is not one point has M >= 2^-25; a mesh of points nearer the origin, or at it, would have a
    // window whose square is 0, which holds nothing)
    m->filter_ok = records_safe && M >= 0x1p-26 && M <= double(kFilterMaxCoord) && tau <= 0x1p-8 ? 1 : 0;
}

namespace {

// Middle and scale of the mesh's box (the union of the nbox boxes box64), and M in that frame: w[0..2] the
// middle and w[6] M as floats, w[4..5] the scale as a double. The scale is 1 for a half size of 2^-26 to 2^28, which
// holds every mesh that the float filter takes (its records have the frame's middle but no scale), and else
// brings the half size into [8, 16): k_obb's fourth powers of lengths and the walks' squared distances then stay
// in float's range. A mesh with a coordinate that is not finite in float gets M < 0: its boxes cull nothing. And the
// nodes a warp-wide walk starts from (DeviceMesh::entry): the root, each node whose children are both nodes
// replaced by them, five times over. One warp.
__global__ void k_box_frame(const float4 *__restrict__ nodes, const double *__restrict__ box64, int nbox,
                            int *__restrict__ w, int *__restrict__ entry) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x;
    if (lane == 0) {
        double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
        for (int i = 0; i < nbox; i++)
            for (int d = 0; d < 3; d++)
                lo[d] = fmin(lo[d], box64[6 * i + 2 * d]), hi[d] = fmax(hi[d], box64[6 * i + 2 * d + 1]);
        float mid[3];
        double m = 0.0;
        bool ok = true;
        for (int d = 0; d < 3; d++) {
            ok = ok && lo[d] <= hi[d] && lo[d] >= -double(FLT_MAX) && hi[d] <= double(FLT_MAX);
            mid[d] = ok ? float(0.5 * lo[d] + 0.5 * hi[d]) : 0.f;
            m = fmax(m, fmax(hi[d] - mid[d], mid[d] - lo[d]));
        }
        double scale = 1.0;
        if (ok && m > 0.0 && !(m >= 0x1p-26 && m <= 0x1p28)) {
            int e = ilogb(m) - 3;
            e = e < -450 ? -450 : e;
            scale = ldexp(1.0, -e);
        }
        for (int d = 0; d < 3; d++) w[d] = ok ? __float_as_int(mid[d]) : 0;
        w[4] = __double2loint(scale);
        w[5] = __double2hiint(scale);
        w[6] = __float_as_int(ok ? __double2float_ru(m * scale) : -1.f);
    }
    int n = 1, node = 0;  // lanes 0 .. n - 1 hold a node each
    for (int round = 0; round < 5; round++) {
        int r0 = -1, r1 = -1;
        if (lane < n) {
            const float4 r = nodes[4 * size_t(node) + 3];
            r0 = __float_as_int(r.x), r1 = __float_as_int(r.y);
        }
        const bool open = r0 >= 0 && r1 >= 0;
        const unsigned m = __ballot_sync(kAll, open);
        const int at = lane < n ? lane + __popc(m & ((1u << lane) - 1u)) : 0;  // at most 2 n <= 32 of them
        if (lane < n) {
            entry[1 + at] = open ? r0 : node;
            if (open) entry[2 + at] = r1;
        }
        n += __popc(m);
        __syncwarp();
        node = lane < n ? entry[1 + lane] : 0;
        __syncwarp();
    }
    if (lane == 0) {
        entry[0] = n;
        if (n == 1) entry[1] = node;
    }
}

__global__ void k_tri_records(int nt, const int *__restrict__ sorted_ids, const int *__restrict__ s0,
                              const int *__restrict__ s1, const int *__restrict__ s2, const double *__restrict__ vx,
                              const double *__restrict__ vy, const double *__restrict__ vz, float4 *__restrict__ t32,
                              double2 *__restrict__ t64, float4 *__restrict__ filt, const int *__restrict__ frame,
                              int *__restrict__ nill) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nt) return;
    const int t = sorted_ids[p];
    const int a = s0[t], b = s1[t], c = s2[t];
    const double ax = vx[a], ay = vy[a], az = vz[a], bx = vx[b], by = vy[b], bz = vz[b];
    const double cx = vx[c], cy = vy[c], cz = vz[c];
    t32[3 * p + 0] = make_float4(float(ax), float(ay), float(az), float(bx));
    t32[3 * p + 1] = make_float4(float(by), float(bz), float(cx), float(cy));
    t32[3 * p + 2] = make_float4(float(cz), __int_as_float(t), 0.f, 0.f);
    if (filt) {
        // the record is taken relative to the mesh's middle, where its corners round least; whether the
        // filter serves the mesh, and its window's width, are judged at the mesh's place too (the larger
        // bound term, both records safe)
        const bool ill = ill_conditioned(ax, ay, az, bx, by, bz, cx, cy, cz);
        if (ill) atomicAdd(nill, 1);
        float4 placed[3];
        float term, term_mid;
        filter_record(ax, ay, az, bx, by, bz, cx, cy, cz, ill, placed);
        const double mx = __int_as_float(frame[0]), my = __int_as_float(frame[1]), mz = __int_as_float(frame[2]);
        filter_record(ax - mx, ay - my, az - mz, bx - mx, by - my, bz - mz, cx - mx, cy - my, cz - mz, ill,
                      filt + 3 * size_t(p));
        const bool safe = filter_bound(placed, &term) && filter_bound(filt + 3 * size_t(p), &term_mid);
        if (safe)
            atomicMax(nill + 1, __float_as_int(fmaxf(term, term_mid)));  // non-negative floats order like their bits
        else
            atomicAdd(nill + 2, 1);
    }
    if (t64) {
        t64[5 * p + 0] = make_double2(ax, ay);
        t64[5 * p + 1] = make_double2(az, bx);
        t64[5 * p + 2] = make_double2(by, bz);
        t64[5 * p + 3] = make_double2(cx, cy);
        t64[5 * p + 4] = make_double2(cz, double(t));
    }
}

// ---- oriented boxes --------------------------------------------------------------------------------
//
// The boxes the query kernels walk (DeviceMesh::obb). On a curved surface an axis-aligned box sticks out
// of the surface by its triangles' tilt, and a query far from small triangles then wants every leaf of a
// wide patch; a box along the patch does not. Per 32-query packet of the torus-knot 256^3 grid
// (131,072 triangles) the walk meets 52 triangle iterations and 79 nodes instead of 187 and 133, on the
// lattice of thin beams 23 and 164 instead of 166 and 225.
//
// Box frame: points are taken as (p - box_c) * box_scale, box_c the middle of the mesh's box (a float,
// so p - box_c has one rounding) and box_scale a power of two (k_box_frame). M below is the
// largest coordinate in that frame, u = 2^-24, d the distance from a query to a point q of the child.
// Why the float box distance is a lower bound of d:
// - With R the matrix of the three float axes, each axis' excess |axis.(p - centre)| - h is at most
//   |axis.(p - q)|, so the box distance is at most |R (p - q)| <= (1 + 20 u) d (axes unit and orthogonal within 2^-20).
// - Roundings of a coordinate along an axis: the vertices (float records against double ones, 1.8 u M),
//   their offsets from the first vertex (3.5 u M), the dot products (10.4 u M), middle and half extent
//   (7 u M), the centre's coordinate (10.4 u M), the query's (10.4 u M + 3 u d), its point (1.8 u M + u d):
//   45 u M + 4 u d. Half extents are stored 64 u M = 2^-18 M larger, and everything scaled by 1 - 64 u, which
//   covers the relative terms (at most 62 u of the squared distance).
// - The float arithmetic (SSDF_PREC_F32) compares distances that may lie below the true ones: its
//   region tests, on dot products within 11 u of their lengths, put the closest point at most D = 90 u
//   alpha R off the triangle (alpha = longest edge / smallest altitude, R <= d + L the distance to the
//   farthest corner, L the longest edge), in its plane. So half extents are also stored 128 u alpha L
//   larger and everything scaled by 1 / (1 + 128 u alpha), alpha and L over the child's triangles. (The closest
//   point's own rounding and the float corners' are of the mesh's place, not of M: box_margin.h.) A child
//   with alpha above kObbMaxAlpha keeps its axis-aligned box, as does one of more than kObbMaxTris
//   triangles (its patch is no longer flat; building it would read every triangle at every level).
constexpr int kObbMaxTris = 64;
constexpr float kObbMaxAlpha = 2048.f;

struct Vec3 {
    float x, y, z;
};
__device__ __forceinline__ Vec3 vsub(Vec3 a, Vec3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ float vdot(Vec3 a, Vec3 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }
__device__ __forceinline__ Vec3 vcross(Vec3 a, Vec3 b) {
    return {fmaf(a.y, b.z, -a.z * b.y), fmaf(a.z, b.x, -a.x * b.z), fmaf(a.x, b.y, -a.y * b.x)};
}

// Corners of the triangle at leaf position p in the box frame.
__device__ __forceinline__ void frame_corners(const float4 *__restrict__ t32, const double2 *__restrict__ t64, int p,
                                              const float (&mid)[3], double s, Vec3 (&v)[3]) {
    if (t64) {
        const double2 *r = t64 + 5 * size_t(p);
        const double2 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2), d = __ldg(r + 3);
        const double e = __ldg(&r[4].x), mx = mid[0], my = mid[1], mz = mid[2];
        v[0] = {float((a.x - mx) * s), float((a.y - my) * s), float((b.x - mz) * s)};
        v[1] = {float((b.y - mx) * s), float((c.x - my) * s), float((c.y - mz) * s)};
        v[2] = {float((d.x - mx) * s), float((d.y - my) * s), float((e - mz) * s)};
    } else {
        const float4 a = __ldg(t32 + 3 * p), b = __ldg(t32 + 3 * p + 1);
        const float e = __ldg(&t32[3 * p + 2].x), scale = float(s);  // beyond float's range: no query walks the boxes
        v[0] = {(a.x - mid[0]) * scale, (a.y - mid[1]) * scale, (a.z - mid[2]) * scale};
        v[1] = {(a.w - mid[0]) * scale, (b.x - mid[1]) * scale, (b.y - mid[2]) * scale};
        v[2] = {(b.z - mid[0]) * scale, (b.w - mid[1]) * scale, (e - mid[2]) * scale};
    }
}

// A warp per child of a node: each lane takes a candidate frame -- the box frame's axes, a normal of one of
// up to seven of the child's triangles with one of its edges, or the sum of the triangles' normals with an
// edge -- and projects every corner on it; the frame of least half surface area wins (the summed normal
// often does: with triangle normals alone the torus knot keeps 75 triangle iterations a packet, not 52).
// Bound by issue: 45 operations a triangle and candidate. The corners are taken into the box frame once, a
// triangle a lane, and shared from there: with every lane converting every triangle's doubles the FP64
// conversions bound it (41,006 / 131,072 triangles: 68 -> 43 us, 186 -> 126).
__global__ void __launch_bounds__(128) k_obb(int nnodes, int L, const int *__restrict__ count,
                                             const int *__restrict__ first_of, const double *__restrict__ pbox64,
                                             const double *__restrict__ nbox64, const int *__restrict__ sorted_ids,
                                             const float4 *__restrict__ nodes, const float4 *__restrict__ t32,
                                             const double2 *__restrict__ t64, const int *__restrict__ frame,
                                             float *__restrict__ obb) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ float4 s_corners[4][3 * kObbMaxTris];  // a warp's child: v0 v1.x, v1.yz v2.xy, v2.z
    float4 *const corners = s_corners[threadIdx.x >> 5];
    auto shared_corners = [&](int t, Vec3(&v)[3]) {
        const float4 a = corners[3 * t], b = corners[3 * t + 1];
        v[0] = {a.x, a.y, a.z}, v[1] = {a.w, b.x, b.y}, v[2] = {b.z, b.w, corners[3 * t + 2].x};
    };
    const long long w = (blockIdx.x * 128ll + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int i = int(w >> 1), h = int(w & 1);
    if (i >= nnodes) return;
    if (i != 0 && (!count || count[i] <= L)) return;  // not a node of the walked tree (one leaf: the root alone is)
    const float4 r4 = nodes[4 * size_t(i) + 3];
    const int ref = __float_as_int(h ? r4.y : r4.x);
    const float mid[3] = {__int_as_float(frame[0]), __int_as_float(frame[1]), __int_as_float(frame[2])};
    const double scale = __hiloint2double(frame[5], frame[4]);
    const float M = __int_as_float(frame[6]);
    // child's axes, -centre coordinates and half extents (a box that culls nothing)
    Vec3 ax[3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
    const float inf = __int_as_float(0x7f800000);
    float off[3] = {0.f, 0.f, 0.f}, half[3] = {inf, inf, inf};
    int writer = 0;
    if (ref != kEmptyRef && M >= 0.f) {
        const bool leaf = ref < 0;
        const int n = leaf ? leaf_count(ref) : count[ref], first = leaf ? leaf_first(ref) : first_of[ref];
        const float margin = 0x1p-18f * M;
        // normals' sum, and the float arithmetic's terms over the child's triangles
        float grow = 0.f, alpha = 0.f;
        Vec3 ns{0.f, 0.f, 0.f};
        const bool small = n <= kObbMaxTris;
        if (small) {
            for (int t = lane; t < n; t += 32) {
                Vec3 v[3];
                frame_corners(t32, t64, first + t, mid, scale, v);
                corners[3 * t] = make_float4(v[0].x, v[0].y, v[0].z, v[1].x);
                corners[3 * t + 1] = make_float4(v[1].y, v[1].z, v[2].x, v[2].y);
                corners[3 * t + 2].x = v[2].z;
                const Vec3 e1 = vsub(v[1], v[0]), e2 = vsub(v[2], v[0]), e3 = vsub(v[2], v[1]);
                const Vec3 c = vcross(e1, e2);
                const float l2 = fmaxf(vdot(e1, e1), fmaxf(vdot(e2, e2), vdot(e3, e3)));
                // all corners equal: no region test can err
                const float al = l2 == 0.f ? 0.f : l2 / sqrtf(vdot(c, c));
                alpha = al <= kObbMaxAlpha ? fmaxf(alpha, al) : FLT_MAX;  // a NaN or an overflow: too thin
                grow = fmaxf(grow, al * sqrtf(l2));
                ns = {ns.x + c.x, ns.y + c.y, ns.z + c.z};
            }
            for (int o = 16; o > 0; o >>= 1) {
                alpha = fmaxf(alpha, __shfl_xor_sync(kAll, alpha, o));
                grow = fmaxf(grow, __shfl_xor_sync(kAll, grow, o));
                ns.x += __shfl_xor_sync(kAll, ns.x, o);
                ns.y += __shfl_xor_sync(kAll, ns.y, o);
                ns.z += __shfl_xor_sync(kAll, ns.z, o);
            }
            __syncwarp();
        }
        if (small && alpha <= kObbMaxAlpha) {
            // this lane's frame
            const int nsample = n < 7 ? n : 7;
            const bool summed = lane >= 22 && lane < 31;
            const int j = summed ? (lane - 22) / 3 : (lane - 1) / 3, e = summed ? (lane - 22) % 3 : (lane + 2) % 3;
            bool ok = lane == 0;
            ax[0] = {1.f, 0.f, 0.f}, ax[1] = {0.f, 1.f, 0.f}, ax[2] = {0.f, 0.f, 1.f};
            if (lane > 0 && lane < 31 && j < nsample) {
                Vec3 v[3];
                shared_corners((j * n) / nsample, v);
                const Vec3 edge = e == 0 ? vsub(v[1], v[0]) : (e == 1 ? vsub(v[2], v[0]) : vsub(v[2], v[1]));
                Vec3 c = summed ? ns : vcross(vsub(v[1], v[0]), vsub(v[2], v[0]));
                const float rc = rsqrtf(vdot(c, c));
                c = {c.x * rc, c.y * rc, c.z * rc};
                const float along = vdot(edge, c);
                Vec3 d{fmaf(-along, c.x, edge.x), fmaf(-along, c.y, edge.y), fmaf(-along, c.z, edge.z)};
                float rd = rsqrtf(vdot(d, d));
                d = {d.x * rd, d.y * rd, d.z * rd};
                const float again = vdot(d, c);  // orthogonal to rounding
                d = {fmaf(-again, c.x, d.x), fmaf(-again, c.y, d.y), fmaf(-again, c.z, d.z)};
                rd = rsqrtf(vdot(d, d));
                d = {d.x * rd, d.y * rd, d.z * rd};
                const Vec3 f = vcross(c, d);
                // unit and orthogonal within 2^-20 (a NaN is not)
                ok = fabsf(vdot(c, c) - 1.f) < 0x1p-20f && fabsf(vdot(d, d) - 1.f) < 0x1p-20f &&
                     fabsf(vdot(c, d)) < 0x1p-20f && fabsf(vdot(f, f) - 1.f) < 0x1p-20f;
                if (ok) ax[0] = d, ax[1] = f, ax[2] = c;
            }
            Vec3 o[3];
            shared_corners(0, o);
            float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
            for (int t = 0; t < n; t++) {
                Vec3 v[3];
                shared_corners(t, v);
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const Vec3 q = vsub(v[k], o[0]);
#pragma unroll
                    for (int a = 0; a < 3; a++) {
                        const float x = vdot(ax[a], q);
                        lo[a] = fminf(lo[a], x), hi[a] = fmaxf(hi[a], x);
                    }
                }
            }
            const float pad = margin + 128.f * 0x1p-24f * grow * 1.001f;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                half[a] = 0.5f * (hi[a] - lo[a]) + pad;
                off[a] = -(vdot(ax[a], o[0]) + 0.5f * (lo[a] + hi[a]));
            }
            const float area = half[0] * half[1] + half[1] * half[2] + half[2] * half[0];
            const unsigned key = ok && area < FLT_MAX ? __float_as_uint(area) : 0x7f800000u;
            const unsigned least = __reduce_min_sync(kAll, key);
            writer = __ffs(__ballot_sync(kAll, key == least)) - 1;
            // lane 0's frame is always a candidate; all keys infinite (an overflow): keep its box
            const float s = (1.f - 0x1p-18f) / (1.f + 128.f * 0x1p-24f * alpha);
#pragma unroll
            for (int a = 0; a < 3; a++) {
                ax[a] = {ax[a].x * s, ax[a].y * s, ax[a].z * s};
                off[a] *= s;
                // an extent the margins cannot bound (an overflow) culls nothing
                half[a] = half[a] < FLT_MAX ? half[a] * s : inf;
            }
        } else {
            // the axis-aligned box of the double corners
            const double *b = leaf && n == 1 ? pbox64 + 6 * size_t(sorted_ids[first])
                                             : (leaf ? nullptr : nbox64 + 6 * size_t(ref));
            double e[6];
            if (b) {
                for (int k = 0; k < 6; k++) e[k] = b[k];
            } else {  // a leaf of several triangles: the union of their boxes
                for (int k = 0; k < 6; k++) e[k] = (k & 1) ? -DBL_MAX : DBL_MAX;
                for (int t = 0; t < n; t++) {
                    const double *q = pbox64 + 6 * size_t(sorted_ids[first + t]);
                    for (int k = 0; k < 6; k += 2) e[k] = fmin(e[k], q[k]), e[k + 1] = fmax(e[k + 1], q[k + 1]);
                }
            }
            const float s = 1.f - 0x1p-18f;
            ax[0] = {s, 0.f, 0.f}, ax[1] = {0.f, s, 0.f}, ax[2] = {0.f, 0.f, s};
            for (int a = 0; a < 3; a++) {
                const float lo = float((e[2 * a] - double(mid[a])) * scale);
                const float hi = float((e[2 * a + 1] - double(mid[a])) * scale);
                half[a] = (0.5f * (hi - lo) + margin) * s;
                off[a] = -0.5f * (lo + hi) * s;
            }
        }
    }
    if (ref == kEmptyRef) {  // never entered, and the farther child
        off[0] = 0x1p60f;
        half[0] = half[1] = half[2] = 0.f;
    }
    if (lane != writer) return;
    float *o = obb + 32 * size_t(i) + h;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        o[8 * a] = ax[a].x, o[8 * a + 2] = ax[a].y, o[8 * a + 4] = ax[a].z, o[8 * a + 6] = off[a];
        o[24 + 2 * a] = half[a];
    }
    o[30] = __int_as_float(ref);
}

// ---- pseudo-normals --------------------------------------------------------------------------------

// Face normals, the per-(face, corner) angle contributions in visit order 3t + v, the vertex and
// edge sort keys; edge normals initialised to the face's own (serial/bvh/bvh.cpp:1681-1710).
__global__ void k_face_normals(int nt, int nv, const int *__restrict__ s0, const int *__restrict__ s1,
                               const int *__restrict__ s2, const double *__restrict__ vx,
                               const double *__restrict__ vy, const double *__restrict__ vz,
                               double *__restrict__ face_n, double *__restrict__ edge_n, double *__restrict__ contrib,
                               uint32_t *__restrict__ vkey, int *__restrict__ vval, uint64_t *__restrict__ ekey,
                               int *__restrict__ eval) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const int id[3] = {s0[t], s1[t], s2[t]};
    double p[3][3];
    for (int v = 0; v < 3; v++) p[v][0] = vx[id[v]], p[v][1] = vy[id[v]], p[v][2] = vz[id[v]];
    const double u[3] = {p[1][0] - p[0][0], p[1][1] - p[0][1], p[1][2] - p[0][2]};
    const double w[3] = {p[2][0] - p[0][0], p[2][1] - p[0][1], p[2][2] - p[0][2]};
    double n[3] = {u[1] * w[2] - u[2] * w[1], u[2] * w[0] - u[0] * w[2], u[0] * w[1] - u[1] * w[0]};
    const double len = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    if (len > 0) {
        for (int d = 0; d < 3; d++) n[d] /= len;
    }
    for (int d = 0; d < 3; d++) face_n[3 * t + d] = n[d];
    for (int v = 0; v < 3; v++) {
        const double *a = p[v], *b = p[(v + 1) % 3], *c = p[(v + 2) % 3];
        const double e1[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]};
        const double e2[3] = {c[0] - a[0], c[1] - a[1], c[2] - a[2]};
        const double l1 = sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
        const double l2 = sqrt(e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2]);
        const double cosine = (l1 > 0 && l2 > 0) ? (e1[0] * e2[0] + e1[1] * e2[1] + e1[2] * e2[2]) / (l1 * l2) : 1.0;
        const double mn = (cosine < 1.0) ? cosine : 1.0;
        const double cl = (-1.0 < mn) ? mn : -1.0;
        const double angle = acos(cl);
        for (int d = 0; d < 3; d++) contrib[3 * (3 * t + v) + d] = angle * n[d];
        vkey[3 * t + v] = uint32_t(id[v]);
        vval[3 * t + v] = 3 * t + v;
    }
    for (int e = 0; e < 3; e++) {
        for (int d = 0; d < 3; d++) edge_n[9 * t + 3 * e + d] = n[d];
        const uint64_t a = uint64_t(id[e]), b = uint64_t(id[(e + 1) % 3]);
        ekey[3 * t + e] = (a < b ? a : b) * uint64_t(nv) + (a < b ? b : a);
        eval[3 * t + e] = 3 * t + e;
    }
}

// One thread per run of equal vertex keys: sums the contributions in visit order.
__global__ void k_vertex_sums(int nocc, const uint32_t *__restrict__ vkey, const int *__restrict__ vval,
                              const double *__restrict__ contrib, double *__restrict__ vertex_n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nocc) return;
    if (i > 0 && vkey[i - 1] == vkey[i]) return;
    double acc[3] = {0.0, 0.0, 0.0};
    int j = i;
    for (; j < nocc && vkey[j] == vkey[i]; j++) {
        const int o = vval[j];
        for (int d = 0; d < 3; d++) acc[d] += contrib[3 * o + d];
    }
    for (int d = 0; d < 3; d++) vertex_n[3 * size_t(vkey[i]) + d] = acc[d];
}

// One thread per run of equal edge keys: replays the reference's first-occurrence map.
__global__ void k_edge_sums(int nocc, const uint64_t *__restrict__ ekey, const int *__restrict__ eval,
                            const double *__restrict__ face_n, double *__restrict__ edge_n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nocc) return;
    if (i > 0 && ekey[i - 1] == ekey[i]) return;
    const int first = eval[i];
    int j = i + 1;
    for (; j < nocc && ekey[j] == ekey[i]; j++) {
        const int o = eval[j];
        for (int d = 0; d < 3; d++) {
            const double sum = face_n[3 * (first / 3) + d] + face_n[3 * (o / 3) + d];
            edge_n[9 * (o / 3) + 3 * (o % 3) + d] = sum;
            edge_n[9 * (first / 3) + 3 * (first % 3) + d] = sum;
        }
    }
}

int bits_for(uint64_t maxval) {
    int b = 1;
    while (b < 64 && (maxval >> b) != 0) b++;
    return b;
}

#define LAUNCH_CHECK(what)                                                  \
    do {                                                                    \
        cudaError_t e_ = cudaGetLastError();                                \
        if (e_ != cudaSuccess) return cuda_fail(e_, what, __FILE__, __LINE__); \
    } while (0)

int build_normals(MeshStorage *s, DeviceMesh *m, const int *s0, const int *s1, const int *s2, const double *vx,
                  const double *vy, const double *vz, cudaStream_t stream) {
    const int nt = m->nt, nv = m->nv, nocc = 3 * nt;
    double *face_n, *edge_n, *vertex_n;
    SSDF_CHECK(dalloc(s, &face_n, 3 * size_t(nt), stream));
    SSDF_CHECK(dalloc(s, &edge_n, 9 * size_t(nt), stream));
    SSDF_CHECK(dalloc(s, &vertex_n, 3 * size_t(nv), stream));
    MeshStorage tmp;
    double *contrib;
    uint32_t *vkey;
    uint64_t *ekey;
    int *vval, *eval;
    int st = SSDF_OK;
    if ((st = dalloc(&tmp, &contrib, 3 * size_t(nocc), stream)) == SSDF_OK &&
        (st = dalloc(&tmp, &vkey, nocc, stream)) == SSDF_OK && (st = dalloc(&tmp, &vval, nocc, stream)) == SSDF_OK &&
        (st = dalloc(&tmp, &ekey, nocc, stream)) == SSDF_OK && (st = dalloc(&tmp, &eval, nocc, stream)) == SSDF_OK) {
        cudaMemsetAsync(vertex_n, 0, sizeof(double) * 3 * size_t(nv), stream);
        k_face_normals<<<grid_blocks(nt, 128), 128, 0, stream>>>(nt, nv, s0, s1, s2, vx, vy, vz, face_n, edge_n,
                                                                 contrib, vkey, vval, ekey, eval);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) st = cuda_fail(e, "k_face_normals", __FILE__, __LINE__);
        if (st == SSDF_OK) st = radix_sort_pairs_u32(vkey, vval, nocc, bits_for(uint64_t(nv)), stream);
        if (st == SSDF_OK)
            st = radix_sort_pairs_u64(ekey, eval, nocc, bits_for(uint64_t(nv) * uint64_t(nv)), stream);
        if (st == SSDF_OK) {
            k_vertex_sums<<<grid_blocks(nocc, 256), 256, 0, stream>>>(nocc, vkey, vval, contrib, vertex_n);
            k_edge_sums<<<grid_blocks(nocc, 256), 256, 0, stream>>>(nocc, ekey, eval, face_n, edge_n);
            e = cudaGetLastError();
            if (e != cudaSuccess) st = cuda_fail(e, "normal sums", __FILE__, __LINE__);
        }
    }
    for (void *p : tmp.blocks) cudaFreeAsync(p, stream);
    m->face_n = face_n;
    m->edge_n = edge_n;
    m->vertex_n = vertex_n;
    return st;
}

}  // namespace

// The storage comes from the stream-ordered pool (cudaMallocAsync): cudaFree on it does not wait for
// work that still reads it, so the caller has ensured that none does (ssdf_mesh_destroy waits for the
// device) -- or frees it in stream order behind that work with mesh_free_async.
void mesh_free(MeshStorage *storage) {
    if (!storage) return;
    for (void *p : storage->blocks) cudaFree(p);
    delete storage;
}

void mesh_free_async(MeshStorage *storage, cudaStream_t stream) {
    if (!storage) return;
    for (void *p : storage->blocks) cudaFreeAsync(p, stream);
    delete storage;
}

size_t mesh_bytes(const MeshStorage *storage) { return storage ? storage->bytes : 0; }

// Page-locked words for the build's read-backs (one set per calling thread, kept until exit), so the
// copies stay asynchronous and the build waits once, at its end.
constexpr int kReadbackWords = 64;
static int readback_words(int **out) {
    static thread_local int *w = nullptr;
    if (!w) SSDF_CUDA(cudaHostAlloc((void **)&w, sizeof(int) * kReadbackWords, cudaHostAllocPortable));
    *out = w;
    return SSDF_OK;
}

static int mesh_build_impl(MeshStorage *s, MeshStorage *tmp, DeviceMesh *m, int nt, const int *s0_in,
                           const int *s1_in, const int *s2_in, int nv, const void *sx, const void *sy, const void *sz,
                           int coord_f64, int device_ptrs, const ssdf_build_opts &opts, bool query_boxes,
                           bool check_indices, cudaStream_t stream) {
    const int L = opts.leaf_size > 0 ? opts.leaf_size : 4;
    m->nt = nt;
    m->nv = nv;
    m->leaf_size = L;
    // indices (kept: the sign step needs the caller's vertex ids)
    int *s0, *s1, *s2;
    SSDF_CHECK(dalloc(s, &s0, nt, stream));
    SSDF_CHECK(dalloc(s, &s1, nt, stream));
    SSDF_CHECK(dalloc(s, &s2, nt, stream));
    const cudaMemcpyKind kind = device_ptrs ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    SSDF_CUDA(cudaMemcpyAsync(s0, s0_in, sizeof(int) * size_t(nt), kind, stream));
    SSDF_CUDA(cudaMemcpyAsync(s1, s1_in, sizeof(int) * size_t(nt), kind, stream));
    SSDF_CUDA(cudaMemcpyAsync(s2, s2_in, sizeof(int) * size_t(nt), kind, stream));
    m->s0 = s0, m->s1 = s1, m->s2 = s2;
    // vertices, widened to double
    const size_t gsz = coord_f64 ? sizeof(double) : sizeof(float);
    void *gx, *gy, *gz;
    double *vx, *vy, *vz;
    SSDF_CHECK(dalloc(tmp, &vx, nv, stream));
    SSDF_CHECK(dalloc(tmp, &vy, nv, stream));
    SSDF_CHECK(dalloc(tmp, &vz, nv, stream));
    if (device_ptrs) {
        gx = const_cast<void *>(sx), gy = const_cast<void *>(sy), gz = const_cast<void *>(sz);
    } else {
        char *g;
        SSDF_CHECK(dalloc(tmp, &g, 3 * gsz * size_t(nv), stream));
        gx = g, gy = g + gsz * nv, gz = g + 2 * gsz * nv;
        SSDF_CUDA(cudaMemcpyAsync(gx, sx, gsz * nv, cudaMemcpyHostToDevice, stream));
        SSDF_CUDA(cudaMemcpyAsync(gy, sy, gsz * nv, cudaMemcpyHostToDevice, stream));
        SSDF_CUDA(cudaMemcpyAsync(gz, sz, gsz * nv, cudaMemcpyHostToDevice, stream));
    }
    if (coord_f64)
        k_widen<double><<<grid_blocks(nv, 256), 256, 0, stream>>>(nv, (const double *)gx, (const double *)gy,
                                                                  (const double *)gz, vx, vy, vz);
    else
        k_widen<float><<<grid_blocks(nv, 256), 256, 0, stream>>>(nv, (const float *)gx, (const float *)gy,
                                                                 (const float *)gz, vx, vy, vz);
    LAUNCH_CHECK("k_widen");
    // validation + per-triangle boxes
    // [0] first bad triangle, [1..6] scene, [7] scale, [8..9] depth / leaves, [10] ill, [11] largest
    // filter bound term (float bits), [12] records unsafe for the float filter, [16..22] the box frame
    int *flags;
    SSDF_CHECK(dalloc(tmp, &flags, 24, stream));
    k_init_flags<<<1, 32, 0, stream>>>(flags);
    LAUNCH_CHECK("k_init_flags");
    if (device_ptrs && check_indices) {
        // host arrays were checked on the host (check_mesh_host); device arrays are checked here,
        // before any kernel indexes the vertices with them
        k_validate<<<grid_blocks(nt, 256), 256, 0, stream>>>(nt, nv, s0, s1, s2, flags);
        LAUNCH_CHECK("k_validate");
        int bad = 0;
        SSDF_CUDA(cudaMemcpyAsync(&bad, flags, sizeof(int), cudaMemcpyDeviceToHost, stream));
        SSDF_CUDA(cudaStreamSynchronize(stream));
        if (bad != 0x7fffffff)
            return fail(SSDF_ERR_INVALID_ARGUMENT, "triangle " + std::to_string(bad) +
                                                       " has a vertex index outside [0, " + std::to_string(nv) + ")");
    }
    float *box32, *cen;
    double *box64;
    SSDF_CHECK(dalloc(tmp, &box32, 6 * size_t(nt), stream));
    SSDF_CHECK(dalloc(tmp, &box64, 6 * size_t(nt), stream));
    SSDF_CHECK(dalloc(tmp, &cen, 3 * size_t(nt), stream));
    k_prep<<<grid_blocks(nt, 256), 256, 0, stream>>>(nt, s0, s1, s2, vx, vy, vz, box32, box64, cen, flags + 1,
                                                     flags + 7);
    LAUNCH_CHECK("k_prep");
    // Morton order
    uint32_t *keys;
    int *ids;
    SSDF_CHECK(dalloc(tmp, &keys, nt, stream));
    SSDF_CHECK(dalloc(tmp, &ids, nt, stream));
    k_morton<<<grid_blocks(nt, 256), 256, 0, stream>>>(nt, cen, flags + 1, keys, ids);
    LAUNCH_CHECK("k_morton");
    SSDF_CHECK(radix_sort_pairs_u32(keys, ids, nt, 30, stream));
    // topology
    const bool keep64 = opts.keep_fp64 != 0;
    const int nint = nt > 1 ? nt - 1 : 0;
    m->nnodes = nint > 0 ? nint : 1;
    float4 *nodes32;
    float4 *obb = nullptr;
    SSDF_CHECK(dalloc(s, &nodes32, 4 * size_t(m->nnodes), stream));
    if (query_boxes) SSDF_CHECK(dalloc(s, &obb, 8 * size_t(m->nnodes), stream));
    // read back in one copy: flag words 7 to 21, the coordinate scale, depth and leaves, the three filter words
    // and (from word 16) the box frame's middle and scale
    constexpr int kFirstWord = 7, kWords = 15;
    static_assert(kWords <= kReadbackWords, "read-back words");
    int *rb = nullptr;
    SSDF_CHECK(readback_words(&rb));
    const int *const scale_word = rb, *const depth_leaves = rb + 8 - kFirstWord;
    const int *const filt_info = rb + 10 - kFirstWord, *const frame_words = rb + 16 - kFirstWord;
    const int *obb_first = nullptr, *obb_count = nullptr;  // subtree ranges (null: the small root)
    const double *obb_nbox = nullptr;
    if (nt <= L) {
        // one leaf over everything (its triangle order is the Morton order)
        k_write_small_root<<<1, 1, 0, stream>>>(nt, box32, nodes32);
        LAUNCH_CHECK("k_write_small_root");
    } else {
        int *child_l, *child_r, *first_of, *parent_int, *parent_leaf, *count;
        float *nbox32;
        double *nbox64;
        SSDF_CHECK(dalloc(tmp, &child_l, nint, stream));
        SSDF_CHECK(dalloc(tmp, &child_r, nint, stream));
        SSDF_CHECK(dalloc(tmp, &first_of, nint, stream));
        SSDF_CHECK(dalloc(tmp, &parent_int, nint, stream));
        SSDF_CHECK(dalloc(tmp, &parent_leaf, nt, stream));
        SSDF_CHECK(dalloc(tmp, &count, nint, stream));
        SSDF_CHECK(dalloc(tmp, &nbox32, 6 * size_t(nint), stream));
        SSDF_CHECK(dalloc(tmp, &nbox64, 6 * size_t(nint), stream));
        k_karras<<<grid_blocks(nint, 256), 256, 0, stream>>>(nt, keys, child_l, child_r, first_of, count,
                                                             parent_int, parent_leaf);
        LAUNCH_CHECK("k_karras");
        const unsigned blocks = grid_blocks(nt, kRefitBlock);
        float *run32, *block32;
        double *run64, *block64;
        SSDF_CHECK(dalloc(tmp, &run32, 6 * size_t(kRuns) * blocks, stream));
        SSDF_CHECK(dalloc(tmp, &run64, 6 * size_t(kRuns) * blocks, stream));
        SSDF_CHECK(dalloc(tmp, &block32, 6 * size_t(blocks), stream));
        SSDF_CHECK(dalloc(tmp, &block64, 6 * size_t(blocks), stream));
        k_boxes_inside<<<blocks, kRefitBlock, 0, stream>>>(nt, ids, child_l, child_r, parent_int, parent_leaf, first_of,
                                                           count, box32, box64, nbox32, nbox64, run32, run64, block32,
                                                           block64);
        LAUNCH_CHECK("k_boxes_inside");
        k_boxes_across<<<grid_blocks(nint, 4 * kAcrossNodes), 128, 0, stream>>>(nt, ids, first_of, count, box32, box64,
                                                                                run32, run64, block32, block64, nbox32,
                                                                                nbox64);
        LAUNCH_CHECK("k_boxes_across");
        for (int round = 0; round < opts.treelet_opt && round < 8; round++) {  // treelet_opt: rounds (0 = none)
            SSDF_CHECK(treelet_optimize(nt, child_l, child_r, parent_int, parent_leaf, first_of, count, nbox32, nbox64,
                                        box32, box64, ids, stream));
        }
        k_write_nodes<<<grid_blocks(nint, 256), 256, 0, stream>>>(nt, L, child_l, child_r, first_of, count, ids,
                                                                  box32, nbox32, nodes32);
        LAUNCH_CHECK("k_write_nodes");
        k_depth<<<grid_blocks(nint, 256), 256, 0, stream>>>(nt, L, count, parent_int, child_l, child_r, flags + 8);
        LAUNCH_CHECK("k_depth");
        obb_first = first_of, obb_count = count, obb_nbox = nbox64;
    }
    // triangle records in leaf order
    float4 *t32, *filt = nullptr;
    double2 *t64 = nullptr;
    SSDF_CHECK(dalloc(s, &t32, 3 * size_t(nt), stream));
    if (keep64) SSDF_CHECK(dalloc(s, &t64, 5 * size_t(nt), stream));
    if (keep64) SSDF_CHECK(dalloc(s, &filt, 3 * size_t(nt), stream));  // the fix-up path's filter records
    int *entry;
    SSDF_CHECK(dalloc(s, &entry, 33, stream));
    k_box_frame<<<1, 32, 0, stream>>>(nodes32, obb_nbox ? obb_nbox : box64, obb_nbox ? 1 : nt, flags + 16, entry);
    LAUNCH_CHECK("k_box_frame");
    k_tri_records<<<grid_blocks(nt, 256), 256, 0, stream>>>(nt, ids, s0, s1, s2, vx, vy, vz, t32, t64, filt,
                                                            flags + 16, flags + 10);
    LAUNCH_CHECK("k_tri_records");
    // oriented boxes of the tree's children, from the triangle records
    if (query_boxes) {
        k_obb<<<grid_blocks(2ll * m->nnodes * 32, 128), 128, 0, stream>>>(
            m->nnodes, L, obb_count, obb_first, box64, obb_nbox, ids, nodes32, t32, t64, flags + 16, (float *)obb);
        LAUNCH_CHECK("k_obb");
    }
    SSDF_CUDA(cudaMemcpyAsync(rb, flags + kFirstWord, kWords * sizeof(int), cudaMemcpyDeviceToHost, stream));
    if (opts.normals) SSDF_CHECK(build_normals(s, m, s0, s1, s2, vx, vy, vz, stream));
    SSDF_CUDA(cudaStreamSynchronize(stream));  // the build's one wait: every read-back has landed
    float scale;
    memcpy(&scale, scale_word, sizeof(float));
    m->coord_scale = scale;
    memcpy(m->box_c, frame_words, 3 * sizeof(float));
    memcpy(&m->box_scale, frame_words + 4, sizeof(double));
    m->box_scale_f = m->box_scale >= 0x1p-126 && m->box_scale <= 0x1p126 ? float(m->box_scale) : NAN;
    m->nill = filt_info[0];
    if (keep64) {
        float term;
        memcpy(&term, &filt_info[1], sizeof(float));
        set_filter_window(m, term, filt_info[2] == 0 && m->box_scale == 1.0);
    }
    m->depth = nt <= L ? 1 : depth_leaves[0];
    m->nleaves = nt <= L ? 1 : depth_leaves[1];
    m->nodes32 = nodes32;
    m->obb = obb;
    m->entry = entry;
    m->tris32 = t32;
    m->tris64 = t64;
    m->filt32 = filt;
    if (m->depth >= kStackSize)
        return fail(SSDF_ERR_NOT_SUPPORTED,
                    "BVH depth " + std::to_string(m->depth) + " exceeds the traversal stack (" +
                        std::to_string(kStackSize) + ")");
    return SSDF_OK;
}

int mesh_build(MeshStorage **storage, DeviceMesh *mesh, ptrdiff_t nt, const int *s0, const int *s1, const int *s2,
               ptrdiff_t nv, const void *sx, const void *sy, const void *sz, int coord_f64, int device_ptrs,
               const ssdf_build_opts &opts, cudaStream_t stream, bool query_boxes, bool check_indices) {
    if (nt <= 0 || nv <= 0) return fail(SSDF_ERR_INVALID_ARGUMENT, "empty mesh");
    if (nt > kMaxTriangles) return fail(SSDF_ERR_NOT_SUPPORTED, "more than 2^26 triangles in one mesh");
    if (nv >= (1ll << 31)) return fail(SSDF_ERR_NOT_SUPPORTED, "more than 2^31 vertices");
    if (opts.leaf_size < 0 || opts.leaf_size > kMaxLeafSize)
        return fail(SSDF_ERR_INVALID_ARGUMENT, "leaf_size must be 0 (default) or 1.." + std::to_string(kMaxLeafSize));
    if (!s0 || !s1 || !s2 || !sx || !sy || !sz) return fail(SSDF_ERR_INVALID_ARGUMENT, "null mesh array");
    retain_pool_memory();
    MeshStorage *s = new MeshStorage();
    MeshStorage tmp;
    *mesh = DeviceMesh();
    int st = mesh_build_impl(s, &tmp, mesh, int(nt), s0, s1, s2, int(nv), sx, sy, sz, coord_f64, device_ptrs, opts,
                             query_boxes, check_indices, stream);
    for (void *p : tmp.blocks) cudaFreeAsync(p, stream);
    if (st == SSDF_OK) {
        cudaError_t e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) st = cuda_fail(e, "mesh build", __FILE__, __LINE__);
    }
    if (st != SSDF_OK) {
        cudaStreamSynchronize(stream);
        mesh_free(s);
        *mesh = DeviceMesh();
        return st;
    }
    *storage = s;
    return SSDF_OK;
}

}  // namespace ssdf_b200
