// treelet_opt.cu -- SAH treelet refinement of the LBVH (after Karras and Aila, "Fast parallel
// construction of high-quality bounding volume hierarchies", HPG 2013).
//
// One bottom-up pass with per-node arrival counters (the second thread to reach a node owns it, so
// its subtree is final; a warp then works on its lanes' treelets together): every node with at least
// kTreeletLeaves triangles below it roots a treelet,
// grown from its two children by opening the largest-area internal member until it has seven
// members. The binary tree over those members with the lowest surface-area cost,
//     cost(node) = area(node) + cost(left) + cost(right),   cost(triangle) = area(triangle),
// is found exactly by dynamic programming over the 127 member subsets (each subset's best split
// among its 2^k - 2 partitions), and replaces the old arrangement when it is cheaper, reusing the
// treelet's six internal nodes (the root keeps its identity, so the walk continues upward). Boxes
// and parent links inside the treelet are rewritten. The pass then re-derives the leaf order (a
// depth-first numbering of the triangles), so every subtree is again a contiguous range of leaf
// positions, as the leaf collapse and the node records require.
#include <cuda_runtime.h>

#include <cfloat>

#include "internal.h"

namespace ssdf_b200 {

namespace {

constexpr int kTreeletLeaves = 7;
constexpr int kSubsets = 1 << kTreeletLeaves;

struct TreeArrays {
    int *child_l, *child_r, *parent_int, *parent_leaf;
    float *nbox32;
    double *nbox64;
    const float *pbox32;
    const double *pbox64;
    const int *ids;  // leaf position -> triangle
    float *cost;     // per internal node: SAH cost of its subtree
    int *count;      // per internal node: triangles below
};

__device__ __forceinline__ float area6(const float *b) {
    const float dx = fmaxf(b[1] - b[0], 0.f), dy = fmaxf(b[3] - b[2], 0.f), dz = fmaxf(b[5] - b[4], 0.f);
    return 2.f * (dx * dy + dy * dz + dz * dx);
}

// Box / cost / count of a child reference (internal >= 0, leaf -(pos + 1)); reads bypass L1 since
// other threads wrote them.
__device__ __forceinline__ void ref_box32(const TreeArrays &t, int ref, float *b) {
    const float *s = ref >= 0 ? t.nbox32 + 6 * ref : t.pbox32 + 6 * t.ids[-ref - 1];
    for (int k = 0; k < 6; k++) b[k] = __ldcg(s + k);
}
__device__ __forceinline__ void ref_box64(const TreeArrays &t, int ref, double *b) {
    const double *s = ref >= 0 ? t.nbox64 + 6 * ref : t.pbox64 + 6 * t.ids[-ref - 1];
    for (int k = 0; k < 6; k++) b[k] = __ldcg(s + k);
}
__device__ __forceinline__ float ref_cost(const TreeArrays &t, int ref) {
    if (ref >= 0) return __ldcg(t.cost + ref);
    float b[6];
    ref_box32(t, ref, b);
    return area6(b);
}

__device__ __forceinline__ void set_parent(const TreeArrays &t, int ref, int parent) {
    if (ref >= 0)
        __stcg(t.parent_int + ref, parent);
    else
        __stcg(t.parent_leaf + (-ref - 1), parent);
}

// A treelet in the making, in shared memory (one per warp): its members and their boxes, the internal nodes
// it reuses, and the dynamic programme's area, cost and best split of every subset.
struct TreeletWork {
    double mb64[kTreeletLeaves][6];
    float mb[kTreeletLeaves][6];
    int mcount[kTreeletLeaves];
    int member[kTreeletLeaves];
    int inner[kTreeletLeaves - 1];
    float old_cost;
    float area[kSubsets];
    float c[kSubsets];
    unsigned char split[kSubsets];
    // the rebuilt arrangement: internal node onode[k] now covers the members of subset oset[k]
    int onode[kTreeletLeaves - 1], oset[kTreeletLeaves - 1];
    int2 oref[kTreeletLeaves - 1], stack[kTreeletLeaves];
    int norder;
};

// The subsets of seven members by size, each size in increasing order, and where each size starts.
struct SubsetTable {
    unsigned char set[kSubsets];
    int start[kTreeletLeaves + 2];
};
constexpr SubsetTable make_subsets() {
    SubsetTable t{};
    int n = 0;
    for (int size = 0; size <= kTreeletLeaves; size++) {
        t.start[size] = n;
        for (int s = 0; s < kSubsets; s++) {
            int bits = 0;
            for (int b = 0; b < kTreeletLeaves; b++) bits += (s >> b) & 1;
            if (bits == size) t.set[n++] = (unsigned char)s;
        }
    }
    t.start[kTreeletLeaves + 1] = n;
    return t;
}
__constant__ SubsetTable kSubsetTable = make_subsets();

// The best split of every subset of SIZE members, from the smaller subsets' costs: 2^LG lanes to
// a subset, each the splits that agree with its number in the lowest bits of the subset without its lowest
// member (each split is met once, by the half that holds that member); the cheapest wins, the larger half
// among equals. Sizes and counts are constants, so a lane's costs are all asked for at once.
constexpr int choose(int n, int k) { return k == 0 ? 1 : choose(n - 1, k - 1) * n / k; }
constexpr int lanes_log(int size, int nsub) {
    int lg = 0;
    while (lg < size - 1 && (2 << lg) * nsub <= 32) lg++;
    return lg;
}
template <int SIZE>
__device__ __forceinline__ void best_splits(TreeletWork &w, const unsigned char *__restrict__ sets, int lane) {
    constexpr int kSub = choose(kTreeletLeaves, SIZE), kLg = lanes_log(SIZE, kSub), kTrips = 1 << (SIZE - 1 - kLg);
    const int before = kSubsetTable.start[SIZE], r = lane & ((1 << kLg) - 1);
#pragma unroll
    for (int first = 0; first < kSub; first += 32 >> kLg) {
        const int j = first + (lane >> kLg);
        const int s = j < kSub ? int(sets[before + j]) : 0;
        float best = FLT_MAX;
        int bp = 0;
        if (s) {
            const int low = s & -s;
            int rest = s ^ low, half = low;
#pragma unroll
            for (int k = 0; k < kLg; k++) {
                const int bit = rest & -rest;
                rest ^= bit;
                if ((r >> k) & 1) half |= bit;
            }
            int q = rest;
#pragma unroll
            for (int k = 0; k < kTrips; k++) {
                const int p = half | q;
                if (p != s) {
                    const float v = w.c[p] + w.c[s ^ p];
                    if (v < best || (v == best && p > bp)) best = v, bp = p;
                }
                q = (q - 1) & rest;
            }
        }
#pragma unroll
        for (int o = 1; o < (1 << kLg); o <<= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int obp = __shfl_xor_sync(0xffffffffu, bp, o);
            if (ob < best || (ob == best && obp > bp)) best = ob, bp = obp;
        }
        if (s && r == 0) w.c[s] = w.area[s] + best, w.split[s] = (unsigned char)bp;
    }
    __syncwarp();
}

// The whole warp: the treelet rooted at internal node x (its subtree is final, of kTreeletLeaves triangles or
// more), grown from its two children by opening the largest-area internal member until it has seven members,
// a lane to each; then the best binary tree over them, by dynamic programming over the member subsets. Bound by
// latency, one treelet after the other up the tree's deepest path: a member's lane asks for its children's
// links together with its box, so an opening waits once, and the programme's sizes are unrolled (11,100 cycles
// as loops, two reads at a time). A round on 5,120 / 41,006 / 81,920 / 131,072 triangles takes 154 / 230 /
// 277 / 331 us, 283 / 394 / 455 / 500 with the loops, two waits an opening and 32 climbers a warp.
__device__ void treelet_best(const TreeArrays &t, int x, TreeletWork &w, const unsigned char *__restrict__ sets,
                             int lane) {
    constexpr unsigned kAll = 0xffffffffu;
    float bx[6], b[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, mcost = 0.f;
    double d[6];
    int ref = -1, cl = 0, cr = 0, mcount = 1;
    // everything an internal member will be asked for, its children for the case that it is opened among it
    auto take = [&](int r) {
        ref = r;
        if (r < 0) return;
        cl = __ldcg(t.child_l + r), cr = __ldcg(t.child_r + r);
        ref_box32(t, r, b);
        ref_box64(t, r, d);
        mcost = __ldcg(t.cost + r), mcount = __ldcg(t.count + r);
    };
    for (int q = 0; q < 6; q++) bx[q] = __ldcg(t.nbox32 + 6 * x + q);
    if (lane < 2) take(__ldcg((lane ? t.child_r : t.child_l) + x));
    float old_cost = area6(bx);  // the old internal nodes' areas, then the members' costs
    if (lane == 0) w.inner[0] = x;
    for (int m = 2; m < kTreeletLeaves; m++) {  // with kTreeletLeaves triangles below x, one is internal
        const int key = lane < m && ref >= 0 ? __float_as_int(area6(b)) : -1;  // areas are not negative
        const int best = __reduce_max_sync(kAll, key);
        const int pick = __ffs(__ballot_sync(kAll, key == best)) - 1;
        const int y = __shfl_sync(kAll, ref, pick), l = __shfl_sync(kAll, cl, pick), r = __shfl_sync(kAll, cr, pick);
        old_cost += __int_as_float(best);
        if (lane == 0) w.inner[m - 1] = y;
        if (lane == pick || lane == m) take(lane == pick ? l : r);
    }
    if (lane < kTreeletLeaves) {
        if (ref < 0) {  // triangles: only now, so that no opening waited for them
            ref_box32(t, ref, b);
            ref_box64(t, ref, d);
            mcost = area6(b), mcount = 1;
        }
        w.member[lane] = ref;
        w.mcount[lane] = mcount;
        for (int q = 0; q < 6; q++) w.mb[lane][q] = b[q];
        for (int q = 0; q < 6; q++) w.mb64[lane][q] = d[q];
    }
    for (int k = 0; k < kTreeletLeaves; k++) old_cost += __shfl_sync(kAll, mcost, k);
    if (lane == 0) w.old_cost = old_cost;
    // areas of all subsets: lane l those of members 2 .. 6 in the bits of l, with and without members 0 and 1
    {
        float u[6] = {FLT_MAX, -FLT_MAX, FLT_MAX, -FLT_MAX, FLT_MAX, -FLT_MAX}, e[2][6];
        for (int k = 0; k < kTreeletLeaves; k++)
            for (int q = 0; q < 6; q++) {
                const float v = __shfl_sync(kAll, b[q], k);
                if (k < 2) e[k][q] = v;
                else if ((lane >> (k - 2)) & 1) u[q] = (q & 1) ? fmaxf(u[q], v) : fminf(u[q], v);
            }
        for (int v = 0; v < 4; v++) {
            float r[6];
            for (int q = 0; q < 6; q++) {
                r[q] = u[q];
                if (v & 1) r[q] = (q & 1) ? fmaxf(r[q], e[0][q]) : fminf(r[q], e[0][q]);
                if (v & 2) r[q] = (q & 1) ? fmaxf(r[q], e[1][q]) : fminf(r[q], e[1][q]);
            }
            w.area[4 * lane + v] = area6(r);
        }
    }
    if (lane < kTreeletLeaves) w.c[1 << lane] = mcost, w.split[1 << lane] = 0;
    __syncwarp();
    best_splits<2>(w, sets, lane);
    best_splits<3>(w, sets, lane);
    best_splits<4>(w, sets, lane);
    best_splits<5>(w, sets, lane);
    best_splits<6>(w, sets, lane);
    best_splits<7>(w, sets, lane);
}

// One lane: the arrangement by the programme's splits when it is cheaper, reusing the treelet's internal nodes
// (the root keeps x): in w.onode / w.oset / w.oref the reused nodes, the members each now covers and its two
// children (w.norder of them; 0 when the old arrangement stays, whose cost is stored here).
__device__ void rebuild_plan(const TreeArrays &t, int x, TreeletWork &w) {
    constexpr int full = kSubsets - 1;
    w.norder = 0;
    if (!(w.c[full] < w.old_cost * (1.f - 1e-6f))) {
        __stcg(t.cost + x, w.old_cost);
        return;
    }
    int sp = 0, used = 1, norder = 0;
    w.stack[sp++] = make_int2(full, x);
    while (sp > 0) {
        const int2 top = w.stack[--sp];
        const int split = w.split[top.x];
        const int halves[2] = {split, top.x ^ split};
        int refs[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int hs = halves[h];
            const bool single = (hs & (hs - 1)) == 0;
            refs[h] = single ? w.member[__ffs(hs) - 1] : w.inner[used];
            if (!single) w.stack[sp++] = make_int2(hs, refs[h]), used++;
        }
        w.onode[norder] = top.y, w.oset[norder] = top.x;
        w.oref[norder++] = make_int2(refs[0], refs[1]);
    }
    w.norder = norder;
}

// The whole warp, after rebuild_plan: lane k writes reused node w.onode[k]'s child and parent links, boxes
// (float and double), triangle count and cost. A node's box is the union of its members' boxes -- the same
// values the union of its two children's boxes gives, min and max being exact -- so no lane waits for
// another. The owner's fence before its next arrival, after the warp's barrier, publishes every lane's stores.
__device__ void rebuild_write(const TreeArrays &t, const TreeletWork &w, int lane) {
    if (lane >= w.norder) return;
    const int node = w.onode[lane], s = w.oset[lane];
    const int2 refs = w.oref[lane];
    __stcg(t.child_l + node, refs.x);
    __stcg(t.child_r + node, refs.y);
    set_parent(t, refs.x, node);
    set_parent(t, refs.y, node);
    float b[6];
    double d[6];
    int cnt = 0;
    bool first = true;
    for (int j = 0; j < kTreeletLeaves; j++) {
        if (!((s >> j) & 1)) continue;
        for (int q = 0; q < 6; q += 2) {
            b[q] = first ? w.mb[j][q] : fminf(b[q], w.mb[j][q]);
            b[q + 1] = first ? w.mb[j][q + 1] : fmaxf(b[q + 1], w.mb[j][q + 1]);
            d[q] = first ? w.mb64[j][q] : fmin(d[q], w.mb64[j][q]);
            d[q + 1] = first ? w.mb64[j][q + 1] : fmax(d[q + 1], w.mb64[j][q + 1]);
        }
        cnt += w.mcount[j];
        first = false;
    }
    for (int q = 0; q < 6; q++) {
        __stcg(t.nbox32 + 6 * node + q, b[q]);
        __stcg(t.nbox64 + 6 * node + q, d[q]);
    }
    __stcg(t.count + node, cnt);
    __stcg(t.cost + node, w.c[s]);
}

constexpr int kTreeletThreads = 128;
// Lanes of a warp that start from a triangle. With fewer, more warps share the treelets close to the triangles,
// where one warp has several at once; with many triangles the GPU is full of warps anyway. us at 16 and 32:
// 5,120 triangles 169 / 196, 41,006 255 / 271, 81,920 305 / 328, 131,072 387 / 357.
constexpr int treelet_climbers(int n) { return n <= 100000 ? 16 : 32; }

// One lane per triangle climbs from its leaf; the second thread to reach a node owns it (its
// subtree is then final). Each round, the warp optimises its lanes' owned treelets one after the
// other, all 32 lanes sharing each one's dynamic programme. Lanes without work stay in the loop (the
// warp-wide votes need every lane) until the whole warp has climbed out.
__global__ void __launch_bounds__(kTreeletThreads) k_treelets(int n, int climbers, TreeArrays t,
                                                             int *arrivals) {
    __shared__ TreeletWork s_work[kTreeletThreads / 32];
    __shared__ unsigned char s_sets[kSubsets];
    for (int k = threadIdx.x; k < kSubsets; k += kTreeletThreads) s_sets[k] = kSubsetTable.set[k];
    __syncthreads();
    TreeletWork &w = s_work[threadIdx.x >> 5];
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int p = int((blockIdx.x * kTreeletThreads + threadIdx.x) >> 5) * climbers + lane;
    int node = lane < climbers && p < n ? __ldcg(t.parent_leaf + p) : -1;
    while (__any_sync(kAll, node >= 0)) {
        bool own = false;
        int parent = -1;
        if (node >= 0) {
            // a node's links and count stay as they are until it is owned, so they don't wait for the arrival
            parent = __ldcg(t.parent_int + node);
            const int cnt = __ldcg(t.count + node), l = __ldcg(t.child_l + node), r = __ldcg(t.child_r + node);
            __threadfence();
            if (atomicAdd(&arrivals[node], 1) == 0) {
                node = -1;  // the first arrival: the other child's thread continues
            } else {
                __threadfence();
                if (cnt >= kTreeletLeaves) {
                    own = true;
                } else {
                    float b[6];
                    for (int q = 0; q < 6; q++) b[q] = __ldcg(t.nbox32 + 6 * node + q);
                    __stcg(t.cost + node, area6(b) + ref_cost(t, l) + ref_cost(t, r));
                }
            }
        }
        unsigned todo = __ballot_sync(kAll, own);
        // every lane reads the owned subtrees, but only their owners met the other arrivals and fenced: a vote or
        // a shuffle orders no memory, this barrier does
        __syncwarp();
        while (todo) {
            const int owner = __ffs(todo) - 1;
            todo &= todo - 1;
            const int x = __shfl_sync(kAll, node, owner);
            treelet_best(t, x, w, s_sets, lane);
            if (lane == owner) rebuild_plan(t, x, w);
            __syncwarp();
            rebuild_write(t, w, lane);
            __syncwarp();
        }
        if (node >= 0) node = parent;
    }
}

// New leaf position of every triangle: its rank in a depth-first, left-first walk of the new tree,
// found by walking up and adding the sizes of left siblings.
__global__ void k_leaf_positions(int n, const int *__restrict__ child_l, const int *__restrict__ parent_int,
                                 const int *__restrict__ parent_leaf, const int *__restrict__ count,
                                 int *__restrict__ newpos) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    int ref = -(p + 1);
    int node = parent_leaf[p];
    int off = 0;
    int guard = 0;
    while (node >= 0 && guard++ < (1 << 20)) {
        const int l = child_l[node];
        if (l != ref) off += l >= 0 ? count[l] : 1;
        ref = node;
        node = parent_int[node];
    }
    newpos[p] = off;
}

__global__ void k_relabel(int n, const int *__restrict__ newpos, const int *__restrict__ ids_old,
                          const int *__restrict__ parent_leaf_old, const int *__restrict__ child_l_old,
                          const int *__restrict__ child_r_old, int *__restrict__ ids_new,
                          int *__restrict__ parent_leaf_new, int *__restrict__ child_l_new,
                          int *__restrict__ child_r_new) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int q = newpos[p];
    ids_new[q] = ids_old[p];
    const int parent = parent_leaf_old[p];
    parent_leaf_new[q] = parent;
    if (child_l_old[parent] == -(p + 1)) child_l_new[parent] = -(q + 1);
    if (child_r_old[parent] == -(p + 1)) child_r_new[parent] = -(q + 1);
}

// first_of: leaf position of the leftmost triangle below each internal node.
__global__ void k_first_of(int nint, const int *__restrict__ child_l, int *__restrict__ first_of) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nint) return;
    int ref = i;
    int guard = 0;
    while (ref >= 0 && guard++ < (1 << 20)) ref = child_l[ref];
    first_of[i] = -ref - 1;
}

}  // namespace

int treelet_optimize(int n, int *child_l, int *child_r, int *parent_int, int *parent_leaf, int *first_of, int *count,
                     float *nbox32, double *nbox64, const float *pbox32, const double *pbox64, int *sorted_ids,
                     cudaStream_t stream) {
    const int nint = n - 1;
    if (nint < kTreeletLeaves) return SSDF_OK;
    float *cost = nullptr;
    int *arrivals = nullptr, *newpos = nullptr, *ids2 = nullptr, *pl2 = nullptr, *cl2 = nullptr,
        *cr2 = nullptr;
    int st = SSDF_OK;
    auto alloc = [&](void **p, size_t b) {
        if (st == SSDF_OK && cudaMallocAsync(p, b, stream) != cudaSuccess) st = fail(SSDF_ERR_OUT_OF_MEMORY, "treelet scratch");
    };
    alloc((void **)&cost, sizeof(float) * nint);
    alloc((void **)&arrivals, sizeof(int) * nint);
    alloc((void **)&newpos, sizeof(int) * n);
    alloc((void **)&ids2, sizeof(int) * n);
    alloc((void **)&pl2, sizeof(int) * n);
    alloc((void **)&cl2, sizeof(int) * nint);
    alloc((void **)&cr2, sizeof(int) * nint);
    cudaError_t e = cudaSuccess;
    if (st == SSDF_OK) {
        TreeArrays t{child_l, child_r, parent_int, parent_leaf, nbox32, nbox64, pbox32, pbox64, sorted_ids, cost, count};
        e = cudaMemsetAsync(arrivals, 0, sizeof(int) * nint, stream);
        if (e == cudaSuccess) {
            const int climbers = treelet_climbers(n);
            k_treelets<<<grid_blocks(n, kTreeletThreads / 32 * climbers), kTreeletThreads, 0, stream>>>(n, climbers, t,
                                                                                                        arrivals);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) {
            k_leaf_positions<<<grid_blocks(n, 256), 256, 0, stream>>>(n, child_l, parent_int, parent_leaf, count,
                                                                       newpos);
            e = cudaMemcpyAsync(cl2, child_l, sizeof(int) * nint, cudaMemcpyDeviceToDevice, stream);
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(cr2, child_r, sizeof(int) * nint, cudaMemcpyDeviceToDevice, stream);
        if (e == cudaSuccess) {
            k_relabel<<<grid_blocks(n, 256), 256, 0, stream>>>(n, newpos, sorted_ids, parent_leaf, child_l, child_r, ids2,
                                                                pl2, cl2, cr2);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(sorted_ids, ids2, sizeof(int) * n, cudaMemcpyDeviceToDevice, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(parent_leaf, pl2, sizeof(int) * n, cudaMemcpyDeviceToDevice, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(child_l, cl2, sizeof(int) * nint, cudaMemcpyDeviceToDevice, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(child_r, cr2, sizeof(int) * nint, cudaMemcpyDeviceToDevice, stream);
        if (e == cudaSuccess) {
            k_first_of<<<grid_blocks(nint, 256), 256, 0, stream>>>(nint, child_l, first_of);
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) st = cuda_fail(e, "treelet refinement", __FILE__, __LINE__);
    }
    for (void *p : {(void *)cost, (void *)arrivals, (void *)newpos, (void *)ids2, (void *)pl2,
                    (void *)cl2, (void *)cr2})
        if (p) cudaFreeAsync(p, stream);
    return st;
}

}  // namespace ssdf_b200
