// internal.h -- shared declarations of the library's host runtime and kernels.
#pragma once

#include <algorithm>
#include <cmath>

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <string>

#include "../../include/ssdf_b200.h"

namespace ssdf_b200 {

// ---- error plumbing ------------------------------------------------------------------------------
void set_error(const std::string &msg);
int fail(int status, const std::string &msg);
int cuda_fail(cudaError_t err, const char *what, const char *file, int line);

#define SSDF_CUDA(call)                                                             \
    do {                                                                            \
        cudaError_t ssdf_err_ = (call);                                             \
        if (ssdf_err_ != cudaSuccess)                                               \
            return ::ssdf_b200::cuda_fail(ssdf_err_, #call, __FILE__, __LINE__);    \
    } while (0)

#define SSDF_CHECK(call)                           \
    do {                                           \
        int ssdf_st_ = (call);                     \
        if (ssdf_st_ != SSDF_OK) return ssdf_st_;  \
    } while (0)

// ---- device layouts ------------------------------------------------------------------------------
//
// BVH: binary, child-box layout. Every internal node holds both children's boxes and references,
// so one visit tests two boxes from one record, 64 bytes (axis-aligned) or 128 (oriented):
//   FP32 node (4 x float4): (c0.lox, c0.hix, c0.loy, c0.hiy), (c1.lox, c1.hix, c1.loy, c1.hiy),
//                           (c0.loz, c0.hiz, c1.loz, c1.hiz), (ref0, ref1, -, -) as int bits
//   oriented node (8 x float4): the same children's oriented boxes in the mesh's box frame (see
//                           DeviceMesh::obb); per axis k = u, v, n of both children: (kx of c0, kx of
//                           c1, ky, ky), (kz, kz, -k.centre, -k.centre), then the half extents (hu, hu,
//                           hv, hv), (hn, hn, ref0, ref1): pairs (c0, c1) throughout, for two-wide FP32
// A reference >= 0 is an internal node; < 0 is a leaf ~((first << 5) | (count - 1)) over the
// triangle records in leaf order; kEmptyRef is an empty slot (its box is inverted).
// Triangles in leaf order:
//   FP32 record (3 x float4): (ax, ay, az, bx), (by, bz, cx, cy), (cz, id bits, -, -)
//   FP64 record (5 x double2): (ax, ay), (az, bx), (by, bz), (cx, cy), (cz, id)
// where id is the triangle's index in the caller's s0/s1/s2 and a, b, c its vertices s0, s1, s2.
constexpr int kEmptyRef = -2147483647 - 1;  // INT_MIN
constexpr int kLeafCountBits = 5;
constexpr int kMaxLeafSize = 16;
constexpr int kMaxTriangles = 1 << 26;
constexpr int kStackSize = 64;

__host__ __device__ inline int leaf_ref(int first, int count) { return ~((first << kLeafCountBits) | (count - 1)); }
__host__ __device__ inline int leaf_first(int ref) { return (~ref) >> kLeafCountBits; }
__host__ __device__ inline int leaf_count(int ref) { return ((~ref) & ((1 << kLeafCountBits) - 1)) + 1; }

struct DeviceMesh {
    int nt = 0;            // triangles
    int nv = 0;            // vertices
    int nnodes = 0;        // node records (>= 1)
    int depth = 0;         // max internal-node depth of the BVH (root = 1)
    int leaf_size = 4;
    int nleaves = 0;
    const float4 *nodes32 = nullptr;   // [4 * nnodes]
    // Oriented boxes of the same tree's children, [8 * nnodes]: what the query kernels walk. Axes
    // and extents are for points (p - box_c) * box_scale, with margins that make the float distance a
    // lower bound of any contained triangle's distance, exact or as the float arithmetic evaluates it
    // (mesh_build.cu, k_obb).
    const float4 *obb = nullptr;
    // where a walk shared by a warp starts: entry[0] nodes (at most 32), entry[1 ..]
    const int *entry = nullptr;
    float box_c[3] = {0.f, 0.f, 0.f};
    double box_scale = 1.0;    // a power of two, 1 for a mesh of half size 2^-26 to 2^28
    float box_scale_f = 1.f;   // the same for the float walk; NaN (every box at distance 0) beyond float's range
    const float4 *tris32 = nullptr;    // [3 * nt], leaf order
    const double2 *tris64 = nullptr;   // [5 * nt], leaf order, or null
    // the fix-up path's FP32 filter records, [3 * nt], leaf order, with the double data or null:
    // (ax, ay, az, ab.ab), (abx, aby, abz, ac.ac), (acx, acy, acz, ab.ac) of the triangle, or of a
    // well-conditioned proxy containing an ill-conditioned one, marked by the sign bit of ab.ab
    // (mesh_build.cu, filter_record)
    const float4 *filt32 = nullptr;
    // sign data, caller's triangle order
    const int *s0 = nullptr, *s1 = nullptr, *s2 = nullptr;  // [nt]
    const double *face_n = nullptr;    // [3 * nt]
    const double *edge_n = nullptr;    // [9 * nt]
    const double *vertex_n = nullptr;  // [3 * nv]
    // scale of the coordinates (max |coordinate| over the mesh), for the fix-up window
    float coord_scale = 0.f;
    // triangles the fix-up filter sees through a proxy (ill-conditioned; 0 without the double data)
    int nill = 0;
    // the fix-up window's smallest relative width for this mesh (at least 2^-16; wider when its
    // records are large against coord_scale), and whether the float filter can serve it at all
    // (coordinates within 2^28, no record that float rounding made degenerate, needle-like or
    // too small); see set_filter_window
    float tau_rel_min = 1.0f / 65536.0f;
    int filter_ok = 0;
};

// Largest coordinate magnitude of a mesh, or of a query point, that the fix-up path's float filter
// takes: every product it forms then stays finite (|p - a| < 2^30, dot products < 2^60, their
// products < 2^120). Points beyond it are answered exactly by the second stage.
constexpr float kFilterMaxCoord = 268435456.0f;  // 2^28
// Sets DeviceMesh::tau_rel_min and ::filter_ok from the largest bound term of the mesh's filter
// records (mesh_build.cu, filter_bound) and whether every record is safe.
void set_filter_window(DeviceMesh *m, float largest_term, bool records_safe);

// Everything a query launch needs; built by the host entry points.
struct QueryArgs {
    DeviceMesh m;
    int output;        // SSDF_OUT_*
    int coord_f64;     // G == double
    int out_f64;       // T == double
    int is_grid;
    long long npoints;
    // point source
    const void *x, *y, *z;
    // grid source: nodes n, origin lo and spacing h in G precision (both views kept)
    long long nx, ny, nz;
    double lo64[3], h64[3];
    float lo32[3], h32[3];
    // outputs
    void *out;
    int *outtri;
    void *outx, *outy, *outz;
    // fix-up window: tau = tau_rel * (coord_scale + d)
    float tau_rel;
    // warp packets: a packet that has tested more than this many triangle records hands
    // its queries to the second stage (a warp per query) with their current windows; 0: no limit;
    // < 0: the default for the launch's size (resolve_hand_over)
    int warp_budget;
    // they may while fewer queries than this are on the list (resolve_hand_over)
    int hand_most;
    // hand-over list (query, threshold), finished by k_window; null without a budget
    int *fallback_ids;
    float *fallback_thr;
    int *fallback_count;
    // optional counters [4]: triangle tests, box tests, fix-up evaluations, fallbacks
    unsigned long long *counters;
    // 0: environment / default; 1 warp packets, 2 thread per query
    int force_traversal;
    // point lists: the visiting order (query index per slot, Morton-sorted), or null (input order)
    const int *order;
    // streamed download of a grid (launch_query_streamed): the blocks of chunk c (blockIdx.x /
    // chunk_blocks, whole slabs of the grid) count themselves in chunk_counts[c] (device memory), and
    // the last one raises chunk_flags[c] (page-locked host memory); null: off
    int *chunk_counts;
    int *chunk_flags;
    int chunk_blocks;
    // grid launches: start each step of a block's column from the triangles found one step below
    int seed;
    // grid launches: z-steps of 2 kQ planes each block walks (1 .. kMaxGridSteps)
    int grid_steps;
    // grid jobs: the z-planes nz of this job are planes z0 .. z0 + nz - 1 of a larger grid with the
    // same origin and spacing (node coordinates use the global plane; outputs are the job's own)
    long long z0;
};

// Job table header of a batch (device memory).
struct BatchHeader {
    int njobs;
    int pad;
    long long total_blocks;
};

// Device pointers and launch shape of one batch launch.
struct BatchLaunch {
    const BatchHeader *hdr;
    const QueryArgs *jobs;
    const long long *first_block;
    unsigned long long *next_item;
    int grid;   // persistent blocks (SMs x resident blocks per SM)
    int sms;
    bool warp;
};

// ---- mesh build (mesh_build.cu) ------------------------------------------------------------------
struct MeshStorage;  // owns the device allocations behind a DeviceMesh
int mesh_build(MeshStorage **storage, DeviceMesh *mesh, ptrdiff_t nt, const int *s0, const int *s1, const int *s2,
               ptrdiff_t nv, const void *sx, const void *sy, const void *sz, int coord_f64, int device_ptrs,
               const ssdf_build_opts &opts, cudaStream_t stream, bool query_boxes = true,
               bool check_indices = true);
// query_boxes false: without the oriented boxes (DeviceMesh::obb null), for walks of the axis-aligned nodes
// only (contact.cu). check_indices false: device index arrays that this library wrote (sdf_rebuild.cu).
void mesh_free(MeshStorage *storage);                            // after the work using it completed
void mesh_free_async(MeshStorage *storage, cudaStream_t stream);  // in stream order
size_t mesh_bytes(const MeshStorage *storage);

// ---- radix sort (radix_sort.cu) ------------------------------------------------------------------
// Stable LSD sort of (key, value) pairs on the device, keys of `key_bits` low bits. Scratch is
// allocated on `stream` (stream-ordered).
int radix_sort_pairs_u32(uint32_t *keys, int *vals, int n, int key_bits, cudaStream_t stream);
int radix_sort_pairs_u64(uint64_t *keys, int *vals, int n, int key_bits, cudaStream_t stream);
// Exclusive prefix sum of n ints (out may alias in).
int exclusive_scan_i32(const int *in, int *out, int n, cudaStream_t stream);

// ---- queries (bvh_query.cu) ----------------------------------------------------------------------
int launch_query(const QueryArgs &args, int precision, cudaStream_t stream);
// launch_query that, on success, hands back the second stage's query list (device ints: count, then the
// query indices) instead of freeing it; *fallback_list stays null where there is none. The caller frees it with cudaFreeAsync on `stream`.
int launch_query_keep(const QueryArgs &args, int precision, cudaStream_t stream, int **fallback_list);
// A grid query whose results go to host arrays: args.out / args.outtri are device buffers of the
// grid's size, and each slab chunk is copied to host_out / host_tri as soon as the kernel has
// finished it (through page-locked staging where an array is pageable), so the download overlaps the
// query. Returns when the host arrays hold the results (the same bits as launch_query followed by a
// copy).
int launch_query_streamed(const QueryArgs &args, int precision, void *host_out, int *host_tri, cudaStream_t stream);
// Host copy split across up to 8 threads (copies of at least 8 MB).
void par_memcpy(void *dst, const void *src, size_t bytes);
// Whether the streamed grid download applies: n queries (at least 2^22) and the switch on.
bool streamed_download_applies(long long n, const void *host_out, const int *host_tri);
int launch_query_noalloc(const QueryArgs &args, cudaStream_t stream);
long long noalloc_max_queries();
int launch_batch(const BatchLaunch &b, int precision, cudaStream_t stream);
// Whether a fix-up request on this mesh runs the FP64 kernel instead (bvh_query.cu).
bool fixup_runs_f64(const DeviceMesh &m);
int batch_capture_graphs(ssdf_batch *b);  // batch.cu
int batch_blocks_per_sm(int precision, bool warp);
bool default_warp(int is_grid);
// Queries each lane of the query kernels answers (two independent arithmetic chains per node visit).
#ifndef SSDF_B200_QUERIES_PER_LANE
#define SSDF_B200_QUERIES_PER_LANE 1
#endif
constexpr int kQ = SSDF_B200_QUERIES_PER_LANE;
// Grid launches: a block of 128 lanes covers an 8 x 4 column of nodes and walks it upwards in
// QueryArgs::grid_steps steps (1 .. kMaxGridSteps) of 4 kQ z-planes, each step an 8 x 4 x 4kQ brick
// of nodes (each warp a 4 x 4 x 2kQ part of it). A lane starts each step from the closest triangle it
// found one step below, 4 kQ nodes away: a tight upper bound (SSDF_B200_SEED=0 starts from the
// incoming bound alone). Large grids take kMaxGridSteps; a grid too small to fill the GPU many times
// over with such columns takes fewer (grid_steps_for).
constexpr int kMaxGridSteps = 8;
__host__ __device__ inline long long grid_blocks_x(long long nx) { return (nx + 7) / 8; }
__host__ __device__ inline long long grid_blocks_y(long long ny) { return (ny + 3) / 4; }
__host__ __device__ inline long long grid_block_planes(int steps) { return 4ll * kQ * steps; }
__host__ __device__ inline long long grid_blocks_z(long long nz, int steps) {
    return (nz + grid_block_planes(steps) - 1) / grid_block_planes(steps);
}
// Blocks of 128 lanes one job needs (grid columns as above, x fastest, then y, then z; or 128 kQ
// consecutive points).
inline long long query_blocks(const QueryArgs &a) {
    if (a.is_grid) return grid_blocks_x(a.nx) * grid_blocks_y(a.ny) * grid_blocks_z(a.nz, a.grid_steps);
    return (a.npoints + 128 * kQ - 1) / (128 * kQ);
}
// Steps per grid block for a launch whose work, at one step per block, is `one_step_blocks` blocks:
// the most steps (1, 2, 4 or kMaxGridSteps) that still leave ten waves of resident blocks on this
// device (SSDF_B200_GRID_STEPS overrides). bvh_query.cu.
int grid_steps_for(long long one_step_blocks);
// Sets QueryArgs::grid_steps of a grid job from its own size (no-op for point lists).
void set_grid_steps(QueryArgs *a);

// The counts ssdf_last_query_counts reports for this thread's last counting launch (bvh_query.cu).
void set_last_counts(unsigned long long tri, unsigned long long box, unsigned long long fix,
                     unsigned long long fallback);
// Warp-summed, one 64-bit atomic per warp: counts of a counting launch (c[0] triangle tests, c[1]
// box tests). Every lane of the warp must call it.
__device__ __forceinline__ void flush_pair_counts(unsigned long long *c, unsigned long long tri,
                                                  unsigned long long box) {
    for (int o = 16; o > 0; o >>= 1) {
        tri += __shfl_xor_sync(0xffffffffu, tri, o);
        box += __shfl_xor_sync(0xffffffffu, box, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(c, tri);
        atomicAdd(c + 1, box);
    }
}

// ---- plain methods (brute_force.cu, celllist.cu) -------------------------------------
// With SSDF_B200_COUNT set, both run a counting instantiation and leave their triangle (Ericson)
// and box tests in ssdf_last_query_counts.
int brute_force_edf(int f64, ptrdiff_t npoints, const void *x, const void *y, const void *z, ptrdiff_t nt,
                    const int *s0, const int *s1, const int *s2, ptrdiff_t nv, const void *sx, const void *sy,
                    const void *sz, void *out, int *outtri, cudaStream_t stream);
int celllist_edf(int f64, ptrdiff_t npoints, const void *x, const void *y, const void *z, ptrdiff_t nt,
                 const int *s0, const int *s1, const int *s2, ptrdiff_t nv, const void *sx, const void *sy,
                 const void *sz, void *out, int *outtri, cudaStream_t stream);

// ---- box helpers (box_helpers.cu) ----------------------------------------------------------------
// Bounding box of n device points as T (xmin, xmax, ymin, ymax, zmin, zmax into device box6).
template <typename G, typename T>
int points_aabb_device(long long n, const G *x, const G *y, const G *z, T *box6, cudaStream_t stream);
// Signed distance of n device points to the box given as host box6 (|.| when absolute).
template <typename G, typename T>
int points_box_sdf_device(long long n, const G *x, const G *y, const G *z, const T box6[6], int absolute, T *out,
                          cudaStream_t stream);

// ---- level sets and field rebuilds (sdf_rebuild.cu) ----------------------------------------------
// A uniform grid: n[d] samples along axis d at o[d] + i h[d], x fastest (G's o and h, widened).
struct GridDesc {
    long long n[3];
    double o[3], h[3];
};
GridDesc grid_strided(const GridDesc &g, long long stride, bool g64);
GridDesc grid_refined(const GridDesc &g, long long factor, bool g64);
template <typename G, typename T>
int level_set_device(const GridDesc &gd, const T *d_f, T level, long long *ntri, G *x, G *y, G *z, int **d_offsets,
                     cudaStream_t stream);
template <typename G, typename T>
int rebuild_device(const GridDesc &gd, const T *d_f, T level, T band, long long stride, T *d_out, cudaStream_t stream);
template <typename G, typename T>
int refine_device(const GridDesc &gd, const T *d_f, long long factor, T *d_fine, cudaStream_t stream);
template <typename G, typename T>
int round_device(const GridDesc &gd, const T *d_f, T radius, T band, bool open, bool close, long long stride, T *d_out,
                 T *d_f0, cudaStream_t stream);

// Treelet refinement rounds of a resident mesh's BVH (built once, queried many times). Measured on the
// current kernels, queries against 1 round: beam lattice (8e6 points + 512^3 grid, float) 335.6 ->
// 313.1 / 308.7 / 304.8 ms for 2 / 3 / 4 rounds; torus knot 256^3 16.70 -> 16.63 ms (3); 64^3
// icosphere 0.470 -> 0.465 ms; the serving leg's heaviest grid 3.74 -> 3.67 ms. Each round adds
// 0.3 ms to the torus knot's build, which calls that build per query do not repay
// (call_treelet_rounds).
constexpr int kResidentTreeletRounds = 3;

// ---- small helpers -------------------------------------------------------------------------------
inline int grid_blocks(long long n, int threads) { return int((n + threads - 1) / threads); }
// QueryArgs::warp_budget of a launch (or of a batch's jobs) that left it to the default (< 0): a launch or
// batch of n queries, a mesh of T triangles. A packet in a region where every triangle is almost
// equidistant (near a sphere's centre), or of scattered points, sets the launch's tail; handing its
// queries to the warp-per-query stage cuts it. The best budget grows with T, faster on grids, whose packets
// start close together, than on point lists; a launch that fills the GPU several times over repays less of
// a shorter tail and takes a larger one. Measured on B200, us
// without a budget and at 64 / 128 / 256 / 450 / 700 records: 64^3 grid on 5,120 triangles 373: 349 / 247 /
// 284 / 348 / 377; 96^3 on 20,480 1,264: 2,740 / 1,098 / 778 / 754 / 887; 110^3 on 81,920 13,872: 11,175 /
// 4,373 / 2,720 / 2,145 / 2,262; 64^3 around the 131,072-triangle knot 1,021: 3,010 / 2,364 / 1,279 / 876 /
// 807; 500,003 points near it 1,467: 2,579 / 1,360 / 978 / 987 / 1,130; 50,000 1,707: 754 / 712 / 546 / 624 /
// 748; 1,000,000 in its box 2,653: 10,229 / 6,473 / 2,882 / 2,102 / 2,054. Above 2^21 queries: 200^3 on 81,920
// triangles 12,950 without, 7,040 / 6,518 / 6,641 / 7,572 at 500 / 700 / 1,000 / 1,500; 48 uneven meshes,
// 42M queries in one batch, 44.2 ms without, 26.4 at 700; the knot's 256^3 unchanged.
// SSDF_B200_WARP_BUDGET sets it for every launch (0 = no limit), and then nothing below holds packets back.
constexpr int kWarpBudgetMin = 64, kWarpBudgetMax = 700;
constexpr long long kBudgetSmallLaunch = 1ll << 21;
// Largest launch of the plain arithmetics (F64, F32) that keeps a hand-over list, 8 bytes a query.
constexpr long long kHandOverMaxQueries = 1ll << 24;
// How many queries of a launch (of a batch's job) may be handed over (QueryArgs::hand_most). The second stage shares
// no triangle between queries: it is worth its 2 to 5 times a packet's work a query where the GPU would else wait
// for a few packets, and not where most packets run out of budget, as among random overlapping triangles, or far from a
// small mesh, whose packets a warp walk's fixed cost exceeds. Where it pays, few are handed over: up to 12,200 on
// grids of up to 160^3 around spheres, tori and the knot; of points in their boxes 33,000 of 200,000, 82,000 of
// 1,000,000. So 8,192 and a 64th of the launch on meshes below 2,048 triangles, 16,384 and a 64th on other grids,
// 32,768 and a 16th (an 8th from 20,000 triangles on) of other point lists. Without a limit: launches too small to fill the
// GPU either way, and fix-up launches up to 2^21 queries or on larger meshes, whose windows' double evaluations share
// out well (64^3 nodes, 5,120 triangles at 1e4: 7,913 us without a budget, 3,437 with).
// us without a budget, handing over without a limit, and by this rule: 127^3 nodes among 500 random triangles, float
// 1,310 / 6,745 / 1,443; 160^3 among 20,000, fix-up 52,898 / 293,992 / 63,100; 1,000,000 points 30 sizes away from 320
// triangles, float 562 / 1,870 / 609; from 131,072, double 26,689 / 17,321 / 26,421, the one that loses by it.
inline void resolve_hand_over(QueryArgs *a, bool fixup, long long n_launch) {
    a->hand_most = 0x7fffffff;
    if (a->warp_budget >= 0) return;
    const long long n = a->is_grid ? a->nx * a->ny * a->nz : a->npoints;
    const double t = a->m.nt > 0 ? a->m.nt : 0;
    auto within = [](double v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : int(v)); };
    const bool grid = a->is_grid != 0, small = n_launch <= kBudgetSmallLaunch;
    a->warp_budget = small ? within(grid ? t / 40 : 1.2 * std::sqrt(t), kWarpBudgetMin, kWarpBudgetMax)
                           : within(3.0 * std::sqrt(t), 2 * kWarpBudgetMin, 1000);
    const bool few = a->m.nt < 2048;
    if (few ? n_launch <= 1 << 15 : (fixup ? small || a->m.nt > 24576 : n_launch <= (grid ? 1 << 17 : 1 << 16))) return;
    const double base = few ? 8192 : (grid ? 16384 : 32768);
    // a batch's small jobs have their share of the launch's
    const double part = std::max(double(n) / double(n_launch), std::min(1.0, double(n) / 262144.0));
    a->hand_most = int(std::max(1024.0, base * part) +
                       double(n / (few || grid ? 64 : (a->m.nt < 20000 ? 16 : 8))));
}
// Whether a budget can matter on a mesh: a packet tests a triangle at most once.
inline bool budget_reachable(const QueryArgs &a) { return a.warp_budget > 0 && a.m.nt > 4ll * a.warp_budget; }
// Point lists of at least this many queries are visited in Morton order (SSDF_B200_SORT_POINTS=0
// keeps input order).
constexpr long long kSortMinPoints = 4096;
// Point lists of at most this many queries are answered a warp per query (k_query_warp), whose time grows
// with the list (about 12 us per 1,000) where packets' does not until they fill the GPU; the lines cross
// between 16,000 and 40,000 points in every mesh and arithmetic measured (SSDF_B200_WARP_POINTS overrides).
constexpr int kWarpPoints = 24576;
// Morton order of n (< 2^31) points over the mesh's root box: *order (n ints, stream-ordered
// allocation the caller frees with cudaFreeAsync) lists the point indices in key order (bvh_query.cu).
int morton_point_order(long long n, const void *x, const void *y, const void *z, int f64, const float4 *nodes32,
                       int **order, cudaStream_t stream);
int env_int(const char *name, int dflt);
const char *env_str(const char *name);
// Treelet refinement rounds for a mesh that one call builds and queries once (host-array calls, rebuilds,
// pedf): none below 2^21 queries (SSDF_B200_TREELET overrides). The refinement is latency bound (0.3 to 0.5
// ms a round whatever the mesh size) and, with oriented boxes, saves 0-10 % of a query on closed surfaces and 30 %
// on the beam lattice. us without it and with one round: 110^3 grid on 81,920 triangles 2,296 / 2,157, 128^3
// around the knot 2,373 / 2,330, 256^3 10,672 / 10,222, 100,000 points near a torus 425 / 427, 4,000,000 on
// the beam lattice 8,472 / 5,986; a 72^3 field rounded (four rebuilds) 9,588 with it, 4,683 without.
inline int call_treelet_rounds(long long nqueries) {
    return env_int("SSDF_B200_TREELET", nqueries >= (1ll << 21) ? 1 : 0);
}
cudaStream_t library_stream();  // per-thread non-blocking stream for the blocking entry points
void retain_pool_memory();      // keep freed scratch in the device's default pool (once per device)

}  // namespace ssdf_b200

// The handle behind ssdf_mesh* (include/ssdf_b200.h).
struct ssdf_mesh {
    ssdf_b200::DeviceMesh m;
    ssdf_b200::MeshStorage *storage = nullptr;
    int device = 0;
};

namespace ssdf_b200 {
// QueryArgs of one grid / point job (validation shared by the direct and the batch entry points).
int fill_grid_args(ssdf_mesh *mesh, ptrdiff_t nx, ptrdiff_t ny, ptrdiff_t nz, const double lo[3], const double hi[3],
                   void *out, int *outtri, const ssdf_query_opts *opts, QueryArgs *a);
int fill_point_args(ssdf_mesh *mesh, ptrdiff_t npoints, const void *x, const void *y, const void *z, void *out,
                    int *outtri, void *outx, void *outy, void *outz, const ssdf_query_opts *opts, QueryArgs *a);
}  // namespace ssdf_b200

