// celllist.cu -- ssdf::edf_celllist on the GPU.
//
// The reference bins the triangles in a 2-D cell list so that a point need not test them all
// (serial/ssdf.hpp:642-963); its value is the brute-force minimum. Here the structure that saves the tests
// is the library's tree of oriented boxes, built for the call, and the query is the library's point query:
// bitwise the reference's value in T's arithmetic, the closest triangle the lowest index at the minimum.
// A cell list of the reference's shape, walked in rings around each point, took 4.6 ms for 150,001 points on
// a 5,120-triangle sphere (3.3x the pairs' tests of the tree, points in input order); this takes 0.73 ms, the
// build included. Few pairs are cheaper without any structure (few_pairs).
#include <cuda_runtime.h>

#include "internal.h"

namespace ssdf_b200 {

namespace {

// The brute force is faster than building a tree (about 300 us) for few pairs on few triangles: 2,000 points on
// 5,120 triangles, 10M pairs, 384 us against 403 in double and 233 against 383 in float; 20,000 on 1,280,
// 26M pairs, 510 / 447 and 350 / 396; 500 on 20,480, 10M pairs in long rows, 807 / 465 and 499 / 443.
inline bool few_pairs(int f64, long long npoints, long long nt) {
    return nt <= 8192 && npoints <= (f64 ? 10000000ll : 24000000ll) / nt;
}

struct MeshInStreamOrder {
    ssdf_mesh mesh;
    cudaStream_t stream;
    ~MeshInStreamOrder() { mesh_free_async(mesh.storage, stream); }
};

}  // namespace

int celllist_edf(int f64, ptrdiff_t npoints, const void *x, const void *y, const void *z, ptrdiff_t nt,
                 const int *s0, const int *s1, const int *s2, ptrdiff_t nv, const void *sx, const void *sy,
                 const void *sz, void *out, int *outtri, cudaStream_t stream) {
    if (npoints <= 0 || nt <= 0 || nv <= 0) return SSDF_OK;
    if (npoints > 0x7fffffff || nt > kMaxTriangles)
        return fail(SSDF_ERR_NOT_SUPPORTED, "cell-list edf: too many points or triangles for one launch");
    if (few_pairs(f64, npoints, nt))
        return brute_force_edf(f64, npoints, x, y, z, nt, s0, s1, s2, nv, sx, sy, sz, out, outtri, stream);
    ssdf_build_opts bo;
    bo.leaf_size = 0, bo.keep_fp64 = f64, bo.normals = 0;
    bo.treelet_opt = call_treelet_rounds(npoints);
    MeshInStreamOrder h{{}, stream};
    cudaGetDevice(&h.mesh.device);
    SSDF_CHECK(mesh_build(&h.mesh.storage, &h.mesh.m, nt, s0, s1, s2, nv, sx, sy, sz, f64, /*device_ptrs=*/1, bo,
                          stream));
    ssdf_query_opts qo{};
    // (a fix-up launch takes one query less than this call)
    qo.precision = !f64 ? SSDF_PREC_F32 : (npoints < 0x7fffffff ? SSDF_PREC_F32_FIXUP : SSDF_PREC_F64);
    qo.output = SSDF_OUT_EDF;
    qo.coord_type = qo.out_type = f64 ? SSDF_F64 : SSDF_F32;
    QueryArgs a;
    SSDF_CHECK(fill_point_args(&h.mesh, npoints, x, y, z, out, outtri, nullptr, nullptr, nullptr, &qo, &a));
    SSDF_CHECK(launch_query(a, qo.precision, stream));
    SSDF_CUDA(cudaStreamSynchronize(stream));
    return SSDF_OK;
}

}  // namespace ssdf_b200
