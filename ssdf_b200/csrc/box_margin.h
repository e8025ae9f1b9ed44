// box_margin.h -- how far above the best float distance a box may lie and still be entered.
//
// SSDF_PREC_F32 compares the reference's float squared distances, which lie off the true ones, so a walk
// must enter every box that can hold a triangle whose float distance is the best or ties with it. With
// u = 2^-24, c the largest coordinate magnitude of the mesh, d the distance, L the triangle's longest edge:
// - The region tests and barycentric coordinates err by lengths of the triangle, which the boxes' own
//   margins cover (mesh_build.cu, above k_obb).
// - The closest point is formed at the triangle's place: a + v ab + w ac takes two sums, u c an axis each,
//   2 sqrt(3) u c = 3.5 u c together (edges and products round by 3.5 u L, which the boxes' margins have to spare).
//   An axis-aligned box of the float corners holds the rounded point all the same, because rounding is
//   monotone; an oriented box does not.
// - The boxes hold the mesh's vertices, which may be doubles; the triangles' corners are those rounded to
//   float: sqrt(3) u c = 1.7 u c.
// - Differences, squares and sums of p less the closest point are relative, 2.5 u d: below 1 + 2^-16.
// 5.2 u c in all; the threshold allows 8 u c. (2 u c lost ties on meshes far from the origin.)
// tests/box_margin_check.c looks for the largest need. Plain C, for that check.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define SSDF_BOX_MARGIN_FN __host__ __device__ __forceinline__
#else
#define SSDF_BOX_MARGIN_FN static inline
#endif

// c as float_box_reach takes it. Squares below the smallest normal float are not relative: at least 2^-63, the root
// of that number, which is as near as the float arithmetic tells distances apart.
SSDF_BOX_MARGIN_FN float float_box_margin(float c) { return fmaxf(c * 0x1p-16f, 0x1p-63f); }

// The squared distance below which a box is entered: (sqrt(best) + 8 u c)^2, and at least best + (2^-16 c)^2.
SSDF_BOX_MARGIN_FN float float_box_reach(float best, float margin) {
    const float d = sqrtf(best) + 0x1p-5f * margin;
    return fmaxf(d * d, best + margin * margin) * (1.0f + 1.0f / 65536.0f);
}

// The same, in a box frame of scale s, where no distance is known: a box farther than this holds no triangle
// whose float squared distance is finite (below 2^128).
SSDF_BOX_MARGIN_FN float float_box_limit(float margin, float s) {
    const float d = (0x1p64f + 0x1p-5f * margin) * s;
    return d * d * (1.0f + 1.0f / 65536.0f);
}
