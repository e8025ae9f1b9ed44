/*
 * Test support (not part of the library): how much of its threshold's allowance the float arithmetic's walk
 * needs. A triangle's oriented box, built as mesh_build.cu's k_obb builds it in the frame of a mesh of half
 * size 1, is restated here with the reference's float distance (device_geom.cuh, tri_dist_sq_exact) and
 * the box distance (obb_pair). The box must be entered while the triangle's own float distance is the best:
 *     box distance < float_box_reach(distance, float_box_margin(c)),   c the mesh's largest coordinate.
 * Triangles lie 1 to 3e5 mesh sizes from the origin, most across the direction to it (where the closest
 * point's rounding adds up), given in floats or doubles; points lie 1e-5 c to 0.06 c off them. Prints the number
 * of cases, of boxes that were not entered, and the largest need: k of (sqrt(distance) + k u c)^2, u = 2^-24.
 *
 * Usage: box_margin_check <cases> <seed>
 */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "box_margin.h"

static uint64_t g_s;
static double uniform(void) {
    g_s ^= g_s << 13, g_s ^= g_s >> 7, g_s ^= g_s << 17;
    return (double)(g_s >> 11) * 0x1p-53;
}
static double normal(void) { return sqrt(-2.0 * log(uniform() + 1e-300)) * cos(6.283185307179586 * uniform()); }

typedef struct {
    float x, y, z;
} V;
static V sub(V a, V b) { return (V){a.x - b.x, a.y - b.y, a.z - b.z}; }
static float dot(V a, V b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }
static V cross(V a, V b) {
    return (V){fmaf(a.y, b.z, -a.z * b.y), fmaf(a.z, b.x, -a.x * b.z), fmaf(a.x, b.y, -a.y * b.x)};
}
static V times(V a, float s) { return (V){a.x * s, a.y * s, a.z * s}; }
static V less(V a, float s, V b) { return (V){fmaf(-s, b.x, a.x), fmaf(-s, b.y, a.y), fmaf(-s, b.z, a.z)}; }

static float dot3(const float *a, const float *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
static float distance_sq(const float *p, const float *a, const float *b, const float *c) {
    float ab[3], ac[3], ap[3], bp[3], cp[3], d[3];
    for (int k = 0; k < 3; k++)
        ab[k] = b[k] - a[k], ac[k] = c[k] - a[k], ap[k] = p[k] - a[k], bp[k] = p[k] - b[k], cp[k] = p[k] - c[k];
    const float d1 = dot3(ab, ap), d2 = dot3(ac, ap);
    if (d1 <= 0 && d2 <= 0) return dot3(ap, ap);
    const float d3 = dot3(ab, bp), d4 = dot3(ac, bp);
    if (d3 >= 0 && d4 <= d3) return dot3(bp, bp);
    const float vc = d1 * d4 - d3 * d2;
    if (vc <= 0 && d1 >= 0 && d3 <= 0) {
        const float v = d1 / (d1 - d3);
        for (int k = 0; k < 3; k++) d[k] = p[k] - (a[k] + v * ab[k]);
        return dot3(d, d);
    }
    const float d5 = dot3(ab, cp), d6 = dot3(ac, cp);
    if (d6 >= 0 && d5 <= d6) return dot3(cp, cp);
    const float vb = d5 * d2 - d1 * d6;
    if (vb <= 0 && d2 >= 0 && d6 <= 0) {
        const float w = d2 / (d2 - d6);
        for (int k = 0; k < 3; k++) d[k] = p[k] - (a[k] + w * ac[k]);
        return dot3(d, d);
    }
    const float va = d3 * d6 - d5 * d4;
    if (va <= 0 && (d4 - d3) >= 0 && (d5 - d6) >= 0) {
        const float w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        for (int k = 0; k < 3; k++) d[k] = p[k] - (b[k] + w * (c[k] - b[k]));
        return dot3(d, d);
    }
    const float denom = 1.f / (va + vb + vc), v = vb * denom, w = vc * denom;
    for (int k = 0; k < 3; k++) d[k] = p[k] - (a[k] + ab[k] * v + ac[k] * w);
    return dot3(d, d);
}

int main(int argc, char **argv) {
    const long cases = argc > 1 ? atol(argv[1]) : 1000000;
    g_s = 88172645463325252ull ^ (argc > 2 ? strtoull(argv[2], 0, 10) * 0x9e3779b97f4a7c15ull : 0);
    long done = 0, left_out = 0;
    double worst = -1.0;
    for (long i = 0; i < cases; i++) {
        const int doubles = uniform() < 0.5;
        const double place = pow(2.0, 18.0 * uniform()), size = pow(2.0, -4.0 * uniform());
        double off[3], n[3], t[3][3];
        for (int k = 0; k < 3; k++) off[k] = place * (uniform() < 0.5 ? 1 : -1) * (uniform() < 0.8 ? 1.0 : uniform());
        const int across = uniform() < 0.9;
        for (int k = 0; k < 3; k++) n[k] = across ? copysign(1.0, off[k]) : normal();
        const double nn = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
        for (int v = 0; v < 3; v++) {
            double q[3], along = 0.0;
            for (int k = 0; k < 3; k++) q[k] = size * 0.4 * normal(), along += q[k] * n[k];
            for (int k = 0; k < 3; k++) t[v][k] = off[k] + q[k] - along * n[k] / nn;
        }
        float f[3][3], mid[3], c = 0.f;
        for (int v = 0; v < 3; v++)
            for (int k = 0; k < 3; k++) {
                f[v][k] = (float)t[v][k];
                if (!doubles) t[v][k] = f[v][k];
            }
        for (int k = 0; k < 3; k++) {
            c = fmaxf(c, (float)(fabs(off[k]) + 1.0));
            mid[k] = (float)(off[k] + 0.5 * (2.0 * uniform() - 1.0));
        }
        V w[3];
        for (int v = 0; v < 3; v++)
            w[v] = (V){(float)(t[v][0] - mid[0]), (float)(t[v][1] - mid[1]), (float)(t[v][2] - mid[2])};
        const V e1 = sub(w[1], w[0]), e2 = sub(w[2], w[0]), e3 = sub(w[2], w[1]);
        V z = cross(e1, e2);
        const float l2 = fmaxf(dot(e1, e1), fmaxf(dot(e2, e2), dot(e3, e3))), alpha = l2 / sqrtf(dot(z, z));
        if (!(alpha <= 2048.f)) continue;
        z = times(z, 1.f / sqrtf(dot(z, z)));
        V d = less(e1, dot(e1, z), z);
        d = times(d, 1.f / sqrtf(dot(d, d)));
        d = less(d, dot(d, z), z);
        d = times(d, 1.f / sqrtf(dot(d, d)));
        V axis[3] = {d, cross(z, d), z};
        const float pad = 0x1p-18f + 128.f * 0x1p-24f * alpha * sqrtf(l2) * 1.001f;
        const float s = (1.f - 0x1p-18f) / (1.f + 128.f * 0x1p-24f * alpha);
        float half[3], at[3];
        for (int a = 0; a < 3; a++) {
            float lo = INFINITY, hi = -INFINITY;
            for (int v = 0; v < 3; v++) {
                const float x = dot(axis[a], sub(w[v], w[0]));
                lo = fminf(lo, x), hi = fmaxf(hi, x);
            }
            half[a] = (0.5f * (hi - lo) + pad) * s;
            at[a] = -(dot(axis[a], w[0]) + 0.5f * (lo + hi)) * s;
            axis[a] = times(axis[a], s);
        }
        const double away = c * pow(2.0, -4.0 - 12.0 * uniform()) * (uniform() < 0.5 ? 1 : -1);
        double b0 = uniform(), b1 = uniform();
        if (b0 + b1 > 1.0) b0 = 1.0 - b0, b1 = 1.0 - b1;
        float p[3];
        for (int k = 0; k < 3; k++)
            p[k] = (float)(t[0][k] + b0 * (t[1][k] - t[0][k]) + b1 * (t[2][k] - t[0][k]) + away * n[k] / sqrt(nn) +
                           0.1 * size * normal() * (i % 4 == 0));
        const float d2 = distance_sq(p, f[0], f[1], f[2]);
        if (!(d2 < INFINITY)) continue; /* corners that collapsed: no distance, never the best */
        const V b = {p[0] - mid[0], p[1] - mid[1], p[2] - mid[2]};
        float box = 0.f;
        for (int a = 0; a < 3; a++) {
            const float x = fmaf(axis[a].x, b.x, fmaf(axis[a].y, b.y, fmaf(axis[a].z, b.z, at[a])));
            const float e = fmaxf(fabsf(x) - half[a], 0.f);
            box = a ? fmaf(e, e, box) : e * e;
        }
        const float margin = float_box_margin(c);
        done++;
        left_out += !(box < float_box_reach(d2, margin));
        if (box >= (d2 + margin * margin) * (1.f + 0x1p-16f))  // else the near margin alone admits it
            worst = fmax(worst, (sqrt(box / (1.0 + 0x1p-16)) - sqrt((double)d2)) / (0x1p-24 * c));
    }
    printf("cases %ld left_out %ld largest_need %.3f\n", done, left_out, worst);
    return 0;
}
