// bvh_margin.hpp — how far the traversal tree's leaf boxes reach past their triangles.
//
// The reference expands every triangle box by 1e-3 (bounding_box.h:30-37), and any tree whose boxes
// hold every hit that the triangle test accepts returns the same hits.  In a fine mesh that margin is
// a quarter of a triangle on every side (the caustic workload's water: triangles of 1/256), so a ray
// through it visits about twice the leaves it needs.  The margin a triangle needs follows from the
// test's rounding: with u = 2^-24, an accepted hit has |a| >= EPS = 1e-5, a = e1 . (d x e2), and
//   * each barycentric numerator, a dot product of s = o - v0 with a cross product, is off by at most
//     8u |s| e (|d| = 1, e the longest edge), a itself by 7u e^2, so the accepted point lies within
//     e * (8u |s| e + 7u e^2) / EPS of the triangle, and t is off by at most 8u |s| e^2 / EPS;
//   * a slab distance (one fused multiply-add on a rounded product) places a plane to within a few
//     u times the coordinates.
// With every vertex and every ray origin within S of zero in each coordinate, |s| and e are at most
// 3.5 S, and all of it is below 128 u S (1 + e^2 / EPS).  The margin is that, and never more than the
// reference's 1e-3: a large or far-away triangle keeps 1e-3.
//
// Measured (B200, 1024 x 1024 caustic workload, S = 2.4, water margin 8e-5): shadow stage 6.5 -> 5.4 ms,
// photon kernel 3.8 -> 3.2 ms, camera kernel 0.90 -> 0.75 ms a round.  The atrium's triangles (edges of
// about 0.05 at S = 14) keep 1e-3 and their times.
#pragma once

#if defined(__CUDACC__)
#define PHX_MARGIN_FN __host__ __device__ inline
#else
#define PHX_MARGIN_FN inline
#endif

namespace phx {

constexpr float BBOX_EPS = 1e-3f; // bounding_box.h expansion

// unit: 128 u S of the scene (tight_margin_unit), or 0 for the reference's margin
PHX_MARGIN_FN float box_margin(const float v[3][3], float unit) {
    if (!(unit > 0.0f))
        return BBOX_EPS;
    float e2 = 0.0f;
    for (int k = 0; k < 3; k++) {
        float l = 0.0f;
        for (int a = 0; a < 3; a++) {
            const float d = v[(k + 1) % 3][a] - v[k][a];
            l = l + d * d;
        }
        e2 = l > e2 ? l : e2;
    }
    const float m = unit * (1.0f + e2 * 1e5f);
    return m < BBOX_EPS ? m : BBOX_EPS;
}

PHX_MARGIN_FN float tight_margin_unit(float s) { return s * (128.0f / 16777216.0f); }

} // namespace phx
