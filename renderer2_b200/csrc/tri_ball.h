// The filter's test of triangles against the balls that hold a voxel's rays.
#pragma once
#include <math.h>

#include "r2_core.h"

namespace r2 {

R2_HD float ball_rcp(float x) {
#if defined(__CUDA_ARCH__)
  return __frcp_rn(x);
#else
  return 1.0f / x;
#endif
}

// Tests of one triangle against balls of radius r whose centres lie within
// `around` of c0.  near() is false only when the ball cannot touch the
// triangle: it is out of reach of the plane, or of all three edges while its
// centre projects outside the triangle.  The radius grows by 2e-6 of the
// vertices' distances, more than the rounding of the products; the plane and
// the side tests give way by the rounding of their cross products, so a sliver
// whose normal is only rounding is left to its edges, and a NaN rejects
// nothing.  The normal is held times `scale`, a power of two near 1 over the square
// of the voxels' size (ball_scale): unscaled, products of the fourth power of an edge
// left the range of a float where edges were beyond 4e9 or below 1e-11.
struct TriBall {
  V3 p0, p1, AB, BC, AC, n, m0, m1, m2;  // vertices, edges, scaled normal, the edges' outward normals
  float i0, i1, i2;                      // 1 / squared edge lengths (0 for an edge without length)
  float rr, plane, side;                 // squared padded radius; bounds of the plane and the side tests
};
R2_HD TriBall tri_ball(V3 p0, V3 p1, V3 p2, V3 c0, float around, float r, float scale) {
  TriBall t;
  t.p0 = p0;
  t.p1 = p1;
  t.AB = p1 - p0;
  t.BC = p2 - p1;
  t.AC = p2 - p0;
  const V3 a = vabs(p0 - c0), b = vabs(p1 - c0), c = vabs(p2 - c0);
  const float far = fmaxf(fmaxf(a.x + a.y + a.z, b.x + b.y + b.z), c.x + c.y + c.z) + around;
  const float rp = r + 2e-6f * far;
  t.rr = rp * rp;
  const float e0 = dot(t.AB, t.AB), e1 = dot(t.BC, t.BC), e2 = dot(t.AC, t.AC);
  t.i0 = e0 > 1e-30f ? ball_rcp(e0) : 0.0f;
  t.i1 = e1 > 1e-30f ? ball_rcp(e1) : 0.0f;
  t.i2 = e2 > 1e-30f ? ball_rcp(e2) : 0.0f;
  t.n = cross(t.AB, t.AC) * scale;
  t.m0 = cross(t.AB, t.n);
  t.m1 = cross(t.BC, t.n);
  t.m2 = cross(t.n, t.AC);
  const float area = e0 + e1 + e2;  // more than |AB| |AC|
  t.plane = rp * sqrtf(dot(t.n, t.n)) + 2e-6f * (far + rp) * (area * scale);
  t.side = 4e-6f * far * (area * scale) * sqrtf(area);
  return t;
}
R2_HD float edge_dist2(V3 a, V3 e, float inv) {  // of the origin from the edge a + [0, 1] e
  const V3 q = a + e * clampf(-dot(a, e) * inv, 0.0f, 1.0f);
  return dot(q, q);
}
R2_HD bool tri_near(const TriBall& t, V3 c) {
  const V3 A = t.p0 - c, B = t.p1 - c;
  const float d2 = fminf(fminf(edge_dist2(A, t.AB, t.i0), edge_dist2(B, t.BC, t.i1)), edge_dist2(A, t.AC, t.i2));
  // the centre lies outside an edge where its outward normal points back to the edge's vertex
  const float out = fminf(fminf(dot(A, t.m0), dot(B, t.m1)), dot(A, t.m2));
  return !(fabsf(dot(A, t.n)) > t.plane) && (!(d2 > t.rr) || !(out < -t.side));
}

// The scale for voxels of the given size: 2^-2k with 2^k near it, k within +-50.
inline float ball_scale(float voxel) {
  int e = 0;
  frexpf(voxel, &e);
  return ldexpf(1.0f, -2 * (e < -50 ? -50 : (e > 50 ? 50 : e)));
}

}  // namespace r2
