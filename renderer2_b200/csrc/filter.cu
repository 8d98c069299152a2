// SGGX mesh-to-volume filter kernels for sm_100a.
//
// Reference path: __raygen__filtering (raytracer/src/backend/shaders.optix.cu:258-284)
// launches one OptiX thread per voxel running CMeshFilter::run
// (raytracer/include/filtering/mesh_filter.hpp:51-122) and estimateDensity (182-204).
//
// B200 design, three kernels per part of the grid:
//  * k_filter_classify (large grids): one thread per brick of 2x2x2 voxels
//    lists the bricks whose bounding box overlaps a triangle's box.
//  * k_filter_lists: one warp per brick walks the BVH once, 32 nodes at a time,
//    and finds for each of the eight voxels the triangles that can touch the
//    ball that holds all of its rays (its centre and 1.1 * |voxelSize| / 2 with
//    ClipRays).  A voxel without any has zero hits for certain and gets the
//    empty payload; the others go to a work list, their candidates to a pool.
//  * k_filter_sample: a persistent kernel; each warp takes one voxel at a time
//    from the work list and its 32 lanes trace the voxel's samples (lane l owns
//    samples l, l+32, ...) against the candidates, the lanes in step.  Voxels
//    with more than kCandMax candidates trace through the BVH from the deepest
//    node that holds them.  Sums are compensated per lane and across the warp.
//    The density fit runs its iterations as warp reductions.
// The sampling kernel issues an instruction in 79 % of the cycles; what it
// waits for is instruction fetch, so its code is kept small: unrolling the
// triangle loop twice took the 256^3 filter (1M triangles, 256 samples) from
// 178 to 237 ms when it was tried.  That filter took 314 ms when each voxel
// walked the BVH by itself, a node at a time, inside the sampling kernel and
// tested the triangles whose boxes overlap the ball's box (8.5 per ray over
// 12.0M voxels); with the ball test, the lists and the smaller kernel (4.6 per
// ray over 6.5M voxels) it takes 95 ms, 16 of them for the lists.
#include "filter.cuh"
#include "filter_math.h"
#include "texture_shade.cuh"
#include "tri_ball.h"

namespace r2 {
namespace {

constexpr int kSampleWarps = 4;  // warps per block of the list and sampling kernels
// Candidate triangles of a brick or a voxel tested without the BVH.  128 / 192 /
// 256 / 512: 256^3 filter of 1M leaf triangles 111.8 / 102.7 / 102.7 / 103.3 ms,
// 24x77x24 voxels of a 40,000-triangle tree 0.99 / 1.01 / 1.02 / 1.27 ms.
constexpr int kCandMax = 256;
constexpr int kCandStage = 40;   // candidates of a voxel whose vertices a warp copies into shared memory
constexpr int kWalkStack = 256;  // nodes waiting in the candidate walk
constexpr int kWalkInts = kWalkStack + 96;  // and its leaves: under 32 kept, up to 64 more in a step
static_assert(kWalkInts * sizeof(int) <= kCandStage * 9 * sizeof(float), "the walk's scratch lies where the staged vertices go");
// Up to so many bricks a resident warp are walked without k_filter_classify: on
// 32^3 voxels its launch alone took 44 us against 27 us for walking every brick;
// on a 256^3 grid it takes 1.4 ms and spares the walks of a quarter of the bricks.
constexpr uint32_t kListAll = 16;
static_assert(kCandStage * 9 * sizeof(float) % 16 == 0 && kCandMax * sizeof(int) % 16 == 0, "a warp's shared memory is counted in 16 bytes");
// Candidates from which a voxel is sampled among the first (the 48^3 grid of
// 400,000 triangles 2.49 ms in any order, 2.12 ms with these first).
constexpr int kLongList = 96;
constexpr uint32_t kNoList = 0xFFFFFFFFu;  // a voxel that k_filter_sample walks the BVH for

// Dynamic shared memory of a sampling block, per warp: the staged candidate
// vertices (kCandStage x 9 floats; the candidate walk and the voxel's sums use
// the place before and after), the candidate list (kCandMax ints), the
// samples' hit lengths (spv floats).
__host__ __device__ constexpr size_t sample_smem_per_warp(uint32_t spv) {
  return (size_t)kCandStage * 9 * sizeof(float) + (size_t)kCandMax * sizeof(int) +
         ((size_t)spv * sizeof(float) + 15) / 16 * 16;
}

// How far from the voxel's centre its rays reach: with ClipRays a ray ends on
// the bounding sphere; otherwise it starts anywhere in the voxel and runs
// voxelSize.x (mesh_filter.hpp:72-82).
__device__ __forceinline__ float ray_reach(const FilterLaunch& L) {
  return L.clip ? 1.1f * length(L.voxelSize) / 2.0f : length(L.voxelSize) / 2.0f + L.voxelSize.x;
}

__device__ __forceinline__ V3 voxel_center(const FilterLaunch& L, int x, int y, int z) {
  V3 pm = xform_point(L.indexToModel, v3((float)x + 0.5f, (float)y + 0.5f, (float)z + 0.5f));
  return xform_point(L.modelToWorld, pm);
}

// The reach of a voxel's rays from its centre c, padded for their rounding.
__device__ __forceinline__ float padded_reach(float reach, V3 c) {
  return reach * 1.01f + 1e-5f * (fabsf(c.x) + fabsf(c.y) + fabsf(c.z) + 1.0f);
}

// A brick of 2x2x2 voxels (at the grid's end some of them lie outside): its
// first voxel and a ball that holds the padded balls of its voxels' rays.
struct Brick {
  int x, y, z;
  V3 center;
  float r;
};
__device__ __forceinline__ Brick brick_at(const FilterLaunch& L, uint32_t id) {
  const uint32_t mx = (uint32_t)(L.nx + 1) / 2, my = (uint32_t)(L.ny + 1) / 2;
  const uint32_t row = id / mx, slice = row / my;
  Brick k;
  k.x = (int)(id - row * mx) * 2;
  k.y = (int)(row - slice * my) * 2;
  k.z = (int)slice * 2;
  k.center = (voxel_center(L, k.x, k.y, k.z) + voxel_center(L, k.x + 1, k.y + 1, k.z + 1)) * 0.5f;
  k.r = padded_reach(ray_reach(L) + L.brickOffset, k.center) +
        1e-6f * (fabsf(k.center.x) + fabsf(k.center.y) + fabsf(k.center.z));
  return k;
}

// A brick's v-th voxel, v < 8; false if it lies outside the grid.
__device__ __forceinline__ bool brick_voxel(const FilterLaunch& L, const Brick& k, int v, int* x, int* y, int* z) {
  *x = k.x + (v & 1);
  *y = k.y + ((v >> 1) & 1);
  *z = k.z + (v >> 2);
  return *x < L.nx && *y < L.ny && *z < L.nz;
}
__device__ __forceinline__ size_t voxel_index(const FilterLaunch& L, int x, int y, int z) {
  return (size_t)x + ((size_t)y + (size_t)z * L.ny) * L.nx;
}

__device__ __forceinline__ bool box_overlap(float lox, float hix, float loy, float hiy, float loz,
                                            float hiz, V3 qlo, V3 qhi) {
  return !(lox > qhi.x || hix < qlo.x || loy > qhi.y || hiy < qlo.y || loz > qhi.z || hiz < qlo.z);
}

__device__ __forceinline__ TriBall load_tri_ball(const FilterLaunch& L, int t, V3 c0, float around, float r) {
  const float4 a = __ldg(&L.bvh.tris[3 * t]), b = __ldg(&L.bvh.tris[3 * t + 1]), c = __ldg(&L.bvh.tris[3 * t + 2]);
  return tri_ball(v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), c0, around, r, L.ballScale);
}

// Does any triangle box overlap the query box?
__device__ bool bvh_any_box(const BvhView& bvh, V3 qlo, V3 qhi) {
  int stack[R2_BVH_STACK];
  int sp = 0;
  int cur = 0;
  while (true) {
    if (cur >= 0) {
      const BvhNode* nd = &bvh.nodes[cur];
      float4 b0 = __ldg(&nd->b0), b1 = __ldg(&nd->b1), bz = __ldg(&nd->bz);
      int4 ch = __ldg(&nd->ch);
      bool h0 = box_overlap(b0.x, b0.y, b0.z, b0.w, bz.x, bz.y, qlo, qhi);
      bool h1 = ch.y != R2_BVH_NONE && box_overlap(b1.x, b1.y, b1.z, b1.w, bz.z, bz.w, qlo, qhi);
      if (h0 && h1) {
        stack[sp++] = ch.y;
        cur = ch.x;
        continue;
      } else if (h0) {
        cur = ch.x;
        continue;
      } else if (h1) {
        cur = ch.y;
        continue;
      }
    } else {
      int first = bvh_leaf_first(cur), count = bvh_leaf_count(cur);
      for (int i = 0; i < count; ++i) {
        int t = first + i;
        float4 a = __ldg(&bvh.tris[3 * t]), b = __ldg(&bvh.tris[3 * t + 1]), c = __ldg(&bvh.tris[3 * t + 2]);
        float lx = fminf(fminf(a.x, b.x), c.x), hx = fmaxf(fmaxf(a.x, b.x), c.x);
        float ly = fminf(fminf(a.y, b.y), c.y), hy = fmaxf(fmaxf(a.y, b.y), c.y);
        float lz = fminf(fminf(a.z, b.z), c.z), hz = fmaxf(fmaxf(a.z, b.z), c.z);
        if (box_overlap(lx, hx, ly, hy, lz, hz, qlo, qhi)) return true;
      }
    }
    if (sp == 0) return false;
    cur = stack[--sp];
  }
}

// The deepest node whose subtree holds every leaf whose box overlaps the
// query box: descend while exactly one child's box overlaps it.  A leaf that
// a ray confined to the query box can hit overlaps it, and so does every box
// above that leaf, so a traversal started here finds the same closest hit as
// one started at the root.
__device__ int bvh_local_root(const BvhView& bvh, V3 qlo, V3 qhi) {
  int cur = 0;
  for (int depth = 0; depth < R2_BVH_STACK && cur >= 0; ++depth) {
    const BvhNode* nd = &bvh.nodes[cur];
    const float4 b0 = __ldg(&nd->b0), b1 = __ldg(&nd->b1), bz = __ldg(&nd->bz);
    const int4 ch = __ldg(&nd->ch);
    const bool h0 = box_overlap(b0.x, b0.y, b0.z, b0.w, bz.x, bz.y, qlo, qhi);
    const bool h1 = ch.y != R2_BVH_NONE && box_overlap(b1.x, b1.y, b1.z, b1.w, bz.z, bz.w, qlo, qhi);
    if (h0 == h1) return cur;  // both children (or neither): start here
    cur = h0 ? ch.x : ch.y;
  }
  return cur;
}

// The triangles of up to 32 leaves, one leaf per lane (refs[lane], lane < n),
// that can touch the ball: appended to list, the lanes' first triangles, then
// their second ones, and so on.  Returns the list's new length, or -1 when it
// would pass kCandMax.
__device__ __forceinline__ int near_triangles(const FilterLaunch& L, const int* refs, int n, V3 qlo, V3 qhi, V3 center,
                                              float r, int* list, int len, int lane) {
  const int ref = lane < n ? refs[lane] : 0;
  const int first = bvh_leaf_first(ref), count = lane < n ? bvh_leaf_count(ref) : 0;
  for (int k = 0; __any_sync(0xFFFFFFFFu, k < count); ++k) {
    bool near = false;
    if (k < count) {
      const int t = first + k;
      const float4 a = __ldg(&L.bvh.tris[3 * t]), b = __ldg(&L.bvh.tris[3 * t + 1]), c = __ldg(&L.bvh.tris[3 * t + 2]);
      near = box_overlap(fminf(fminf(a.x, b.x), c.x), fmaxf(fmaxf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y),
                         fmaxf(fmaxf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z), fmaxf(fmaxf(a.z, b.z), c.z), qlo,
                         qhi) &&
             tri_near(tri_ball(v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), center, 0.0f, r, L.ballScale),
                      center);
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, near);
    const int added = __popc(m);
    if (len + added > kCandMax) return -1;
    if (near) list[len + __popc(m & ((1u << lane) - 1u))] = first + k;
    len += added;
  }
  return len;
}

// The candidate triangles of a brick of voxels: every triangle that can touch
// the ball of radius r about center, which holds every sample ray of the
// brick, so these are all the triangles its rays can hit.  The warp walks the
// BVH together from the root: each step takes up to 32 nodes off a stack in
// shared memory, one per lane, and puts the children whose boxes overlap the
// ball's box [qlo, qhi] back with ballots, leaves on a list of their own that
// is worked off 32 at a time.  A walk of 100 nodes is then about 15 dependent
// fetches (the tree's depth) and not 100.  scratch: kWalkInts ints.  Returns
// the number of candidates, or -1 when there are more than kCandMax or the
// stack is full.  nodes: inner nodes visited by this lane (the counting build).
__device__ int gather_candidates(const FilterLaunch& L, V3 qlo, V3 qhi, V3 center, float r, int* list, int* scratch,
                                 int lane, uint32_t* nodes) {
  int* stack = scratch;
  int* leaves = scratch + kWalkStack;
  int sp = 1, nleaf = 0, len = 0;
  if (lane == 0) stack[0] = 0;
  __syncwarp();
  const unsigned below = (1u << lane) - 1u;
  while (sp > 0) {
    const int take = min(sp, 32);
    sp -= take;
    int c0 = R2_BVH_NONE, c1 = R2_BVH_NONE;
    if (lane < take) {
      ++*nodes;
      const BvhNode* nd = &L.bvh.nodes[stack[sp + lane]];
      const float4 b0 = __ldg(&nd->b0), b1 = __ldg(&nd->b1), bz = __ldg(&nd->bz);
      const int4 ch = __ldg(&nd->ch);
      if (box_overlap(b0.x, b0.y, b0.z, b0.w, bz.x, bz.y, qlo, qhi)) c0 = ch.x;
      if (ch.y != R2_BVH_NONE && box_overlap(b1.x, b1.y, b1.z, b1.w, bz.z, bz.w, qlo, qhi)) c1 = ch.y;
    }
    const unsigned i0 = __ballot_sync(0xFFFFFFFFu, c0 >= 0), i1 = __ballot_sync(0xFFFFFFFFu, c1 >= 0);
    const unsigned l0 = __ballot_sync(0xFFFFFFFFu, c0 < 0 && c0 != R2_BVH_NONE);
    const unsigned l1 = __ballot_sync(0xFFFFFFFFu, c1 < 0 && c1 != R2_BVH_NONE);
    if (sp + __popc(i0) + __popc(i1) > kWalkStack) return -1;
    if (c0 >= 0) stack[sp + __popc(i0 & below)] = c0;
    else if (c0 != R2_BVH_NONE) leaves[nleaf + __popc(l0 & below)] = c0;
    sp += __popc(i0);
    nleaf += __popc(l0);
    if (c1 >= 0) stack[sp + __popc(i1 & below)] = c1;
    else if (c1 != R2_BVH_NONE) leaves[nleaf + __popc(l1 & below)] = c1;
    sp += __popc(i1);
    nleaf += __popc(l1);
    __syncwarp();
    while (nleaf >= 32 || (sp == 0 && nleaf > 0)) {
      const int n = min(nleaf, 32);
      nleaf -= n;
      len = near_triangles(L, leaves + nleaf, n, qlo, qhi, center, r, list, len, lane);
      if (len < 0) return -1;
    }
  }
  return len;
}

// Two floats in one 64-bit register pair: sm_100's packed additions
// round each half like the scalar ones and issue once for both.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float lo(F2 a) { return __uint_as_float((unsigned)a.v); }
__device__ __forceinline__ float hi(F2 a) { return __uint_as_float((unsigned)(a.v >> 32)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

// The closest hit of one ray among the candidate triangles list[0 .. n-1],
// with tri_test's arithmetic and (t, triangle) order: the same hit as
// bvh_trace over the whole scene.  Every lane walks the same list.  A vertex's
// coordinates are fetched in the ray's axis order (three words of three banks,
// so a warp reads them at once), which saves tri_test's 18 selects a triangle;
// tri_test also swaps the first two axes of rays against the third, which only
// changes the sign of U, V, W, det and T and none of t, b1 and b2.
template <bool kAlpha>
__device__ __forceinline__ Hit trace_candidates(const BvhView& bvh, const int* list, int n, const float* staged,
                                                V3 o, V3 d, float tmax) {
  const V3 ad = vabs(d);
  const int kz = (ad.x > ad.y) ? ((ad.x > ad.z) ? 0 : 2) : ((ad.y > ad.z) ? 1 : 2);
  const int kx = kz == 2 ? 0 : kz + 1, ky = kx == 2 ? 0 : kx + 1;
  const float dz = comp(d, kz);
  const float Sx = comp(d, kx) / dz, Sy = comp(d, ky) / dz, Sz = 1.0f / dz;
  const F2 oxy = f2(comp(o, kx), comp(o, ky));
  const float oz = comp(o, kz);
  Hit best;
  best.t = tmax;
  best.b1 = best.b2 = 0.0f;
  best.tri = -1;  // place in the list
#pragma unroll 1
  for (int c = 0; c < n; ++c) {
    float Ax, Ay, Az0, Bx, By, Bz0, Cx, Cy, Cz0;
    if (c < kCandStage) {
      const float* v = staged + 9 * c;
      Ax = v[kx]; Ay = v[ky]; Az0 = v[kz];
      Bx = v[3 + kx]; By = v[3 + ky]; Bz0 = v[3 + kz];
      Cx = v[6 + kx]; Cy = v[6 + ky]; Cz0 = v[6 + kz];
    } else {
      const float* v = reinterpret_cast<const float*>(bvh.tris + 3 * list[c]);
      Ax = __ldg(v + kx); Ay = __ldg(v + ky); Az0 = __ldg(v + kz);
      Bx = __ldg(v + 4 + kx); By = __ldg(v + 4 + ky); Bz0 = __ldg(v + 4 + kz);
      Cx = __ldg(v + 8 + kx); Cy = __ldg(v + 8 + ky); Cz0 = __ldg(v + 8 + kz);
    }
    Az0 = Az0 - oz;
    Bz0 = Bz0 - oz;
    Cz0 = Cz0 - oz;
    const F2 A = (f2(Ax, Ay) - oxy) - f2(Sx * Az0, Sy * Az0);
    const F2 B = (f2(Bx, By) - oxy) - f2(Sx * Bz0, Sy * Bz0);
    const F2 C = (f2(Cx, Cy) - oxy) - f2(Sx * Cz0, Sy * Cz0);
    Ax = lo(A); Ay = hi(A);
    Bx = lo(B); By = hi(B);
    Cx = lo(C); Cy = hi(C);
    float U = Cx * By - Cy * Bx;
    float V = Ax * Cy - Ay * Cx;
    float W = Bx * Ay - By * Ax;
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
      U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
      V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
      W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
    }
    if (fminf(fminf(U, V), W) < 0.0f && fmaxf(fmaxf(U, V), W) > 0.0f) continue;
    const float det = U + V + W;
    if (det == 0.0f) continue;
    const float T = U * (Sz * Az0) + V * (Sz * Bz0) + W * (Sz * Cz0);
    const float rcp = 1.0f / det;
    const float t = T * rcp;
    if (!(t > 0.0f) || !(t <= best.t)) continue;
    if (t == best.t && best.tri >= 0 && list[c] > list[best.tri]) continue;
    const float b1 = V * rcp, b2 = W * rcp;
    if (kAlpha && !alpha_opaque(bvh.alpha, list[c], b1, b2)) continue;
    best.t = t;
    best.b1 = b1;
    best.b2 = b2;
    best.tri = c;
  }
  if (best.tri >= 0) best.tri = list[best.tri];
  return best;
}

__device__ __forceinline__ void write_voxel(r2_voxel* out, size_t vid, const r2_voxel& v) {
  const uint4* src = reinterpret_cast<const uint4*>(&v);
  uint4* dst = reinterpret_cast<uint4*>(out + vid);
  dst[0] = src[0];
  dst[1] = src[1];
}

__device__ __forceinline__ void write_empty(const FilterLaunch& L, size_t vid) {
  write_voxel(L.out, vid, empty_voxel());
  if (L.wide) {
    float* w = L.wide + vid * kWideFloats;
    for (int k = 0; k < kWideFloats; ++k) w[k] = 0.0f;
    w[16] = 1.0f;
  }
  if (L.fp16) {
    uint4* f = reinterpret_cast<uint4*>(L.fp16 + vid * 8);
    *f = make_uint4(0, 0, 0, 0);
  }
  if (L.eig) {
    float4* e = reinterpret_cast<float4*>(L.eig + vid * 12);
    e[0] = e[1] = e[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}

// FP64 eigendecomposition of the voxel's mean SGGX matrix (compensated FP32
// sums promoted to double), written to L.eig (lanes 0..11, one float each),
// and, with the projection on, the projected matrix in the shared record wv[1..6].
// Every lane computes the same values.  Out of line: only this tail uses double registers.
__device__ __noinline__ void sggx_eig_tail(const FilterLaunch& L, uint32_t vid, int lane, const float2* S,
                                           uint32_t hits, float* wv) {
  double m[6], w[3], V[3][3];
  const double inv = 1.0 / (double)hits;
  for (int k = 0; k < 6; ++k) m[k] = ((double)S[k].x + (double)S[k].y) * inv;
  sym3_eig_jacobi(m, w, V);
  if (L.eig && lane < 12) {
    const double v = lane < 3 ? w[lane] : V[(lane - 3) % 3][(lane - 3) / 3];
    L.eig[(size_t)vid * 12 + lane] = (float)v;
  }
  if (L.project) {
    double P[6];
    sym3_project(w, V, (double)L.floor, P);
    if (lane == 0)
      for (int k = 0; k < 6; ++k) wv[1 + k] = (float)P[k];
  }
  __syncwarp();
}

// One thread per brick: the brick goes to the brick list when its ball's box
// overlaps a triangle's box; the others' voxels get the empty payload here.
__global__ void __launch_bounds__(256) k_filter_classify(FilterLaunch L) {
  const int lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < L.brickCount; base += stride) {
    const uint32_t id = L.brickFirst + base + lane;
    bool cand = false;
    if (base + lane < L.brickCount) {
      const Brick k = brick_at(L, id);
      cand = bvh_any_box(L.bvh, k.center - v3(k.r), k.center + v3(k.r));
      int x, y, z;
      if (!cand)
        for (int v = 0; v < 8; ++v)
          if (brick_voxel(L, k, v, &x, &y, &z)) write_empty(L, voxel_index(L, x, y, z));
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, cand);
    if (m) {
      uint32_t slot = 0;
      const int leader = __ffs(m) - 1;
      if (lane == leader) slot = atomicAdd(&L.counters[kCountBricks], (uint32_t)__popc(m));
      slot = __shfl_sync(0xFFFFFFFFu, slot, leader);
      if (cand) L.bricks[slot + __popc(m & ((1u << lane) - 1u))] = id;
    }
  }
}

// One warp per brick (kAll: every brick of the part, else the listed ones):
// the brick's candidates by one walk of the BVH, then, a candidate per lane,
// which of the brick's voxels each can reach.  A voxel with any goes to the
// work list, its candidates to the pool; one without gets the empty payload.
// Of a brick with more than kCandMax candidates, or whose lists do not fit,
// the voxels go to the work list without a candidate list.  Walking per brick
// of 8 voxels shares the dependent fetches of the walk, and keeping it out of
// the sampling kernel keeps that kernel's code small.
template <bool kAll>
__global__ void __launch_bounds__(kSampleWarps * 32) k_filter_lists(FilterLaunch L) {
  __shared__ int sCand[kSampleWarps][kCandMax], sScratch[kSampleWarps][kWalkInts];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* cand = sCand[warp];
  unsigned* masks = reinterpret_cast<unsigned*>(sScratch[warp]);  // after the walk: of 32 candidates, who reach voxel v
  static_assert(kCandMax / 32 * 8 <= kWalkInts, "eight masks for every 32 candidates");
  const uint32_t nbricks = kAll ? L.brickCount : *(volatile uint32_t*)&L.counters[kCountBricks];
  const float reach = ray_reach(L);
  uint32_t cNodes = 0;  // counting build: a walk counts for every voxel it serves
  for (uint32_t w = blockIdx.x * kSampleWarps + warp; w < nbricks; w += gridDim.x * kSampleWarps) {
    const Brick k = brick_at(L, kAll ? L.brickFirst + w : L.bricks[w]);
    uint32_t walked = 0;
    const int n = gather_candidates(L, k.center - v3(k.r), k.center + v3(k.r), k.center, k.r, cand, sScratch[warp],
                                    lane, &walked);
    __syncwarp();
    int x, y, z;
    const bool mine = lane < 8 && brick_voxel(L, k, lane, &x, &y, &z);  // this lane's voxel
    const size_t vid = mine ? voxel_index(L, x, y, z) : 0;
    int count = 0;  // its candidates
    for (int base = 0; base < n; base += 32) {
      const bool valid = base + lane < n;
      const float r = padded_reach(reach, k.center) + 1e-5f * L.brickOffset * 2.0f;  // any of its voxels' padded reach
      const TriBall t = load_tri_ball(L, cand[valid ? base + lane : base], k.center, 2.0f * k.r, r);
      for (int v = 0; v < 8; ++v) {
        int vx, vy, vz;
        const bool in = brick_voxel(L, k, v, &vx, &vy, &vz);
        const bool near = in && valid && tri_near(t, voxel_center(L, vx, vy, vz));
        const unsigned m = __ballot_sync(0xFFFFFFFFu, near);
        if (lane == v) {
          masks[(base >> 2) + v] = m;
          count += __popc(m);
        }
      }
    }
    __syncwarp();
    if (mine && n >= 0 && count == 0) write_empty(L, vid);
    const bool entry = mine && (n < 0 || count > 0);
    const unsigned entries = __ballot_sync(0xFFFFFFFFu, entry);
    cNodes += walked * (uint32_t)__popc(entries);
    if (entries == 0) continue;
    // places in the pool: every voxel's list is its length and its triangles
    int end = entry && n >= 0 ? count + 1 : 0;
    const int words = end;
    for (int off = 1; off < 8; off <<= 1) {
      const int o = __shfl_up_sync(0xFFFFFFFFu, end, off);
      if (lane >= off) end += o;
    }
    const int used = __shfl_sync(0xFFFFFFFFu, end, 7);
    // the long ones go to the front of the work list, the others to its end,
    // so that the sampling kernel's last voxels are short
    const unsigned lo = (1u << lane) - 1u;
    const unsigned front = __ballot_sync(0xFFFFFFFFu, entry && (n < 0 || count > kLongList)), back = entries & ~front;
    unsigned long long base = 0;  // places: in the list's front, and in the pool
    uint32_t atBack = 0;
    if (lane == 0) {
      base = atomicAdd(reinterpret_cast<unsigned long long*>(L.counters + kCountFront),
                       ((unsigned long long)(uint32_t)used << 32) | (unsigned long long)__popc(front));
      if (back) atBack = atomicAdd(&L.counters[kCountBack], (uint32_t)__popc(back));
    }
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    atBack = __shfl_sync(0xFFFFFFFFu, atBack, 0);
    const uint32_t pool = (uint32_t)(base >> 32);
    const bool lists = n >= 0 && (unsigned long long)pool + (uint32_t)used <= L.poolWords;
    const uint32_t at = pool + (uint32_t)(end - words);
    if (entry) {
      const uint32_t slot = front >> lane & 1u ? (uint32_t)base + (uint32_t)__popc(front & lo)
                                               : 8u * L.brickCount - 1u - (atBack + (uint32_t)__popc(back & lo));
      L.entries[slot] = make_uint2((uint32_t)vid, lists ? at : kNoList);
      if (lists) L.pool[at] = count;
    }
    if (lists)
      for (int v = 0; v < 8; ++v) {
        if (!(entries >> v & 1u)) continue;
        uint32_t to = __shfl_sync(0xFFFFFFFFu, at, v) + 1;
        for (int b = 0; b < n; b += 32) {
          const unsigned m = masks[(b >> 2) + v];
          if (m >> lane & 1u) L.pool[to + __popc(m & ((1u << lane) - 1u))] = cand[b + lane];
          to += __popc(m);
        }
      }
    __syncwarp();
  }
  if (L.ops) {
    for (int off = 16; off > 0; off >>= 1) cNodes += __shfl_xor_sync(0xFFFFFFFFu, cNodes, off);
    if (lane == 0 && cNodes) atomicAdd(&L.ops[1], (unsigned long long)cNodes);
  }
}

__device__ __forceinline__ CSum shfl_xor_csum(CSum v, int off) {
  CSum o;
  o.s = __shfl_xor_sync(0xFFFFFFFFu, v.s, off);
  o.c = __shfl_xor_sync(0xFFFFFFFFu, v.c, off);
  return o;
}

__device__ __forceinline__ CSum warp_csum(CSum v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = ccombine(v, shfl_xor_csum(v, off));
  return v;
}

// The sums of a voxel, in the order of the reduction.
enum SumIndex { kSumS = 0, kSumNormal = 6, kSumDist = 9, kSumDiffuse = 10, kSumSpecular = 13, kSumRough = 16, kSumIor = 17, kSums = 18 };

// Two compensated sums at once (cadd of each half).
struct CSum2 {
  F2 s, c;
};
__device__ __forceinline__ void cadd(CSum2& x, F2 v) {
  const F2 sum = x.s + v, bb = sum - x.s;
  x.c = x.c + ((x.s - (sum - bb)) + (v - bb));
  x.s = sum;
}

// Reduces v[0 .. kSums-1] over the warp into out (shared): recursive halving,
// each step exchanging half of the values still held with the lane `off` away
// and adding the other half, so that a value's additions are those of a
// butterfly over the same offsets (the sums are symmetric), at 20 additions a
// lane in place of 90.
__device__ __forceinline__ void warp_csums(CSum (&v)[kSums + 2], float2* out, int lane) {
  v[kSums] = v[kSums + 1] = csum0();
  int base = 0, have = kSums;  // this lane holds the values base .. base + have - 1
  int n = kSums;               // (the same number of slots on every lane)
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const int half = (n + 1) / 2;
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < (kSums + 1) / 2; ++i) {
      if (i >= half) break;
      const CSum hi = half + i < n ? v[half + i] : csum0();
      v[i] = ccombine(up ? hi : v[i], shfl_xor_csum(up ? v[i] : hi, off));
    }
    base += up ? half : 0;
    have = up ? have - half : min(have, half);
    n = half;
  }
  if (have > 0) out[base] = make_float2(v[0].s, v[0].c);
  __syncwarp();
}

// The closest hit of a ray through the BVH, from the node root.
template <bool kCount, bool kAlpha>
__device__ Hit trace_bvh(const BvhView& bvh, V3 o, V3 d, float tmax, int root, uint32_t* nodes, uint32_t* tris) {
  TraceState s;
  trace_begin(s, o, d, tmax, root);
  int stack[R2_BVH_STACK];
  float stackT[R2_BVH_STACK];
  while (!trace_advance<kCount, kAlpha>(bvh, s, stack, stackT, 1 << 30)) {
  }
  if (kCount) {
    *nodes += s.nodes;
    *tris += s.tris;
  }
  return s.best;
}

// Writes a voxel's record w (the wide layout, in shared memory: [0] density,
// [1..6] Sxx Syy Szz Sxy Sxz Syz, [7..9] diffuse, [10..12] specular, [13..15] normal,
// [16] ior): its 32-byte payload (SFilteredDataCompact(const SFilteredData&),
// filtered_data.hpp:91-107, a field per lane; tmp: 8 words of shared memory), the
// wide record and the FP16 payload.
__device__ __forceinline__ void write_record(const FilterLaunch& L, uint32_t vid, const float* w, uint32_t* tmp,
                                             int lane) {
  const float M16 = 65535.0f, M8 = 255.0f;
  const V3 n = normalize(v3(w[13], w[14], w[15]));  // SFilteredData::n()
  uint16_t* h = reinterpret_cast<uint16_t*>(tmp);
  if (lane < 9) {
    // 0..2 sigma, 3..5 r of xy, xz, yz, 6..8 normal
    const int i = lane < 3 ? lane : (lane == 5 ? 1 : 0), j = lane == 3 ? 1 : 2;
    const float q = sqrtf(lane < 3 ? w[1 + lane] : w[1 + i] * w[1 + j]);
    float v = M16 * q;
    if (lane >= 3) v = M16 * 0.5f * ((lane < 6 ? w[1 + lane] / q : comp(n, lane - 6)) + 1.0f);
    h[lane < 6 ? 2 + lane : 5 + lane] = to_u16(clampf(v, 0.0f, M16));
  } else if (lane < 15) {
    reinterpret_cast<uint8_t*>(tmp)[7 + lane] = to_u8(clampf(M8 * w[lane - 2], 0.0f, M8));
  } else if (lane == 15) {
    h[14] = f32_to_f16_bits(w[16]);
    h[15] = 0;
  } else if (lane == 16) {
    tmp[0] = __float_as_uint(w[0]);
  }
  __syncwarp();
  if (lane < 8) reinterpret_cast<uint32_t*>(L.out + vid)[lane] = tmp[lane];
  if (L.wide && lane < kWideFloats) L.wide[(size_t)vid * kWideFloats + lane] = w[lane];
  if (L.fp16 && lane < 8) L.fp16[(size_t)vid * 8 + lane] = lane < 7 ? f32_to_f16_bits(w[lane]) : (uint16_t)0;
}

// 8 resident blocks per SM (64 registers a thread): traversal is issue and
// latency bound, and the extra warps hide more than the few spilled values of
// the shading tail cost (measured on the 256^3 filter: 96 registers and 5
// blocks 18.6 M voxels/s, 64 and 8 blocks 21.6 M).
// Its warps are in different places of the kernel, so instruction fetch counts
// as much as issue: the loops of one or a few turns (hit lengths, packing,
// copies, iterations) are kept rolled, where the compiler's four-fold unrolling
// cost more to fetch than it spared (256^3 filter 102.4 -> 94.9 ms, 24x77x24
// tree 1.04 -> 1.00 ms, 48^3 of 400,000 triangles 2.09 -> 1.95 ms).
// kEig: the build with the FP64 eigendecomposition tail (eigen output or
// projection requested), kTex: with texture and opacity maps; the default
// build carries none of their code.
template <bool kCount, bool kEig, bool kTex>
__global__ void __launch_bounds__(kSampleWarps * 32, 8) k_filter_sample(FilterLaunch L) {
  extern __shared__ float4 sSample[];  // sample_smem_per_warp(L.spv) bytes per warp
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* myV = reinterpret_cast<float*>(sSample + warp * (sample_smem_per_warp(L.spv) / sizeof(float4)));
  int* myCand = reinterpret_cast<int*>(myV + kCandStage * 9);
  float* myTs = reinterpret_cast<float*>(myCand + kCandMax);
  float2* mySum = reinterpret_cast<float2*>(myV);            // after the rays: the voxel's sums,
  float* myRec = reinterpret_cast<float*>(mySum + kSums);    // its wide record
  uint32_t* myOut = reinterpret_cast<uint32_t*>(myRec + kWideFloats);  // and its payload
  const uint32_t nfront = *(volatile uint32_t*)&L.counters[kCountFront];
  const uint32_t nwork = nfront + *(volatile uint32_t*)&L.counters[kCountBack];
  const float radius = 1.1f * length(L.voxelSize) / 2.0f;
  const float tMaxFixed = L.voxelSize.x;
  uint32_t cRays = 0, cNodes = 0, cTris = 0;  // counting build only
  uint32_t sampled = 0;                       // voxels with candidates
  while (true) {
    uint32_t w = 0;
    if (lane == 0) w = atomicAdd(&L.counters[kCountTaken], 1u);
    w = __shfl_sync(0xFFFFFFFFu, w, 0);
    if (w >= nwork) break;
    const uint2 entry = L.entries[w < nfront ? w : 8u * L.brickCount - 1u - (w - nfront)];
    const uint32_t vid = entry.x;
    const int x = (int)(vid % (uint32_t)L.nx);
    const int y = (int)((vid / (uint32_t)L.nx) % (uint32_t)L.ny);
    const int z = (int)(vid / ((uint32_t)L.nx * (uint32_t)L.ny));
    const V3 center = voxel_center(L, x, y, z);
    const V3 cv = v3((float)x, (float)y, (float)z);
    // few candidate triangles (the usual case): every ray tests them all, the
    // warp's lanes in step; otherwise the rays traverse the BVH from the
    // voxel's local root
    int ncand, root = 0;
    if (entry.y != kNoList) {
      ncand = L.pool[entry.y];
#pragma unroll 1
      for (int i = lane; i < ncand; i += 32) myCand[i] = L.pool[entry.y + 1 + i];
    } else {
      const float pad = padded_reach(ray_reach(L), center);  // every sample ray stays within it
      ncand = gather_candidates(L, center - v3(pad), center + v3(pad), center, pad, myCand,
                                reinterpret_cast<int*>(myV), lane, &cNodes);
      if (ncand < 0) root = bvh_local_root(L.bvh, center - v3(pad), center + v3(pad));
    }
    if (ncand == 0) {  // no triangle within reach
      if (lane == 0) write_empty(L, vid);
      continue;
    }
    ++sampled;
    __syncwarp();
#pragma unroll 1
    for (int i = lane; i < min(ncand, kCandStage); i += 32) {
      const int t = myCand[i];
      const float4 a = __ldg(&L.bvh.tris[3 * t]), b = __ldg(&L.bvh.tris[3 * t + 1]), c = __ldg(&L.bvh.tris[3 * t + 2]);
      float* v = myV + 9 * i;
      v[0] = a.x; v[1] = a.y; v[2] = a.z;
      v[3] = b.x; v[4] = b.y; v[5] = b.z;
      v[6] = c.x; v[7] = c.y; v[8] = c.z;
    }
    __syncwarp();

    // this lane's sums in the order of SumIndex, two by two: S, the normal and
    // the length compensated, the last eight plain until the warp adds them
    CSum2 comp2[kSumDiffuse / 2];
    F2 plain[(kSums - kSumDiffuse) / 2];
    const F2 zero = f2(0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < kSumDiffuse / 2; ++k) comp2[k].s = comp2[k].c = zero;
#pragma unroll
    for (int k = 0; k < (kSums - kSumDiffuse) / 2; ++k) plain[k] = zero;
    uint32_t hits = 0;

#pragma unroll 1
    for (uint32_t s = lane; s < L.spv; s += 32) {
      const U4 r0 = philox4x32_10(u4(s, 0u, L.lod, 0u), vid, L.seed);
      const U4 r1 = philox4x32_10(u4(s, 1u, L.lod, 0u), vid, L.seed);
      const V3 oi = cv + v3(u01(r0.x), u01(r0.y), u01(r0.z));
      const V3 o = xform_point(L.indexToWorld, oi);
      const V3 d = uniform_sample_sphere(u01(r0.w), u01(r1.x));
      const float tmax = L.clip ? sphere_exit(o, d, center, radius) : tMaxFixed;
      Hit h;
      if (ncand >= 0) {
        h = kTex && L.bvh.alpha.alphaTex ? trace_candidates<true>(L.bvh, myCand, ncand, myV, o, d, tmax)
                                         : trace_candidates<false>(L.bvh, myCand, ncand, myV, o, d, tmax);
        if (kCount) cTris += (uint32_t)ncand;
      } else {
        h = kTex && L.bvh.alpha.alphaTex ? trace_bvh<kCount, true>(L.bvh, o, d, tmax, root, &cNodes, &cTris)
                                         : trace_bvh<kCount, false>(L.bvh, o, d, tmax, root, &cNodes, &cTris);
      }
      if (kCount) ++cRays;
      float tsv = -1.0f;
      if (h.tri >= 0) {
        const float4 n0 = __ldg(&L.triN[3 * h.tri]);
        const float4 n1 = __ldg(&L.triN[3 * h.tri + 1]);
        const float4 n2 = __ldg(&L.triN[3 * h.tri + 2]);
        const float b0 = (1.0f - h.b1) - h.b2;
        V3 gn = v3(n0.x, n0.y, n0.z) * b0 + v3(n1.x, n1.y, n1.z) * h.b1 + v3(n2.x, n2.y, n2.z) * h.b2;
        gn = normalize(gn);
        V3 n = normalize(xform_vector(L.objModelToWorld, gn));
        const uint32_t mi = __ldg(&L.triMat[h.tri]);
        const r2_material& m = L.mats[mi];
        V3 kd = v3(m.diffuse[0], m.diffuse[1], m.diffuse[2]), ks = v3(m.specular[0], m.specular[1], m.specular[2]);
        if (kTex) {  // diffuse(tc), glossy(tc) and the normal-mapped normal (mesh_filter.hpp:300-371)
          const int4 mt = L.matTex[mi];
          if (mt.x >= 0 || mt.y >= 0 || mt.z >= 0) {
            const TexView tv = {L.triUV, L.texels, L.texInfo, L.bvh.tris};
            const TexShade ts = textured_surface(tv, mt.x, mt.y, mt.z, h.tri, h.b1, h.b2, n, kd, ks);
            n = ts.n;
            kd = ts.diffuse;
            ks = ts.specular;
          }
        }
        float bs[6];
        build_s(n, m.alpha_x, bs);
        cadd(comp2[0], f2(bs[0], bs[1]));
        cadd(comp2[1], f2(bs[2], bs[3]));
        cadd(comp2[2], f2(bs[4], bs[5]));
        cadd(comp2[3], f2(n.x, n.y));
        cadd(comp2[4], f2(n.z, tmax));
        plain[0] = plain[0] + f2(kd.x, kd.y);
        plain[1] = plain[1] + f2(kd.z, ks.x);
        plain[2] = plain[2] + f2(ks.y, ks.z);
        plain[3] = plain[3] + f2(m.alpha_x, m.eta_t);
        ++hits;
        tsv = tmax;
      }
      myTs[s] = tsv;
    }
    hits = __reduce_add_sync(0xFFFFFFFFu, hits);
    if (hits == 0) {  // also: every lane is done with the staged vertices
      if (lane == 0) write_empty(L, vid);
      __syncwarp();
      continue;
    }
    CSum sum[kSums + 2];
#pragma unroll
    for (int k = 0; k < kSums; ++k) {
      const F2 v = k < kSumDiffuse ? comp2[k / 2].s : plain[(k - kSumDiffuse) / 2];
      const F2 c = k < kSumDiffuse ? comp2[k / 2].c : zero;
      sum[k].s = k & 1 ? hi(v) : lo(v);
      sum[k].c = k & 1 ? hi(c) : lo(c);
    }
    warp_csums(sum, mySum, lane);

    // the hit samples' lengths packed into myTs[0 .. hits-1] in sample order, so
    // that every iteration of the density fit visits the hits only
    if (L.clip) {
      uint32_t packed = 0;
#pragma unroll 1
      for (uint32_t base = 0; base < L.spv; base += 32) {
        const uint32_t s = base + lane;
        const float t = s < L.spv ? myTs[s] : -1.0f;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, t >= 0.0f);
        __syncwarp();  // every lane has read its entry before any is overwritten
        if (t >= 0.0f) myTs[packed + __popc(m & ((1u << lane) - 1u))] = t;
        packed += (uint32_t)__popc(m);
      }
      __syncwarp();
    }

    const auto total = [&](int k) { return mySum[k].x + mySum[k].y; };  // cvalue
    // estimateDensity (mesh_filter.hpp:182-204)
    const float avgDist = total(kSumDist) / (float)hits;
    const float pMesh = (float)hits / (float)L.spv;
    float density = -logf(1.0f - pMesh) / (avgDist * L.sigma_t);
    const float nAlpha = L.alpha / L.sigma_t;
#pragma unroll 1
    for (uint32_t it = 0; it < L.iters; ++it) {
      float pVol;
      if (L.clip) {
        CSum p = csum0();
#pragma unroll 1
        for (uint32_t s = lane; s < hits; s += 32) cadd(p, expf(-density * L.sigma_t * myTs[s]));
        p = warp_csum(p);
        pVol = 1.0f - cvalue(p) / (float)hits;
      } else {
        pVol = 1.0f - expf(-density * L.sigma_t * tMaxFixed);
      }
      density = density - nAlpha * (pVol - pMesh);
    }
    // the wide record, an entry per lane
    const float inv = 1.0f / (float)hits;
    const V3 nm = normalize(xform_vector(
        L.worldToModel, v3(total(kSumNormal), total(kSumNormal + 1), total(kSumNormal + 2)) * inv));
    if (lane < kWideFloats) {
      float v = lane == 0 ? density : (lane == 17 ? (float)hits : avgDist);
      if (lane >= 13 && lane < 16) v = comp(nm, lane - 13);
      const int k = lane < 7 ? kSumS + lane - 1 : (lane < 13 ? kSumDiffuse + lane - 7 : (lane == 16 ? kSumIor : kSumRough));
      if ((lane >= 1 && lane < 13) || lane == 16 || lane == 19) v = total(k) * inv;
      myRec[lane] = v;
    }
    __syncwarp();
    if (kEig) sggx_eig_tail(L, vid, lane, mySum + kSumS, hits, myRec);
    write_record(L, vid, myRec, myOut, lane);
    __syncwarp();
  }
  if (lane == 0 && sampled) atomicAdd(&L.counters[kCountSampled], sampled);
  if (kCount) {
    unsigned long long r = cRays, n = cNodes, t = cTris;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      r += __shfl_xor_sync(0xFFFFFFFFu, r, off);
      n += __shfl_xor_sync(0xFFFFFFFFu, n, off);
      t += __shfl_xor_sync(0xFFFFFFFFu, t, off);
    }
    if (lane == 0) {
      atomicAdd(&L.ops[0], r);
      atomicAdd(&L.ops[1], n);
      atomicAdd(&L.ops[2], t);
    }
  }
}

}  // namespace

void launch_filter_lists(const FilterLaunch& L, cudaStream_t s) {
  const uint32_t warps = (uint32_t)sm_count() * 8 * kSampleWarps;
  const int blocks = (int)((std::min(L.brickCount, warps) + kSampleWarps - 1) / kSampleWarps);
  if (L.brickCount <= kListAll * warps) {
    k_filter_lists<true><<<blocks, kSampleWarps * 32, 0, s>>>(L);
  } else {
    k_filter_classify<<<sm_count() * 16, 256, 0, s>>>(L);
    k_filter_lists<false><<<blocks, kSampleWarps * 32, 0, s>>>(L);
  }
  R2_CUDA(cudaGetLastError());
}

template <bool kCount, bool kEig, bool kTex>
static void launch_sample(const FilterLaunch& L, cudaStream_t s) {
  const size_t smem = kSampleWarps * sample_smem_per_warp(L.spv);  // <= 4 x 7.5 KB at spv 1024
  int n = 0;
  R2_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_filter_sample<kCount, kEig, kTex>, kSampleWarps * 32, smem));
  k_filter_sample<kCount, kEig, kTex><<<sm_count() * std::max(n, 1), kSampleWarps * 32, smem, s>>>(L);
}

template <bool kCount>
static void launch_sample(const FilterLaunch& L, cudaStream_t s) {
  const bool eig = L.eig || L.project;
  if (L.triUV) {
    if (eig) launch_sample<kCount, true, true>(L, s);
    else launch_sample<kCount, false, true>(L, s);
  } else {
    if (eig) launch_sample<kCount, true, false>(L, s);
    else launch_sample<kCount, false, false>(L, s);
  }
}

void launch_filter_sample(const FilterLaunch& L, cudaStream_t s) {
  if (L.ops) launch_sample<true>(L, s);
  else launch_sample<false>(L, s);
  R2_CUDA(cudaGetLastError());
}

}  // namespace r2
