// Eight-wide BVH of the path tracer's surface queries (Ylitie, Karras, Laine,
// "Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide BVHs",
// HPG 2017): the builder's binary tree collapsed to nodes of up to eight
// children whose boxes are 8-bit offsets in the node's own frame.  A ray visits
// about a third of the nodes it visits in the binary tree, each one dependent
// fetch, and the nodes of 327,680 triangles take 4 MB in place of 21.
//
// A child's decoded box holds its exact one with room for the rounding of the
// decoded test, so no child that the exact test would enter is skipped, and
// hits are the least (t, code) of the triangles tested: the same as the binary
// tree's.
//
// Node, seven 16-byte words:
//   w0  frame origin x y z | exponent bytes x y z, mask of inner children
//   w1  first inner child, mask of leaf children, 1 if they are instances, -
//   w2  lo.x of children 0-3, 4-7, lo.y 0-3, 4-7
//   w3  lo.z, hi.x      w4  hi.y, hi.z
//   w5, w6  of the slots that are leaves: the complement of bvh_leaf_ref, or the
//           instance
// Inner children are consecutive nodes in slot order.  A slot's bits are the
// octant of the node that the child lies in (1: the greater half of x, y, z),
// so that slot ^ octant of the direction orders the children along the ray.
//
// Traversal (wide_rays): a warp's lanes take one node step each, together, and
// put the leaves they enter on a queue of the warp; whenever 32 wait, the warp
// turns them into triangles, and whenever 32 of those wait, it tests them, one
// per lane, whichever lanes they came from.  A ray's closest hit is a 64-bit
// minimum in shared memory.  With every lane testing its own leaves 8.8 of 32
// lanes were active and the wide tree was no faster than the binary one; now
// 21 are, and the kernels are bound by issue and the integer pipe (72 % and
// 64 % busy: the box test unpacks 48 bytes a node).  64 spheres of 5,120
// triangles, 1024x1024, 64 samples: 123.2 -> 100.2 ms a frame; 60,000
// alpha-tested leaf triangles at 641x479, 16 samples: 35.1 -> 21.3 ms; 144
// instances of 20,480 triangles at 1280x720, 8 samples: 27.9 -> 23.5 ms.
// Leaves of fewer triangles (as many as fill the node's slots), nodes of 128
// bytes, 6 or 10 blocks an SM instead of 8 and queues of triangles without the
// queue of leaves were each slower.
#pragma once
#include "bvh.h"
#include "runtime.h"

namespace r2 {

constexpr int kWideWords = 7;  // 16-byte words of a node

struct WideView {
  const uint4* nodes;
};

struct WideBox {
  V3 lo, hi;
};
R2_HD float wide_area(const WideBox& b) {
  const V3 e = b.hi - b.lo;
  return e.x * e.y + e.y * e.z + e.z * e.x;
}
R2_HD void wide_children_of(const BvhNode* nd, WideBox* b, int* ref) {
  const float4 b0 = nd->b0, b1 = nd->b1, bz = nd->bz;
  const int4 ch = nd->ch;
  b[0] = WideBox{v3(b0.x, b0.z, bz.x), v3(b0.y, b0.w, bz.y)};
  b[1] = WideBox{v3(b1.x, b1.z, bz.z), v3(b1.y, b1.w, bz.w)};
  ref[0] = ch.x;
  ref[1] = ch.y;
}

// The children of the wide node over binary node `node`: box[0 .. n-1] and
// ref[0 .. n-1] (room for nine each), n returned.  The inner child of largest
// area is opened until there are eight or none is left; of areas that are not
// numbers any is, so that the capacity below holds for every tree.
R2_HD int wide_open(const BvhNode* nodes, uint32_t node, WideBox* box, int* ref) {
  wide_children_of(&nodes[node], box, ref);
  int n = ref[1] == R2_BVH_NONE ? 1 : 2;
  while (n < 8) {
    int open = -1;
    float largest = 0.0f;
    for (int i = 0; i < n; ++i)
      if (ref[i] >= 0 && (open < 0 || wide_area(box[i]) > largest)) {
        open = i;
        largest = wide_area(box[i]);
      }
    if (open < 0) break;
    WideBox b[2];
    int r[2];
    wide_children_of(&nodes[ref[open]], b, r);
    box[open] = b[0];
    ref[open] = r[0];
    box[n] = b[1];
    ref[n] = r[1];
    if (r[1] != R2_BVH_NONE) ++n;
  }
  return n;
}

// Wide nodes that trees of nleaves leaves in all below nroots roots can take.
// A node with fewer than eight children has leaves alone: of W nodes with L
// leaves below R roots, 7 L / 12 + R bounds W (L / 2 nodes of two leaves, an
// inner node per eight nodes).
R2_HD size_t wide_capacity(uint32_t nleaves, uint32_t nroots) { return (size_t)nleaves * 7 / 12 + nroots + 8; }

// Collapses binary BVHs into wide ones, keeping its buffers between builds.
class WideBvh {
 public:
  // nodes: binary nodes, trees below roots[0 .. nroots-1] (host; null: one
  // root, node 0) with at most nleaves leaves in all.
  // Wide node i < nroots is the root of tree i.  Asynchronous on s.
  void build(const BvhNode* nodes, const uint32_t* roots, uint32_t nroots, uint32_t nleaves, cudaStream_t s);
  WideView view() const { return WideView{nodes_.get()}; }
  static constexpr int kLaunches = 5;  // kernels of a build

 private:
  DBuf<uint8_t> mem_;
  DBuf<uint4> nodes_;
  DBuf<uint32_t> queue_, state_;  // binary node of each wide node; counters
};

#if defined(__CUDACC__)

// A warp's rays in shared memory, as the lanes that test their triangles read
// them, and the triangles that wait.
struct WideWarp {
  float4 a[32];  // origin, Sx
  float4 b[32];  // Sy, Sz, kz, hit code - triangle (int bits)
  unsigned long long key[32];  // closest hit so far: t (float bits) << 32 | code; kWideNoHit without one
  float2 bary[32];             // its b1, b2
  uint2 leaves[64];            // lane, leaf's word of the nodes
  uint32_t tris[32 + 32 * 8];  // lane << 26 | triangle (a BVH has fewer than 2^26)
};
constexpr uint32_t kWideNoHit = 0x7FFFFFFFu;

// One lane's ray: what its node steps need.  group: the inner children still
// to visit of the last node (first child; inner mask << 8 | their slots ^ oct).
struct WideRay {
  V3 o, invd;
  uint32_t oct;
  uint2 group;
  int sp;
  float tmax;  // its closest hit's t when the queue was last emptied
};

constexpr uint32_t kWideExit = 0x40000000u;  // stack marker: leave the instance
constexpr uint32_t kWideLeafGroup = 0x80000000u;  // stacked instance slots of a node: word of slot 0; slots

// 1 / x within an ulp or two, far inside what the box tests give way; of an x
// near zero (positive: its sign as the ray's octant has it) 2^88.  Units lie
// between 2^-42 and 2^23, so that nothing overflows in wide_axis, and a plane 1/64
// unit away still lies 2^40 or more from the ray in t, beyond every tmax (1e12), on
// the side that the exact one does: a ray along an axis is culled by what it does
// not pass.  Left to infinities its axis culled nothing, and of the 20M shadow rays
// of a forest's bounce one that ran straight through 267 trees took 90 ms.
__device__ __forceinline__ float wide_rcp(float x, bool positive) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  r = fminf(fabsf(r), 3.0948500982134507e26f);
  return positive ? r : -r;
}

// Sets a lane's ray up (make_ray_pre without its swap of the first two axes,
// which changes the sign of U, V, W, det and T alone) with root still to visit.
__device__ __forceinline__ void wide_set(WideRay& r, WideWarp& w, int lane, V3 o, V3 d, int vdelta, uint32_t root) {
  r.o = o;
  r.oct = (d.x < 0.0f ? 0u : 1u) | (d.y < 0.0f ? 0u : 2u) | (d.z < 0.0f ? 0u : 4u);
  r.invd = v3(wide_rcp(d.x, r.oct & 1u), wide_rcp(d.y, r.oct & 2u), wide_rcp(d.z, r.oct & 4u));
  const V3 ad = vabs(d);
  const int kz = (ad.x > ad.y) ? ((ad.x > ad.z) ? 0 : 2) : ((ad.y > ad.z) ? 1 : 2);
  const float dx = kz == 0 ? d.y : (kz == 1 ? d.z : d.x), dy = kz == 0 ? d.z : (kz == 1 ? d.x : d.y);
  const float dz = comp(d, kz);
  w.a[lane] = make_float4(o.x, o.y, o.z, dx / dz);
  w.b[lane] = make_float4(dy / dz, 1.0f / dz, __int_as_float(kz), __int_as_float(vdelta));
  r.group = make_uint2(root, 0x0100u | (1u << r.oct));  // a group of one child, in slot 0
}

// Byte k of w as the float 2^23 + 256 * byte (exact): a permute in place of a
// conversion.
template <int k>
__device__ __forceinline__ float wide_byte(uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7404u | (k << 4)));
}

// Entry or exit distances of a child on one axis: scale * byte + base for the
// near and the far plane, one packed operation.
__device__ __forceinline__ void wide_planes(float nearQ, float farQ, unsigned long long scale, unsigned long long base,
                                            float* tn, float* tf) {
  unsigned long long q;
  asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(nearQ), "f"(farQ));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(q) : "l"(q), "l"(scale), "l"(base));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(*tn), "=f"(*tf) : "l"(q));
}
// The axis's scale and base: t = byte * 2^e / d + (origin - o) / d, for bytes
// read as 2^23 + 256 * byte.
__device__ __forceinline__ void wide_axis(float origin, float o, float invd, uint32_t exponent, unsigned long long* scale,
                                          unsigned long long* base) {
  const float s = __uint_as_float(exponent << 23) * (1.0f / 256.0f) * invd;
  const float b = fmaf(-8388608.0f, s, (origin - o) * invd);
  asm("mov.b64 %0, {%1, %1};" : "=l"(*scale) : "f"(s));
  asm("mov.b64 %0, {%1, %1};" : "=l"(*base) : "f"(b));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Slots of the children of a node whose boxes the ray enters before tmax.  The
// far distance counts 4e-6 more, which exceeds the rounding of the distances
// here and slab's factor.  An axis whose frame is
// not finite is NaN, which the minima and maxima ignore: it culls nothing.  A child
// is out when far * 1.000004 - near has its sign set.
__device__ __forceinline__ uint32_t wide_hits(const WideRay& s, uint4 w0, uint4 w2, uint4 w3, uint4 w4) {
  unsigned long long sx, bx, sy, by, sz, bz;
  wide_axis(__uint_as_float(w0.x), s.o.x, s.invd.x, w0.w & 255u, &sx, &bx);
  wide_axis(__uint_as_float(w0.y), s.o.y, s.invd.y, (w0.w >> 8) & 255u, &sy, &by);
  wide_axis(__uint_as_float(w0.z), s.o.z, s.invd.z, (w0.w >> 16) & 255u, &sz, &bz);
  const bool px = s.oct & 1u, py = s.oct & 2u, pz = s.oct & 4u;
  uint32_t out = 0;  // from slot 7 down, one sign after the other
#define R2_WIDE_CHILD(half, k)                                                                        \
  {                                                                                                   \
    float nx, fx, ny, fy, nz, fz;                                                                     \
    wide_planes(wide_byte<k>(n##half##x), wide_byte<k>(f##half##x), sx, bx, &nx, &fx);                \
    wide_planes(wide_byte<k>(n##half##y), wide_byte<k>(f##half##y), sy, by, &ny, &fy);                \
    wide_planes(wide_byte<k>(n##half##z), wide_byte<k>(f##half##z), sz, bz, &nz, &fz);                \
    const float tn = fmaxf(max3(nx, ny, nz), 0.0f), tf = fminf(min3(fx, fy, fz), s.tmax);             \
    out = __funnelshift_l(__float_as_uint(fmaf(tf, 1.000004f, -tn)), out, 1);                         \
  }
  {
    const uint32_t n1x = px ? w2.y : w3.w, f1x = px ? w3.w : w2.y;
    const uint32_t n1y = py ? w2.w : w4.y, f1y = py ? w4.y : w2.w;
    const uint32_t n1z = pz ? w3.y : w4.w, f1z = pz ? w4.w : w3.y;
    R2_WIDE_CHILD(1, 3) R2_WIDE_CHILD(1, 2) R2_WIDE_CHILD(1, 1) R2_WIDE_CHILD(1, 0)
  }
  {
    const uint32_t n0x = px ? w2.x : w3.z, f0x = px ? w3.z : w2.x;
    const uint32_t n0y = py ? w2.z : w4.x, f0y = py ? w4.x : w2.z;
    const uint32_t n0z = pz ? w3.x : w4.z, f0z = pz ? w4.z : w3.x;
    R2_WIDE_CHILD(0, 3) R2_WIDE_CHILD(0, 2) R2_WIDE_CHILD(0, 1) R2_WIDE_CHILD(0, 0)
  }
#undef R2_WIDE_CHILD
  return ~out & 0xFFu;
}

// Slots to places along the ray: bit s to bit s ^ oct.
__device__ __forceinline__ uint32_t wide_permute(uint32_t m, uint32_t oct) {
  m = oct & 1u ? ((m & 0x55u) << 1) | ((m >> 1) & 0x55u) : m;
  m = oct & 2u ? ((m & 0x33u) << 2) | ((m >> 2) & 0x33u) : m;
  return oct & 4u ? ((m & 0x0Fu) << 4) | (m >> 4) : m;
}

// Tests w.tris[first .. first + n-1], n <= 32, one per lane: tri_test's
// arithmetic with the ray of the lane that entered the leaf.
template <bool kAnyHit, bool kAlpha>
__device__ __forceinline__ void wide_test(const BvhView& bvh, WideWarp& w, int first, int n, int lane) {
  __syncwarp();
  int owner = 0;
  unsigned long long key = 0;
  float b1 = 0.0f, b2 = 0.0f;
  bool hit = false;
  if (lane < n) {
    const uint32_t item = w.tris[first + lane];
    owner = (int)(item >> 26);
    const int tri = (int)(item & 0x03FFFFFFu);
    const float4 a = __ldg(&bvh.tris[3 * (size_t)tri]), b = __ldg(&bvh.tris[3 * (size_t)tri + 1]),
                 c = __ldg(&bvh.tris[3 * (size_t)tri + 2]);
    const float4 ra = w.a[owner], rb = w.b[owner];
    const V3 o = v3(ra.x, ra.y, ra.z);
    const float Sx = ra.w, Sy = rb.x, Sz = rb.y;
    const int kz = __float_as_int(rb.z);
    const V3 A = v3(a.x, a.y, a.z) - o, B = v3(b.x, b.y, b.z) - o, C = v3(c.x, c.y, c.z) - o;
    const bool z0 = kz == 0, z1 = kz == 1;
    const float Az0 = z0 ? A.x : (z1 ? A.y : A.z), Bz0 = z0 ? B.x : (z1 ? B.y : B.z), Cz0 = z0 ? C.x : (z1 ? C.y : C.z);
    const float Ax = (z0 ? A.y : (z1 ? A.z : A.x)) - Sx * Az0, Ay = (z0 ? A.z : (z1 ? A.x : A.y)) - Sy * Az0;
    const float Bx = (z0 ? B.y : (z1 ? B.z : B.x)) - Sx * Bz0, By = (z0 ? B.z : (z1 ? B.x : B.y)) - Sy * Bz0;
    const float Cx = (z0 ? C.y : (z1 ? C.z : C.x)) - Sx * Cz0, Cy = (z0 ? C.z : (z1 ? C.x : C.y)) - Sy * Cz0;
    float U = Cx * By - Cy * Bx;
    float V = Ax * Cy - Ay * Cx;
    float W = Bx * Ay - By * Ax;
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
      U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
      V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
      W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
    }
    const float det = U + V + W;
    if (!(fminf(fminf(U, V), W) < 0.0f && fmaxf(fmaxf(U, V), W) > 0.0f) && det != 0.0f) {
      const float T = U * (Sz * Az0) + V * (Sz * Bz0) + W * (Sz * Cz0);
      const float rcp = 1.0f / det;
      const float t = T * rcp;
      b1 = V * rcp;
      b2 = W * rcp;
      key = ((unsigned long long)__float_as_uint(t) << 32) | (uint32_t)(tri + __float_as_int(rb.w));
      hit = t > 0.0f && key < w.key[owner] && (!kAlpha || alpha_opaque(bvh.alpha, tri, b1, b2));
      if (hit) atomicMin(&w.key[owner], key);
    }
  }
  __syncwarp();
  if (!kAnyHit && hit && w.key[owner] == key) w.bary[owner] = make_float2(b1, b2);
  __syncwarp();
}

// Takes the last n <= 32 of the waiting leaves (nl of them, counted down) and
// tests triangles while 32 wait (all: until none do).
template <bool kAnyHit, bool kAlpha>
__device__ __forceinline__ void wide_leaves(const BvhView& bvh, const WideView& wide, WideWarp& w, int& nl, int& nt,
                                            int n, bool all, int lane) {
  __syncwarp();
  nl -= n;
  uint32_t owner = 0, tri = 0;
  int count = 0;
  if (lane < n) {
    const uint2 leaf = w.leaves[nl + lane];
    const uint32_t ref = __ldg(reinterpret_cast<const uint32_t*>(wide.nodes) + leaf.y);
    owner = leaf.x;
    tri = ref & 0x03FFFFFFu;
    count = (int)(ref >> 26);
  }
  int end = count;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, end, off);
    if (lane >= off) end += o;
  }
  uint32_t* out = w.tris + nt + end - count;
  for (int k = 0; k < count; ++k) out[k] = (owner << 26) | (tri + (uint32_t)k);
  nt += __shfl_sync(0xffffffffu, end, 31);
  while (nt >= 32 || (all && nt > 0)) {
    const int m = min(nt, 32);
    nt -= m;
    wide_test<kAnyHit, kAlpha>(bvh, w, nt, m, lane);
  }
}

// Traces items 0 .. n-1 of a queue that all warps of the grid share (taken: its
// head).  begin(k, &o, &d, &tmax, &item) starts item k (false: no ray);
// end(item, hit) takes the closest hit, kAnyHit: any (tri -1: none).  Lanes
// whose ray is done wait until `refill` of them do; then the queued triangles
// are tested, the rays end and the lanes take new ones, after at most `visits`
// node steps between looks at the others.  Results depend on neither.  The
// stack holds at most one group of nodes per level of the tree and, in
// two-level scenes (kInst), a group of leaves and a marker for the instance:
// the builder bounds the height of the binary tree, which is no less, so
// R2_BVH_STACK entries suffice.  A ray unfinished after kMaxTraceVisits steps (a
// correct traversal visits each node once) ends as a miss, counted in *bound.
constexpr int kMaxTraceVisits = 1 << 26;
// Once no items are left a warp tests what waits every so many steps, not
// whenever lanes are idle (moving spheres at 853x480: 3.89 -> 3.81 ms).
constexpr int kWideDrain = 4;

template <bool kAnyHit, bool kAlpha, bool kInst, class Begin, class End>
__device__ __forceinline__ void wide_rays(const BvhView& bvh, const WideView& wide, WideWarp& w, uint32_t n,
                                          uint32_t* taken, int visits, int refill, unsigned int* bound, Begin begin,
                                          End end) {
  uint2 stack[R2_BVH_STACK];
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  WideRay r;
  r.sp = 0;
  r.group = make_uint2(0u, 0u);
  V3 wo, wd;          // the ray in world space
  uint32_t item = 0;
  int spent = 0;
  bool has = false;   // the lane has a ray
  bool run = false;   // and nodes to visit for it
  int enter = -1;     // two-level: the instance to enter (or, -2, to leave) once its triangles are tested
  bool queued = false;  // two-level: some may still wait
  bool more = true;   // warp-uniform: the queue may still hold items
  int drained = 0;    // rounds since the queue ran out
  int nl = 0, nt = 0; // warp-uniform: leaves and triangles that wait
  while (true) {
    const unsigned running = __ballot_sync(0xffffffffu, run || (kInst && has && enter != -1 && !queued));
    if ((more && 32 - __popc(running) >= refill) || running == 0u || (!more && ++drained >= kWideDrain)) {
      drained = 0;
      if (nl + nt > 0) wide_leaves<kAnyHit, kAlpha>(bvh, wide, w, nl, nt, nl, true, lane);
      queued = false;
      if (has) r.tmax = __uint_as_float((uint32_t)(w.key[lane] >> 32));
      if (kAnyHit && has && (uint32_t)w.key[lane] != kWideNoHit) run = false;
      if (has && !run) {
        if (!kInst || enter == -1 || (kAnyHit && (uint32_t)w.key[lane] != kWideNoHit)) {
          const unsigned long long key = w.key[lane];
          Hit h;
          h.t = __uint_as_float((uint32_t)(key >> 32));
          h.tri = (uint32_t)key == kWideNoHit ? -1 : (int)(uint32_t)key;
          h.b1 = h.b2 = 0.0f;
          if (!kAnyHit && h.tri >= 0) {
            h.b1 = w.bary[lane].x;
            h.b2 = w.bary[lane].y;
          }
          end(item, wo, wd, h);
          has = false;
        }
      }
      const unsigned want = __ballot_sync(0xffffffffu, !has);
      if (more && want) {
        const uint32_t count = (uint32_t)__popc(want);
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(taken, count);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base + count >= n) more = false;
        const uint32_t k = base + (uint32_t)__popc(want & below);
        if (!has && k < n) {
          float tmax;
          if (begin(k, &wo, &wd, &tmax, &item)) {
            has = run = true;
            enter = -1;
            spent = 0;
            r.sp = 0;
            r.tmax = tmax;
            w.key[lane] = ((unsigned long long)__float_as_uint(tmax) << 32) | kWideNoHit;
            wide_set(r, w, lane, wo, wd, 0, 0u);
            if (!(tmax > 0.0f)) run = false;  // nothing in (0, tmax]
          }
        }
      } else if (want == 0xffffffffu) {
        break;
      }
      __syncwarp();
    }
    // Rays that enter an instance, or leave one without a leaf in the queue, need
    // not wait for the queue to be emptied (144 instances of 20,480 triangles
    // 19.2 -> 18.6 ms, 225 of 320 triangles at 605x252 3.85 -> 3.64 ms; looking
    // for them sooner, at 4 or 8 such lanes, gained no more).
    if (kInst) {
      if (has && enter != -1 && !queued) {
        if (enter == -2) {
          wide_set(r, w, lane, wo, wd, 0, 0u);
          r.group.y = 0u;
        } else {
          const BvhInstance& in = bvh.inst[enter];
          if (in.identity) wide_set(r, w, lane, wo, wd, in.vdelta, (uint32_t)in.wide);
          else wide_set(r, w, lane, inst_point(in, wo), inst_vector(in, wd), in.vdelta, (uint32_t)in.wide);
        }
        enter = -1;
        run = true;
      }
      __syncwarp();
    }
    for (int step = 0; step < visits; ++step) {
      uint32_t leaves = 0, word = 0;  // leaf slots of the node to test, the word of slot 0
      if (run) {
        bool instances = false;
        if ((r.group.y & 0xFFu) == 0u) {  // the next group
          if (r.sp == 0) {
            run = false;
          } else {
            const uint2 e = stack[--r.sp];
            if (kInst && e.y == kWideExit) {
              run = false;
              enter = -2;
            } else if (kInst && (e.y & kWideLeafGroup)) {
              instances = true;
              leaves = e.y & 0xFFu;
              word = e.x;
            } else {
              r.group = e;
            }
          }
        }
        if (run && !instances) {
          // the group's nearest child
          const uint32_t place = 31u - __clz(r.group.y & 0xFFu), slot = place ^ r.oct;
          r.group.y ^= 1u << place;
          const uint32_t node = r.group.x + __popc((r.group.y >> 8) & ((1u << slot) - 1u));
          if (r.group.y & 0xFFu) stack[r.sp++] = r.group;
          const uint4* nd = wide.nodes + kWideWords * (size_t)node;
          const uint4 w0 = __ldg(nd), w1 = __ldg(nd + 1), w2 = __ldg(nd + 2), w3 = __ldg(nd + 3), w4 = __ldg(nd + 4);
          const uint32_t hits = wide_hits(r, w0, w2, w3, w4), inner = w0.w >> 24;
          r.group = make_uint2(w1.x, (inner << 8) | wide_permute(hits & inner, r.oct));
          leaves = hits & w1.y;
          word = node * (4u * kWideWords) + 20u;
          if (kInst) instances = w1.z != 0u && leaves != 0u;
          if (++spent >= kMaxTraceVisits) {
            run = false;
            leaves = 0u;
            w.key[lane] = kWideNoHit;
            atomicAdd(bound, 1u);
          }
        }
        if (kInst && instances && leaves) {  // one is entered, what is left of the node waits on the stack
          if (r.group.y & 0xFFu) stack[r.sp++] = r.group;
          enter = (int)__ldg(reinterpret_cast<const uint32_t*>(wide.nodes) + word + (__ffs(leaves) - 1));
          leaves &= leaves - 1u;
          if (leaves) stack[r.sp++] = make_uint2(word, kWideLeafGroup | leaves);
          stack[r.sp++] = make_uint2(0u, kWideExit);
          r.group.y = 0u;
          leaves = 0u;
          run = false;
        }
      }
      // to the queue, one per lane at a time
      while (true) {
        const unsigned m = __ballot_sync(0xffffffffu, leaves != 0u);
        if (m == 0u) break;
        if (leaves) {
          w.leaves[nl + __popc(m & below)] = make_uint2((uint32_t)lane, word + __ffs(leaves) - 1u);
          leaves &= leaves - 1u;
          queued = true;
        }
        nl += __popc(m);
        if (nl >= 32) {
          wide_leaves<kAnyHit, kAlpha>(bvh, wide, w, nl, nt, 32, false, lane);
          if (has) r.tmax = __uint_as_float((uint32_t)(w.key[lane] >> 32));
          if (kAnyHit && has && (uint32_t)w.key[lane] != kWideNoHit) {
            run = false;
            leaves = 0u;
          }
        }
      }
      if (32 - __popc(__ballot_sync(0xffffffffu, run)) >= refill) break;
    }
  }
}

#endif  // __CUDACC__

}  // namespace r2
