// What tests call below the library's C interface: the filter's test of a
// triangle against a ball (no GPU); of the eight-wide BVH the collapse's choice of children over a host-built binary tree (no GPU), and
// the closest hits of given rays through the wide tree and through the binary
// one over the same build.  Compiled and loaded by wide_probe.py.
#include <cstring>
#include <vector>

#include "bvh_build.cuh"
#include "tri_ball.h"
#include "wide_bvh.cuh"

using namespace r2;

namespace {

struct HostTree {
  std::vector<BvhNode> nodes;
  const float* boxes;  // 6 floats a leaf: lo, hi
  uint32_t state;

  uint32_t random() { return state = state * 1664525u + 1013904223u; }
  // The subtree over leaves first .. first + n - 1; box: its bounds (fminf and fmaxf of its leaves', as the builders').
  int add(uint32_t first, uint32_t n, int skew, WideBox* box) {
    if (n == 1) {
      const float* b = boxes + 6 * (size_t)first;
      *box = WideBox{v3(b[0], b[1], b[2]), v3(b[3], b[4], b[5])};
      return bvh_leaf_ref((int)first, 1);
    }
    const uint32_t left = skew == 0 ? n / 2 : 1 + (random() >> 8) % (n - 1);
    const int me = (int)nodes.size();
    nodes.push_back(BvhNode());
    WideBox b[2];
    const int l = add(first, left, skew, &b[0]), r = add(first + left, n - left, skew, &b[1]);
    BvhNode& nd = nodes[me];
    nd.b0 = make_float4(b[0].lo.x, b[0].hi.x, b[0].lo.y, b[0].hi.y);
    nd.b1 = make_float4(b[1].lo.x, b[1].hi.x, b[1].lo.y, b[1].hi.y);
    nd.bz = make_float4(b[0].lo.z, b[0].hi.z, b[1].lo.z, b[1].hi.z);
    nd.ch = make_int4(l, r, 0, 0);
    *box = WideBox{vmin(b[0].lo, b[1].lo), vmax(b[0].hi, b[1].hi)};
    return me;
  }
};

struct Ray {
  float o[3], d[3], tmax;
};

__global__ void k_wide(BvhView bvh, WideView wide, const Ray* rays, uint32_t n, uint32_t* taken, unsigned int* bound,
                       float4* closest, int* any) {
  __shared__ WideWarp warps[4];
  auto begin = [&](uint32_t k, V3* o, V3* d, float* tmax, uint32_t* item) {
    *item = k;
    *o = v3(rays[k].o[0], rays[k].o[1], rays[k].o[2]);
    *d = v3(rays[k].d[0], rays[k].d[1], rays[k].d[2]);
    *tmax = rays[k].tmax;
    return true;
  };
  auto put = [&](uint32_t k, V3, V3, const Hit& h) {
    closest[k] = make_float4(h.t, h.b1, h.b2, __int_as_float(h.tri));
  };
  auto seen = [&](uint32_t k, V3, V3, const Hit& h) { any[k] = h.tri >= 0; };
  wide_rays<false, false, false>(bvh, wide, warps[threadIdx.x >> 5], n, &taken[0], 32, 16, bound, begin, put);
  __syncwarp();
  wide_rays<true, false, false>(bvh, wide, warps[threadIdx.x >> 5], n, &taken[1], 32, 16, bound, begin, seen);
}

__global__ void k_binary(BvhView bvh, const Ray* rays, uint32_t n, float4* closest) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const Hit h = bvh_trace(bvh, v3(rays[k].o[0], rays[k].o[1], rays[k].o[2]),
                                   v3(rays[k].d[0], rays[k].d[1], rays[k].d[2]), rays[k].tmax);
    closest[k] = make_float4(h.t, h.b1, h.b2, __int_as_float(h.tri));
  }
}

__global__ void k_all(BvhView bvh, const Ray* rays, uint32_t n, float4* closest) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const RayPre r = make_ray_pre(v3(rays[k].o[0], rays[k].o[1], rays[k].o[2]),
                                  v3(rays[k].d[0], rays[k].d[1], rays[k].d[2]));
    Hit h;
    h.t = rays[k].tmax;
    h.b1 = h.b2 = 0.0f;
    h.tri = 0x7FFFFFFF;
    for (uint32_t t = 0; t < bvh.ntris; ++t) {
      const float4 a = bvh.tris[3 * t], b = bvh.tris[3 * t + 1], c = bvh.tris[3 * t + 2];
      tri_test(r, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z), (int)t, (int)t, &h);
    }
    closest[k] = make_float4(h.t, h.b1, h.b2, __int_as_float(h.tri == 0x7FFFFFFF ? -1 : h.tri));
  }
}

// Wide nodes whose boxes each ray enters before its tmax.
__global__ void k_visits(WideView wide, const Ray* rays, uint32_t n, uint32_t* visits) {
  __shared__ WideWarp warps[4];
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    WideRay r;
    wide_set(r, warps[threadIdx.x >> 5], threadIdx.x & 31, v3(rays[k].o[0], rays[k].o[1], rays[k].o[2]),
             v3(rays[k].d[0], rays[k].d[1], rays[k].d[2]), 0, 0u);
    r.tmax = rays[k].tmax;
    uint2 stack[R2_BVH_STACK];  // first child, inner children to visit and, above them, all
    int sp = 0;
    stack[sp++] = make_uint2(0u, 0x0101u);
    uint32_t count = 0;
    while (sp > 0) {
      const uint32_t hits = stack[sp - 1].y & 0xFFu, slot = __ffs(hits) - 1u;
      const uint32_t node = stack[sp - 1].x + __popc((stack[sp - 1].y >> 8) & ((1u << slot) - 1u));
      stack[sp - 1].y &= ~(1u << slot);
      if (!(stack[sp - 1].y & 0xFFu)) --sp;
      const uint4* nd = wide.nodes + kWideWords * (size_t)node;
      const uint32_t inner = nd[0].w >> 24, in = wide_hits(r, nd[0], nd[2], nd[3], nd[4]) & inner;
      ++count;
      if (in) stack[sp++] = make_uint2(nd[1].x, inner << 8 | in);
    }
    visits[k] = count;
  }
}

}  // namespace

extern "C" {

// near[k]: whether tri_near keeps triangle k (9 floats) for a ball of radius r[k] about c[3k..], whose test was set up
// for centres within around[k] of c0[3k..], among voxels of the given size.
void probe_tri_near(const float* tris, const float* c0, const float* around, const float* c, const float* r, float voxel,
                    uint32_t n, int* near) {
  const float scale = ball_scale(voxel);
  const auto at = [](const float* p) { return v3(p[0], p[1], p[2]); };
  for (uint32_t k = 0; k < n; ++k) {
    const float* t = tris + 9 * (size_t)k;
    near[k] = tri_near(tri_ball(at(t), at(t + 3), at(t + 6), at(c0 + 3 * (size_t)k), around[k], r[k], scale),
                       at(c + 3 * (size_t)k));
  }
}

// Wide nodes of the collapse of a binary tree over the leaf boxes (skew: 0 halves, 1 splits anywhere); *capacity: what
// the builder has room for.
uint64_t probe_wide_nodes(const float* boxes, uint32_t nleaves, int skew, uint32_t seed, uint64_t* capacity) {
  HostTree t;
  t.boxes = boxes;
  t.state = seed;
  WideBox all;
  t.add(0, nleaves, skew, &all);
  *capacity = wide_capacity(nleaves, 1);
  uint64_t count = 0;
  std::vector<uint32_t> todo(1, 0u);
  while (!todo.empty()) {
    const uint32_t node = todo.back();
    todo.pop_back();
    ++count;
    WideBox box[9];
    int ref[9];
    const int n = wide_open(t.nodes.data(), node, box, ref);
    for (int i = 0; i < n; ++i)
      if (ref[i] >= 0) todo.push_back((uint32_t)ref[i]);
  }
  return count;
}

// Buffers placed in one allocation by two users that ask for different parts of it in turn, as a builder does for
// triangles (large) and for boxes (none of the first part, more of the others): how often a buffer moved after the
// first turn of each.
int probe_reserve_moves(uint32_t large, uint32_t more, int turns) {
  try {
    DBuf<uint8_t> mem;
    DBuf<float4> boxes;
    DBuf<uint64_t> keys;
    int moves = 0;
    for (int k = 0; k < turns; ++k) {
      reserve_together(mem, part(boxes, large), part(keys, large));
      const void *a = boxes.get(), *b = keys.get();
      reserve_together(mem, part(boxes, 0), part(keys, more));
      const void *c = boxes.get(), *d = keys.get();
      if (k > 0) moves += (a != c) + (b != d);
      if (boxes.size() < large || keys.size() < more) return -1;
    }
    return moves;
  } catch (const Error&) {
    return -2;
  }
}

// Closest hits (t, b1, b2, BVH-order triangle as int bits, t free without a hit) of n rays through the wide tree,
// through the binary one and among all triangles, whether the wide
// any-hit query sees one, and the wide nodes whose boxes the ray enters.  0 on success.
int probe_trace(const float* pos, uint32_t nverts, const uint32_t* idx, uint32_t ntris, const float* rays, uint32_t n,
                float* wideHits, float* binaryHits, float* allHits, int* any, uint32_t* visits) {
  try {
    cudaStream_t s = nullptr;
    DBuf<float> dpos;
    DBuf<uint32_t> didx, taken(2);
    DBuf<unsigned int> bound(1);
    DBuf<Ray> drays;
    DBuf<float4> a(n), b(n), c(n);
    DBuf<int> dany(n);
    DBuf<uint32_t> dvisits(n);
    dpos.upload(pos, 3 * (size_t)nverts, s);
    didx.upload(idx, 3 * (size_t)ntris, s);
    drays.upload(reinterpret_cast<const Ray*>(rays), n, s);
    BvhBuilder builder;
    DeviceBvh bvh;
    builder.build(dpos.get(), didx.get(), ntris, &bvh, s);
    WideBvh wide;
    wide.build(bvh.nodes.get(), nullptr, 1, ntris, s);
    R2_CUDA(cudaMemsetAsync(taken.get(), 0, 2 * sizeof(uint32_t), s));
    R2_CUDA(cudaMemsetAsync(bound.get(), 0, sizeof(unsigned int), s));
    k_wide<<<sm_count() * 4, 128, 0, s>>>(bvh.view(), wide.view(), drays.get(), n, taken.get(), bound.get(), a.get(),
                                          dany.get());
    k_binary<<<sm_count() * 8, 128, 0, s>>>(bvh.view(), drays.get(), n, b.get());
    k_all<<<sm_count() * 8, 128, 0, s>>>(bvh.view(), drays.get(), n, c.get());
    k_visits<<<sm_count() * 8, 128, 0, s>>>(wide.view(), drays.get(), n, dvisits.get());
    R2_CUDA(cudaGetLastError());
    unsigned int ended = 0;
    a.download(reinterpret_cast<float4*>(wideHits), n, s);
    b.download(reinterpret_cast<float4*>(binaryHits), n, s);
    c.download(reinterpret_cast<float4*>(allHits), n, s);
    dany.download(any, n, s);
    dvisits.download(visits, n, s);
    bound.download(&ended, 1, s);
    R2_CUDA(cudaStreamSynchronize(s));
    return ended ? 1 : 0;
  } catch (const Error& e) {
    return 2;
  }
}

}  // extern "C"
