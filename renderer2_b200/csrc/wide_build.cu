// Collapse of a binary BVH into the eight-wide one (wide_bvh.cuh).
//
// Top down: a wide node takes the two children of its binary node and opens
// the inner child of largest area until it has eight or only leaves.  Wide
// nodes are numbered as they are allocated (the children of a node in a row),
// and queue[i] keeps the binary node of wide node i, so the work of a level is
// a range of numbers.  The first levels, a few hundred nodes, run in one block
// (a barrier costs less than a launch), the next in launches of their own,
// and whatever lies deeper is finished by a thread per subtree.
#include <algorithm>

#include "bvh_build.cuh"
#include "wide_bvh.cuh"

namespace r2 {
namespace {

constexpr int kTopThreads = 1024;
constexpr uint32_t kTopItems = 1024;  // items of a level from which it is a launch of its own
constexpr int kLevels = 3;            // levels in launches of their own
// counters: nodes allocated, blocks done, then per launch the range of its level
enum { kWideNodes = 0, kWideDone = 1, kWideRange = 2, kWideState = kWideRange + 2 * (kLevels + 1) };

struct WideBuild {
  const BvhNode* nodes;
  uint4* out;
  uint32_t* queue;
  uint32_t* state;
};

// One axis of a node's frame: the smallest power of two 2^e in whose units the
// box and one unit below it take at most 254, and an origin at least one unit
// below the box, so that a child's planes and 1/64 unit around them (far more
// than the traversal's rounding in units) lie within 0 .. 255.  Far from zero a
// unit can be less than lo's unit in the last place: the origin is rounded down
// and the unit grown until the box fits above it; a box without extent counts as
// one of about a unit in the last place.  Units stay between 2^-42 and 2^23 (see
// wide_rcp); a box of more than 2e9 or an infinite one gets an infinite unit, whose planes are no numbers: the axis then culls nothing.
__device__ __forceinline__ void frame_axis(float lo, float hi, float* origin, uint32_t* exponent) {
  int e = 0;
  const float ext = fmaxf(hi - lo, 1.2e-7f * fmaxf(fabsf(lo), fabsf(hi)));
  frexpf(ext / 252.0f, &e);
  if (!(ext > 0.0f)) e = -42;
  float from = lo;
  for (e = max(e, -42); isfinite(ext) && e <= 23; ++e) {
    from = __fsub_rd(lo, __uint_as_float((uint32_t)(e + 127) << 23));
    if (__fsub_ru(hi, from) * __uint_as_float((uint32_t)(127 - e) << 23) <= 254.0f) break;
  }
  *exponent = isfinite(ext) && e <= 23 ? (uint32_t)(e + 127) : 255u;
  *origin = from;
}
// (x - origin and the scaling are exact or within 2e-5 of a unit.)
__device__ __forceinline__ uint32_t plane(float x, float origin, float perUnit, bool upper) {
  const float q = (x - origin) * perUnit;
  const float r = upper ? ceilf(q + 0.015625f) : floorf(q - 0.015625f);
  if (!(r >= 0.0f)) return upper && !(r < 0.0f) ? 255u : 0u;  // NaN: the whole frame
  return (uint32_t)fminf(r, 255.0f);
}

static_assert(kLeafMax <= 8, "a warp's triangle queue has room for eight of each of 32 leaves");

__device__ void collapse(const WideBuild& B, uint32_t w) {
  WideBox box[9];
  int ref[9];
  const int n = wide_open(B.nodes, B.queue[w], box, ref);
  WideBox all = box[0];
  for (int i = 1; i < n; ++i) all = WideBox{vmin(all.lo, box[i].lo), vmax(all.hi, box[i].hi)};
  // children to slots, the largest child first: the free slot whose octant fits its offset best
  int childAt[8];
  for (int k = 0; k < 8; ++k) childAt[k] = -1;
  uint32_t placed = 0;
  for (int round = 0; round < n; ++round) {
    int c = -1;
    for (int i = 0; i < n; ++i)
      if (!(placed >> i & 1u) && (c < 0 || wide_area(box[i]) > wide_area(box[c]))) c = i;
    placed |= 1u << c;
    const V3 off = (box[c].lo + box[c].hi) - (all.lo + all.hi);
    int slot = -1;
    float best = 0.0f;
    for (int k = 0; k < 8; ++k) {
      const float fit = (k & 1 ? off.x : -off.x) + (k & 2 ? off.y : -off.y) + (k & 4 ? off.z : -off.z);
      if (childAt[k] < 0 && (slot < 0 || fit > best)) {
        slot = k;
        best = fit;
      }
    }
    childAt[slot] = c;
  }
  uint32_t inner = 0, leaf = 0;
  for (int k = 0; k < 8; ++k)
    if (childAt[k] >= 0) (ref[childAt[k]] >= 0 ? inner : leaf) |= 1u << k;
  const uint32_t firstChild = inner ? atomicAdd(&B.state[kWideNodes], (uint32_t)__popc(inner)) : 0u;
  float px, py, pz;
  uint32_t ex, ey, ez;
  frame_axis(all.lo.x, all.hi.x, &px, &ex);
  frame_axis(all.lo.y, all.hi.y, &py, &ey);
  frame_axis(all.lo.z, all.hi.z, &pz, &ez);
  const float ux = __uint_as_float((254u - ex) << 23), uy = __uint_as_float((254u - ey) << 23), uz = __uint_as_float((254u - ez) << 23);
  uint32_t q[6][2] = {};  // lo.x lo.y lo.z hi.x hi.y hi.z of the eight slots
  uint32_t child = firstChild, leafWord[8] = {}, instances = 0;
  for (int k = 0; k < 8; ++k) {
    const int c = childAt[k];
    if (c < 0) continue;
    const WideBox& b = box[c];
    const int half = k >> 2, shift = 8 * (k & 3);
    q[0][half] |= plane(b.lo.x, px, ux, false) << shift;
    q[1][half] |= plane(b.lo.y, py, uy, false) << shift;
    q[2][half] |= plane(b.lo.z, pz, uz, false) << shift;
    q[3][half] |= plane(b.hi.x, px, ux, true) << shift;
    q[4][half] |= plane(b.hi.y, py, uy, true) << shift;
    q[5][half] |= plane(b.hi.z, pz, uz, true) << shift;
    if (ref[c] >= 0) {
      B.queue[child++] = (uint32_t)ref[c];
    } else {
      leafWord[k] = (uint32_t)~ref[c];
      if (bvh_leaf_count(ref[c]) == 0) instances = 1u;
    }
  }
  uint4* out = B.out + kWideWords * (size_t)w;
  out[0] = make_uint4(__float_as_uint(px), __float_as_uint(py), __float_as_uint(pz), ex | ey << 8 | ez << 16 | inner << 24);
  out[1] = make_uint4(firstChild, leaf, instances, 0u);
  out[2] = make_uint4(q[0][0], q[0][1], q[1][0], q[1][1]);
  out[3] = make_uint4(q[2][0], q[2][1], q[3][0], q[3][1]);
  out[4] = make_uint4(q[4][0], q[4][1], q[5][0], q[5][1]);
  out[5] = make_uint4(leafWord[0], leafWord[1], leafWord[2], leafWord[3]);
  out[6] = make_uint4(leafWord[4], leafWord[5], leafWord[6], leafWord[7]);
}

// The first levels: wide nodes 0 .. nroots-1, whose binary nodes are in the
// queue, and down from them.
__global__ void __launch_bounds__(kTopThreads) k_wide_top(WideBuild B, uint32_t nroots) {
  if (threadIdx.x == 0) B.state[kWideNodes] = nroots;
  __syncthreads();
  uint32_t first = 0, end = nroots;
  while (first < end && end - first < kTopItems) {
    for (uint32_t w = first + threadIdx.x; w < end; w += kTopThreads) collapse(B, w);
    __syncthreads();
    first = end;
    end = *(volatile uint32_t*)&B.state[kWideNodes];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    B.state[kWideRange] = first;
    B.state[kWideRange + 1] = end;
  }
}

// One level; the last block to finish writes the range of the next.
__global__ void __launch_bounds__(64) k_wide_level(WideBuild B, int level) {
  const uint32_t first = B.state[kWideRange + 2 * level], end = B.state[kWideRange + 2 * level + 1];
  for (uint32_t w = first + blockIdx.x * blockDim.x + threadIdx.x; w < end; w += gridDim.x * blockDim.x) collapse(B, w);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&B.state[kWideDone], 1u) == gridDim.x - 1) {
    B.state[kWideDone] = 0u;
    B.state[kWideRange + 2 * (level + 1)] = end;
    B.state[kWideRange + 2 * (level + 1) + 1] = *(volatile uint32_t*)&B.state[kWideNodes];
  }
}

// The rest, each subtree depth first by one thread: the stack holds the
// children still to do of every node above, one entry per level.
__global__ void __launch_bounds__(64) k_wide_rest(WideBuild B) {
  const uint32_t first = B.state[kWideRange + 2 * kLevels], end = B.state[kWideRange + 2 * kLevels + 1];
  for (uint32_t w = first + blockIdx.x * blockDim.x + threadIdx.x; w < end; w += gridDim.x * blockDim.x) {
    uint2 stack[R2_BVH_STACK];  // next node, nodes left
    int sp = 0;
    stack[sp++] = make_uint2(w, 1u);
    while (sp > 0) {
      const uint32_t node = stack[sp - 1].x;
      ++stack[sp - 1].x;
      if (--stack[sp - 1].y == 0u) --sp;
      collapse(B, node);
      const uint4* n = B.out + kWideWords * (size_t)node;
      const uint32_t children = (uint32_t)__popc(n[0].w >> 24);
      if (children) stack[sp++] = make_uint2(n[1].x, children);
    }
  }
}

}  // namespace

void WideBvh::build(const BvhNode* nodes, const uint32_t* roots, uint32_t nroots, uint32_t nleaves,
                    cudaStream_t s) {
  const size_t cap = wide_capacity(nleaves, nroots);
  reserve_together(mem_, part(nodes_, cap * kWideWords), part(queue_, cap), part(state_, kWideState));
  R2_CUDA(cudaMemsetAsync(state_.get(), 0, kWideState * sizeof(uint32_t), s));
  if (roots) R2_CUDA(cudaMemcpyAsync(queue_.get(), roots, nroots * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
  else R2_CUDA(cudaMemsetAsync(queue_.get(), 0, sizeof(uint32_t), s));
  const WideBuild B = {nodes, nodes_.get(), queue_.get(), state_.get()};
  k_wide_top<<<1, kTopThreads, 0, s>>>(B, nroots);
  const int blocks = sm_count() * 4;
  for (int level = 0; level < kLevels; ++level) k_wide_level<<<blocks, 64, 0, s>>>(B, level);
  k_wide_rest<<<blocks, 64, 0, s>>>(B);
  R2_CUDA(cudaGetLastError());
}

}  // namespace r2
