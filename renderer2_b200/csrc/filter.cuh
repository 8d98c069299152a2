// SGGX mesh-to-volume filter: device kernels and their launch description.
#pragma once
#include "bvh_build.cuh"

namespace r2 {

constexpr uint32_t kFilterMaxSpv = 1024;  // per-voxel sample cap (reference: rayTs[1000])
constexpr int kWideFloats = 20;           // floats per voxel of the wide (pre-quantisation) output

// Everything the per-voxel kernels read.  Passed by value (kernel parameter
// space), so each launch is self-contained and graph-capturable.
struct FilterLaunch {
  M43 indexToWorld;   // mat4(modelToWorld) * mat4(indexToModel)
  M43 indexToModel;   // voxel index -> model space (COpenvdbBackend::setupGrid)
  M43 modelToWorld;   // grid model -> world (voxel centres, COpenvdbBackend::setupGrid)
  M43 objModelToWorld;  // the object's own transform (hit normals, shaders.optix.cu:106)
  M43 worldToModel;   // mean-normal transform back to model space
  int nx, ny, nz;
  V3 voxelSize;       // (worldBB.max - worldBB.min) / numVoxels
  uint32_t spv, iters, clip, seed, lod;
  float sigma_t, alpha;
  uint32_t project;          // FP64 eigendecomposition + projection of S (r2_filter_params::sggx_projection)
  float floor;               // relative eigenvalue floor of the projection
  BvhView bvh;
  const float4* triN;        // 3 per BVH-order triangle: model-space vertex normals
  const uint32_t* triMat;    // per BVH-order triangle: material index
  const r2_material* mats;
  r2_voxel* out;
  float* wide;               // nullable
  uint16_t* fp16;            // nullable
  float* eig;                // nullable: 12 floats per voxel, eigenvalues and eigenvectors of the mean S
  // Work of this launch: the bricks brickFirst .. brickFirst + brickCount - 1
  // (2x2x2 voxels, x fastest), the ones near triangles
  // (bricks), the voxels to sample (entries: index and place of the candidate
  // list in the pool, from both ends) and the counters.
  uint32_t brickFirst, brickCount;
  float brickOffset;         // from a brick's centre to its farthest voxel centre
  float ballScale;           // of the triangle tests (tri_ball.h)
  uint32_t* bricks;
  uint2* entries;
  int* pool;                 // candidate lists: their length, then triangles
  uint32_t poolWords;
  uint32_t* counters;        // kFilterCounters of them, see below
  unsigned long long* ops;   // nullable: counting build, [0] rays, [1] inner nodes visited, [2] triangles tested
  // texture maps (nullable): 3 texture coordinates per BVH-order triangle, the
  // texels, and per material its {albedo, glossy, normal, opacity} texture (-1: none)
  const float2* triUV;
  const float4* texels;
  const TexInfo* texInfo;
  const int4* matTex;
};

// Counters of a launch: voxels with a triangle within reach (of the whole
// grid); then, cleared for every part of it, the bricks listed, the entries
// taken, the entries at the end of the list, and those at its front and the
// pool words used (one 64-bit word).
enum { kCountSampled = 0, kCountBricks = 1, kCountTaken = 2, kCountBack = 3, kCountFront = 4, kFilterCounters = 6 };

// Bricks of the grid, x fastest.
R2_HD uint32_t brick_count(const FilterLaunch& L) {
  return ((uint32_t)(L.nx + 1) / 2) * ((uint32_t)(L.ny + 1) / 2) * ((uint32_t)(L.nz + 1) / 2);
}

// Host launchers of one part of a grid.  `lists` writes the empty payload of
// voxels that no triangle is near and collects the others and their candidate
// triangles; `sample` is the persistent warp-per-voxel kernel.
void launch_filter_lists(const FilterLaunch& L, cudaStream_t s);
void launch_filter_sample(const FilterLaunch& L, cudaStream_t s);

}  // namespace r2
