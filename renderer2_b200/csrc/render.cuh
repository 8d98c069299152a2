// Wavefront path tracer: launch description shared by the kernels (render.cu)
// and the host runtime (render_host.cu).
#pragma once
#include "bvh_build.cuh"
#include "media.cuh"
#include "wide_bvh.cuh"

namespace r2 {

// Analytic scene objects of the reference's scene description (Circle,
// Sphere; include/shapes/circle.hpp:35-60, sphere.hpp:33-90).
enum ShapeType : int { kShapeSphere = 0, kShapeCircle = 1 };

struct Shape {
  int type;
  int material;
  float radius;
  float pad;
  V3 center;
  V3 normal;
};

// Device view of a committed scene.
struct SceneView {
  BvhView bvh;
  WideView wide;           // the wide nodes that the surface kernels traverse
  const float4* triN;      // 3 per BVH-order triangle: world-space vertex normals
  const uint32_t* triMat;  // per BVH-order triangle: material index
  const Material* mats;
  const Shape* shapes;
  int nshapes;
  int hasTris;
  const MediumView* media;  // medium instances (device array), nullable
  int nmedia;
  const BvhNode* mediaNodes;    // BVH over the instances' world boxes (more than kMediaLinearMax), nullable
  const uint32_t* mediaOrder;   // BVH leaf position -> instance index
  EnvMap env;
  const float2* triUV;      // 3 texture coordinates per BVH-order triangle, nullable
  const float4* texels;     // texture maps of the materials (TexInfo offsets), nullable
  const TexInfo* texInfo;
  // two-level scenes (bvh.inst set): per instance the first hit code (ascending)
  // and the object-to-world 3x3 | translation rows that take its normals to world space
  const int* instCode;
  const float4* instO2W;
  int ninst;
};

// Per-path SoA state of one wave (one sample of every pixel).
struct PathState {
  float4* rayO;     // origin, .w = current medium index as int bits (-1: none)
  float4* rayD;     // direction, .w = ray tmax
  float4* T;        // throughput
  float4* L;        // radiance
  float4* hit;      // t, b1, b2, event code (int bits: >= 0 triangle, -1 miss, -2 - i shape i,
                    // kEventScatter medium collision, kEventDead path ended by a medium rule)
  uint32_t* q[2];   // ping-pong queues of live path ids
  uint32_t* qe[2];  // event lists of even and odd bounces: paths that hit a surface from the front, paths with
                    // a medium collision from the back (also the ray sort's output, before they are filled)
  uint32_t* sortBins;  // 256 key counters of the ray sort
  uint32_t* counts; // [bounce] live path count entering the bounce; from kTravCounters on,
                    // per bounce the rays taken by the persistent surface traversals
  // shadow records, two per queue slot (0: light sample, 1: BSDF sample)
  float4* shO;      // origin.xyz, pdf (0 = no ray)
  float4* shD;      // direction.xyz, unused
  float4* shPre;    // (mis * f) * Le
  float4* shT;      // throughput at the bounce (one per slot pair)
  float* shTr;      // transmittance of each shadow ray (0 or 1 without media)
  // media scenes only
  float2* shX;      // shadow ray tmax, medium index (int bits)
  float4* evA;      // collision position, ior
  float4* evB;      // collision normal, medium index (int bits)
  float4* evC;      // SGGX S xx yy zz xy
  float2* evD;      // SGGX S xz yz
  uint32_t* mc;     // per-bounce media counters
  uint32_t* pj;     // per path: medium boundaries met in the bounce up to the segment it tracks
  uint32_t* cl;     // paths whose segment ended in a collision
  float4* swP;      // shadow walk: origin of the segment it tracks, transmittance before it
  int2* swM;        // shadow walk: medium of the segment, draw index of the slot's stream
  float* swT;       // shadow walk: length of the segment
  uint32_t* pq[2];  // queued rounds: paths with a segment to track, paths that go on after one
  uint32_t* sq[2];  // the same of shadow slots
};

// top_nodes of a tuning, largest: accepted, without effect.
constexpr uint32_t kMaxTopNodes = 256;
// Launch tuning defaults (RenderLaunch::trackSteps, travVisits, travRefill);
// no result depends on them.
constexpr uint32_t kDefaultTrackSteps = 16;  // tracking steps a lane takes between refills
constexpr uint32_t kDefaultTravVisits = 32;  // BVH visits between refill checks
constexpr uint32_t kDefaultTravRefill = 16;  // finished lanes that trigger a refill
// Paths per wave a frame's samples are grouped to.  A wave's later bounces hold
// a few per cent of its paths, so larger waves keep the traversals' lanes and
// the launches full: 64 samples of 1024x1024, 98.3 / 87.3 / 81.5 ms with 4M / 8M /
// 16M paths (3.6 GB of state at 16M, 6.3 with media; 0.9 and 1.6 at 4M).  They are
// taken while memory is plenty (RenderContext::take_large); otherwise, and for
// served jobs, which share the device, waves have kServeWavePaths.
constexpr uint32_t kDefaultWavePaths = 1u << 24;
constexpr uint32_t kServeWavePaths = 1u << 22;
// Queued rounds of medium boundaries (media_rounds of a tuning) in bounces of at
// least kRoundPaths paths (shadow rays: events), of waves of at least twice as
// many; k_walk alone takes the others, and what the rounds leave.  Frames with
// rounds in bounces of 2^17 and more / of 2^18 / without: 256^3 foliage at 1920x1080,
// 16 samples 228 / 227 / 278 ms; 24,000 trees, 4 samples 133 / 133 / 144; eight
// 1080p volumes in one graph 560 / 567 / 707; 1,200 trees at 640x360, 4 samples
// 19.1 / 19.7 / 19.9.  In waves below 2^18 paths the launches cost more than they
// bring: 820x114, 2 samples 4.04 ms against 3.56, 191x439, 3 samples 7.9 against 7.2.
// One round or two or four: 227 / 228 / 230 ms of the volume, 133 / 129 / 130 of the
// trees, in waves of 4M paths 314 / 327 of the volume, 128^3 foliage at 960x540, 8
// samples 6.3 / 6.7.  In a batch of n
// frames a wave is of one sample and runs beside the others': two rounds, from
// 2 / n of the paths on, and the second stream for shadow rays only where the waves
// have no more than kBatchForkPaths in all.  Sixteen 1080p volumes, 4 samples, 4
// tracker blocks an SM: 1082 ms with one round and the second stream, 1046 without
// the stream, 1033 with two rounds, 1004 with two and without.  Twelve volumes at
// 640x360, 8 samples: 266 ms, 317 with rounds from kRoundPaths on (264 with rounds in
// every bounce, inline ends and no second stream); two at 160x90 5.6 ms, 7.5 without the
// second stream.
constexpr uint32_t kDefaultMediaRounds = 1, kBatchMediaRounds = 2, kMaxMediaRounds = 32;
constexpr size_t kBatchForkPaths = (size_t)1 << 24;
constexpr uint32_t kRoundPaths = 1u << 17;
// What the tuner tries of each setting: the default among them (the current value
// is not timed against itself), and the waves of served jobs.
constexpr uint32_t kTuneWavePaths[] = {1u << 20, 1u << 21, 1u << 22, 1u << 23, 1u << 24};
constexpr uint32_t kTuneTravRefill[] = {4, 8, 12, 16, 24}, kTuneTravVisits[] = {8, 16, 32, 64, 256};
constexpr uint32_t kTuneTrackSteps[] = {2, 4, 8, 16, 32}, kTuneMediaRounds[] = {1, 2, 4, 8};
constexpr uint32_t kTuneTrackBlocks[] = {0, 2, 3, 4, 6}, kTuneSortRays[] = {0, 1};
template <size_t N>
constexpr bool tunes(const uint32_t (&values)[N], uint32_t value) {
  for (uint32_t v : values)
    if (v == value) return true;
  return false;
}
static_assert(tunes(kTuneWavePaths, kDefaultWavePaths) && tunes(kTuneWavePaths, kServeWavePaths) &&
                  tunes(kTuneTravRefill, kDefaultTravRefill) && tunes(kTuneTravVisits, kDefaultTravVisits) &&
                  tunes(kTuneTrackSteps, kDefaultTrackSteps) && tunes(kTuneMediaRounds, kDefaultMediaRounds),
              "a default left the tuner's lists when it changed");

// Media counters of a bounce (PathState::mc): [3r] segments queued in round r,
// [3r + 1] segments taken, [3r + 2] paths that go on, for paths and, from
// kShadowCounters on, shadow slots; then paths and slots taken by k_walk, entries of
// the collision list.
constexpr int kShadowCounters = 3 * kMaxMediaRounds;
enum { kPathCounter = 2 * kShadowCounters, kShadowCounter, kCollideCounter, kCountersPerBounce = kPathCounter + 4 };

// PathState::counts layout: [0, 64) live paths per bounce, then two counters
// per bounce (extension rays taken, shadow records taken), then the surface
// hits and the medium collisions per bounce.  Shading, shadow records and
// accumulation run over the bounce's events: item i < hits is qh[i], the
// others qs[i - hits].
constexpr int kTravCounters = 64;
constexpr int kHitCounters = kTravCounters + 2 * 64;
constexpr int kScatterCounters = kHitCounters + 64;
constexpr int kCountsSize = kScatterCounters + 64;

// Scenes with at most this many medium instances test every box along a ray;
// larger ones walk the instance BVH (same result either way).
constexpr int kMediaLinearMax = 8;
constexpr size_t kMaxMediumInstances = size_t(1) << 22;

constexpr int kEventScatter = -2147483647;  // INT_MIN + 1
constexpr int kEventDead = -2147483646;     // INT_MIN + 2

struct RenderLaunch {
  SceneView scene;
  Camera cam;
  PathState st;
  float* frame;       // W*H*3 linear RGB, row 0 = bottom (SFrame layout)
  uint32_t npix;      // pixels of the frame
  uint32_t waveSpp;   // samples per wave (>= 1): path p is pixel p % npix, sample `sample` + p / npix
  uint32_t wavePaths; // npix * waveSpp
  uint32_t sample;    // first sample index of the wave
  uint32_t* sampleDev;  // nullable: device sample counter of a captured wave (read instead of `sample`)
  uint32_t spp;
  uint32_t maxDepth;
  uint32_t seed;
  uint32_t bounce;
  uint32_t dda;       // brick-grid DDA tracking (UseBrickGrid) instead of the global majorant
  uint32_t trackSteps;  // tracking steps a lane takes between refills (tuning, >= 1)
  uint32_t travVisits;  // BVH node steps a lane takes between refill checks of the surface kernels (tuning, >= 1)
  uint32_t travRefill;  // finished lanes of a warp that trigger a refill (tuning, 1..32)
  uint32_t trackBlocks; // persistent tracker blocks per SM (tuning; 0: every resident block)
  uint32_t mediaRounds; // queued rounds of a bounce's medium boundaries (tuning; 0: the default)
  uint32_t roundPaths;  // paths of a bounce from which they are used (0: kRoundPaths)
  uint32_t trackLimit;  // steps of one tracking loop after which the path ends (1..kMaxTrackingSteps)
  uint32_t sortRays;    // surface scenes: reorder each bounce's rays by a coherence key before k_extend
  unsigned long long* stats;  // nullable: [0] path segments traced, [1] shadow rays traced
  unsigned int* bound;        // paths and shadow rays ended by a loop bound (tracking steps, boundaries)
};

// Optional timing of one wave: events recorded after each stage; kind: -1
// start, 0 camera, 1 extend, 2 shade, 3 shadow, 4 accum, 5 finish; since: the
// event the stage's time counts from (the last on its stream).
struct WaveTimer {
  static constexpr int events(int depth) { return 6 + 6 * depth; }
  static constexpr int kMax = 6 + 6 * 64;
  int made = 0;  // events created
  cudaEvent_t ev[kMax];
  int kind[kMax], since[kMax];
  int n = 0;
};

// The second stream of a wave, on which a bounce's shadow rays are traced and
// accumulated while the next bounce is extended (the tail of a persistent
// kernel leaves most of the GPU free), and the events that fork and join it:
// 1,200 trees 24.1 -> 21.3 ms, moving spheres at 853x480 4.16 -> 3.95 ms.
struct WaveSide {
  cudaStream_t stream = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  uint32_t bounces = 64;  // of which the shadow rays go to it; the others' stay on the wave's own stream
};
// Bounces of a served job's captured wave that fork to it, in waves of at least so
// many paths: every fork costs in the graph's instantiation and launch.  Without
// forks / in the first 2 / 4 / 8 / 16 bounces, eight jobs on four slots, ms (one
// stream and the binary tree before: in brackets): 64x64, 4 samples, 50 bounces
// 9.2 / 8.4 / 10.2 / 13.0 / 18.5 (12.2; 46.6 with all bounces forked); 256x256, 1 sample
// 4.5 / 5.6 / 7.3 / 9.6 / 9.3 (5.5); 512x512, 4 samples, 50 bounces 26.9 / 26.1 / 25.2 /
// 24.1 / 24.5 (34.6); 1280x720, 32 samples 329 / 322 / 314 / 304 / 304 (428).
constexpr uint32_t kCapturedForks = 8, kCapturedForkPaths = 1u << 18;

// One wave (L.waveSpp consecutive samples of every pixel) on s and side, which
// rejoins s before the wave ends.  With L.sampleDev the last launch advances
// the device sample counter by L.waveSpp, so a captured wave replays as the
// next samples.
void launch_render_wave(const RenderLaunch& L, int nblocks, cudaStream_t s, const WaveSide& side,
                        WaveTimer* tm = nullptr);
// Occupancy queries of the persistent kernels, done before any capture.
void prepare_render_launches();

}  // namespace r2
