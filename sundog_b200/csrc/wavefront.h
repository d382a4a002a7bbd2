// Wavefront path tracer (wavefront.cu): pool buffers and the host driver.
#pragma once

#include <cuda_runtime.h>

#include <memory>

#include "render_session.h"
#include "sd_types.h"

namespace sdb {

struct LateVertex;
struct GuideTrail;

// A pool entry at a 16-byte boundary, moved with 128-bit loads and stores.
template <typename T>
struct __align__(16) PoolSlot {
  T v;
};

// Counters of one iteration (cleared on the device before it).
struct WfCounts {
  unsigned live;         // rays the iteration traces (its live list's length)
  unsigned shadow;       // shadow rays it queued
  unsigned late;         // vertices finished after their shadow ray
  unsigned traced;       // radiance rays shaded (live without tile padding)
  unsigned fetchRay, fetchShadow;  // rays taken by the dynamic fetches
  unsigned flame;        // rays that may meet a flame
  unsigned pad;
};
// Iterations launched between two looks at the live count. More waste empty
// launches where paths end early, fewer wait for the count more often: 4 / 8 /
// 16 at depth 16 take 0.67 / 0.61 / 0.58 ms (Cornell 96x96), 3.82 / 3.76 / 3.73
// (512x512) and 1.49 / 1.39 / 1.48 (instancing 333x217), at depth 64 0.79 /
// 0.78 / 0.84 (Cornell 96x96); with a look at every iteration, before groups,
// 1.08, 7.83, 2.04 and 1.22.
constexpr int kWfGroup = 8;

// Device view of the slot pool (one path per slot). A path's state is three
// 32-byte records in arrays of their own, so each stage moves whole sectors
// of what it needs and nothing else:
//   ray    o.xyz d.xyz, previous BSDF density, flags (specular | medDepth << 1);
//          of a camera ray the last two words are the random state
//   sum    L.xyz, sample slot, throughput.xyz, -
//   rest   previous vertex.xyz, -, random state, medium stack
// (the depth is the iteration; the random increment is the launch's).
struct WfPool {
  float4 *ray, *sum, *rest;   // two float4 each
  float4* hits;               // two: t, inst, prim | media << 30 | front << 31, u / v, normal.xyz
  float4* shadowRays;         // two: origin.xyz dir.xyz, tmax, flags
  float4* shadowTerms;        // the NEE term; for a late vertex its transmittance
  PoolSlot<LateVertex>* verts;  // late vertices (WfBuffers::lateCap slots have one)
  int* lists[2];              // live slot lists, ping-pong between iterations
  int *shadowList;
  int *lateList;              // late vertices; before shading, the rays that may meet a flame
  WfCounts* counts;           // kWfGroup + 1
  PoolSlot<GuideTrail>* trails;  // guided vertices awaiting their path's end (record passes)
  unsigned char* jobs;        // serving batches: the job slot of each slot's path
  unsigned long long* seen;   // host memory: the last report (wfReport)
};

// Host-owned pool storage, grown on demand.
struct WfBuffers {
  // One device allocation holds every per-slot array (carved at 256-byte
  // boundaries), so a pool costs one cudaMalloc and one cudaFree.
  DevBuf slab, counts;
  WfPool pool = {};
  DevBuf trails;  // allocated by the first training-record pass
  DevBuf verts;   // late vertices, where the slab was made without them
  // Pinned words, from a process-wide free list: counters read back, WfPool::seen.
  unsigned *hostCount = nullptr, *hostSeen = nullptr;
  cudaEvent_t ev[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};  // stage timing
  cudaStream_t side = nullptr;  // the shadow stage's, beside the next trace
  cudaEvent_t shaded = nullptr, shadowDone = nullptr;
  int cap = 0;
  int lateCap = 0;   // slots with room for a late vertex, in the slab or in verts
  int trailCap = 0;
  int gridStart = 0, gridTrace = 0, gridShade = 0, gridShadow = 0, gridLate = 0,
      gridFlame = 0;
  WfBuffers() = default;
  WfBuffers(const WfBuffers&) = delete;
  WfBuffers& operator=(const WfBuffers&) = delete;
  ~WfBuffers();
  // Room for `slots` paths (fewer when device memory is short), and with
  // withLate for their late vertices: in the slab where it is made now.
  void ensure(int slots, bool withLate);
  // Room for the late vertices of `slots` of the pool's paths (fewer when
  // device memory is short; `keep` bytes of it are left free).
  void ensureLate(int slots, size_t keep = 0);
  void ensureTrails();  // one GuideTrail per slot

 private:
  void grow(int slots, bool withLate);
};

// Whether paths of the launch may have late vertices: those whose next draws
// depend on their shadow ray (flames along it draw a random number) or whose
// training record needs its radiance.
bool wfHasLate(const SdLaunch& lp, int guide);

// Device bytes per pool slot, and per late vertex.
size_t wfSlotBytes();
size_t wfLateBytes();
// A pool for the current device: the idle one kept from an earlier session,
// or a new empty one. wfRelease keeps a finished session's pool for reuse.
std::unique_ptr<WfBuffers> wfAcquire();
void wfRelease(std::unique_ptr<WfBuffers> b);
// Frees the idle pools of every device.
void wfReleaseIdle();
// Whether finished sessions keep their device buffers for the next one
// (sundog_set_device_memory_cache; render.cpp).
bool keepDeviceMemory();
// Renders lp.numPaths camera paths (counters cleared by the caller) into
// lp.sampleL; returns the number of kernels launched. Synchronises st every
// kWfGroup iterations to read the live-path count, where paths may be longer.
// guide: 0, or a combination of
// kGuideSample (draw directions by MIS with the learned guide of lp) and
// kGuideRecord (keep each path's guided vertices in its slot's trail and turn
// them into training records when the path ends).
// times: when non-null, per-stage event times and ray counts are added to it.
int wfRender(const SdLaunch& lp, WfBuffers& b, cudaStream_t st, int guide = 0,
             WfStageTimes* times = nullptr);

// Serving batches (serve.h): the engine's whole job table (kMaxServeJobs
// launch blocks, host memory), and one batch of tile-passes rendered through
// the pool into batch.sampleL at each path's id (the caller folds them).
// Returns the kernels launched.
// jobs: the same table, for what its scenes need (the shadow-ray kernel, as a
// render picks it by its own scene's instance count; late vertices).
struct ServeBatch;
cudaError_t wfSetJobs(const SdLaunch* table, cudaStream_t st);
int wfRenderBatch(const ServeBatch& batch, WfBuffers& b, cudaStream_t st, const SdLaunch* jobs);

// Scenes with at least this many instances trace their shadow rays with
// dynamic fetch (wfShadowFetch), smaller ones one ray per thread (wfShadow).
#ifndef SDB_SHADOW_FETCH_INSTANCES
#define SDB_SHADOW_FETCH_INSTANCES 64
#endif
constexpr int kShadowFetchInstances = SDB_SHADOW_FETCH_INSTANCES;

}  // namespace sdb
