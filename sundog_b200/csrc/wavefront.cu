// Wavefront path tracer: the plain path kernel's per-path computation split
// into stages over a pool of path slots held in global memory.
//
//   wfStart        a camera ray in every slot
//   per iteration (path depth), over the slots in the live list:
//   wfTraceFetch   trace the radiance ray (traversal only)
//   wfFlameScan, wfFlame  (scenes with flames) march the rays that may meet one
//   wfShade        media, escape, shading, emission, the NEE light draw, the
//                  BSDF sample and roulette; queues the slot's shadow ray
//                  with the radiance it would add
//   wfShadow       trace the queued shadow rays (transparent shadows) and
//                  add that radiance
//   wfLate         the end of the few vertices that must know their shadow
//                  ray's result before they go on
//
// All paths of a pool are at the same depth, so the iterations of a pool are
// known to end with the deepest path and are launched in groups without a
// look at the live count. Each stage's code is small next to the
// megakernel's and keeps its state in registers instead of a 1 KB spilled
// frame; the price is the path state's round trip through global memory
// between stages (about 200 bytes per path segment).
//
// The stages call the megakernel's own per-path functions in the same order
// with the same random draws, so every sample is ptPersistent's up to FP32
// rounding (Rounding, sd_bsdf.cuh: a path may part from the megakernel's in
// its last bits; test_gpu_entry_points.py), and the film fold is the same.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <thread>
#include <vector>

#include "pt_path.cuh"
#include "serve.h"
#include "wavefront.h"

namespace sdb {

namespace cg = cooperative_groups;

__constant__ SdLaunch c_wlp;
__constant__ WfPool c_pool;

// Serving batches (GUIDE & kWfServe): tile-passes of many jobs in one pool.
// Each slot's path reads its job's launch block from this table (pool.jobs
// holds the job slot); path ids map to tile-passes as in ptServe (serve.cu),
// and finished samples go to the batch's sample buffer at their path id.
constexpr int kWfServe = 4;
__constant__ SdLaunch c_wjobs[kMaxServeJobs];
__constant__ ServeBatch c_wbatch;

// Launch block of the path in `slot`.
template <int GUIDE>
__device__ __forceinline__ const SdLaunch& slotLaunch(int slot) {
  if (GUIDE & kWfServe) return c_wjobs[c_pool.jobs[slot]];
  return c_wlp;
}

template <int GUIDE>
constexpr int kRound = (GUIDE & kWfServe) ? kRoundServe : kRoundStage;  // sd_bsdf.cuh

#ifndef SDB_WF_TRACE_BLOCKS
#define SDB_WF_TRACE_BLOCKS 8
#endif
// Resident blocks per SM the stage kernels are compiled for: traversal 8 of
// 128 threads (64 registers), the flame march and late vertices 5 (up to 96),
// shading 2 of 384 (80 registers, 228 bytes of spill stores and 304 of loads;
// 320 threads at 102 registers: instancing 1080p 90.6 against 89.1 ms).
#ifndef SDB_WF_LATE_BLOCKS
#define SDB_WF_LATE_BLOCKS 5
#endif
#ifndef SDB_WF_FLAME_BLOCKS
#define SDB_WF_FLAME_BLOCKS 5
#endif
#ifndef SDB_WF_SHADE_BLOCKS
#define SDB_WF_SHADE_BLOCKS 2
#endif

// A 32-byte record in one 256-bit load or store.
struct Rec {
  float4 a, b;
};
__device__ __forceinline__ Rec ldRec(const float4* p, int slot) {
  Rec r;
  asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y),
                 "=f"(r.b.z), "=f"(r.b.w)
               : "l"(p + 2 * (size_t)slot)
               : "memory");
  return r;
}
__device__ __forceinline__ void stRec(float4* p, int slot, float4 a, float4 b) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p + 2 * (size_t)slot),
               "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}
__device__ __forceinline__ float bitsF(unsigned v) { return __uint_as_float(v); }
__device__ __forceinline__ unsigned bitsU(float v) { return __float_as_uint(v); }

// Slot index for an append to a list by the calling lanes together.
__device__ __forceinline__ unsigned appendSlot(unsigned* count) {
  cg::coalesced_group g = cg::coalesced_threads();
  unsigned base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(count, g.size());
  return g.shfl(base, 0) + g.thread_rank();
}

// Serving: path id -> its tile-pass's pixel and sample (false for block
// padding), as serveStart in serve.cu.
__device__ __forceinline__ bool servePixel(unsigned long long id, int& job, int& px, int& py,
                                           int& sample) {
  const ServeBatch& b = c_wbatch;
  int lo = 0, hi = b.numItems - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (b.items[mid].pathBegin <= id) lo = mid;
    else hi = mid - 1;
  }
  const ServeItem& it = b.items[lo];
  int rem, sLocal;
  splitPathId(id - it.pathBegin, it.sampleCount, rem, sLocal);
  int blk = rem >> 6, within = rem & 63;
  int lx = (blk % it.bw) * 8 + tileX(within), ly = (blk / it.bw) * 8 + tileY(within);
  if (lx >= it.w || ly >= it.h) return false;
  job = it.job;
  px = it.x0 + lx;
  py = it.y0 + ly;
  sample = it.sampleBegin + sLocal;
  return true;
}

// What a late vertex keeps beyond its path and its queued shadow ray (which
// holds so, wi and tmaxS): the rest of Vertex.
struct LateVertex {
  float3 x, ns, albedo, Li;
  float etaExt, etaRel, pdf, cosS;
  int matId, lightK;
  bool front, delta;
};

// Hit record markers (in place of the instance).
constexpr int kMiss = -1;
constexpr int kNoPath = -2;  // a slot of tile padding

// Camera rays into the first n slots: slot i takes path base + i. Only the
// ray and the random state are stored (32 bytes); the rest of a fresh path
// is constant and the first shading stage fills it in.
template <int GUIDE>
__global__ void __launch_bounds__(kRenderBlock) wfStart(unsigned long long base, unsigned n) {
  const WfPool& pool = c_pool;
  if (blockIdx.x == 0 && threadIdx.x == 0) pool.counts[0].live = n;
  for (unsigned slot = blockIdx.x * blockDim.x + threadIdx.x; slot < n;
       slot += gridDim.x * blockDim.x) {
    Path p;
    bool ok;
    if (GUIDE & kWfServe) {
      int job = 0, px, py, s;
      ok = servePixel(base + slot, job, px, py, s);
      pool.jobs[slot] = (unsigned char)job;
      if (ok) startPathAt(c_wjobs[job], px, py, s, p);
    } else {
      ok = startPath(c_wlp, base + slot, p);
    }
    if (!ok) {  // tile padding (isPadding)
      p.o = p.d = v3(0.0f);
      p.rng.state = 0;
    }
    stRec(pool.ray, slot, make_float4(p.o.x, p.o.y, p.o.z, p.d.x),
          make_float4(p.d.y, p.d.z, bitsF((unsigned)p.rng.state),
                      bitsF((unsigned)(p.rng.state >> 32))));
  }
}

// Whether a camera record is tile padding: no direction and no random state.
// The state tells it from a camera ray whose direction vanished (a focus
// distance whose square overflows), which is traced like any other.
__device__ __forceinline__ bool isPadding(const Rec& r) {
  return r.a.w == 0.0f && r.b.x == 0.0f && r.b.y == 0.0f && (bitsU(r.b.z) | bitsU(r.b.w)) == 0u;
}

// Lanes of each warp that take work from a list of n items: all of them when
// the list fills the grid's lanes, else as few as spread it over every warp.
// A short list is bound by the longest walk among the lanes that share a
// warp, not by issue slots, so fewer lanes per warp end it sooner.
__device__ __forceinline__ unsigned spreadLanes(unsigned n) {
  const unsigned warps = gridDim.x * blockDim.x >> 5;
  const unsigned per = max(1u, min(32u, (n + warps - 1) / warps));
  return per == 32u ? 0xFFFFFFFFu : (1u << per) - 1u;
}

// Slot of ray i of the live list: the identity for the camera rays.
template <bool CAM>
__device__ __forceinline__ int liveSlot(int it, unsigned i) {
  return CAM ? (int)i : c_pool.lists[it & 1][i];
}

// Stores a closest-hit candidate straight into the slot's hit record (one
// 32-byte store), so the trace loop keeps no hit fields in registers: each
// closer hit overwrites the record, and a ray whose tmax was never lowered
// stores the miss marker when it ends.
__device__ __forceinline__ void putHit(float4* hits, int slot, float t, int inst, int prim, float u,
                                       float v, float3 nq, bool front) {
  stRec(hits, slot,
        make_float4(t, __int_as_float(inst),
                    bitsF((unsigned)prim | (front ? 0x80000000u : 0u)), u),
        make_float4(v, nq.x, nq.y, nq.z));
}
__device__ __forceinline__ void putMiss(float4* hits, int slot) {
  hits[2 * (size_t)slot] = make_float4(0.0f, __int_as_float(kMiss), 0.0f, 0.0f);
}
__device__ __forceinline__ void putNoPath(float4* hits, int slot) {
  hits[2 * (size_t)slot] = make_float4(0.0f, __int_as_float(kNoPath), 0.0f, 0.0f);
}

// A lane's next action.
constexpr int kAtNode = 0, kAtTriangle = 1, kAtInstance = 2, kNoRay = 3;
#if !SDB_WIDE_BVH
__device__ __forceinline__ int travKind(const BinTrav& t) {
  return t.cur >= 0 ? kAtNode : (t.inBlas ? kAtTriangle : kAtInstance);
}
#endif
// A round of the walk takes waiting instances if at least SDB_WF_INST_MIN
// lanes have one (any, once the list is used up), then triangles one at a time
// while at least SDB_WF_TRI_MIN lanes hold one, then node visits while at least
// SDB_WF_NODE_MIN lanes are at one. Instancing 1080p, ms: every lane's own next
// step, then descents (before) 96.0; 6 / 4 / 4 92.7; instances at 1 93.4; nodes
// at 2 / 7 / 10 95.3 / 93.0 / 94.2; triangles at 1 / 8 95.1 / 94.4; always the
// action most lanes wait for 98.6 (three small groups take turns).
#ifndef SDB_WF_NODE_MIN
#define SDB_WF_NODE_MIN 4
#endif
#ifndef SDB_WF_TRI_MIN
#define SDB_WF_TRI_MIN 4
#endif
#ifndef SDB_WF_INST_MIN
#define SDB_WF_INST_MIN 6
#endif
// Idle lanes a warp gathers before it fetches new rays (on the instancing
// frame with the one-action loop: 894 Mrays/s at 24, 869 with a grid-stride
// loop, 752 when every idle lane fetches at once: fresh rays at the TLAS
// root diverge from the warp's deep BLAS walks; with the 4-wide walk and
// descent runs, instancing 1080p / Cornell 256x256: 1,717 / 2,798 at 20, 1,706 / 2,801 at
// 24, 1,678 / 2,799 at 28).
#ifndef SDB_WF_FETCH_IDLE
#define SDB_WF_FETCH_IDLE 20
#endif

// Radiance rays with dynamic ray fetch (Aila and Laine, "Understanding the
// Efficiency of Ray Traversal on GPUs", 2009): the traversal loop runs per
// warp, and a lane whose ray is done writes its hit and, once
// SDB_WF_FETCH_IDLE lanes of the warp are idle, takes the next ray of the
// live list (one warp-aggregated atomicAdd on fetchRay), so a warp no longer
// waits for its longest ray. Each ray visits the nodes of traverse<false>
// (sd_trace.cuh) in the same order with the same tests: the same closest
// accepted hit. (Shadow rays take the same form in scenes of many instances,
// wfShadowFetch.) SERVE: a serving batch, each lane tracing in its own job's
// scene.
#if SDB_WIDE_BVH
// The same stage over the compressed 8-wide BVH (CwNode, sd_trace.cuh): each
// loop iteration a lane either tests one primitive of its current leaf group
// (a triangle, or a TLAS instance: quadric roots or entry into its BLAS),
// tests the 8 child boxes of the nearest remaining child node, or pops a
// group. The visit order and tests are those of traverse<false> in the
// 8-wide build: the same closest accepted hit.
template <bool SERVE, bool CAM>
__global__ void __launch_bounds__(kRenderBlock, SDB_WF_TRACE_BLOCKS) wfTraceFetch(int it, bool) {
  const WfPool& pool = c_pool;
  const unsigned n = pool.counts[it].live;
  const unsigned full = 0xFFFFFFFFu;
  const unsigned ltMask = (1u << (threadIdx.x & 31)) - 1u;
  int job = 0;  // SERVE: the lane's job slot
  const float tmin = 0.0f;
  int slot = -1;
  bool exhausted = false;  // warp-uniform
  float3 O = v3(0.0f), D = v3(0.0f);
  RayCtx ray;
  rayInit(ray, O, v3(1.0f), false);
  float tmax = 0.0f;
  TraceHit hit = {};
  bool found = false, inBlas = false;
  int curInst = -1, sp = 0;
  uint32_t gBase = 0, gHits = 0, gImask = 0, tBase = 0, tBits = 0;
  uint2 stack[kCwStack];
  while (true) {
    const unsigned idle = __ballot_sync(full, slot < 0);
    if (!exhausted && (idle == full || __popc(idle) >= SDB_WF_FETCH_IDLE)) {
      const int leader = __ffs(idle) - 1;
      unsigned base = 0;
      if ((int)(threadIdx.x & 31) == leader) base = atomicAdd(&pool.counts[it].fetchRay, (unsigned)__popc(idle));
      base = __shfl_sync(full, base, leader);
      if (base + __popc(idle) >= n) exhausted = true;
      if (slot < 0) {
        unsigned i = base + __popc(idle & ltMask);
        if (i < n) {
          slot = liveSlot<CAM>(it, i);
          if (SERVE) job = pool.jobs[slot];
          const SdLaunch& jl = SERVE ? c_wjobs[job] : c_wlp;
          const Rec r = ldRec(pool.ray, slot);
          O = v3(r.a.x, r.a.y, r.a.z);
          D = v3(r.a.w, r.b.x, r.b.y);
          if (CAM && isPadding(r)) {
            putNoPath(pool.hits, slot);
            slot = -1;
          }
          rayInit(ray, O, D, false);
          tmax = 1e16f;
          found = false;
          inBlas = false;
          curInst = -1;
          sp = 0;
          gBase = (uint32_t)jl.tlasRoot;
          gHits = jl.numInstances > 0 ? 1u << (0u ^ ray.rayOct) : 0u;
          gImask = 1u;
          tBits = 0;
        }
      }
    }
    if (__ballot_sync(full, slot >= 0) == 0) {
      if (exhausted) break;
      continue;
    }
    if (slot < 0) continue;
    const SdLaunch& lp = SERVE ? c_wjobs[job] : c_wlp;
    if (tBits) {
      const int j = __ffs(tBits) - 1;
      tBits &= tBits - 1u;
      const int prim = (int)tBase + j;
      if (!inBlas) {
        const SdInstance& inst = lp.inst[prim];
        float3 o2 = xfPoint(inst.w2o, O), d2 = xfVec(inst.w2o, D);
        if (inst.kind == GK_MESH) {
          // Suspend this level (the scene build keeps TLAS + BLAS depth
          // within the stack) and walk the BLAS in object space.
          if (sp + 3 > kCwStack) continue;
          if (gHits) stack[sp++] = make_uint2(gBase, gHits | (gImask << 8));
          if (tBits) stack[sp++] = make_uint2(tBase, tBits | kGroupPrims);
          stack[sp++] = make_uint2(0xFFFFFFFFu, kGroupMarker);
          inBlas = true;
          curInst = prim;
          rayInit(ray, o2, d2, true);
          gBase = (uint32_t)lp.meshes[inst.mesh].root;
          gHits = 1u << (0u ^ ray.rayOct);
          gImask = 1u;
          tBits = 0;
          continue;
        }
        QHits qh = hitQuadric(inst.kind, o2, d2, tmin, tmax);
        for (int k = 0; k < qh.n; k++) {
          const QHit& q = qh.h[k];
          if (q.t >= tmax) continue;
          bool front = dot(q.n, d2) < 0.0f;
          if ((inst.flags & kInstMasked) && !faceAccepts(lp, inst, front, q.u, q.v)) continue;
          tmax = q.t;
          found = true;
          hit.t = q.t;
          hit.inst = prim;
          hit.prim = 0;
          hit.u = q.u;
          hit.v = q.v;
          hit.nq = q.n;
          hit.front = front;
        }
        continue;
      }
      // Triangle of the current BLAS, in object space.
      const float4* tp = lp.tris + 3 * (size_t)prim;
      float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
      float t, b1, b2;
      float3 p0 = v3(a.x, a.y, a.z), p1 = v3(b.x, b.y, b.z), p2 = v3(c.x, c.y, c.z);
      if (!wtHit(ray.wt, ray.o, p0, p1, p2, tmin, tmax, t, b1, b2)) continue;
      const int tri = __float_as_int(a.w);
      const SdInstance& inst = lp.inst[curInst];
      bool front;
      if (!(inst.flags & (kInstMasked | kInstTransmissive))) {
        front = dot(cross(p1 - p0, p2 - p0), ray.d) < 0.0f;
      } else {
        ShadePt spt = triShade(lp, inst, tri, b1, b2, D);
        if ((inst.flags & kInstMasked) && !faceAccepts(lp, inst, spt.front, spt.u, spt.v)) continue;
        front = spt.front;
      }
      tmax = t;
      found = true;
      hit.t = t;
      hit.inst = curInst;
      hit.prim = tri;
      hit.u = b1;
      hit.v = b2;
      hit.front = front;
      continue;
    }
    if (gHits) {
      const int b = __ffs(gHits) - 1;
      gHits &= gHits - 1u;
      const uint32_t cs = (uint32_t)b ^ ray.rayOct;
      const int child = (int)(gBase + __popc(gImask & ((1u << cs) - 1u)));
      if (gHits && sp < kCwStack) stack[sp++] = make_uint2(gBase, gHits | (gImask << 8));
      CwHits h = cwIntersect(lp.cw, child, ray.o, ray.id, ray.rayOct, tmin, tmax);
      gBase = h.childBase;
      gHits = h.hits;
      gImask = h.imask;
      tBase = h.primBase;
      tBits = h.leafBits;
      continue;
    }
    if (sp == 0) {  // ray done
      if (found) putHit(pool.hits, slot, hit.t, hit.inst, hit.prim, hit.u, hit.v, hit.nq, hit.front);
      else putMiss(pool.hits, slot);
      slot = -1;
      continue;
    }
    const uint2 e = stack[--sp];
    if (e.y & kGroupMarker) {
      inBlas = false;
      rayInit(ray, O, D, false);
    } else if (e.y & kGroupPrims) {
      tBase = e.x;
      tBits = e.y & 0xFFFFFFu;
    } else {
      gBase = e.x;
      gHits = e.y & 0xFFu;
      gImask = (e.y >> 8) & 0xFFu;
    }
  }
}
#else
// Sink of the trace stage's walks (binTravStep, sd_trace.cuh): closer hits go
// straight to the slot's hit record and the world ray is re-read from the
// slot when a walk leaves a BLAS, so neither stays in registers.
struct PoolSink {
  const WfPool& pool;
  int slot;
  __device__ __forceinline__ void world(float3& ro, float3& rd) const {
    const Rec r = ldRec(pool.ray, slot);
    ro = v3(r.a.x, r.a.y, r.a.z);
    rd = v3(r.a.w, r.b.x, r.b.y);
  }
  __device__ __forceinline__ float3 worldDir() const {
    const Rec r = ldRec(pool.ray, slot);
    return v3(r.a.w, r.b.x, r.b.y);
  }
  __device__ __forceinline__ void hit(float t, int inst, int prim, float u, float v, float3 nq,
                                      bool front) const {
    putHit(pool.hits, slot, t, inst, prim, u, v, nq, front);
  }
};

constexpr float kRayMax = 1e16f;  // tmax of a radiance ray: any hit lowers it

template <bool SERVE, bool CAM>
__global__ void __launch_bounds__(kRenderBlock, SDB_WF_TRACE_BLOCKS) wfTraceFetch(int it, bool spread) {
  const WfPool& pool = c_pool;
  const unsigned n = pool.counts[it].live;
  const unsigned full = 0xFFFFFFFFu;
  const unsigned ltMask = (1u << (threadIdx.x & 31)) - 1u;
  const unsigned lanes = spread ? spreadLanes(n) : full;
  int job = 0;  // SERVE: the lane's job slot
  int slot = -1;
  bool exhausted = false;  // warp-uniform
  BinTrav t;
  TravStack stack;
  float trUnused = 1.0f;
  float3 tauUnused = v3(0.0f);
  while (true) {
    const unsigned idle = __ballot_sync(full, slot < 0) & lanes;
    if (!exhausted && (idle == lanes || __popc(idle) >= SDB_WF_FETCH_IDLE)) {
      const int leader = __ffs(idle) - 1;
      unsigned base = 0;
      if ((int)(threadIdx.x & 31) == leader)
        base = atomicAdd(&pool.counts[it].fetchRay, (unsigned)__popc(idle));
      base = __shfl_sync(full, base, leader);
      if (base + __popc(idle) >= n) exhausted = true;
      if (idle >> (threadIdx.x & 31) & 1u) {
        unsigned i = base + __popc(idle & ltMask);
        if (i < n) {
          slot = liveSlot<CAM>(it, i);
          if (SERVE) job = pool.jobs[slot];
          const SdLaunch& jl = SERVE ? c_wjobs[job] : c_wlp;
          const Rec r = ldRec(pool.ray, slot);
          const float3 o = v3(r.a.x, r.a.y, r.a.z), d = v3(r.a.w, r.b.x, r.b.y);
          binTravStart(t, jl, o, d, kRayMax);
          if (CAM && isPadding(r)) {
            putNoPath(pool.hits, slot);
            slot = -1;
          }
        }
      }
    }
    if (__ballot_sync(full, slot >= 0) == 0) {
      if (exhausted) break;
      continue;
    }
    const SdLaunch& lp = SERVE ? c_wjobs[job] : c_wlp;
    PoolSink sink{pool, slot};
    int r = kTravMore;
    // Leaves first (instances, then triangles one at a time while enough
    // lanes hold one), then node visits in a row while enough lanes are at
    // one; lanes that reach a leaf meanwhile wait for the next round.
    int kind = slot < 0 ? kNoRay : travKind(t);
    {
      const int insts = __popc(__ballot_sync(full, kind == kAtInstance));
      if (insts >= (exhausted ? 1 : SDB_WF_INST_MIN) || __ballot_sync(full, kind == kAtNode || kind == kAtTriangle) == 0) {
        if (kind == kAtInstance) {
          r = t.cur == kPop ? binTravPop(t, stack, sink)
                            : binTravInstance<false, false, true>(t, stack, lp, sink, trUnused, tauUnused, nullptr);
          kind = r == kTravMore ? travKind(t) : kNoRay;
        }
      }
    }
    for (int tris = __popc(__ballot_sync(full, kind == kAtTriangle)); tris > 0;) {
      if (kind == kAtTriangle) {
        r = binTravTriangle<false, false>(t, stack, lp, sink, trUnused, tauUnused, nullptr);
        kind = r == kTravLeaf ? kAtTriangle : (r == kTravMore ? travKind(t) : kNoRay);
      }
      tris = __popc(__ballot_sync(full, kind == kAtTriangle));
      if (tris < SDB_WF_TRI_MIN) break;
    }
    for (int nodes = __popc(__ballot_sync(full, kind == kAtNode)); nodes > 0;) {
      if (kind == kAtNode) {
        r = binTravNode<false, false, false, true>(t, stack, lp, sink, nullptr);
        kind = r == kTravMore ? travKind(t) : kNoRay;
      }
      nodes = __popc(__ballot_sync(full, kind == kAtNode));
      if (nodes < SDB_WF_NODE_MIN) break;
    }
    if (slot >= 0 && r == kTravDone) {
      if (t.tmax == kRayMax) putMiss(pool.hits, slot);
      slot = -1;
    }
  }
}
#endif

// ---- shading ---------------------------------------------------------------------

// Rays of a tile, shaded together by one block: sorted by what their hit
// needs (kClass*), so a warp runs one material's code instead of stepping
// through all of them with a few lanes each.
#ifndef SDB_SHADE_THREADS
#define SDB_SHADE_THREADS 384
#endif
#ifndef SDB_SHADE_TILE
#define SDB_SHADE_TILE 1536
#endif
constexpr int kShadeBlock = SDB_SHADE_THREADS;
constexpr int kTileMax = SDB_SHADE_TILE;
constexpr int kClasses = 8;       // miss, then 1 + MatKind, then tile padding
constexpr int kClassNone = 7;
constexpr int kWarps = kShadeBlock / 32;

// Hides a value from the optimiser as a trip through memory does: the two
// halves of a vertex round the same whether one kernel computes both or the
// second runs later from stored state (no product of the first half fuses
// into a sum of the second).
__device__ __forceinline__ void opaque(float& x) { asm volatile("" : "+f"(x)); }
__device__ __forceinline__ void opaque(int& x) { asm volatile("" : "+r"(x)); }
__device__ __forceinline__ void opaque(float3& a) {
  opaque(a.x);
  opaque(a.y);
  opaque(a.z);
}

__device__ __forceinline__ unsigned long long rngInc(const SdLaunch& lp) {
  return ((unsigned long long)lp.seed << 1) | 1ull;  // Pcg::seeded's stream
}

// The finished path's sample; record passes also turn its trail of guided
// vertices into training records.
template <int GUIDE>
__device__ __forceinline__ void finishPath(float3 radiance, int sample, int slot) {
  float3 L = sanitize3(radiance);
  if (GUIDE & kGuideRecord) guideFlush(c_wlp, c_pool.trails[slot].v, L);
  float4* sampleL = (GUIDE & kWfServe) ? c_wbatch.sampleL : c_wlp.sampleL;
  sampleL[sample] = make_float4(L.x, L.y, L.z, 1.0f);
}

__device__ __forceinline__ void storeSum(const WfPool& pool, const Path& p, int slot) {
  stRec(pool.sum, slot, make_float4(p.L.x, p.L.y, p.L.z, __int_as_float(p.slot)),
        make_float4(p.beta.x, p.beta.y, p.beta.z, 0.0f));
}
__device__ __forceinline__ void storePath(const WfPool& pool, const Path& p, int slot) {
  stRec(pool.ray, slot, make_float4(p.o.x, p.o.y, p.o.z, p.d.x),
        make_float4(p.d.y, p.d.z, p.prevPdf,
                    bitsF((p.specular ? 1u : 0u) | ((unsigned)p.medDepth << 1))));
  storeSum(pool, p, slot);
  stRec(pool.rest, slot, make_float4(p.prevX.x, p.prevX.y, p.prevX.z, 0.0f),
        make_float4(bitsF((unsigned)p.rng.state), bitsF((unsigned)(p.rng.state >> 32)),
                    bitsF((unsigned)p.med), bitsF((unsigned)(p.med >> 32))));
}
__device__ __forceinline__ unsigned long long join64(float lo, float hi) {
  return (unsigned long long)bitsU(lo) | ((unsigned long long)bitsU(hi) << 32);
}
__device__ __forceinline__ void loadSum(const WfPool& pool, int slot, Path& p) {
  const Rec s = ldRec(pool.sum, slot);
  p.L = v3(s.a.x, s.a.y, s.a.z);
  p.slot = __float_as_int(s.a.w);
  p.beta = v3(s.b.x, s.b.y, s.b.z);
}
// The path in `slot` at `depth` (not a camera ray).
__device__ __forceinline__ void loadPath(const WfPool& pool, const SdLaunch& lp, int slot, int depth,
                                         Path& p) {
  const Rec r = ldRec(pool.ray, slot), q = ldRec(pool.rest, slot);
  loadSum(pool, slot, p);
  p.o = v3(r.a.x, r.a.y, r.a.z);
  p.d = v3(r.a.w, r.b.x, r.b.y);
  p.prevPdf = r.b.z;
  p.specular = (bitsU(r.b.w) & 1u) != 0;
  p.medDepth = (int)(bitsU(r.b.w) >> 1);
  p.prevX = v3(q.a.x, q.a.y, q.a.z);
  p.rng.state = join64(q.b.x, q.b.y);
  p.rng.inc = rngInc(lp);
  p.med = join64(q.b.z, q.b.w);
  p.depth = depth;
  opaque(p.depth);
}
// The camera path with id `id` in `slot`.
template <int GUIDE>
__device__ __forceinline__ void loadCamera(const WfPool& pool, const SdLaunch& lp, int slot,
                                           unsigned long long id, Path& p) {
  const Rec r = ldRec(pool.ray, slot);
  p.o = v3(r.a.x, r.a.y, r.a.z);
  p.d = v3(r.a.w, r.b.x, r.b.y);
  p.rng.state = join64(r.b.z, r.b.w);
  p.rng.inc = rngInc(lp);
  p.beta = v3(1.0f);
  p.L = v3(0.0f);
  p.prevX = p.o;
  p.prevPdf = 0.0f;
  p.specular = true;
  p.med = 0ull;
  p.medDepth = 0;
  p.depth = 0;
  if (GUIDE & kWfServe) {
    p.slot = (int)id;
  } else {
    int px, py, s;
    pathPixel(lp, id, px, py, s);
    p.slot = sampleSlot(lp, px, py, s);
  }
  opaque(p.beta);
  opaque(p.L);
  opaque(p.prevPdf);
  int specular = 1;
  opaque(specular);
  p.specular = specular != 0;
  opaque(p.depth);
}

constexpr unsigned kPrimMask = 0x3FFFFFFFu;  // hit record: the triangle
constexpr unsigned kMediaDone = 0x40000000u;  // its segment's media are in the path already

constexpr unsigned kShadowFinal = 1u;  // shadow ray flags: its path has ended
constexpr unsigned kShadowLate = 2u;   // its vertex is finished by wfLate

// One ray's shading. Returns what follows: bit 0 the path lives on, bit 1 it
// queued a shadow ray, bit 2 its vertex waits for that ray.
template <int GUIDE, bool CAM>
__device__ __forceinline__ unsigned shadeRay(const WfPool& pool, int slot, unsigned long long id,
                                             int depth) {
  const SdLaunch& lp = slotLaunch<GUIDE>(slot);
  Path p;
  if (CAM) loadCamera<GUIDE>(pool, lp, slot, id, p);
  else loadPath(pool, lp, slot, depth, p);
  if (CAM && (GUIDE & kGuideRecord)) pool.trails[slot].v.n = 0;
  const Rec hr = ldRec(pool.hits, slot);
  const bool mediaDone = (bitsU(hr.a.z) & kMediaDone) != 0;
  TraceHit h;
  h.t = hr.a.x;
  h.inst = __float_as_int(hr.a.y);
  h.prim = (int)(bitsU(hr.a.z) & kPrimMask);
  h.front = (bitsU(hr.a.z) >> 31) != 0;
  h.u = hr.a.w;
  h.v = hr.b.x;
  h.nq = v3(hr.b.y, hr.b.z, hr.b.w);
  const bool hit = h.inst >= 0;
  if (mediaDone) {
    if (CAM) loadSum(pool, slot, p);
  } else {
    absorbMedium(lp, p, hit, h.t);
    // No flame on the segment: nothing added (but a non-finite throughput
    // still shows, as it would with flames marched).
    if (lp.numFlames > 0) addClamped(lp, p, p.beta * 0.0f);
  }
  Vertex v;
  unsigned long long raysUnused = 0;
  if (!shadeSurface(lp, p, hit, h, raysUnused, v)) {
    finishPath<GUIDE>(p.L, p.slot, slot);
    return 0;
  }
  bool late = false;
  if (v.nee) {
    if (GUIDE & kGuideRecord) {
      late = true;
    } else if (lp.numFlames > 0 && lp.transparentShadows) {
      const int skip = v.lightK < lp.numLights ? lp.lights[v.lightK].flameId : -1;
      late = flamesMayMeet(lp.flames, lp.numFlames, v.so, v.wi, v.tmaxS, skip);
    }
  }
  if (v.nee)
    stRec(pool.shadowRays, slot, make_float4(v.so.x, v.so.y, v.so.z, v.wi.x),
          make_float4(v.wi.y, v.wi.z, v.tmaxS, bitsF(late ? kShadowLate : 0u)));
  if (late) {
    storePath(pool, p, slot);
    pool.verts[slot].v = {v.x,   v.ns,   v.albedo, v.Li,    v.etaExt, v.etaRel,
                          v.pdf, v.cosS, v.matId,  v.lightK, v.front,  v.delta};
    return 6;
  }
  int flags = (v.nee ? 1 : 0) | (v.delta ? 2 : 0) | (v.front ? 4 : 0);
  opaque(flags);
  v.nee = (flags & 1) != 0;
  v.delta = (flags & 2) != 0;
  v.front = (flags & 4) != 0;
  opaque(v.matId);
  opaque(v.x);
  opaque(v.ns);
  opaque(v.albedo);
  opaque(v.etaExt);
  opaque(v.etaRel);
  opaque(v.wi);
  opaque(v.Li);
  opaque(v.pdf);
  opaque(v.cosS);
  opaque(p.beta);
  opaque(p.L);
  const SdMaterial mat = lp.materials[v.matId];
  if (v.nee) {
    const float3 c = neeTerm(lp, p, mat, v);
    pool.shadowTerms[slot] = make_float4(c.x, c.y, c.z, 0.0f);
  }
  GuideTrail* trail = (GUIDE & kGuideRecord) ? &pool.trails[slot].v : nullptr;
  if (sampleNext<GUIDE, kRound<GUIDE>>(lp, p, mat, v, trail)) {
    storePath(pool, p, slot);
    return v.nee ? 3 : 1;
  }
  if (v.nee) {  // the shadow ray adds the last term and finishes the sample
    pool.sum[2 * (size_t)slot] = make_float4(p.L.x, p.L.y, p.L.z, __int_as_float(p.slot));
    reinterpret_cast<unsigned*>(pool.shadowRays + 2 * (size_t)slot)[7] = kShadowFinal;
    return 2;
  }
  finishPath<GUIDE>(p.L, p.slot, slot);
  return 0;
}

// Lists the traced rays whose segment may meet a flame.
template <int GUIDE, bool CAM>
__global__ void __launch_bounds__(kRenderBlock) wfFlameScan(int it) {
  const WfPool& pool = c_pool;
  const unsigned n = pool.counts[it].live;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int slot = liveSlot<CAM>(it, i);
    const float4 h = pool.hits[2 * (size_t)slot];
    const int inst = __float_as_int(h.y);
    if (inst == kNoPath) continue;
    const SdLaunch& lp = slotLaunch<GUIDE>(slot);
    if (lp.numFlames == 0) continue;
    const Rec r = ldRec(pool.ray, slot);
    if (flamesMayMeet(lp.flames, lp.numFlames, v3(r.a.x, r.a.y, r.a.z), v3(r.a.w, r.b.x, r.b.y),
                      inst >= 0 ? h.x : 1e16f, -1))
      pool.lateList[appendSlot(&pool.counts[it].flame)] = slot;
  }
}

// Their media: absorption and the flame march, ahead of the shading stage.
// In that stage a few lanes of a warp marched while the others waited; here
// every lane of a warp marches.
template <int GUIDE, bool CAM>
__global__ void __launch_bounds__(kRenderBlock, SDB_WF_FLAME_BLOCKS) wfFlame(
    int it, int depth, unsigned long long base) {
  const WfPool& pool = c_pool;
  const unsigned n = pool.counts[it].flame;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int slot = pool.lateList[i];
    const SdLaunch& lp = slotLaunch<GUIDE>(slot);
    Path p;
    if (CAM) loadCamera<GUIDE>(pool, lp, slot, base + slot, p);
    else loadPath(pool, lp, slot, depth, p);
    float4 h = pool.hits[2 * (size_t)slot];
    crossMedia(lp, p, __float_as_int(h.y) >= 0, h.x);
    storeSum(pool, p, slot);
    // The random state: in a camera ray's record, else in the rest.
    float2* rng = reinterpret_cast<float2*>((CAM ? pool.ray : pool.rest) + 2 * (size_t)slot) +
                  (CAM ? 3 : 2);
    *rng = make_float2(bitsF((unsigned)p.rng.state), bitsF((unsigned)(p.rng.state >> 32)));
    reinterpret_cast<unsigned*>(pool.hits + 2 * (size_t)slot)[2] = bitsU(h.z) | kMediaDone;
  }
}

// What the shading of a traced ray runs: 0 a miss, 1 + the kind of the hit
// face's material, kClassNone for tile padding.
template <int GUIDE>
__device__ __forceinline__ int hitClass(const WfPool& pool, int slot) {
  const float4 h = pool.hits[2 * (size_t)slot];
  const int inst = __float_as_int(h.y);
  if (inst < 0) return inst == kNoPath ? kClassNone : 0;
  const SdLaunch& lp = slotLaunch<GUIDE>(slot);
  const unsigned mats = lp.inst[inst].mats;
  const unsigned m = (bitsU(h.z) >> 31) ? (mats & 0xFFFFu) : (mats >> 16);
  return 1 + lp.materials[m].kind;
}

// Exclusive prefix sum of v over the calling warp; total gets the sum.
__device__ __forceinline__ unsigned warpPrefix(unsigned v, unsigned& total) {
  const int lane = threadIdx.x & 31;
  unsigned x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned y = __shfl_up_sync(0xFFFFFFFFu, x, off);
    if (lane >= off) x += y;
  }
  total = __shfl_sync(0xFFFFFFFFu, x, 31);
  return x - v;
}

// Shades the rays of the live list, a tile of up to kTileMax consecutive
// list entries per block at a time: the tile is sorted by class in shared
// memory and shaded in that order, and what lives on (and the shadow rays)
// joins the next lists in the tile's own order, so the pixel order of the
// camera rays is kept from bounce to bounce. Small lists take smaller tiles
// so that every block has one.
template <int GUIDE, bool CAM>
__global__ void __launch_bounds__(kShadeBlock, SDB_WF_SHADE_BLOCKS) wfShade(
    int it, int depth, unsigned long long base) {
  __shared__ int sSlot[kTileMax];
  __shared__ unsigned short sKey[kTileMax];    // class << 8 | rank
  __shared__ unsigned char sFlag[kTileMax];
  __shared__ unsigned short sOrder[kTileMax];
  constexpr int kGroups = kTileMax / 32;       // warps' worth of entries in a tile
  __shared__ unsigned short sCount[kClasses * kGroups];
  __shared__ unsigned sList[3][kGroups];
  __shared__ unsigned sBase[3];
  __shared__ unsigned sPart[kWarps];
  __shared__ unsigned sNext;
  const WfPool& pool = c_pool;
  WfCounts& cnt = pool.counts[it];
  const unsigned full = 0xFFFFFFFFu;
  const unsigned n = cnt.live;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned ltMask = (1u << lane) - 1u;
  const unsigned per = (n + gridDim.x * kShadeBlock - 1) / (gridDim.x * kShadeBlock);
  // Record passes keep the records of the paths that end first: small tiles
  // there, so those are not the misses of large ones.
  const unsigned most = (GUIDE & kGuideRecord) ? 1u : (unsigned)(kTileMax / kShadeBlock);
  const int K = (int)min(max(per, 1u), most);
  const unsigned T = (unsigned)K * kShadeBlock;
  for (unsigned t0 = blockIdx.x * T; t0 < n; t0 += gridDim.x * T) {
    // Classes, and each entry's rank among its warp's entries of the class.
    for (int k = tid; k < kClasses * kGroups; k += kShadeBlock) sCount[k] = 0;
    if (tid == 0) sNext = 0;
    __syncthreads();
    for (int k = 0; k < K; k++) {
      const int e = k * kShadeBlock + tid;
      const unsigned i = t0 + e;
      int slot = -1, cls = kClassNone;
      if (i < n) {
        slot = liveSlot<CAM>(it, i);
        cls = hitClass<GUIDE>(pool, slot);
      }
      const unsigned same = __match_any_sync(full, cls);
      const int rank = __popc(same & ltMask);
      if (rank == 0) sCount[cls * kGroups + (e >> 5)] = (unsigned short)__popc(same);
      sSlot[e] = slot;
      sKey[e] = (unsigned short)(cls << 8 | rank);
      sFlag[e] = 0;
    }
    __syncthreads();
    // Prefix over the counts, class by class (two entries per thread).
    static_assert(kClasses * kGroups <= 2 * kShadeBlock, "two counts per thread");
    {
      const bool in = 2 * tid < kClasses * kGroups;
      const unsigned c0 = in ? sCount[2 * tid] : 0u, c1 = in ? sCount[2 * tid + 1] : 0u;
      unsigned total;
      const unsigned ex = warpPrefix(c0 + c1, total);
      if (lane == 0) sPart[warp] = total;
      __syncthreads();
      unsigned before = 0;
      for (int w = 0; w < warp; w++) before += sPart[w];
      if (in) {
        sCount[2 * tid] = (unsigned short)(before + ex);
        sCount[2 * tid + 1] = (unsigned short)(before + ex + c0);
      }
    }
    __syncthreads();
    const int shaded = sCount[kClassNone * kGroups];  // entries that hold a path
    for (int k = 0; k < K; k++) {
      const int e = k * kShadeBlock + tid;
      const unsigned key = sKey[e];
      sOrder[sCount[(key >> 8) * kGroups + (e >> 5)] + (key & 0xFFu)] = (unsigned short)e;
    }
    __syncthreads();
    // Warps take the sorted rays 32 at a time: classes cost unevenly.
    while (true) {
      unsigned j = 0;
      if (lane == 0) j = atomicAdd(&sNext, 32u);
      j = __shfl_sync(full, j, 0);
      if (j >= (unsigned)shaded) break;
      if (j + lane < (unsigned)shaded) {
        const int e = sOrder[j + lane];
        sFlag[e] = (unsigned char)shadeRay<GUIDE, CAM>(pool, sSlot[e], base + t0 + e, depth);
      }
      __syncwarp();
    }
    __syncthreads();
    // The tile's contributions to the next lists, in its own order.
    for (int k = 0; k < K; k++) {
      const int e = k * kShadeBlock + tid;
      const unsigned f = sFlag[e];
      const unsigned live = __ballot_sync(full, f & 1u), shadow = __ballot_sync(full, f & 2u),
                     late = __ballot_sync(full, f & 4u);
      if (lane == 0) {
        sList[0][e >> 5] = __popc(live);
        sList[1][e >> 5] = __popc(shadow);
        sList[2][e >> 5] = __popc(late);
      }
    }
    __syncthreads();
    if (warp < 3) {
      // Two groups per lane.
      static_assert(kGroups <= 64, "groups of a tile");
      unsigned total;
      const bool in0 = 2 * lane < K * kWarps, in1 = 2 * lane + 1 < K * kWarps;
      const unsigned v0 = in0 ? sList[warp][2 * lane] : 0u, v1 = in1 ? sList[warp][2 * lane + 1] : 0u;
      const unsigned ex = warpPrefix(v0 + v1, total);
      if (in0) sList[warp][2 * lane] = ex;
      if (in1) sList[warp][2 * lane + 1] = ex + v0;
      if (lane == 0 && total) {
        unsigned* c = warp == 0 ? &pool.counts[it + 1].live : (warp == 1 ? &cnt.shadow : &cnt.late);
        sBase[warp] = atomicAdd(c, total);
      }
      if (warp == 1 && lane == 0) {
        unsigned long long* rays = (GUIDE & kWfServe) ? c_wbatch.rayCounter : c_wlp.rayCounter;
        atomicAdd(rays, (unsigned long long)shaded + total);
      }
    } else if (warp == 3 && lane == 0) {
      atomicAdd(&cnt.traced, (unsigned)shaded);
    }
    __syncthreads();
    for (int k = 0; k < K; k++) {
      const int e = k * kShadeBlock + tid;
      const unsigned f = sFlag[e];
      const unsigned live = __ballot_sync(full, f & 1u), shadow = __ballot_sync(full, f & 2u),
                     late = __ballot_sync(full, f & 4u);
      const int slot = sSlot[e];
      if (f & 1u) pool.lists[(it + 1) & 1][sBase[0] + sList[0][e >> 5] + __popc(live & ltMask)] = slot;
      if (f & 2u) pool.shadowList[sBase[1] + sList[1][e >> 5] + __popc(shadow & ltMask)] = slot;
      if (f & 4u) pool.lateList[sBase[2] + sList[2][e >> 5] + __popc(late & ltMask)] = slot;
    }
    __syncthreads();
  }
}

// ---- shadow rays --------------------------------------------------------------------

// A shadow ray's result: the transmittance to a late vertex, or its NEE term
// added to the path's radiance, which for an ended path is its sample.
template <int GUIDE>
__device__ __forceinline__ void finishShadow(const WfPool& pool, int slot, unsigned flags, float3 tr,
                                             int depth) {
  if (flags & kShadowLate) {
    pool.shadowTerms[slot] = make_float4(tr.x, tr.y, tr.z, 0.0f);
    return;
  }
  const bool lit = hmax(tr) > 0.0f;
  if (!lit && !(flags & kShadowFinal)) return;
  float4 s = pool.sum[2 * (size_t)slot];
  float3 L = v3(s.x, s.y, s.z);
  if (lit) {
    const float4 c = pool.shadowTerms[slot];
    float3 z = v3(__fmul_rn(c.x, tr.x), __fmul_rn(c.y, tr.y), __fmul_rn(c.z, tr.z));
    z = neeRadiance(z, v3(1.0f), depth >= 1, slotLaunch<GUIDE>(slot).clampVal);
    L = v3(__fadd_rn(L.x, z.x), __fadd_rn(L.y, z.y), __fadd_rn(L.z, z.z));
  }
  if (flags & kShadowFinal) finishPath<GUIDE & kWfServe>(L, __float_as_int(s.w), slot);
  else pool.sum[2 * (size_t)slot] = make_float4(L.x, L.y, L.z, s.w);
}

// Shadow rays, one per thread to the end of its walk (grid-stride over the
// shadow list).
template <int GUIDE>
__global__ void __launch_bounds__(kRenderBlock, SDB_WF_TRACE_BLOCKS) wfShadow(int it, int depth) {
  const WfPool& pool = c_pool;
  const unsigned n = pool.counts[it].shadow;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int slot = pool.shadowList[i];
    const SdLaunch& lp = slotLaunch<GUIDE>(slot);
    const Rec r = ldRec(pool.shadowRays, slot);
    const float3 so = v3(r.a.x, r.a.y, r.a.z), wi = v3(r.a.w, r.b.x, r.b.y);
    const float3 tr = shadowTransmittance<false>(lp, so, wi, r.b.z, nullptr);
    finishShadow<GUIDE>(pool, slot, bitsU(r.b.w), tr, depth);
  }
}

#if !SDB_WIDE_BVH
// Sink of the shadow stage's walks: the world ray is the slot's queued
// shadow ray, re-read when a walk leaves a BLAS.
struct ShadowSink {
  const WfPool& pool;
  int slot;
  __device__ __forceinline__ void world(float3& ro, float3& rd) const {
    const Rec r = ldRec(pool.shadowRays, slot);
    ro = v3(r.a.x, r.a.y, r.a.z);
    rd = v3(r.a.w, r.b.x, r.b.y);
  }
  __device__ __forceinline__ float3 worldDir() const {
    const Rec r = ldRec(pool.shadowRays, slot);
    return v3(r.a.w, r.b.x, r.b.y);
  }
  __device__ __forceinline__ void hit(float, int, int, float, float, float3, bool) const {}
};

// Shadow rays with the trace stage's dynamic fetch and
// node-descent runs: the walk and transmittance of shadowTransmittance, many
// rays interleaved per warp. Faster than wfShadow where walks are long and
// uneven (1024 instances, 1080p: 29.3 -> 24.5 ms per frame), slower on small
// scenes (Cornell: 2,730 -> 2,672 Mrays/s; volumes 1440p: 113.7 -> 122.2
// ms), so renders choose by instance count (kShadowFetchInstances).
template <int GUIDE>
__global__ void __launch_bounds__(kRenderBlock, SDB_WF_TRACE_BLOCKS) wfShadowFetch(int it, int depth) {
  const WfPool& pool = c_pool;
  const unsigned n = pool.counts[it].shadow;
  const unsigned full = 0xFFFFFFFFu;
  const unsigned ltMask = (1u << (threadIdx.x & 31)) - 1u;
  const unsigned lanes = spreadLanes(n);
  int slot = -1;
  bool exhausted = false;  // warp-uniform
  BinTrav t;
  TravStack stack;
  float trProd = 1.0f;
  float3 tau = v3(0.0f);
  while (true) {
    const unsigned idle = __ballot_sync(full, slot < 0) & lanes;
    if (!exhausted && (idle == lanes || __popc(idle) >= SDB_WF_FETCH_IDLE)) {
      const int leader = __ffs(idle) - 1;
      unsigned base = 0;
      if ((int)(threadIdx.x & 31) == leader)
        base = atomicAdd(&pool.counts[it].fetchShadow, (unsigned)__popc(idle));
      base = __shfl_sync(full, base, leader);
      if (base + __popc(idle) >= n) exhausted = true;
      if (idle >> (threadIdx.x & 31) & 1u) {
        unsigned i = base + __popc(idle & ltMask);
        if (i < n) {
          slot = pool.shadowList[i];
          const Rec r = ldRec(pool.shadowRays, slot);
          binTravStart(t, slotLaunch<GUIDE>(slot), v3(r.a.x, r.a.y, r.a.z),
                       v3(r.a.w, r.b.x, r.b.y), r.b.z);
          trProd = 1.0f;
          tau = v3(0.0f);
        }
      }
    }
    if (__ballot_sync(full, slot >= 0) == 0) {
      if (exhausted) break;
      continue;
    }
    const SdLaunch& lp = slotLaunch<GUIDE>(slot >= 0 ? slot : 0);
    ShadowSink sink{pool, slot};
    int r = kTravMore;
    // Leaves first (instances, then triangles one at a time while enough
    // lanes hold one), then node visits in a row while enough lanes are at
    // one; lanes that reach a leaf meanwhile wait for the next round.
    int kind = slot < 0 ? kNoRay : travKind(t);
    {
      const int insts = __popc(__ballot_sync(full, kind == kAtInstance));
      if (insts >= (exhausted ? 1 : SDB_WF_INST_MIN) || __ballot_sync(full, kind == kAtNode || kind == kAtTriangle) == 0) {
        if (kind == kAtInstance) {
          r = t.cur == kPop ? binTravPop(t, stack, sink)
                            : binTravInstance<true, false, true>(t, stack, lp, sink, trProd, tau, nullptr);
          kind = r == kTravMore ? travKind(t) : kNoRay;
        }
      }
    }
    for (int tris = __popc(__ballot_sync(full, kind == kAtTriangle)); tris > 0;) {
      if (kind == kAtTriangle) {
        r = binTravTriangle<true, false>(t, stack, lp, sink, trProd, tau, nullptr);
        kind = r == kTravLeaf ? kAtTriangle : (r == kTravMore ? travKind(t) : kNoRay);
      }
      tris = __popc(__ballot_sync(full, kind == kAtTriangle));
      if (tris < SDB_WF_TRI_MIN) break;
    }
    for (int nodes = __popc(__ballot_sync(full, kind == kAtNode)); nodes > 0;) {
      if (kind == kAtNode) {
        r = binTravNode<true, false, false, true>(t, stack, lp, sink, nullptr);
        kind = r == kTravMore ? travKind(t) : kNoRay;
      }
      nodes = __popc(__ballot_sync(full, kind == kAtNode));
      if (nodes < SDB_WF_NODE_MIN) break;
    }
    if (slot >= 0 && (r == kTravDone || r == kTravOccluded)) {
      float3 tr = v3(0.0f);
      if (r == kTravDone) {
        tau = v3(fmaxf(0.0f, tau.x), fmaxf(0.0f, tau.y), fmaxf(0.0f, tau.z));
        tr = v3(trProd);
        if (hmax(tau) > 0.0f) tr = tr * vexp(-tau);
      }
      const unsigned flags = reinterpret_cast<const unsigned*>(pool.shadowRays + 2 * (size_t)slot)[7];
      finishShadow<GUIDE>(pool, slot, flags, tr, depth);
      slot = -1;
    }
  }
}
#else
// The 8-wide build traces shadow rays one per thread.
template <int GUIDE>
__global__ void wfShadowFetch(int, int) {}
#endif

// Late vertices (their shadow ray's transmittance is in shadowTerms): the
// NEE contribution, the BSDF sample, roulette. GUIDE & kGuideRecord: the
// guided vertex joins the slot's trail.
template <int GUIDE>
__global__ void __launch_bounds__(kRenderBlock, SDB_WF_LATE_BLOCKS) wfLate(int it, int depth) {
  const WfPool& pool = c_pool;
  const unsigned n = pool.counts[it].late;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int slot = pool.lateList[i];
    const SdLaunch& lp = slotLaunch<GUIDE>(slot);
    Path p;
    loadPath(pool, lp, slot, depth, p);
    const LateVertex l = pool.verts[slot].v;
    const Rec r = ldRec(pool.shadowRays, slot);
    Vertex v;
    v.x = l.x;
    v.ns = l.ns;
    v.albedo = l.albedo;
    v.etaExt = l.etaExt;
    v.etaRel = l.etaRel;
    v.matId = l.matId;
    v.front = l.front;
    v.nee = true;  // it waited for its shadow ray
    v.lightK = l.lightK;
    v.so = v3(r.a.x, r.a.y, r.a.z);
    v.wi = v3(r.a.w, r.b.x, r.b.y);
    v.Li = l.Li;
    v.tmaxS = r.b.z;
    v.pdf = l.pdf;
    v.cosS = l.cosS;
    v.delta = l.delta;
    const float4 tr = pool.shadowTerms[slot];
    GuideTrail* trail = (GUIDE & kGuideRecord) ? &pool.trails[slot].v : nullptr;
    if (finishVertex<GUIDE, kRound<GUIDE>>(lp, p, v, v3(tr.x, tr.y, tr.z), trail)) {
      storePath(pool, p, slot);
      pool.lists[(it + 1) & 1][appendSlot(&pool.counts[it + 1].live)] = slot;
    } else {
      finishPath<GUIDE>(p.L, p.slot, slot);
    }
  }
}

// Reports to the host how many rays iteration it + 1 has, under the ticket of
// iteration it.
constexpr int kRaysBits = 28;  // a pool holds fewer rays
__global__ void wfReport(int it, unsigned long long ticket) {
  *c_pool.seen = ticket << kRaysBits | c_pool.counts[it + 1].live;
}

// Between two groups of iterations: the last list's length moves to the
// front (kWfGroup is even, so the list keeps its place), the rest clears.
__global__ void wfNextGroup() {
  WfCounts* c = c_pool.counts;
  const unsigned live = c[kWfGroup].live;
  __syncwarp();
  for (int k = threadIdx.x; k < (int)((kWfGroup + 1) * sizeof(WfCounts) / 4); k += 32)
    reinterpret_cast<unsigned*>(c)[k] = 0;
  __syncwarp();
  if (threadIdx.x == 0) c[0].live = live;
}
static_assert(kWfGroup % 2 == 0, "lists ping-pong back to their place");

// ---- host ---------------------------------------------------------------------

template <typename K>
static int gridFor(K kernel, int block = kRenderBlock) {
  int dev = 0, sms = 0, perSm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, block, 0);
  return sms * (perSm < 1 ? 1 : perSm);
}

bool wfHasLate(const SdLaunch& lp, int guide) {
  return (guide & kGuideRecord) || (lp.numFlames > 0 && lp.transparentShadows);
}

void WfBuffers::ensure(int slots, bool withLate) {
  if (slots > cap) grow(slots, withLate);
  if (withLate) ensureLate(slots);
}

void WfBuffers::grow(int slots, bool withLate) {
  // At most half of the device memory that is free (counting the pool about
  // to be replaced), so films, scenes and other work keep room; at least
  // 1 M slots.
  size_t freeB = 0, totB = 0;
  cudaCheck(cudaMemGetInfo(&freeB, &totB), "cudaMemGetInfo");
  const bool within = withLate && !verts.ptr;  // late vertices in the slab
  const size_t per = wfSlotBytes() + (within ? wfLateBytes() : 0);
  const size_t fit = std::max<size_t>((freeB + slab.bytes) / 2 / per, (size_t)1 << 20);
  slots = (int)std::min<size_t>((size_t)slots, fit);
  if (slots <= cap) return;
  const size_t n = (size_t)slots;
  const size_t sizes[12] = {n * 32, n * 32, n * 32, n * 32, n * 32, n * 16,
                            n * sizeof(int), n * sizeof(int), n * sizeof(int), n * sizeof(int), n,
                            within ? n * wfLateBytes() : 0};
  size_t offs[12], total = 0;
  for (int k = 0; k < 12; k++) {
    offs[k] = total;
    total += (sizes[k] + 255) & ~(size_t)255;
  }
  cap = 0;
  if (!verts.ptr) lateCap = 0;  // those in the slab go with it
  slab.release();
  slab.alloc(total);
  char* base = (char*)slab.ptr;
  pool.ray = (float4*)(base + offs[0]);
  pool.sum = (float4*)(base + offs[1]);
  pool.rest = (float4*)(base + offs[2]);
  pool.hits = (float4*)(base + offs[3]);
  pool.shadowRays = (float4*)(base + offs[4]);
  pool.shadowTerms = (float4*)(base + offs[5]);
  pool.lists[0] = (int*)(base + offs[6]);
  pool.lists[1] = (int*)(base + offs[7]);
  pool.shadowList = (int*)(base + offs[8]);
  pool.lateList = (int*)(base + offs[9]);
  pool.jobs = (unsigned char*)(base + offs[10]);
  if (within) {
    pool.verts = (PoolSlot<LateVertex>*)(base + offs[11]);
    lateCap = slots;
  }
  if (!counts.ptr) counts.alloc((kWfGroup + 1) * sizeof(WfCounts));
  pool.counts = (WfCounts*)counts.ptr;
  if (!hostCount) hostCount = pinnedWords();
  if (!hostSeen) {
    hostSeen = pinnedWords();
    pool.seen = reinterpret_cast<unsigned long long*>(hostSeen);
    *pool.seen = 0;
  }
  if (!side) {
    cudaCheck(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking), "shadow stream");
    cudaCheck(cudaEventCreateWithFlags(&shaded, cudaEventDisableTiming), "shadow events");
    cudaCheck(cudaEventCreateWithFlags(&shadowDone, cudaEventDisableTiming), "shadow events");
  }
  cap = slots;
  gridTrace = gridFor(wfTraceFetch<false, false>);
  gridShade = gridFor(wfShade<0, false>, kShadeBlock);
  gridShadow = gridFor(wfShadow<0>);
  gridLate = gridFor(wfLate<0>);
  gridStart = gridFor(wfStart<0>);
  gridFlame = gridFor(wfFlame<0, false>);
}

void WfBuffers::ensureLate(int slots, size_t keep) {
  slots = std::min(slots, cap);
  if (slots <= lateCap) return;
  // A buffer of its own: a pool kept from a large frame is not made again for
  // the late vertices of a small one. Half of the free memory at most, as the
  // pool's.
  size_t freeB = 0, totB = 0;
  cudaCheck(cudaMemGetInfo(&freeB, &totB), "cudaMemGetInfo");
  freeB += verts.bytes;
  const size_t fit = std::max<size_t>((freeB > keep ? freeB - keep : 0) / 2 / wfLateBytes(),
                                      (size_t)1 << 20);
  slots = (int)std::min<size_t>((size_t)slots, fit);
  if (slots <= lateCap) return;
  lateCap = 0;
  verts.alloc((size_t)slots * wfLateBytes());
  pool.verts = (PoolSlot<LateVertex>*)verts.ptr;
  lateCap = slots;
}

void WfBuffers::ensureTrails() {
  if (trailCap >= cap) return;
  trails.alloc((size_t)cap * sizeof(PoolSlot<GuideTrail>));
  trailCap = cap;
}

WfBuffers::~WfBuffers() {
  if (hostCount) returnPinnedWords(hostCount);
  if (hostSeen) returnPinnedWords(hostSeen);
  for (cudaEvent_t& e : ev)
    if (e) cudaEventDestroy(e);
  if (shaded) cudaEventDestroy(shaded);
  if (shadowDone) cudaEventDestroy(shadowDone);
  if (side) cudaStreamDestroy(side);
}

// One idle pool per device, kept between sessions while the device-memory
// cache is on (sundog_set_device_memory_cache); otherwise a finished
// session's pool is freed with it.
static std::mutex g_poolMu;
static std::unique_ptr<WfBuffers> g_idle[64];

std::unique_ptr<WfBuffers> wfAcquire() {
  int dev = 0;
  cudaCheck(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> lock(g_poolMu);
  if (dev >= 0 && dev < 64 && g_idle[dev]) return std::move(g_idle[dev]);
  return std::unique_ptr<WfBuffers>(new WfBuffers());
}

void wfRelease(std::unique_ptr<WfBuffers> b) {
  if (!b) return;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
  if (!keepDeviceMemory()) return;  // b frees its buffers here
  std::lock_guard<std::mutex> lock(g_poolMu);
  if (!g_idle[dev] || g_idle[dev]->cap < b->cap) g_idle[dev] = std::move(b);
}

void wfReleaseIdle() {
  int cur = 0;
  if (cudaGetDevice(&cur) != cudaSuccess) return;
  std::lock_guard<std::mutex> lock(g_poolMu);
  for (int d = 0; d < 64; d++) {
    if (!g_idle[d]) continue;
    if (cudaSetDevice(d) == cudaSuccess) g_idle[d].reset();
  }
  cudaSetDevice(cur);
}

size_t wfSlotBytes() { return 6 * 32 - 16 + 4 * sizeof(int) + 1; }
size_t wfLateBytes() { return sizeof(PoolSlot<LateVertex>); }

// What the launches of a render or batch need.
struct WfPlan {
  int mode;           // guide bits, or kWfServe
  bool shadowFetch;   // the shadow-ray kernel (kShadowFetchInstances)
  bool lights;        // any NEE strategy: shadow rays can exist
  bool late;          // late vertices can exist
  bool flames;        // some scene has flames
  int maxDepth;
};

// The shadow rays of an iteration and the radiance rays of the next need
// nothing of each other: without late vertices the shadow stage runs on the
// pool's second stream, beside the next trace, until the next flame march or
// shading.
static bool shadowBeside(const WfPlan& plan, bool timed) {
  return plan.lights && !plan.late && !timed;
}

// One iteration's stage kernels for mode GUIDE (guide bits, or kWfServe).
// With `timed`, events ev[1..5] bracket the stage launches.
template <int GUIDE, bool CAM>
static int wfIteration(const WfBuffers& b, cudaStream_t st, int it, int depth,
                       unsigned long long base, const WfPlan& plan, unsigned long long ticket,
                       bool timed) {
  constexpr int kScene = GUIDE & kWfServe;  // stages that neither guide nor record
  int launches = 2;
  const bool beside = shadowBeside(plan, timed);
  if (timed) cudaEventRecord(b.ev[1], st);
  wfTraceFetch<kScene != 0, CAM><<<b.gridTrace, kRenderBlock, 0, st>>>(it, plan.shadowFetch);
  if (timed) cudaEventRecord(b.ev[2], st);
  // The flame march and shading read and write the radiance it adds to.
  if (beside && !CAM) cudaCheck(cudaStreamWaitEvent(st, b.shadowDone, 0), "shadow stage");
  if (plan.flames) {
    wfFlameScan<kScene, CAM><<<b.gridStart, kRenderBlock, 0, st>>>(it);
    wfFlame<kScene, CAM><<<b.gridFlame, kRenderBlock, 0, st>>>(it, depth, base);
    launches += 2;
  }
  wfShade<GUIDE, CAM><<<b.gridShade, kShadeBlock, 0, st>>>(it, depth, base);
  if (timed) cudaEventRecord(b.ev[3], st);
  if (plan.lights) {
    cudaStream_t ss = st;
    if (beside) {
      ss = b.side;
      cudaCheck(cudaEventRecord(b.shaded, st), "shading stage");
      cudaCheck(cudaStreamWaitEvent(ss, b.shaded, 0), "shading stage");
    }
    if (plan.shadowFetch && !SDB_WIDE_BVH)
      wfShadowFetch<kScene><<<b.gridShadow, kRenderBlock, 0, ss>>>(it, depth);
    else
      wfShadow<kScene><<<b.gridShadow, kRenderBlock, 0, ss>>>(it, depth);
    launches++;
    if (beside) {
      cudaCheck(cudaEventRecord(b.shadowDone, ss), "shadow stage");
      if (depth + 1 >= plan.maxDepth || it + 1 == kWfGroup)  // back to one stream
        cudaCheck(cudaStreamWaitEvent(st, b.shadowDone, 0), "shadow stage");
    }
  }
  if (timed) cudaEventRecord(b.ev[4], st);
  if (plan.late) {
    wfLate<GUIDE><<<b.gridLate, kRenderBlock, 0, st>>>(it, depth);
    launches++;
  }
  if (timed) cudaEventRecord(b.ev[5], st);
  if (ticket) {  // on the second stream: no stage waits for it
    if (!beside) {
      cudaCheck(cudaEventRecord(b.shaded, st), "ray report");
      cudaCheck(cudaStreamWaitEvent(b.side, b.shaded, 0), "ray report");
    }
    wfReport<<<1, 1, 0, b.side>>>(it, ticket);
    launches++;
  }
  return launches;
}

template <int GUIDE>
static int wfIterationAny(const WfBuffers& b, cudaStream_t st, int it, int depth,
                          unsigned long long base, const WfPlan& plan,
                          unsigned long long ticket, bool timed) {
  return depth == 0 ? wfIteration<GUIDE, true>(b, st, it, depth, base, plan, ticket, timed)
                    : wfIteration<GUIDE, false>(b, st, it, depth, base, plan, ticket, timed);
}

// Tickets grow over all pools of the process: words that another pool's
// reports were written to hold smaller ones.
static unsigned long long nextTicket() {
  static std::atomic<unsigned long long> last{0};
  return ++last;
}

// Whether a report under this ticket or a later one says that no rays are
// left; waits for one. The report is queued on the second stream, so it comes,
// or that stream ends in an error.
static bool raysEnded(const WfBuffers& b, unsigned long long ticket) {
  const volatile unsigned long long* seen = b.pool.seen;
  for (unsigned spins = 1;; spins++) {
    const bool check = spins % 4096 == 0;
    const cudaError_t e = check ? cudaStreamQuery(b.side) : cudaErrorNotReady;
    const unsigned long long v = *seen;
    if (v >> kRaysBits >= ticket) return (v & ((1ull << kRaysBits) - 1)) == 0;
    if (e == cudaErrorNotReady) {
      if (check) std::this_thread::yield();
      continue;
    }
    cudaCheck(e, "wavefront iteration");
    throw std::runtime_error("wavefront: an iteration did not report");
  }
}

static double evMs(cudaEvent_t a, cudaEvent_t b) {
  float ms = 0.0f;
  cudaCheck(cudaEventElapsedTime(&ms, a, b), "stage timing");
  return ms;
}

constexpr unsigned kReportPaths = 1u << 18;  // runPool

// Renders path ids [0, numPaths), a pool of them at a time, each through
// stage iterations until no path is live (the launch block or batch is
// already in constant memory). Paths of a pool share their depth, so
// plan.maxDepth iterations end them all; in groups of kWfGroup, with a look
// at the live count between groups. In small pools, where an empty iteration
// (9 us) is much of a render, the host also stops within a group when a report
// says that no rays are left, an iteration or two behind the one being
// launched: a view of the sky at 64x48 and 4 samples takes 144 us, 193 with all
// eight iterations launched and 165 with a look after each; views that last all
// eight are within 0.4%. From 262,144 paths on the reports cost more than they
// save (instancing 333x217 at 5 samples 1,359 -> 1,377). Returns the kernels
// launched.
static int runPool(WfBuffers& b, cudaStream_t st, unsigned long long numPaths, const WfPlan& plan,
                   WfStageTimes* times = nullptr) {
  const bool timed = times != nullptr;
  if (timed && !b.ev[0])
    for (cudaEvent_t& e : b.ev) cudaCheck(cudaEventCreate(&e), "stage timing events");
  WfPool pool = b.pool;
  pool.trails = (PoolSlot<GuideTrail>*)b.trails.ptr;
  // Paths in flight at once: slots, with a late vertex each where there can be some.
  const int cap = plan.late ? std::min(b.cap, b.lateCap) : b.cap;
  if (cap < 1) throw std::runtime_error("wavefront: no path slots");
  cudaCheck(cudaMemcpyToSymbolAsync(c_pool, &pool, sizeof pool, 0, cudaMemcpyHostToDevice, st),
            "wavefront pool");
  int launches = 0;
  for (unsigned long long base = 0; base < numPaths; base += (unsigned long long)cap) {
    const unsigned n = (unsigned)std::min<unsigned long long>((unsigned long long)cap,
                                                              numPaths - base);
    cudaCheck(cudaMemsetAsync(b.counts.ptr, 0, b.counts.bytes, st), "wavefront counts");
    if (timed) cudaEventRecord(b.ev[0], st);
    if (plan.mode & kWfServe) wfStart<kWfServe><<<b.gridStart, kRenderBlock, 0, st>>>(base, n);
    else wfStart<0><<<b.gridStart, kRenderBlock, 0, st>>>(base, n);
    cudaCheck(cudaGetLastError(), "wfStart");
    launches++;
    if (timed) {
      cudaEventRecord(b.ev[1], st);
      cudaCheck(cudaEventSynchronize(b.ev[1]), "wfStart");
      times->startMs += evMs(b.ev[0], b.ev[1]);
      times->launches++;
    }
    unsigned long long tickets[kWfGroup] = {};  // of the group's reports
    for (int depth = 0;; depth++) {
      const int it = depth % kWfGroup;
      if (depth > 0 && it == 0) {  // the next group of iterations
        unsigned* live = &((WfCounts*)b.counts.ptr)[kWfGroup].live;
        cudaCheck(cudaMemcpyAsync(b.hostCount, live, sizeof(unsigned), cudaMemcpyDeviceToHost, st),
                  "wavefront count");
        cudaCheck(cudaStreamSynchronize(st), "wavefront group");
        if (b.hostCount[0] == 0) break;
        wfNextGroup<<<1, 32, 0, st>>>();
        launches++;
      }
      if (it >= 2 && tickets[it - 2] && raysEnded(b, tickets[it - 2])) {
        cudaCheck(cudaEventRecord(b.shadowDone, b.side), "shadow stage");  // back to one stream
        cudaCheck(cudaStreamWaitEvent(st, b.shadowDone, 0), "shadow stage");
        break;
      }
      // Asked for before the iteration after the next one of the group; every
      // other one (each takes 0.9 us of a small render).
      const bool asked = !timed && n <= kReportPaths && it % 2 == 0 && it + 2 < kWfGroup &&
                         depth + 2 < plan.maxDepth;
      const unsigned long long ticket = tickets[it] = asked ? nextTicket() : 0;
      int k;
      switch (plan.mode) {
        case 0: k = wfIterationAny<0>(b, st, it, depth, base, plan, ticket, timed); break;
        case kGuideSample:
          k = wfIterationAny<kGuideSample>(b, st, it, depth, base, plan, ticket, timed);
          break;
        case kGuideRecord:
          k = wfIterationAny<kGuideRecord>(b, st, it, depth, base, plan, ticket, timed);
          break;
        case kGuideSample | kGuideRecord:
          k = wfIterationAny<kGuideSample | kGuideRecord>(b, st, it, depth, base, plan, ticket, timed);
          break;
        default: k = wfIterationAny<kWfServe>(b, st, it, depth, base, plan, ticket, timed); break;
      }
      cudaCheck(cudaGetLastError(), "wavefront stage");
      launches += k;
      if (timed) {
        static_assert(offsetof(WfCounts, traced) == 3 * sizeof(unsigned), "counter order");
        cudaCheck(cudaMemcpyAsync(b.hostCount, (WfCounts*)b.counts.ptr + it, 4 * sizeof(unsigned),
                                  cudaMemcpyDeviceToHost, st),
                  "wavefront count");
        cudaCheck(cudaStreamSynchronize(st), "wavefront iteration");
        times->traceMs += evMs(b.ev[1], b.ev[2]);
        times->shadeAMs += evMs(b.ev[2], b.ev[3]);
        times->shadowMs += evMs(b.ev[3], b.ev[4]);
        times->shadeBMs += evMs(b.ev[4], b.ev[5]);
        times->iterations++;
        times->launches += k;
        times->radianceRays += b.hostCount[3];
        times->shadowRays += b.hostCount[1];
      }
      if (depth + 1 >= plan.maxDepth) break;
    }
  }
  return launches;
}

int wfRender(const SdLaunch& lp, WfBuffers& b, cudaStream_t st, int guide, WfStageTimes* times) {
  if (guide < 0 || guide > (kGuideSample | kGuideRecord))
    throw std::runtime_error("wavefront: invalid guide mode");
  if (guide & kGuideRecord) b.ensureTrails();
  cudaCheck(cudaMemcpyToSymbolAsync(c_wlp, &lp, sizeof lp, 0, cudaMemcpyHostToDevice, st),
            "wavefront launch block");
  const WfPlan plan = {guide, lp.numInstances >= kShadowFetchInstances,
                       lp.numLights > 0 || lp.bgKind == BG_ENVMAP, wfHasLate(lp, guide),
                       lp.numFlames > 0, lp.maxDepth};
  return runPool(b, st, lp.numPaths, plan, times);
}

cudaError_t wfSetJobs(const SdLaunch* table, cudaStream_t st) {
  return cudaMemcpyToSymbolAsync(c_wjobs, table, kMaxServeJobs * sizeof(SdLaunch), 0,
                                 cudaMemcpyHostToDevice, st);
}

int wfRenderBatch(const ServeBatch& batch, WfBuffers& b, cudaStream_t st, const SdLaunch* jobs) {
  cudaCheck(cudaMemcpyToSymbolAsync(c_wbatch, &batch, sizeof batch, 0, cudaMemcpyHostToDevice, st),
            "wavefront batch");
  WfPlan plan = {kWfServe, false, false, false, false, 0};
  for (int k = 0; k < kMaxServeJobs; k++) {  // unused slots are zero
    const SdLaunch& lp = jobs[k];
    plan.shadowFetch = plan.shadowFetch || lp.numInstances >= kShadowFetchInstances;
    plan.lights = plan.lights || lp.numLights > 0 || (lp.width > 0 && lp.bgKind == BG_ENVMAP);
    plan.late = plan.late || wfHasLate(lp, 0);
    plan.flames = plan.flames || lp.numFlames > 0;
    plan.maxDepth = std::max(plan.maxDepth, lp.maxDepth);
  }
  return runPool(b, st, batch.numPaths, plan);
}

}  // namespace sdb
