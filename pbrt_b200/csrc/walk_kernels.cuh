// walk_kernels.cuh — the persistent walks over a wave's queues, for one kind of scene source.
#pragma once

#include <cstdio>
#include <cstdlib>

#include "scene_walk.cuh"
#include "walk.cuh"

// Resident 256-thread blocks per SM the walks are compiled for (4: at most 64 registers a thread).
#ifndef PBRT_WALK_BLOCKS
#define PBRT_WALK_BLOCKS 4
#endif
#ifndef PBRT_WALK_OBJ_BLOCKS
#define PBRT_WALK_OBJ_BLOCKS 4
#endif

namespace pbrt {

// Scene::find_nearest for the queued paths.
template <class Src>
struct PathRays {
  const WaveBuffers& w;
  const Src& src;
  const uint32_t* q;
  uint32_t p;
  typename Src::Cursor c;
  PBRT_DEV void load(uint64_t k, F3& o, F3& d) {
    p = q[k];
    c = src.cursor(w, p);
    o = mk3(w.ox[p], w.oy[p], w.oz[p]);
    d = mk3(w.dx[p], w.dy[p], w.dz[p]);
  }
  PBRT_DEV float near() const { return src.settings(c).near; }
  PBRT_DEV float far() const { return src.settings(c).far; }
  PBRT_DEV const SceneView& scene() const { return src.view(c); }
  PBRT_DEV void store(bool have, float t, uint32_t leaf, uint32_t prim) {
    w.ht[p] = have ? t : 0.f;
    w.hobj[p] = have ? leaf : 0xFFFFFFFFu;
    w.hprim[p] = prim;
  }
};

// The walks are built without the code of primitives that are not merged meshes, and of solids,
// where the scenes have none: it takes registers from every other query.
template <class Src, bool kObj, bool kCsg, bool kEach>
__global__ void __launch_bounds__(256, kObj ? PBRT_WALK_OBJ_BLOCKS : PBRT_WALK_BLOCKS) k_nearest(const __grid_constant__ WaveBuffers w,
                                                               const __grid_constant__ Src src,
                                                               const uint32_t* __restrict__ q,
                                                               const uint32_t* __restrict__ qcount, uint32_t* fetch,
                                                               uint32_t* next_count, WalkSchedule ws, uint32_t* err,
                                                               unsigned long long* stats) {
  const uint32_t n = *qcount;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // the words this bounce's shading and shadow kernels count in, last used in the bounce before
    *next_count = 0u;
    w.counts[2] = 0u;
    w.counts[4] = 0u;
    if (stats) atomicAdd(stats, (unsigned long long)n);
  }
  PathRays<Src> job{w, src, q, 0u, {}};
  static_assert(!kEach || !kObj, "one thread per ray: merged meshes only");
  if constexpr (kEach) each_nearest(job, n, err);
  else walk_nearest<kObj, kCsg>(job, walk_queue(fetch, n), ws, err);
}

// The shadow queue: an unoccluded entry adds its light sample (VisibilityTester::unoccluded,
// lights.rs:67-69).
template <class Src>
struct ShadowRays {
  const WaveBuffers& w;
  const Src& src;
  uint32_t k;
  typename Src::Cursor c;
  PBRT_DEV void load(uint64_t kk, F3& o, F3& d) {
    k = uint32_t(kk);
    c = src.cursor(w, w.s_path[k]);
    o = mk3(w.s_ox[k], w.s_oy[k], w.s_oz[k]);
    d = mk3(w.s_dx[k], w.s_dy[k], w.s_dz[k]);
  }
  PBRT_DEV float near() const { return kShadowEps; }
  PBRT_DEV float far() const { return w.s_tmax[k]; }
  PBRT_DEV const SceneView& scene() const { return src.view(c); }
  PBRT_DEV void store(bool occluded) {
    if (occluded) return;
    const uint32_t p = w.s_path[k];
    w.lr[p] = fa(w.lr[p], w.s_cr[k]);
    w.lg[p] = fa(w.lg[p], w.s_cg[k]);
    w.lb[p] = fa(w.lb[p], w.s_cb[k]);
  }
};

template <class Src, bool kObj, bool kCsg, bool kEach>
__global__ void __launch_bounds__(256, kObj ? PBRT_WALK_OBJ_BLOCKS : PBRT_WALK_BLOCKS) k_shadow(const __grid_constant__ WaveBuffers w,
                                                              const __grid_constant__ Src src, uint32_t* fetch,
                                                              WalkSchedule ws, uint32_t* err,
                                                              unsigned long long* stats) {
  const uint32_t n = w.counts[2];
  if (stats && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(stats + 1, (unsigned long long)n);
  ShadowRays<Src> job{w, src, 0u, {}};
  static_assert(!kEach || !kObj, "one thread per ray: merged meshes only");
  if constexpr (kEach) each_any(job, n, err);
  else walk_any<kObj, kCsg>(job, walk_queue(fetch, n), ws, err);
}

// The walks' step schedules: a leaf step once `leaf_min` lanes of a warp stand on a leaf, a refill
// once `refill_min` lanes are idle, up to `burst` nodes per node step. PBRT_WALK_SCHEDULE=
// "leaf_min,refill_min[,burst]" (each in 1..32) overrides them for measurements; answers do not
// depend on it.
inline WalkSchedule walk_schedule(bool objects) {
  static const WalkSchedule v = [] {
    WalkSchedule d{0, 0, 0};
    if (const char* e = std::getenv("PBRT_WALK_SCHEDULE")) {
      int a = 0, b = 0, c = 4;
      if (std::sscanf(e, "%d,%d,%d", &a, &b, &c) >= 2 && a >= 1 && a <= 32 && b >= 1 && b <= 32 && c >= 1 && c <= 32)
        d = WalkSchedule{a, b, c};
    }
    return d;
  }();
  if (v.leaf_min) return v;
  return objects ? WalkSchedule{16, 8, 8} : WalkSchedule{16, 8, 4};
}

// Blocks of a persistent walk: no more than are resident.
template <bool kObj>
unsigned walk_blocks(const WalkLaunch& l) {
  const unsigned resident = 256u * (kObj ? PBRT_WALK_OBJ_BLOCKS : PBRT_WALK_BLOCKS) / l.shape.trace_threads;
  return unsigned(l.sm_count) * (l.shape.trace_blocks_per_sm < resident ? l.shape.trace_blocks_per_sm : resident);
}

// One thread per ray for a wave of at most kEachMaxPaths in mesh scenes of at most kEachMaxNodes
// wide nodes. A closed box of 34 triangles (some 20 nodes), two chains of waves, persistent
// against one thread per ray: 0.52 M paths a wave 1.82 / 1.78 ms, 0.36 M at depth 20 2.72 / 2.43,
// 0.56 M at depth 6 1.51 / 1.50; but 0.85 M 2.68 / 2.77, 1.7 M 5.06 / 5.94, 3.4 M 9.82 / 13.2.
// Larger trees are persistent throughout.
constexpr uint32_t kEachMaxNodes = 128, kEachMaxPaths = 3u << 18;
inline bool walk_each(const WalkLaunch& l) { return l.nodes <= kEachMaxNodes && l.paths <= kEachMaxPaths; }

template <bool kObj, bool kCsg, bool kEach, class Src>
cudaError_t run_nearest(const WaveBuffers& w, const Src& src, const uint32_t* q, const uint32_t* qcount,
                        uint32_t* fetch, uint32_t* next_count, const WalkLaunch& l) {
  const unsigned g = kEach ? unsigned(l.sm_count) * l.shape.trace_blocks_per_sm : walk_blocks<kObj>(l);
  k_nearest<Src, kObj, kCsg, kEach><<<g, l.shape.trace_threads, 0, l.st>>>(w, src, q, qcount, fetch, next_count,
                                                                           walk_schedule(kObj), l.err, l.stats);
  return cudaGetLastError();
}

template <bool kObj, bool kCsg, bool kEach, class Src>
cudaError_t run_shadow(const WaveBuffers& w, const Src& src, uint32_t* fetch, const WalkLaunch& l) {
  const unsigned g = kEach ? unsigned(l.sm_count) * l.shape.trace_blocks_per_sm : walk_blocks<kObj>(l);
  k_shadow<Src, kObj, kCsg, kEach><<<g, l.shape.trace_threads, 0, l.st>>>(w, src, fetch, walk_schedule(kObj), l.err,
                                                                          l.stats);
  return cudaGetLastError();
}

template <class Src>
cudaError_t launch_nearest_for(const WaveBuffers& w, const Src& src, const uint32_t* q, const uint32_t* qcount,
                               uint32_t* fetch, uint32_t* next_count, const WalkLaunch& l) {
  if (l.csg) return run_nearest<true, true, false>(w, src, q, qcount, fetch, next_count, l);
  if (l.objects) return run_nearest<true, false, false>(w, src, q, qcount, fetch, next_count, l);
  if (walk_each(l)) return run_nearest<false, false, true>(w, src, q, qcount, fetch, next_count, l);
  return run_nearest<false, false, false>(w, src, q, qcount, fetch, next_count, l);
}

template <class Src>
cudaError_t launch_shadow_for(const WaveBuffers& w, const Src& src, uint32_t* fetch, const WalkLaunch& l) {
  if (l.csg) return run_shadow<true, true, false>(w, src, fetch, l);
  if (l.objects) return run_shadow<true, false, false>(w, src, fetch, l);
  if (walk_each(l)) return run_shadow<false, false, true>(w, src, fetch, l);
  return run_shadow<false, false, false>(w, src, fetch, l);
}

}  // namespace pbrt
