// kernels_scene_rays.cu — ray casting over any scene: the walks over a caller's rays, and the
// counted forms on the binary trees.
#include <cfloat>
#include <cstdint>

#include "walk_kernels.cuh"

namespace pbrt {

// Adds a thread's counters to cnt[0..2] (one atomic per warp and counter).
PBRT_DEV void flush_counts(const SceneCount& c, unsigned long long* cnt) {
  unsigned long long v[3] = {c.nodes, c.boxes, c.objects};
  for (int k = 0; k < 3; ++k) {
    for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xFFFFFFFFu, v[k], off);
    if ((threadIdx.x & 31) == 0 && v[k]) atomicAdd(cnt + k, v[k]);
  }
}

// Nearest hit per ray with the scene accelerator's counters (Scene::intersect_instrumented) added
// into cnt, one thread per ray on the binary trees; object ids are the description's (the leaf's
// desc_id).
__global__ void __launch_bounds__(128) k_scene_closest_counted(SceneView s, const float* __restrict__ rays,
                                                               uint64_t stride, uint64_t n, uint32_t* __restrict__ prim,
                                                               float* __restrict__ tout, uint32_t* __restrict__ obj,
                                                               unsigned long long* cnt, uint32_t* err) {
  SceneCount c{0, 0, 0};
  // whole warps run the same trip count so the counter reduction sees full warps
  const uint64_t step = uint64_t(gridDim.x) * blockDim.x;
  const uint64_t iters = (n + step - 1) / step;
  for (uint64_t it = 0; it < iters; ++it) {
    const uint64_t i = it * step + uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) continue;
    const F3 o = mk3(__ldcs(rays + i), __ldcs(rays + stride + i), __ldcs(rays + 2 * stride + i));
    const F3 d = mk3(__ldcs(rays + 3 * stride + i), __ldcs(rays + 4 * stride + i), __ldcs(rays + 5 * stride + i));
    const float near = __ldcs(rays + 6 * stride + i), far = __ldcs(rays + 7 * stride + i);
    float t = 0.f;
    uint32_t leaf = 0, pr = 0;
    const bool hit = scene_closest_t<true, true>(s, o, d, near, far, t, leaf, pr, err, &c);
    __stcs(prim + i, hit ? pr : 0xFFFFFFFFu);
    __stcs(tout + i, hit ? t : __int_as_float(0x7f800000));
    if (obj) __stcs(obj + i, hit ? s.objects[leaf].desc_id : 0xFFFFFFFFu);
  }
  flush_counts(c, cnt);
}

__global__ void __launch_bounds__(128) k_scene_any_counted(SceneView s, const float* __restrict__ rays, uint64_t stride,
                                                           uint64_t n, uint8_t* __restrict__ occ,
                                                           unsigned long long* cnt, uint32_t* err) {
  SceneCount c{0, 0, 0};
  const uint64_t step = uint64_t(gridDim.x) * blockDim.x;
  const uint64_t iters = (n + step - 1) / step;
  for (uint64_t it = 0; it < iters; ++it) {
    const uint64_t i = it * step + uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) continue;
    const F3 o = mk3(__ldcs(rays + i), __ldcs(rays + stride + i), __ldcs(rays + 2 * stride + i));
    const F3 d = mk3(__ldcs(rays + 3 * stride + i), __ldcs(rays + 4 * stride + i), __ldcs(rays + 5 * stride + i));
    occ[i] = scene_any_t<true, true>(s, o, d, __ldcs(rays + 6 * stride + i), __ldcs(rays + 7 * stride + i), err, &c)
                 ? 1
                 : 0;
  }
  flush_counts(c, cnt);
}

// The rays of a caller's planes.
struct PlaneRays {
  const SceneView& s;
  const float* rays;
  uint64_t stride;
  uint32_t* prim;
  float* tout;
  uint32_t* obj;
  uint8_t* occ;
  uint64_t i;
  PBRT_DEV void load(uint64_t k, F3& o, F3& d) {
    i = k;
    o = mk3(__ldcs(rays + k), __ldcs(rays + stride + k), __ldcs(rays + 2 * stride + k));
    d = mk3(__ldcs(rays + 3 * stride + k), __ldcs(rays + 4 * stride + k), __ldcs(rays + 5 * stride + k));
  }
  PBRT_DEV float near() const { return __ldg(rays + 6 * stride + i); }
  PBRT_DEV float far() const { return __ldg(rays + 7 * stride + i); }
  PBRT_DEV const SceneView& scene() const { return s; }
  PBRT_DEV void store(bool have, float t, uint32_t leaf, uint32_t pr) {
    prim[i] = have ? pr : 0xFFFFFFFFu;
    tout[i] = have ? t : __int_as_float(0x7f800000);
    if (obj) obj[i] = have ? s.objects[leaf].desc_id : 0xFFFFFFFFu;
  }
  PBRT_DEV void store(bool occluded) { occ[i] = occluded ? 1 : 0; }
};

// Nearest hit / occlusion per ray. The warps take their own chunks of 32 rays: nothing is shared
// between calls, and a captured call replays beside any other.
template <bool kAny, bool kObj, bool kCsg>
__global__ void __launch_bounds__(128, kObj ? 6 : 8) k_scene_rays(const __grid_constant__ SceneView s,
                                                                  const float* __restrict__ rays, uint64_t stride,
                                                                  uint64_t n, uint32_t* __restrict__ prim,
                                                                  float* __restrict__ tout, uint32_t* __restrict__ obj,
                                                                  uint8_t* __restrict__ occ, WalkSchedule ws,
                                                                  uint32_t* err) {
  PlaneRays job{s, rays, stride, prim, tout, obj, occ, 0};
  if constexpr (kAny)
    walk_any<kObj, kCsg>(job, walk_queue(nullptr, n), ws, err);
  else
    walk_nearest<kObj, kCsg>(job, walk_queue(nullptr, n), ws, err);
}

static unsigned grid_cap(uint64_t n, int threads, int sm_count, int per_sm) {
  const uint64_t want = (n + threads - 1) / threads;
  const uint64_t cap = uint64_t(sm_count) * per_sm;
  return unsigned(want < cap ? (want ? want : 1) : cap);
}

template <bool kAny>
static cudaError_t launch_scene_rays(const SceneView& s, const float* rays, uint64_t stride, uint64_t n, uint32_t* prim,
                                     float* t, uint32_t* obj, uint8_t* occ, uint32_t* err, int sm_count,
                                     cudaStream_t st) {
  const WalkSchedule ws = walk_schedule(s.has_objects != 0);
  const unsigned g = grid_cap(n, 128, sm_count, s.has_objects ? 6 : 8);
  if (s.has_csg)
    k_scene_rays<kAny, true, true><<<g, 128, 0, st>>>(s, rays, stride, n, prim, t, obj, occ, ws, err);
  else if (s.has_objects)
    k_scene_rays<kAny, true, false><<<g, 128, 0, st>>>(s, rays, stride, n, prim, t, obj, occ, ws, err);
  else
    k_scene_rays<kAny, false, false><<<g, 128, 0, st>>>(s, rays, stride, n, prim, t, obj, occ, ws, err);
  return cudaGetLastError();
}

cudaError_t launch_scene_closest(const SceneView& s, const float* rays, uint64_t stride, uint64_t n, uint32_t* prim,
                                 float* t, uint32_t* obj, unsigned long long* cnt, uint32_t* err, int sm_count,
                                 cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (!cnt) return launch_scene_rays<false>(s, rays, stride, n, prim, t, obj, nullptr, err, sm_count, st);
  k_scene_closest_counted<<<grid_cap(n, 128, sm_count, 32), 128, 0, st>>>(s, rays, stride, n, prim, t, obj, cnt, err);
  return cudaGetLastError();
}

cudaError_t launch_scene_any(const SceneView& s, const float* rays, uint64_t stride, uint64_t n, uint8_t* occ,
                             unsigned long long* cnt, uint32_t* err, int sm_count, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (!cnt) return launch_scene_rays<true>(s, rays, stride, n, nullptr, nullptr, nullptr, occ, err, sm_count, st);
  k_scene_any_counted<<<grid_cap(n, 128, sm_count, 32), 128, 0, st>>>(s, rays, stride, n, occ, cnt, err);
  return cudaGetLastError();
}

}  // namespace pbrt
