// walk.cuh — what the wavefront's shading and walking kernels share: where a path's scene comes
// from, and the launchers of the walks (walk_kernels.cuh; one translation unit per source, so
// that they compile side by side).
#pragma once

#include "render.hpp"
#include "scene_device.cuh"

namespace pbrt {

constexpr float kShadowEps = 0.00001f;  // SHADOW_RAY_EPSILON (src/lights.rs:21)

// ---- where a path's scene comes from ------------------------------------------------------------
// The wavefront kernels are written once over a scene source: one scene passed as a kernel
// parameter (pbrt_render, the cached render), or the batch table indexed by the path's scene.
struct PathSettings {
  uint32_t max_depth, rr_start, integrator;  // integrator: 0 path, 1 naive, 2 normal
  float near, far;
};

// A cursor names a path's scene while a lane works on it.
struct OneScene {
  SceneView v;
  PathSettings ps;
  struct Cursor {};
  PBRT_DEV Cursor cursor(const WaveBuffers&, uint32_t) const { return {}; }
  PBRT_DEV const SceneView& view(const Cursor&) const { return v; }
  PBRT_DEV PathSettings settings(const Cursor&) const { return ps; }
};

struct ManyScenes {
  const BatchScene* b;
  struct Cursor {
    const BatchScene* e;
  };
  PBRT_DEV Cursor cursor(const WaveBuffers& w, uint32_t p) const { return {b + w.scene[p]}; }
  PBRT_DEV const SceneView& view(const Cursor& c) const { return c.e->view; }
  PBRT_DEV PathSettings settings(const Cursor& c) const {
    const BatchScene& e = *c.e;
    return PathSettings{e.max_depth, e.rr_start, e.integrator, e.cam.near, e.cam.far};
  }
};

struct WalkLaunch {
  bool objects, csg;  // some scene has primitives that are not merged meshes; constructive solids
  uint32_t nodes;     // wide nodes of the largest scene
  uint32_t paths;     // of the wave
  LaunchShape shape;
  unsigned long long* stats;
  uint32_t* err;
  int sm_count;
  cudaStream_t st;
};

// Scene::find_nearest for the paths of queue q (its length *qcount); `fetch` is a zeroed word.
// Zeroes the bounce's other counters: *next_count, the shadow queue's length and fetch position.
cudaError_t launch_nearest(const WaveBuffers& w, const OneScene& src, const uint32_t* q, const uint32_t* qcount,
                           uint32_t* fetch, uint32_t* next_count, const WalkLaunch& l);
cudaError_t launch_nearest(const WaveBuffers& w, const ManyScenes& src, const uint32_t* q, const uint32_t* qcount,
                           uint32_t* fetch, uint32_t* next_count, const WalkLaunch& l);
// Scene::any_hit for the shadow queue; unoccluded entries add their light sample.
cudaError_t launch_shadow(const WaveBuffers& w, const OneScene& src, uint32_t* fetch, const WalkLaunch& l);
cudaError_t launch_shadow(const WaveBuffers& w, const ManyScenes& src, uint32_t* fetch, const WalkLaunch& l);

}  // namespace pbrt
