// scene_walk.cuh — Scene::find_nearest and Scene::any_hit for many rays: persistent warps over
// the scene's wide tree (wide_bvh.cuh).
//
// Each lane walks one ray; idle lanes take the next rays once `refill_min` of a warp's lanes are
// idle (or all are). Each iteration is one warp-voted step: up to `burst` wide nodes for the
// lanes standing on one or, once `leaf_min` lanes stand on a leaf (or no lane has a node to
// visit), a leaf for those. Once the warp can take no more rays an iteration is both, the leaf
// first: a lane that waits then only lengthens the launch. One thread per ray left 3-5 of 32 lanes
// active per instruction on the torus-knot and 10,000-sphere renders and 10 on a closed box; and a
// mesh answered in a kernel of its own, or a per-object query inside the top-level walk, repeated
// the set-up of every ray for every object.
//
// A Job names the rays:
//   void load(k, o, d): fetches ray k into the lane
//   float near(), far(): its interval (read again where needed rather than held in registers)
//   const SceneView& scene(): the lane's scene
//   void store(...): the lane's answer
#pragma once

#include "scene_device.cuh"

namespace pbrt {

struct WalkSchedule {
  int leaf_min, refill_min, burst;
};

// The rays a warp takes: from a shared counter, or (fetch NULL: no memory to share, as for a
// stream under capture) its own chunks of 32, warp w of W taking chunks w, w + W, ... When the
// grid has a lane for every ray a warp takes rays once; and 8 to 16 of them instead of 32 when
// they are few (up to half the grid's lanes): the launch then lasts as long as its slowest warp,
// and a warp as long as its lanes' different paths one after another. Frames of a torus knot of
// 164,000 triangles (81x431, 3 samples, depth 19; 948x110, 2 samples, depth 12) took 2.35 and 1.99 ms
// with 32, 2.09 and 1.75 with 8 at least; between half and all of the lanes 32 was faster.
struct WalkQueue {
  uint32_t* fetch;
  uint64_t n, own;  // own: rays this warp has taken (fetch NULL)
  uint32_t per;     // rays a warp takes when it takes once, else 0
  bool drained;     // warp-uniform
};

PBRT_DEV WalkQueue walk_queue(uint32_t* fetch, uint64_t n) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  uint32_t per = 0;
  if (n <= uint64_t(warps) * 16u) {
    per = uint32_t((n + warps - 1) / warps);
    per = per < 8u ? 8u : per;
  } else if (n <= uint64_t(warps) * 32u) {
    per = 32u;
  }
  return WalkQueue{fetch, n, 0, per, false};
}

// The ray of each idle lane, n or beyond when there is none left; every lane of the warp calls it.
PBRT_DEV uint64_t walk_take(WalkQueue& q, unsigned idle) {
  const unsigned lane = threadIdx.x & 31u, before = __popc(idle & ((1u << lane) - 1u)), want = __popc(idle);
  const uint64_t warps = uint64_t(gridDim.x) * (blockDim.x >> 5);
  const uint64_t w = uint64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (q.per) {
    q.drained = true;
    return before < q.per ? w * q.per + before : q.n;
  }
  if (q.fetch) {
    const int leader = __ffs(idle) - 1;
    uint32_t base = 0;
    if (int(lane) == leader) base = atomicAdd(q.fetch, want);
    base = __shfl_sync(0xffffffffu, base, leader);
    q.drained = uint64_t(base) + want >= q.n;
    return uint64_t(base) + before;
  }
  const uint64_t k = q.own + before;
  q.own += want;
  q.drained = ((q.own >> 5) * warps + w) * 32u >= q.n;  // its next chunk starts beyond the end
  return ((k >> 5) * warps + w) * 32u + (k & 31u);
}

// The exact queries, for rays the wide walk does not cover; calls, so that their stacks and
// registers are not the walk's (one per kernel: ptxas fails on a function shared by kernels of
// different register bounds).
template <class Job, bool kObj, bool kCsg, bool kEach>
__device__ __noinline__ bool exact_nearest(const SceneView& s, F3 o, F3 d, float near, float far, float& t,
                                           uint32_t& leaf, uint32_t& prim, uint32_t* err) {
  return scene_closest<kCsg>(s, o, d, near, far, t, leaf, prim, err);
}
template <class Job, bool kObj, bool kCsg, bool kEach>
__device__ __noinline__ bool exact_any(const SceneView& s, F3 o, F3 d, float near, float far, uint32_t* err) {
  return scene_any<kCsg>(s, o, d, near, far, err);
}

// The nearest hit of a walk so far: `t` is the ray's far end before there is one.
struct Nearest {
  float t;
  bool have;
};

// ---- a leaf ---------------------------------------------------------------------------------------
// The nearest hit of the leaf `cur`, whose slot is entered at `e`, adopted when it is nearer than the
// best so far, as scene_closest_t does. Slots are entered up to and including best.t, as a mesh's own
// boxes are; an object is asked when its box is entered below best.t only. A merged mesh's leaf
// entered at exactly best.t is asked or not as the box of the whole mesh has it: true, the ray must be
// answered by the exact query.
template <bool kObj, bool kCsg>
PBRT_DEV bool nearest_in_leaf(const SceneView& s, const WRay& r, float near, uint32_t cur, float e, Nearest& best,
                              uint32_t& leaf, uint32_t& prim, uint32_t* err) {
  float t;
  uint32_t lf = 0, pr = 0;
  if (kObj && (cur & kObjectRef)) {
    if (!(e < best.t) || !prim_closest<kCsg>(s, __ldg(&s.order[cur & 0x3FFFFFFFu]), r.o, r.d, near, best.t, t, lf, pr, err) ||
        (best.have && !(t < best.t)))
      return false;
  } else {
    uint32_t first, count;
    triangle_range(s.wide, cur, first, count);
    // (a mesh's own search starts at FLT_MAX, bvh.rs:459: its hits lie below that)
    if (!nearest_triangle(s.wide.tri, s.wide.tri_c, first, count, r.o, r.d, near, fminf(best.t, 0x1.fffffcp127f), t, pr) ||
        (best.have && !(t < best.t)))
      return false;
    const uint2 info = __ldg(&s.wide.leaf[first]);
    // (the slot of a mesh of one leaf is its top-level box: the leaf's own is asked)
    if (!leaf_hit(s.wide.nodes + 2 * size_t(info.x), r, near, e) || e > best.t) return false;
    if (e == best.t) return true;
    lf = info.y;
  }
  best = Nearest{t, true};
  leaf = lf;
  prim = pr;
  return false;
}

// Whether the leaf `cur` blocks the ray.
template <bool kObj, bool kCsg>
PBRT_DEV bool blocked_in_leaf(const SceneView& s, const WRay& r, float near, float far, uint32_t cur, uint32_t* err) {
  const float4* node = nullptr;
  if (kObj && (cur & kObjectRef)) {
    const uint32_t slot = cur & 0x3FFFFFFFu;
    if (prim_any<kCsg>(s, __ldg(&s.order[slot]), r.o, r.d, near, far, err))
      node = s.top + 2 * size_t(__ldg(&s.wide.slot_node[slot]));
  } else {
    uint32_t first, count;
    triangle_range(s.wide, cur, first, count);
    if (blocking_triangle(s.wide.tri, s.wide.tri_c, first, count, r.o, r.d, near, far))
      node = s.wide.nodes + 2 * size_t(__ldg(&s.wide.leaf[first]).x);
  }
  float e;
  return node && leaf_hit(node, r, near, e) && e <= far;
}

// ---- many rays: persistent warps ----------------------------------------------------------------
// kObj: some primitive of some scene is not a mesh merged into its wide tree (kCsg: or is a
// constructive solid).
template <bool kObj, bool kCsg, class Job>
PBRT_DEV void walk_nearest(Job& job, WalkQueue q, WalkSchedule ws, uint32_t* err) {
  bool active = false;
  WRay r;
  Nearest best{0.f, false};
  uint32_t leaf = 0, prim = 0, cur = 0, budget = 0;
  float e = 0.f;  // the entry into the slot of `cur`
  int sp = 0;
  WideStack stk;
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, !active);
    if (!q.drained && idle && (__popc(idle) >= ws.refill_min || idle == 0xffffffffu)) {
      const uint64_t k = walk_take(q, idle);
      F3 o, d;
      if (!active && k < q.n) {
        job.load(k, o, d);
        const SceneView& s = job.scene();
        const float near = job.near(), far = job.far();
        r = wide_ray(o, d, near, far, s.wide.bounded);
        best = Nearest{far, false};
        if (kObj && !r.exact) {
          for (uint32_t u = 0; u < s.unbounded_count; ++u) {  // nearest_among + closer (scene.rs:222-249)
            float t;
            uint32_t lf, pr;
            if (prim_closest<kCsg>(s, __ldg(&s.unbounded[u]), o, d, near, far, t, lf, pr, err) &&
                (!best.have || t < best.t)) {
              best = Nearest{t, true};
              leaf = lf;
              prim = pr;
            }
          }
        }
        cur = s.wide.root;
        if (kObj && (cur & kObjectRef) && (cur & kLeafRef) && !leaf_hit(s.top, r, near, e)) cur = 0u;  // the only primitive
        sp = 0;
        budget = 4u * s.wide.count + 4u;  // every iteration visits a node or a leaf it has not visited
        active = true;
      }
    }
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (act == 0) {
      if (q.drained) break;
      continue;
    }
    const bool at_leaf = (cur & kLeafRef) != 0u;
    const unsigned on_leaf = __ballot_sync(0xffffffffu, active && at_leaf);
    const bool leaf_step = q.drained || __popc(on_leaf) >= ws.leaf_min || on_leaf == act;
    if (active && (q.drained || at_leaf == leaf_step || cur == 0u || r.exact)) {
      const SceneView& s = job.scene();
      const float near = job.near();
      bool restart = r.exact;
      if (leaf_step && at_leaf && !restart) {
        restart = nearest_in_leaf<kObj, kCsg>(s, r, near, cur, e, best, leaf, prim, err);
        cur = wide_pop(stk, sp, next_up(best.t), e);
      }
      if (!leaf_step || q.drained) {
        const float reach = next_up(best.t);
        for (int b = 0; b < ws.burst && cur != 0u && !(cur & kLeafRef); ++b)
          cur = wide_step(s.wide.exact + cur, r, near, reach, stk, sp, e);
        if (--budget == 0u) {
          atomicOr(err, kErrBudget);
          cur = 0u;
        }
      }
      if (restart) {
        float t = 0.f;
        best.have = exact_nearest<Job, kObj, kCsg, false>(s, r.o, r.d, near, job.far(), t, leaf, prim, err);
        best.t = t;
        cur = 0u;
      }
      if (cur == 0u) {
        job.store(best.have, best.t, leaf, prim);
        active = false;
      }
    }
  }
}

template <bool kObj, bool kCsg, class Job>
PBRT_DEV void walk_any(Job& job, WalkQueue q, WalkSchedule ws, uint32_t* err) {
  bool active = false;
  WRay r;
  float far = 0.f;
  uint32_t cur = 0, budget = 0;
  int sp = 0;
  WideStack stk;
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, !active);
    if (!q.drained && idle && (__popc(idle) >= ws.refill_min || idle == 0xffffffffu)) {
      const uint64_t k = walk_take(q, idle);
      F3 o, d;
      if (!active && k < q.n) {
        job.load(k, o, d);
        const SceneView& s = job.scene();
        const float near = job.near();
        far = job.far();
        r = wide_ray(o, d, near, far, s.wide.bounded);
        bool hit = false;
        if (kObj && !r.exact)
          for (uint32_t u = 0; u < s.unbounded_count && !hit; ++u)  // any_blocks (scene.rs:170-184)
            hit = prim_any<kCsg>(s, __ldg(&s.unbounded[u]), o, d, near, far, err);
        cur = s.wide.root;
        sp = 0;
        budget = 4u * s.wide.count + 4u;  // every iteration visits a node or a leaf it has not visited
        active = !hit;
        if (hit) job.store(true);
      }
    }
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (act == 0) {
      if (q.drained) break;
      continue;
    }
    const bool at_leaf = (cur & kLeafRef) != 0u;
    const unsigned on_leaf = __ballot_sync(0xffffffffu, active && at_leaf);
    const bool leaf_step = q.drained || __popc(on_leaf) >= ws.leaf_min || on_leaf == act;
    if (active && (q.drained || at_leaf == leaf_step || cur == 0u || r.exact)) {
      const SceneView& s = job.scene();
      const float near = job.near();
      bool hit = false;
      if (r.exact) {
        hit = exact_any<Job, kObj, kCsg, false>(s, r.o, r.d, near, far, err);
        cur = 0u;
      } else if (leaf_step && at_leaf) {
        hit = blocked_in_leaf<kObj, kCsg>(s, r, near, far, cur, err);
        cur = hit ? 0u : wide_pop_any(stk, sp);
      }
      if (!leaf_step || q.drained) {
        for (int b = 0; b < ws.burst && cur != 0u && !(cur & kLeafRef); ++b)
          cur = wide_step_any(s.wide.wide + cur, r, near, far, stk, sp);
        if (--budget == 0u) {
          atomicOr(err, kErrBudget);
          cur = 0u;
          hit = true;  // reported, the sample dropped
        }
      }
      if (cur == 0u) {
        job.store(hit);
        active = false;
      }
    }
  }
}

// ---- one thread per ray -------------------------------------------------------------------------
// For scenes of a few wide nodes, merged meshes only: their walks are too short for the votes and
// refills to pay.
template <class Job>
PBRT_DEV void each_nearest(Job& job, uint64_t n, uint32_t* err) {
  for (uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; k < n; k += uint64_t(gridDim.x) * blockDim.x) {
    F3 o, d;
    job.load(k, o, d);
    const SceneView& s = job.scene();
    const float near = job.near(), far = job.far();
    const WRay r = wide_ray(o, d, near, far, s.wide.bounded);
    Nearest best{far, false};
    uint32_t leaf = 0, prim = 0, cur = s.wide.root, budget = 4u * s.wide.count + 4u;
    int sp = 0;
    WideStack stk;
    bool restart = r.exact;
    while (cur != 0u && !restart) {
      const float reach = next_up(best.t);
      while (cur != 0u && !(cur & kLeafRef)) {
        cur = wide_step(s.wide.exact + cur, r, near, reach, stk, sp);
        if (--budget == 0u) {
          atomicOr(err, kErrBudget);
          cur = 0u;
        }
      }
      if (cur == 0u) break;
      restart = nearest_in_leaf<false, false>(s, r, near, cur, 0.f, best, leaf, prim, err);
      cur = wide_pop(stk, sp, next_up(best.t));
    }
    if (restart) {
      float t = 0.f;
      best.have = exact_nearest<Job, false, false, true>(s, r.o, r.d, near, job.far(), t, leaf, prim, err);
      best.t = t;
    }
    job.store(best.have, best.t, leaf, prim);
  }
}

template <class Job>
PBRT_DEV void each_any(Job& job, uint64_t n, uint32_t* err) {
  for (uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; k < n; k += uint64_t(gridDim.x) * blockDim.x) {
    F3 o, d;
    job.load(k, o, d);
    const SceneView& s = job.scene();
    const float near = job.near(), far = job.far();
    const WRay r = wide_ray(o, d, near, far, s.wide.bounded);
    uint32_t cur = s.wide.root, budget = 4u * s.wide.count + 4u;
    int sp = 0;
    WideStack stk;
    bool hit = false;
    if (r.exact) {
      hit = exact_any<Job, false, false, true>(s, r.o, r.d, near, far, err);
      cur = 0u;
    }
    while (cur != 0u && !hit) {
      while (cur != 0u && !(cur & kLeafRef)) {
        cur = wide_step_any(s.wide.wide + cur, r, near, far, stk, sp);
        if (--budget == 0u) {
          atomicOr(err, kErrBudget);
          cur = 0u;
          hit = true;  // reported, the sample dropped
        }
      }
      if (cur == 0u) break;
      hit = blocked_in_leaf<false, false>(s, r, near, far, cur, err);
      if (!hit) cur = wide_pop_any(stk, sp);
    }
    job.store(hit);
  }
}

}  // namespace pbrt
