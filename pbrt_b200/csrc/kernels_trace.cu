// kernels_trace.cu — batched ray-cast kernels (nearest hit / any hit) over one mesh.
//
// Ray planes are read and results written with streaming cache hints (each byte is touched
// once), so L1/L2 stay dedicated to the tree and triangles, which every ray revisits.
//
// A pass over a batch (nearest hit or occlusion) runs in two stages:
//   1. the cull streams every ray once (four rays per thread), tests the root box, writes a
//      miss for every ray, and appends the rays that enter the root to a queue with one
//      atomicAdd per block, each with a 32-byte copy of the ray beside its index (when a
//      record buffer is given), so that stage 2 reads its rays coalesced instead of gathering
//      eight planes per ray;
//   2. k_mesh_walk: persistent warps over the queue, idle lanes refilled with ballot/popc and
//      one atomicAdd per warp; each iteration is one warp-voted step, a burst of wide nodes
//      or a leaf step. Each lane tests its triangles in the reference's order, so ids and t
//      stay bit-exact.
// k_mesh_closest (one thread per ray, the binary tree) is the instrumented form that counts
// the work.
#include <cfloat>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "kernels.hpp"
#include "mesh_bvh.hpp"
#include "tcgen05.cuh"
#include "trace_mesh.cuh"
#include "wide_bvh.cuh"

namespace pbrt {

template <bool kCount>
__global__ void __launch_bounds__(128) k_mesh_closest(MeshView m, const float* __restrict__ rays, uint64_t stride,
                                                      uint64_t n, uint32_t* __restrict__ prim, float* __restrict__ tout,
                                                      uint32_t* __restrict__ obj, unsigned long long* __restrict__ counters,
                                                      uint32_t* __restrict__ err) {
  const uint64_t step = uint64_t(gridDim.x) * blockDim.x;
  unsigned long long acc[3] = {0, 0, 0};
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += step) {
    const F3 o = mk3(__ldcs(rays + i), __ldcs(rays + stride + i), __ldcs(rays + 2 * stride + i));
    const F3 d = mk3(__ldcs(rays + 3 * stride + i), __ldcs(rays + 4 * stride + i), __ldcs(rays + 5 * stride + i));
    const float near = __ldcs(rays + 6 * stride + i), far = __ldcs(rays + 7 * stride + i);
    const PRay r = prepare_ray(o, d);
    TraceCounters c{0, 0, 0};
    float t;
    const uint32_t id = mesh_closest<kCount>(m, r, near, far, &t, &c, err);
    __stcs(prim + i, id);
    __stcs(tout + i, id == 0xFFFFFFFFu ? __int_as_float(0x7f800000) : t);
    if (obj) __stcs(obj + i, id == 0xFFFFFFFFu ? 0xFFFFFFFFu : 0u);
    if (kCount) {
      acc[0] += c.nodes_visited;
      acc[1] += c.box_tests;
      acc[2] += c.triangle_tests;
    }
  }
  if (kCount) {
    // Every lane reaches this point, so a full-warp reduction is safe.
    for (int k = 0; k < 3; ++k) {
      unsigned long long v = acc[k];
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if ((threadIdx.x & 31) == 0 && v) atomicAdd(&counters[k], v);
    }
  }
}

// Occlusion, one thread per ray on the binary nodes (PBRT_TRACE_KERNEL=simple).
__global__ void __launch_bounds__(128) k_mesh_any(MeshView m, const float* __restrict__ rays, uint64_t stride, uint64_t n,
                                                  uint8_t* __restrict__ occ, uint32_t* __restrict__ err) {
  const uint64_t step = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += step) {
    const F3 o = mk3(__ldcs(rays + i), __ldcs(rays + stride + i), __ldcs(rays + 2 * stride + i));
    const F3 d = mk3(__ldcs(rays + 3 * stride + i), __ldcs(rays + 4 * stride + i), __ldcs(rays + 5 * stride + i));
    const float near = __ldcs(rays + 6 * stride + i), far = __ldcs(rays + 7 * stride + i);
    const PRay r = prepare_ray(o, d);
    occ[i] = mesh_any(m, r, near, far, err) ? 1 : 0;
  }
}

// ---------------------------------------------------------------------------------------
// Stage 1: root-box cull and compaction.
// ---------------------------------------------------------------------------------------
constexpr int kCullThreads = 128;
constexpr int kCullRays = 4;  // rays per thread and iteration

// Whether a ray is handed to stage 2: it enters the root box and, for a nearest hit, is not
// dropped at its first pop for entry >= min_t = FLT_MAX (bvh.rs:462-472).
template <bool kAny>
PBRT_DEV bool enters_root(const float (&v)[8][kCullRays], int j, const float4& rlo, const float4& rhi) {
  float entry;
  const PRay r = prepare_ray(mk3(v[0][j], v[1][j], v[2][j]), mk3(v[3][j], v[4][j], v[5][j]));
  return box_hit(r, rlo, rhi, v[6][j], v[7][j], entry) && (kAny || entry < FLT_MAX);
}

// The same for ray i of the planes, whose miss answer is written.
template <bool kAny>
PBRT_DEV bool enters_root_of(const MeshView& m, const float* rays, uint64_t stride, uint64_t i, uint32_t* prim, float* tout,
                             uint32_t* obj) {
  const F3 o = mk3(__ldg(rays + i), __ldg(rays + stride + i), __ldg(rays + 2 * stride + i));
  const F3 d = mk3(__ldg(rays + 3 * stride + i), __ldg(rays + 4 * stride + i), __ldg(rays + 5 * stride + i));
  const float near = __ldg(rays + 6 * stride + i), far = __ldg(rays + 7 * stride + i);
  if (kAny) {
    reinterpret_cast<uint8_t*>(prim)[i] = 0;
  } else {
    __stcs(prim + i, 0xFFFFFFFFu);
    __stcs(tout + i, __int_as_float(0x7f800000));
    if (obj) __stcs(obj + i, 0xFFFFFFFFu);
  }
  float entry;
  return box_hit(prepare_ray(o, d), __ldg(&m.nodes[0]), __ldg(&m.nodes[1]), near, far, entry) &&
         (kAny || entry < FLT_MAX);
}

// The miss answer of rays i0 .. i0 + 3 (those below n); stage 2 overwrites the hits. For an
// any-hit pass `prim` holds the occlusion bytes.
template <bool kVec, bool kAny>
PBRT_DEV void write_misses(uint64_t i0, uint64_t n, uint32_t* prim, float* tout, uint32_t* obj) {
  const float inf = __int_as_float(0x7f800000);
  if (kAny) {
    uint8_t* occ = reinterpret_cast<uint8_t*>(prim);
    if (kVec && i0 + kCullRays <= n) {
      __stcs(reinterpret_cast<uint32_t*>(occ + i0), 0u);
    } else {
      for (int j = 0; j < kCullRays; ++j)
        if (i0 + j < n) __stcs(occ + i0 + j, uint8_t(0));
    }
  } else if (kVec && i0 + kCullRays <= n) {
    __stcs(reinterpret_cast<uint4*>(prim + i0), make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu));
    __stcs(reinterpret_cast<float4*>(tout + i0), make_float4(inf, inf, inf, inf));
    if (obj)
      __stcs(reinterpret_cast<uint4*>(obj + i0), make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu));
  } else {
    for (int j = 0; j < kCullRays; ++j)
      if (i0 + j < n) {
        __stcs(prim + i0 + j, 0xFFFFFFFFu);
        __stcs(tout + i0 + j, inf);
        if (obj) __stcs(obj + i0 + j, 0xFFFFFFFFu);
      }
  }
}

// Appends the block's survivors (bit j of `enter`: the thread's ray i0 + j) to the queue, in
// ray order within the block: a block-wide scan and one atomicAdd. Every thread of the block
// calls it; `buf` alternates between iterations.
PBRT_DEV void push_survivors(unsigned enter, const float (&v)[8][kCullRays], uint64_t i0, int buf,
                             uint32_t (&warp_off)[2][kCullThreads / 32], unsigned long long (&blk_base)[2],
                             uint32_t* queue, unsigned long long* queue_count, float4* rec) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t c = __popc(enter);
  uint32_t incl = c;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= unsigned(off)) incl += y;
  }
  if (lane == 31) warp_off[buf][warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0;
    for (int w = 0; w < kCullThreads / 32; ++w) {
      const uint32_t t = warp_off[buf][w];
      warp_off[buf][w] = run;
      run += t;
    }
    blk_base[buf] = run ? atomicAdd(queue_count, (unsigned long long)run) : 0ull;
  }
  __syncthreads();
  uint64_t pos = blk_base[buf] + warp_off[buf][warp] + (incl - c);
#pragma unroll
  for (int j = 0; j < kCullRays; ++j)
    if (enter & (1u << j)) {
      if (rec) {  // read back soon by stage 2: default caching, the planes stream past
        rec[2 * pos] = make_float4(v[0][j], v[1][j], v[2][j], v[6][j]);
        rec[2 * pos + 1] = make_float4(v[3][j], v[4][j], v[5][j], v[7][j]);
      }
      queue[pos] = uint32_t(i0 + j);
      ++pos;
    }
}

// The cull by direct loads: any alignment (kVec: every plane and output 16-byte aligned, the
// plane stride a multiple of 4, so a thread's four rays are one float4 per plane; only the
// allocation-free pass takes it, the others run k_cull_root_bulk then).
template <bool kVec, bool kAny>
__global__ void __launch_bounds__(kCullThreads) k_cull_root(MeshView m, const float* __restrict__ rays, uint64_t stride,
                                                            uint64_t n, uint32_t* __restrict__ prim,
                                                            float* __restrict__ tout, uint32_t* __restrict__ obj,
                                                            uint32_t* __restrict__ queue,
                                                            unsigned long long* __restrict__ queue_count,
                                                            float4* __restrict__ rec) {
  __shared__ uint32_t warp_off[2][kCullThreads / 32];
  __shared__ unsigned long long blk_base[2];
  const float4 rlo = __ldg(&m.nodes[0]);
  const float4 rhi = __ldg(&m.nodes[1]);
  const uint64_t per_iter = uint64_t(gridDim.x) * blockDim.x * kCullRays;
  const uint64_t iters = (n + per_iter - 1) / per_iter;  // uniform across the grid: __syncthreads is safe
  for (uint64_t it = 0; it < iters; ++it) {
    const uint64_t i0 = it * per_iter + (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * kCullRays;
    float v[8][kCullRays];
    if (kVec && i0 + kCullRays <= n) {
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const float4 q = __ldcs(reinterpret_cast<const float4*>(rays + p * stride + i0));
        v[p][0] = q.x; v[p][1] = q.y; v[p][2] = q.z; v[p][3] = q.w;
      }
    } else {
#pragma unroll
      for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int j = 0; j < kCullRays; ++j) v[p][j] = (i0 + j < n) ? __ldcs(rays + p * stride + i0 + j) : 0.f;
    }
    unsigned enter = 0;
#pragma unroll
    for (int j = 0; j < kCullRays; ++j)
      if (i0 + j < n && enters_root<kAny>(v, j, rlo, rhi)) enter |= 1u << j;
    write_misses<kVec, kAny>(i0, n, prim, tout, obj);
    push_survivors(enter, v, i0, int(it & 1), warp_off, blk_base, queue, queue_count, rec);
  }
}

// The cull with its rays staged through shared memory by bulk asynchronous copies (the plain
// cp.async.bulk, no tensor map, no multicast), double-buffered: while a block tests, scans and
// compacts one 512-ray chunk, the next chunk's eight plane segments (2 KB each) are already on
// their way. Same tests, compaction and records as k_cull_root; 0.8 % faster per 16M-ray step
// than direct 16-byte loads. Requires kVec's alignment (planes and outputs 16-byte aligned,
// stride a multiple of 4). The last, partial chunk is read directly. A copy wait that runs out
// of its budget sets kErrCopy.
constexpr uint32_t kBulkChunk = kCullThreads * kCullRays;  // rays per chunk
constexpr uint32_t kBulkPlaneBytes = kBulkChunk * 4;       // one plane's segment

template <bool kAny>
__global__ void __launch_bounds__(kCullThreads) k_cull_root_bulk(MeshView m, const float* __restrict__ rays,
                                                                 uint64_t stride, uint64_t n,
                                                                 uint32_t* __restrict__ prim, float* __restrict__ tout,
                                                                 uint32_t* __restrict__ obj, uint32_t* __restrict__ queue,
                                                                 unsigned long long* __restrict__ queue_count,
                                                                 float4* __restrict__ rec, uint32_t* __restrict__ err) {
  __shared__ __align__(128) float sbuf[2][8][kBulkChunk];  // 32 KB
  __shared__ __align__(8) uint64_t mbar[2];
  __shared__ uint32_t warp_off[2][kCullThreads / 32];
  __shared__ unsigned long long blk_base[2];
  const float4 rlo = __ldg(&m.nodes[0]);
  const float4 rhi = __ldg(&m.nodes[1]);
  const uint64_t full_chunks = n / kBulkChunk;  // chunks read by bulk copies
  const uint64_t chunks = (n + kBulkChunk - 1) / kBulkChunk;
  const uint64_t iters = (chunks + gridDim.x - 1) / gridDim.x;  // uniform across the grid
  // thread 0 starts chunk c's copies into buffer b (c < full_chunks)
  auto issue = [&](uint64_t c, int b) {
    tc::fence_smem_to_async();  // the buffer's previous contents were read by ordinary loads
    tc::mbar_arrive_expect_tx(&mbar[b], 8u * kBulkPlaneBytes);
#pragma unroll
    for (int p = 0; p < 8; ++p) tc::bulk_g2s(&sbuf[b][p][0], rays + p * stride + c * kBulkChunk, kBulkPlaneBytes, &mbar[b]);
  };
  if (threadIdx.x == 0) {
    tc::mbar_init(&mbar[0], 1);
    tc::mbar_init(&mbar[1], 1);
    if (uint64_t(blockIdx.x) < full_chunks) issue(blockIdx.x, 0);
  }
  __syncthreads();
  bool copies_ok = true;  // false after a wait ran out: this thread reads directly from then on
  for (uint64_t it = 0; it < iters; ++it) {
    const uint64_t c = uint64_t(blockIdx.x) + it * gridDim.x;
    const int b = int(it & 1);
    // The next chunk's copies go out now; its buffer was last read in the previous
    // iteration, before that iteration's barriers.
    if (threadIdx.x == 0 && c + gridDim.x < full_chunks) issue(c + gridDim.x, b ^ 1);
    const uint64_t i0 = c * kBulkChunk + uint64_t(threadIdx.x) * kCullRays;
    float v[8][kCullRays];
    // buffer b's (it >> 1)-th use: full chunks come first, so every earlier use was a copy
    if (c < full_chunks && copies_ok && !tc::mbar_wait(&mbar[b], uint32_t((it >> 1) & 1u))) {
      atomicOr(err, kErrCopy);
      copies_ok = false;
    }
    if (c < full_chunks && copies_ok) {
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const float4 q = *reinterpret_cast<const float4*>(&sbuf[b][p][threadIdx.x * kCullRays]);
        v[p][0] = q.x; v[p][1] = q.y; v[p][2] = q.z; v[p][3] = q.w;
      }
    } else {
#pragma unroll
      for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int j = 0; j < kCullRays; ++j) v[p][j] = (i0 + j < n) ? __ldcs(rays + p * stride + i0 + j) : 0.f;
    }
    unsigned enter = 0;
#pragma unroll
    for (int j = 0; j < kCullRays; ++j)
      if (i0 + j < n && enters_root<kAny>(v, j, rlo, rhi)) enter |= 1u << j;
    write_misses<true, kAny>(i0, n, prim, tout, obj);
    push_survivors(enter, v, i0, b, warp_off, blk_base, queue, queue_count, rec);
  }
}

// ---------------------------------------------------------------------------------------
// Stage 2: persistent traversal of the survivors.
// ---------------------------------------------------------------------------------------
// Resident 128-thread blocks per SM the traversal kernels are compiled for (the register cap
// follows: 8 -> 64 registers a thread).
#ifndef PBRT_TRAVERSAL_MIN_BLOCKS
#define PBRT_TRAVERSAL_MIN_BLOCKS 8
#endif

// Persistent warps over the survivors' queue, each lane walking the wide tree (wide_bvh.cuh).
// One warp-voted step per iteration: either a node step for the lanes standing on a wide node
// (up to `burst` nodes each, fewer when a lane reaches a leaf) or a leaf step for the lanes
// standing on a leaf, never both. A leaf step is taken once at least `leaf_min` lanes stand on
// a leaf (or no lane has interior work left); until then the lanes on a leaf wait and the
// others keep descending. Idle lanes are refilled from the queue (one atomicAdd per warp) once
// at least `refill_min` of them are idle (or all are). leaf_min and burst carry the schedule of
// the drained queue in their second byte. Each lane tests its triangles in the reference's
// order, so ids and t are unchanged.
// kFrom: the survivors' rays come from the records stage 1 wrote beside the queue, from the planes
// by the queue's indices, or (kPlanes: no scratch, for a stream under capture) from the planes of
// `n_planes` rays: warp w of W then culls its own chunks of 128, w, w + W, ..., into a queue of its
// own in shared memory. (16,777,216 rays, 327,680 triangles, nearest hits, recorded: 943 us; 1,419
// with a warp's rays tested as its lanes take them, 2,496 by k_mesh_few.) kAny: the
// first triangle hit ends a ray, `prim` holds the occlusion bytes. Rays outside the wide nodes'
// arithmetic walk m's binary nodes.
constexpr uint32_t kOwnChunk = 128;
enum RaySource : int { kRecords, kQueue, kPlanes };
template <int kFrom, bool kAny>
__global__ void __launch_bounds__(128, PBRT_TRAVERSAL_MIN_BLOCKS) k_mesh_walk(
    MeshView m, WideView w, const float* __restrict__ rays, uint64_t stride, const uint32_t* __restrict__ queue,
    const unsigned long long* __restrict__ queue_count, uint32_t* __restrict__ prim, float* __restrict__ tout,
    uint32_t* __restrict__ obj, unsigned long long* __restrict__ next_ray, uint32_t* __restrict__ err,
    const float4* __restrict__ rec, uint64_t n_planes, int leaf_min, int refill_min, int burst) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  const uint64_t n = kFrom == kPlanes ? n_planes : *queue_count;
  // kPlanes: the warp's queue, its length, and its next chunk
  __shared__ uint32_t own_queue[kFrom == kPlanes ? 4 : 1][kFrom == kPlanes ? kOwnChunk + 32 : 1];
  uint32_t* own = own_queue[kFrom == kPlanes ? threadIdx.x >> 5 : 0];
  uint32_t held = 0;
  uint64_t chunk = uint64_t(blockIdx.x) * 4u + (threadIdx.x >> 5);
  bool active = false, exhausted = false;  // exhausted is warp-uniform
  uint32_t idx = 0;
  WRay r;
  float near = 0.f, lim = 0.f;  // a nearest hit counts below lim, any hit up to it
  uint32_t best = 0xFFFFFFFFu, cur = 0, budget = 0;
  int sp = 0;
  WideStack stk;
  const uint32_t exact_root = binary_ref(__ldg(&m.nodes[0]), __ldg(&m.nodes[1]), 0u);

  for (;;) {
    // Refill the idle lanes: one atomicAdd per warp.
    const unsigned idle = __ballot_sync(0xffffffffu, !active);
    if (!exhausted && idle && (__popc(idle) >= refill_min || idle == 0xffffffffu)) {
      uint64_t k = __popc(idle & lt_mask);
      if (kFrom == kPlanes) {
        const uint32_t want = __popc(idle);
        for (; held < want && chunk * kOwnChunk < n; chunk += uint64_t(gridDim.x) * 4u) {
#pragma unroll 2
          for (uint32_t j = 0; j < kOwnChunk; j += 32u) {
            const uint64_t i = chunk * kOwnChunk + j + lane;
            const bool enters = i < n && enters_root_of<kAny>(m, rays, stride, i, prim, tout, obj);
            const unsigned in = __ballot_sync(0xffffffffu, enters);
            if (enters) own[held + __popc(in & lt_mask)] = uint32_t(i);
            held += __popc(in);
          }
        }
        __syncwarp();
        k = k < held ? uint64_t(own[held - 1u - uint32_t(k)]) : n;
        __syncwarp();
        held -= held < want ? held : want;
        exhausted = held == 0u && chunk * kOwnChunk >= n;
      } else {
        const int leader = __ffs(idle) - 1;
        unsigned long long base = 0;
        if (int(lane) == leader) base = atomicAdd(next_ray, (unsigned long long)__popc(idle));
        base = __shfl_sync(0xffffffffu, base, leader);
        exhausted = base + __popc(idle) >= n;
        k += base;
      }
      if (!active && k < n) {
        F3 o, d;
        float far;
        if (kFrom == kRecords) {  // the copy stage 1 wrote: consecutive lanes read consecutive records
          idx = __ldg(queue + k);
          const float4 a = __ldcs(rec + 2 * k), b = __ldcs(rec + 2 * k + 1);
          o = mk3(a.x, a.y, a.z);
          d = mk3(b.x, b.y, b.z);
          near = a.w;
          far = b.w;
        } else {
          const uint64_t i = kFrom == kPlanes ? k : uint64_t(__ldg(queue + k));
          o = mk3(__ldg(rays + i), __ldg(rays + stride + i), __ldg(rays + 2 * stride + i));
          d = mk3(__ldg(rays + 3 * stride + i), __ldg(rays + 4 * stride + i), __ldg(rays + 5 * stride + i));
          near = __ldg(rays + 6 * stride + i);
          far = __ldg(rays + 7 * stride + i);
          idx = uint32_t(i);
        }
        r = wide_ray(o, d, near, far, w.bounded);
        // a nearest hit: t <= far, and t < min_t (which starts at FLT_MAX, bvh.rs:459)
        lim = kAny ? far : fminf(FLT_MAX, next_up(far));
        best = 0xFFFFFFFFu;
        cur = r.exact ? exact_root : w.root;  // the root has been entered (bvh.rs:458-461)
        sp = 0;
        budget = m.node_count;
        active = true;
      }
    }
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (act == 0) {
      if (exhausted) break;
      continue;  // all idle and the queue not yet drained: the next iteration refills
    }
    const bool at_leaf = (cur & kLeafRef) != 0u;
    const unsigned on_leaf = __ballot_sync(0xffffffffu, active && at_leaf);
    const int lmin = exhausted ? (leaf_min >> 8) : (leaf_min & 255);
    const bool leaf_step = __popc(on_leaf) >= lmin || on_leaf == act;
    if (active && at_leaf == leaf_step) {
      if (leaf_step) {
        uint32_t first, count;
        if (r.exact) {
          const uint32_t node = cur & ~kLeafRef;
          first = __float_as_uint(__ldg(&m.nodes[2 * size_t(node)]).w);
          count = __float_as_uint(__ldg(&m.nodes[2 * size_t(node) + 1]).w);
        } else {
          triangle_range(w, cur, first, count);
        }
        const float4* tri = r.exact ? m.tri : w.tri;
        const float2* tri_c = r.exact ? m.tri_c : w.tri_c;
        bool done = false;
        if (kAny) {  // (the grid's boxes are wider than a leaf's own)
          float e;
          done = blocking_triangle(tri, tri_c, first, count, r.o, r.d, near, lim) &&
                 (r.exact || (leaf_hit(w.nodes + 2 * size_t(__ldg(&w.leaf[first]).x), r, near, e) && e <= lim));
        } else {
          float t;
          uint32_t id;
          if (nearest_triangle(tri, tri_c, first, count, r.o, r.d, near, lim, t, id) && t < lim) {
            lim = t;
            best = id;
          }
        }
        if (done) {
          best = 0u;
          cur = 0u;
        } else {
          cur = kAny ? wide_pop_any(stk, sp) : wide_pop(stk, sp, lim);
        }
      } else {
        // up to `burst` nodes before the next vote (fewer when a leaf is reached)
        const int nb = exhausted ? (burst >> 8) : (burst & 255);
        for (int b = 0; b < nb && cur != 0u && !(cur & kLeafRef); ++b) {
          if (budget-- == 0) {
            atomicOr(err, kErrBudget);
            cur = 0u;
            break;
          }
          cur = r.exact ? binary_step<kAny>(m.nodes, cur, r, near, lim, stk, sp)
                : kAny  ? wide_step_any(w.wide + cur, r, near, lim, stk, sp)
                        : wide_step(w.exact + cur, r, near, lim, stk, sp);
        }
      }
      if (cur == 0u) {
        if (best != 0xFFFFFFFFu) {  // the miss answer has been written
          if (kAny) {
            reinterpret_cast<uint8_t*>(prim)[idx] = 1;
          } else {
            __stcs(prim + idx, best);
            __stcs(tout + idx, lim);
            if (obj) __stcs(obj + idx, 0u);
          }
        }
        active = false;
      }
    }
  }
}

// Few rays, one launch and no scratch: `lanes` rays to a warp, each through the root test and its
// own walk of the wide tree. The answers are the two stages' (see k_mesh_walk). What bounds a
// small call is the launches and a ray's own chain of node loads, not the lanes left idle: 4,099
// device rays against 20,480 triangles take 40 us a call so, 61 with a memset and two kernels.
template <bool kAny>
__global__ void __launch_bounds__(128) k_mesh_few(MeshView m, WideView w, const float* __restrict__ rays,
                                                  uint64_t stride, uint64_t n, uint32_t* __restrict__ prim,
                                                  float* __restrict__ tout, uint32_t* __restrict__ obj,
                                                  uint32_t* __restrict__ err, uint32_t lanes) {
  const uint32_t lane = threadIdx.x & 31u;
  if (lane >= lanes) return;
  const float4 rlo = __ldg(&m.nodes[0]), rhi = __ldg(&m.nodes[1]);
  const uint64_t warps = uint64_t(gridDim.x) * (blockDim.x / 32u);
  for (uint64_t i = (blockIdx.x * uint64_t(blockDim.x / 32u) + threadIdx.x / 32u) * lanes + lane; i < n;
       i += warps * lanes) {
    const F3 o = mk3(__ldcs(rays + i), __ldcs(rays + stride + i), __ldcs(rays + 2 * stride + i));
    const F3 d = mk3(__ldcs(rays + 3 * stride + i), __ldcs(rays + 4 * stride + i), __ldcs(rays + 5 * stride + i));
    const float near = __ldcs(rays + 6 * stride + i), far = __ldcs(rays + 7 * stride + i);
    const PRay pr = prepare_ray(o, d);
    uint32_t best = 0xFFFFFFFFu;
    float t = 0.f, entry;
    if (box_hit(pr, rlo, rhi, near, far, entry) && (kAny || entry < FLT_MAX)) {
      const WRay r = wide_ray(o, d, near, far, w.bounded);
      float lim = kAny ? far : fminf(FLT_MAX, next_up(far));
      uint32_t cur = r.exact ? 0u : w.root, budget = m.node_count;
      int sp = 0;
      WideStack stk;
      while (cur != 0u) {
        while (cur != 0u && !(cur & kLeafRef)) {
          if (budget-- == 0u) {
            atomicOr(err, kErrBudget);
            cur = 0u;
            break;
          }
          cur = kAny ? wide_step_any(w.wide + cur, r, near, lim, stk, sp)
                     : wide_step(w.exact + cur, r, near, lim, stk, sp);
        }
        if (cur == 0u) break;
        uint32_t first, count, id;
        triangle_range(w, cur, first, count);
        if (kAny) {
          float e;
          if (blocking_triangle(w.tri, w.tri_c, first, count, o, d, near, lim) &&
              leaf_hit(w.nodes + 2 * size_t(__ldg(&w.leaf[first]).x), r, near, e) && e <= lim) {
            best = 0u;
            break;
          }
        } else if (nearest_triangle(w.tri, w.tri_c, first, count, o, d, near, lim, t, id) && t < lim) {
          lim = t;
          best = id;
        }
        cur = kAny ? wide_pop_any(stk, sp) : wide_pop(stk, sp, lim);
      }
      t = lim;
      if (r.exact) {
        TraceCounters c{0, 0, 0};
        best = kAny ? (mesh_any(m, pr, near, far, err) ? 0u : 0xFFFFFFFFu)
                    : mesh_closest<false>(m, pr, near, far, &t, &c, err);
      }
    }
    if (kAny) {
      reinterpret_cast<uint8_t*>(prim)[i] = best == 0u ? 1 : 0;
    } else {
      prim[i] = best;
      tout[i] = best == 0xFFFFFFFFu ? __int_as_float(0x7f800000) : t;
      if (obj) obj[i] = best == 0xFFFFFFFFu ? 0xFFFFFFFFu : 0u;
    }
  }
}

// The wide nodes of a tree: one thread per node of the binary tree; those of every second level write
// the wide node of their grandchildren. A mesh's leaves become triangle references and note their
// node and object beside their first triangle; a top-level tree's leaves become their primitive's
// reference (`slot_ref`: the root of a merged mesh, or an object leaf) and note their node beside the
// slot.
__global__ void k_widen(WidenArgs a) {
  auto ref_of = [&](uint32_t q) -> uint32_t {
    const uint32_t first = __float_as_uint(__ldg(&a.nodes[2 * size_t(q)]).w);
    const uint32_t count = __float_as_uint(__ldg(&a.nodes[2 * size_t(q) + 1]).w);
    if (count == 0u) return a.wide_base + __ldg(&a.wide_id[q]);
    return a.slot_ref ? __ldg(&a.slot_ref[first]) : triangle_ref(a.tri_base + first, count, a.direct);
  };
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.count; i += gridDim.x * blockDim.x) {
    if (i == 1u) continue;  // the padding slot
    const float4 nlo = __ldg(&a.nodes[2 * size_t(i)]), nhi = __ldg(&a.nodes[2 * size_t(i) + 1]);
    const uint32_t pair = __float_as_uint(nlo.w);
    if (__float_as_uint(nhi.w) != 0u) {
      if (a.slot_ref) a.slot_node[pair] = i;
      else a.leaf[a.tri_base + pair] = make_uint2(a.node_base + i, a.owner);
      continue;
    }
    const uint32_t id = __ldg(&a.wide_id[i]);
    if (id == kNoWide) continue;
    uint32_t slot[4], ref[4];  // the slots' nodes; a leaf child stands in slot 0 (2), slot 1 (3) is empty
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const uint32_t c = pair + side;
      const uint32_t cl = __float_as_uint(__ldg(&a.nodes[2 * size_t(c)]).w);
      const bool leaf = __float_as_uint(__ldg(&a.nodes[2 * size_t(c) + 1]).w) != 0u;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int k = 2 * side + g;
        slot[k] = leaf ? c : cl + g;
        ref[k] = leaf && g == 1 ? 0u : ref_of(slot[k]);
      }
    }
    WideNode w;
    ExactNode x4;
    uint32_t pl[3] = {0u, 0u, 0u}, ph[3] = {0u, 0u, 0u};
    const float blo[3] = {nlo.x, nlo.y, nlo.z}, bhi[3] = {nhi.x, nhi.y, nhi.z};
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      // 255 steps span the node (a step of at least 2^-70; beyond kWideLimit: never walked), so
      // that a plane on the node's own faces stands on the grid: the flat boxes of a room's walls
      // stay flat
      const double extent = double(bhi[x]) - double(blo[x]);
      float step = float(fmin(fmax(extent / 255.0, 0x1p-70), 0x1p100));
      if (double(step) * 255.0 < extent) step = nextafterf(step, FLT_MAX);
      const double s = double(step);
      w.org[x] = blo[x];
      w.step[x] = step * 0x1p-8f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 lo = __ldg(&a.nodes[2 * size_t(slot[k])]), hi = __ldg(&a.nodes[2 * size_t(slot[k]) + 1]);
        const float l = x == 0 ? lo.x : (x == 1 ? lo.y : lo.z), h = x == 0 ? hi.x : (x == 1 ? hi.y : hi.z);
        (x == 0 ? x4.lo_x : (x == 1 ? x4.lo_y : x4.lo_z))[k] = l;
        (x == 0 ? x4.hi_x : (x == 1 ? x4.hi_y : x4.hi_z))[k] = h;
        // (within a thousandth of a step a plane snaps to the grid, inwards too: the walk's margin
        // of a 256th of a step covers it)
        const double fl = floor((double(l) - double(blo[x])) / s + 1e-3);
        const double fh = ceil((double(h) - double(blo[x])) / s - 1e-3);
        const uint32_t ql = uint32_t(fmin(fmax(fl, 0.0), 255.0)), qh = uint32_t(fmin(fmax(fh, 0.0), 255.0));
        pl[x] |= ql << (8 * k);
        ph[x] |= qh << (8 * k);
      }
    }
    w.lo_x = pl[0]; w.lo_y = pl[1]; w.lo_z = pl[2];
    w.hi_x = ph[0]; w.hi_y = ph[1]; w.hi_z = ph[2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      w.ref[k] = x4.ref[k] = ref[k];
      x4.pad[k] = 0u;
    }
    a.wide[a.wide_base + id] = w;
    a.exact[a.wide_base + id] = x4;
  }
}

// The persistent traversal's schedule. Once the queue is drained no refill can come, and a
// lane waiting on a leaf only lengthens the launch's tail: there a leaf step is taken as soon
// as one lane stands on a leaf. PBRT_TRACE_SCHEDULE="leaf_min,refill_min[,burst[,tail_leaf_min
// [,tail_burst]]]" (each in 1..32; without tail values the bulk's apply) overrides it for
// measurements; results do not depend on it.
struct TraversalSchedule {
  int leaf_min = 12, refill_min = 12, burst = 4;
  int tail_leaf_min = 1, tail_burst = 4;  // once the queue is drained (no refill can come)
  int leaf_arg() const { return leaf_min | (tail_leaf_min << 8); }
  int burst_arg() const { return burst | (tail_burst << 8); }
};

static TraversalSchedule traversal_schedule() {
  static const TraversalSchedule v = [] {
    TraversalSchedule d;
    if (const char* e = std::getenv("PBRT_TRACE_SCHEDULE")) {
      int a = 0, b = 0, c = 1, ta = 0, tc = 0;
      const int got = std::sscanf(e, "%d,%d,%d,%d,%d", &a, &b, &c, &ta, &tc);
      if (got >= 2 && a >= 1 && a <= 32 && b >= 1 && b <= 32 && c >= 1 && c <= 32) {
        d.leaf_min = a;
        d.refill_min = b;
        d.burst = got >= 3 ? c : 1;
        d.tail_leaf_min = got >= 4 && ta >= 1 && ta <= 32 ? ta : d.leaf_min;
        d.tail_burst = got >= 5 && tc >= 1 && tc <= 32 ? tc : d.burst;
      }
    }
    return d;
  }();
  return v;
}

static unsigned grid_for(uint64_t n, int threads, int sm_count) {
  const uint64_t want = (n + threads - 1) / threads;
  const uint64_t cap = uint64_t(sm_count) * 64;  // grid-stride beyond this
  return unsigned(want < cap ? (want ? want : 1) : cap);
}

cudaError_t launch_widen(const WidenArgs& a, int sm_count, cudaStream_t s) {
  if (a.count == 0) return cudaSuccess;
  k_widen<<<grid_for(a.count, 128, sm_count), 128, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_mesh_closest(const MeshView& m, const float* rays, uint64_t stride, uint64_t n, uint32_t* prim,
                                float* t, uint32_t* obj, unsigned long long* counters, uint32_t* err, int sm_count,
                                cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const unsigned g = grid_for(n, 128, sm_count);
  if (counters)
    k_mesh_closest<true><<<g, 128, 0, s>>>(m, rays, stride, n, prim, t, obj, counters, err);
  else
    k_mesh_closest<false><<<g, 128, 0, s>>>(m, rays, stride, n, prim, t, obj, nullptr, err);
  return cudaGetLastError();
}

static bool aligned(const void* p, uintptr_t a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; }

// Resident 128-thread blocks per SM of the persistent traversal (the same on every B200);
// computed once, thread-safely, by the first launch.
template <int kFrom, bool kAny>
static int walk_blocks_per_sm() {
  static const int v = [] {
    int b = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_mesh_walk<kFrom, kAny>, 128, 0);
    return e == cudaSuccess && b > 0 ? b : 4;
  }();
  return v;
}

// The walk over the survivors of n rays (kPlanes: over all of them).
template <int kFrom, bool kAny>
static cudaError_t walk(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                        uint32_t* prim, float* t, uint32_t* obj, const uint32_t* queue, unsigned long long* counters,
                        uint32_t* err, int sm_count, cudaStream_t s, const float4* rec) {
  const uint64_t full = uint64_t(sm_count) * walk_blocks_per_sm<kFrom, kAny>();
  const uint64_t need = (n + 127) / 128;
  const TraversalSchedule ts = traversal_schedule();
  k_mesh_walk<kFrom, kAny><<<unsigned(need < full ? need : full), 128, 0, s>>>(
      m, w, rays, stride, queue, counters, prim, t, obj, counters + 1, err, rec, n, ts.leaf_arg(), ts.refill_min,
      ts.burst_arg());
  return cudaGetLastError();
}

// The two stages over n rays; kAny: `prim` is the occlusion buffer, t and obj are NULL.
template <bool kRec, bool kAny>
static cudaError_t two_stage(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n, uint32_t* prim, float* t,
                             uint32_t* obj, uint32_t* queue, unsigned long long* counters, uint32_t* err, int sm_count,
                             cudaStream_t s, float4* rec) {
  const bool vec = stride % 4 == 0 && aligned(rays, 16) &&
                   (kAny ? aligned(prim, 4) : aligned(prim, 16) && aligned(t, 16) && (!obj || aligned(obj, 16)));
  const uint64_t chunks = (n + kBulkChunk - 1) / kBulkChunk;
  if (vec && kRec) {
    static const int bulk_per_sm = [] {
      int b = 0;
      const cudaError_t oe =
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_cull_root_bulk<kAny>, kCullThreads, 0);
      return oe == cudaSuccess && b > 0 ? b : 4;
    }();
    const uint64_t cap = uint64_t(sm_count) * bulk_per_sm;
    k_cull_root_bulk<kAny><<<unsigned(chunks < cap ? chunks : cap), kCullThreads, 0, s>>>(
        m, rays, stride, n, prim, t, obj, queue, counters, rec, err);
  } else {
    const uint64_t cap = uint64_t(sm_count) * 16;
    const unsigned g = unsigned(chunks < cap ? chunks : cap);
    if (vec)
      k_cull_root<true, kAny><<<g, kCullThreads, 0, s>>>(m, rays, stride, n, prim, t, obj, queue, counters, rec);
    else
      k_cull_root<false, kAny><<<g, kCullThreads, 0, s>>>(m, rays, stride, n, prim, t, obj, queue, counters, rec);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return walk<kRec ? kRecords : kQueue, kAny>(m, w, rays, stride, n, prim, t, obj, queue, counters, err, sm_count, s, rec);
}

cudaError_t launch_mesh_closest_persistent(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                           uint32_t* prim, float* t, uint32_t* obj, uint32_t* queue,
                                           unsigned long long* counters, uint32_t* err, int sm_count, cudaStream_t s,
                                           float4* rec) {
  if (n == 0) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(counters, 0, 2 * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  return two_stage<true, false>(m, w, rays, stride, n, prim, t, obj, queue, counters, err, sm_count, s, rec);
}

cudaError_t launch_mesh_any_persistent(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n, uint8_t* occ,
                                       uint32_t* queue, unsigned long long* counters, uint32_t* err, int sm_count,
                                       cudaStream_t s, float4* rec) {
  if (n == 0) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(counters, 0, 2 * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  return two_stage<true, true>(m, w, rays, stride, n, reinterpret_cast<uint32_t*>(occ), nullptr, nullptr, queue, counters,
                               err, sm_count, s, rec);
}

// Rays per warp of k_mesh_few: 8 (a 32-byte sector of each plane) while the GPU has room for the
// warps, more for more rays.
static uint32_t few_lanes(uint64_t n, int sm_count) {
  uint32_t lanes = 8;
  while (lanes < 32 && n > uint64_t(sm_count) * 32u * lanes) lanes *= 2;
  return lanes;
}
template <bool kAny>
static cudaError_t launch_few(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                              uint32_t* prim, float* t, uint32_t* obj, uint32_t* err, int sm_count, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const uint32_t lanes = few_lanes(n, sm_count);
  k_mesh_few<kAny><<<grid_for(n, int(4 * lanes), sm_count), 128, 0, s>>>(m, w, rays, stride, n, prim, t, obj, err, lanes);
  return cudaGetLastError();
}

cudaError_t launch_mesh_closest_planes(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                       uint32_t* prim, float* t, uint32_t* obj, uint32_t* err, int sm_count,
                                       cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  return walk<kPlanes, false>(m, w, rays, stride, n, prim, t, obj, nullptr, nullptr, err, sm_count, s, nullptr);
}

cudaError_t launch_mesh_any_planes(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                   uint8_t* occ, uint32_t* err, int sm_count, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  return walk<kPlanes, true>(m, w, rays, stride, n, reinterpret_cast<uint32_t*>(occ), nullptr, nullptr, nullptr, nullptr, err,
                             sm_count, s, nullptr);
}

cudaError_t launch_mesh_closest_few(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                    uint32_t* prim, float* t, uint32_t* obj, uint32_t* err, int sm_count,
                                    cudaStream_t s) {
  return launch_few<false>(m, w, rays, stride, n, prim, t, obj, err, sm_count, s);
}

cudaError_t launch_mesh_any_few(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                uint8_t* occ, uint32_t* err, int sm_count, cudaStream_t s) {
  return launch_few<true>(m, w, rays, stride, n, reinterpret_cast<uint32_t*>(occ), nullptr, nullptr, err, sm_count, s);
}

// ---------------------------------------------------------------------------------------
// Allocation-free variant of the two-stage nearest-hit pass.
//
// Its scratch (the two 64-bit counters, the device error word and the survivor queue) is
// this file-scope array instead of memory the context allocates: 256 header bytes plus
// kNoAllocMaxRays queue entries, i.e. 4 MiB + 256 B that every GPU which loads the library
// holds until the process exits. Header layout in 32-bit words: [0..1] queue length,
// [2..3] fetch position, [4] error word; the queue starts at word 64.
// ---------------------------------------------------------------------------------------
static __device__ __align__(256) uint32_t g_noalloc_scratch[64 + kNoAllocMaxRays];

// Device address of g_noalloc_scratch on the current device (host code cannot use the
// symbol itself as a device address). The context looks it up when it is created, with its
// device current, and keeps it: a context made after a device reset gets the new address.
cudaError_t noalloc_scratch_lookup(uint32_t** out) {
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return e;
  *out = static_cast<uint32_t*>(p);
  return cudaSuccess;
}

cudaError_t launch_mesh_closest_noalloc(const MeshView& m, const WideView& w, const float* rays, uint64_t n, uint32_t* prim, float* t,
                                        uint32_t* scratch, int sm_count, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (n > kNoAllocMaxRays || !scratch) return cudaErrorInvalidValue;
  // The array keeps the previous call's contents: the counters and the error word must
  // start at zero; the queue is written before it is read.
  cudaError_t e = cudaMemsetAsync(scratch, 0, 64 * sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  unsigned long long* counters = reinterpret_cast<unsigned long long*>(scratch);
  uint32_t* err = scratch + 4;
  uint32_t* queue = scratch + 64;
  return two_stage<false, false>(m, w, rays, n, n, prim, t, nullptr, queue, counters, err, sm_count, s, nullptr);
}

cudaError_t launch_mesh_any(const MeshView& m, const float* rays, uint64_t stride, uint64_t n, uint8_t* occ,
                            uint32_t* err, int sm_count, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_mesh_any<<<grid_for(n, 128, sm_count), 128, 0, s>>>(m, rays, stride, n, occ, err);
  return cudaGetLastError();
}

}  // namespace pbrt
