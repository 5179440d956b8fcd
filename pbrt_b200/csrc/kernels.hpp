// kernels.hpp — host-side launchers of the device kernels (no device code here).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace pbrt {

struct MeshView;
struct WideView;
struct WideNode;
struct ExactNode;

// Ray buffers: eight planes (ox oy oz dx dy dz tmin tmax) of `stride` floats each, of which
// the first `n` are used.
cudaError_t launch_mesh_closest(const MeshView& m, const float* rays, uint64_t stride, uint64_t n, uint32_t* prim,
                                float* t, uint32_t* obj, unsigned long long* counters, uint32_t* err, int sm_count,
                                cudaStream_t s);
// Two-stage nearest hit: a streaming root-box cull that answers misses and compacts the
// survivors' indices into `queue` (scratch, capacity >= n, n < 2^32), then the persistent
// dynamic-fetch traversal over the queue. `counters` is two 64-bit words of scratch (queue
// length, fetch position), zeroed on `s` by the launcher. `rec` (scratch, 2 x n float4): the
// survivors' rays copied beside their queue entries, read back coalesced.
cudaError_t launch_mesh_closest_persistent(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                           uint32_t* prim, float* t, uint32_t* obj, uint32_t* queue,
                                           unsigned long long* counters, uint32_t* err, int sm_count, cudaStream_t s,
                                           float4* rec);
// The same two stages for occlusion.
cudaError_t launch_mesh_any_persistent(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n, uint8_t* occ,
                                       uint32_t* queue, unsigned long long* counters, uint32_t* err, int sm_count,
                                       cudaStream_t s, float4* rec);
// Both queries for many rays without scratch: one launch that tests the root itself (n <= 2^32).
cudaError_t launch_mesh_closest_planes(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                       uint32_t* prim, float* t, uint32_t* obj, uint32_t* err, int sm_count,
                                       cudaStream_t s);
cudaError_t launch_mesh_any_planes(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                   uint8_t* occ, uint32_t* err, int sm_count, cudaStream_t s);
// Both queries for few rays: one launch, no scratch; the rays and answers may be pinned host memory.
cudaError_t launch_mesh_closest_few(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                    uint32_t* prim, float* t, uint32_t* obj, uint32_t* err, int sm_count,
                                    cudaStream_t s);
cudaError_t launch_mesh_any_few(const MeshView& m, const WideView& w, const float* rays, uint64_t stride, uint64_t n,
                                uint8_t* occ, uint32_t* err, int sm_count, cudaStream_t s);
// One binary tree's part of a scene's wide tree (wide_bvh.cuh): a mesh's (slot_ref NULL), or the
// top level's: `wide_id` names each node's wide node (number_wide), from wide_base on.
struct WidenArgs {
  const float4* nodes;
  uint32_t count;
  WideNode* wide;
  ExactNode* exact;
  const uint32_t* wide_id;
  uint32_t wide_base;
  bool direct;
  uint32_t tri_base, node_base, owner;  // a mesh: its first triangle, first node and object in the scene's arrays
  uint2* leaf;
  const uint32_t* slot_ref;  // the top level: each primitive's reference
  uint32_t* slot_node;
};
cudaError_t launch_widen(const WidenArgs& a, int sm_count, cudaStream_t s);
// Allocation-free form of launch_mesh_closest_persistent for device buffers (plane stride
// = n): its scratch is a file-scope __device__ array of kNoAllocMaxRays queue entries
// shared by every call on a device. `scratch` is that array's device address on the current
// device, from noalloc_scratch_lookup (word 4 is the error word). cudaErrorInvalidValue when
// n > kNoAllocMaxRays. Calls that overlap on the GPU race.
constexpr uint64_t kNoAllocMaxRays = uint64_t(1) << 20;
cudaError_t launch_mesh_closest_noalloc(const MeshView& m, const WideView& w, const float* rays, uint64_t n, uint32_t* prim, float* t,
                                        uint32_t* scratch, int sm_count, cudaStream_t s);
// Device address of the allocation-free pass's scratch array on the current device. The
// lookup loads this file's module there (under lazy loading), which commits the array.
cudaError_t noalloc_scratch_lookup(uint32_t** scratch);
cudaError_t launch_mesh_any(const MeshView& m, const float* rays, uint64_t stride, uint64_t n, uint8_t* occ,
                            uint32_t* err, int sm_count, cudaStream_t s);

}  // namespace pbrt
