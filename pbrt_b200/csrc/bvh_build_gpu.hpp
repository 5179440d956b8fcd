// bvh_build_gpu.hpp — a triangle mesh's BVH built on the GPU (bvh_build_gpu.cu): the same tree,
// triangle order and flattened layout as build_mesh_bvh (mesh_bvh.hpp), left in device memory.
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "mesh_bvh.hpp"

namespace pbrt {

struct DeviceMeshBuild {
  GpuNode* nodes = nullptr;     // node_slots records, GPU numbering (root 0, padding 1)
  uint64_t node_slots = 0;
  float4* tri = nullptr;        // the triangle streams of mesh_bvh.hpp, in leaf order
  float2* tri_c = nullptr;
  uint32_t* tri_index = nullptr;  // leaf order -> original triangle index
  float* v = nullptr;             // the mesh's own copy of its vertices and indices, for shading
  uint32_t* idx = nullptr;
  uint32_t* wide_id = nullptr;    // per node: its wide node (number_wide, in an order of its own)
  uint32_t wide_count = 0;
  MeshBuildStats stats;
  float bounds_min[3] = {0, 0, 0}, bounds_max[3] = {0, 0, 0};  // vertex bounds
};

// vertices (3 floats each) and indices (3 per triangle) in device memory of the current
// device; runs on `st` and returns when the build is complete (its memory comes from `pool`).
// On failure returns false with `err` set (bad input is reported, not read out of range).
bool build_mesh_bvh_device(const float* vertices, uint32_t vertex_count, const uint32_t* indices, uint32_t tri_count,
                           const MeshBuildParams& params, cudaStream_t st, cudaMemPool_t pool, int sm_count,
                           DeviceMeshBuild* out, std::string* err);
void free_device_mesh_build(DeviceMeshBuild* build);

}  // namespace pbrt
