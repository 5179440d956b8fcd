// api.cu — implementation of the C ABI declared in include/pbrt_b200.h.
//
// Host responsibilities: validate descriptions, build acceleration structures, own device
// memory, pick the host- or device-buffer path, and turn device-side error flags into
// status codes. No computation of the hot path happens on the host.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <string>
#include <vector>
#include <atomic>
#include <thread>

#include "../../include/pbrt_b200.h"
#include "cache.hpp"
#include "kernels.hpp"
#include "mesh_bvh.hpp"
#include "render.hpp"
#include "scene_device.cuh"
#include "bvh_build_gpu.hpp"
#include "scene_host.hpp"
#include "trace_mesh.cuh"
#include "context.hpp"

using namespace pbrt;
using namespace pbrt::api;

namespace {

int ensure_slots(pbrt_ctx* c) {
  if (c->slots_ready) return PBRT_OK;
  for (Slot& s : c->slots) {
    PBRT_TRY(c->cuda(cudaStreamCreateWithFlags(&s.s, cudaStreamNonBlocking), "cudaStreamCreate"));
    PBRT_TRY(c->cuda(cudaMalloc(&s.rays, sizeof(float) * 8 * kSlotRays), "cudaMalloc(staging rays)"));
    PBRT_TRY(c->cuda(cudaMalloc(&s.prim, sizeof(uint32_t) * kSlotRays), "cudaMalloc(staging)"));
    PBRT_TRY(c->cuda(cudaMalloc(&s.t, sizeof(float) * kSlotRays), "cudaMalloc(staging)"));
    PBRT_TRY(c->cuda(cudaMalloc(&s.obj, sizeof(uint32_t) * kSlotRays), "cudaMalloc(staging)"));
    PBRT_TRY(c->cuda(cudaMalloc(&s.occ, kSlotRays), "cudaMalloc(staging)"));
    PBRT_TRY(c->cuda(cudaMalloc(&s.queue, sizeof(uint32_t) * kSlotRays), "cudaMalloc(staging)"));
    PBRT_TRY(c->cuda(cudaMalloc(&s.rec, sizeof(float4) * 2 * kSlotRays), "cudaMalloc(staging)"));
    PBRT_TRY(c->cuda(cudaMalloc(&s.fetch, 2 * sizeof(unsigned long long)), "cudaMalloc(staging)"));
  }
  c->slots_ready = true;
  return PBRT_OK;
}

int ensure_queue(pbrt_ctx* c) {
  if (c->queue && c->queue_rec) return PBRT_OK;
  if (!c->queue) PBRT_TRY(c->cuda(cudaMalloc(&c->queue, sizeof(uint32_t) * kDevChunk), "cudaMalloc(survivor queue)"));
  if (!c->queue_rec)
    PBRT_TRY(c->cuda(cudaMalloc(&c->queue_rec, sizeof(float4) * 2 * kDevChunk), "cudaMalloc(survivor records)"));
  return PBRT_OK;
}

// The survivor queue is the context's: a call waits for the last asynchronous call's use of it,
// whatever the stream (one created after that call's was destroyed may have the same handle).
int acquire_queue(pbrt_ctx* c, cudaStream_t st) {
  if (!c->queue_used) return PBRT_OK;
  return c->cuda(cudaStreamWaitEvent(st, c->queue_used, 0), "cudaStreamWaitEvent(survivor queue)");
}

int release_queue(pbrt_ctx* c, cudaStream_t st) {
  if (!c->queue_used)
    PBRT_TRY(c->cuda(cudaEventCreateWithFlags(&c->queue_used, cudaEventDisableTiming), "cudaEventCreate"));
  return c->cuda(cudaEventRecord(c->queue_used, st), "cudaEventRecord(survivor queue)");
}

}  // namespace

extern "C" {

int pbrt_ctx_create(int device, pbrt_ctx** out) {
  if (!out) return PBRT_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
    cudaGetLastError();
    return PBRT_ERR_INVALID_ARGUMENT;
  }
  std::unique_ptr<pbrt_ctx> c(new pbrt_ctx);
  c->device = device;
  DeviceGuard g(device);
  cudaDeviceProp prop;
  if (c->cuda(cudaGetDeviceProperties(&prop, device), "cudaGetDeviceProperties") != PBRT_OK) return PBRT_ERR_CUDA;
  if (prop.major < 10) return PBRT_ERR_UNSUPPORTED;  // built for sm_100a only
  c->sm_count = prop.multiProcessorCount;
  // PBRT_TRACE_KERNEL=simple selects the one-thread-per-ray kernel (same results) for A/B runs.
  if (const char* k = std::getenv("PBRT_TRACE_KERNEL")) c->persistent = std::strcmp(k, "simple") != 0;
  if (c->cuda(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking), "cudaStreamCreate") != PBRT_OK)
    return PBRT_ERR_CUDA;
  cudaMemPoolProps pp{};
  pp.allocType = cudaMemAllocationTypePinned;
  pp.location.type = cudaMemLocationTypeDevice;
  pp.location.id = device;
  if (c->cuda(cudaMemPoolCreate(&c->pool, &pp), "cudaMemPoolCreate") != PBRT_OK) return PBRT_ERR_CUDA;
  uint64_t keep = kPoolKeep;
  if (c->cuda(cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &keep), "cudaMemPoolSetAttribute") !=
      PBRT_OK)
    return PBRT_ERR_CUDA;
  if (c->cuda(cudaHostAlloc(&c->d_err, sizeof(uint32_t), cudaHostAllocMapped), "cudaHostAlloc") != PBRT_OK)
    return PBRT_ERR_OUT_OF_MEMORY;
  *c->d_err = 0;
  if (c->cuda(cudaMalloc(&c->d_counters, 16 * sizeof(unsigned long long)), "cudaMalloc") != PBRT_OK)
    return PBRT_ERR_OUT_OF_MEMORY;
  if (c->cuda(cudaMemsetAsync(c->d_counters, 0, 16 * sizeof(unsigned long long), c->stream), "cudaMemset") !=
      PBRT_OK)
    return PBRT_ERR_CUDA;
  // The allocation-free trace's scratch array: its address on this device (which loads the
  // trace kernels' module now, under lazy loading, so its 4 MiB are committed here and not
  // inside a later call).
  if (c->cuda(noalloc_scratch_lookup(&c->noalloc_scratch), "cudaGetSymbolAddress") != PBRT_OK) return PBRT_ERR_CUDA;
  if (c->cuda(cudaStreamSynchronize(c->stream), "cudaStreamSynchronize") != PBRT_OK) return PBRT_ERR_CUDA;
  *out = c.release();
  return PBRT_OK;
}

void pbrt_ctx_destroy(pbrt_ctx* c) {
  if (!c) return;
  DeviceGuard g(c->device);
  cudaStreamSynchronize(c->stream);
  for (Slot& s : c->slots) {
    if (s.s) cudaStreamSynchronize(s.s);
    cudaFree(s.rays);
    cudaFree(s.prim);
    cudaFree(s.t);
    cudaFree(s.obj);
    cudaFree(s.occ);
    cudaFree(s.queue);
    cudaFree(s.fetch);
    cudaFree(s.rec);
    if (s.s) cudaStreamDestroy(s.s);
  }
  if (c->side) {
    cudaStreamSynchronize(c->side);
    cudaStreamDestroy(c->side);
  }
  if (c->fork) cudaEventDestroy(c->fork);
  if (c->join) cudaEventDestroy(c->join);
  c->waves.release();
  c->train_waves.release();
  for (uint32_t k = 0; k < kMaxBatchBranches; ++k) {
    if (c->branch_st[k]) {
      cudaStreamSynchronize(c->branch_st[k]);
      cudaStreamDestroy(c->branch_st[k]);
    }
    if (c->branch_join[k]) cudaEventDestroy(c->branch_join[k]);
    if (k + 1 < kMaxBatchBranches) c->branch_waves[k].release();
  }
  if (c->branch_fork) cudaEventDestroy(c->branch_fork);
  if (c->queue_used) cudaEventDestroy(c->queue_used);
  cudaFreeHost(c->d_err);
  cudaFreeHost(c->stage);
  cudaFree(c->d_counters);
  cudaFree(c->queue);
  cudaFree(c->queue_rec);
  cudaStreamDestroy(c->stream);
  if (c->pool) cudaMemPoolDestroy(c->pool);  // (memory of scenes still alive goes with them)
  delete c;
}

const char* pbrt_last_error(const pbrt_ctx* c) { return c ? c->err.c_str() : "null context"; }

int pbrt_ctx_set_stream(pbrt_ctx* c, void* stream) {
  if (!c) return PBRT_ERR_INVALID_ARGUMENT;
  c->user = (cudaStream_t)stream;
  return PBRT_OK;
}

int pbrt_ctx_sync(pbrt_ctx* c) {
  if (!c) return PBRT_ERR_INVALID_ARGUMENT;
  DeviceGuard g(c->device);
  return check_device_error(c, c->work_stream());
}

}  // extern "C"

namespace {

// The device half of scene creation: checks the built structure, uploads it, fills the view.
// Meshes listed in `dev` (non-null nodes) were built on the GPU: their arrays are taken over.
int upload_scene(pbrt_ctx* c, const pbrt_scene_desc* d, const FlatScene& fs, pbrt_scene** out,
                 std::vector<DeviceMeshBuild>* dev = nullptr) {
  for (uint32_t i = 0; i < fs.meshes.size(); ++i)
    if (fs.meshes[i].stats.max_depth >= uint32_t(kTraceStack))
      return c->fail(PBRT_ERR_CAPACITY, "mesh " + std::to_string(i) + ": BVH depth " +
                                             std::to_string(fs.meshes[i].stats.max_depth) +
                                             " exceeds the traversal stack");
  if (fs.top_depth >= uint32_t(kTraceStack))
    return c->fail(PBRT_ERR_CAPACITY, "scene BVH depth exceeds the traversal stack");

  std::unique_ptr<pbrt_scene> s(new pbrt_scene);
  s->ctx = c;
  const uint32_t nm = uint32_t(fs.meshes.size());
  auto built = [&](uint32_t i) { return dev && i < dev->size() && (*dev)[i].nodes; };  // on the GPU
  // All meshes' nodes and triangles end to end, and one wide tree: the top level's nodes first
  // (index 0 stays unused), then each mesh's.
  std::vector<uint64_t> node_at(nm + 1, 0), tri_at(nm + 1, 0), wide_at(nm + 1, 0);
  wide_at[0] = 1 + fs.top_wide_count;
  uint32_t deepest = 0;
  for (uint32_t i = 0; i < nm; ++i) {
    const uint64_t slots = built(i) ? (*dev)[i].node_slots : fs.meshes[i].nodes.size();
    node_at[i + 1] = node_at[i] + slots;
    tri_at[i + 1] = tri_at[i] + d->meshes[i].triangle_count;
    wide_at[i + 1] = wide_at[i] + (built(i) ? (*dev)[i].wide_count : fs.meshes[i].wide_count);
    deepest = std::max(deepest, fs.meshes[i].stats.max_depth);
  }
  const uint64_t total_nodes = node_at[nm], total_tris = tri_at[nm], total_wide = wide_at[nm];
  if (total_tris >= (uint64_t(1) << 30) || total_nodes >= (uint64_t(1) << 32) || total_wide >= (uint64_t(1) << 30))
    return c->fail(PBRT_ERR_CAPACITY, "a scene holds at most 2^30 triangles");
  const bool direct = total_tris <= (uint64_t(1) << 26);
  s->meshes.resize(nm);
  std::vector<MeshView> views(nm);
  std::vector<MeshShade> shades(nm);
  void *nodes = nullptr, *tri = nullptr, *tri_c = nullptr, *wide = nullptr, *exact = nullptr, *leaf = nullptr;
  int rc = PBRT_OK;
  if (nm == 1 && built(0)) {  // the only mesh's arrays are the scene's
    DeviceMeshBuild& b = (*dev)[0];
    s->take(nodes = b.nodes, total_nodes * sizeof(GpuNode));
    s->take(tri = b.tri, total_tris * 32);
    s->take(tri_c = b.tri_c, total_tris * 8);
    b.nodes = nullptr;
    b.tri = nullptr;
    b.tri_c = nullptr;
  } else if (nm) {
    // One kind of array after another, a build's own given back behind its copy: no more than one
    // kind is held twice, and what was given back serves the wide nodes below (as far as the pool
    // finds it in one piece).
    std::vector<char> on_gpu(nm);
    for (uint32_t i = 0; i < nm; ++i) on_gpu[i] = built(i);
    for (int part = 0; part < 3 && rc == PBRT_OK; ++part) {
      void** dst = part == 0 ? &nodes : (part == 1 ? &tri : &tri_c);
      const std::vector<uint64_t>& at = part == 0 ? node_at : tri_at;
      const size_t each = part == 2 ? 8 : 32;
      rc = s->alloc(dst, at[nm] * each);
      for (uint32_t i = 0; i < nm && rc == PBRT_OK; ++i) {
        const FlatMesh& fm = fs.meshes[i];
        const void* src = part == 0 ? (const void*)fm.nodes.data() : (part == 1 ? fm.tri.data() : fm.tri_c.data());
        if (on_gpu[i]) {
          DeviceMeshBuild& b = (*dev)[i];
          src = part == 0 ? (const void*)b.nodes : (part == 1 ? (const void*)b.tri : b.tri_c);
        }
        rc = c->cuda(cudaMemcpyAsync(static_cast<char*>(*dst) + at[i] * each, src, (at[i + 1] - at[i]) * each,
                                     cudaMemcpyDefault, c->stream),
                     "cudaMemcpy(scene)");
        if (rc == PBRT_OK && on_gpu[i]) {
          DeviceMeshBuild& b = (*dev)[i];
          rc = c->cuda(cudaFreeAsync(const_cast<void*>(src), c->stream), "cudaFree(scene)");
          if (part == 0) b.nodes = nullptr;
          if (part == 1) b.tri = nullptr;
          if (part == 2) b.tri_c = nullptr;
        }
      }
    }
  }
  if (rc == PBRT_OK) rc = s->alloc(&wide, total_wide * sizeof(WideNode));
  if (rc == PBRT_OK) rc = s->alloc(&exact, total_wide * sizeof(ExactNode));
  if (rc == PBRT_OK && nm) rc = s->alloc(&leaf, total_tris * sizeof(uint2));
  // A tree's wide nodes, by its own device array of their numbers or a host one.
  auto widen = [&](WidenArgs a, const std::vector<uint32_t>& id) -> int {
    void* copy = nullptr;
    if (!a.wide_id) {
      PBRT_TRY(c->cuda(cudaMallocFromPoolAsync(&copy, id.size() * 4, c->pool, c->stream), "cudaMalloc(scene)"));
      a.wide_id = static_cast<const uint32_t*>(copy);
    }
    int r = copy ? c->cuda(cudaMemcpyAsync(copy, id.data(), id.size() * 4, cudaMemcpyHostToDevice, c->stream),
                           "cudaMemcpy(scene)")
                 : PBRT_OK;
    if (r == PBRT_OK) r = c->cuda(launch_widen(a, c->sm_count, c->stream), "scene upload");
    if (copy) cudaFreeAsync(copy, c->stream);
    return r;
  };
  // The primitives' references: a mesh placed untransformed, once, is merged (its wide root),
  // anything else is an object leaf.
  std::vector<uint32_t> slot_ref(fs.order.size()), owner(nm, 0xFFFFFFFFu);
  bool objects = !fs.unbounded.empty();
  for (uint32_t k = 0; k < fs.order.size(); ++k) {
    const uint32_t ref = fs.order[k];
    const ObjRec* ob = ref & kGroupBit ? nullptr : &fs.objects[ref];
    if (ob && ob->shape == kShapeMesh && ob->xf_count == 0 && owner[ob->mesh] == 0xFFFFFFFFu) {
      const uint32_t m = ob->mesh;
      owner[m] = ref;
      const uint32_t count = uint32_t(tri_at[m + 1] - tri_at[m]);
      slot_ref[k] = node_at[m + 1] - node_at[m] > 2 ? uint32_t(wide_at[m])  // the root's
                                                    : triangle_ref(uint32_t(tri_at[m]), count, direct);
    } else {
      slot_ref[k] = kLeafRef | kObjectRef | k;
      objects = true;
    }
  }
  for (uint32_t i = 0; i < nm && rc == PBRT_OK; ++i) {
    const pbrt_mesh_desc& md = d->meshes[i];
    MeshView& v = views[i];
    v.nodes = static_cast<const float4*>(nodes) + 2 * node_at[i];
    v.tri = static_cast<const float4*>(tri) + 2 * tri_at[i];
    v.tri_c = static_cast<const float2*>(tri_c) + tri_at[i];
    v.node_count = uint32_t(node_at[i + 1] - node_at[i]);
    s->meshes[i] = v;
    WidenArgs a{};
    a.nodes = v.nodes;
    a.count = v.node_count;
    a.wide = static_cast<WideNode*>(wide);
    a.exact = static_cast<ExactNode*>(exact);
    a.wide_base = uint32_t(wide_at[i]);
    a.direct = direct;
    a.tri_base = uint32_t(tri_at[i]);
    a.node_base = uint32_t(node_at[i]);
    a.owner = owner[i];
    a.leaf = static_cast<uint2*>(leaf);
    a.wide_id = dev && i < dev->size() ? (*dev)[i].wide_id : nullptr;
    rc = widen(a, fs.meshes[i].wide_id);
    void* pv = nullptr;
    void* pi = nullptr;
    if (built(i) || (dev && i < dev->size() && (*dev)[i].v)) {  // the build's copies of the mesh's arrays
      DeviceMeshBuild& b = (*dev)[i];
      s->take(pv = b.v, size_t(md.vertex_count) * 12);
      s->take(pi = b.idx, size_t(md.triangle_count) * 12);
      b.v = nullptr;
      b.idx = nullptr;
    } else {
      if (rc == PBRT_OK) rc = s->upload(&pv, md.vertices, size_t(md.vertex_count) * 3 * sizeof(float));
      if (rc == PBRT_OK) rc = s->upload(&pi, md.indices, size_t(md.triangle_count) * 3 * sizeof(uint32_t));
    }
    void* pf = nullptr;
    if (rc == PBRT_OK && md.face_materials) rc = s->upload(&pf, md.face_materials, size_t(md.triangle_count) * 4);
    shades[i] = MeshShade{(const float*)pv, (const uint32_t*)pi, (const uint32_t*)pf};
    const FlatMesh& fm = fs.meshes[i];
    s->info.triangle_count += md.triangle_count;
    s->info.mesh_node_count += fm.stats.node_count;
    s->info.mesh_leaf_count += fm.stats.leaf_count;
    s->info.mesh_max_depth = std::max(s->info.mesh_max_depth, fm.stats.max_depth);
    s->info.mesh_max_leaf_tris = std::max(s->info.mesh_max_leaf_tris, fm.stats.max_leaf_tris);
  }
  void *top = nullptr, *order = nullptr, *objs = nullptr, *mviews = nullptr, *mshades = nullptr, *mats = nullptr,
       *lights = nullptr, *ltris = nullptr, *lcdf = nullptr, *unb = nullptr, *xfs = nullptr, *grps = nullptr,
       *csgs = nullptr, *srefs = nullptr, *snodes = nullptr;
  if (rc == PBRT_OK && !slot_ref.empty()) rc = s->upload(&srefs, slot_ref.data(), slot_ref.size() * sizeof(uint32_t));
  if (rc == PBRT_OK && !slot_ref.empty()) rc = s->alloc(&snodes, slot_ref.size() * sizeof(uint32_t));
  if (rc == PBRT_OK && !fs.top.empty()) rc = s->upload(&top, fs.top.data(), fs.top.size() * sizeof(GpuNode));
  if (rc == PBRT_OK && !fs.order.empty()) rc = s->upload(&order, fs.order.data(), fs.order.size() * sizeof(uint32_t));
  if (rc == PBRT_OK) rc = s->upload(&objs, fs.objects.data(), fs.objects.size() * sizeof(ObjRec));
  if (rc == PBRT_OK && !fs.unbounded.empty())
    rc = s->upload(&unb, fs.unbounded.data(), fs.unbounded.size() * sizeof(uint32_t));
  if (rc == PBRT_OK && !fs.xforms.empty()) rc = s->upload(&xfs, fs.xforms.data(), fs.xforms.size() * sizeof(XfRec));
  if (rc == PBRT_OK && !fs.groups.empty()) rc = s->upload(&grps, fs.groups.data(), fs.groups.size() * sizeof(GroupRec));
  if (rc == PBRT_OK && !fs.csg.empty()) rc = s->upload(&csgs, fs.csg.data(), fs.csg.size() * sizeof(CsgRec));
  if (rc == PBRT_OK && !views.empty()) rc = s->upload(&mviews, views.data(), views.size() * sizeof(MeshView));
  if (rc == PBRT_OK && !shades.empty()) rc = s->upload(&mshades, shades.data(), shades.size() * sizeof(MeshShade));
  if (rc == PBRT_OK) rc = s->upload(&mats, fs.materials.data(), fs.materials.size() * sizeof(MatRec));
  if (rc == PBRT_OK && !fs.lights.empty()) rc = s->upload(&lights, fs.lights.data(), fs.lights.size() * sizeof(LightRec));
  if (rc == PBRT_OK && !fs.light_tris.empty())
    rc = s->upload(&ltris, fs.light_tris.data(), fs.light_tris.size() * sizeof(float));
  if (rc == PBRT_OK && !fs.light_cdf.empty())
    rc = s->upload(&lcdf, fs.light_cdf.data(), fs.light_cdf.size() * sizeof(float));
  if (rc != PBRT_OK) {
    pbrt_scene_destroy(s.release());
    return rc;
  }
  SceneView& v = s->view;
  v.top = (const float4*)top;
  v.top_node_count = uint32_t(fs.top.size());
  v.order = (const uint32_t*)order;
  v.unbounded = (const uint32_t*)unb;
  v.unbounded_count = uint32_t(fs.unbounded.size());
  v.objects = (const ObjRec*)objs;
  v.xforms = (const XfRec*)xfs;
  v.groups = (const GroupRec*)grps;
  v.csg = (const CsgRec*)csgs;
  v.meshes = (const MeshView*)mviews;
  v.shade = (const MeshShade*)mshades;
  v.materials = (const MatRec*)mats;
  v.lights = (const LightRec*)lights;
  v.light_count = uint32_t(fs.lights.size());
  v.light_tris = (const float*)ltris;
  v.light_cdf = (const float*)lcdf;
  v.has_csg = 0;
  for (const ObjRec& ob : fs.objects) v.has_csg |= ob.shape == kShapeCsg ? 1u : 0u;
  v.has_objects = objects ? 1u : 0u;
  WideView& w = v.wide;
  w.exact = (const ExactNode*)exact;
  w.wide = (const WideNode*)wide;
  w.tri = (const float4*)tri;
  w.tri_c = (const float2*)tri_c;
  w.leaf = (const uint2*)leaf;
  w.nodes = (const float4*)nodes;
  w.slot_node = (const uint32_t*)snodes;
  w.count = uint32_t(total_wide);
  w.direct = direct;
  // (a top level of one leaf has no wide node: its primitive's reference is the root)
  w.root = fs.top.empty() ? 0u : (fs.top.size() > 2 ? 1u : slot_ref[0]);
  // The wide walk needs its coordinates inside the grid's arithmetic and its pending slots,
  // three per two levels, inside its stack; otherwise every ray takes the binary nodes.
  w.bounded = 3 * ((fs.top_depth + 1) / 2 + (deepest + 1) / 2 + 2) <= uint32_t(kWideStack);
  for (const GpuNode& g : fs.top)
    for (int x = 0; x < 3; ++x)
      if (!(std::fabs(g.bmin[x]) <= kWideLimit) || !(std::fabs(g.bmax[x]) <= kWideLimit)) w.bounded = false;
  if (!fs.top.empty()) {
    WidenArgs a{};
    a.nodes = (const float4*)top;
    a.count = uint32_t(fs.top.size());
    a.wide = static_cast<WideNode*>(wide);
    a.exact = static_cast<ExactNode*>(exact);
    a.direct = direct;
    a.wide_base = 1;
    a.slot_ref = (const uint32_t*)srefs;
    a.slot_node = (uint32_t*)snodes;
    const int rc1 = widen(a, fs.top_wide);
    if (rc1 != PBRT_OK) {
      pbrt_scene_destroy(s.release());
      return rc1;
    }
  }
  s->info.object_count = fs.primitive_count;
  s->info.device_bytes += s->extra_bytes;
  s->max_radiance = fs.max_radiance;
  s->has_dielectric = fs.has_dielectric;
  for (int a = 0; a < 3; ++a) {  // the bounded primitives' box (none: an empty box)
    s->bounds[a] = fs.top.empty() ? 0.0f : fs.top[0].bmin[a];
    s->bounds[3 + a] = fs.top.empty() ? 0.0f : fs.top[0].bmax[a];
  }
  s->single_mesh = fs.single_mesh;
  const int rc2 = c->cuda(cudaStreamSynchronize(c->stream), "scene upload");
  if (rc2 != PBRT_OK) {
    pbrt_scene_destroy(s.release());
    return rc2;
  }
  *out = s.release();
  return PBRT_OK;
}

// The meshes' BVHs built on the GPU (pbrt_scene_desc::device_build). Mesh arrays in device
// memory are copied to the host for the scene build's host part (validation of face
// materials, area-light triangles, the shading copies); `md` receives the description's
// meshes pointing at host memory.
int build_meshes_on_device(pbrt_ctx* c, const pbrt_scene_desc* d, std::vector<pbrt_mesh_desc>* md,
                           std::vector<std::vector<float>>* hv, std::vector<std::vector<uint32_t>>* hi,
                           std::vector<std::vector<uint32_t>>* hf, std::vector<MeshPrebuilt>* pre,
                           std::vector<DeviceMeshBuild>* builds) {
  const uint32_t n = d->mesh_count;
  md->assign(d->meshes, d->meshes + n);
  hv->resize(n);
  hi->resize(n);
  hf->resize(n);
  pre->resize(n);
  builds->resize(n);
  MeshBuildParams bp;
  bp.bins = d->bvh_bins ? int(d->bvh_bins) : 8;
  bp.max_leaf = d->bvh_max_leaf ? d->bvh_max_leaf : 1;
  cudaStream_t st = c->stream;
  for (uint32_t i = 0; i < n; ++i) {
    const pbrt_mesh_desc& m = d->meshes[i];
    if (!m.vertices || !m.indices || m.triangle_count == 0)
      return c->fail(PBRT_ERR_INVALID_ARGUMENT, "mesh " + std::to_string(i) + ": a TriangleMesh needs triangles");
    const size_t vb = size_t(m.vertex_count) * 3 * sizeof(float), ib = size_t(m.triangle_count) * 3 * sizeof(uint32_t);
    const bool vdev = mem_kind(m.vertices) == MemKind::Device, idev = mem_kind(m.indices) == MemKind::Device;
    float* dv = nullptr;
    uint32_t* di = nullptr;
    int rc = PBRT_OK;
    // the mesh's own copies: the build reads them, and the scene keeps them for shading
    rc = c->cuda(cudaMallocFromPoolAsync(&dv, std::max<size_t>(vb, 4), c->pool, st), "cudaMalloc(build vertices)");
    if (rc == PBRT_OK)
      rc = c->cuda(cudaMallocFromPoolAsync(&di, std::max<size_t>(ib, 4), c->pool, st), "cudaMalloc(build indices)");
    if (rc == PBRT_OK) rc = c->cuda(cudaMemcpyAsync(dv, m.vertices, vb, cudaMemcpyDefault, st), "cudaMemcpy(vertices)");
    if (rc == PBRT_OK) rc = c->cuda(cudaMemcpyAsync(di, m.indices, ib, cudaMemcpyDefault, st), "cudaMemcpy(indices)");
    if (rc == PBRT_OK && vdev) {  // the scene's host part reads them too
      (*hv)[i].resize(size_t(m.vertex_count) * 3);
      rc = c->cuda(cudaMemcpyAsync((*hv)[i].data(), m.vertices, vb, cudaMemcpyDeviceToHost, st), "cudaMemcpy(vertices)");
      (*md)[i].vertices = (*hv)[i].data();
    }
    if (rc == PBRT_OK && idev) {
      (*hi)[i].resize(size_t(m.triangle_count) * 3);
      rc = c->cuda(cudaMemcpyAsync((*hi)[i].data(), m.indices, ib, cudaMemcpyDeviceToHost, st), "cudaMemcpy(indices)");
      (*md)[i].indices = (*hi)[i].data();
    }
    if (rc == PBRT_OK && m.face_materials && mem_kind(m.face_materials) == MemKind::Device) {
      (*hf)[i].resize(m.triangle_count);
      rc = c->cuda(cudaMemcpyAsync((*hf)[i].data(), m.face_materials, size_t(m.triangle_count) * 4,
                                   cudaMemcpyDeviceToHost, st),
                   "cudaMemcpy(face materials)");
      (*md)[i].face_materials = (*hf)[i].data();
    }
    std::string e;
    if (rc == PBRT_OK &&
        !build_mesh_bvh_device(dv, m.vertex_count, di, m.triangle_count, bp, st, c->pool, c->sm_count, &(*builds)[i], &e))
      rc = c->fail(PBRT_ERR_INVALID_ARGUMENT, "mesh " + std::to_string(i) + ": " + e);
    (*builds)[i].v = dv;
    (*builds)[i].idx = di;
    if (rc != PBRT_OK) {
      cudaStreamSynchronize(st);
      for (DeviceMeshBuild& b : *builds) free_device_mesh_build(&b);
      return rc;
    }
    MeshPrebuilt& p = (*pre)[i];
    p.used = true;
    p.stats = (*builds)[i].stats;
    for (int a = 0; a < 3; ++a) {
      p.bounds_min[a] = (*builds)[i].bounds_min[a];
      p.bounds_max[a] = (*builds)[i].bounds_max[a];
    }
  }
  return c->cuda(cudaStreamSynchronize(st), "device BVH build");
}

int check_scene_desc(pbrt_ctx* c, const pbrt_scene_desc* d) {
  if (!d) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "scene description is NULL");
  if (d->object_count == 0) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "a scene needs at least one object");
  if (d->mesh_count && !d->meshes) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "meshes is NULL");
  if (!d->objects) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "objects is NULL");
  return PBRT_OK;
}

}  // namespace

extern "C" {

int pbrt_scene_create(pbrt_ctx* c, const pbrt_scene_desc* d, pbrt_scene** out) {
  if (!c || !d || !out) return PBRT_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  DeviceGuard g(c->device);
  PBRT_TRY(check_scene_desc(c, d));
  FlatScene fs;
  std::string e;
  if (d->device_build && d->mesh_count) {
    std::vector<pbrt_mesh_desc> md;
    std::vector<std::vector<float>> hv;
    std::vector<std::vector<uint32_t>> hi, hf;
    std::vector<MeshPrebuilt> pre;
    std::vector<DeviceMeshBuild> builds;
    PBRT_TRY(build_meshes_on_device(c, d, &md, &hv, &hi, &hf, &pre, &builds));
    pbrt_scene_desc d2 = *d;
    d2.meshes = md.data();
    int rc = PBRT_OK;
    if (!build_scene(d2, &fs, &e, &pre)) rc = c->fail(PBRT_ERR_INVALID_ARGUMENT, e);
    if (rc == PBRT_OK) rc = upload_scene(c, &d2, fs, out, &builds);
    for (DeviceMeshBuild& b : builds) free_device_mesh_build(&b);  // those not taken over
    return rc;
  }
  if (!build_scene(*d, &fs, &e)) return c->fail(PBRT_ERR_INVALID_ARGUMENT, e);
  return upload_scene(c, d, fs, out);
}

int pbrt_scene_create_many(pbrt_ctx* c, const pbrt_scene_desc* descs, uint32_t n, uint32_t threads,
                           pbrt_scene** out) {
  if (!c || !descs || !out) return PBRT_ERR_INVALID_ARGUMENT;
  DeviceGuard g(c->device);
  for (uint32_t i = 0; i < n; ++i) out[i] = nullptr;
  for (uint32_t i = 0; i < n; ++i) PBRT_TRY(check_scene_desc(c, descs + i));
  // GPU mesh builds first (device_build scenes), one scene after another on the context's stream
  struct DevParts {
    std::vector<pbrt_mesh_desc> md;
    std::vector<std::vector<float>> hv;
    std::vector<std::vector<uint32_t>> hi, hf;
    std::vector<MeshPrebuilt> pre;
    std::vector<DeviceMeshBuild> builds;
  };
  std::vector<DevParts> parts(n);
  std::vector<pbrt_scene_desc> d2(descs, descs + n);
  auto free_builds = [&]() {
    for (DevParts& p : parts)
      for (DeviceMeshBuild& b : p.builds) free_device_mesh_build(&b);
  };
  for (uint32_t i = 0; i < n; ++i) {
    if (!descs[i].device_build || !descs[i].mesh_count) continue;
    DevParts& p = parts[i];
    const int rc = build_meshes_on_device(c, descs + i, &p.md, &p.hv, &p.hi, &p.hf, &p.pre, &p.builds);
    if (rc != PBRT_OK) {
      free_builds();
      return rc;
    }
    d2[i].meshes = p.md.data();
  }
  // host builds on a pool of threads (no device calls), then uploads in order
  std::vector<FlatScene> flat(n);
  std::vector<std::string> errs(n);
  std::vector<char> ok(n, 0);
  std::atomic<uint32_t> next{0};
  unsigned T = threads ? threads : std::max(1u, std::thread::hardware_concurrency());
  T = std::min<unsigned>(T, n);
  auto work = [&]() {
    for (uint32_t i = next++; i < n; i = next++)
      ok[i] = build_scene(d2[i], &flat[i], &errs[i], parts[i].pre.empty() ? nullptr : &parts[i].pre) ? 1 : 0;
  };
  std::vector<std::thread> pool;
  for (unsigned t = 1; t < T; ++t) pool.emplace_back(work);
  work();
  for (std::thread& t : pool) t.join();
  for (uint32_t i = 0; i < n; ++i)
    if (!ok[i]) {
      free_builds();
      return c->fail(PBRT_ERR_INVALID_ARGUMENT, "scene " + std::to_string(i) + ": " + errs[i]);
    }
  for (uint32_t i = 0; i < n; ++i) {
    const int rc = upload_scene(c, &d2[i], flat[i], out + i, parts[i].builds.empty() ? nullptr : &parts[i].builds);
    if (rc != PBRT_OK) {
      for (uint32_t j = 0; j < i; ++j) {
        pbrt_scene_destroy(out[j]);
        out[j] = nullptr;
      }
      free_builds();
      return rc;
    }
    FlatScene().meshes.swap(flat[i].meshes);  // release host copies as we go
  }
  free_builds();  // anything not taken over
  return PBRT_OK;
}

void pbrt_scene_destroy(pbrt_scene* s) {
  if (!s) return;
  DeviceGuard g(s->ctx->device);
  wait_for_device();
  for (void* p : s->allocs) cudaFree(p);
  delete s;
}

int pbrt_mesh_bvh_build_device(pbrt_ctx* c, const pbrt_mesh_desc* md, uint32_t bins, uint32_t max_leaf, void* nodes,
                               uint64_t node_capacity, uint32_t* tri_order, uint64_t* node_count, float* build_ms) {
  if (!c || !md || !node_count) return PBRT_ERR_INVALID_ARGUMENT;
  DeviceGuard g(c->device);
  pbrt_scene_desc d{};
  d.meshes = md;
  d.mesh_count = 1;
  d.bvh_bins = bins;
  d.bvh_max_leaf = max_leaf;
  std::vector<pbrt_mesh_desc> m2;
  std::vector<std::vector<float>> hv;
  std::vector<std::vector<uint32_t>> hi, hf;
  std::vector<MeshPrebuilt> pre;
  std::vector<DeviceMeshBuild> b;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (build_ms) {
    PBRT_TRY(c->cuda(cudaEventCreate(&e0), "cudaEventCreate"));
    PBRT_TRY(c->cuda(cudaEventCreate(&e1), "cudaEventCreate"));
    PBRT_TRY(c->cuda(cudaEventRecord(e0, c->stream), "cudaEventRecord"));
  }
  int rc = build_meshes_on_device(c, &d, &m2, &hv, &hi, &hf, &pre, &b);
  if (rc == PBRT_OK && build_ms) {
    rc = c->cuda(cudaEventRecord(e1, c->stream), "cudaEventRecord");
    if (rc == PBRT_OK) rc = c->cuda(cudaEventSynchronize(e1), "cudaEventSynchronize");
    if (rc == PBRT_OK) rc = c->cuda(cudaEventElapsedTime(build_ms, e0, e1), "cudaEventElapsedTime");
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (rc != PBRT_OK) return rc;
  DeviceMeshBuild& r = b[0];
  *node_count = r.node_slots;  // 32-byte records, the padding slot included (as the host variant)
  if (nodes && node_capacity < r.node_slots) rc = PBRT_ERR_CAPACITY;
  if (rc == PBRT_OK && nodes)
    rc = c->cuda(cudaMemcpy(nodes, r.nodes, r.node_slots * sizeof(GpuNode), cudaMemcpyDeviceToHost), "cudaMemcpy(nodes)");
  if (rc == PBRT_OK && nodes && tri_order)
    rc = c->cuda(cudaMemcpy(tri_order, r.tri_index, size_t(md->triangle_count) * 4, cudaMemcpyDeviceToHost),
                 "cudaMemcpy(order)");
  free_device_mesh_build(&r);
  return rc;
}

int pbrt_mesh_bvh_build_host(const pbrt_mesh_desc* md, uint32_t bins, uint32_t max_leaf, void* nodes,
                             uint64_t node_capacity, uint32_t* tri_order, uint64_t* node_count) {
  if (!md || !node_count) return PBRT_ERR_INVALID_ARGUMENT;
  MeshBuildParams bp;
  bp.bins = bins ? int(bins) : 8;
  bp.max_leaf = max_leaf ? max_leaf : 1;
  FlatMesh fm;
  std::string e;
  if (!build_mesh_bvh(md->vertices, md->vertex_count, md->indices, md->triangle_count, bp, &fm, &e))
    return PBRT_ERR_INVALID_ARGUMENT;
  *node_count = fm.nodes.size();
  if (!nodes) return PBRT_OK;
  if (node_capacity < fm.nodes.size()) return PBRT_ERR_CAPACITY;
  std::memcpy(nodes, fm.nodes.data(), fm.nodes.size() * sizeof(GpuNode));
  if (tri_order) std::memcpy(tri_order, fm.tri_index.data(), fm.tri_index.size() * sizeof(uint32_t));
  return PBRT_OK;
}

// Loader::load_scene (src/loader.rs:29-45): the scene file parsed, then built like any scene.
int pbrt_scene_load(pbrt_ctx* c, const char* text, const pbrt_stage_options* options, pbrt_scene** scene,
                    pbrt_camera_desc* camera) {
  if (!c || !scene) return PBRT_ERR_INVALID_ARGUMENT;
  *scene = nullptr;
  char err[512];
  pbrt_stage* st = nullptr;
  const int rc = pbrt_stage_parse(text, options, &st, err, sizeof(err));
  if (rc != PBRT_OK) return c->fail(rc, std::string("scene file: ") + err);
  pbrt_scene_desc d;
  pbrt_stage_describe(st, &d, camera, nullptr);
  const int rc2 = pbrt_scene_create(c, &d, scene);
  pbrt_stage_destroy(st);
  return rc2;
}

int pbrt_scene_get_info(const pbrt_scene* s, pbrt_scene_info* info) {
  if (!s || !info) return PBRT_ERR_INVALID_ARGUMENT;
  *info = s->info;
  return PBRT_OK;
}

}  // extern "C"

namespace {

// Runs the nearest-hit (or, with occ != NULL, any-hit) kernel over host or device buffers.
// stats with scene_stats: the scene accelerator's counters (any scene); stats alone: the
// mesh traversal's (scenes of one untransformed mesh).
int trace_impl(pbrt_scene* s, const float* rays, uint64_t n, uint32_t* prim, float* t, uint32_t* obj, uint8_t* occ,
               uint64_t* stats, bool scene_stats = false) {
  if (!s) return PBRT_ERR_INVALID_ARGUMENT;
  pbrt_ctx* c = s->ctx;
  DeviceGuard g(c->device);
  if (n == 0) return PBRT_OK;
  if (!rays || (!occ && (!prim || !t))) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "ray or result buffer is NULL");
  if (stats && !scene_stats && s->single_mesh < 0)
    return c->fail(PBRT_ERR_UNSUPPORTED, "work counters are reported for scenes made of one untransformed mesh");
  const bool one_mesh = s->single_mesh >= 0 && !scene_stats;
  const MeshView mv = one_mesh ? s->meshes[s->single_mesh] : MeshView{};
  const WideView& wv = s->view.wide;
  // Nearest hit / any hit of one chunk of `m` rays (planes `stride` apart) on `st`; without a queue
  // one thread per ray.
  auto launch = [&](const float* r, uint64_t stride, uint64_t m, uint32_t* p, float* tt, uint32_t* ob, uint8_t* oc,
                    unsigned long long* cnt, uint32_t* queue, unsigned long long* qc, float4* rec,
                    cudaStream_t st) -> cudaError_t {
    if (!one_mesh)
      return oc ? launch_scene_any(s->view, r, stride, m, oc, cnt, c->d_err, c->sm_count, st)
                : launch_scene_closest(s->view, r, stride, m, p, tt, ob, cnt, c->d_err, c->sm_count, st);
    if (!c->persistent || cnt)
      return oc ? launch_mesh_any(mv, r, stride, m, oc, c->d_err, c->sm_count, st)
                : launch_mesh_closest(mv, r, stride, m, p, tt, ob, cnt, c->d_err, c->sm_count, st);
    if (m <= kFewRays)
      return oc ? launch_mesh_any_few(mv, wv, r, stride, m, oc, c->d_err, c->sm_count, st)
                : launch_mesh_closest_few(mv, wv, r, stride, m, p, tt, ob, c->d_err, c->sm_count, st);
    if (!queue)
      return oc ? launch_mesh_any_planes(mv, wv, r, stride, m, oc, c->d_err, c->sm_count, st)
                : launch_mesh_closest_planes(mv, wv, r, stride, m, p, tt, ob, c->d_err, c->sm_count, st);
    return oc ? launch_mesh_any_persistent(mv, wv, r, stride, m, oc, queue, qc, c->d_err, c->sm_count, st, rec)
              : launch_mesh_closest_persistent(mv, wv, r, stride, m, p, tt, ob, queue, qc, c->d_err, c->sm_count, st, rec);
  };

  const MemKind kr = mem_kind(rays);
  const MemKind ko = occ ? mem_kind(occ) : mem_kind(prim);
  const MemKind kt = occ ? ko : mem_kind(t);
  const MemKind kb = obj ? mem_kind(obj) : ko;
  if (kr != ko || ko != kt || kt != kb)
    return c->fail(PBRT_ERR_INVALID_ARGUMENT, "ray and result buffers must all be host memory or all device memory");

  unsigned long long* counters = nullptr;
  if (stats) {
    counters = c->d_counters;
    PBRT_TRY(c->cuda(cudaMemsetAsync(counters, 0, 3 * sizeof(unsigned long long), c->work_stream()), "cudaMemset"));
  }

  if (kr == MemKind::Device) {
    cudaStream_t st = c->work_stream();
    // Few rays take one kernel without scratch. So does a call on a stream under capture, of any
    // size: a graph replayed later may run beside another call's use of the queue.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (c->user) PBRT_TRY(c->cuda(cudaStreamIsCapturing(st, &cap), "cudaStreamIsCapturing"));
    const bool queued = one_mesh && c->persistent && !counters && n > kFewRays && cap == cudaStreamCaptureStatusNone;
    if (queued) {
      PBRT_TRY(ensure_queue(c));
      PBRT_TRY(acquire_queue(c, st));
    }
    // Chunks of at most kDevChunk rays bound the survivor queue (scratch) to 64 MiB.
    const uint64_t chunk = one_mesh ? kDevChunk : n;
    for (uint64_t base = 0; base < n; base += chunk) {
      const uint64_t m = std::min<uint64_t>(chunk, n - base);
      PBRT_TRY(c->cuda(launch(rays + base, n, m, occ ? nullptr : prim + base, occ ? nullptr : t + base,
                              obj ? obj + base : nullptr, occ ? occ + base : nullptr, counters,
                              queued ? c->queue : nullptr, c->d_counters + 4, c->queue_rec, st),
                       "kernel launch"));
    }
    if (queued && c->user) PBRT_TRY(release_queue(c, st));
    if (stats) {
      unsigned long long h[3];
      PBRT_TRY(c->cuda(cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, st), "cudaMemcpy"));
      PBRT_TRY(check_device_error(c, st));
      for (int k = 0; k < 3; ++k) stats[k] = h[k];
      return PBRT_OK;
    }
    if (c->user) return PBRT_OK;  // ordered on the caller's stream; errors surface at pbrt_ctx_sync
    return check_device_error(c, st);
  }

  // A small host call on one mesh: the rays are copied into pinned memory that one kernel reads,
  // and it writes its answers there, so that no copy engine, no second kernel and no memset stand
  // in its way. (20,480 triangles, nearest hits through the Python call, staged against chunks:
  // 100 rays 26 / 54 us, 4,099 rays 50 / 79, 32,768 rays 160 / 168.)
  if (one_mesh && c->persistent && !counters && n <= kStageRays) {
    if (!c->stage) PBRT_TRY(c->cuda(cudaHostAlloc(&c->stage, kStageBytes, cudaHostAllocMapped), "cudaHostAlloc(stage)"));
    if (c->user) PBRT_TRY(c->cuda(cudaStreamSynchronize(c->user), "cudaStreamSynchronize"));
    const uint64_t stride = (n + 31) & ~uint64_t(31);  // planes on 128-byte lines
    float* in = reinterpret_cast<float*>(c->stage);
    uint32_t* out = reinterpret_cast<uint32_t*>(in + 8 * stride);
    for (int k = 0; k < 8; ++k) std::memcpy(in + k * stride, rays + k * n, n * 4);
    uint32_t* p = out;
    float* tt = reinterpret_cast<float*>(out + stride);
    uint32_t* ob = out + 2 * stride;
    uint8_t* oc = reinterpret_cast<uint8_t*>(out);
    PBRT_TRY(c->cuda(launch(in, stride, n, p, tt, obj ? ob : nullptr, occ ? oc : nullptr, nullptr, nullptr, nullptr,
                            nullptr, c->stream),
                     "kernel launch"));
    PBRT_TRY(check_device_error(c, c->stream));
    if (occ) {
      std::memcpy(occ, oc, n);
      return PBRT_OK;
    }
    std::memcpy(prim, p, n * 4);
    std::memcpy(t, tt, n * 4);
    if (obj) std::memcpy(obj, ob, n * 4);
    return PBRT_OK;
  }

  // Host buffers: pipeline chunks through three staging slots, each on its own stream, so
  // the copy engines and the SMs overlap (H2D of chunk k+1 and D2H of k-1 run under the
  // kernel of chunk k). With 1M-ray chunks and one 2D copy per chunk a 16M-ray call takes the
  // time of its bare copies (512 MiB in, 128 MiB out concurrently: 10.3 ms on PCIe 5).
  PBRT_TRY(ensure_slots(c));
  if (c->user) PBRT_TRY(c->cuda(cudaStreamSynchronize(c->user), "cudaStreamSynchronize"));
  if (stats)
    PBRT_TRY(c->cuda(cudaStreamSynchronize(c->work_stream()), "cudaStreamSynchronize"));
  uint64_t chunk = 0;
  for (uint64_t base = 0; base < n; base += kSlotRays, ++chunk) {
    Slot& sl = c->slots[chunk % kSlots];
    const uint64_t m = std::min<uint64_t>(kSlotRays, n - base);
    // the chunk's eight planes as one 2D copy (rows = planes): one DMA job instead of eight
    PBRT_TRY(c->cuda(cudaMemcpy2DAsync(sl.rays, kSlotRays * sizeof(float), rays + base, n * sizeof(float),
                                       m * sizeof(float), 8, cudaMemcpyHostToDevice, sl.s),
                     "cudaMemcpy2DAsync(rays)"));
    PBRT_TRY(c->cuda(launch(sl.rays, kSlotRays, m, sl.prim, sl.t, obj ? sl.obj : nullptr, occ ? sl.occ : nullptr,
                            counters, c->persistent ? sl.queue : nullptr, sl.fetch, sl.rec, sl.s),
                     "kernel launch"));
    if (occ) {
      PBRT_TRY(c->cuda(cudaMemcpyAsync(occ + base, sl.occ, m, cudaMemcpyDeviceToHost, sl.s), "cudaMemcpyAsync"));
    } else {
      PBRT_TRY(c->cuda(cudaMemcpyAsync(prim + base, sl.prim, m * 4, cudaMemcpyDeviceToHost, sl.s), "cudaMemcpyAsync"));
      PBRT_TRY(c->cuda(cudaMemcpyAsync(t + base, sl.t, m * 4, cudaMemcpyDeviceToHost, sl.s), "cudaMemcpyAsync"));
      if (obj)
        PBRT_TRY(c->cuda(cudaMemcpyAsync(obj + base, sl.obj, m * 4, cudaMemcpyDeviceToHost, sl.s), "cudaMemcpyAsync"));
    }
  }
  int rc = PBRT_OK;
  for (Slot& sl : c->slots) {
    int r = c->cuda(cudaStreamSynchronize(sl.s), "kernel execution");
    if (rc == PBRT_OK) rc = r;
  }
  PBRT_TRY(rc);
  if (stats) {
    unsigned long long h[3];
    PBRT_TRY(c->cuda(cudaMemcpy(h, counters, sizeof(h), cudaMemcpyDeviceToHost), "cudaMemcpy"));
    for (int k = 0; k < 3; ++k) stats[k] = h[k];
  }
  return check_device_error(c, c->stream);
}

}  // namespace

extern "C" {

int pbrt_trace_closest(pbrt_scene* s, const float* rays, uint64_t n, uint32_t* prim_id, float* t, uint32_t* object_id) {
  return trace_impl(s, rays, n, prim_id, t, object_id, nullptr, nullptr);
}

int pbrt_trace_closest_instrumented(pbrt_scene* s, const float* rays, uint64_t n, uint32_t* prim_id, float* t,
                                    uint64_t* stats) {
  if (!stats) return PBRT_ERR_INVALID_ARGUMENT;
  return trace_impl(s, rays, n, prim_id, t, nullptr, nullptr, stats);
}

static_assert(kNoAllocMaxRays == PBRT_NOALLOC_MAX_RAYS, "header and kernels disagree on the no-alloc capacity");

// For callers that cannot call cudaMalloc (see the header): the same two kernels as the
// device-buffer path of pbrt_trace_closest, with their scratch in a static __device__ array
// whose address the context looked up when it was created.
int pbrt_trace_closest_noalloc(pbrt_scene* s, const float* rays, uint64_t n, uint32_t* prim_id, float* t) {
  if (!s) return PBRT_ERR_INVALID_ARGUMENT;
  pbrt_ctx* c = s->ctx;
  if (n == 0) return PBRT_OK;  // as pbrt_trace_closest: nothing to do, whatever the scene
  DeviceGuard g(c->device);
  if (n > kNoAllocMaxRays)
    return c->fail(PBRT_ERR_CAPACITY, "pbrt_trace_closest_noalloc: n = " + std::to_string(n) +
                                          " exceeds its fixed scratch capacity of " + std::to_string(kNoAllocMaxRays) +
                                          " rays; split the batch or use pbrt_trace_closest");
  cudaStream_t st = c->work_stream();
  // The call waits for its results (it reads the error word back), which a stream under
  // capture cannot do: refuse before any other CUDA call, so the caller's capture survives.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  PBRT_TRY(c->cuda(cudaStreamIsCapturing(st, &cap), "cudaStreamIsCapturing"));
  if (cap != cudaStreamCaptureStatusNone)
    return c->fail(PBRT_ERR_UNSUPPORTED,
                   "pbrt_trace_closest_noalloc waits for its results and cannot run on a stream being captured");
  if (!rays || !prim_id || !t) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "ray or result buffer is NULL");
  if (mem_kind(rays) != MemKind::Device || mem_kind(prim_id) != MemKind::Device || mem_kind(t) != MemKind::Device)
    return c->fail(PBRT_ERR_INVALID_ARGUMENT,
                   "pbrt_trace_closest_noalloc takes device buffers only (host buffers need staging memory)");
  if (s->single_mesh < 0)
    return c->fail(PBRT_ERR_UNSUPPORTED, "pbrt_trace_closest_noalloc traces scenes made of one untransformed mesh");
  const MeshView& mv = s->meshes[s->single_mesh];
  uint32_t* scratch = c->noalloc_scratch;
  PBRT_TRY(c->cuda(launch_mesh_closest_noalloc(mv, s->view.wide, rays, n, prim_id, t, scratch, c->sm_count, st),
                   "pbrt_trace_closest_noalloc"));
  uint32_t h = 0;  // the error word, read back on the same stream (no legacy-stream wait)
  PBRT_TRY(c->cuda(cudaMemcpyAsync(&h, scratch + 4, sizeof(h), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync"));
  PBRT_TRY(c->cuda(cudaStreamSynchronize(st), "kernel execution"));
  if (h & kErrStack) return c->fail(PBRT_ERR_CAPACITY, "traversal stack capacity exceeded");
  if (h) return c->fail(PBRT_ERR_DEVICE_BUDGET, "a traversal exceeded its iteration budget (malformed tree)");
  return PBRT_OK;
}

int pbrt_trace_any(pbrt_scene* s, const float* rays, uint64_t n, uint8_t* occluded) {
  if (!occluded) return s ? s->ctx->fail(PBRT_ERR_INVALID_ARGUMENT, "occluded is NULL") : PBRT_ERR_INVALID_ARGUMENT;
  return trace_impl(s, rays, n, nullptr, nullptr, nullptr, occluded, nullptr);
}

int pbrt_trace_closest_counted(pbrt_scene* s, const float* rays, uint64_t n, uint32_t* prim_id, float* t,
                               uint32_t* object_id, uint64_t* stats) {
  if (!stats) return s ? s->ctx->fail(PBRT_ERR_INVALID_ARGUMENT, "stats is NULL") : PBRT_ERR_INVALID_ARGUMENT;
  for (int k = 0; k < 3; ++k) stats[k] = 0;
  return trace_impl(s, rays, n, prim_id, t, object_id, nullptr, stats, true);
}

int pbrt_trace_any_counted(pbrt_scene* s, const float* rays, uint64_t n, uint8_t* occluded, uint64_t* stats) {
  if (!occluded || !stats)
    return s ? s->ctx->fail(PBRT_ERR_INVALID_ARGUMENT, "occluded or stats is NULL") : PBRT_ERR_INVALID_ARGUMENT;
  for (int k = 0; k < 3; ++k) stats[k] = 0;
  return trace_impl(s, rays, n, nullptr, nullptr, nullptr, occluded, stats, true);
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Rendering
// ---------------------------------------------------------------------------------------
int pbrt::api::ensure_wave(pbrt_ctx* c, WaveAlloc* wa, uint32_t cap) {
  if (wa->capacity >= cap) return PBRT_OK;
  cudaFree(wa->block);
  wa->block = nullptr;
  wa->capacity = 0;
  const size_t n = cap;
  // 4-byte arrays: 6 ray + 3 beta + 3 L + pixel + scene + flags + ht + hobj + hprim + qa + qb + 11 shadow
  // = 32 words, plus the 8-byte rng state, plus 4 counters.
  const size_t bytes = n * (32 * 4 + 8) + 64;
  PBRT_TRY(c->cuda(cudaMalloc(&wa->block, bytes), "cudaMalloc(wave state)"));
  char* p = static_cast<char*>(wa->block);
  auto f32 = [&]() { float* r = reinterpret_cast<float*>(p); p += n * 4; return r; };
  auto u32 = [&]() { uint32_t* r = reinterpret_cast<uint32_t*>(p); p += n * 4; return r; };
  WaveBuffers& w = wa->w;
  w.rng = reinterpret_cast<unsigned long long*>(p);
  p += n * 8;
  w.ox = f32(); w.oy = f32(); w.oz = f32(); w.dx = f32(); w.dy = f32(); w.dz = f32();
  w.br = f32(); w.bg = f32(); w.bb = f32(); w.lr = f32(); w.lg = f32(); w.lb = f32();
  w.pixel = u32(); w.scene = u32(); w.flags = u32(); w.ht = f32(); w.hobj = u32(); w.hprim = u32(); w.qa = u32(); w.qb = u32();
  w.s_path = u32(); w.s_ox = f32(); w.s_oy = f32(); w.s_oz = f32(); w.s_dx = f32(); w.s_dy = f32(); w.s_dz = f32();
  w.s_tmax = f32(); w.s_cr = f32(); w.s_cg = f32(); w.s_cb = f32();
  w.counts = reinterpret_cast<uint32_t*>(p);
  wa->capacity = cap;
  return PBRT_OK;
}

// The query buffers of a wave. They are the context's, as the waves are, so that a new cache's first
// frame maps no memory: with blocks of its own (830 MB at 1920x1080, 2 samples, of which 332 were
// used) it took 11.7 ms beside another state, 6.9 so.
int pbrt::api::ensure_queries(pbrt_ctx* c, WaveAlloc* wa, uint32_t cap) {
  if (wa->qblock && wa->qcap >= cap) return PBRT_OK;
  cudaFree(wa->qblock);
  wa->qblock = nullptr;
  wa->qcap = 0;
  wa->q = CacheWave{};
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  const size_t rec = up(size_t(cap) * kCacheRecordFloats * 4), out = up(size_t(cap) * 12), path = up(size_t(cap) * 4);
  PBRT_TRY(c->cuda(cudaMalloc(&wa->qblock, 256 + rec + out + path), "cudaMalloc(cache queries)"));
  char* p = static_cast<char*>(wa->qblock);
  wa->q.counts = reinterpret_cast<uint32_t*>(p);
  wa->q.qrec = reinterpret_cast<float*>(p + 256);
  wa->q.qout = reinterpret_cast<float*>(p + 256 + rec);
  wa->q.qpath = reinterpret_cast<uint32_t*>(p + 256 + rec + out);
  wa->q.qcap = wa->qcap = cap;
  return PBRT_OK;
}

int pbrt::api::check_render_params(pbrt_ctx* c, const pbrt_render_params* p, bool allow_no_samples) {
  const pbrt_camera_desc& cd = p->camera;
  if (cd.width == 0 || cd.height == 0) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "empty image");
  if (p->spp == 0 && !allow_no_samples) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "spp must be >= 1");
  if (p->max_depth == 0 || p->max_depth > 0xFFFF)
    return c->fail(PBRT_ERR_INVALID_ARGUMENT, "max_depth must be in [1, 65535]");
  if (p->integrator > PBRT_INTEGRATOR_NORMAL) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "unknown integrator");
  if (!(cd.fov > 0.f) || !(cd.fov < 3.14159265f) || !(cd.far > cd.near))
    return c->fail(PBRT_ERR_INVALID_ARGUMENT, "bad camera");
  if (cd.thin_lens && (!(cd.lens_radius >= 0.f) || !std::isfinite(cd.lens_radius) || !std::isfinite(cd.focal_distance)))
    return c->fail(PBRT_ERR_INVALID_ARGUMENT, "bad thin lens");
  if (uint64_t(cd.width) * cd.height > 0xFFFFFFFFull) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "image too large");
  if (p->pixel_stride > cd.width || p->pixel_stride > cd.height)
    return c->fail(PBRT_ERR_INVALID_ARGUMENT, "pixel_stride exceeds the image");
  return PBRT_OK;
}

RenderSettings pbrt::api::settings_of(pbrt_ctx* c, const pbrt_render_params* p) {
  RenderSettings rs;
  rs.stats = c->d_counters + 8;
  rs.shape = c->shape;
  rs.max_depth = p->max_depth;
  rs.rr_start = p->integrator == PBRT_INTEGRATOR_PATH ? p->rr_start : 0u;
  rs.sample_offset = p->sample_offset;
  rs.integrator = p->integrator;
  rs.seed = p->seed;
  rs.stride = p->pixel_stride > 1 ? p->pixel_stride : 1u;
  rs.film_w = (p->camera.width + rs.stride - 1) / rs.stride;
  return rs;
}

// Film pixels of a render: the image's, or the strided subset's.
uint64_t pbrt::api::film_pixels(const pbrt_render_params* p, const RenderSettings& rs) {
  return uint64_t(rs.film_w) * ((p->camera.height + rs.stride - 1) / rs.stride);
}

namespace {

// Training paths of the cached render go this many hits past the render's cache hit before
// they end into the cache themselves.
constexpr uint32_t kTrainTail = 3;

// Concurrent branches of one pbrt_render: the frame's paths split into this many contiguous
// parts, each a chain of waves on its own stream with its own wave buffers, so that one
// part's per-bounce kernel tails overlap another part's work. PBRT_RENDER_BRANCHES (1..8)
// overrides it for measurements; films do not depend on it.
uint32_t render_branches(uint64_t total) {
  static const uint32_t v = [] {
    const char* e = std::getenv("PBRT_RENDER_BRANCHES");
    const int k = e ? std::atoi(e) : int(kDefaultRenderBranches);
    return uint32_t(k >= 1 && k <= int(kMaxBatchBranches) ? k : kDefaultRenderBranches);
  }();
  return uint32_t(std::min<uint64_t>(v, std::max<uint64_t>(1, total / 1024)));
}

unsigned long long host_mix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  return x ^ (x >> 31);
}

}  // namespace

extern "C" {

int pbrt_render(pbrt_scene* s, const pbrt_render_params* p, double* film) {
  if (!s) return PBRT_ERR_INVALID_ARGUMENT;
  pbrt_ctx* c = s->ctx;
  DeviceGuard g(c->device);
  if (!p || !film) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "params or film is NULL");
  PBRT_TRY(check_render_params(c, p, false));
  const pbrt_camera_desc& cd = p->camera;
  const CameraRec cam = build_camera(cd);
  const RenderSettings rs = settings_of(c, p);
  const uint64_t npix = film_pixels(p, rs);
  const uint64_t total = npix * p->spp;

  // the paths in `nb` contiguous parts [j * part, (j + 1) * part), part j on branch j
  const uint32_t nb = render_branches(total);
  const uint64_t part = (total + nb - 1) / nb;
  const uint32_t wave = uint32_t(std::min<uint64_t>(part, c->wave_paths));
  PBRT_TRY(ensure_wave(c, &c->waves, wave));
  for (uint32_t j = 1; j < nb; ++j) {
    PBRT_TRY(ensure_wave(c, &c->branch_waves[j - 1], wave));
    if (!c->branch_st[j])
      PBRT_TRY(c->cuda(cudaStreamCreateWithFlags(&c->branch_st[j], cudaStreamNonBlocking), "cudaStreamCreate"));
    if (!c->branch_join[j])
      PBRT_TRY(c->cuda(cudaEventCreateWithFlags(&c->branch_join[j], cudaEventDisableTiming), "cudaEventCreate"));
  }
  if (nb > 1 && !c->branch_fork)
    PBRT_TRY(c->cuda(cudaEventCreateWithFlags(&c->branch_fork, cudaEventDisableTiming), "cudaEventCreate"));
  cudaStream_t st = c->work_stream();
  const size_t film_n = size_t(npix) * 3;
  double* dfilm = film;
  const bool host_film = mem_kind(film) != MemKind::Device;
  if (host_film) PBRT_TRY(c->cuda(cudaMalloc(&dfilm, film_n * sizeof(double)), "cudaMalloc(film)"));
  int rc = c->cuda(cudaMemsetAsync(dfilm, 0, film_n * sizeof(double), st), "cudaMemset(film)");
  if (rc == PBRT_OK) rc = c->cuda(cudaMemsetAsync(rs.stats, 0, 3 * sizeof(unsigned long long), st), "cudaMemset");
  if (rc == PBRT_OK && nb > 1) rc = c->cuda(cudaEventRecord(c->branch_fork, st), "cudaEventRecord");
  for (uint32_t j = 1; j < nb && rc == PBRT_OK; ++j)
    rc = c->cuda(cudaStreamWaitEvent(c->branch_st[j], c->branch_fork, 0), "cudaStreamWaitEvent");
  for (uint32_t j = 0; j < nb && rc == PBRT_OK; ++j) {
    cudaStream_t bs = j ? c->branch_st[j] : st;
    const WaveBuffers& bw = j ? c->branch_waves[j - 1].w : c->waves.w;
    const uint64_t end = std::min<uint64_t>(total, (j + 1) * part);
    for (uint64_t base = j * part; base < end && rc == PBRT_OK; base += wave) {
      const uint32_t n = uint32_t(std::min<uint64_t>(wave, end - base));
      rc = c->cuda(render_wave(s->view, bw, cam, base, n, uint32_t(npix), rs, dfilm, c->d_err, c->sm_count, bs),
                   "render");
    }
  }
  // the branches join `st` again (also after a failed launch, so that no branch is left behind)
  for (uint32_t j = 1; j < nb; ++j) {
    const int jr = c->cuda(cudaEventRecord(c->branch_join[j], c->branch_st[j]), "cudaEventRecord");
    if (jr == PBRT_OK) cudaStreamWaitEvent(st, c->branch_join[j], 0);
    if (rc == PBRT_OK) rc = jr;
  }
  if (rc == PBRT_OK) rc = c->cuda(scale_film(dfilm, film_n, 1.0 / double(p->spp), c->sm_count, st), "render");
  if (host_film) {
    if (rc == PBRT_OK)
      rc = c->cuda(cudaMemcpyAsync(film, dfilm, film_n * sizeof(double), cudaMemcpyDeviceToHost, st), "cudaMemcpy(film)");
    if (rc == PBRT_OK) rc = check_device_error(c, st);
    cudaStreamSynchronize(st);
    cudaFree(dfilm);
    return rc;
  }
  PBRT_TRY(rc);
  if (c->user) return PBRT_OK;
  return check_device_error(c, st);
}

int pbrt_render_cached(pbrt_scene* s, pbrt_cache* k, const pbrt_render_params* p, uint32_t train_rounds,
                       double* film) {
  if (!s || !k) return PBRT_ERR_INVALID_ARGUMENT;
  pbrt_ctx* c = s->ctx;
  DeviceGuard g(c->device);
  if (k->ctx != c) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "the cache belongs to another context");
  if (!p) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "params is NULL");
  PBRT_TRY(check_render_params(c, p, true));
  if (p->spp && !film) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "film is NULL");
  if (p->integrator != PBRT_INTEGRATOR_PATH)
    return c->fail(PBRT_ERR_UNSUPPORTED, "the radiance cache ends path-integrator paths only");
  pbrt_cache_params& cp = k->params;
  if (cp.scene_min[0] == cp.scene_max[0] && cp.scene_min[1] == cp.scene_max[1] && cp.scene_min[2] == cp.scene_max[2])
    for (int a = 0; a < 3; ++a) {
      cp.scene_min[a] = s->bounds[a];
      cp.scene_max[a] = s->bounds[3 + a];
    }
  const pbrt_camera_desc& cd = p->camera;
  const CameraRec cam = build_camera(cd);
  const RenderSettings rs = settings_of(c, p);
  const uint64_t npix = film_pixels(p, rs);
  const uint64_t total = npix * p->spp;
  const uint32_t train_paths = std::max(128u, cp.train_samples / 4);
  const uint32_t steps = cp.train_steps;
  const uint32_t batch = std::max(128u, cp.train_samples / steps);
  // the frame's paths in `nbr` contiguous parts on concurrent branches, as pbrt_render's; branch
  // j >= 1 has its own wave buffers and query buffers
  const uint32_t nbr = render_branches(total);
  const uint64_t part = (total + nbr - 1) / nbr;
  const uint32_t fwave = uint32_t(std::min<uint64_t>(part, c->wave_paths));
  const bool beside = train_rounds > 0 && p->spp > 0;

  // One query per path at most. The rounds share the frame's first wave, or run beside it on one of
  // their own.
  WaveAlloc& wa = c->waves;
  const uint32_t first_cap = beside || train_rounds == 0 ? fwave : std::max(fwave, train_paths);
  PBRT_TRY(ensure_wave(c, &wa, first_cap));
  PBRT_TRY(ensure_queries(c, &wa, first_cap));
  if (train_rounds) PBRT_TRY(k->ensure_train_buffers(cp.train_samples, batch));
  cudaStream_t st = c->work_stream();
  PBRT_TRY(c->cuda(cudaMemsetAsync(rs.stats, 0, 3 * sizeof(unsigned long long), st), "cudaMemset"));

  // A call that trains and renders runs its rounds beside the frame: the rounds on the
  // context's side stream with their own wave, the frame on `st`, reading a snapshot of the weights the call started with. The rounds' few thousand paths
  // leave most of the GPU idle; this way the frame's work fills it.
  cudaStream_t ts = st;            // the training rounds' stream
  WaveAlloc* twa = &wa;            // and their wave
  mlp::Net fnet{k->wfwd, k->wbwd};  // the weights the frame reads
  if (beside) {
    if (!c->side) PBRT_TRY(c->cuda(cudaStreamCreateWithFlags(&c->side, cudaStreamNonBlocking), "cudaStreamCreate"));
    if (!c->fork) PBRT_TRY(c->cuda(cudaEventCreateWithFlags(&c->fork, cudaEventDisableTiming), "cudaEventCreate"));
    if (!c->join) PBRT_TRY(c->cuda(cudaEventCreateWithFlags(&c->join, cudaEventDisableTiming), "cudaEventCreate"));
    twa = &c->train_waves;
    PBRT_TRY(ensure_wave(c, twa, train_paths));
    PBRT_TRY(ensure_queries(c, twa, train_paths));
    PBRT_TRY(c->cuda(cudaMemcpyAsync(k->wsnap, k->wfwd, mlp::kParams * 2, cudaMemcpyDeviceToDevice, st),
                     "cudaMemcpy(weight snapshot)"));
    PBRT_TRY(c->cuda(cudaEventRecord(c->fork, st), "cudaEventRecord"));
    PBRT_TRY(c->cuda(cudaStreamWaitEvent(c->side, c->fork, 0), "cudaStreamWaitEvent"));
    ts = c->side;
    fnet.wpk_fwd = k->wsnap;
  }
  CacheWave cw = k->cw;  // the rounds' training vertices, and their wave's queries
  cw.qrec = twa->q.qrec;
  cw.qout = twa->q.qout;
  cw.qpath = twa->q.qpath;
  cw.qcap = twa->q.qcap;

  // Online training. Training paths start at random pixels, go kTrainTail hits past the
  // render's cache hit and end into the cache there; their earlier Lambertian and metal
  // vertices become training samples. No host synchronisation: counts stay on the device.
  const uint32_t term_hit = cp.terminate_bounce + 1;
  const uint32_t tail_hit = term_hit + kTrainTail;
  const mlp::Net net{k->wfwd, k->wbwd};
  const mlp::Bounds nb = k->bounds();
  int trc = PBRT_OK;
  {
    auto train = [&]() -> int {
      for (uint32_t r = 0; r < train_rounds; ++r) {
        RenderSettings tr = rs;
        tr.cache_mode = kCacheRecord;
        tr.term_hit = tail_hit;
        tr.random_pixels = 1;
        tr.sample_offset = 0;
        tr.seed = host_mix64(p->seed ^ host_mix64(0x747261696e696e67ULL + k->rounds));
        if (!s->has_dielectric) tr.loop_depth = std::min(rs.max_depth, tail_hit);
        PBRT_TRY(c->cuda(cudaMemsetAsync(cw.counts, 0, 3 * sizeof(uint32_t), ts), "cudaMemset(cache counts)"));
        PBRT_TRY(c->cuda(trace_wave(s->view, twa->w, cw, cam, 0, train_paths, uint32_t(npix), tr, c->d_err, c->sm_count, ts),
                         "cache training paths"));
        PBRT_TRY(c->cuda(mlp::launch_infer_dev(net, nb, cw.qrec, cw.counts, train_paths, cw.qout, c->d_err, c->sm_count,
                                               ts),
                         "cache training tails"));
        PBRT_TRY(c->cuda(apply_cache(twa->w, cw, train_paths, s->max_radiance, c->sm_count, ts), "cache training tails"));
        for (uint32_t step = 0; step < steps; ++step) {
          PBRT_TRY(c->cuda(train_batch(twa->w, cw, batch, step, tr.seed, s->max_radiance, k->brec, k->btgt, c->sm_count, ts),
                           "cache training batch"));
          PBRT_TRY(k->gradient_device(k->brec, k->btgt, batch, ts));
          PBRT_TRY(k->adam_device(ts, cw.counts + 2));
        }
        ++k->rounds;
      }
      return PBRT_OK;
    };
    trc = train();
  }
  if (beside) {  // the call ends when its rounds have: `st` waits for them at the end
    const int jr = c->cuda(cudaEventRecord(c->join, c->side), "cudaEventRecord");
    if (trc == PBRT_OK) trc = jr;
  }
  if (trc != PBRT_OK) {
    if (beside) cudaStreamWaitEvent(st, c->join, 0);
    return trc;
  }
  if (p->spp == 0) {
    if (c->user) return PBRT_OK;
    return check_device_error(c, st);
  }

  // rendering: paths end into the cache at hit terminate_bounce + 1
  RenderSettings qr = rs;
  qr.cache_mode = kCacheQuery;
  qr.term_hit = term_hit;
  if (!s->has_dielectric) qr.loop_depth = std::min(rs.max_depth, term_hit);
  const size_t film_n = size_t(npix) * 3;
  double* dfilm = film;
  const bool host_film = mem_kind(film) != MemKind::Device;
  if (host_film) PBRT_TRY(c->cuda(cudaMalloc(&dfilm, film_n * sizeof(double)), "cudaMalloc(film)"));
  int rc = PBRT_OK;
  for (uint32_t j = 1; j < nbr && rc == PBRT_OK; ++j) {
    rc = ensure_wave(c, &c->branch_waves[j - 1], fwave);
    if (rc == PBRT_OK) rc = ensure_queries(c, &c->branch_waves[j - 1], fwave);
    if (rc == PBRT_OK && !c->branch_st[j])
      rc = c->cuda(cudaStreamCreateWithFlags(&c->branch_st[j], cudaStreamNonBlocking), "cudaStreamCreate");
    if (rc == PBRT_OK && !c->branch_join[j])
      rc = c->cuda(cudaEventCreateWithFlags(&c->branch_join[j], cudaEventDisableTiming), "cudaEventCreate");
  }
  if (rc == PBRT_OK && nbr > 1 && !c->branch_fork)
    rc = c->cuda(cudaEventCreateWithFlags(&c->branch_fork, cudaEventDisableTiming), "cudaEventCreate");
  if (rc != PBRT_OK) {
    if (beside) cudaStreamWaitEvent(st, c->join, 0);
    if (host_film) cudaFree(dfilm);
    return rc;
  }
  rc = c->cuda(cudaMemsetAsync(dfilm, 0, film_n * sizeof(double), st), "cudaMemset(film)");
  if (rc == PBRT_OK && nbr > 1) rc = c->cuda(cudaEventRecord(c->branch_fork, st), "cudaEventRecord");
  for (uint32_t j = 1; j < nbr && rc == PBRT_OK; ++j)
    rc = c->cuda(cudaStreamWaitEvent(c->branch_st[j], c->branch_fork, 0), "cudaStreamWaitEvent");
  for (uint32_t j = 0; j < nbr && rc == PBRT_OK; ++j) {
    cudaStream_t bs = j ? c->branch_st[j] : st;
    const WaveBuffers& bw = j ? c->branch_waves[j - 1].w : wa.w;
    const CacheWave& q = j ? c->branch_waves[j - 1].q : wa.q;
    const uint64_t end = std::min<uint64_t>(total, (j + 1) * part);
    for (uint64_t base = j * part; base < end && rc == PBRT_OK; base += fwave) {
      const uint32_t n = uint32_t(std::min<uint64_t>(fwave, end - base));
      rc = c->cuda(cudaMemsetAsync(q.counts, 0, sizeof(uint32_t), bs), "cudaMemset(cache counts)");
      if (rc == PBRT_OK)
        rc = c->cuda(trace_wave(s->view, bw, q, cam, base, n, uint32_t(npix), qr, c->d_err, c->sm_count, bs),
                     "cached render");
      if (rc == PBRT_OK)
        rc = c->cuda(mlp::launch_infer_dev(fnet, nb, q.qrec, q.counts, n, q.qout, c->d_err, c->sm_count, bs),
                     "cache query");
      if (rc == PBRT_OK) rc = c->cuda(apply_cache(bw, q, n, s->max_radiance, c->sm_count, bs), "cache apply");
      if (rc == PBRT_OK) rc = c->cuda(accumulate_wave(bw, n, dfilm, cd.width, qr, c->sm_count, bs), "cached render");
    }
  }
  for (uint32_t j = 1; j < nbr; ++j) {  // the branches join `st` again
    const int jr = c->cuda(cudaEventRecord(c->branch_join[j], c->branch_st[j]), "cudaEventRecord");
    if (jr == PBRT_OK) cudaStreamWaitEvent(st, c->branch_join[j], 0);
    if (rc == PBRT_OK) rc = jr;
  }
  if (rc == PBRT_OK) rc = c->cuda(scale_film(dfilm, film_n, 1.0 / double(p->spp), c->sm_count, st), "render");
  if (beside) {
    const int jr = c->cuda(cudaStreamWaitEvent(st, c->join, 0), "cudaStreamWaitEvent");
    if (rc == PBRT_OK) rc = jr;
  }
  if (host_film) {
    if (rc == PBRT_OK)
      rc = c->cuda(cudaMemcpyAsync(film, dfilm, film_n * sizeof(double), cudaMemcpyDeviceToHost, st), "cudaMemcpy(film)");
    if (rc == PBRT_OK) rc = check_device_error(c, st);
    cudaStreamSynchronize(st);
    cudaFree(dfilm);
    return rc;
  }
  PBRT_TRY(rc);
  if (c->user) return PBRT_OK;
  return check_device_error(c, st);
}

int pbrt_ctx_set_tuning(pbrt_ctx* c, const pbrt_tuning* t) {
  if (!c) return PBRT_ERR_INVALID_ARGUMENT;
  pbrt_tuning d{};
  if (t) d = *t;
  LaunchShape sh;
  const uint32_t wave = d.wave_paths ? d.wave_paths : (1u << 26);
  if (d.trace_threads) sh.trace_threads = d.trace_threads;
  if (d.trace_blocks_per_sm) sh.trace_blocks_per_sm = d.trace_blocks_per_sm;
  if (d.shade_threads) sh.shade_threads = d.shade_threads;
  if (d.shade_blocks_per_sm) sh.shade_blocks_per_sm = d.shade_blocks_per_sm;
  auto bad_threads = [](uint32_t x) { return x < 32 || x > 256 || x % 32 != 0; };
  auto bad_blocks = [](uint32_t x) { return x < 1 || x > 64; };
  if (bad_threads(sh.trace_threads) || bad_threads(sh.shade_threads))
    return c->fail(PBRT_ERR_INVALID_ARGUMENT, "threads per block must be a multiple of 32 in [32, 256]");
  if (bad_blocks(sh.trace_blocks_per_sm) || bad_blocks(sh.shade_blocks_per_sm))
    return c->fail(PBRT_ERR_INVALID_ARGUMENT, "blocks per SM must be in [1, 64]");
  if (wave < 1024 || wave > (1u << 26)) return c->fail(PBRT_ERR_INVALID_ARGUMENT, "wave_paths must be in [1024, 2^26]");
  c->shape = sh;
  c->wave_paths = wave;
  return PBRT_OK;
}

int pbrt_ctx_get_tuning(pbrt_ctx* c, pbrt_tuning* t) {
  if (!c || !t) return PBRT_ERR_INVALID_ARGUMENT;
  t->wave_paths = c->wave_paths;
  t->trace_threads = c->shape.trace_threads;
  t->trace_blocks_per_sm = c->shape.trace_blocks_per_sm;
  t->shade_threads = c->shape.shade_threads;
  t->shade_blocks_per_sm = c->shape.shade_blocks_per_sm;
  return PBRT_OK;
}

int pbrt_ctx_render_stats(pbrt_ctx* c, uint64_t* stats) {
  if (!c || !stats) return PBRT_ERR_INVALID_ARGUMENT;
  DeviceGuard g(c->device);
  PBRT_TRY(c->cuda(cudaStreamSynchronize(c->work_stream()), "sync"));
  unsigned long long h[3];
  PBRT_TRY(c->cuda(cudaMemcpy(h, c->d_counters + 8, sizeof(h), cudaMemcpyDeviceToHost), "cudaMemcpy(render stats)"));
  for (int i = 0; i < 3; ++i) stats[i] = h[i];
  return PBRT_OK;
}

int pbrt_film_to_rgba8(const double* film, uint32_t w, uint32_t h, uint8_t* rgba) {
  if (!film || !rgba) return PBRT_ERR_INVALID_ARGUMENT;
  for (size_t i = 0; i < size_t(w) * h; ++i) {
    for (int ch = 0; ch < 3; ++ch) {
      const double v = std::sqrt(film[3 * i + ch]);           // gamma_correct (spectrum.rs:19-23)
      const double b = std::fmin(1.0, std::fmax(0.0, v));      // in_bound (spectrum.rs:134-136)
      rgba[4 * i + ch] = uint8_t(b * 255.0);                   // `as u8` truncates (spectrum.rs:13-17)
    }
    rgba[4 * i + 3] = 255;
  }
  return PBRT_OK;
}

}  // extern "C"
