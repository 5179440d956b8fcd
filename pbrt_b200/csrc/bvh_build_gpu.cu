// bvh_build_gpu.cu — a triangle mesh's BVH built on the GPU: node for node, and triangle for
// triangle in every leaf, the tree mesh_bvh.cpp builds on the host (and so the reference's
// binned-SAH tree, src/shapes/triangle_mesh/bvh.rs:221-309, 609-735).
//
// What has to be identical, and how it is kept so:
//   - the centroid extents, bins, SAH costs and split decisions: min / max / counts are
//     order-independent, and the cost arithmetic is the host's, operation for operation
//     (FP32, round-to-nearest intrinsics, no FMA);
//   - the order of the triangles inside every node: the host partitions with one forward
//     pass that swaps each left triangle to the front (bvh.rs:260-267). Its result is
//     computed here in parallel: a left triangle with ordinal q (q lefts before it) lands at
//     q; a right triangle at i >= nl (nl lefts in all) stays; a right triangle at p < nl moves
//     along p -> pos(p) -> pos(pos(p)) ... (pos(q) = where the left of ordinal q stands) to
//     the first position >= nl — resolved by pointer jumping;
//   - the node numbering: the host numbers nodes depth first (children pushed as a pair when
//     their parent splits, left subtree first); here nodes are made in any order and
//     renumbered from their subtree sizes;
//   - stored zero bounds are +0 in both builders (the sign of a zero bound depends on visiting
//     order and no slab test can observe it).
// Large nodes (more than kSmall triangles) are split level by level by many blocks at once;
// a subtree of at most kSmall triangles is built by one warp in shared memory with the host's
// algorithm. The children of a split are made on the device (their boxes are the unions of the
// bins on either side); the host reads one record of counts per level, to size its launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <string>
#include <vector>

#include "bvh_build_gpu.hpp"

namespace pbrt {
namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kSmall = 128;     // subtrees of at most this many triangles: one warp each
constexpr uint32_t kChunk = 2048;    // elements per block in the level kernels
constexpr int kLevelThreads = 256;
constexpr int kMaxBins = 64;
constexpr int kBinWords = 7;         // a bin: orderable box (lo xyz, hi xyz), count
constexpr int kJumpHops = 8;         // chain links a pointer-jumping round follows
constexpr int kMaxJumpRounds = 16;
enum : uint32_t { kBuildErrInput = 1u };

struct __align__(16) TriRec {
  float4 c;   // centroid xyz, w = bits of the original triangle index
  float4 lo;  // triangle box
  float4 hi;
};

struct PoolNode {  // a node in making, in any order; renumbered at the end
  float lo[3], hi[3];
  uint32_t first, count, depth, child;  // child: the left child's pool index (right = +1), or kNone
};

struct LevelNode {  // a large node split by the level kernels
  uint32_t pool, first, count, depth;
  uint32_t ext[6];  // orderable centroid min xyz, max xyz
  float cmin[3], width[3];
  uint32_t use;     // bit a: axis a has distinct centroids
  uint32_t split, axis, boundary, nl;
  uint32_t cfirst, nchunks;  // its chunks in the level's list
  uint32_t next[2];          // the children: a node of the next level, or kToBuffer / kFinal
};
// A child that is not a node of the next level: its triangles wait for its warp, or are final.
constexpr uint32_t kToBuffer = 0xFFFFFFFEu, kFinal = 0xFFFFFFFFu;

struct Chunk {
  uint32_t node, start, len;  // start relative to the node's first triangle
};

struct SmallJob {
  uint32_t pool, first, count, depth_buf;  // depth | buffer << 31
};

struct Counters {  // on the device; the host reads them once per level
  uint32_t err, pool, jobs, changed[kMaxJumpRounds + 1];
  uint32_t nodes[2], chunks[2];  // of the levels, ping-pong
  uint32_t root_box[6], vertex_box[6];
};

// ---- FP32 helpers (the host builder's expressions) ----------------------------------------
__device__ __forceinline__ float mn(float x, float y) { return y < x ? y : x; }
__device__ __forceinline__ float mx(float x, float y) { return x < y ? y : x; }
__device__ __forceinline__ float canon(float x) { return x == 0.0f ? 0.0f : x; }
// a monotone map of floats to unsigned integers, for atomic min / max
__device__ __forceinline__ uint32_t f2o(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}
__device__ __forceinline__ float half_area(const float* lo, const float* hi) {
  if (lo[0] > hi[0] || lo[1] > hi[1] || lo[2] > hi[2]) return 0.0f;
  const float dx = __fsub_rn(hi[0], lo[0]), dy = __fsub_rn(hi[1], lo[1]), dz = __fsub_rn(hi[2], lo[2]);
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dy), __fmul_rn(dy, dz)), __fmul_rn(dz, dx));
}
// bin_index (bvh.rs:173-176) as the host restates it
__device__ __forceinline__ int bin_of(float pos, float cmin, float width, int bins) {
  const float q = __fdiv_rn(__fsub_rn(pos, cmin), width);
  if (!(q >= 0.0f)) return 0;
  if (q >= float(bins - 1)) return bins - 1;
  return int(q);
}
__device__ __forceinline__ float comp(const float4& v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// ---- block reductions ---------------------------------------------------------------------
__device__ __forceinline__ uint32_t warp_min(uint32_t v) {
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  return v;
}
__device__ __forceinline__ uint32_t warp_max(uint32_t v) {
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  return v;
}
// Reduces k values per thread (min for the first half, max for the second) across the block
// and applies one atomic per value into dst.
template <int K>
__device__ void block_minmax_atomic(uint32_t (&v)[K], uint32_t* dst) {
  __shared__ uint32_t red[K][kLevelThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int k = 0; k < K; ++k) {
    const uint32_t r = k < K / 2 ? warp_min(v[k]) : warp_max(v[k]);
    if (lane == 0) red[k][w] = r;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    const int k = threadIdx.x;
    uint32_t r = red[k][0];
    for (int j = 1; j < kLevelThreads / 32; ++j) r = k < K / 2 ? min(r, red[k][j]) : max(r, red[k][j]);
    if (k < K / 2) atomicMin(dst + k, r);
    else atomicMax(dst + k, r);
  }
  __syncthreads();
}

// ---- preparation ----------------------------------------------------------------------------
// tri_centroid and aabound_from_triangle (bvh.rs:564-584) per triangle; bad input sets err
__global__ void k_tri_prep(const float* __restrict__ v, uint32_t nv, const uint32_t* __restrict__ idx, uint32_t n,
                           TriRec* __restrict__ out, uint32_t* err) {
  const float third = __fdiv_rn(1.0f, 3.0f);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t i0 = idx[3 * size_t(i)], i1 = idx[3 * size_t(i) + 1], i2 = idx[3 * size_t(i) + 2];
    if (i0 >= nv || i1 >= nv || i2 >= nv) {
      atomicOr(err, kBuildErrInput);
      out[i] = TriRec{};
      continue;
    }
    float p[3][3];
    for (int a = 0; a < 3; ++a) {
      p[0][a] = v[3 * size_t(i0) + a];
      p[1][a] = v[3 * size_t(i1) + a];
      p[2][a] = v[3 * size_t(i2) + a];
    }
    float c[3], lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
      lo[a] = mn(mn(p[0][a], p[1][a]), p[2][a]);
      hi[a] = mx(mx(p[0][a], p[1][a]), p[2][a]);
      c[a] = __fmul_rn(__fadd_rn(__fadd_rn(p[0][a], p[1][a]), p[2][a]), third);
    }
    out[i] = TriRec{make_float4(c[0], c[1], c[2], __uint_as_float(i)), make_float4(lo[0], lo[1], lo[2], 0.f),
                    make_float4(hi[0], hi[1], hi[2], 0.f)};
  }
}

// vertex bounds (TriangleMesh::get_bounding_box) and finiteness of every coordinate
__global__ void k_vertex_bounds(const float* __restrict__ v, uint32_t nv, uint32_t* box, uint32_t* err) {
  uint32_t r[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x)
    for (int a = 0; a < 3; ++a) {
      const float x = v[3 * size_t(i) + a];
      if (!isfinite(x)) atomicOr(err, kBuildErrInput);
      const uint32_t o = f2o(canon(x));
      r[a] = min(r[a], o);
      r[3 + a] = max(r[3 + a], o);
    }
  block_minmax_atomic<6>(r, box);
}

// the root's box: bounds over every triangle (bvh.rs:232-238)
__global__ void k_root_box(const TriRec* __restrict__ t, uint32_t n, uint32_t* box) {
  uint32_t r[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const TriRec x = t[i];
    r[0] = min(r[0], f2o(canon(x.lo.x))); r[1] = min(r[1], f2o(canon(x.lo.y))); r[2] = min(r[2], f2o(canon(x.lo.z)));
    r[3] = max(r[3], f2o(canon(x.hi.x))); r[4] = max(r[4], f2o(canon(x.hi.y))); r[5] = max(r[5], f2o(canon(x.hi.z)));
  }
  block_minmax_atomic<6>(r, box);
}

__global__ void k_root_node(PoolNode* pool, const uint32_t* box, uint32_t n) {
  PoolNode& p = pool[0];
  for (int a = 0; a < 3; ++a) {
    p.lo[a] = canon(o2f(box[a]));
    p.hi[a] = canon(o2f(box[3 + a]));
  }
  p.first = 0;
  p.count = n;
  p.depth = 1;
  p.child = kNone;
}

// ---- the split decision -----------------------------------------------------------------------
__device__ __forceinline__ void clear_bin(uint32_t* e) {
  e[0] = e[1] = e[2] = f2o(FLT_MAX);
  e[3] = e[4] = e[5] = f2o(-FLT_MAX);
  e[6] = 0u;
}

// One triangle into its bin of axis a (fill_bins, bvh.rs:694-711); shared memory.
__device__ __forceinline__ void add_to_bin(uint32_t* e, const float4& lo, const float4& hi) {
  atomicMin(e, f2o(lo.x));
  atomicMin(e + 1, f2o(lo.y));
  atomicMin(e + 2, f2o(lo.z));
  atomicMax(e + 3, f2o(hi.x));
  atomicMax(e + 4, f2o(hi.y));
  atomicMax(e + 5, f2o(hi.z));
  atomicAdd(e + 6, 1u);
}

// One warp: the split of a node from its bins (3 * B of them in shared memory), as the host
// evaluates it: axes in order, boundaries in order, the first strictly cheapest candidate, taken
// when it is cheaper than the leaf. A lane evaluates a candidate at a time. False: a leaf.
__device__ bool best_split(const uint32_t* bins, int B, uint32_t use, float leaf_cost, int& axis, int& boundary) {
  const int lane = threadIdx.x & 31, S = B - 1;
  uint32_t best = 0xFFFFFFFFu;  // orderable cost
  int bestj = 1 << 30, firstj = 1 << 30;
  bool first_nan = false;
  for (int j = lane; j < 3 * S; j += 32) {
    const int a = j / S, m = j - a * S;
    if (!(use & (1u << a))) continue;
    float lo[2][3], hi[2][3];
    uint32_t cnt[2] = {0u, 0u};
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        lo[s][q] = FLT_MAX;
        hi[s][q] = -FLT_MAX;
      }
    for (int b = 0; b < B; ++b) {  // boundary m: bins 0..m on the left
      const uint32_t* e = bins + kBinWords * (a * B + b);
      const int s = b <= m ? 0 : 1;
      float l[3], h[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        l[q] = o2f(e[q]);
        h[q] = o2f(e[3 + q]);
      }
      const uint32_t c = e[6];
      if (s == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          lo[0][q] = mn(lo[0][q], l[q]);
          hi[0][q] = mx(hi[0][q], h[q]);
        }
        cnt[0] += c;
      } else {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          lo[1][q] = mn(lo[1][q], l[q]);
          hi[1][q] = mx(hi[1][q], h[q]);
        }
        cnt[1] += c;
      }
    }
    if (cnt[0] == 0u || cnt[1] == 0u) continue;
    const float cost = __fadd_rn(__fmul_rn(half_area(lo[0], hi[0]), __uint2float_rn(cnt[0])),
                                 __fmul_rn(half_area(lo[1], hi[1]), __uint2float_rn(cnt[1])));
    const bool nan = !(cost == cost);
    if (j < firstj) {
      firstj = j;
      first_nan = nan;
    }
    if (!nan && f2o(cost) < best) {
      best = f2o(cost);
      bestj = j;
    }
  }
  const uint32_t least = __reduce_min_sync(0xFFFFFFFFu, best);
  const int j = __reduce_min_sync(0xFFFFFFFFu, best == least ? bestj : 1 << 30);
  // (a NaN as the first candidate is never beaten, nor cheaper than the leaf)
  const int f = __reduce_min_sync(0xFFFFFFFFu, firstj);
  if (__any_sync(0xFFFFFFFFu, firstj == f && first_nan)) return false;
  if (j >= 3 * S) return false;
  axis = j / S;
  boundary = j - axis * S;
  return o2f(least) < leaf_cost;
}

// One warp: the children's boxes, the unions of the split axis's bins on either side. Lane v < 12
// returns component v % 6 (lo xyz, hi xyz) of child v / 6.
__device__ float child_box(const uint32_t* bins, int B, int axis, int boundary) {
  const int v = threadIdx.x & 31, side = v / 6, q = v % 6;
  uint32_t r = q < 3 ? 0xFFFFFFFFu : 0u;
  if (v < 12)
    for (int b = side ? boundary + 1 : 0; b < (side ? B : boundary + 1); ++b) {
      const uint32_t* e = bins + kBinWords * (axis * B + b);
      if (e[6] != 0u) r = q < 3 ? min(r, e[q]) : max(r, e[q]);
    }
  return canon(o2f(r));
}

// ---- the level kernels (large nodes) -------------------------------------------------------
// The first level: one node over every triangle, its chunks.
__global__ void k_root_level(LevelNode* nodes, Chunk* chunks, uint32_t n, Counters* ctr) {
  const uint32_t nc = (n + kChunk - 1) / kChunk;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nc; k += gridDim.x * blockDim.x)
    chunks[k] = Chunk{0u, k * kChunk, min(kChunk, n - k * kChunk)};
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    LevelNode& r = nodes[0];
    r.pool = 0;
    r.first = 0;
    r.count = n;
    r.depth = 1;
    r.cfirst = 0;
    r.nchunks = nc;
    for (int q = 0; q < 6; ++q) r.ext[q] = q < 3 ? 0xFFFFFFFFu : 0u;
    ctr->nodes[0] = 1;
    ctr->chunks[0] = nc;
  }
}

// The root's centroid extents (every later level's come from k_permute).
__global__ void k_ext(const TriRec* __restrict__ t, LevelNode* nodes, const Chunk* __restrict__ chunks) {
  const Chunk ch = chunks[blockIdx.x];
  LevelNode& nd = nodes[ch.node];
  const uint32_t base = nd.first + ch.start;
  uint32_t r[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
  for (uint32_t k = threadIdx.x; k < ch.len; k += blockDim.x) {
    const float4 c = t[base + k].c;
    r[0] = min(r[0], f2o(c.x)); r[1] = min(r[1], f2o(c.y)); r[2] = min(r[2], f2o(c.z));
    r[3] = max(r[3], f2o(c.x)); r[4] = max(r[4], f2o(c.y)); r[5] = max(r[5], f2o(c.z));
  }
  block_minmax_atomic<6>(r, nd.ext);
}

// per node: the splittable axes and bin widths (find_best_split_plane's first lines), bins reset
__global__ void k_bin_prep(LevelNode* nodes, uint32_t* bins, int B) {
  LevelNode& nd = nodes[blockIdx.x];
  if (threadIdx.x == 0) {
    nd.use = 0;
    for (int a = 0; a < 3; ++a) {
      const float lo = o2f(nd.ext[a]), hi = o2f(nd.ext[3 + a]);
      nd.cmin[a] = lo;
      nd.width[a] = __fdiv_rn(__fsub_rn(hi, lo), float(B));
      if (!(lo == hi)) nd.use |= 1u << a;
    }
  }
  uint32_t* b = bins + size_t(blockIdx.x) * 3 * B * kBinWords;
  for (int k = threadIdx.x; k < 3 * B; k += blockDim.x) clear_bin(b + kBinWords * k);
}

// fill_bins for the three axes: box of the triangles whose centroid falls in each bin, and
// their count
__global__ void k_bins(const TriRec* __restrict__ t, const LevelNode* __restrict__ nodes,
                       const Chunk* __restrict__ chunks, uint32_t* bins, int B) {
  __shared__ uint32_t sb[3 * kMaxBins * kBinWords];
  const Chunk ch = chunks[blockIdx.x];
  const LevelNode& nd = nodes[ch.node];
  for (int k = threadIdx.x; k < 3 * B; k += blockDim.x) clear_bin(sb + kBinWords * k);
  __syncthreads();
  const uint32_t base = nd.first + ch.start;
  for (uint32_t k = threadIdx.x; k < ch.len; k += blockDim.x) {
    const TriRec x = t[base + k];
    for (int a = 0; a < 3; ++a)
      if (nd.use & (1u << a))
        add_to_bin(sb + kBinWords * (a * B + bin_of(comp(x.c, a), nd.cmin[a], nd.width[a], B)), x.lo, x.hi);
  }
  __syncthreads();
  uint32_t* g = bins + size_t(ch.node) * 3 * B * kBinWords;
  for (int k = threadIdx.x; k < 3 * B; k += blockDim.x) {
    const uint32_t* e = sb + kBinWords * k;
    if (e[6] == 0) continue;
    uint32_t* d = g + kBinWords * k;
    for (int q = 0; q < 3; ++q) {
      atomicMin(d + q, e[q]);
      atomicMax(d + 3 + q, e[3 + q]);
    }
    atomicAdd(d + 6, e[6]);
  }
}

// One warp per node: the split; a split node gets its two children in the pool, with their
// boxes. (The counts of the bins on either side are the children's counts.)
__global__ void __launch_bounds__(32) k_sah(LevelNode* nodes, const uint32_t* __restrict__ bins, int B, PoolNode* pool,
                                            Counters* ctr) {
  __shared__ uint32_t sb[3 * kMaxBins * kBinWords];
  LevelNode& nd = nodes[blockIdx.x];
  const int lane = threadIdx.x;
  const uint32_t* g = bins + size_t(blockIdx.x) * 3 * B * kBinWords;
  for (int k = lane; k < 3 * B * kBinWords; k += 32) sb[k] = g[k];
  __syncwarp();
  PoolNode& p = pool[nd.pool];
  const float leaf_cost = __fmul_rn(half_area(p.lo, p.hi), __uint2float_rn(nd.count));
  int axis = 0, boundary = 0;
  const bool split = best_split(sb, B, nd.use, leaf_cost, axis, boundary);
  if (!split) {
    if (lane == 0) nd.split = 0;
    return;
  }
  uint32_t c = 0, nl = 0;
  for (int b = lane; b <= boundary; b += 32) nl += sb[kBinWords * (axis * B + b) + 6];
  nl = __reduce_add_sync(0xFFFFFFFFu, nl);
  if (lane == 0) c = atomicAdd(&ctr->pool, 2u);
  c = __shfl_sync(0xFFFFFFFFu, c, 0);
  const float box = child_box(sb, B, axis, boundary);
  if (lane < 12) {
    PoolNode& q = pool[c + lane / 6];
    const int k = lane % 6;
    if (k < 3) q.lo[k] = box;
    else q.hi[k - 3] = box;
  }
  if (lane < 2) {
    PoolNode& q = pool[c + lane];
    q.first = nd.first + (lane ? nl : 0u);
    q.count = lane ? nd.count - nl : nl;
    q.depth = nd.depth + 1;
    q.child = kNone;
  }
  if (lane == 0) {
    p.child = c;
    p.count = 0;
    nd.split = 1;
    nd.axis = uint32_t(axis);
    nd.boundary = uint32_t(boundary);
    nd.nl = nl;
  }
}

// The partition's classification: each triangle's ordinal among its chunk's lefts, and whether
// it is one.
__global__ void __launch_bounds__(kLevelThreads) k_classify(const TriRec* __restrict__ t,
                                                            const LevelNode* __restrict__ nodes,
                                                            const Chunk* __restrict__ chunks,
                                                            uint32_t* __restrict__ ord, uint32_t* chunk_tot, int B) {
  constexpr int kRounds = kChunk / kLevelThreads, kWarps = kLevelThreads / 32;
  __shared__ uint32_t tot[kRounds * kWarps + 1];
  const Chunk ch = chunks[blockIdx.x];
  const LevelNode& nd = nodes[ch.node];
  if (!nd.split) return;
  const uint32_t base = nd.first + ch.start;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int axis = int(nd.axis), boundary = int(nd.boundary);
  const float cmin = nd.cmin[axis], width = nd.width[axis];
  uint32_t bal[kRounds];
#pragma unroll
  for (int j = 0; j < kRounds; ++j) {
    const uint32_t k = j * kLevelThreads + threadIdx.x;
    const bool left = k < ch.len && bin_of(comp(t[base + k].c, axis), cmin, width, B) <= boundary;
    bal[j] = __ballot_sync(0xFFFFFFFFu, left);
    if (lane == 0) tot[j * kWarps + w] = __popc(bal[j]);
  }
  __syncthreads();
  if (w == 0) {  // exclusive scan of the 64 counts, two per lane
    static_assert(kRounds * kWarps == 64, "two counts per lane");
    const uint32_t a = tot[2 * lane], b = tot[2 * lane + 1];
    uint32_t incl = a + b;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, off);
      if (lane >= off) incl += y;
    }
    tot[2 * lane] = incl - a - b;
    tot[2 * lane + 1] = incl - b;
    if (lane == 31) chunk_tot[blockIdx.x] = incl;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRounds; ++j) {
    const uint32_t k = j * kLevelThreads + threadIdx.x;
    if (k < ch.len)
      ord[base + k] = (tot[j * kWarps + w] + __popc(bal[j] & ((1u << lane) - 1u))) |
                      ((bal[j] >> lane & 1u) ? 0x80000000u : 0u);
  }
}

// One warp per node: its chunks' offsets among its lefts; the children that are large become
// nodes of the next level with their chunks, the others jobs of the small-subtree kernel unless
// they are leaves already.
__global__ void __launch_bounds__(32) k_children(LevelNode* nodes, uint32_t* chunk_tot, LevelNode* next, Chunk* nchunks,
                                                 const PoolNode* __restrict__ pool, SmallJob* jobs, uint32_t max_leaf,
                                                 int parity, Counters* ctr) {
  LevelNode& nd = nodes[blockIdx.x];
  if (!nd.split) return;
  const int lane = threadIdx.x;
  uint32_t run = 0;
  for (uint32_t c0 = 0; c0 < nd.nchunks; c0 += 32) {
    const uint32_t c = c0 + lane;
    const uint32_t v = c < nd.nchunks ? chunk_tot[nd.cfirst + c] : 0u;
    uint32_t incl = v;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, off);
      if (lane >= off) incl += y;
    }
    if (c < nd.nchunks) chunk_tot[nd.cfirst + c] = run + incl - v;
    run += __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  for (int s = 0; s < 2; ++s) {
    const uint32_t first = nd.first + (s ? nd.nl : 0u), count = s ? nd.count - nd.nl : nd.nl;
    const uint32_t q = pool[nd.pool].child + s;
    uint32_t where;
    if (count <= max_leaf) {
      where = kFinal;
    } else if (count <= kSmall) {
      where = kToBuffer;
      if (lane == 0)
        jobs[atomicAdd(&ctr->jobs, 1u)] = SmallJob{q, first, count, (nd.depth + 1) | (uint32_t(parity ^ 1) << 31)};
    } else {
      const uint32_t nc = (count + kChunk - 1) / kChunk;
      uint32_t at = 0, cf = 0;
      if (lane == 0) {
        at = atomicAdd(&ctr->nodes[parity ^ 1], 1u);
        cf = atomicAdd(&ctr->chunks[parity ^ 1], nc);
      }
      at = __shfl_sync(0xFFFFFFFFu, at, 0);
      cf = __shfl_sync(0xFFFFFFFFu, cf, 0);
      where = at;
      if (lane == 0) {
        LevelNode& c = next[at];
        c.pool = q;
        c.first = first;
        c.count = count;
        c.depth = nd.depth + 1;
        c.cfirst = cf;
        c.nchunks = nc;
        for (int k = 0; k < 6; ++k) c.ext[k] = k < 3 ? 0xFFFFFFFFu : 0u;
      }
      for (uint32_t k = lane; k < nc; k += 32) nchunks[cf + k] = Chunk{at, k * kChunk, min(kChunk, count - k * kChunk)};
    }
    if (lane == 0) nd.next[s] = where;
  }
}

// each left's ordinal in its node; pos[q] = where the left of ordinal q stands (relative)
__global__ void k_scatter(const LevelNode* __restrict__ nodes, const Chunk* __restrict__ chunks,
                          const uint32_t* __restrict__ chunk_off, uint32_t* ord, uint32_t* pos) {
  const Chunk ch = chunks[blockIdx.x];
  const LevelNode& nd = nodes[ch.node];
  if (!nd.split) return;
  const uint32_t base = nd.first + ch.start;
  for (uint32_t k = threadIdx.x; k < ch.len; k += blockDim.x) {
    const uint32_t o = ord[base + k];
    const uint32_t q = chunk_off[blockIdx.x] + (o & 0x7FFFFFFFu);
    ord[base + k] = q | (o & 0x80000000u);
    if (o & 0x80000000u) pos[nd.first + q] = ch.start + k;
  }
}

// Pointer jumping on pos[] over [0, nl): a misplaced right at p follows p -> pos(p) -> ... to the
// first position >= nl (its final place). A round follows up to kJumpHops links of every chain,
// so that a chain of c links is resolved after ceil(log_9 c) rounds; a round after one that
// left nothing unresolved returns at once.
__global__ void k_jump(const LevelNode* __restrict__ nodes, const Chunk* __restrict__ chunks, uint32_t* pos, int round,
                       Counters* ctr) {
  if (round > 0 && *static_cast<volatile uint32_t*>(&ctr->changed[round - 1]) == 0u) return;
  const Chunk ch = chunks[blockIdx.x];
  const LevelNode& nd = nodes[ch.node];
  if (!nd.split || ch.start >= nd.nl) return;
  uint32_t open = 0;
  volatile uint32_t* p = pos + nd.first;  // other threads shorten the same chains
  for (uint32_t k = threadIdx.x; k < ch.len; k += blockDim.x) {
    const uint32_t q = ch.start + k;
    if (q >= nd.nl) break;
    uint32_t j = p[q];
    if (j < nd.nl && j != q) {  // (a left already in place points at itself: no chain ends there)
      for (int hop = 0; hop < kJumpHops && j < nd.nl; ++hop) j = p[j];
      p[q] = j;
      open |= j < nd.nl ? 1u : 0u;
    }
  }
  if (__syncthreads_or(open) && threadIdx.x == 0) atomicOr(&ctr->changed[round], 1u);
}

// The partition's result written to the next buffer, with the centroid extents of the children
// that are split next; the triangles of final leaves go to their place in the order.
__global__ void __launch_bounds__(kLevelThreads) k_permute(const TriRec* __restrict__ cur, TriRec* __restrict__ nxt,
                                                           uint32_t* __restrict__ order,
                                                           const LevelNode* __restrict__ nodes,
                                                           const Chunk* __restrict__ chunks,
                                                           const uint32_t* __restrict__ ord,
                                                           const uint32_t* __restrict__ pos, LevelNode* next) {
  __shared__ uint32_t red[12];
  const Chunk ch = chunks[blockIdx.x];
  const LevelNode& nd = nodes[ch.node];
  const uint32_t base = nd.first + ch.start;
  if (!nd.split) {
    for (uint32_t k = threadIdx.x; k < ch.len; k += blockDim.x) order[base + k] = __float_as_uint(cur[base + k].c.w);
    return;
  }
  if (threadIdx.x < 12) red[threadIdx.x] = threadIdx.x % 6 < 3 ? 0xFFFFFFFFu : 0u;
  __syncthreads();
  uint32_t r[2][6];
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int q = 0; q < 6; ++q) r[s][q] = q < 3 ? 0xFFFFFFFFu : 0u;
  for (uint32_t k = threadIdx.x; k < ch.len; k += blockDim.x) {
    const TriRec x = cur[base + k];
    const uint32_t i = ch.start + k, o = ord[base + k];
    uint32_t dest;
    if (o & 0x80000000u) dest = o & 0x7FFFFFFFu;  // a left: its ordinal
    else if (i >= nd.nl) dest = i;                // a right already on the right
    else dest = pos[nd.first + i];                // a misplaced right: the end of its chain
    const bool right = dest >= nd.nl;
    const uint32_t where = nd.next[right ? 1 : 0];
    if (where == kFinal) order[nd.first + dest] = __float_as_uint(x.c.w);
    else nxt[nd.first + dest] = x;
#pragma unroll
    for (int s = 0; s < 2; ++s)
      if (right == (s == 1)) {
        r[s][0] = min(r[s][0], f2o(x.c.x)); r[s][1] = min(r[s][1], f2o(x.c.y)); r[s][2] = min(r[s][2], f2o(x.c.z));
        r[s][3] = max(r[s][3], f2o(x.c.x)); r[s][4] = max(r[s][4], f2o(x.c.y)); r[s][5] = max(r[s][5], f2o(x.c.z));
      }
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    if (nd.next[s] >= kToBuffer) continue;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const uint32_t v = q < 3 ? __reduce_min_sync(0xFFFFFFFFu, r[s][q]) : __reduce_max_sync(0xFFFFFFFFu, r[s][q]);
      if ((threadIdx.x & 31u) == 0u) {
        if (q < 3) atomicMin(&red[6 * s + q], v);
        else atomicMax(&red[6 * s + q], v);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int s = threadIdx.x / 6, q = threadIdx.x % 6;
    const uint32_t at = nd.next[s];
    if (at < kToBuffer) {
      if (q < 3) atomicMin(&next[at].ext[q], red[threadIdx.x]);
      else atomicMax(&next[at].ext[q], red[threadIdx.x]);
    }
  }
}

// ---- small subtrees: one warp runs the host's algorithm in shared memory ---------------------
// One thread per subtree (the earlier form) read its triangles from memory one after another,
// 3.1 ms of serial chains for 327,680 triangles; a warp holds them in shared memory, bins with
// shared atomics and evaluates the SAH candidates a lane each: 0.63 ms. 9.5 KB of shared memory
// (16 bins) let 24 warps stand on an SM.
struct SmallShared {
  float4 c[kSmall], lo[kSmall], hi[kSmall];
  uint8_t ord[kSmall], pos[kSmall];  // the current order; the lefts' positions
  uint32_t st_pool[kSmall];          // pending nodes (each holds 2 or more triangles)
  float st_area[kSmall];
  uint16_t st_first[kSmall], st_count[kSmall], st_depth[kSmall];
};
static_assert(kSmall <= 128, "four triangles per lane, 8-bit positions");

__global__ void __launch_bounds__(32) k_small(const SmallJob* __restrict__ jobs, const TriRec* __restrict__ b0,
                                              const TriRec* __restrict__ b1, uint32_t* __restrict__ order,
                                              PoolNode* pool, int B, uint32_t max_leaf, Counters* ctr) {
  __shared__ SmallShared sh;
  extern __shared__ uint32_t sb[];  // 3 * B bins
  const int lane = threadIdx.x;
  const SmallJob jb = jobs[blockIdx.x];
  const TriRec* src = (jb.depth_buf >> 31) ? b1 : b0;
  for (uint32_t k = lane; k < jb.count; k += 32) {
    const TriRec x = src[jb.first + k];
    sh.c[k] = x.c;
    sh.lo[k] = x.lo;
    sh.hi[k] = x.hi;
    sh.ord[k] = uint8_t(k);
  }
  int sp = 1;  // the same in every lane
  if (lane == 0) {
    sh.st_pool[0] = jb.pool;
    sh.st_area[0] = half_area(pool[jb.pool].lo, pool[jb.pool].hi);
    sh.st_first[0] = 0;
    sh.st_count[0] = uint16_t(jb.count);
    sh.st_depth[0] = uint16_t(jb.depth_buf & 0x7FFFFFFFu);
  }
  __syncwarp();
  while (sp > 0) {
    --sp;
    const uint32_t ni = sh.st_pool[sp], first = sh.st_first[sp], count = sh.st_count[sp], depth = sh.st_depth[sp];
    const float leaf_cost = __fmul_rn(sh.st_area[sp], __uint2float_rn(count));
    __syncwarp();
    uint32_t id[4];  // this lane's triangles of the node: positions lane, lane + 32, ...
    uint32_t ext[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t k = lane + 32u * j;
      id[j] = k < count ? sh.ord[first + k] : 0u;
      if (k < count) {
        const float4 c = sh.c[id[j]];
        ext[0] = min(ext[0], f2o(c.x)); ext[1] = min(ext[1], f2o(c.y)); ext[2] = min(ext[2], f2o(c.z));
        ext[3] = max(ext[3], f2o(c.x)); ext[4] = max(ext[4], f2o(c.y)); ext[5] = max(ext[5], f2o(c.z));
      }
    }
    float cmin[3], width[3];
    uint32_t use = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float lo = o2f(__reduce_min_sync(0xFFFFFFFFu, ext[a])), hi = o2f(__reduce_max_sync(0xFFFFFFFFu, ext[3 + a]));
      cmin[a] = lo;
      width[a] = __fdiv_rn(__fsub_rn(hi, lo), float(B));
      if (!(lo == hi)) use |= 1u << a;
    }
    for (int k = lane; k < 3 * B; k += 32) clear_bin(sb + kBinWords * k);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (lane + 32u * j < count) {
        const float4 c = sh.c[id[j]], lo = sh.lo[id[j]], hi = sh.hi[id[j]];
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if (use & (1u << a)) add_to_bin(sb + kBinWords * (a * B + bin_of(comp(c, a), cmin[a], width[a], B)), lo, hi);
      }
    __syncwarp();
    int axis = 0, boundary = 0;
    if (!best_split(sb, B, use, leaf_cost, axis, boundary)) continue;
    // forward-swap partition by bin index (bvh.rs:260-267), resolved as in the level kernels
    const float bm = axis == 0 ? cmin[0] : (axis == 1 ? cmin[1] : cmin[2]);
    const float bw = axis == 0 ? width[0] : (axis == 1 ? width[1] : width[2]);
    uint32_t bal[4], before = 0, nl = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool left = lane + 32u * j < count && bin_of(comp(sh.c[id[j]], axis), bm, bw, B) <= boundary;
      bal[j] = __ballot_sync(0xFFFFFFFFu, left);
      nl += __popc(bal[j]);
    }
    uint32_t dest[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      dest[j] = lane + 32u * j;
      if (bal[j] >> lane & 1u) {
        dest[j] = before + __popc(bal[j] & ((1u << lane) - 1u));
        sh.pos[dest[j]] = uint8_t(lane + 32 * j);
      }
      before += __popc(bal[j]);
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (!(bal[j] >> lane & 1u) && lane + 32u * j < count)
        while (dest[j] < nl) dest[j] = sh.pos[dest[j]];  // positions only grow: at most `count` links
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (lane + 32u * j < count) sh.ord[first + dest[j]] = uint8_t(id[j]);
    uint32_t c = 0;
    if (lane == 0) c = atomicAdd(&ctr->pool, 2u);
    c = __shfl_sync(0xFFFFFFFFu, c, 0);
    const float box = child_box(sb, B, axis, boundary);
    float lo[2][3], hi[2][3];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        lo[s][q] = __shfl_sync(0xFFFFFFFFu, box, 6 * s + q);
        hi[s][q] = __shfl_sync(0xFFFFFFFFu, box, 6 * s + 3 + q);
      }
    if (lane < 2) {
      PoolNode p;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        p.lo[q] = lane ? lo[1][q] : lo[0][q];
        p.hi[q] = lane ? hi[1][q] : hi[0][q];
      }
      p.first = jb.first + first + (lane ? nl : 0u);
      p.count = lane ? count - nl : nl;
      p.depth = depth + 1;
      p.child = kNone;
      pool[c + lane] = p;
    }
    if (lane == 0) {
      pool[ni].child = c;
      pool[ni].count = 0;
    }
#pragma unroll
    for (int s = 1; s >= 0; --s) {
      const uint32_t cc = s ? count - nl : nl;
      if (cc > max_leaf) {  // (pending nodes hold disjoint triangles: never more than kSmall of them)
        if (lane == 0) {
          sh.st_pool[sp] = c + s;
          sh.st_area[sp] = half_area(lo[s], hi[s]);
          sh.st_first[sp] = uint16_t(first + (s ? nl : 0u));
          sh.st_count[sp] = uint16_t(cc);
          sh.st_depth[sp] = uint16_t(depth + 1);
        }
        ++sp;
      }
    }
    __syncwarp();
  }
  __syncwarp();
  for (uint32_t k = lane; k < jb.count; k += 32) order[jb.first + k] = __float_as_uint(sh.c[sh.ord[k]].w);
}

__global__ void k_identity(uint32_t* order, uint32_t n) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) order[i] = i;
}

// ---- depth-first renumbering and the GPU layout -----------------------------------------------
// Nodes grouped by depth. Every node adds to one of a few dozen counters, so the lanes of a
// warp that share a depth (neighbouring nodes usually do) add once, together; the order
// within a depth does not matter to the sizes and numbers computed from it.
__global__ void k_depth_hist(const PoolNode* __restrict__ pool, uint32_t n, uint32_t* hist) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t dep = min(pool[i].depth, 255u);
    const unsigned peers = __match_any_sync(__activemask(), dep);
    if ((threadIdx.x & 31u) == unsigned(__ffs(peers) - 1)) atomicAdd(hist + dep, uint32_t(__popc(peers)));
  }
}
__global__ void k_depth_scatter(const PoolNode* __restrict__ pool, uint32_t n, uint32_t* cursor, uint32_t* by_depth) {
  const unsigned lane = threadIdx.x & 31u;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t dep = min(pool[i].depth, 255u);
    const unsigned peers = __match_any_sync(__activemask(), dep);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (int(lane) == leader) base = atomicAdd(cursor + dep, uint32_t(__popc(peers)));
    base = __shfl_sync(peers, base, leader);
    by_depth[base + __popc(peers & ((1u << lane) - 1u))] = i;
  }
}
// subtree sizes, deepest level first; and how many of a subtree's nodes become wide nodes (`wide`:
// this level's interior nodes do)
__global__ void k_sizes(const PoolNode* __restrict__ pool, const uint32_t* __restrict__ ids, uint32_t n, uint32_t wide,
                        uint32_t* size, uint32_t* wsize) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t i = ids[k];
  const uint32_t c = pool[i].child;
  size[i] = c == kNone ? 1u : 1u + size[c] + size[c + 1];
  wsize[i] = c == kNone ? 0u : wide + wsize[c] + wsize[c + 1];
}
// depth-first indexes, root level first: a node's children take the next two free indexes,
// its left subtree's descendants follow, then the right's; wide nodes likewise, the node itself first
__global__ void k_number(const PoolNode* __restrict__ pool, const uint32_t* __restrict__ ids, uint32_t n, uint32_t wide,
                         const uint32_t* __restrict__ size, const uint32_t* __restrict__ wsize, uint32_t* ref,
                         uint32_t* cbase, uint32_t* wbase) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t i = ids[k];
  const uint32_t c = pool[i].child;
  if (c == kNone) return;
  const uint32_t b = cbase[i];
  ref[c] = b;
  ref[c + 1] = b + 1;
  cbase[c] = b + 2;
  cbase[c + 1] = b + 2 + (size[c] - 1u);
  wbase[c] = wbase[i] + wide;
  wbase[c + 1] = wbase[c] + wsize[c];
}
__global__ void k_layout(const PoolNode* __restrict__ pool, uint32_t n, const uint32_t* __restrict__ ref,
                         const uint32_t* __restrict__ wbase, GpuNode* out, uint32_t* wide_id, uint32_t* stats) {
  uint32_t leaves = 0, most = 0, deepest = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const PoolNode& p = pool[i];
    const uint32_t r = ref[i];
    GpuNode g;
    for (int a = 0; a < 3; ++a) {
      g.bmin[a] = p.lo[a];
      g.bmax[a] = p.hi[a];
    }
    if (p.child == kNone) {
      g.left_first = p.first;
      g.count = p.count;
      leaves++;
      most = max(most, p.count);
    } else {
      g.left_first = ref[p.child] + 1;
      g.count = 0;
    }
    deepest = max(deepest, p.depth);
    out[r == 0 ? 0 : r + 1] = g;
    wide_id[r == 0 ? 0 : r + 1] = p.child != kNone && (p.depth & 1u) ? wbase[i] : kNoWide;
  }
  leaves = __reduce_add_sync(0xFFFFFFFFu, leaves);  // one atomic per warp and figure
  most = __reduce_max_sync(0xFFFFFFFFu, most);
  deepest = __reduce_max_sync(0xFFFFFFFFu, deepest);
  if ((threadIdx.x & 31u) == 0u) {
    atomicAdd(stats, leaves);
    atomicMax(stats + 1, most);
    atomicMax(stats + 2, deepest);
  }
}

// the triangles in leaf order, with their precomputed edges (mesh_bvh.hpp)
__global__ void k_tri_layout(const uint32_t* __restrict__ order, uint32_t n, const float* __restrict__ v,
                             const uint32_t* __restrict__ idx, float4* tri, float2* tc) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const uint32_t t = order[k];
    const float* p0 = v + 3 * size_t(idx[3 * size_t(t)]);
    const float* p1 = v + 3 * size_t(idx[3 * size_t(t) + 1]);
    const float* p2 = v + 3 * size_t(idx[3 * size_t(t) + 2]);
    const float e1[3] = {__fsub_rn(p1[0], p0[0]), __fsub_rn(p1[1], p0[1]), __fsub_rn(p1[2], p0[2])};
    const float e2[3] = {__fsub_rn(p2[0], p0[0]), __fsub_rn(p2[1], p0[1]), __fsub_rn(p2[2], p0[2])};
    tri[2 * size_t(k)] = make_float4(p0[0], p0[1], p0[2], e1[0]);
    tri[2 * size_t(k) + 1] = make_float4(e1[1], e1[2], e2[0], e2[1]);
    tc[k] = make_float2(e2[2], __uint_as_float(t));
  }
}

// ---- host driver ------------------------------------------------------------------------------
struct Scratch {
  cudaStream_t st;
  cudaMemPool_t mem;
  std::vector<void*> ptrs;
  Scratch(cudaStream_t s, cudaMemPool_t m) : st(s), mem(m) {}
  ~Scratch() {
    for (void* p : ptrs) cudaFreeAsync(p, st);
  }
  template <class T>
  cudaError_t alloc(T** p, size_t count) {
    const cudaError_t e = keep(p, count);
    if (e == cudaSuccess) ptrs.push_back(*p);
    return e;
  }
  template <class T>
  cudaError_t keep(T** p, size_t count) {  // not freed here
    void* q = nullptr;
    const cudaError_t e = cudaMallocFromPoolAsync(&q, std::max<size_t>(count, 1) * sizeof(T), mem, st);
    *p = static_cast<T*>(q);
    return e;
  }
};

#define BUILD_TRY(x)                                                                  \
  do {                                                                                \
    const cudaError_t e_ = (x);                                                       \
    if (e_ != cudaSuccess) {                                                          \
      *err = std::string("device BVH build: ") + cudaGetErrorString(e_) + " at " #x; \
      return false;                                                                   \
    }                                                                                 \
  } while (0)

const char* const kBadInput = "a triangle vertex index out of range or a non-finite vertex coordinate";

unsigned grid_for(uint64_t n, int threads, int sm_count) {
  const uint64_t want = (n + threads - 1) / threads;
  const uint64_t cap = uint64_t(sm_count) * 16;
  return unsigned(std::max<uint64_t>(1, std::min(want, cap)));
}

}  // namespace

bool build_mesh_bvh_device(const float* d_v, uint32_t nv, const uint32_t* d_idx, uint32_t n,
                           const MeshBuildParams& p, cudaStream_t st, cudaMemPool_t mem, int sm_count,
                           DeviceMeshBuild* out, std::string* err) {
  *out = DeviceMeshBuild{};
  if (n == 0) { *err = "a TriangleMesh needs at least one triangle"; return false; }
  if (p.bins < 2 || p.bins > kMaxBins) { *err = "bvh_bins must be in [2, 64]"; return false; }
  const int B = p.bins;
  Scratch s(st, mem);
  // large nodes hold more than kSmall triangles each; a job at least two
  const size_t cap_nodes = size_t(n) / (kSmall + 1) + 1, cap_chunks = size_t(n) / kChunk + cap_nodes + 1;
  TriRec* bufs[2];
  PoolNode* pool;
  LevelNode* nodes[2];
  Chunk* chunks[2];
  SmallJob* jobs;
  uint32_t *ord, *pos, *ctot, *bins;
  Counters* ctr;
  for (int k = 0; k < 2; ++k) {
    BUILD_TRY(s.alloc(&bufs[k], n));
    BUILD_TRY(s.alloc(&nodes[k], cap_nodes));
    BUILD_TRY(s.alloc(&chunks[k], cap_chunks));
  }
  BUILD_TRY(s.alloc(&pool, size_t(2) * n));
  BUILD_TRY(s.alloc(&ord, n));
  BUILD_TRY(s.alloc(&pos, n));
  BUILD_TRY(s.alloc(&ctot, cap_chunks));
  BUILD_TRY(s.alloc(&bins, cap_nodes * 3 * B * kBinWords));
  BUILD_TRY(s.alloc(&jobs, size_t(n) / 2 + 1));
  BUILD_TRY(s.alloc(&ctr, 1));
  Counters h{};
  h.pool = 1;
  for (int q = 0; q < 3; ++q) h.root_box[q] = h.vertex_box[q] = 0xFFFFFFFFu;
  BUILD_TRY(cudaMemcpyAsync(ctr, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  k_tri_prep<<<grid_for(n, 256, sm_count), 256, 0, st>>>(d_v, nv, d_idx, n, bufs[0], &ctr->err);
  k_vertex_bounds<<<grid_for(nv, kLevelThreads, sm_count), kLevelThreads, 0, st>>>(d_v, nv, ctr->vertex_box, &ctr->err);
  k_root_box<<<grid_for(n, kLevelThreads, sm_count), kLevelThreads, 0, st>>>(bufs[0], n, ctr->root_box);
  k_root_node<<<1, 1, 0, st>>>(pool, ctr->root_box, n);
  DeviceMeshBuild o{};
  struct Outputs {  // freed unless the build succeeds
    DeviceMeshBuild* b;
    ~Outputs() {
      if (b) free_device_mesh_build(b);
    }
  } guard{&o};
  BUILD_TRY(s.keep(&o.tri_index, n));

  // large nodes, level by level; `small` jobs follow
  int cur = 0;
  uint32_t nn = 0, nc = 0, nj = 0;
  if (n > kSmall && n > p.max_leaf) {
    nn = 1;
    nc = (n + kChunk - 1) / kChunk;
    k_root_level<<<grid_for(nc, 128, sm_count), 128, 0, st>>>(nodes[0], chunks[0], n, ctr);
    k_ext<<<nc, kLevelThreads, 0, st>>>(bufs[0], nodes[0], chunks[0]);
  } else if (n > p.max_leaf) {
    nj = 1;
    const SmallJob root{0, 0, n, 1};
    BUILD_TRY(cudaMemcpyAsync(jobs, &root, sizeof(root), cudaMemcpyHostToDevice, st));
    BUILD_TRY(cudaStreamSynchronize(st));  // `root` is on the stack
  } else {
    k_identity<<<grid_for(n, 256, sm_count), 256, 0, st>>>(o.tri_index, n);
  }
  BUILD_TRY(cudaGetLastError());
  uint32_t longest = n;  // no chain of a level is longer than its largest node
  for (int level = 0; nn > 0; ++level) {
    if (level >= 256) { *err = "device BVH build: the tree is deeper than 254 levels"; return false; }
    BUILD_TRY(cudaMemsetAsync(ctr->changed, 0, sizeof(ctr->changed), st));
    BUILD_TRY(cudaMemsetAsync(&ctr->nodes[cur ^ 1], 0, sizeof(uint32_t), st));
    BUILD_TRY(cudaMemsetAsync(&ctr->chunks[cur ^ 1], 0, sizeof(uint32_t), st));
    k_bin_prep<<<nn, 64, 0, st>>>(nodes[cur], bins, B);
    k_bins<<<nc, kLevelThreads, 0, st>>>(bufs[cur], nodes[cur], chunks[cur], bins, B);
    k_sah<<<nn, 32, 0, st>>>(nodes[cur], bins, B, pool, ctr);
    k_classify<<<nc, kLevelThreads, 0, st>>>(bufs[cur], nodes[cur], chunks[cur], ord, ctot, B);
    k_children<<<nn, 32, 0, st>>>(nodes[cur], ctot, nodes[cur ^ 1], chunks[cur ^ 1], pool, jobs, p.max_leaf, cur, ctr);
    k_scatter<<<nc, kLevelThreads, 0, st>>>(nodes[cur], chunks[cur], ctot, ord, pos);
    int rounds = 1;
    for (uint64_t reach = kJumpHops + 1; reach < longest; reach *= kJumpHops + 1) ++rounds;
    for (int r = 0; r < rounds; ++r) k_jump<<<nc, kLevelThreads, 0, st>>>(nodes[cur], chunks[cur], pos, r, ctr);
    k_permute<<<nc, kLevelThreads, 0, st>>>(bufs[cur], bufs[cur ^ 1], o.tri_index, nodes[cur], chunks[cur], ord, pos,
                                            nodes[cur ^ 1]);
    BUILD_TRY(cudaGetLastError());
    BUILD_TRY(cudaMemcpyAsync(&h, ctr, sizeof(h), cudaMemcpyDeviceToHost, st));
    BUILD_TRY(cudaStreamSynchronize(st));
    if (h.err & kBuildErrInput) {
      *err = kBadInput;
      return false;
    }
    cur ^= 1;
    nn = h.nodes[cur];
    nc = h.chunks[cur];
    nj = h.jobs;
    if (nn > cap_nodes || nc > cap_chunks) { *err = "device BVH build: a level outgrew its buffers"; return false; }
  }
  if (nj > 0) {
    k_small<<<nj, 32, size_t(3) * B * kBinWords * sizeof(uint32_t), st>>>(jobs, bufs[0], bufs[1], o.tri_index, pool, B,
                                                                         p.max_leaf, ctr);
    BUILD_TRY(cudaGetLastError());
  }
  BUILD_TRY(cudaMemcpyAsync(&h, ctr, sizeof(h), cudaMemcpyDeviceToHost, st));
  BUILD_TRY(cudaStreamSynchronize(st));
  if (h.err & kBuildErrInput) {
    *err = kBadInput;
    return false;
  }
  const uint32_t made = h.pool;  // nodes

  // renumbering: nodes grouped by depth, subtree sizes bottom-up, indexes top-down
  uint32_t *hist, *by_depth, *size, *wsize, *ref, *cbase, *wbase, *stats;
  BUILD_TRY(s.alloc(&hist, 512));
  BUILD_TRY(s.alloc(&by_depth, made));
  BUILD_TRY(s.alloc(&size, made));
  BUILD_TRY(s.alloc(&wsize, made));
  BUILD_TRY(s.alloc(&ref, made));
  BUILD_TRY(s.alloc(&cbase, made));
  BUILD_TRY(s.alloc(&wbase, made));
  BUILD_TRY(s.alloc(&stats, 4));
  BUILD_TRY(cudaMemsetAsync(hist, 0, 512 * sizeof(uint32_t), st));
  k_depth_hist<<<grid_for(made, 256, sm_count), 256, 0, st>>>(pool, made, hist);
  uint32_t hh[256];
  BUILD_TRY(cudaMemcpyAsync(hh, hist, sizeof(hh), cudaMemcpyDeviceToHost, st));
  BUILD_TRY(cudaStreamSynchronize(st));
  if (hh[255]) { *err = "device BVH build: the tree is deeper than 254 levels"; return false; }
  uint32_t off[257];
  off[0] = 0;
  uint32_t maxd = 0;
  for (int d = 0; d < 256; ++d) {
    off[d + 1] = off[d] + hh[d];
    if (hh[d]) maxd = uint32_t(d);
  }
  BUILD_TRY(cudaMemcpyAsync(hist + 256, off, 256 * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  k_depth_scatter<<<grid_for(made, 256, sm_count), 256, 0, st>>>(pool, made, hist + 256, by_depth);
  for (uint32_t d = maxd; d >= 1; --d) {
    const uint32_t cnt = hh[d];
    if (cnt) k_sizes<<<(cnt + 255) / 256, 256, 0, st>>>(pool, by_depth + off[d], cnt, d & 1u, size, wsize);
  }
  const uint32_t zero = 0, one = 1;
  BUILD_TRY(cudaMemcpyAsync(ref, &zero, sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  BUILD_TRY(cudaMemcpyAsync(cbase, &one, sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  BUILD_TRY(cudaMemcpyAsync(wbase, &zero, sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  for (uint32_t d = 1; d <= maxd; ++d) {
    const uint32_t cnt = hh[d];
    if (cnt)
      k_number<<<(cnt + 255) / 256, 256, 0, st>>>(pool, by_depth + off[d], cnt, d & 1u, size, wsize, ref, cbase, wbase);
  }
  BUILD_TRY(cudaGetLastError());

  // outputs
  BUILD_TRY(s.keep(&o.nodes, size_t(made) + 1));
  BUILD_TRY(s.keep(&o.wide_id, size_t(made) + 1));
  o.node_slots = uint64_t(made) + 1;
  BUILD_TRY(s.keep(&o.tri, size_t(n) * 2));
  BUILD_TRY(s.keep(&o.tri_c, n));
  BUILD_TRY(cudaMemsetAsync(o.nodes + 1, 0, sizeof(GpuNode), st));  // the padding slot
  BUILD_TRY(cudaMemsetAsync(stats, 0, 4 * sizeof(uint32_t), st));
  BUILD_TRY(cudaMemcpyAsync(stats + 3, wsize, sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  k_layout<<<grid_for(made, 256, sm_count), 256, 0, st>>>(pool, made, ref, wbase, o.nodes, o.wide_id, stats);
  k_tri_layout<<<grid_for(n, 256, sm_count), 256, 0, st>>>(o.tri_index, n, d_v, d_idx, o.tri, o.tri_c);
  BUILD_TRY(cudaGetLastError());
  uint32_t hs[4] = {0, 0, 0, 0};
  BUILD_TRY(cudaMemcpyAsync(hs, stats, sizeof(hs), cudaMemcpyDeviceToHost, st));
  BUILD_TRY(cudaStreamSynchronize(st));
  o.stats.node_count = made;
  o.stats.leaf_count = hs[0];
  o.stats.max_leaf_tris = hs[1];
  o.stats.max_depth = hs[2];
  o.wide_count = hs[3];
  for (int a = 0; a < 3; ++a) {
    auto dec = [](uint32_t x) {
      const uint32_t u = (x & 0x80000000u) ? (x & 0x7FFFFFFFu) : ~x;
      float f;
      std::memcpy(&f, &u, sizeof(f));
      return f == 0.0f ? 0.0f : f;
    };
    o.bounds_min[a] = dec(h.vertex_box[a]);
    o.bounds_max[a] = dec(h.vertex_box[3 + a]);
  }
  guard.b = nullptr;
  *out = o;
  return true;
}

void free_device_mesh_build(DeviceMeshBuild* b) {
  cudaFree(b->v);
  cudaFree(b->idx);
  cudaFree(b->nodes);
  cudaFree(b->tri);
  cudaFree(b->tri_c);
  cudaFree(b->tri_index);
  cudaFree(b->wide_id);
  *b = DeviceMeshBuild{};
}

}  // namespace pbrt
