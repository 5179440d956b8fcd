// cache.hpp — the radiance cache object behind the C ABI's pbrt_cache handle (host code).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <initializer_list>
#include <vector>

#include "../../include/pbrt_b200.h"
#include "mlp.hpp"
#include "render.hpp"

struct pbrt_cache {
  pbrt_ctx* ctx = nullptr;
  pbrt_cache_params params{};
  float *w = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr, *loss = nullptr;
  uint16_t *wfwd = nullptr, *wbwd = nullptr;
  float *partials = nullptr, *tile_loss = nullptr;
  uint32_t tile_cap = 0;
  uint32_t step = 0;
  uint64_t rounds = 0;  // training rounds run by cached renders (keys their path streams)

  // the cached render's training vertices and one training batch (its queries are the context's)
  void* train_block = nullptr;
  uint32_t bcap = 0;
  pbrt::CacheWave cw{};
  float *brec = nullptr, *btgt = nullptr;
  int ensure_train_buffers(uint32_t train_vertices, uint32_t batch);
  // the weights a frame reads while training rounds beside it update them
  uint16_t* wsnap = nullptr;

  int take_bytes(void** p, size_t bytes);
  template <class T>
  int take(T** p, size_t bytes) {
    return take_bytes(reinterpret_cast<void**>(p), bytes);
  }
  void give_back(std::initializer_list<void*> blocks);
  int device_arrays();
  int ensure_tiles(uint32_t tiles);
  int reset();
  pbrt::mlp::Bounds bounds() const;
  int gradient_device(const float* records, const float* targets, uint64_t n, cudaStream_t s);
  int adam_device(cudaStream_t s, const uint32_t* active = nullptr);
  int query_device(const float* records, uint64_t n, float* rgb, cudaStream_t s);
  void release();
};
