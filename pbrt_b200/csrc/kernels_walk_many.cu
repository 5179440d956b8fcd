// kernels_walk_many.cu — the walks of a wave over a batch's scene table.
#include "walk_kernels.cuh"

namespace pbrt {

cudaError_t launch_nearest(const WaveBuffers& w, const ManyScenes& src, const uint32_t* q, const uint32_t* qcount,
                           uint32_t* fetch, uint32_t* next_count, const WalkLaunch& l) {
  return launch_nearest_for(w, src, q, qcount, fetch, next_count, l);
}

cudaError_t launch_shadow(const WaveBuffers& w, const ManyScenes& src, uint32_t* fetch, const WalkLaunch& l) {
  return launch_shadow_for(w, src, fetch, l);
}

}  // namespace pbrt
