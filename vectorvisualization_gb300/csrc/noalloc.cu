// Noise-gradient precompute that allocates nothing, for callers that may not allocate device memory
// at that point: a host application that reserves its whole GPU memory budget up front (a render or
// simulation host embedding this library as a plugin), or a frame loop that cannot take allocator
// latency.  The gradient kernel keeps its raw gradients in shared memory, so this is
// vvlic_noise_gradients_device with the entry point's own limits, and calls on different streams or
// threads are independent.
//
// Compiled with -fmad=false like preprocess.cu.
#include <cuda_runtime.h>

#include "../../include/vvlic.h"
#include "vvlic_host.hpp"
#include "vvlic_launch.hpp"

extern "C" vvlic_status vvlic_noise_gradients_device_noalloc(const uint8_t* d_noise, int32_t mx, int32_t my,
                                                            int32_t mz, int32_t mode, const float* slice_dist,
                                                            uint8_t* d_rgba, void* stream) {
  if (!d_noise || !d_rgba) return VVLIC_ERR_INVALID_ARGUMENT;
  if (mode != VVLIC_NOISE_GRAD_SOBEL && mode != VVLIC_NOISE_GRAD_CENTRAL) return VVLIC_ERR_INVALID_ARGUMENT;
  // two voxels per axis (the border differences read the +1 neighbour) and the fixed maximum
  if (mx < 2 || my < 2 || mz < 2) return VVLIC_ERR_INVALID_ARGUMENT;
  if ((uint64_t)mx * (uint64_t)my * (uint64_t)mz > (uint64_t)VVLIC_NOALLOC_MAX_VOXELS) return VVLIC_ERR_INVALID_ARGUMENT;
  float sd[3] = {1.f, 1.f, 1.f};
  if (slice_dist)
    for (int i = 0; i < 3; ++i) sd[i] = slice_dist[i];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return VVLIC_ERR_NO_DEVICE;
  float w27[27];
  vvlic::noise_filter_weights(w27);
  const int m[3] = {mx, my, mz};
  const cudaError_t e = vvlic::launch_noise_gradients(d_noise, m, mode, sd, d_rgba, w27, (cudaStream_t)stream);
  return e == cudaSuccess ? VVLIC_OK : VVLIC_ERR_CUDA;
}
