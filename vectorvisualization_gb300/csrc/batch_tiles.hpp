// Pixels of a batch tile's lanes (batch.cuh).  Plain C++, so that a host compiler can test the mapping.
#pragma once

#ifdef __CUDACC__
#define VVLIC_HOST_DEVICE_INLINE __host__ __device__ __forceinline__
#else
#define VVLIC_HOST_DEVICE_INLINE inline
#endif

namespace vvlic {

struct BatchPixel {
  int x, y;
};

// Pixel of ray r (0..7) of group sub (0..3) of a tile `tw` pixels wide (8, 4, 16 or 32; 32 pixels in all), tile
// `tile` of an image of tiles_x tiles across: groups of 4x2 rays, 8x1 in one-row tiles.
VVLIC_HOST_DEVICE_INLINE BatchPixel batch_pixel(int tw, unsigned tile, int tiles_x, int sub, int r) {
  constexpr int R = 8;
  const int th = 32 / tw, gw = th == 1 ? R : 4, gx = tw / gw;
  return {(int)(tile % tiles_x) * tw + (sub % gx) * gw + r % gw, (int)(tile / tiles_x) * th + (sub / gx) * (R / gw) + r / gw};
}

}  // namespace vvlic
