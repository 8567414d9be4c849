// How the drop-in shading covers a strip of rows, shared by the procedural (shade.cu) and
// the surrogate form (neural.cu): warps take 8x4-pixel tiles.
//
// A strip of at most one wave (1,024 threads an SM, the 64 registers of the kernels that do
// both halves of a pixel) is shaded by one launch, a warp a tile: there the time is one
// pixel's chain and the launches, not the code's size.  More is shaded in two launches,
// material and light, of grids the device holds.  Street, aerial and avenue views together
// by two launches and by one: 64x36 139 / 114 us, 320x180 145 / 122, 500x281 (4,473 tiles of
// 4,736) 163 / 156, 560x315 (5,530) 176 / 178, 640x360 194 / 210, 1600x900 790 / 952; in
// 64-row strips 640x360 579 / 420, 1600x900 1,593 / 1,316.
#pragma once
#include <mutex>

#include "common_api.cuh"
#include "frame_init.cuh"

namespace st {

constexpr int kShadeThreads = 128;

// Tile `i` of a strip of rows: whether this lane has a pixel there, and which.
SD bool stripPixel(int i, int tilesX, int width, int rowStart, int rowEnd, int& x, int& y) {
  const int lane = int(threadIdx.x & 31);
  x = (i % tilesX) * 8 + (lane & 7);
  y = rowStart + (i / tilesX) * 4 + (lane >> 3);
  return x < width && y < rowEnd;
}

// Blocks that cover a strip, a warp a tile.
inline int tileBlocks(int width, int rows) {
  return ((width + 7) / 8 * ((rows + 3) / 4) + kShadeThreads / 32 - 1) / (kShadeThreads / 32);
}
inline int tileBlocks(int width, int rows, int most) {
  const int need = tileBlocks(width, rows);
  return need < most ? need : most;
}
// Blocks of one wave at 1,024 threads an SM on the current device, asked for once; 0 if
// there is none.
inline int shadeWave() {
  constexpr int kDevices = 64;
  static std::once_flag once[kDevices];
  static int blocks[kDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
  std::call_once(once[dev], [dev] {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    blocks[dev] = sms * (1024 / kShadeThreads);
  });
  return blocks[dev];
}

}  // namespace st
