// Multi-view batch: scratch layout shared by the batched kernels.
#pragma once
#include <cstdint>
#include "../../include/stratum.h"
#include "shading.cuh"

namespace st {

constexpr int kTileW = 8, kTileH = 4;  // one warp per 8x4 pixel tile

// Scratch: 16 u32 counters, the resolve taps, then one FrameConst per view.
enum : int {
  kTraceNext = 0,   // next tile to claim (trace)
  kTraceDone = 1,   // warps that found the queue empty (trace)
  kShadeNext = 2,
  kShadeDone = 3,
  kTotalTiles = 4,  // tiles over all views (written by the prologue)
  kResolveNext = 5,
  kResolveDone = 6,
  kLightNext = 7,
  kLightDone = 8,
  kBandTiles = 9,   // band tiles over all views (written by the prologue)
  kCounters = 16
};
// The trace draws a band of tile rows around the horizon first, in tiles one
// pixel high, then everything else in whole tiles, nearest the horizon first.
// A ray near the horizon crosses the most lots: the slowest tiles took 1 ms where
// the mean took 25 us, so a frame waited for the few that were claimed late, and
// a frame of fewer tiles than the device holds warps waited for its slowest tile.
struct Band {
  int base;        // first of the view's band tiles
  int row0, row1;  // the band's tile rows
  int horizon;     // pixel row of the horizon, inside the frame
};
struct ViewFrame {
  FrameConst frame;
  Band band;
};
struct BatchScratch {
  uint32_t counters[kCounters];
  ResolveTaps taps;
  ViewFrame view[1];  // n entries
};
constexpr size_t batchScratchBytes(int views) {
  return sizeof(BatchScratch) + size_t(views > 1 ? views - 1 : 0) * sizeof(ViewFrame);
}

// Tile count of a view under an order: row-major tiles, or whole 4x4-tile
// super-tiles (Morton order inside each) whose out-of-frame tiles are skipped.
SD int tileCount(int width, int height, int order) {
  int tx = (width + kTileW - 1) / kTileW, ty = (height + kTileH - 1) / kTileH;
  if (order == 1) return ((tx + 3) / 4) * ((ty + 3) / 4) * 16;
  return tx * ty;
}
// Rows in the order of their distance from row `h` (0 <= k, h < rows): h, then
// its neighbours on either side by turns, then what is left of the longer side.
HD int nearRow(int k, int h, int rows) {
  const int side = h < rows - 1 - h ? h : rows - 1 - h;
  if (k <= 2 * side) return (k & 1) ? h + (k + 1) / 2 : h - k / 2;
  return side == h ? k : rows - 1 - k;
}
// The pixel row the camera's horizon falls on, kept inside the frame.
SD int horizonRow(const Camera& c, int height) {
  const float sy = -c.fwd.y / c.up.y, y = 0.5f * float(height) - 0.5f - c.jy - sy * float(height) / 1.08f;
  return int(fminf(fmaxf(y, 0.0f), float(height - 1)));  // NaN (looking straight down): 0
}

// Tile `local` of a view: row-major, or super-tile rows of Morton-ordered
// super-tiles; with `first` >= 0 the (super-)rows in the order of their distance
// from tile row `first`.
SD bool tileCoord(int local, int tilesX, int tilesY, int order, int& tx, int& ty, int first = -1) {
  if (order == 1) {
    int st = local >> 4, w = local & 15, superX = (tilesX + 3) / 4, row = st / superX;
    if (first >= 0) row = nearRow(row, first / 4, (tilesY + 3) / 4);
    tx = (st % superX) * 4 + ((w & 1) | ((w >> 1) & 2));
    ty = row * 4 + (((w >> 1) & 1) | ((w >> 2) & 2));
  } else {
    tx = local % tilesX;
    ty = local / tilesX;
    if (first >= 0) ty = nearRow(ty, first, tilesY);
  }
  return tx < tilesX && ty < tilesY;
}
SD int bandCount(const Band& b, int tilesX, int height) {
  return (min(b.row1 * kTileH, height) - b.row0 * kTileH) * tilesX;
}

// Last view whose first tile is <= tile (binary search; warp-uniform).
SD int viewOf(const stratum_view* __restrict__ V, int n, int tile) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (V[mid].tileBase <= tile) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Claim `grab` tiles for this warp; returns the first, or >= total when empty.
SD int claim(uint32_t* next, int grab) {
  int t0 = 0;
  if ((threadIdx.x & 31) == 0) t0 = int(atomicAdd(next, uint32_t(grab)));
  return __shfl_sync(0xffffffffu, t0, 0);
}
// The last warp to see the queue empty resets it for the next launch.
SD void retire(uint32_t* next, uint32_t* done, int threads) {
  if ((threadIdx.x & 31) == 0) {
    __threadfence();
    uint32_t warps = gridDim.x * uint32_t(threads / 32);
    if (atomicAdd(done, 1u) == warps - 1) { *next = 0u; *done = 0u; }
  }
}

// Blocks of a kernel that the current device holds.
template <class K>
inline int residentBlocks(K kernel, int threads, size_t smem = 0) {
  int dev = 0, sms = 148, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
  return sms * (per > 0 ? per : 1);
}

// The block-pooled trace of at most kPoolViews views, with the device's ordinal (pooled.cu).
constexpr int kPoolViews = 4095, kGridDevices = 64;
template <int THREADS>
void launchPooled(const stratum_view* V, int n, int order, BatchScratch* S, int dev, cudaStream_t stream);

}  // namespace st
