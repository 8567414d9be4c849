// shadePixels and resolveFrame drop-ins (kernels/shade.cu:45-123 of the
// reference).
//
// Warps take 8x4-pixel tiles, strided over a grid the device holds at once, and a
// block works out the frame's constants once, an angle a lane: with 64-pixel
// blocks of a wave each, every block waited for one thread's eight double sines.
// Material and light are two kernels, as in the batched path (albedo into Linear,
// then lit in place): half the code for the instruction cache; short strips are shaded by
// one (strips.cuh).  One 1600x900 frame
// (mean of six poses): shade 275 us in one kernel of 8x8 blocks, now 220 us; resolve
// 118 us, now 89 us.
#include <mutex>

#include "shading.cuh"
#include "strips.cuh"

namespace st {

__global__ void __launch_bounds__(kShadeThreads, 1280 / kShadeThreads)
    albedoPixelsK(const float* __restrict__ W, const uint32_t* __restrict__ O, const float* __restrict__ C,
                  const float4* __restrict__ Hit, const float4* __restrict__ Surface, float4* Linear, int width,
                  int height, int rowStart, int rowEnd) {
  __shared__ FrameConst F;
  frameInit(F, C, O);
  const int tilesX = (width + 7) / 8, tiles = tilesX * ((rowEnd - rowStart + 3) / 4), warps = kShadeThreads / 32;
#pragma unroll 1
  for (int i = int(blockIdx.x) * warps + int(threadIdx.x >> 5); i < tiles; i += int(gridDim.x) * warps) {
    int x, y;
    if (!stripPixel(i, tilesX, width, rowStart, rowEnd, x, y)) continue;
    const size_t b = size_t(y) * width + x;
    const float4 h = Hit[b];
    const f3 rd = primaryDir(F.cam, x, y, width, height);
    f3 c;
    if (int(h.y) == kSkyId) {
      c = skyColor(rd, F.sun);
    } else {
      SurfacePoint sp;
      surfacePoint(W, F, h, Surface[b], rd, height, sp);
      c = pixelAlbedo(sp);
    }
    Linear[b] = make_float4(c.x, c.y, c.z, 1.0f);
  }
}

__global__ void __launch_bounds__(kShadeThreads, 1536 / kShadeThreads)
    lightPixelsK(const float* __restrict__ W, const uint32_t* __restrict__ O, const float* __restrict__ C,
                 const float4* __restrict__ Hit, const float4* __restrict__ Surface, float4* Linear, int width, int height,
                 int rowStart, int rowEnd) {
  __shared__ FrameConst F;
  frameInit(F, C, O);
  const int tilesX = (width + 7) / 8, tiles = tilesX * ((rowEnd - rowStart + 3) / 4), warps = kShadeThreads / 32;
#pragma unroll 1
  for (int i = int(blockIdx.x) * warps + int(threadIdx.x >> 5); i < tiles; i += int(gridDim.x) * warps) {
    int x, y;
    if (!stripPixel(i, tilesX, width, rowStart, rowEnd, x, y)) continue;
    const size_t b = size_t(y) * width + x;
    const float4 h = Hit[b];
    if (int(h.y) == kSkyId) continue;
    const f3 rd = primaryDir(F.cam, x, y, width, height);
    const float4 a = Linear[b];
    SurfacePoint sp;
    surfacePoint(W, F, h, Surface[b], rd, height, sp);
    const f3 c = pixelLight(W, F, sp, rd, int(h.y), mk(a.x, a.y, a.z));
    Linear[b] = make_float4(c.x, c.y, c.z, 1.0f);
  }
}

// Both halves at once, for strips of at most one wave (strips.cuh).
__global__ void __launch_bounds__(kShadeThreads, 1024 / kShadeThreads)
    shadePixelsK(const float* __restrict__ W, const uint32_t* __restrict__ O, const float* __restrict__ C,
                 const float4* __restrict__ Hit, const float4* __restrict__ Surface, float4* Linear, int width,
                 int height, int rowStart, int rowEnd) {
  __shared__ FrameConst F;
  frameInit(F, C, O);
  int x, y;
  if (!stripPixel(int(blockIdx.x) * (kShadeThreads / 32) + int(threadIdx.x >> 5), (width + 7) / 8, width, rowStart, rowEnd,
                  x, y))
    return;
  const size_t b = size_t(y) * width + x;
  const float4 h = Hit[b];
  const f3 rd = primaryDir(F.cam, x, y, width, height);
  f3 c;
  if (int(h.y) == kSkyId) {
    c = skyColor(rd, F.sun);
  } else {
    SurfacePoint sp;
    surfacePoint(W, F, h, Surface[b], rd, height, sp);
    c = pixelLight(W, F, sp, rd, int(h.y), pixelAlbedo(sp));
  }
  Linear[b] = make_float4(c.x, c.y, c.z, 1.0f);
}

__global__ void __launch_bounds__(kShadeThreads, 1024 / kShadeThreads)
    resolveFrameK(const float4* __restrict__ Linear, float4* History, uint32_t* Pixels, const float* __restrict__ C,
                  const float4* __restrict__ Hit, const float4* __restrict__ Surface, int width, int height) {
  __shared__ FrameConst F;
  __shared__ ResolveTaps taps;
  tapsInit(taps);
  frameInit(F, C, nullptr);
  const int tilesX = (width + 7) / 8, tiles = tilesX * ((height + 3) / 4), warps = kShadeThreads / 32;
#pragma unroll 1
  for (int i = int(blockIdx.x) * warps + int(threadIdx.x >> 5); i < tiles; i += int(gridDim.x) * warps) {
    int x, y;
    if (!stripPixel(i, tilesX, width, 0, height, x, y)) continue;
    const float4 l = Linear[size_t(y) * width + x];
    resolvePixel(mk(l.x, l.y, l.z), History, Pixels, F, taps, Hit, Surface, width, height, x, y);
  }
}

// Blocks of each kernel the current device holds, computed once per device.
struct ShadeGrids { int albedo, light, resolve; };
const ShadeGrids* shadeGrids() {
  constexpr int kDevices = 64;
  static std::once_flag once[kDevices];
  static ShadeGrids grids[kDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return nullptr;
  std::call_once(once[dev], [dev] {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    auto held = [sms](auto kernel) {
      int per = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kShadeThreads, 0);
      return sms * (per > 0 ? per : 1);
    };
    grids[dev] = ShadeGrids{held(albedoPixelsK), held(lightPixelsK), held(resolveFrameK)};
  });
  return &grids[dev];
}
// The lighting half alone, over an albedo that is already in Linear.
int lightRows(const float* World, const unsigned* Origin, const float* C, const float* Hit, const float* Surface,
              float* Linear, int width, int height, int rowStart, int rows, cudaStream_t stream) {
  const ShadeGrids* g = shadeGrids();
  if (!g) return STRATUM_EINVAL;
  lightPixelsK<<<tileBlocks(width, rows, g->light), kShadeThreads, 0, stream>>>(
      World, Origin, C, reinterpret_cast<const float4*>(Hit), reinterpret_cast<const float4*>(Surface),
      reinterpret_cast<float4*>(Linear), width, height, rowStart, rowStart + rows);
  return launchStatus();
}

}  // namespace st

using namespace st;

extern "C" {

int stratum_shadePixels(const float* World, const unsigned* Origin, const float* C, const float* Hit,
                        const float* Surface, float* Linear, int width, int height, int rowStart, int rowCount,
                        stratum_stream_t stream) {
  if (!World || !Origin || !C || !Hit || !Surface || !Linear || !frameOk(width, height)) return STRATUM_EINVAL;
  if (rowStart < 0 || rowCount < 0) return STRATUM_EINVAL;
  int rows = rowCount < height - rowStart ? rowCount : height - rowStart;
  if (rows <= 0) return STRATUM_OK;
  const ShadeGrids* g = shadeGrids();
  if (!g) return STRATUM_EINVAL;
  if (tileBlocks(width, rows) <= shadeWave()) {
    shadePixelsK<<<tileBlocks(width, rows), kShadeThreads, 0, asStream(stream)>>>(
        World, Origin, C, reinterpret_cast<const float4*>(Hit), reinterpret_cast<const float4*>(Surface),
        reinterpret_cast<float4*>(Linear), width, height, rowStart, rowStart + rows);
    return launchStatus();
  }
  albedoPixelsK<<<tileBlocks(width, rows, g->albedo), kShadeThreads, 0, asStream(stream)>>>(
      World, Origin, C, reinterpret_cast<const float4*>(Hit), reinterpret_cast<const float4*>(Surface),
      reinterpret_cast<float4*>(Linear), width, height, rowStart, rowStart + rows);
  const int s = launchStatus();
  return s != STRATUM_OK ? s
                         : lightRows(World, Origin, C, Hit, Surface, Linear, width, height, rowStart, rows, asStream(stream));
}

int stratum_resolveFrame(const float* Linear, float* History, unsigned* Pixels, const float* C, const float* Hit,
                         const float* Surface, int width, int height, stratum_stream_t stream) {
  if (!Linear || !History || !Pixels || !C || !Hit || !Surface || !frameOk(width, height)) return STRATUM_EINVAL;
  const ShadeGrids* g = shadeGrids();
  if (!g) return STRATUM_EINVAL;
  resolveFrameK<<<tileBlocks(width, height, g->resolve), kShadeThreads, 0, asStream(stream)>>>(
      reinterpret_cast<const float4*>(Linear), reinterpret_cast<float4*>(History), Pixels, C,
      reinterpret_cast<const float4*>(Hit), reinterpret_cast<const float4*>(Surface), width, height);
  return launchStatus();
}

}  // extern "C"
