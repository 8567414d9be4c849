// tracePrimary drop-in (kernels/trace.cu:29-61 of the reference): every pixel of
// a strip of rows.
//
// A block covers 16x16 pixels with eight warps, each tracing one 8x4 tile with
// the warp-cooperative traversal of the batched renderer (traverse_coop.cuh):
// lanes walk their own rays to the hierarchy leaves, and the warp evaluates one
// (lot, group) at a time for every lane waiting on it.  The drop-in has only
// the reference's buffers, so there is no table-wide group cache; instead the
// block keeps the groups its warps build (by the random-access grammar) in a
// shared-memory table, and a warp that needs a group another warp of the block
// has built, or is building, reads it from there (neighbouring tiles reach the same
// groups: on the bench poses a 16x16 block needs 6-9x fewer group builds than its
// warps would alone).  Warps that came to a group while it was being built used to
// build it too: six 1600x900 views, one call each, 5.69 ms, now 5.23 (16x16 blocks;
// of 32x16 pixels 5.37, 8x16 6.65, fewer warps resident 6.07).  Each ray still visits its leaves in the reference's order with
// the same running best, so Hit and Surface equal the reference's bit for bit.
//
// The reference's 64-row strips leave each launch a tail of partly idle SMs:
// six 1600x900 views in 15 strips each took 24.4 ms, in one call per view
// (rowCount = height, which the entry point accepts) 14.3 ms, and in one call take
// 4.95 now.  A
// programmatic dependent launch of each strip was tried and measured no
// faster: a dependent grid may be scheduled early, but its griddepcontrol.wait
// returns only once the preceding grid has completed, and skipping that wait is
// safe only when the preceding kernel is known to be another strip.
#include <mutex>

// (written out: six 1600x900 views 5.23 ms, with one copy of each division 5.31; the
// eight warps of a block share more of their way through the code)
#define STRATUM_QUOTIENT WrittenOut
#include "batch.cuh"
#include "common_api.cuh"
#include "traverse_coop.cuh"

// Block shape in 8x4-pixel warp tiles, and resident blocks per SM the register
// allocation must allow (2 blocks of 2 x 4 tiles: 512 threads, up to 128
// registers a thread).
#ifndef STRATUM_DROPIN_TILES_X
#define STRATUM_DROPIN_TILES_X 2
#endif
#ifndef STRATUM_DROPIN_TILES_Y
#define STRATUM_DROPIN_TILES_Y 4
#endif
#ifndef STRATUM_DROPIN_BLOCKS
#define STRATUM_DROPIN_BLOCKS 2
#endif

namespace st {

constexpr int kDropInTilesX = STRATUM_DROPIN_TILES_X, kDropInTilesY = STRATUM_DROPIN_TILES_Y;
constexpr int kDropInThreads = 32 * kDropInTilesX * kDropInTilesY;
constexpr int kDropInW = 8 * kDropInTilesX, kDropInH = 4 * kDropInTilesY;
struct DropInShared {
  WarpStage stage[kDropInThreads / 32];
  BlockCache cache;
};

// `bandRows` block rows nearest the horizon are drawn first, each by four blocks
// whose warps take tiles one pixel high (see Band in batch.cuh), then the others,
// nearest the horizon first.
__global__ void __launch_bounds__(kDropInThreads, STRATUM_DROPIN_BLOCKS)
    tracePrimaryK(const float* __restrict__ W, const float* __restrict__ N, const uint32_t* __restrict__ O,
                  const float* __restrict__ C, float* Hit, float* Surface, int width, int height, int rowStart,
                  int rowCount, int blocksX, int bandRows) {
  extern __shared__ __align__(16) unsigned char dropInBytes[];
  DropInShared& sh = *reinterpret_cast<DropInShared*>(dropInBytes);
  __shared__ Camera cam;
  __shared__ uint32_t org[4];
  if (threadIdx.x == 0) {
    cam = makeCamera(C);
    for (int i = 0; i < 4; i++) org[i] = O[i];
  }
  blockCacheInit(sh.cache);
  __syncthreads();
  const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
  const int strip = min(rowCount, height - rowStart), rows = (strip + kDropInH - 1) / kDropInH;
  const int horizon = min(max(horizonRow(cam, height) - rowStart, 0), strip - 1), mid = horizon / kDropInH;
  const int row0 = min(max(mid - bandRows / 2, 0), rows - bandRows);  // of the band
  const int blockRow = int(blockIdx.x) / blocksX, blockX = int(blockIdx.x) % blocksX;
  const int tileX = blockX * kDropInW + (warp % kDropInTilesX) * 8;
  int x, y;
  bool mine;
  if (blockRow < 4 * bandRows) {
    x = tileX + lane;
    y = row0 * kDropInH + nearRow(blockRow, min(horizon / 4 - row0 * (kDropInH / 4), 4 * bandRows - 1), 4 * bandRows) * 4 +
        warp / kDropInTilesX;
    mine = lane < 8;
  } else {
    const int row = nearRow(blockRow - 4 * bandRows, mid, rows);
    if (row >= row0 && row < row0 + bandRows) return;  // uniform over the block
    x = tileX + (lane & 7);
    y = row * kDropInH + (warp / kDropInTilesX) * 4 + (lane >> 3);
    mine = true;
  }
  const bool active = mine && x < width && y < strip;
  y += rowStart;
  const f3 rd = primaryDir<Quotient>(cam, active ? x : 0, active ? y : 0, width, height);
  const TraceResult r = traceWarp<true>(W, reinterpret_cast<const float4*>(N), org[0], org[2], cam.pos, rd,
                                        1.08f / float(height), active, sh.stage[warp], groupCache(nullptr),
                                        &sh.cache);
  if (!active) return;
  storeTrace(Hit, Surface, size_t(y) * width + x, r);
}

}  // namespace st

using namespace st;

namespace {
constexpr int kSmemDevices = 64;
static_assert(kDropInTilesY == 4 && kDropInH == 16, "a band block is a quarter of a block high");
}

extern "C" int stratum_tracePrimary(const float* World, const float* Nodes, const unsigned* Origin, const float* C,
                                    float* Hit, float* Surface, int width, int height, int rowStart, int rowCount,
                                    stratum_stream_t stream) {
  if (!World || !Nodes || !Origin || !C || !Hit || !Surface || !frameOk(width, height)) return STRATUM_EINVAL;
  if (rowStart < 0 || rowCount < 0) return STRATUM_EINVAL;
  int rows = rowCount < height - rowStart ? rowCount : height - rowStart;
  if (rows <= 0) return STRATUM_OK;
  static std::once_flag once[kSmemDevices];
  static int resident[kSmemDevices];  // blocks the device holds
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kSmemDevices) return STRATUM_EINVAL;
  std::call_once(once[dev], [dev] {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(tracePrimaryK, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(DropInShared)));
    resident[dev] = sms * STRATUM_DROPIN_BLOCKS;
  });
  // Band rows: up to twice the blocks the device holds in quarter blocks, but at
  // most a sixth of a launch that fills the device by itself (a band row takes about
  // two rows' time; so a 64-row strip that does gets none), and none in one that fills it
  // more than 14 times, whose other rows hide the slow tiles.  One call for each of six
  // poses, sum in us, without / with: 320x180 2,045 / 1,507, 640x360 2,454 / 2,118, 1024x576
  // (7.8 times) 3,380 / 3,167, 1283x721 (12.6) 4,199 / 4,151, 1344x756 (13.6) 4,359 / 4,235,
  // 1440x810 (15.5) 4,463 / 4,632, 1600x900 (19) 5,031 / 5,305, 3840x2160 18,635 / 18,970.
  // A launch that does not fill the device may be all band: a small frame has to be, but
  // most strips of a larger one hold no horizon, and a strip of over 0.6 of the device
  // gets none.  Frames in 64-row strips: 320x180 (strips of 0.3 of the device) 3,115 / 2,116,
  // 640x360 (0.5) 4,674 / 4,315, 800x450 (0.7) 5,314 / 6,321, 1024x576 (0.9) 6,146 / 8,231.
  const int blocksX = (width + kDropInW - 1) / kDropInW, blockRows = (rows + kDropInH - 1) / kDropInH;
  const int blocks = blocksX * blockRows, held = resident[dev];
  const bool all = blocks <= held && (rows == height || 5 * blocks <= 3 * held);
  const int most = all ? blockRows : blocks <= 14 * held ? blockRows / 6 : 0;
  const int want = (2 * resident[dev] - 1) / (4 * blocksX) + 1, bandRows = want < most ? want : most;
  tracePrimaryK<<<blocksX * (blockRows + 4 * bandRows), kDropInThreads, sizeof(DropInShared), asStream(stream)>>>(
      World, Nodes, static_cast<const uint32_t*>(Origin), C, Hit, Surface, width, height, rowStart, rowCount, blocksX,
      bandRows);
  return launchStatus();
}
