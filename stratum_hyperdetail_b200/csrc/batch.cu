// Batched multi-view frame path: many views of any resolution, pose and world
// seed per launch.  Each kernel reads a device table of stratum_view; every
// per-ray / per-pixel / per-lot computation is the single-view code, so a
// view's results in a batch are bit-identical to rendering it alone.
//
//   stepViewsK      one thread per view: stepCamera
//   clearViewsK,
//   refreshViewsK   clearQueue + prepareLots of all views (grid: slots x views)
//   buildViewsK     all views' queued lots, eight to a block (hierarchy.cuh)
//   prologueK       tile bases of every view under the chosen tile order, the
//                   per-view frame constants (camera basis, sun, origin), the
//                   resolve taps and the group caches' launch epochs, computed
//                   once per frame
//   cacheResetK     clears the directory of a full group cache the prologue
//                   chose to reset (group_cache.cuh)
//   traceViewsK     persistent: each warp claims `grab` 8x4-pixel tiles at a
//                   time from a device queue over all views and traces them
//   shadeViewsK     persistent: material colour of the same tiles (albedo into
//                   Linear; sky pixels get their final colour)
//   lightViewsK     persistent: lighting of the hit pixels from that albedo
//                   (relief normal, sun shadow, ambient, GGX, reflections, fog)
//                   into Linear -- two kernels because the shading code split in
//                   two measured faster than one (instruction fetch)
//   resolveViewsK   persistent: contact occlusion, accumulation and tone map
//                   (History, Pixels); a kernel of its own because the two
//                   fused measured slower (the shading code alone fills the
//                   instruction cache)
//
// The tile queues reset themselves: the last warp to find a queue empty zeroes
// its counters, so consecutive launches (and graph replays) need no memset.
#include <mutex>

#include "batch.cuh"
#include "common_api.cuh"
#include "hierarchy.cuh"
#include "traverse_coop.cuh"
#include "world.cuh"

static_assert(sizeof(stratum_view) == 128, "stratum_view layout is part of the ABI");

namespace st {

__global__ void stepViewsK(stratum_view* V, int n) {
  int v = int(blockIdx.x * blockDim.x + threadIdx.x);
  if (v >= n) return;
  stratum_view& w = V[v];
  stepOne(w.C, w.Origin, w.I, w.dt, w.width, w.height);
}

__global__ void applyPosesK(const stratum_view* V, const stratum_pose* P, const int* flags, int n) {
  int v = int(blockIdx.x * blockDim.x + threadIdx.x);
  if (v >= n) return;
  const stratum_view& w = V[v];
  const int f = flags[v];
  if (f & 1) {
    const stratum_pose& p = P[v];
    w.C[0] = p.pos[0]; w.C[1] = p.pos[1]; w.C[2] = p.pos[2]; w.C[3] = p.yaw; w.C[4] = p.pitch;
    for (int i = 0; i < 4; i++) w.Origin[i] = p.origin[i];
  }
  const_cast<float*>(w.I)[23] = (f & 2) ? 1.0f : 0.0f;
}

__global__ void clearViewsK(const stratum_view* V, int n) {
  int v = int(blockIdx.x * blockDim.x + threadIdx.x);
  if (v < n) V[v].Queue[0] = 0u;
}

__global__ void refreshViewsK(const stratum_view* __restrict__ V, int n) {
  int slot = int(blockIdx.x * blockDim.x + threadIdx.x), v = int(blockIdx.y);
  if (slot >= kLots || v >= n) return;
  const stratum_view& w = V[v];
  refreshSlot(slot, w.Origin, int(w.C[14]), w.World, w.Tags, w.Queue);
}

__global__ void __launch_bounds__(kBuildThreads, kBuildBlocks) buildViewsK(const stratum_view* __restrict__ V, int n) {
  __shared__ BuildShared sh;
  const int v = int(blockIdx.y);
  if (v >= n) return;
  buildQueue(V[v].Queue, V[v].World, V[v].Nodes, int(blockIdx.x), int(gridDim.x), sh);
}

// The directory of a group cache whose reset the prologue just decided.
__global__ void cacheResetK(const stratum_view* __restrict__ V, int n) {
  const int v = int(blockIdx.y);
  if (v >= n || !V[v].Groups) return;
  const GroupCacheHeader* h = reinterpret_cast<const GroupCacheHeader*>(V[v].Groups);
  if (h->capacity == 0u || h->resetAt != h->launches || h->resets == 0u) return;
  uint4* d = reinterpret_cast<uint4*>(groupCache(V[v].Groups).dir(0, 0));
  for (int i = int(blockIdx.x * blockDim.x + threadIdx.x); i < kCacheDirWords / 4; i += int(gridDim.x * blockDim.x))
    d[i] = make_uint4(0u, 0u, 0u, 0u);
}
__global__ void cacheInitK(uint32_t* base, uint32_t entries) {
  GroupCacheHeader* h = reinterpret_cast<GroupCacheHeader*>(base);
  h->next = 0u; h->capacity = entries; h->resets = 0u; h->fills = 0u; h->launches = 0u; h->resetAt = 0u;
}

// `bandTiles`: band tiles to give out over all views: twice the warps the device
// holds.  Warm trace of one 640x360 view, street / rooftop / aerial / canal / avenue:
// no band 417 / 486 / 637 / 399 / 460 us, once the warps 363 / 484 / 629 / 359 / 285,
// twice 309 / 355 / 634 / 248 / 291, four times 324 / 377 / 723 / 262 / 310.  Views
// of a large batch get none: there the other views' tiles fill the device (one tile row
// each made twelve mixed views 0.5 % slower).
__global__ void prologueK(stratum_view* V, int n, int order, int bandTiles, BatchScratch* S) {
  for (int v = int(threadIdx.x); v < n; v += int(blockDim.x)) {
    S->view[v].frame = makeFrame(V[v].C, V[v].Origin);
    const int W = V[v].width, H = V[v].height;
    V[v].tilesX = (W + kTileW - 1) / kTileW;
    Band& b = S->view[v].band;
    b.horizon = b.row0 = b.row1 = 0;
    if (W > 0 && H > 0) {
      const int rows = (H + kTileH - 1) / kTileH, want = bandTiles / n / (V[v].tilesX * kTileH), band = min(want, rows);
      b.horizon = horizonRow(S->view[v].frame.cam, H);
      b.row0 = min(max(b.horizon / kTileH - band / 2, 0), rows - band);  // may be none
      b.row1 = b.row0 + band;
    }
    if (V[v].Groups) {  // this launch's epoch; a full cache starts again now and then
      GroupCacheHeader* h = reinterpret_cast<GroupCacheHeader*>(V[v].Groups);
      h->launches++;
      if (h->capacity != 0u && h->next >= h->capacity && h->launches - h->resetAt >= kCacheResetInterval) {
        h->next = 0u;
        h->resets++;
        h->resetAt = h->launches;  // cacheResetK clears the directory next
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int base = 0, band = 0;
    for (int v = 0; v < n; v++) {
      V[v].tileBase = base;
      S->view[v].band.base = band;
      // a view with no pixels owns no tiles (and is never looked up)
      if (V[v].width > 0 && V[v].height > 0) {
        base += tileCount(V[v].width, V[v].height, order);
        band += bandCount(S->view[v].band, V[v].tilesX, V[v].height);
      }
    }
    S->counters[kTotalTiles] = uint32_t(base);
    S->counters[kBandTiles] = uint32_t(band);
    S->taps = makeTaps();
  }
}

SD int bandViewOf(const BatchScratch* S, int n, int tile) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (S->view[mid].band.base <= tile) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// STRATUM_TRACE_OCC / THREADS resident blocks (rounded down).  At 576 threads per SM
// the compiler takes 96 registers, which is ten 64-thread blocks: six-view 1600x900
// trace 3.45 ms, aerial 1.54; 512 (128 registers) 3.73 / 1.69, 640 3.51 / 1.57.  768
// (80 registers, spills) is equal over whole frames, but the slowest tiles, which bound
// small views, take 5-10 % longer.  128- and 256-thread blocks come to four and two an SM
// (127 registers, 16 warps): 3.49 and 3.48 ms.
#ifndef STRATUM_TRACE_OCC
#define STRATUM_TRACE_OCC 576
#endif
template <int THREADS>
__global__ void __launch_bounds__(THREADS, STRATUM_TRACE_OCC / THREADS)
    traceViewsK(const stratum_view* __restrict__ V, int n, int grab, int order, BatchScratch* S) {
  extern __shared__ __align__(16) unsigned char stageBytes[];  // THREADS / 32 WarpStage
  const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
  const int bands = int(S->counters[kBandTiles]), total = bands + int(S->counters[kTotalTiles]);
#pragma unroll 1
  for (;;) {
    const int t0 = claim(&S->counters[kTraceNext], grab);
    if (t0 >= total) break;
    const int t1 = min(t0 + grab, total);
#pragma unroll 1
    for (int tile = t0; tile < t1; tile++) {
      const int v = tile < bands ? bandViewOf(S, n, tile) : viewOf(V, n, tile - bands);
      const int W = V[v].width, H = V[v].height;
      const Band band = S->view[v].band;
      int x, y;
      bool inFrame;
      if (tile < bands) {
        const int local = tile - band.base, first = band.row0 * kTileH, rows = min(band.row1 * kTileH, H) - first;
        x = (local % V[v].tilesX) * kTileW + lane;
        y = first + nearRow(local / V[v].tilesX, min(max(band.horizon - first, 0), rows - 1), rows);
        inFrame = lane < kTileW && x < W;
      } else {
        int tx, ty;
        if (!tileCoord(tile - bands - V[v].tileBase, V[v].tilesX, (H + kTileH - 1) / kTileH, order, tx, ty,
                       band.horizon / kTileH) ||
            (ty >= band.row0 && ty < band.row1))
          continue;
        x = tx * kTileW + (lane & 7);
        y = ty * kTileH + (lane >> 3);
        inFrame = x < W && y < H;
      }
      const Camera cam = S->view[v].frame.cam;
      const uint32_t o0 = S->view[v].frame.o[0], o2 = S->view[v].frame.o[2];
      f3 rd = primaryDir<Quotient>(cam, inFrame ? x : 0, inFrame ? y : 0, W, H);
      TraceResult r = traceWarp(V[v].World, reinterpret_cast<const float4*>(V[v].Nodes), o0, o2, cam.pos, rd,
                                1.08f / float(H), inFrame, reinterpret_cast<WarpStage*>(stageBytes)[warp],
                                groupCache(V[v].Groups));
      if (!inFrame) continue;
      storeTrace(V[v].Hit, V[v].Surface, size_t(y) * W + x, r);
    }
  }
  retire(&S->counters[kTraceNext], &S->counters[kTraceDone], THREADS);
}

// STRATUM_SHADE_OCC / THREADS resident blocks of the material pass: 1280 threads
// per SM (six 1600x900 views 392 us; 1024 397, 1536 404); STRATUM_LIGHT_OCC of
// the lighting pass: 1536 (40 registers, some spills: 736 us; 1024 764).
#ifndef STRATUM_SHADE_OCC
#define STRATUM_SHADE_OCC 1280
#endif
#ifndef STRATUM_LIGHT_OCC
#define STRATUM_LIGHT_OCC 1536
#endif
template <int THREADS>
__global__ void __launch_bounds__(THREADS, STRATUM_SHADE_OCC / THREADS) shadeViewsK(const stratum_view* __restrict__ V, int n, int grab, int order,
                                                      BatchScratch* S) {
  const int lane = int(threadIdx.x & 31);
  const int total = int(S->counters[kTotalTiles]);
#pragma unroll 1
  for (;;) {
    const int t0 = claim(&S->counters[kShadeNext], grab);
    if (t0 >= total) break;
    const int t1 = min(t0 + grab, total);
#pragma unroll 1
    for (int tile = t0; tile < t1; tile++) {
      const int v = viewOf(V, n, tile);
      const int W = V[v].width, H = V[v].height;
      int tx, ty;
      if (!tileCoord(tile - V[v].tileBase, V[v].tilesX, (H + kTileH - 1) / kTileH, order, tx, ty)) continue;
      const int x = tx * kTileW + (lane & 7), y = ty * kTileH + (lane >> 3);
      if (x >= W || y >= H) continue;
      const FrameConst F = S->view[v].frame;
      const size_t b = size_t(y) * W + x;
      const float4* hit = reinterpret_cast<const float4*>(V[v].Hit);
      const float4* surf = reinterpret_cast<const float4*>(V[v].Surface);
      const float4 h4 = hit[b];
      const f3 rd = primaryDir(F.cam, x, y, W, H);
      f3 c;
      if (int(h4.y) == kSkyId) {
        c = skyColor(rd, F.sun);
      } else {
        SurfacePoint sp;
        surfacePoint(V[v].World, F, h4, surf[b], rd, H, sp);
        c = pixelAlbedo(sp);
      }
      reinterpret_cast<float4*>(V[v].Linear)[b] = make_float4(c.x, c.y, c.z, 1.0f);
    }
  }
  retire(&S->counters[kShadeNext], &S->counters[kShadeDone], THREADS);
}

// STRATUM_RESOLVE_OCC / THREADS resident blocks: the taps' loads are what it waits
// for (1024 threads per SM 611 us for the six views; 1280 630, 1536 648, the
// compiler's choice of 72 registers 639).
#ifndef STRATUM_RESOLVE_OCC
#define STRATUM_RESOLVE_OCC 1024
#endif
template <int THREADS>
__global__ void __launch_bounds__(THREADS, STRATUM_LIGHT_OCC / THREADS) lightViewsK(const stratum_view* __restrict__ V,
                                                                                int n, int grab, int order,
                                                                                BatchScratch* S) {
  const int lane = int(threadIdx.x & 31);
  const int total = int(S->counters[kTotalTiles]);
#pragma unroll 1
  for (;;) {
    const int t0 = claim(&S->counters[kLightNext], grab);
    if (t0 >= total) break;
    const int t1 = min(t0 + grab, total);
#pragma unroll 1
    for (int tile = t0; tile < t1; tile++) {
      const int v = viewOf(V, n, tile);
      const int W = V[v].width, H = V[v].height;
      int tx, ty;
      if (!tileCoord(tile - V[v].tileBase, V[v].tilesX, (H + kTileH - 1) / kTileH, order, tx, ty)) continue;
      const int x = tx * kTileW + (lane & 7), y = ty * kTileH + (lane >> 3);
      if (x >= W || y >= H) continue;
      const size_t b = size_t(y) * W + x;
      const float4 h4 = reinterpret_cast<const float4*>(V[v].Hit)[b];
      if (int(h4.y) == kSkyId) continue;
      const FrameConst F = S->view[v].frame;
      const f3 rd = primaryDir(F.cam, x, y, W, H);
      float4* lin = reinterpret_cast<float4*>(V[v].Linear) + b;
      const float4 a = *lin;
      SurfacePoint sp;
      surfacePoint(V[v].World, F, h4, reinterpret_cast<const float4*>(V[v].Surface)[b], rd, H, sp);
      const f3 c = pixelLight(V[v].World, F, sp, rd, int(h4.y), mk(a.x, a.y, a.z));
      *lin = make_float4(c.x, c.y, c.z, 1.0f);
    }
  }
  retire(&S->counters[kLightNext], &S->counters[kLightDone], THREADS);
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, STRATUM_RESOLVE_OCC / THREADS) resolveViewsK(const stratum_view* __restrict__ V, int n, int grab, int order,
                                                        BatchScratch* S) {
  const int lane = int(threadIdx.x & 31);
  const int total = int(S->counters[kTotalTiles]);
#pragma unroll 1
  for (;;) {
    const int t0 = claim(&S->counters[kResolveNext], grab);
    if (t0 >= total) break;
    const int t1 = min(t0 + grab, total);
#pragma unroll 1
    for (int tile = t0; tile < t1; tile++) {
      const int v = viewOf(V, n, tile);
      const int W = V[v].width, H = V[v].height;
      int tx, ty;
      if (!tileCoord(tile - V[v].tileBase, V[v].tilesX, (H + kTileH - 1) / kTileH, order, tx, ty)) continue;
      const int x = tx * kTileW + (lane & 7), y = ty * kTileH + (lane >> 3);
      if (x >= W || y >= H) continue;
      const FrameConst F = S->view[v].frame;
      const size_t b = size_t(y) * W + x;
      const float4 l = reinterpret_cast<const float4*>(V[v].Linear)[b];
      resolvePixel(mk(l.x, l.y, l.z), reinterpret_cast<float4*>(V[v].History), V[v].Pixels, F, S->taps,
                   reinterpret_cast<const float4*>(V[v].Hit), reinterpret_cast<const float4*>(V[v].Surface), W, H, x, y);
    }
  }
  retire(&S->counters[kResolveNext], &S->counters[kResolveDone], THREADS);
}

// Dynamic shared memory of a trace block: one WarpStage per warp.
constexpr size_t traceSmem(int threads) { return size_t(threads / 32) * sizeof(WarpStage); }

enum Parts { kTrace = 1, kShade = 2 };

// Persistent grids of one block size on one device: the resident-block count of
// each kernel, computed once per (block size, device) and published through
// std::call_once, so concurrent first calls (the render server's scheduler and
// a direct caller) all see the four grids complete.
struct PersistentGrids { int trace, shade, light, resolve; };

template <int T>
int launchParts(stratum_view* V, int n, const stratum_tune& t, BatchScratch* S, cudaStream_t s, int parts) {
  static std::once_flag once[kGridDevices];
  static PersistentGrids grids[kGridDevices];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return -int(e);
  if (dev < 0 || dev >= kGridDevices) return STRATUM_EINVAL;
  std::call_once(once[dev], [&] {
    PersistentGrids g;
    g.trace = residentBlocks(traceViewsK<T>, T, traceSmem(T));
    g.shade = residentBlocks(shadeViewsK<T>, T);
    g.light = residentBlocks(lightViewsK<T>, T);
    g.resolve = residentBlocks(resolveViewsK<T>, T);
    grids[dev] = g;
  });
  const PersistentGrids& g = grids[dev];
  const int order = t.order & 1;  // tile order; bit 1 selects the block-pooled trace
  if (parts & kTrace) {
    prologueK<<<1, 256, 0, s>>>(V, n, order, 2 * g.trace * (T / 32), S);
    cacheResetK<<<dim3(64, n), 256, 0, s>>>(V, n);
  }
  if ((parts & kTrace) && (t.order & 2) && n <= kPoolViews)
    launchPooled<T>(V, n, order, S, dev, s);
  else if (parts & kTrace)
    traceViewsK<T><<<g.trace, T, traceSmem(T), s>>>(V, n, t.grab, order, S);
  if (parts & kShade) shadeViewsK<T><<<g.shade, T, 0, s>>>(V, n, t.grab, order, S);
  if (parts & kShade) lightViewsK<T><<<g.light, T, 0, s>>>(V, n, t.grab, order, S);
  if (parts & kShade) resolveViewsK<T><<<g.resolve, T, 0, s>>>(V, n, t.grab, order, S);
  return launchStatus();
}

bool tuneOk(const stratum_tune& t) {
  return (t.threads == 64 || t.threads == 128 || t.threads == 256) && t.grab >= 1 && t.grab <= 16 &&
         t.order >= 0 && t.order <= 3;
}

// parts: kTrace (with the prologue), kShade (uses the prologue's scratch), or both.
int render(stratum_view* V, int n, void* scratch, unsigned long long bytes, const stratum_tune* tune, cudaStream_t s,
           int parts) {
  if (!V || !scratch || n <= 0 || n > 65535 || bytes < batchScratchBytes(n)) return STRATUM_EINVAL;
  stratum_tune t = tune ? *tune : stratum_tune{128, 1, 1};
  if (!tuneOk(t)) return STRATUM_EINVAL;
  BatchScratch* S = static_cast<BatchScratch*>(scratch);
  if (t.threads == 64) return launchParts<64>(V, n, t, S, s, parts);
  if (t.threads == 256) return launchParts<256>(V, n, t, S, s, parts);
  return launchParts<128>(V, n, t, S, s, parts);
}

// ---- allocation-free variant -------------------------------------------------
// The renderer's scratch (queue counters, resolve taps, per-view frame
// constants) for callers that cannot give the library device memory, held in
// one static device array.  Every GPU that loads the library holds this array
// (about 7.8 KB) until the process exits.
constexpr int kNoAllocMaxViews = STRATUM_NOALLOC_MAX_VIEWS;
constexpr size_t kNoAllocBytes = batchScratchBytes(kNoAllocMaxViews);
static __device__ __align__(256) unsigned char gNoAllocScratch[kNoAllocBytes];

}  // namespace st

#include <cuda.h>
#include <mutex>

namespace {
// Device address of gNoAllocScratch per device ordinal, looked up with that
// device current on the first call in each of its contexts.  Host code must
// not use the array's name as an address: on the host it is only a stand-in
// for the device symbol.  The address belongs to the context the module was
// loaded into, so it is cached with that context's unique id: after a
// cudaDeviceReset the next call finds a new context and looks it up again.
constexpr int kMaxDevices = 128;
std::mutex gNoAllocLock;
struct NoAllocSlot { unsigned long long ctx; void* addr; };
NoAllocSlot gNoAllocAddr[kMaxDevices] = {};

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

// Unique id of the calling thread's current context (0 if none or unknown),
// through the driver entry points the runtime hands out.
unsigned long long currentContextId() {
  static std::once_flag once;
  static CtxGetCurrentFn getCurrent = nullptr;
  static CtxGetIdFn getId = nullptr;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      getCurrent = reinterpret_cast<CtxGetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      getId = reinterpret_cast<CtxGetIdFn>(f);
  });
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (!getCurrent || !getId || getCurrent(&ctx) != CUDA_SUCCESS || !ctx || getId(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

int noAllocScratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return -int(e);
  if (dev < 0 || dev >= kMaxDevices) return STRATUM_EINVAL;
  std::lock_guard<std::mutex> hold(gNoAllocLock);
  NoAllocSlot& slot = gNoAllocAddr[dev];
  const unsigned long long ctx = currentContextId();
  if (!slot.addr || ctx == 0 || slot.ctx != ctx) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, st::gNoAllocScratch);
    if (e != cudaSuccess || !p) return e != cudaSuccess ? -int(e) : STRATUM_EINVAL;
    slot.addr = p;
    slot.ctx = currentContextId();  // the lookup has made the device's context current
  }
  *out = slot.addr;
  return STRATUM_OK;
}
}  // namespace

using namespace st;
int stratumHierarchyGrid();

extern "C" {

unsigned long long stratum_batchScratchBytes(int views) { return views > 0 ? batchScratchBytes(views) : 0; }

unsigned long long stratum_groupCacheBytes(int entries) { return entries >= 0 ? groupCacheBytes(entries) : 0; }
int stratum_groupCacheInit(unsigned* Groups, int entries, stratum_stream_t stream) {
  if (!Groups || entries < 0 || uint32_t(entries) > kCacheMaxEntries) return STRATUM_EINVAL;
  cudaError_t e = cudaMemsetAsync(Groups, 0, kCacheEntryOffset, asStream(stream));
  if (e != cudaSuccess) return -int(e);
  cacheInitK<<<1, 1, 0, asStream(stream)>>>(Groups, uint32_t(entries));
  return launchStatus();
}

int stratum_applyPoses(stratum_view* views, const stratum_pose* poses, const int* flags, int n,
                       stratum_stream_t stream) {
  if (!views || !poses || !flags || n <= 0) return STRATUM_EINVAL;
  applyPosesK<<<(n + 63) / 64, 64, 0, asStream(stream)>>>(views, poses, flags, n);
  return launchStatus();
}
int stratum_stepViews(stratum_view* views, int n, stratum_stream_t stream) {
  if (!views || n <= 0) return STRATUM_EINVAL;
  stepViewsK<<<(n + 63) / 64, 64, 0, asStream(stream)>>>(views, n);
  return launchStatus();
}
int stratum_refreshViews(stratum_view* views, int n, stratum_stream_t stream) {
  if (!views || n <= 0 || n > 65535) return STRATUM_EINVAL;
  clearViewsK<<<(n + 63) / 64, 64, 0, asStream(stream)>>>(views, n);
  refreshViewsK<<<dim3(kLots / 128, n), 128, 0, asStream(stream)>>>(views, n);
  return launchStatus();
}
int stratum_buildViews(stratum_view* views, int n, stratum_stream_t stream) {
  if (!views || n <= 0 || n > 65535) return STRATUM_EINVAL;
  int per = stratumHierarchyGrid() / n;
  buildViewsK<<<dim3(per < 16 ? 16 : per, n), kBuildThreads, 0, asStream(stream)>>>(views, n);
  return launchStatus();
}
int stratum_traceViews(stratum_view* views, int n, void* scratch, unsigned long long scratchBytes,
                       const stratum_tune* tune, stratum_stream_t stream) {
  return render(views, n, scratch, scratchBytes, tune, asStream(stream), kTrace);
}
int stratum_shadeViews(stratum_view* views, int n, void* scratch, unsigned long long scratchBytes,
                       const stratum_tune* tune, stratum_stream_t stream) {
  return render(views, n, scratch, scratchBytes, tune, asStream(stream), kShade);
}
int stratum_renderViews(stratum_view* views, int n, void* scratch, unsigned long long scratchBytes,
                        const stratum_tune* tune, stratum_stream_t stream) {
  return render(views, n, scratch, scratchBytes, tune, asStream(stream), kTrace | kShade);
}
// renderViews with the library's static scratch: allocates nothing, calls no
// allocating routine.  The queue counters are cleared on the stream first, so
// the call does not depend on how an earlier call ended.
int stratum_renderViewsNoAlloc(stratum_view* views, int n, const stratum_tune* tune, stratum_stream_t stream) {
  if (!views || n <= 0) return STRATUM_EINVAL;
  if (n > kNoAllocMaxViews) return STRATUM_ELIMIT;
  void* scratch = nullptr;
  int s = noAllocScratch(&scratch);
  if (s != STRATUM_OK) return s;
  cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(uint32_t) * kCounters, asStream(stream));
  if (e != cudaSuccess) return -int(e);
  return render(views, n, scratch, kNoAllocBytes, tune, asStream(stream), kTrace | kShade);
}
int stratum_frameViews(stratum_view* views, int n, void* scratch, unsigned long long scratchBytes,
                       const stratum_tune* tune, stratum_stream_t stream) {
  int s;
  if ((s = stratum_stepViews(views, n, stream)) != STRATUM_OK) return s;
  if ((s = stratum_refreshViews(views, n, stream)) != STRATUM_OK) return s;
  if ((s = stratum_buildViews(views, n, stream)) != STRATUM_OK) return s;
  return stratum_renderViews(views, n, scratch, scratchBytes, tune, stream);
}

}  // extern "C"
