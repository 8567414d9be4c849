// The block-pooled trace (traverse_pool.cuh): a block claims THREADS / 32 tiles at once,
// one per warp, and its warps serve one another's groups.
//
// 512 threads per SM (128 registers) and divisions written out: the warps of a block
// share more of their way through the code than those of the per-warp trace, and wait for
// one another's spills.  One view with a filled cache, street and aerial together, 64 / 128
// threads in us, as the per-warp trace has it (576 threads, one copy of each division) and
// so: 64x64 2,399 / 2,316 and 1,862 / 2,122, 320x180 2,631 / 2,524 and 2,059 / 2,223, 1600x900
// 9,773 / 9,793 and 8,665 / 8,630.  What is left against a descent of each lane through its
// own lot (64x64 1,772 / 1,941) is the packet test of a lot's leaves, which gains from
// 320x180 on (2,008 / 2,184; 1600x900 11,407 / 11,621).
#include <mutex>

#define STRATUM_QUOTIENT WrittenOut
#include "batch.cuh"
#include "common_api.cuh"
#include "traverse_pool.cuh"

namespace st {

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS)
    tracePooledK(const stratum_view* __restrict__ V, int n, int order, BatchScratch* S) {
  constexpr int P = THREADS / 32;
  extern __shared__ __align__(16) unsigned char poolBytes[];
  PoolShared<P>& sh = *reinterpret_cast<PoolShared<P>*>(poolBytes);
  __shared__ int firstTile;
  const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
  const int total = int(S->counters[kTotalTiles]);
#pragma unroll 1
  for (;;) {
    if (threadIdx.x == 0) firstTile = int(atomicAdd(&S->counters[kTraceNext], uint32_t(P)));
    __syncthreads();
    const int t0 = firstTile;
    __syncthreads();  // every thread has read it before it is written again
    if (t0 >= total) break;
    const int tile = t0 + warp;
    int v = 0, W = 1, H = 1, tx = 0, ty = 0;
    bool ok = tile < total;
    if (ok) {
      v = viewOf(V, n, tile);
      W = V[v].width;
      H = V[v].height;
      ok = tileCoord(tile - V[v].tileBase, V[v].tilesX, (H + kTileH - 1) / kTileH, order, tx, ty);
    }
    const int x = tx * kTileW + (lane & 7), y = ty * kTileH + (lane >> 3);
    const bool inFrame = ok && x < W && y < H;
    const Camera cam = S->view[v].frame.cam;
    const uint32_t o0 = S->view[v].frame.o[0], o2 = S->view[v].frame.o[2];
    const f3 rd = primaryDir<Quotient>(cam, inFrame ? x : 0, inFrame ? y : 0, W, H);
    const TraceResult r = tracePooled<P>(sh, V, v, V[v].World, reinterpret_cast<const float4*>(V[v].Nodes), o0, o2,
                                         cam.pos, rd, 1.08f / float(H), inFrame);
    if (inFrame) storeTrace(V[v].Hit, V[v].Surface, size_t(y) * W + x, r);
  }
  retire(&S->counters[kTraceNext], &S->counters[kTraceDone], THREADS);
}

template <int THREADS>
void launchPooled(const stratum_view* V, int n, int order, BatchScratch* S, int dev, cudaStream_t stream) {
  static std::once_flag once[kGridDevices];
  static int blocks[kGridDevices];
  constexpr size_t smem = sizeof(PoolShared<THREADS / 32>);
  std::call_once(once[dev], [dev] { blocks[dev] = residentBlocks(tracePooledK<THREADS>, THREADS, smem); });
  tracePooledK<THREADS><<<blocks[dev], THREADS, smem, stream>>>(V, n, order, S);
}
template void launchPooled<64>(const stratum_view*, int, int, BatchScratch*, int, cudaStream_t);
template void launchPooled<128>(const stratum_view*, int, int, BatchScratch*, int, cudaStream_t);
template void launchPooled<256>(const stratum_view*, int, int, BatchScratch*, int, cudaStream_t);

}  // namespace st
