// Ray-batch queries against a view's lot table: the nearest feature hit of
// arbitrary rays, through the hierarchy (kernels/trace.cu:8-61 of the
// reference) or exhaustively -- the same lot DDA, but every group of every
// visited lot evaluated in index order with no node culling.  The second form
// is the check of the first (the reference's own hierarchy-vs-exhaustive test,
// tests/native_harness.cpp:68-79, at any scale).
//
// Nothing is shared between arbitrary rays, so both forms spread one ray's
// features over threads.  A feature's distance does not depend on the best so
// far, so the nearest of a group (the first of equal distances) is the least
// (distance, index) in whatever order the features are tested.
#include <mutex>

// (written out: the features of one ray keep coming back to the same code; with one
// copy of each 65,536 rays take 0.62 ms instead of 0.47)
#define STRATUM_QUOTIENT WrittenOut
#include "common_api.cuh"
#include "grammar_ra.cuh"
#include "traverse.cuh"

namespace st {

static __device__ __noinline__ Feat rayFeature(LotDesc L, int g, int i) { return featureAt(L, g, i); }

// Distance of one feature, with the ray's inverse directions in the lot's frame
// given; same value as featureHitCall.
SD float rayFeatureHit(const Feat& f, f3 ro, f3 rd, f3 inv0, float cone) {
  const bool odd = f.turn % 2 == 1;
  const f3 inv = odd ? mk(inv0.z, inv0.y, rd.x == 0.0f ? guardedInv(-rd.x) : -inv0.x) : inv0;
  const f3 p = intoFeature(ro - f.p, f.turn);
  const Span rg = featureSlab(f, p, inv);
  if (featureSlabMiss(f, rg)) return kFar;
  return featureAfterSlab(f, ro, rd, p, intoFeature(rd, f.turn), rg, cone);
}

// The lot DDA of one ray (kernels/trace.cu:33-57).
struct RayDda {
  f3 ro, rd;
  float cone, best, t, tx, tz, dx, dz, farT;
  int fid, slot, wslot, wcx, wcz;  // winner: group * 64 + index, its lot and cell
  int cx, cz, sx, sz, steps;
  f3 lr, ld, inv0;  // the ray in the current lot's frame
};
// Returns whether there is anything to visit.
SD bool ddaBegin(RayDda& r, const float* __restrict__ q) {
  r.ro = mk(q[0], q[1], q[2]); r.rd = mk(q[3], q[4], q[5]); r.cone = q[6];
  r.best = kFar; r.fid = kSkyId; r.wslot = -1; r.wcx = r.wcz = 0; r.slot = 0; r.steps = 0;
  if (r.rd.y < -0.000001f) {
    float ground = -r.ro.y / r.rd.y;
    if (ground > 0.001f && ground < r.best) { r.best = ground; r.fid = kGroundId; }
  }
  float nearT = 0.001f;
  r.farT = r.best;
  if (fabsf(r.rd.y) > 0.0000001f) {
    float a = (-0.5f - r.ro.y) / r.rd.y, c = (kTop - r.ro.y) / r.rd.y;
    nearT = fmaxf(nearT, fminf(a, c));
    r.farT = fminf(r.farT, fmaxf(a, c));
  } else if (r.ro.y > kTop || r.ro.y < -0.5f) r.farT = -1.0f;
  if (!(nearT <= r.farT)) return false;
  r.t = nearT + 0.0002f;
  f3 start = r.ro + r.rd * r.t;
  r.cx = int(floorf((start.x + 18.0f) / kCell));
  r.cz = int(floorf((start.z + 18.0f) / kCell));
  r.sx = r.rd.x > 0.0f ? 1 : -1;
  r.sz = r.rd.z > 0.0f ? 1 : -1;
  float ix = guardedInv(r.rd.x), iz = guardedInv(r.rd.z);
  r.tx = (float(r.cx) * kCell + (r.sx > 0 ? 18.0f : -18.0f) - r.ro.x) * ix;
  r.tz = (float(r.cz) * kCell + (r.sz > 0 ? 18.0f : -18.0f) - r.ro.z) * iz;
  r.dx = kCell * fabsf(ix);
  r.dz = kCell * fabsf(iz);
  return true;
}
// Whether the ray visits its next cell, and the step past it.
SD bool ddaOpen(const RayDda& r) { return r.steps < 160 && !(r.t > r.best || r.t > r.farT || r.t > kFar); }
SD void ddaStep(RayDda& r) {
  r.steps++;
  if (r.tx < r.tz) { r.t = r.tx; r.tx += r.dx; r.cx += r.sx; } else { r.t = r.tz; r.tz += r.dz; r.cz += r.sz; }
}
// The ray in the frame of the lot in its cell.
SD void ddaFrame(RayDda& r, const float* __restrict__ W, uint32_t o0, uint32_t o2) {
  r.slot = tableSlot(o0, o2, r.cx, r.cz);
  const float4 c = __ldg(reinterpret_cast<const float4*>(W + r.slot * kLotFloats) + 2);  // roofScale, turn, ox, oz
  const int turn = int(c.y);
  const f3 cp = mk(float(r.cx) * kCell + c.z, 0.0f, float(r.cz) * kCell + c.w);
  r.lr = toLot(r.ro - cp, turn);
  r.ld = toLot(r.rd, turn);
  r.inv0 = invDir(r.ld);
}
// Out: [t, fid, material, seed, n.xyz, slot] of the finished ray.
SD void ddaStore(const RayDda& r, const float* __restrict__ W, float* out) {
  float4 a = make_float4(r.best, float(r.fid), 10.0f, 0.0f), b = make_float4(0.0f, 1.0f, 0.0f, -1.0f);
  if (r.fid >= 0) {
    const LotDesc L = loadLot(W, r.wslot);
    const Feat f = rayFeature(L, r.fid / kMaxFeatures, r.fid % kMaxFeatures);
    const f3 cp = mk(float(r.wcx) * kCell + L.ox, 0.0f, float(r.wcz) * kCell + L.oz);
    const f3 lr = toLot(r.ro - cp, L.turn), ld = toLot(r.rd, L.turn);
    const f3 n = fromLot(featureNormal(f, lr + ld * r.best), L.turn);
    a.z = float(f.material);
    a.w = f.seed;
    b = make_float4(n.x, n.y, n.z, float(r.wslot));
  }
  reinterpret_cast<float4*>(out)[0] = a;
  reinterpret_cast<float4*>(out)[1] = b;
}

// ---- through the hierarchy ----------------------------------------------------
// A warp owns up to 32 rays.  Each lane descends its own lot's hierarchy near
// first until it reaches a leaf; the warp then evaluates one lane's leaf at a time,
// a feature a lane (random access), and the lane goes on with the best it found.
// What bounds it is instruction issue.  A lane evaluating its own leaves with
// the sequential grammar ran 32 groups' branches one after another (65,536 random
// rays 3.95 ms).
__global__ void __launch_bounds__(64) traceRaysK(const float* __restrict__ W, const float4* __restrict__ N,
                                                const uint32_t* __restrict__ O, const float* __restrict__ rays, int n,
                                                int perWarp, float* out) {
  const int lane = int(threadIdx.x & 31), warp = int(blockIdx.x * 2 + (threadIdx.x >> 5));
  const int i = warp * perWarp + lane;
  const bool active = lane < perWarp && i < n;
  const uint32_t o0 = O[0], o2 = O[2];
  RayDda r;
  r.best = kFar; r.fid = kSkyId; r.cone = 0.0f; r.slot = 0;
  r.lr = r.ld = r.inv0 = mk(0.0f, 0.0f, 0.0f);
  bool more = active && ddaBegin(r, rays + size_t(i) * 7);
  unsigned long long stack = 0ull;  // 7 bits a node, at most 6 entries
  int node = 0, steps = 0, cx = 0, cz = 0, g = -1;
  bool fresh = false;
#pragma unroll 1
  for (;;) {
    // walk to the next leaf (node 0: the lot is finished)
#pragma unroll 1
    while (more && g < 0) {
      if (node == 0 || steps >= kNodes) {
        more = ddaOpen(r);
        node = 0;
        if (!more) continue;
        cx = r.cx; cz = r.cz;
        ddaFrame(r, W, o0, o2);
        ddaStep(r);
        if (nodeEntry(N, r.slot * kNodes + 1, r.lr, r.inv0, r.best) < r.best) {
          node = 1; stack = 0ull; steps = 0; fresh = true;
        }
        continue;
      }
      steps++;
      const int base = r.slot * kNodes;
      // a node reached from its parent was tested against the same best a
      // moment ago; one popped from the stack is tested against the current best
      const bool near = fresh || nodeEntry(N, base + node, r.lr, r.inv0, r.best) < r.best;
      fresh = false;
      if (near && node < kGroups) {
        const float ln = nodeEntry(N, base + 2 * node, r.lr, r.inv0, r.best);
        const float rn = nodeEntry(N, base + 2 * node + 1, r.lr, r.inv0, r.best);
        const bool lh = ln < r.best, rh = rn < r.best;
        if (lh || rh) {
          const bool left = lh && (!rh || ln < rn);
          if (lh && rh) stack = (stack << 7) | (unsigned long long)(2 * node + (left ? 1 : 0));
          node = 2 * node + (left ? 0 : 1);
          fresh = true;
          continue;
        }
      } else if (near) {
        g = node - kGroups;
      }
      node = int(stack & 127ull);
      stack >>= 7;
    }
    unsigned pending = __ballot_sync(0xffffffffu, g >= 0);
    if (!pending) break;
#pragma unroll 1
    for (; pending; pending &= pending - 1u) {
      const int src = __ffs(pending) - 1;
      const int slot = __shfl_sync(0xffffffffu, r.slot, src), sg = __shfl_sync(0xffffffffu, g, src);
      const f3 lr = mk(__shfl_sync(0xffffffffu, r.lr.x, src), __shfl_sync(0xffffffffu, r.lr.y, src),
                       __shfl_sync(0xffffffffu, r.lr.z, src));
      const f3 ld = mk(__shfl_sync(0xffffffffu, r.ld.x, src), __shfl_sync(0xffffffffu, r.ld.y, src),
                       __shfl_sync(0xffffffffu, r.ld.z, src));
      const f3 inv0 = mk(__shfl_sync(0xffffffffu, r.inv0.x, src), __shfl_sync(0xffffffffu, r.inv0.y, src),
                         __shfl_sync(0xffffffffu, r.inv0.z, src));
      const float cone = __shfl_sync(0xffffffffu, r.cone, src), best = __shfl_sync(0xffffffffu, r.best, src);
      const LotDesc L = loadLot(W, slot);
      const int count = groupCount(L, sg);
      float least = kFar;
      int which = kMaxFeatures;
#pragma unroll 1
      for (int j = lane; j < count; j += 32) {
        const float th = rayFeatureHit(rayFeature(L, sg, j), lr, ld, inv0, cone);
        if (th > 0.001f && th < best && th < least) { least = th; which = j; }
      }
      __syncwarp();
      const float t = warpMin(least);
      if (t < kFar) {  // uniform
        const int first = __reduce_min_sync(0xffffffffu, least == t ? which : kMaxFeatures);
        if (lane == src) { r.best = t; r.fid = sg * kMaxFeatures + first; r.wslot = slot; r.wcx = cx; r.wcz = cz; }
      }
    }
    g = -1;
  }
  if (active) ddaStore(r, W, out + size_t(i) * 8);
}

// ---- exhaustively -------------------------------------------------------------
// A block takes eight rays through their next four lots at once: lanes are those
// 32 (ray, lot) pairs, and each of 16 warps evaluates four groups of one kind (the
// same storey of the four facades) for all of them with the sequential grammar,
// so a warp runs one section of it.  The lots of a ray are then merged in order,
// those past the point where the ray ends unused.  What bounds it is instruction
// issue at the lanes that are left: lots differ in family and floors, and the last
// rays of a block in length.  8,192 random rays: a thread per ray (256 warps for
// 592 schedulers, 1,859 features a lot one after another) 59 ms; one lot of eight rays at
// a time with four groups across the lanes 6.0 ms (6.6 of 32 lanes active).
// Rays differ several times over in the lots they cross, so no slot is given rays
// of its own: the block's next ray goes to whichever slot is free.  2,000 rays take
// 1.43 ms and 8,192 2.29 (fixed slots 2.55 and 3.5; a contiguous run of the rays to a
// block, whose neighbours are alike, 1.98 and 7.2).
constexpr int kExRays = 8, kExLots = 4, kExWarps = 16;
// Group k of a warp's four.
SD int warpGroup(int w, int k) {
  if (w < 6) return 6 + 6 * k + w;
  if (w < 12) return 32 + 6 * k + (w - 6);
  if (w == 12) return 2 + k;
  if (w == 13) return 56 + k;
  if (w == 14) return k < 2 ? k : 28 + k;
  return 60 + k;
}
static __device__ __noinline__ float sinkHit(Feat f, f3 ro, f3 rd, f3 inv0, float cone) {
  return rayFeatureHit(f, ro, rd, inv0, cone);
}
struct NearestSink {
  f3 ro, rd, inv0;
  float cone, t;
  int id;
  SD void take(const Feat& f, int k) {
    const float th = sinkHit(f, ro, rd, inv0, cone);
    if (th > 0.001f && th < t) { t = th; id = k; }
  }
};
// (128 registers: at 64, two blocks an SM, 6.3 ms against 3.6 with fixed slots)
__global__ void __launch_bounds__(32 * kExWarps, 1)
    traceExhaustiveK(const float* __restrict__ W, const uint32_t* __restrict__ O, const float* __restrict__ rays, int n,
                     float* out) {
  // least (distance bits, group, index) of each (ray, lot); three in turn, so that
  // one can be cleared while another is read and the third written
  __shared__ unsigned long long least[3][32];
  const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5), mine = lane & (kExRays - 1), ahead = lane / kExRays;
  const unsigned long long none = ~0ull;
  const uint32_t o0 = O[0], o2 = O[2];
  if (threadIdx.x < 96) least[threadIdx.x / 32][threadIdx.x % 32] = none;
  __syncthreads();
  // the block's rays are blockIdx.x, blockIdx.x + gridDim.x, ...; a slot that has
  // finished its own takes the next of them
  const unsigned share = (unsigned(n) - blockIdx.x + gridDim.x - 1u) / gridDim.x;
  unsigned next = 0u, i = 0u;
  int turn = 0;
  bool begun = false;
  RayDda r;  // before the next four lots; the same on every lane of the ray in every warp
#pragma unroll 1
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, !begun) & ((1u << kExRays) - 1u);
    if (!begun) i = next + __popc(idle & ((1u << mine) - 1u));
    next += __popc(idle);
    if (!begun && i < share) {
      if (!ddaBegin(r, rays + (size_t(i) * gridDim.x + blockIdx.x) * 7)) r.steps = 160;  // nothing to visit
      begun = true;
    }
    if (!__any_sync(0xffffffffu, begun)) break;  // every warp holds the same rays: uniform over the block
    RayDda a = r;  // at this lane's lot
    bool in = begun && ddaOpen(a);
#pragma unroll 1
    for (int s = 0; s < ahead && in; s++) {
      ddaStep(a);
      in = ddaOpen(a);
    }
    if (in) {
      ddaFrame(a, W, o0, o2);
      const LotDesc lot = loadLot(W, a.slot);
      unsigned long long key = none;
#pragma unroll 1
      for (int k = 0; k < 4; k++) {
        const int g = warpGroup(warp, k);
        NearestSink s{a.lr, a.ld, a.inv0, a.cone, a.best, -1};
        runGroup(lot, g, s);
        if (s.id >= 0) {
          const unsigned long long c = (unsigned long long)__float_as_uint(s.t) << 32 | unsigned(g * kMaxFeatures + s.id);
          key = c < key ? c : key;
        }
      }
      if (key != none) atomicMin(&least[turn][lane], key);
    }
    const int after = turn == 2 ? 0 : turn + 1;
    if (threadIdx.x < 32) least[after][threadIdx.x] = none;
    __syncthreads();
    if (begun) {
      bool open = true;
#pragma unroll 1
      for (int s = 0; s < kExLots && open; s++) {
        open = ddaOpen(r);
        if (!open) break;
        const unsigned long long key = least[turn][s * kExRays + mine];
        const float t = __uint_as_float(unsigned(key >> 32));
        if (key != none && t < r.best) {
          r.best = t;
          r.fid = int(unsigned(key));
          r.wslot = tableSlot(o0, o2, r.cx, r.cz);
          r.wcx = r.cx; r.wcz = r.cz;
        }
        ddaStep(r);
      }
      if (!open) {
        if (warp == 0 && ahead == 0) ddaStore(r, W, out + (size_t(i) * gridDim.x + blockIdx.x) * 8);
        begun = false;
      }
    }
    turn = after;
  }
}

// One named feature of a table against one ray: the lot of `slot` (its
// descriptor, cell and turn, kernels/world.cu:37-56), record fid % 64 of group
// fid / 64 (the enumeration sink of kernels/sink.cu:21), intersected in that
// lot's frame exactly as the trace forms it (kernels/trace.cu:49-50).
// Out: [t, normal.xyz] (t = FAR if the ray misses it or the id names nothing).
__global__ void __launch_bounds__(64) retestFeaturesK(const float* __restrict__ W, const uint32_t* __restrict__ O,
                                                     const float* __restrict__ rays, const int* __restrict__ ids,
                                                     int n, float* out) {
  int i = int(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n) return;
  const float* q = rays + size_t(i) * 7;
  const int slot = ids[2 * i], fid = ids[2 * i + 1];
  float4 r = make_float4(kFar, 0.0f, 0.0f, 0.0f);
  if (slot >= 0 && slot < kLots && fid >= 0 && fid < kGroups * kMaxFeatures) {
    const LotDesc lot = loadLot(W, slot);
    int cx, cz;
    slotCell(O[0], O[2], slot, cx, cz);
    const f3 ro = mk(q[0], q[1], q[2]), rd = mk(q[3], q[4], q[5]);
    const f3 cp = mk(float(cx) * kCell + lot.ox, 0.0f, float(cz) * kCell + lot.oz);
    const f3 lr = toLot(ro - cp, lot.turn), ld = toLot(rd, lot.turn);
    PickSink pick{fid % kMaxFeatures};
    runGroup(lot, fid / kMaxFeatures, pick);
    if (pick.f.shape >= 0) {
      const float t = featureHitCall(pick.f, lr, ld, q[6]);
      if (t > 0.001f && t < kFar) {
        const f3 nn = fromLot(featureNormal(pick.f, lr + ld * t), lot.turn);
        r = make_float4(t, nn.x, nn.y, nn.z);
      }
    }
  }
  reinterpret_cast<float4*>(out)[i] = r;
}

}  // namespace st

using namespace st;

extern "C" int stratum_retestFeatures(const float* World, const unsigned* Origin, const float* Rays, const int* Ids,
                                      int n, float* Out, stratum_stream_t stream) {
  if (!World || !Origin || !Rays || !Ids || !Out || n < 0) return STRATUM_EINVAL;
  if (n == 0) return STRATUM_OK;
  retestFeaturesK<<<(n + 63) / 64, 64, 0, asStream(stream)>>>(World, Origin, Rays, Ids, n, Out);
  return launchStatus();
}

// Warps the device holds of the hierarchy form, and blocks of the exhaustive form.
struct RayGrids { int warps, blocks; };
static const RayGrids* rayGrids() {
  constexpr int kDevices = 64;
  static std::once_flag once[kDevices];
  static RayGrids grids[kDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return nullptr;
  std::call_once(once[dev], [dev] {
    int sms = 148, a = 0, b = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, traceRaysK, 64, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, traceExhaustiveK, 32 * kExWarps, 0);
    grids[dev] = RayGrids{sms * 2 * (a > 0 ? a : 1), sms * (b > 0 ? b : 1)};
  });
  return &grids[dev];
}

extern "C" int stratum_traceRays(const float* World, const float* Nodes, const unsigned* Origin, const float* Rays,
                                 int n, int exhaustive, float* Out, stratum_stream_t stream) {
  if (!World || !Origin || !Rays || !Out || n < 0 || (!exhaustive && !Nodes)) return STRATUM_EINVAL;
  if (n == 0) return STRATUM_OK;
  const RayGrids* grid = rayGrids();
  if (!grid) return STRATUM_EINVAL;
  if (exhaustive) {
    const int blocks = (n - 1) / kExRays + 1;
    traceExhaustiveK<<<blocks < grid->blocks ? blocks : grid->blocks, 32 * kExWarps, 0, asStream(stream)>>>(World, Origin,
                                                                                                          Rays, n, Out);
    return launchStatus();
  }
  // few rays: fewer to a warp, so that every warp the device holds has some
  const int each = (n - 1) / grid->warps + 1, perWarp = each < 32 ? each : 32;
  const int warps = (n - 1) / perWarp + 1;
  traceRaysK<<<(warps + 1) / 2, 64, 0, asStream(stream)>>>(World, reinterpret_cast<const float4*>(Nodes), Origin, Rays, n,
                                                          perWarp, Out);
  return launchStatus();
}
