// The 127-node bounding hierarchies of eight lots in one 256-thread block
// (kernels/accel.cu of the reference, fused): lanes are (lot, group) pairs, four
// groups of one kind (the same storey of the four facades) times eight lots, so
// a warp runs one branch of the group bounds (group_bounds.cuh); then each warp
// reduces one lot by shuffles and writes its 4 KiB with coalesced 16-byte
// stores.  Min/max and small-integer sums are exact, so this equals the
// reference's two-kernel form bit for bit.  Node 0 of a lot block is never
// written.
//
// What bounds it is instruction issue, not the 4 KiB a lot (64 MiB a table:
// 10.5 us at the copy rate).  One 64-thread block a lot with a thread a group,
// each walking the whole grammar, ran its 32 branches of a warp one after another:
// 417 us a table (eight tables 3,333 us).  These lanes with the whole grammar
// took 305 us (226 registers, one block an SM), with the attaining features
// alone 66 us, and 47 us (eight tables 378 us) with the trees of parks shared out
// over the warps.  Four blocks an SM (64 registers) measured best: two 432 us,
// three 390 us, six 401 us for the eight tables.
#pragma once
#include "group_bounds.cuh"

namespace st {

// Queue length clamped to the table, so a stale count never reads past the queue.
SD int queued(const uint32_t* Q) { return int(min(Q[0], uint32_t(kLots))); }

constexpr int kBuildLots = 8, kBuildThreads = 256, kBuildBlocks = 4;
constexpr int kLeafWords = 7;                          // bounds and count
constexpr int kLeafRow = kGroups * kLeafWords + 1;     // odd: lots of a warp fall into different banks
static_assert(kBuildThreads / 32 == kBuildLots, "one warp reduces one lot");
struct BuildShared {
  float leaf[kBuildLots][kLeafRow];
  float4 node[kBuildLots][kGroups * 2];  // internal nodes 0..63 (0 is never written out)
  int slot[kBuildLots];
};

// Group k of quad q: the four facades' groups of one kind and storey, so a quad
// runs one branch of the grammar; what is left over makes the last two quads.
SD int quadGroup(int q, int k) {
  if (q == 0) return 2 + k;
  if (q <= 6) return 6 + 6 * k + (q - 1);
  if (q <= 12) return 32 + 6 * k + (q - 7);
  if (q == 13) return 56 + k;
  if (q == 14) return k < 2 ? k : 28 + k;
  return 60 + k;
}

// Up to eight queued lots: lanes are (lot, group of a quad).
SD void lotHierarchies(const uint32_t* Q, const float* W, float* N, int first, int lots, BuildShared& sh) {
  const int lane = int(threadIdx.x & 31), warp = int(threadIdx.x >> 5);
  if (threadIdx.x < kBuildLots) {
    const int s = int(threadIdx.x) < lots ? int(Q[first + int(threadIdx.x) + 1]) : -1;
    sh.slot[threadIdx.x] = s >= 0 && s < kLots ? s : -1;
  }
  __syncthreads();
  const int li = lane & (kBuildLots - 1), slot = sh.slot[li];
  bool park = false;
  if (slot >= 0) {
    const LotDesc lot = loadLotRW(W, slot);
    const bool regular = regularLot(lot);
    park = regular && isTree(lot, 1);
#pragma unroll 1
    for (int q = warp; q < kGroups / 4; q += kBuildThreads / 32) {
      const int g = quadGroup(q, lane / kBuildLots);
      if (regular && isTree(lot, g)) continue;  // the warps share these below
      groupBounds(lot, regular, g, &sh.leaf[li][g * kLeafWords]);
    }
  }
  // The trees of a park's lot: one warp a tree, one lane an envelope.  (As lanes
  // of the quads above, one park lot among eight made five of the eight
  // warps run 28 envelopes for it alone.)
#pragma unroll 1
  for (unsigned parks = __ballot_sync(0xffffffffu, park) & ((1u << kBuildLots) - 1u); parks; parks &= parks - 1u) {
    const int k = __ffs(parks) - 1, g = 1 + warp;
    const LotDesc lot = loadLotRW(W, sh.slot[k]);
    BoundsOf b{lot, BoxUnion{}};
    const float th = treeHeight(lot, g);
    if (lane < 28) treeCrown(b, g, th, lane);
    if (lane == 28) treeTrunk(b, g, th);
    const float v[7] = {warpMin(b.u.lo.x), warpMin(b.u.lo.y), warpMin(b.u.lo.z), 29.0f,
                        warpMax(b.u.hi.x), warpMax(b.u.hi.y), warpMax(b.u.hi.z)};
#pragma unroll
    for (int i = 0; i < 7; i++)
      if (lane == i) sh.leaf[k][g * kLeafWords + i] = v[i];
  }
  __syncthreads();
  const int mine = sh.slot[warp];
  if (mine >= 0) {
    // lane i: node 32 + i from leaves 2i and 2i + 1, then the levels above by
    // shuffles; a lane that is a multiple of the level's step holds its node
    const float* a = &sh.leaf[warp][2 * lane * kLeafWords];
    const float* c = a + kLeafWords;
    float v[7];
#pragma unroll
    for (int k = 0; k < 3; k++) { v[k] = fminf(a[k], c[k]); v[4 + k] = fmaxf(a[4 + k], c[4 + k]); }
    v[3] = a[3] + c[3];
    float4* nodes = sh.node[warp];
#pragma unroll
    for (int step = 1; step <= 32; step <<= 1) {
      if ((lane & (step - 1)) == 0) {
        const int j = (32 + lane) / step;
        nodes[2 * j] = make_float4(v[0], v[1], v[2], v[3]);
        nodes[2 * j + 1] = make_float4(v[4], v[5], v[6], 0.0f);
      }
      if (step == 32) break;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], step));
        v[4 + k] = fmaxf(v[4 + k], __shfl_xor_sync(0xffffffffu, v[4 + k], step));
      }
      v[3] = v[3] + __shfl_xor_sync(0xffffffffu, v[3], step);
    }
    __syncwarp();
    float4* dst = reinterpret_cast<float4*>(N + size_t(mine) * kNodes * 8);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = lane + 32 * k;  // float4 index; 0 and 1 are node 0
      if (i >= 2) dst[i] = nodes[i];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = lane + 32 * k, g = i >> 1;
      const float* l = &sh.leaf[warp][g * kLeafWords + (i & 1) * 4];
      dst[2 * kGroups + i] = make_float4(l[0], l[1], l[2], i & 1 ? float(g) : l[3]);
    }
  }
  __syncthreads();
}

// Grid-stride over one queue: block b takes eight entries at a time.
SD void buildQueue(const uint32_t* Q, const float* W, float* N, int block, int blocks, BuildShared& sh) {
  const int count = queued(Q);
#pragma unroll 1
  for (int q = block * kBuildLots; q < count; q += blocks * kBuildLots)
    lotHierarchies(Q, W, N, q, min(kBuildLots, count - q), sh);
}

}  // namespace st
