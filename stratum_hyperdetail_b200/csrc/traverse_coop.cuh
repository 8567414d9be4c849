// Warp-cooperative primary traversal for the batched renderer.
//
// Same algorithm as traverse.cuh (kernels/trace.cu of the reference), same
// results bit for bit, organised for a warp of 32 coherent rays (one 8x4 tile):
//
//  * each lane steps its own lot DDA to the next lot whose root it enters;
//  * the warp takes the lots its lanes wait in one at a time, the one fewest cells
//    from the camera's first: a ray that reaches a lot has come through nearer
//    ones, so each lot is met once with every ray that will enter it (all lanes'
//    next lots in turn, whatever their distance: 3.88 ms against 3.45, below).  Lanes
//    stand for leaves: all 64 groups of the lot are tested at once against the
//    waiting rays, taken as a packet (packetMayEnter), and each ray then tests the few
//    leaves left (3-7) itself and orders its own by the reference's near-first descent,
//    which needs the hierarchy only where the paths to two of its leaves part;
//  * the warp evaluates one group of that lot at a time for all the lanes that wait
//    on it, the one whose ray has the most leaves to go first, since a ray that is
//    behind may yet come to a group others wait on (the first lane's group instead
//    4.14 ms against 3.88, the nearest 4.34).  Its records come
//    from the table's group cache (group_cache.cuh), the block's table (the
//    drop-in), or the random-access grammar (grammar_ra.cuh), which stores them
//    when the cache has room.  Lanes now stand for records and test them against
//    the packet (packetMayHit): many evaluations end there (64 % on the street pose,
//    30 % on the aerial one, keep no record, the others 2-7 of up to 56), and the
//    waiting lanes test the records kept, in index order, with one inlined
//    intersection routine;
//  * the winner's normal, material and seed are recomputed once per ray.
//
// What bounds the kernel is waiting for instructions (a third of a warp's waiting: a
// tile runs once through most of its 87 KB of code), then dependent
// arithmetic and loads.  One copy of each division, square root and of the step to
// the next leaf took the six-view trace from 4.62 to 4.14 ms at 108 -> 87 KB; at 150 KB
// the aerial pose took twice as long.  Lots and groups in the order above: 3.45 ms
// (street 0.61 -> 0.43, aerial 1.89 -> 1.54).  Six-view 1600x900 trace: each ray walking all records of
// a group behind a box test per run of four, 1,000 (aerial) to 2,500 (street)
// instructions an evaluation, 7.61 ms; records by packet 6.80 ms; without the
// arithmetic of masonry relief and prisms that is certain to come to nothing
// 5.72 ms; leaves by packet instead of a 25-node descent per lane 4.76 ms (street
// 1.18 -> 0.82, aerial 2.29 -> 2.11).  Measured and left out: per-ray candidate
// masks by a ballot per (ray, record) 7.27 ms against 6.80; culling a lot's
// records for all its leaves before the rays order them (street 0.86, aerial 4.43:
// it evaluates groups no ray reaches, which no longer fit the cache); 640 and 768
// threads per SM (spills) 5.16 and 5.01 ms against 4.86.
//
// Each lane's leaves are visited in the reference's order and each test sees
// the same running best, so identity, distance and normal equal the
// per-thread traversal exactly.
#pragma once
#include "geometry.cuh"
#include "grammar_ra.cuh"
#include "group_cache.cuh"
#include "traverse.cuh"

namespace st {

// featureAt out of line: one copy, away from the hot test loop in the
// instruction cache (measured faster than inlining it).
static __device__ __noinline__ Feat featureAtOOL(LotDesc L, int g, int i) { return featureAt(L, g, i); }

// A box (in the lot frame) that contains every distance a feature can return: a
// lane tests a feature only when its ray enters that box nearer than its
// current best (and kReliefReach beyond it), so a skipped feature could only have
// been rejected and results are unchanged.  That holds for the features whose
// computed distance is a slab entry of their own box or follows from it: plain
// boxes and prisms (the slab entry, or a roof plane behind it), masonry boxes (see
// kReliefReach) and foliage envelopes (leaf discs reach at most one 0.18 m grid
// cell, 0.31 m diagonal, beyond the envelope's box: 0.35 m pad).  Ellipsoids,
// cylinders and arches/rings solve a quadratic whose float result can land
// well outside the box at long range (cancellation; 0.17 m at 1.4 km was
// seen), so their box is only bounded along the axis the intersection code
// itself checks: a cylinder's side hit is kept only when its height is within
// +-h.y and its caps lie at +-h.y, so its distance is inside the y slab; an
// arch or ring keeps hits within +-h.z of its own frame (lot x or z by its
// turn); an ellipsoid's root is not checked at all, so its box is unbounded.
// Cache entries also hold the union of these boxes over every run of kRun
// records (the block-pooled trace culls by them).
#ifndef STRATUM_COOP_RUN
#define STRATUM_COOP_RUN 4
#endif
constexpr int kRun = STRATUM_COOP_RUN;
static_assert(kRun * kEntryBoxes >= kEntryRecords, "a group cache entry holds every chunk box of a group");
struct ChunkBox { float lo[3], hi[3]; };
// How far the entry of a masonry box's padded box may lie behind its hit.  Relief moves
// the hit up to 0.0025 m off the face, and faces of a slant down to 0.08 have it: 0.03125 m
// along the ray.  The entry of the box by another axis, which the ray may cross at
// right angles, lies no more than the pad's 0.025 m before the unmoved hit.  So 0.00625 m,
// and the rounding at 2 km.
constexpr float kReliefReach = 0.01f;
HD void hitBox(const Feat& f, f3& lo, f3& hi) {
  const bool foliage = f.shape == 1 && f.material == 7;
  f3 ext = f.h;
  if (f.turn % 2 == 1) ext = mk(f.h.z, f.h.y, f.h.x);
  const float pad = foliage ? 0.35f : 0.025f;
  lo = f.p - ext - mk(pad, pad, pad);
  hi = f.p + ext + mk(pad, pad, pad);
  const float open = 1e30f;
  if (f.shape == 1 && !foliage) {  // ellipsoid: unbounded
    lo = mk(-open, -open, -open);
    hi = mk(open, open, open);
  } else if (f.shape == 2) {  // cylinder: the y slab only
    lo.x = lo.z = -open;
    hi.x = hi.z = open;
  } else if (f.shape == 4 || f.shape == 7) {  // arch, ring: its own z slab only (lot x when the turn is odd)
    lo.y = -open;
    hi.y = open;
    if (f.turn % 2 == 1) { lo.z = -open; hi.z = open; } else { lo.x = -open; hi.x = open; }
  }
}

// The rays a warp serves together, as one packet: they leave one point (the
// camera in the lot's frame) with inverse directions between lo and hi, and
// none wants a hit beyond `best`.
struct Packet { f3 ro, lo, hi; float best; };

// Whether some ray of the packet may hit this record nearer than its own best.
// A ray's slab times of an axis are linear in its inverse direction, so over the
// packet they lie between the extremes of the four products of the box's two
// planes with the interval's two ends; a record is out when the latest of the
// axes' earliest entries is past the earliest of their latest exits, or past
// every ray's best by more than kReliefReach.  The latter holds for boxes (masonry
// relief included) and prisms only: quadrics and foliage are bounded by the box test alone.
// The 0.025 m pad covers every rounding of this test and of the exact one: at
// |ro| <= 2,100 m (a visited lot is at most 2,000 m along a ray) they sum to
// less than 0.001 m.
HD bool packetEnters(const Packet& k, f3 lo, f3 hi, float& in) {
  const float ax = lo.x - k.ro.x, bx = hi.x - k.ro.x, ay = lo.y - k.ro.y, by = hi.y - k.ro.y;
  const float az = lo.z - k.ro.z, bz = hi.z - k.ro.z;
  const float x0 = ax * k.lo.x, x1 = ax * k.hi.x, x2 = bx * k.lo.x, x3 = bx * k.hi.x;
  const float y0 = ay * k.lo.y, y1 = ay * k.hi.y, y2 = by * k.lo.y, y3 = by * k.hi.y;
  const float z0 = az * k.lo.z, z1 = az * k.hi.z, z2 = bz * k.lo.z, z3 = bz * k.hi.z;
  in = fmaxf(fmaxf(fminf(fminf(x0, x1), fminf(x2, x3)), fminf(fminf(y0, y1), fminf(y2, y3))),
             fminf(fminf(z0, z1), fminf(z2, z3)));
  const float out = fminf(fminf(fmaxf(fmaxf(x0, x1), fmaxf(x2, x3)), fmaxf(fmaxf(y0, y1), fmaxf(y2, y3))),
                          fmaxf(fmaxf(z0, z1), fmaxf(z2, z3)));
  return in <= out && out >= 0.001f;
}
// Whether some ray may enter this node's box nearer than its own best.
HD bool packetMayEnter(float4 a, float4 b, const Packet& k) {
  const float pad = 0.01f;
  float in;
  return packetEnters(k, mk(a.x - pad, a.y - pad, a.z - pad), mk(b.x + pad, b.y + pad, b.z + pad), in) && in <= k.best;
}
HD bool packetMayHit(const StagedFeat& s, const Packet& k) {
  const int shape = (s.packed & 255) - 1;
  const bool odd = (s.packed >> 16) & 1, base = shape == 3 || shape == 4;  // these stand on p.y
  const float hx = (odd ? s.hz : s.hx) + 0.025f, hz = (odd ? s.hx : s.hz) + 0.025f, hy = s.hy + 0.025f;
  float in;
  return packetEnters(k, mk(s.px - hx, base ? s.py - 0.025f : s.py - hy, s.pz - hz), mk(s.px + hx, s.py + hy, s.pz + hz), in) &&
         (in <= k.best + kReliefReach || !(shape == 0 || shape == 3));
}
// Whether a ray may hit this record, neither a plain box nor a prism, nearer than `best`.
HD bool mayWin(const Feat& f, f3 ro, f3 inv, float best) {
  f3 lo, hi;
  hitBox(f, lo, hi);
  const Span r = slabInv(ro, inv, lo, hi);
  return !(r.hi < fmaxf(0.001f, r.lo) || r.lo > best + kReliefReach);
}

enum LaneState : int { kEnterLot = 0, kLotPending = 1, kLeafPending = 2, kDone = 3, kNextLeaf = 4 };

struct CoopRay {
  // ray and result
  f3 ro, rd;
  float cone, best;
  int fid, wslot, wcx, wcz;  // winner: group*64+index, slot and DDA cell of its lot
  // lot DDA
  float t, tx, tz, farT;
  f3 inv;  // inverse of rd
  int cx, cz, sx, sz, ddaSteps;
  // current lot
  int slot, lcx, lcz;
  f3 lr, ld, inv0;
  // leaves (groups) of the current lot still to be evaluated, the inner nodes whose
  // right child comes first, the leaf that is next, and whether best has changed
  // since the leaves were found
  unsigned long long leaves, rightFirst;
  int pend, state;
  bool moved;
};

// Ray set-up: ground plane and vertical slab (trace.cu:33-45).
SD void coopBegin(CoopRay& r, f3 ro, f3 rd, float cone, bool active) {
  r.ro = ro; r.rd = rd; r.cone = cone;
  r.best = kFar; r.fid = kSkyId; r.wslot = -1; r.wcx = r.wcz = 0;
  r.state = active ? kEnterLot : kDone;
  r.leaves = r.rightFirst = 0ull; r.moved = false; r.pend = 0; r.slot = 0; r.lcx = r.lcz = 0;
  r.ddaSteps = 0;
  if (!active) return;
  if (rd.y < -0.000001f) {
    float ground = Quotient::div(-ro.y, rd.y);
    if (ground > 0.001f && ground < r.best) { r.best = ground; r.fid = kGroundId; }
  }
  float nearT = 0.001f, farT = r.best;
  if (fabsf(rd.y) > 0.0000001f) {
    float a = Quotient::div(-0.5f - ro.y, rd.y), c = Quotient::div(kTop - ro.y, rd.y);
    nearT = fmaxf(nearT, fminf(a, c));
    farT = fminf(farT, fmaxf(a, c));
  } else if (ro.y > kTop || ro.y < -0.5f) farT = -1.0f;
  r.farT = farT;
  if (!(nearT <= farT)) { r.state = kDone; return; }
  r.t = nearT + 0.0002f;
  f3 start = ro + rd * r.t;
  r.cx = int(floorf(Quotient::div(start.x + 18.0f, kCell)));
  r.cz = int(floorf(Quotient::div(start.z + 18.0f, kCell)));
  r.sx = rd.x > 0.0f ? 1 : -1;
  r.sz = rd.z > 0.0f ? 1 : -1;
  r.inv = invDir<Quotient>(rd);
  r.tx = (float(r.cx) * kCell + (r.sx > 0 ? 18.0f : -18.0f) - ro.x) * r.inv.x;
  r.tz = (float(r.cz) * kCell + (r.sz > 0 ? 18.0f : -18.0f) - ro.z) * r.inv.z;
}

// Inner node where the paths to two leaves part.
SD int forkOf(int a, int b) { return (kGroups + a) >> (32 - __clz(a ^ b)); }

// The order of the lane's leaves: the reference's near-first descent decides
// between two leaves at the node where their paths part, by the entries of its
// two children (ties go right).  Those nodes are the forks of neighbouring
// leaves; nothing else of the hierarchy is read.
SD void orderLeaves(CoopRay& r, const float4* __restrict__ N) {
  const int base = r.slot * kNodes;
  r.rightFirst = 0ull;
  r.moved = false;
  unsigned long long rest = r.leaves;
#pragma unroll 1
  while (rest & (rest - 1ull)) {
    const int a = __ffsll(rest) - 1;
    rest &= rest - 1ull;
    const int fork = forkOf(a, __ffsll(rest) - 1);
    const float ln = nodeEntry(N, base + 2 * fork, r.lr, r.inv0, r.best);
    const float rn = nodeEntry(N, base + 2 * fork + 1, r.lr, r.inv0, r.best);
    if (!(ln < rn)) r.rightFirst |= 1ull << fork;
  }
}

// Take the lane's next leaf in that order, or send it to its next lot.  Once best
// has moved a leaf is tested again and dropped when it has fallen behind, as the
// reference drops it when it gets there: best only falls and a node's entry is
// never after its children's, so a leaf is visited exactly when its own test
// passes then.
SD void nextLeaf(CoopRay& r, const float4* __restrict__ N) {
  r.state = kEnterLot;
#pragma unroll 1
  while (r.leaves) {
    unsigned long long cur = r.leaves;
#pragma unroll 1
    while (cur & (cur - 1ull)) {
      const int first = __ffsll(cur) - 1, last = 63 - __clzll(cur), level = 31 - __clz(first ^ last);
      const unsigned long long below = cur & ((1ull << (((first >> level) | 1) << level)) - 1ull);
      cur = (r.rightFirst >> ((kGroups + first) >> (level + 1))) & 1ull ? cur ^ below : below;
    }
    r.leaves ^= cur;
    const int leaf = __ffsll(cur) - 1;
    if (!r.moved || nodeEntry(N, r.slot * kNodes + kGroups + leaf, r.lr, r.inv0, r.best) < r.best) {
      r.pend = leaf;
      r.state = kLeafPending;
      return;
    }
  }
}

// Step the lane's DDA to the next lot whose root it enters before its best, or to its end.
SD void coopEnterLot(CoopRay& r, const float* __restrict__ W, const float4* __restrict__ N, uint32_t o0, uint32_t o2) {
#pragma unroll 1
  while (r.state == kEnterLot) {
    if (r.ddaSteps >= 160 || r.t > r.best || r.t > r.farT || r.t > kFar) { r.state = kDone; break; }
    r.ddaSteps++;
    r.slot = tableSlot(o0, o2, r.cx, r.cz);
    r.lcx = r.cx; r.lcz = r.cz;
    const float4 c = __ldg(reinterpret_cast<const float4*>(W + r.slot * kLotFloats) + 2);  // roofScale, turn, ox, oz
    const int turn = int(c.y);
    f3 cp = mk(float(r.cx) * kCell + c.z, 0.0f, float(r.cz) * kCell + c.w);
    r.lr = toLot(r.ro - cp, turn);
    r.ld = toLot(r.rd, turn);
    r.inv0 = invToLot(r.inv, r.rd, turn);
    // the DDA steps to the next cell now; the reference does it after the
    // lot's query, and the next test reads only t and the (later) best
    if (r.tx < r.tz) { r.t = r.tx; r.tx += kCell * fabsf(r.inv.x); r.cx += r.sx; }
    else { r.t = r.tz; r.tz += kCell * fabsf(r.inv.z); r.cz += r.sz; }
    if (nodeEntry(N, r.slot * kNodes + 1, r.lr, r.inv0, r.best) < r.best) r.state = kLotPending;
  }
}

// The rays of `peer` lanes, all in the same lot, as one packet.  Warp-collective.
SD Packet lotPacket(const CoopRay& r, bool peer, int src) {
  const float big = 1e30f;
  Packet k;
  k.ro = mk(__shfl_sync(0xffffffffu, r.lr.x, src), __shfl_sync(0xffffffffu, r.lr.y, src),
            __shfl_sync(0xffffffffu, r.lr.z, src));
  k.lo = mk(warpMin(peer ? r.inv0.x : big), warpMin(peer ? r.inv0.y : big), warpMin(peer ? r.inv0.z : big));
  k.hi = mk(warpMax(peer ? r.inv0.x : -big), warpMax(peer ? r.inv0.y : -big), warpMax(peer ? r.inv0.z : -big));
  k.best = warpMax(peer ? r.best : 0.0f);
  return k;
}

// Inverse of the turn-1 direction (ld.z, ld.y, -ld.x): a permutation of inv0
// with one sign flipped, except for an exactly zero ld.x, whose guarded inverse
// keeps the sign of the zero.
SD f3 inv1Of(const CoopRay& r) {
  return mk(r.inv0.z, r.inv0.y, r.ld.x == 0.0f ? guardedInv<Quotient>(-r.ld.x) : -r.inv0.x);
}

// The winner's record for one lane: from the group cache when it holds the
// group, else from the grammar.
SD Feat winnerFeature(const GroupCache& c, const float* __restrict__ W, int slot, int g, int i) {
  const LotDesc L = loadLot(W, slot);
  const int e = c.base ? usableEntry(c, __ldcg(c.dir(slot, g))) : -1;
  if (e >= 0) {
    // the tag (nine descriptor words, group, count) and the record in one round trip
    const uint4* t4 = reinterpret_cast<const uint4*>(entryTag(c, uint32_t(e)));
    const uint4 t0 = __ldg(t4), t1 = __ldg(t4 + 1), t2 = __ldg(t4 + 2);
    const StagedFeat rec = cacheRecord(c, e, i);
    const uint4* r4 = reinterpret_cast<const uint4*>(W + size_t(slot) * kLotFloats);
    const uint4 w0 = __ldg(r4), w1 = __ldg(r4 + 1), w2 = __ldg(r4 + 2);
    const bool same = t0.x == w0.x && t0.y == w0.y && t0.z == w0.z && t0.w == w0.w && t1.x == w1.x &&
                      t1.y == w1.y && t1.z == w1.z && t1.w == w1.w && t2.x == w2.x &&
                      t2.y == uint32_t(g) && t2.z == uint32_t(groupCount(L, g));
    if (same) return unstage(rec);
  }
  return featureAtOOL(L, g, i);
}

constexpr int kRunsPerGroup = (kEntryRecords + kRun - 1) / kRun;
// Shared memory of one warp: the records of the group it serves.
struct WarpStage { StagedFeat feats[kEntryRecords]; };

// Group records shared by the warps of one block, for a trace with no
// table-wide group cache (the drop-in entry point).  Write-once for the
// block's life: a warp that needs a group no entry names claims the next free
// entry for it, builds the records there and marks it ready; a warp that needs a
// group another warp is building waits for that, since the warps of a block set out
// together and come to the same groups at the same time.  Entries are never
// replaced, so the records are read in place.  At most 32 entries: one lane
// checks each entry per lookup.
#ifndef STRATUM_BLOCK_CACHE_ENTRIES
#define STRATUM_BLOCK_CACHE_ENTRIES 32
#endif
constexpr int kBlockEntries = STRATUM_BLOCK_CACHE_ENTRIES;
static_assert(kBlockEntries >= 1 && kBlockEntries <= 32, "one lane per block-cache entry");
constexpr int kBlockWaits = 1024;  // of 64 ns or more; a build takes 2-5 us
struct BlockCache {
  StagedFeat feats[kBlockEntries][kEntryRecords];
  int key[kBlockEntries];  // -1: free
  int count[kBlockEntries];
  volatile int ready[kBlockEntries];
};
// Every thread of the block calls this before any lookup (followed by a
// block-wide barrier).
SD void blockCacheInit(BlockCache& bc) {
  for (int i = int(threadIdx.x); i < kBlockEntries; i += int(blockDim.x)) {
    bc.ready[i] = 0;
    bc.key[i] = -1;
  }
}
// The entry for `key`, which this warp has to fill when `mine`; -1 when the table is
// full.  Entries are claimed in order, so a warp that finds its key in none of them
// and claims the first free one knows that no other has it; losing that entry to
// another warp it looks again (at most once per entry).  Warp-collective.
SD int blockCacheEntry(BlockCache& bc, int key, bool& mine) {
  const int lane = int(threadIdx.x & 31);
  mine = false;
#pragma unroll 1
  for (;;) {
    const int held = lane < kBlockEntries ? reinterpret_cast<volatile int*>(bc.key)[lane] : -2;
    const unsigned same = __ballot_sync(0xffffffffu, held == key), open = __ballot_sync(0xffffffffu, held == -1);
    if (same) return __ffs(same) - 1;
    if (!open) return -1;
    const int e = __ffs(open) - 1;
    int won = 0;
    if (lane == 0) won = atomicCAS(&bc.key[e], -1, key) == -1;
    if (__shfl_sync(0xffffffffu, won, 0)) {
      mine = true;
      return e;
    }
  }
}
// Whether the entry's records can be read, after a bounded wait.  Warp-collective.
SD bool blockCacheReady(const BlockCache& bc, int e) {
#pragma unroll 1
  for (int i = 0; i < kBlockWaits; i++) {
    if (__any_sync(0xffffffffu, bc.ready[e] != 0)) {
      __threadfence_block();  // its records and count were written before its flag
      __syncwarp();           // which some lanes may not have seen yet
      return true;
    }
    __nanosleep(64);
  }
  return false;
}
// Mark an entry this warp has filled.  Warp-collective.
SD void blockCachePublish(BlockCache& bc, int e, int count) {
  if ((threadIdx.x & 31) == 0) bc.count[e] = count;
  __threadfence_block();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) bc.ready[e] = 1;
}

// Build one group's records by the grammar, one feature a lane, storing them
// (with the chunk boxes) when the cache gives an entry; `word` is the directory
// word the caller read.  Warp-collective, out of line: the rare path of a warm
// cache.  `boxes` may be null.
static __device__ __noinline__ void buildGroup(const float* __restrict__ W, GroupCache cache, int key, int count,
                                               uint32_t word, StagedFeat* feats, ChunkBox* boxes) {
  const int lane = int(threadIdx.x & 31);
  const int slot = key >> 6, g = key & 63;
  const LotDesc L = loadLot(W, slot);
  const int e = cacheClaim(cache, slot, g, word);  // -1: build without storing
#pragma unroll 1
  for (int base = 0; base < count; base += 32) {
    const int j = base + lane;
    f3 lo = mk(1e30f, 1e30f, 1e30f), hi = mk(-1e30f, -1e30f, -1e30f);
    if (j < count) {
      StagedFeat s;
      stage(s, featureAtOOL(L, g, j));
      if (e >= 0) entryRecords(cache, uint32_t(e))[j] = s;
      feats[j] = s;
      hitBox(unstage(s), lo, hi);
    }
    if (e < 0 && !boxes) continue;
#pragma unroll
    for (int o = 1; o < kRun; o <<= 1) {
      lo = vmin(lo, mk(__shfl_xor_sync(0xffffffffu, lo.x, o), __shfl_xor_sync(0xffffffffu, lo.y, o),
                       __shfl_xor_sync(0xffffffffu, lo.z, o)));
      hi = vmax(hi, mk(__shfl_xor_sync(0xffffffffu, hi.x, o), __shfl_xor_sync(0xffffffffu, hi.y, o),
                       __shfl_xor_sync(0xffffffffu, hi.z, o)));
    }
    if ((lane & (kRun - 1)) == 0 && j < count) {
      if (boxes) boxes[j / kRun] = ChunkBox{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}};
      if (e >= 0) {
        float* bp = entryBoxes(cache, uint32_t(e)) + (j / kRun) * 6;
        bp[0] = lo.x; bp[1] = lo.y; bp[2] = lo.z; bp[3] = hi.x; bp[4] = hi.y; bp[5] = hi.z;
      }
    }
  }
  if (e >= 0) cachePublish(cache, W, slot, g, count, e);
}

// Stage one group's records and chunk boxes, from the group cache or built.
// Warp-collective; returns the group's record count.
SD int stageGroup(const float* __restrict__ W, const GroupCache& cache, int key, StagedFeat* feats, ChunkBox* boxes) {
  const int lane = int(threadIdx.x & 31);
  const int slot = key >> 6, g = key & 63;
  // the directory word, the lot row, the entry's tag and its records in as few
  // dependent round trips as possible: the records are loaded with the tag and
  // kept only if every tag word matches the slot's current descriptor (else a miss)
  const uint32_t word = cache.base ? __ldcg(cache.dir(slot, g)) : 0u;
  const int count = groupCount(loadLot(W, slot), g);
  const int e = cache.base ? warpEntry(cache, word) : -1;
  if (e >= 0) {
    bool same = true;
    if (lane < kEntryTagWords)
      same = __ldg(entryTag(cache, uint32_t(e)) + lane) == tagWord(W + size_t(slot) * kLotFloats, g, count, lane);
    StagedFeat r0{}, r1{};
    if (lane < count) r0 = cacheRecord(cache, e, lane);
    if (lane + 32 < count) r1 = cacheRecord(cache, e, lane + 32);
    const int runs = (count + kRun - 1) / kRun;
    float2 ba{}, bb{}, bc{};
    if (lane < runs) {
      const float2* bp = reinterpret_cast<const float2*>(entryBoxes(cache, uint32_t(e)) + lane * 6);
      ba = __ldg(bp); bb = __ldg(bp + 1); bc = __ldg(bp + 2);
    }
    if (__all_sync(0xffffffffu, same)) {  // records and chunk boxes as stored
      if (lane < count) feats[lane] = r0;
      if (lane + 32 < count) feats[lane + 32] = r1;
      if (lane < runs) boxes[lane] = ChunkBox{{ba.x, ba.y, bb.x}, {bb.y, bc.x, bc.y}};
      return count;
    }
  }
  buildGroup(W, cache, key, count, word, feats, boxes);
  return count;
}

// Records lane and lane + 32 of a group: from its cache entry, whose tag and
// records are read in one round trip and kept if the tag holds the slot's
// current descriptor words, else from the block's table or built.
// Warp-collective; returns the record count.
template <bool kBlockCache>
SD int groupRecords(const float* __restrict__ W, const GroupCache& cache, BlockCache* bc, int key, WarpStage& ws,
                    StagedFeat& r0, StagedFeat& r1) {
  const int lane = int(threadIdx.x & 31);
  const int slot = key >> 6, g = key & 63;
  StagedFeat* feats = ws.feats;
  uint32_t word = 0u;
  int count, entry = -1;
  bool mine = true;
  if constexpr (kBlockCache) {
    entry = blockCacheEntry(*bc, key, mine);
    if (entry >= 0 && !mine) {
      if (blockCacheReady(*bc, entry)) count = bc->count[entry];
      else { entry = -1; mine = true; }
    } else mine = true;
    if (entry >= 0) feats = bc->feats[entry];
  } else if (cache.base) {
    const uint32_t row = lane < 9 ? __float_as_uint(__ldg(W + slot * kLotFloats + lane)) : 0u;
    word = __ldcg(cache.dir(slot, g));
    const int e = warpEntry(cache, word);
    if (e >= 0) {
      const uint32_t tag = lane < kEntryTagWords ? __ldg(entryTag(cache, uint32_t(e)) + lane) : 0u;
      r0 = cacheRecord(cache, e, lane);
      r1 = cacheRecord(cache, e, min(lane + 32, kEntryRecords - 1));
      const bool same = lane < 9 ? tag == row : lane != 9 || tag == uint32_t(g);
      if (__all_sync(0xffffffffu, same)) return int(__shfl_sync(0xffffffffu, tag, 10));
    } else {
      const int f = filledNow(cache, word, slot, g);
      if (f >= 0) {
        const uint32_t tag = lane < kEntryTagWords ? __ldcg(entryTag(cache, uint32_t(f)) + lane) : 0u;
        r0 = freshRecord(cache, f, lane);
        r1 = freshRecord(cache, f, min(lane + 32, kEntryRecords - 1));
        const bool same = lane < 9 ? tag == row : lane != 9 || tag == uint32_t(g);
        if (__all_sync(0xffffffffu, same)) return int(__shfl_sync(0xffffffffu, tag, 10));
      }
    }
  }
  if (mine) {
    count = groupCount(loadLot(W, slot), g);
    buildGroup(W, cache, key, count, word, feats, nullptr);
    __syncwarp();
    if constexpr (kBlockCache)
      if (entry >= 0) blockCachePublish(*bc, entry, count);
  }
  r0 = feats[lane];
  r1 = feats[min(lane + 32, kEntryRecords - 1)];
  __syncwarp();
  return count;
}

// Find and order the leaves of every lane that waits in lane `src`'s lot; those lanes.  Warp-collective.
SD unsigned coopLot(CoopRay& r, const float4* __restrict__ N, int src) {
  const int lane = int(threadIdx.x & 31), slot = __shfl_sync(0xffffffffu, r.slot, src);
  const bool peer = r.state == kLotPending && r.slot == slot;
  // lanes are leaves: which of the lot's 64 can any peer's ray enter
  const float4* leaf = N + 2 * (slot * kNodes + kGroups + lane);
  const float4 a0 = __ldg(leaf), b0 = __ldg(leaf + 1), a1 = __ldg(leaf + 64), b1 = __ldg(leaf + 65);
  const Packet pk = lotPacket(r, peer, src);
  const unsigned m0 = __ballot_sync(0xffffffffu, a0.w > 0.5f && packetMayEnter(a0, b0, pk));
  const unsigned m1 = __ballot_sync(0xffffffffu, a1.w > 0.5f && packetMayEnter(a1, b1, pk));
  if (peer) {
    const int base = slot * kNodes + kGroups;
    r.leaves = 0ull;
#pragma unroll 1
    for (unsigned long long rest = (unsigned long long)m1 << 32 | m0; rest; rest &= rest - 1ull) {
      const int k = __ffsll(rest) - 1;
      if (nodeEntry(N, base + k, r.lr, r.inv0, r.best) < r.best) r.leaves |= 1ull << k;
    }
    orderLeaves(r, N);
    r.state = kNextLeaf;
  }
  return __ballot_sync(0xffffffffu, peer);
}

// Advance every lane until it has a leaf to evaluate or is done.  Warp-collective.
SD void coopAdvance(CoopRay& r, const float* __restrict__ W, const float4* __restrict__ N, uint32_t o0, uint32_t o2) {
#pragma unroll 1
  for (;;) {
    coopEnterLot(r, W, N, o0, o2);
    unsigned lots = __ballot_sync(0xffffffffu, r.state == kLotPending);
    if (!lots) return;
#pragma unroll 1
    while (lots) lots &= ~coopLot(r, N, __ffs(lots) - 1);
    if (r.state == kNextLeaf) nextLeaf(r, N);
  }
}

// The whole warp traces its 32 rays.  Every lane of the warp must call this
// (inactive lanes with active = false).  `ws` is this warp's shared-memory
// staging area; `cache` is the table's group cache (null base: none).
// kBlockCache: the block's warps share the groups they build through `bc`
// (the drop-in trace); otherwise `bc` is unused.
template <bool kBlockCache = false>
SD TraceResult traceWarp(const float* __restrict__ W, const float4* __restrict__ N, uint32_t o0, uint32_t o2, f3 ro,
                         f3 rd, float cone, bool active, WarpStage& ws, const GroupCache& cache,
                         BlockCache* bc = nullptr) {
  const int lane = int(threadIdx.x & 31);
  CoopRay r;
  coopBegin(r, ro, rd, cone, active);
#pragma unroll 1
  for (;;) {
    if (r.state == kNextLeaf) nextLeaf(r, N);
    if (!__any_sync(0xffffffffu, r.state == kLeafPending)) {
      coopEnterLot(r, W, N, o0, o2);
      // the lot fewest cells away (the camera is in cell 0 or next to it)
      const unsigned far = r.state == kLotPending ? unsigned(abs(r.lcx) + abs(r.lcz)) : ~0u;
      const unsigned nearest = __reduce_min_sync(0xffffffffu, far);
      if (nearest == ~0u) break;  // every lane is done
      coopLot(r, N, __ffs(__ballot_sync(0xffffffffu, far == nearest)) - 1);
      continue;
    }
    // a lane's group, the one with most leaves to go, for every lane that waits on it
    const int myKey = (r.slot << 6) | r.pend;
    const unsigned left = r.state == kLeafPending ? unsigned(__popcll(r.leaves)) + 1u : 0u;
    const int from = __ffs(__ballot_sync(0xffffffffu, left == __reduce_max_sync(0xffffffffu, left))) - 1;
    const int key = __shfl_sync(0xffffffffu, myKey, from);
    const bool peer = r.state == kLeafPending && myKey == key;
    const unsigned peers = __ballot_sync(0xffffffffu, peer);
    // lanes are records: which of the group's can any peer's ray hit
    StagedFeat r0, r1;
    const int count = groupRecords<kBlockCache>(W, cache, bc, key, ws, r0, r1);
    const Packet pk = lotPacket(r, peer, __ffs(peers) - 1);
    unsigned m0 = 0u, m1 = 0u;
#pragma unroll 1
    for (int half = 0; half < count; half += 32) {
      if (half) r0 = r1;
      const unsigned m = __ballot_sync(0xffffffffu, lane + half < count && packetMayHit(r0, pk));
      if ((m >> lane) & 1u) ws.feats[lane + half] = r0;
      if (half) m1 = m; else m0 = m;
    }
    __syncwarp();
    if (peer) {
      // those records in index order: the first feature wins ties
      const int g = r.pend;
      unsigned mlo = m0, mhi = m1;
#pragma unroll 1
      while (mlo | mhi) {
        const int k = mlo ? __ffs(mlo) - 1 : __ffs(mhi) + 31;
        if (mlo) mlo &= mlo - 1u; else mhi &= mhi - 1u;
        const Feat f = unstage(ws.feats[k]);
        const bool odd = f.turn % 2 == 1;
        const f3 inv = odd ? inv1Of(r) : r.inv0, p = intoFeature(r.lr - f.p, f.turn);
        const Span rg = featureSlab(f, p, inv);
        if (featureSlabMiss(f, rg)) continue;
        float th;
        if (plainBox(f)) {
          th = plainBoxHit(rg);
        } else {
          const f3 d = odd ? mk(r.ld.z, r.ld.y, -r.ld.x) : r.ld;
          if (f.shape == 3) {  // its distance is never before the slab's entry
            if (rg.lo > r.best || prismMiss(f, p, d, rg)) continue;
          } else if (!mayWin(f, r.lr, r.inv0, r.best)) {
            continue;
          }
          th = featureInSlabOOL(f, r.lr, r.ld, p, d, rg, r.cone);
        }
        if (th > 0.001f && th < r.best) {
          r.best = th; r.fid = g * kMaxFeatures + k; r.wslot = r.slot; r.wcx = r.lcx; r.wcz = r.lcz;
          r.moved = true;
        }
      }
      r.state = kNextLeaf;
    }
    __syncwarp();
  }
  TraceResult out;
  out.t = r.best; out.fid = r.fid; out.material = 10; out.seed = 0.0f; out.slot = -1;
  out.normal = mk(0.0f, 1.0f, 0.0f);
  if (r.fid >= 0) {  // the winner's record, lot frame and normal (trace.cu:53-54)
    const LotDesc L = loadLot(W, r.wslot);
    const Feat f = winnerFeature(cache, W, r.wslot, r.fid >> 6, r.fid & 63);
    f3 cp = mk(float(r.wcx) * kCell + L.ox, 0.0f, float(r.wcz) * kCell + L.oz);
    f3 lr = toLot(ro - cp, L.turn), ld = toLot(rd, L.turn);
    out.normal = fromLot(featureNormal(f, lr + ld * r.best), L.turn);
    out.material = f.material;
    out.seed = f.seed;
    out.slot = r.wslot;
  }
  return out;
}

}  // namespace st
