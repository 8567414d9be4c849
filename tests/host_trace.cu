// Test infrastructure: what the traces decide by, compiled for the HOST: the record
// culls against the distance of the same record, and the heads of the block-pooled form.
#define STRATUM_QUOTIENT WrittenOut
#include "common_api.cuh"
#include "traverse_pool.cuh"

using namespace st;

// One ray in the lot's frame against a box of turn 0: its distance (kFar: a miss), with
// the relief of tall stone and brick.
static float boxHit(const Feat& f, f3 ro, f3 rd, float cone) {
  const f3 p = ro - f.p;
  const Span rg = featureSlab(f, p, invDir(rd));
  if (featureSlabMiss(f, rg)) return kFar;
  float t = rg.lo > 0.001f ? rg.lo : rg.hi;
  if ((f.material == 0 || f.material == 1) && f.h.y > 1.0f) t = masonryRelief(f, ro, rd, p, rd, t, cone);
  return t <= 0.001f ? kFar : t;
}

// n boxes (centre, half extent, material) and rays (origin, direction): of those hit, the
// distance in t[], and in kept[] whether the record passes the packet's cull (bit 0)
// and the ray's own (bit 1) when the ray's best lies just behind that distance.
extern "C" void ht_culls(const float* boxes, const float* rays, int n, float cone, float* t, int* kept) {
  for (int i = 0; i < n; i++) {
    const float *b = boxes + 7 * i, *q = rays + 6 * i;
    const Feat f{mk(b[0], b[1], b[2]), mk(b[3], b[4], b[5]), 0, int(b[6]), 0, 0.0f};
    const f3 ro = mk(q[0], q[1], q[2]), rd = mk(q[3], q[4], q[5]), inv = invDir(rd);
    t[i] = boxHit(f, ro, rd, cone);
    const float best = t[i] * 1.0000002f;
    StagedFeat s;
    stage(s, f);
    kept[i] = (packetMayHit(s, Packet{ro, inv, inv, best}) ? 1 : 0) | (mayWin(f, ro, inv, best) ? 2 : 0);
  }
}

// The block-pooled trace's heads of n (view, slot, group): whether each is told from an
// idle lane and read back as it was.
extern "C" int ht_heads(const int* heads, int n) {
  int good = 0;
  for (int i = 0; i < n; i++) {
    const int v = heads[3 * i], slot = heads[3 * i + 1], g = heads[3 * i + 2];
    const unsigned long long k = poolKey(v, slot, g);
    good += k != kPoolIdle && poolView(k) == v && poolGroupKey(k) == (slot << 6 | g);
  }
  return good;
}
