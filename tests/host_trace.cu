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
    const unsigned k = poolKey(v, slot, g);
    good += k != kPoolIdle && poolView(k) == v && poolGroupKey(k) == (slot << 6 | g);
  }
  return good;
}

// The relief of n walls (turn 0): the trace's, and its four steps written out with
// nothing left out.  Arguments as ht_culls, and the distance to start from.
static float allSteps(const Feat& f, f3 ro, f3 rd, f3 p, f3 d, float t, float cone) {
  const f3 hp = p + d * t;
  const float ex = fabsf(fabsf(hp.x) - f.h.x), ez = fabsf(fabsf(hp.z) - f.h.z);
  if (!(fabsf(fabsf(hp.y) - f.h.y) > 0.01f)) return t;
  const f3 n = ex < ez ? mk(hp.x < 0.0f ? -1.0f : 1.0f, 0.0f, 0.0f) : mk(0.0f, 0.0f, hp.z < 0.0f ? -1.0f : 1.0f);
  const float denom = dot(n, d), initial = t;
  if (!(denom < -0.08f)) return t;
  for (int k = 0; k < 4; k++) {
    const f3 wp = ro + rd * t;
    float u, v;
    masonryUV(wp, n, u, v);
    const float bw = f.material == 1 ? 0.46f : 0.92f, bh = f.material == 1 ? 0.215f : 0.46f;
    const int row = int(floorf(v / bh));
    const float x = fract(u / bw + float(imod(row, 2)) * 0.5f), y = fract(v / bh);
    const float edge = fminf(fminf(x, 1.0f - x) * bw, fminf(y, 1.0f - y) * bh), grain = noise2(u * 24.0f, v * 24.0f);
    const float chipped = edge - 0.006f * smooth(0.34f, 0.73f, noise2(u * 117.0f, v * 117.0f));
    const float height = -0.018f * (1.0f - smooth(0.008f, 0.023f, chipped)) + 0.0025f * grain;
    t = initial + height * freqWeight(t * cone, 40.0f) / denom;
  }
  return t;
}
extern "C" void ht_relief(const float* boxes, const float* rays, const float* start, const float* cone, int n, float* t,
                          float* whole) {
  for (int i = 0; i < n; i++) {
    const float *b = boxes + 7 * i, *q = rays + 6 * i;
    const Feat f{mk(b[0], b[1], b[2]), mk(b[3], b[4], b[5]), 0, int(b[6]), 0, 0.0f};
    const f3 ro = mk(q[0], q[1], q[2]), rd = mk(q[3], q[4], q[5]), p = ro - f.p;
    t[i] = masonryRelief(f, ro, rd, p, rd, start[i], cone[i]);
    whole[i] = allSteps(f, ro, rd, p, rd, start[i], cone[i]);
  }
}
