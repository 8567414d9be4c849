// Test infrastructure: the device's group bounds compiled for the HOST, by the
// whole grammar and by the features that attain them, for a CPU comparison.
#include "group_bounds.cuh"

using namespace st;

extern "C" int hb_regular(const float* lot16) { return regularLot(loadLotRW(lot16, 0)); }

// out = lo.xyz, count, hi.xyz; whole = 1: the whole grammar
extern "C" void hb_bounds(const float* lot16, int group, int whole, float* out) {
  const LotDesc l = loadLotRW(lot16, 0);
  groupBounds(l, !whole && regularLot(l), group, out);
}

// Rows whose fast and whole bounds differ in any bit, over all 64 groups.
extern "C" int hb_differ(const float* lots, int n, int* where) {
  int bad = 0;
  for (int i = 0; i < n; i++)
    for (int g = 0; g < 64; g++) {
      float a[7], b[7];
      hb_bounds(lots + 16 * i, g, 0, a);
      hb_bounds(lots + 16 * i, g, 1, b);
      for (int k = 0; k < 7; k++)
        if (__builtin_memcmp(a + k, b + k, 4) != 0) {
          if (bad < 64) { where[3 * bad] = i; where[3 * bad + 1] = g; where[3 * bad + 2] = k; }
          bad++;
          break;
        }
    }
  return bad;
}
