// What the traversals share (kernels/trace.cu of the reference): a traced ray's
// result, the node test and the frame stores.
#pragma once
#include "geometry.cuh"

namespace st {

struct TraceResult {
  float t, seed;
  int fid, material, slot;
  f3 normal;
};

// Node = two 128-bit loads: [lo.xyz, count], [hi.xyz, group].
SD float nodeEntry(const float4* __restrict__ N, int node, f3 ro, f3 inv, float best) {
  float4 a = __ldg(N + 2 * node);
  if (a.w < 0.5f) return kFar;
  float4 b = __ldg(N + 2 * node + 1);
  Span r = slabInv(ro, inv, mk(a.x, a.y, a.z), mk(b.x, b.y, b.z));
  if (r.hi < fmaxf(0.001f, r.lo) || r.lo > best) return kFar;
  return fmaxf(0.001f, r.lo);
}

SD void storeTrace(float* Hit, float* Surface, size_t px, const TraceResult& r) {
  reinterpret_cast<float4*>(Hit)[px] = make_float4(r.t, float(r.fid), float(r.material), r.seed);
  reinterpret_cast<float4*>(Surface)[px] = make_float4(r.normal.x, r.normal.y, r.normal.z, float(r.slot));
}

}  // namespace st
