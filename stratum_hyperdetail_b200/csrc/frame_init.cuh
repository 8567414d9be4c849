// A frame's constants worked out by the first warp of a block, one angle a lane:
// the sines and cosines are evaluated in double precision (stratum_math.cuh) and
// take most of the time of makeFrame, makeCamera and makeTaps.  Same values.
#pragma once
#include "shading.cuh"

namespace st {

// Every thread of the block calls these; frameInit and cameraInit end in a block barrier.
SD Camera cameraOf(const float* C, float s3, float c3, float s4, float c4, float hx, float hy) {
  Camera c;
  c.pos = mk(C[0], C[1], C[2]);
  c.fwd = mk(s3 * c4, s4, c3 * c4);
  c.right = mk(c3, 0.0f, -s3);
  c.up = cross(c.fwd, c.right);
  const int sample = int(C[19]) - 1;
  c.jx = sample > 0 ? hx - 0.5f : 0.0f;
  c.jy = sample > 0 ? hy - 0.5f : 0.0f;
  return c;
}
// Lane 2i: sine, lane 2i + 1: cosine of angle i (yaw, pitch, sun's two); lanes 8 and 9: the jitter.
SD float frameTerm(const float* C, int lane) {
  const int sample = int(C[19]) - 1;
  if (lane < 8) {
    const float a = C[lane < 4 ? 3 + (lane >> 1) : 5 + (lane >> 1)];
    return (lane & 1) ? cosR(a) : sinR(a);
  }
  return lane < 10 && sample > 0 ? halton(sample, lane == 8 ? 2 : 3) : 0.0f;
}
SD void frameInit(FrameConst& F, const float* C, const uint32_t* O) {
  if (threadIdx.x < 32) {
    const float v = frameTerm(C, int(threadIdx.x));
    float t[10];
#pragma unroll
    for (int i = 0; i < 10; i++) t[i] = __shfl_sync(0xffffffffu, v, i);
    if (threadIdx.x == 0) {
      F.cam = cameraOf(C, t[0], t[1], t[2], t[3], t[8], t[9]);
      F.sun = unit(mk(t[5] * t[7], t[6], t[4] * t[7]));
      for (int i = 0; i < 4; i++) F.o[i] = O ? O[i] : 0u;
      F.exposure = C[9]; F.view = C[11]; F.shadowsOff = C[18]; F.sample = C[19];
      F.seed = int(C[14]);
    }
  }
  __syncthreads();
}
SD void tapsInit(ResolveTaps& r) {
  if (threadIdx.x >= 32 && threadIdx.x < 48) {
    const int k = int(threadIdx.x) - 32 >> 1;
    const float a = float(k) * kPi * 0.25f + 0.2f;
    if (threadIdx.x & 1) r.s[k] = sinR(a); else r.c[k] = cosR(a);
  }
}

}  // namespace st
