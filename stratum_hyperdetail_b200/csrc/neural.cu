// The optional material surrogate's kernels (kernels/learning.cu of the
// reference, see neural.cuh): parameter initialisation, one training step and
// the surrogate-shaded drop-in.
//
// A training step is ~64 samples x 291 parameters of work, so the reference's
// five launches (prepare, forward, score, gradient, Adam) are one block here:
// the samples' work rows and the gradient stay in shared memory and the phases
// are separated by block barriers.
#include "neural.cuh"
#include "strips.cuh"

namespace st {

// learning.cu:5-10
__global__ void initNeuralK(float* W, float* M, float* V, float* Brain, int seed) {
  const int i = int(blockIdx.x * blockDim.x + threadIdx.x);
  if (i < kNnParams) {
    W[i] = (hash1(i + seed) - 0.5f) * 0.08f;
    M[i] = 0.0f;
    V[i] = 0.0f;
    if (i >= kNnW2) W[i] = 0.0f;
  }
  if (i < 32) Brain[i] = 0.0f;
  if (i == kNnB2) W[i] = 0.36f;
  if (i == kNnB2 + 1) W[i] = 0.29f;
  if (i == kNnB2 + 2) W[i] = 0.20f;
}

constexpr int kStepThreads = 320;  // >= 291 parameters and >= 64 samples

// One training step (learning.cu:11-58) on a frame's Hit/Surface.  One block, so
// what bounds it is the longest chain of dependent steps, not work: every phase is
// spread over all threads as far as its sums allow (their order is kept).  With
// a thread a sample, and then a thread a parameter, it took 25 us, now 23.
__global__ void __launch_bounds__(kStepThreads) materialStepK(const float* __restrict__ World,
                                                             const uint32_t* __restrict__ O,
                                                             const float* __restrict__ C,
                                                             const float* __restrict__ Hit,
                                                             const float* __restrict__ Surface, float* W, float* M,
                                                             float* V, float* Brain, float* WorkOut, int width,
                                                             int height) {
  constexpr int kTrials = 6;
  __shared__ float work[kNnBatch * kNnWs];
  __shared__ float weight[kNnParams], grad[kNnParams], delta[kNnTrain * kNnHidden], decay[2];
  __shared__ float su[kNnBatch], sv[kNnBatch], seedOf[kNnBatch];
  __shared__ int pick[kNnBatch];
  __shared__ FrameConst F;
  if (!materialTrainNow(C)) return;  // uniform over the block
  const int i = int(threadIdx.x);
  for (int k = i; k < kNnBatch * kNnWs; k += kStepThreads) work[k] = 0.0f;
  if (i < kNnBatch) pick[i] = -1;
  if (i < kNnParams) weight[i] = W[i];
  frameInit(F, C, O);
  // prepare (learning.cu:11-24): the last of six hashed pixels that hit brick or stone
  auto pixelOf = [&](int sample, int trial) {
    return int(hash1(sample * 1877 + trial * 331 + int(C[6]) * 59) * float(width * height));
  };
  for (int k = i; k < kNnBatch * kTrials; k += kStepThreads) {
    const int sample = k / kTrials, trial = k % kTrials;
    const float4 h = reinterpret_cast<const float4*>(Hit)[pixelOf(sample, trial)];
    if (int(h.y) >= 0) {
      const int mat = int(h.z);
      if (mat == 0 || mat == 1) atomicMax(&pick[sample], trial);
    }
  }
  __syncthreads();
  if (i < kNnBatch && pick[i] >= 0) {
    float* w = work + i * kNnWs;
    const int chosen = pixelOf(i, pick[i]), x = chosen % width, y = chosen / width;
    const f3 rd = primaryDir(F.cam, x, y, width, height);
    const float4 h = reinterpret_cast<const float4*>(Hit)[chosen];
    const float4 s = reinterpret_cast<const float4*>(Surface)[chosen];
    SurfacePoint sp;
    surfacePoint(World, F, h, s, rd, height, sp);
    su[i] = sp.u; sv[i] = sp.v; seedOf[i] = h.w;
    w[kNnValid] = 1.0f;
    w[kNnMat] = float(int(h.z));
  }
  __syncthreads();
  for (int k = i; k < kNnBatch * (kNnInputs + 1); k += kStepThreads) {  // target and inputs, a kind to a run of threads
    const int j = k / kNnBatch, sample = k % kNnBatch;
    float* w = work + sample * kNnWs;
    if (pick[sample] < 0) continue;
    const int mat = int(w[kNnMat]);
    if (j == 0) {
      const f3 target = substrate(su[sample], sv[sample], seedOf[sample], mat);
      w[kNnTarget] = target.x; w[kNnTarget + 1] = target.y; w[kNnTarget + 2] = target.z;
    } else {
      w[j - 1] = nnFeature(j - 1, su[sample], sv[sample], seedOf[sample], mat);
    }
  }
  __syncthreads();
  // forward (learning.cu:25-29)
  for (int k = i; k < kNnBatch * kNnHidden; k += kStepThreads) {
    const int h = k / kNnBatch;
    float* w = work + (k % kNnBatch) * kNnWs;
    float z = weight[kNnB1 + h];
    for (int j = 0; j < kNnInputs; j++) z += weight[h * 8 + j] * w[j];
    w[kNnHid + h] = nnActivate(z);
  }
  __syncthreads();
  for (int k = i; k < kNnBatch * 3; k += kStepThreads) {
    const int o = k / kNnBatch;
    float* w = work + (k % kNnBatch) * kNnWs;
    float z = weight[kNnB2 + o];
    for (int h = 0; h < kNnHidden; h++) z += weight[kNnW2 + o * 24 + h] * w[kNnHid + h];
    w[kNnOut + o] = z;
  }
  __syncthreads();
  // a hidden unit's error on each training sample (learning.cu:42-52)
  for (int k = i; k < kNnTrain * kNnHidden; k += kStepThreads) {
    const int h = k / kNnTrain, sample = k % kNnTrain;
    const float* w = work + sample * kNnWs;
    float d = 0.0f;
    for (int o = 0; o < 3; o++) d += (w[kNnOut + o] - w[kNnTarget + o]) * weight[kNnW2 + o * 24 + h];
    const float a = w[kNnHid + h];
    d *= 1.0f - a * a;
    delta[h * kNnTrain + sample] = d;
  }
  // score on the 8 held-out samples and the validation gate (learning.cu:30-41)
  if (i == kStepThreads - 1) {
    float err = 0.0f, baseline = 0.0f, n = 0.0f;
    for (int k = kNnTrain; k < kNnBatch; k++) {
      const float* w = work + k * kNnWs;
      if (w[kNnValid] > 0.5f) {
        n += 1.0f;
        const f3 mean = substrateMean(int(w[kNnMat]));
        for (int o = 0; o < 3; o++) {
          const float d = w[kNnOut + o] - w[kNnTarget + o];
          err += d * d;
          const float m = o == 0 ? mean.x : (o == 1 ? mean.y : mean.z);
          const float e = m - w[kNnTarget + o];
          baseline += e * e;
        }
      }
    }
    if (n > 0.0f) {
      const float a = Brain[1] < 1.0f ? 1.0f : 0.065f;
      Brain[2] = lerp(Brain[2], err / (n * 3.0f), a);
      Brain[3] = lerp(Brain[3], baseline / (n * 3.0f), a);
      Brain[1] += n;
    }
    Brain[4] = Brain[1] >= 256.0f && Brain[2] < Brain[3] * 0.90f && Brain[2] < 0.0012f ? 1.0f : 0.0f;
  }
  __syncthreads();
  // gradient over the 56 training samples (learning.cu:42-52)
  float count = 0.0f;
  for (int k = 0; k < kNnTrain; k++) count += work[k * kNnWs + kNnValid] > 0.5f ? 1.0f : 0.0f;
  const float steps = Brain[0] + (count > 0.0f ? 1.0f : 0.0f);
  if (i < kNnParams) {
    float g = 0.0f;
    for (int k = 0; k < kNnTrain; k++) {
      const float* w = work + k * kNnWs;
      if (w[kNnValid] > 0.5f) {
        if (i < kNnB1) g += delta[(i / 8) * kNnTrain + k] * w[i % 8];
        else if (i < kNnW2) g += delta[(i - kNnB1) * kNnTrain + k];
        else if (i < kNnB2) g += (w[kNnOut + (i - kNnW2) / 24] - w[kNnTarget + (i - kNnW2) / 24]) * w[kNnHid + (i - kNnW2) % 24];
        else g += w[kNnOut + i - kNnB2] - w[kNnTarget + i - kNnB2];
      }
    }
    grad[i] = clampv(g / fmaxf(1.0f, count), -0.8f, 0.8f);
  } else if (i == 296 || i == 297) {
    decay[i - 296] = 1.0f - powR(i == 296 ? 0.9f : 0.999f, steps);
  }
  __syncthreads();
  if (i == 0) {
    Brain[0] = steps;
    Brain[5] = count;
  }
  // Adam (learning.cu:53-58)
  if (i < kNnParams && count >= 1.0f) {
    const float g = grad[i];
    const float m = 0.9f * M[i] + 0.1f * g, v = 0.999f * V[i] + 0.001f * g * g;
    M[i] = m;
    V[i] = v;
    const float mh = m / decay[0], vh = v / decay[1];
    W[i] = weight[i] - 0.002f * (mh / (sqrtf(vh) + 0.00001f) + 0.0001f * weight[i]);
  }
  if (WorkOut)
    for (int k = i; k < kNnBatch * kNnWs; k += kStepThreads) WorkOut[k] = work[k];
}

// The surrogate's colour for n queries [u, v, seed, material].
__global__ void predictSubstrateK(const float* __restrict__ W, const float* __restrict__ Q, int n, float* Out) {
  const int i = int(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n) return;
  const float* q = Q + size_t(i) * 4;
  const f3 c = predictSubstrate(W, q[0], q[1], q[2], int(q[3]));
  Out[size_t(i) * 3] = c.x; Out[size_t(i) * 3 + 1] = c.y; Out[size_t(i) * 3 + 2] = c.z;
}

// The albedo of a hit pixel with the surrogate in place of the procedural substrate of
// brick and stone when `useNet` (Stratum.cu:854); otherwise exactly the drop-in's.
SD f3 neuralAlbedo(const float* __restrict__ W, const SurfacePoint& sp, bool useNet) {
  f3 base = substrateMean(sp.mat);
  if (sp.mat == 0 || sp.mat == 1)
    base = useNet ? predictSubstrate(W, sp.u, sp.v, sp.seed, sp.mat) : substrate(sp.u, sp.v, sp.seed, sp.mat);
  return surfaceColor(sp.q, sp.qn, sp.mat, sp.seed, sp.sfp, base) * paletteTint(sp.palette, sp.mat);
}
// The material half of shadePixels with the surrogate, when C[16] enables it and the
// gate Brain[4] is open.  The lighting half follows as its own kernel (shade.cu).
__global__ void __launch_bounds__(kShadeThreads, 1024 / kShadeThreads)
    albedoNeuralK(const float* __restrict__ World, const uint32_t* __restrict__ O, const float* __restrict__ C,
                  const float4* __restrict__ Hit, const float4* __restrict__ Surface, float4* Linear,
                  const float* __restrict__ W, const float* __restrict__ Brain, int width, int height, int rowStart,
                  int rowEnd) {
  __shared__ FrameConst F;
  frameInit(F, C, O);
  const bool useNet = C[16] > 0.5f && Brain[4] > 0.5f;
  const int tilesX = (width + 7) / 8, tiles = tilesX * ((rowEnd - rowStart + 3) / 4), warps = kShadeThreads / 32;
#pragma unroll 1
  for (int i = int(blockIdx.x) * warps + int(threadIdx.x >> 5); i < tiles; i += int(gridDim.x) * warps) {
    int x, y;
    if (!stripPixel(i, tilesX, width, rowStart, rowEnd, x, y)) continue;
    const size_t b = size_t(y) * width + x;
    const f3 rd = primaryDir(F.cam, x, y, width, height);
    const float4 h = Hit[b];
    f3 c;
    if (int(h.y) == kSkyId) {
      c = skyColor(rd, F.sun);
    } else {
      SurfacePoint sp;
      surfacePoint(World, F, h, Surface[b], rd, height, sp);
      c = neuralAlbedo(W, sp, useNet);
    }
    Linear[b] = make_float4(c.x, c.y, c.z, 1.0f);
  }
}
// Both halves at once, for strips of at most one wave (strips.cuh).
__global__ void __launch_bounds__(kShadeThreads, 1024 / kShadeThreads)
    shadePixelsNeuralK(const float* __restrict__ World, const uint32_t* __restrict__ O, const float* __restrict__ C,
                       const float4* __restrict__ Hit, const float4* __restrict__ Surface, float4* Linear,
                       const float* __restrict__ W, const float* __restrict__ Brain, int width, int height, int rowStart,
                       int rowEnd) {
  __shared__ FrameConst F;
  frameInit(F, C, O);
  int x, y;
  if (!stripPixel(int(blockIdx.x) * (kShadeThreads / 32) + int(threadIdx.x >> 5), (width + 7) / 8, width, rowStart, rowEnd,
                  x, y))
    return;
  const size_t b = size_t(y) * width + x;
  const f3 rd = primaryDir(F.cam, x, y, width, height);
  const float4 h = Hit[b];
  f3 c;
  if (int(h.y) == kSkyId) {
    c = skyColor(rd, F.sun);
  } else {
    SurfacePoint sp;
    surfacePoint(World, F, h, Surface[b], rd, height, sp);
    c = pixelLight(World, F, sp, rd, int(h.y), neuralAlbedo(W, sp, C[16] > 0.5f && Brain[4] > 0.5f));
  }
  Linear[b] = make_float4(c.x, c.y, c.z, 1.0f);
}

// The lighting half of shadePixels (shade.cu).
int lightRows(const float* World, const unsigned* Origin, const float* C, const float* Hit, const float* Surface,
              float* Linear, int width, int height, int rowStart, int rows, cudaStream_t stream);

}  // namespace st

using namespace st;

extern "C" {

int stratum_initNeural(float* W, float* M, float* V, float* Brain, int seed, stratum_stream_t stream) {
  if (!W || !M || !V || !Brain) return STRATUM_EINVAL;
  initNeuralK<<<2, 256, 0, asStream(stream)>>>(W, M, V, Brain, seed);
  return launchStatus();
}

int stratum_materialStep(const float* World, const unsigned* Origin, const float* C, const float* Hit,
                         const float* Surface, float* W, float* M, float* V, float* Brain, float* Work, int width,
                         int height, stratum_stream_t stream) {
  if (!World || !Origin || !C || !Hit || !Surface || !W || !M || !V || !Brain || !frameOk(width, height))
    return STRATUM_EINVAL;
  materialStepK<<<1, kStepThreads, 0, asStream(stream)>>>(World, Origin, C, Hit, Surface, W, M, V, Brain, Work,
                                                          width, height);
  return launchStatus();
}

int stratum_predictSubstrate(const float* W, const float* Queries, int n, float* Out, stratum_stream_t stream) {
  if (!W || !Queries || !Out || n < 0) return STRATUM_EINVAL;
  if (n == 0) return STRATUM_OK;
  predictSubstrateK<<<(n + 127) / 128, 128, 0, asStream(stream)>>>(W, Queries, n, Out);
  return launchStatus();
}

int stratum_shadePixelsNeural(const float* World, const unsigned* Origin, const float* C, const float* Hit,
                              const float* Surface, float* Linear, const float* W, const float* Brain, int width,
                              int height, int rowStart, int rowCount, stratum_stream_t stream) {
  if (!World || !Origin || !C || !Hit || !Surface || !Linear || !W || !Brain || !frameOk(width, height))
    return STRATUM_EINVAL;
  if (rowStart < 0 || rowCount < 0) return STRATUM_EINVAL;
  const int rows = rowCount < height - rowStart ? rowCount : height - rowStart;
  if (rows <= 0) return STRATUM_OK;
  const int wave = shadeWave();
  if (!wave) return STRATUM_EINVAL;
  if (tileBlocks(width, rows) <= wave) {
    shadePixelsNeuralK<<<tileBlocks(width, rows), kShadeThreads, 0, asStream(stream)>>>(
        World, Origin, C, reinterpret_cast<const float4*>(Hit), reinterpret_cast<const float4*>(Surface),
        reinterpret_cast<float4*>(Linear), W, Brain, width, height, rowStart, rowStart + rows);
    return launchStatus();
  }
  albedoNeuralK<<<tileBlocks(width, rows, wave), kShadeThreads, 0, asStream(stream)>>>(
      World, Origin, C, reinterpret_cast<const float4*>(Hit), reinterpret_cast<const float4*>(Surface),
      reinterpret_cast<float4*>(Linear), W, Brain, width, height, rowStart, rowStart + rows);
  const int s = launchStatus();
  return s != STRATUM_OK ? s
                         : lightRows(World, Origin, C, Hit, Surface, Linear, width, height, rowStart, rows, asStream(stream));
}

}  // extern "C"
