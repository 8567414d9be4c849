// Test infrastructure: the render server on the HOST, over stand-ins for the CUDA runtime
// and the batched renderer (memory is host memory, work is done at once), with thread
// creation that can be made to fail.
//
// A frame is filled with its pose's yaw and the number of samples since the pose was set.
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../include/stratum.h"

static std::atomic<int> threadsLeft{1 << 30}, allocations{0};

extern "C" {
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static const Create real = reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"));
  return threadsLeft-- > 0 ? real(t, a, f, arg) : EAGAIN;
}
static cudaError_t take(void** p, size_t n) { allocations++; return (*p = calloc(n ? n : 1, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
static cudaError_t give(void* p) { if (p) allocations--; free(p); return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeHost(void* p) { return give(p); }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(to, from, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return take(reinterpret_cast<void**>(s), 1); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return give(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return take(reinterpret_cast<void**>(e), 1); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return give(e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }

unsigned long long stratum_batchScratchBytes(int) { return 256; }
unsigned long long stratum_groupCacheBytes(int) { return 256; }
int stratum_groupCacheInit(unsigned*, int, stratum_stream_t) { return STRATUM_OK; }
int stratum_initCamera(float* C, unsigned*, int, stratum_stream_t) { C[19] = 0.0f; return STRATUM_OK; }
int stratum_applyPoses(stratum_view* v, const stratum_pose* p, const int* flags, int n, stratum_stream_t) {
  for (int i = 0; i < n; i++) {
    if (flags[i] & 1) v[i].C[3] = p[i].yaw;
    if (flags[i] & 2) v[i].C[19] = 0.0f;
  }
  return STRATUM_OK;
}
int stratum_stepViews(stratum_view* v, int n, stratum_stream_t) {
  for (int i = 0; i < n; i++) v[i].C[19] += 1.0f;
  return STRATUM_OK;
}
int stratum_refreshViews(stratum_view*, int, stratum_stream_t) { return STRATUM_OK; }
int stratum_buildViews(stratum_view*, int, stratum_stream_t) { return STRATUM_OK; }
int stratum_renderViews(stratum_view* v, int n, void*, unsigned long long, const stratum_tune*, stratum_stream_t) {
  for (int i = 0; i < n; i++)
    for (int k = 0; k < v[i].width * v[i].height; k++) v[i].Pixels[k] = unsigned(v[i].C[3]) * 256u + unsigned(v[i].C[19]);
  return STRATUM_OK;
}
}

#define EXPECT(x) \
  if (!(x)) { printf("%s:%d: %s\n", __FILE__, __LINE__, #x); return 1; }

// Thread number `k` cannot be started: no server, nothing left behind; then one that works.
static int noThread(int k) {
  const int before = allocations;
  threadsLeft = k;
  stratum_server* S = stratum_server_create(1ull << 30, 4, 2, nullptr);
  threadsLeft = 1 << 30;
  if (k >= 5) {
    EXPECT(S);
    stratum_server_destroy(S);
  } else {
    EXPECT(!S);
  }
  EXPECT(allocations == before);
  return 0;
}

// Requests queued behind one another on every session get each its own frame.
static int ownFrames(int w, int h) {
  stratum_server* S = stratum_server_create(4ull << 30, 3, 2, nullptr);
  EXPECT(S);
  const int sessions = 4, deep = 5;
  int id[sessions];
  std::vector<std::vector<unsigned>> out(sessions * deep, std::vector<unsigned>(size_t(w) * h, 7u));
  std::vector<long long> req(sessions * deep);
  for (int s = 0; s < sessions; s++) EXPECT(stratum_server_open(S, s, w, h, &id[s]) == STRATUM_OK);
  for (int d = 0; d < deep; d++)
    for (int s = 0; s < sessions; s++) {
      stratum_pose p{};
      p.yaw = float(1 + s + 10 * d);
      unsigned char* to = (d + s) % 4 == 3 ? nullptr : reinterpret_cast<unsigned char*>(out[s * deep + d].data());
      EXPECT(stratum_server_submit(S, id[s], &p, 1 + d % 3, to, &req[s * deep + d]) == STRATUM_OK);
    }
  for (int s = 0; s < sessions; s++)
    for (int d = 0; d < deep; d++) {
      EXPECT(stratum_server_wait(S, req[s * deep + d], 60000, nullptr) == STRATUM_OK);
      const unsigned want = (d + s) % 4 == 3 ? 7u : unsigned(1 + s + 10 * d) * 256u + unsigned(1 + d % 3);
      for (unsigned v : out[s * deep + d]) EXPECT(v == want);
    }
  for (int s = 0; s < sessions; s++) EXPECT(stratum_server_close(S, id[s]) == STRATUM_OK);
  stratum_server_destroy(S);
  return 0;
}

int main(int argc, char** argv) {
  const int a = argc > 2 ? atoi(argv[2]) : 0, b = argc > 3 ? atoi(argv[3]) : 0;
  if (argc > 1 && !strcmp(argv[1], "threads")) return noThread(a);
  if (argc > 1 && !strcmp(argv[1], "frames")) return ownFrames(a, b);
  return 2;
}
