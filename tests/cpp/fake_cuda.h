// A CUDA runtime of host memory for tests of the solvers' host code: device
// buffers are host allocations kept in a table, kernels are the test's own
// launchers, stream capture counts.  As CUDA does, a failed call leaves its
// code for the next cudaGetLastError.
#pragma once

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

#include <cuda_runtime.h>

static std::map<const char*, size_t> g_live;
[[maybe_unused]] static bool g_capturing = false;
[[maybe_unused]] static int g_captures = 0, g_replays = 0;
[[maybe_unused]] static bool g_fail_pin = false;  // no MB of host memory can be pinned
static int g_fail_in = 0;  // 1: the next device allocation fails
static cudaError_t g_last = cudaSuccess;

static void need(const void* p, size_t bytes, const char* what) {
  const char* c = static_cast<const char*>(p);
  auto it = g_live.upper_bound(c);
  if (it != g_live.begin()) {
    --it;
    if (c >= it->first && c + bytes <= it->first + it->second) return;
  }
  std::printf("%s: %zu bytes at %p are not in a device buffer\n", what, bytes, p);
  std::exit(1);
}
static cudaError_t last() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}

// ------------------------------------------------------------ runtime
extern "C" {
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) {
  if (g_fail_in > 0 && --g_fail_in == 0) return g_last = cudaErrorMemoryAllocation;
  *p = std::calloc(n, 1);
  g_live[static_cast<char*>(*p)] = n;
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  g_live.erase(static_cast<char*>(p));
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (g_fail_pin && n >= size_t(1) << 20) return g_last = cudaErrorMemoryAllocation;
  *p = std::calloc(n, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  if (k == cudaMemcpyDeviceToHost) need(s, n, "copy to the host");
  if (k == cudaMemcpyHostToDevice) need(d, n, "copy to the device");
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  need(d, n, "memset");
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return last(); }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  g_capturing = true;
  g_captures++;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  g_capturing = false;
  *g = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(&g_captures);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  g_replays++;
  return cudaSuccess;
}
}

