// A CUDA runtime on the host for tests of the library's host code: device
// memory is host memory (filled with a byte pattern), kernels are recorded and
// not run, and allocations can be made to fail.  Linked with the library's
// object files in place of libcudart.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <vector>

#include "gemm.cuh"
#include "common.cuh"

namespace host {
struct Launch {
  const void *func;
  cudaStream_t stream;
  dim3 grid;
  bool overlapped;   // may be set up while the kernel before it runs
  bool cluster;      // CTA pairs
};
inline std::vector<Launch> launches;
inline std::map<void *, size_t> blocks;          // live device blocks
inline size_t live = 0, budget = ~size_t(0);     // bytes in use and at most
inline std::map<cudaStream_t, int> pending;      // launches since the stream was waited for
inline std::function<void()> on_launch = [] {};
inline cudaError_t last = cudaSuccess;

inline void launch(const void *f, cudaStream_t s, dim3 grid, bool overlapped,
                   bool cluster = false) {
  launches.push_back({f, s, grid, overlapped, cluster});
  ++pending[s];
  on_launch();
}
inline cudaError_t fail(cudaError_t e) { return last = e; }
}  // namespace host

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
  if (host::live + n > host::budget) return host::fail(cudaErrorMemoryAllocation);
  *p = std::aligned_alloc(512, (n + 511) / 512 * 512);
  if (!*p) return host::fail(cudaErrorMemoryAllocation);
  std::memset(*p, 0xA5, n);
  host::blocks[*p] = n;
  host::live += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  auto it = host::blocks.find(p);
  if (it == host::blocks.end()) return host::fail(cudaErrorInvalidValue);
  host::live -= it->second;
  host::blocks.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *t = size_t(180) << 30;
  *f = *t - host::live;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { host::pending.clear(); return cudaSuccess; }
cudaError_t cudaGetLastError() {
  cudaError_t e = host::last;
  host::last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "host runtime error"; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) {
  return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void *d, const void *, size_t n, size_t, cudaMemcpyKind) {
  std::memset(d, 0, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
  static char *scratch = (char *)std::calloc(1, (size_t(1) << 23) + 512);
  *p = scratch;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t) new int(0);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { host::pending[s] = 0; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) {
  *c = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  return cudaErrorNotSupported;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) {
  return cudaErrorNotSupported;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t) new int(0); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int,
                                                                   size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
  *n = 74;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **, size_t, cudaStream_t s) {
  host::launch(f, s, grid, false);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  bool over = false, cluster = false;
  for (unsigned i = 0; i < c->numAttrs; ++i) {
    over = over || (c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization &&
                    c->attrs[i].val.programmaticStreamSerializationAllowed);
    cluster = cluster || c->attrs[i].id == cudaLaunchAttributeClusterDimension;
  }
  host::launch(f, c->stream, c->gridDim, over, cluster);
  return cudaSuccess;
}
static CUresult host_encode(CUtensorMap *, ...) { return CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **p, unsigned long long,
                                    cudaDriverEntryPointQueryResult *q) {
  *p = (void *)host_encode;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
}

#define CHECK(cond)                                                   \
  do {                                                                \
    if (!(cond)) {                                                    \
      std::printf("line %d: %s\n", __LINE__, #cond);                  \
      return 1;                                                       \
    }                                                                 \
  } while (0)
