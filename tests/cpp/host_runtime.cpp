// host_runtime.cpp — the CUDA runtime calls that the library makes, without a
// GPU: device memory is host memory, kernels do not run, and every launch is
// written down with its arguments.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "host_only.h"

namespace {
std::mutex mu;
std::vector<HostLaunch> launches;
std::map<const void*, uint64_t> limits;

void record(const void* fn, size_t smem, const cudaLaunchAttribute* attr, int attrs,
            void** args) {
  std::lock_guard<std::mutex> lock(mu);
  HostLaunch l{};
  l.fn = fn;
  l.cluster = 1;
  l.smem = smem;
  auto limit = limits.find(fn);
  l.limit = limit == limits.end() ? 48 << 10 : limit->second;
  for (int k = 0; k < attrs; k++) {
    if (attr[k].id == cudaLaunchAttributeClusterDimension) l.cluster = attr[k].val.clusterDim.x;
    if (attr[k].id == cudaLaunchAttributeCooperative) l.cooperative = attr[k].val.cooperative;
    if (attr[k].id == cudaLaunchAttributeProgrammaticStreamSerialization)
      l.pdl = attr[k].val.programmaticStreamSerializationAllowed;
  }
  host_describe(fn, args, &l);
  launches.push_back(l);
}
}  // namespace

extern "C" {

HostState host_state;

int32_t host_launches(HostLaunch* out, int32_t cap) {
  std::lock_guard<std::mutex> lock(mu);
  int32_t n = 0;
  for (const HostLaunch& l : launches)
    if (n < cap) out[n++] = l;
  launches.clear();
  return n;
}

// ---------------------------------------------------------------------------
// The runtime.
// ---------------------------------------------------------------------------
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*,
                            dim3*, int*) {}
cudaError_t __cudaGetKernel(cudaKernel_t* kernel, const void* fn) {
  *kernel = (cudaKernel_t)fn;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = *block = dim3(1);
  *smem = 0;
  *static_cast<void**>(stream) = nullptr;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3, dim3, void** args, size_t smem,
                               cudaStream_t) {
  record((const void*)kernel, smem, nullptr, 0, args);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void** args) {
  record(fn, c->dynamicSmemBytes, c->attrs, c->numAttrs, args);
  return c->dynamicSmemBytes > launches.back().limit ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute attr, int value) {
  std::lock_guard<std::mutex> lock(mu);
  if (host_state.fail_attribute > 0) {
    host_state.fail_attribute--;
    return cudaErrorUnknown;
  }
  if (attr != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
  auto it = limits.find(fn);
  if (it != limits.end() && (uint64_t)value < it->second) host_state.limits_lowered++;
  limits[fn] = value;
  return cudaSuccess;
}
// How many clusters of a size a GB300 holds with a CTA to an SM, and with more.
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* fn, const cudaLaunchConfig_t* c) {
  std::lock_guard<std::mutex> lock(mu);
  auto it = limits.find(fn);
  if (c->dynamicSmemBytes > (it == limits.end() ? 48 << 10 : it->second))
    return cudaErrorInvalidValue;
  static const std::map<int, int> alone = {{2, 76}, {4, 36}, {6, 23}, {8, 15}, {10, 13}, {12, 8}, {16, 7}};
  const int cluster = c->attrs[0].val.clusterDim.x;
  const int share = (int)((228 << 10) / (c->dynamicSmemBytes + 1024));
  auto a = alone.find(cluster);
  *n = a == alone.end() ? 0 : a->second * (share < 1 ? 1 : share);
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes) {
  *p = nullptr;
  if (host_state.fail_malloc_from > 0 && bytes >= (size_t)host_state.fail_malloc_from)
    return cudaErrorMemoryAllocation;
  *p = calloc(1, bytes);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
  *p = calloc(1, bytes);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int x, size_t n) {
  memset(d, x, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int x, size_t n, cudaStream_t) {
  memset(d, x, n);
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr attr, int) {
  *value = attr == cudaDevAttrMultiProcessorCount ? 152 : 0;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "success" : "refused"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) {
  return cudaErrorUnknown;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorUnknown; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = nullptr;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)1;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) {
  *g = (cudaGraphExec_t)1;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}

}  // extern "C"
