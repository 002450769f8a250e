// The CUDA runtime calls that the library's host code makes, without a GPU: device memory is host memory
// (zeroed), launches do nothing, and every call is written to a log. `limit` bounds the memory that
// can be held, blocks that a pool keeps included.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace fake {
std::vector<std::string> log;
size_t limit = ~size_t(0), held = 0, idle = 0, peak = 0;   // idle: of held, kept by the pool
std::map<void*, size_t> blocks;
int launches = 0;

cudaError_t take(void** p, size_t n, bool pool) {
  *p = nullptr;
  const size_t reuse = pool && idle < n ? idle : (pool ? n : 0);
  if (held - reuse + n > limit) return cudaErrorMemoryAllocation;
  if (pool) idle -= reuse;
  held += n - reuse;
  if (held > peak) peak = held;
  *p = std::calloc(n ? n : 1, 1);
  blocks[*p] = n;
  return cudaSuccess;
}
void give(void* p, bool pool) {
  if (!p) return;
  const size_t n = blocks.at(p);
  blocks.erase(p);
  if (pool) idle += n; else held -= n;
  std::free(p);
}
}  // namespace fake

#define FAKE(name, ...) extern "C" cudaError_t name(__VA_ARGS__)
FAKE(cudaMalloc, void** p, size_t n) { fake::log.push_back("cudaMalloc"); return fake::take(p, n, false); }
FAKE(cudaFree, void* p) { fake::log.push_back("cudaFree"); fake::give(p, false); return cudaSuccess; }
FAKE(cudaMallocFromPoolAsync, void** p, size_t n, cudaMemPool_t, cudaStream_t) { fake::log.push_back("cudaMallocFromPoolAsync"); return fake::take(p, n, true); }
FAKE(cudaFreeAsync, void* p, cudaStream_t) { fake::log.push_back("cudaFreeAsync"); fake::give(p, true); return cudaSuccess; }
FAKE(cudaMemPoolTrimTo, cudaMemPool_t, size_t) { fake::log.push_back("cudaMemPoolTrimTo"); fake::held -= fake::idle; fake::idle = 0; return cudaSuccess; }
FAKE(cudaMemPoolCreate, cudaMemPool_t* p, const cudaMemPoolProps*) { *p = reinterpret_cast<cudaMemPool_t>(16); return cudaSuccess; }
FAKE(cudaMemPoolDestroy, cudaMemPool_t) { fake::held -= fake::idle; fake::idle = 0; return cudaSuccess; }
FAKE(cudaMemPoolSetAttribute, cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
FAKE(cudaMemcpy, void* d, const void* s, size_t n, cudaMemcpyKind) { fake::log.push_back("cudaMemcpy"); std::memcpy(d, s, n); return cudaSuccess; }
FAKE(cudaMemcpyAsync, void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { fake::log.push_back("cudaMemcpyAsync"); std::memcpy(d, s, n); return cudaSuccess; }
FAKE(cudaMemsetAsync, void* d, int v, size_t n, cudaStream_t) { fake::log.push_back("cudaMemsetAsync"); std::memset(d, v, n); return cudaSuccess; }
FAKE(cudaStreamCreateWithFlags, cudaStream_t* s, unsigned) { static char* at = nullptr; at += 16; *s = reinterpret_cast<cudaStream_t>(at); return cudaSuccess; }
FAKE(cudaStreamDestroy, cudaStream_t) { return cudaSuccess; }
FAKE(cudaStreamSynchronize, cudaStream_t s) { fake::log.push_back("cudaStreamSynchronize " + std::to_string(reinterpret_cast<size_t>(s))); return cudaSuccess; }
FAKE(cudaStreamWaitEvent, cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
FAKE(cudaStreamBeginCapture, cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
FAKE(cudaStreamEndCapture, cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
FAKE(cudaDeviceSynchronize, void) { fake::log.push_back("cudaDeviceSynchronize"); return cudaSuccess; }
FAKE(cudaDeviceGetAttribute, int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
FAKE(cudaGetDevice, int* d) { *d = 0; return cudaSuccess; }
FAKE(cudaGetDeviceCount, int* n) { *n = 1; return cudaSuccess; }
FAKE(cudaSetDevice, int) { return cudaSuccess; }
FAKE(cudaGetLastError, void) { return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
FAKE(cudaEventCreate, cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
FAKE(cudaEventCreateWithFlags, cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
FAKE(cudaEventDestroy, cudaEvent_t) { return cudaSuccess; }
FAKE(cudaEventElapsedTime, float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }
FAKE(cudaEventRecord, cudaEvent_t, cudaStream_t) { return cudaSuccess; }
FAKE(cudaEventSynchronize, cudaEvent_t) { return cudaSuccess; }
FAKE(cudaFreeHost, void* p) { std::free(p); return cudaSuccess; }
FAKE(cudaFuncGetAttributes, cudaFuncAttributes* a, const void*) { std::memset(a, 0, sizeof(*a)); return cudaSuccess; }
FAKE(cudaFuncSetAttribute, const void*, cudaFuncAttribute, int) { return cudaSuccess; }
FAKE(cudaGetSymbolAddress, void** p, const void*) { *p = nullptr; return cudaErrorInvalidSymbol; }
FAKE(cudaGraphDestroy, cudaGraph_t) { return cudaSuccess; }
FAKE(cudaGraphExecDestroy, cudaGraphExec_t) { return cudaSuccess; }
FAKE(cudaGraphInstantiate, cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
FAKE(cudaGraphLaunch, cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
FAKE(cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags, int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
// What the compiler puts around a launch.
FAKE(__cudaGetKernel, cudaKernel_t* k, const void*) { *k = nullptr; return cudaSuccess; }
FAKE(__cudaLaunchKernel, cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { ++fake::launches; fake::log.push_back("launch"); return cudaSuccess; }
FAKE(__cudaPopCallConfiguration, dim3* g, dim3* b, size_t* s, void* t) { *g = dim3(); *b = dim3(); *s = 0; *static_cast<cudaStream_t*>(t) = nullptr; return cudaSuccess; }
extern "C" unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
extern "C" void** __cudaRegisterFatBinary(void*) { return nullptr; }
extern "C" void __cudaRegisterFatBinaryEnd(void**) {}
extern "C" void __cudaUnregisterFatBinary(void**) {}
extern "C" void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
extern "C" void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
