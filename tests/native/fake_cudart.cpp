// See fake_cudart.h.
#include "fake_cudart.h"

#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstring>
#include <map>

namespace fake {
int unordered, copies_in, copies_out, events, launches, graphs, fail_malloc, fail_copy_in, fail_memset;
size_t bytes, peak, limit;
static bool pending;                       // legacy-stream work that may still run
static cudaError_t last;                   // what cudaGetLastError gives
static std::map<char*, size_t> dev, host;  // allocations
static cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
static bool hit(int& n) { return n > 0 && --n == 0; }
static bool pinned(const void* p) {
  auto it = host.upper_bound((char*)p);
  if (it == host.begin()) return false;
  --it;
  return (char*)p < it->first + it->second;
}
static void queued(cudaStream_t s) {
  if (s && pending) unordered++;
}
static void* pages(size_t n) {
  void* p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  return p == MAP_FAILED ? nullptr : p;
}
template <class H>
static H handle() {
  static size_t next = 0x1000;
  return reinterpret_cast<H>(next += 16);
}
}  // namespace fake
using namespace fake;

extern "C" {
// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
  if (hit(fail_malloc) || (limit && bytes + n > limit)) return ret(cudaErrorMemoryAllocation);
  *p = pages(n);
  if (!*p) return ret(cudaErrorMemoryAllocation);
  dev[(char*)*p] = n;
  bytes += n;
  if (bytes > peak) peak = bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  auto it = dev.find((char*)p);
  if (it == dev.end()) return p ? ret(cudaErrorInvalidValue) : cudaSuccess;
  bytes -= it->second;
  munmap(p, it->second);
  dev.erase(it);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = pages(n);
  host[(char*)*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  auto it = host.find((char*)p);
  if (it != host.end()) {
    munmap(p, it->second);
    host.erase(it);
  }
  return cudaSuccess;
}
static cudaError_t copy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  if (k == cudaMemcpyHostToDevice) {
    if (hit(fail_copy_in)) return ret(cudaErrorInvalidValue);
    copies_in++;
  }
  if (k == cudaMemcpyDeviceToHost) copies_out++;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  const cudaError_t e = copy(d, s, n, k);
  if (k == cudaMemcpyHostToDevice && !pinned(s)) pending = true;
  else pending = false;  // waits for the legacy stream's earlier work too
  return e;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  queued(st);
  return copy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  if (hit(fail_memset)) return ret(cudaErrorInvalidValue);
  std::memset(d, v, n);
  pending = true;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  if (hit(fail_memset)) return ret(cudaErrorInvalidValue);
  queued(st);
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbolAsync(const void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t st) {
  queued(st);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static char mem[1 << 20];
  *p = mem;
  return cudaSuccess;
}
// ---- launches
static thread_local struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} call;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, CUstream_st* s) {
  call = {g, b, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = call.grid;
  *b = call.block;
  *smem = call.smem;
  *(cudaStream_t*)s = call.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t st) {
  queued(st);
  launches++;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  *a = cudaFuncAttributes{};
  a->maxThreadsPerBlock = 1024;
  a->ptxVersion = a->binaryVersion = 100;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
// ---- device, errors
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  switch (a) {
    case cudaDevAttrMultiProcessorCount: *v = 148; break;
    case cudaDevAttrComputeCapabilityMajor: *v = 10; break;
    case cudaDevAttrComputeCapabilityMinor: *v = 0; break;
    default: *v = 1024; break;
  }
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) {
  *lo = *hi = 0;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = handle<cudaStream_t>();
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (!s) pending = false;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = handle<cudaEvent_t>();
  events++;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) {
  events--;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0;
  return cudaSuccess;
}
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) {
  *g = handle<cudaGraph_t>();
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  *x = handle<cudaGraphExec_t>();
  graphs++;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) {
  queued(st);
  return cudaSuccess;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) {
  *h = 1;
  return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t* n, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraphNodeParams* p) {
  static cudaGraph_t body;
  *n = handle<cudaGraphNode_t>();
  body = handle<cudaGraph_t>();
  if (p->type == cudaGraphNodeTypeConditional) p->conditional.phGraph_out = &body;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*,
                                          size_t, cudaStreamCaptureMode) {
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = handle<cudaGraph_t>();
  return cudaSuccess;
}
}
