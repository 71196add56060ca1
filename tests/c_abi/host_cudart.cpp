// host_cudart.cpp -- a stand-in for the CUDA runtime in host tests of the
// library's planning and launch code, linked in place of libcudart: device
// memory is host memory (filled with a pattern, as a device's is with what was
// there before), copies are done at once, kernels are not run.  Every call that
// a test may look at is written to a trace, a line each.
//
// An event counts the blocks launched before it, and the time between two
// events is those in between: a launch of fewer blocks is the faster one.  A
// graph holds the launches captured into it and repeats them once a launch,
// whatever its conditions.
#include <cuda_runtime_api.h>

#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <string>
#include <vector>

// The library's own host allocations of more than `largest` bytes fail.
static long long largest = LLONG_MAX;
void *operator new(size_t n) {
  void *p = (long long)n > largest ? nullptr : std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

struct CUgraph_st {
  std::vector<std::string> lines;  // captured launches
  CUgraph_st *body = nullptr;      // of its conditional node
};

namespace {

std::string trace;
std::map<void *, size_t> blocks;  // allocations
size_t held = 0;
int device = 0, streams = 0;
long long launched = 0, failing = -1;
CUgraph_st *capturing = nullptr;

struct Config {
  dim3 grid, block;
  size_t smem;
  void *stream;
} config;

// (kernels register themselves while the library is loaded, perhaps before this
// file's own objects exist)
std::map<const void *, std::string> &kernels() {
  static std::map<const void *, std::string> m;
  return m;
}

void say(const std::string &s) { trace += s + "\n"; }

std::string name(const void *f) {
  auto it = kernels().find(f);
  return it == kernels().end() ? "?" : it->second;
}

// Created streams are numbered from 1; 0 is the legacy stream.
std::string stream(const void *s) { return std::to_string((long long)(size_t)s); }

cudaError_t take(void **p, size_t n) {
  *p = std::malloc(n ? n : 1);
  if (!*p) return cudaErrorMemoryAllocation;
  std::memset(*p, 0xa5, n);
  blocks[*p] = n;
  held += n;
  return cudaSuccess;
}

cudaError_t give(void *p) {
  auto it = blocks.find(p);
  if (it == blocks.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
  held -= it->second;
  blocks.erase(it);
  std::free(p);
  return cudaSuccess;
}

}  // namespace

extern "C" {

// for the tests
const char *host_trace() { return trace.c_str(); }
void host_trace_clear() { trace.clear(); }
void host_set_device(int d) { device = d; }
long long host_bytes() { return (long long)held; }
void host_largest(long long bytes) { largest = bytes; }
// the next copy of that many bytes fails
void host_fail_copy(long long bytes) { failing = bytes; }

cudaError_t cudaGetDevice(int *d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "host runtime"; }

cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) {
  *p = std::malloc(n ? n : 1);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return give(p); }
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  say("memcpy " + stream(st) + " " + std::to_string(n));
  if ((long long)n == failing) {
    failing = -1;
    return cudaErrorInvalidValue;
  }
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  return cudaMemcpyAsync(d, s, n, k, nullptr);
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  say("memset " + stream(st) + " " + std::to_string(n));
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorInvalidSymbol; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)(size_t)++streams;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  say("synchronize " + stream(s));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t)std::calloc(1, sizeof(long long));
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  *(long long *)e = launched;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(*(long long *)b - *(long long *)a);
  return cudaSuccess;
}

cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize)
    say("optin " + std::to_string(device) + " " + name(f) + " " + std::to_string(v));
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}

cudaError_t cudaGraphCreate(cudaGraph_t *g, unsigned) {
  *g = new CUgraph_st;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete g->body;
  delete g;
  return cudaSuccess;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *h, cudaGraph_t, unsigned, unsigned) {
  *h = 1;
  return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t *, cudaGraph_t g, const cudaGraphNode_t *, const cudaGraphEdgeData *,
                             size_t, cudaGraphNodeParams *p) {
  g->body = new CUgraph_st;
  p->conditional.phGraph_out = &g->body;
  return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t *nodes, size_t *n) {
  if (!nodes) *n = g->lines.size();
  return cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType *t) {
  *t = cudaGraphNodeTypeKernel;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t g, unsigned long long) {
  *e = (cudaGraphExec_t)g;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  for (const std::string &l : ((cudaGraph_t)e)->body->lines) say(l);
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t g, const cudaGraphNode_t *,
                                          const cudaGraphEdgeData *, size_t, cudaStreamCaptureMode) {
  say("capture");
  capturing = g;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = capturing;
  capturing = nullptr;
  return cudaSuccess;
}

// what nvcc's host code calls for a launch and at load time
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *s) {
  config = {grid, block, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *(void **)s = config.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3, void **, size_t smem, cudaStream_t s) {
  const std::string line = "launch " + stream(s) + " " + name((const void *)k) + " " + std::to_string(grid.x) +
                           " " + std::to_string(smem);
  if (capturing) {
    capturing->lines.push_back(line);
  } else {
    launched += (long long)grid.x * grid.y * grid.z;
    say(line);
  }
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
  static void *handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *n, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  kernels()[f] = n;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}

}  // extern "C"
