// A CUDA runtime on host memory, for tests of the library's host code on a
// machine without a GPU: allocations and copies are real (host pages), kernel
// launches are recorded and not run.  It answers with errors where the real
// runtime would: an allocation that the test refuses, a launch whose dynamic
// shared memory is above the kernel's limit.  As in the real runtime, an error
// stays pending until cudaGetLastError reads it, and successful calls leave it.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {

struct Launch {
  std::string name;
  dim3 grid, block;
  size_t smem;
  bool captured;
};

std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> m;
  return m;
}
std::map<const void*, size_t> g_smem_limit;
std::map<void*, size_t> g_live;
std::map<size_t, void*> g_pinned;  // the last page-locked block of each size
std::vector<Launch> g_launches;
size_t g_bytes = 0, g_peak = 0;
int g_mallocs = 0, g_refuse = 0, g_refusals = 0;
size_t g_at_refusal = 0;  // launches before the refused allocation
bool g_capturing = false;
int g_captured = 0;
std::string g_fail_launch;
cudaError_t g_last = cudaSuccess;

cudaError_t ret(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
constexpr size_t kSmemDefault = 48 * 1024, kSmemMost = 227 * 1024;

cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t smem) {
  const auto it = names().find(f);
  const std::string name = it == names().end() ? "?" : it->second;
  const auto lim = g_smem_limit.find(f);
  const size_t most = lim == g_smem_limit.end() ? kSmemDefault : lim->second;
  if (smem > most || grid.x == 0 || grid.y == 0 || grid.z == 0 || grid.x > 0x7fffffffu || grid.y > 65535u ||
      grid.z > 65535u || block.x * block.y * block.z > 1024u || block.x == 0)
    return ret(cudaErrorInvalidValue);
  if (!g_fail_launch.empty() && name.find(g_fail_launch) != std::string::npos) return ret(cudaErrorLaunchOutOfResources);
  g_launches.push_back({name, grid, block, smem, g_capturing});
  if (g_capturing) ++g_captured;
  return cudaSuccess;
}

struct Graph {
  int kernels = 0;
};

// null, or an offset from null
bool bad(const void* p) { return (uintptr_t)p < (1u << 20); }

}  // namespace

extern "C" {

// ------------------------------------------------------------- for the tests
void host_cudart_reset() {
  g_launches.clear();
  g_mallocs = g_refuse = g_refusals = 0;
  g_at_refusal = 0;
  g_peak = g_bytes;
  g_fail_launch.clear();
  g_last = cudaSuccess;
}
void host_cudart_refuse(int nth) { g_refuse = nth; }  // the nth cudaMalloc from the reset on fails; 0: none
void host_cudart_fail_launch(const char* part) { g_fail_launch = part; }
void* host_cudart_pinned(long long size) {
  const auto it = g_pinned.find((size_t)size);
  return it == g_pinned.end() ? nullptr : it->second;
}
int host_cudart_blocks(long long size, void** out, int most) {  // live device arrays of this size
  int n = 0;
  for (const auto& b : g_live)
    if (b.second == (size_t)size && n < most) out[n++] = b.first;
  return n;
}
int host_cudart_mallocs() { return g_mallocs; }
int host_cudart_refusals() { return g_refusals; }
long long host_cudart_bytes() { return (long long)g_bytes; }
long long host_cudart_peak() { return (long long)g_peak; }
int host_cudart_pending() { return (int)g_last; }
int host_cudart_launches_after_refusal() { return g_refusals ? (int)(g_launches.size() - g_at_refusal) : 0; }
int host_cudart_launches(const char* part, long long* most_smem) {
  int n = 0;
  long long most = 0;
  for (const Launch& l : g_launches)
    if (l.name.find(part) != std::string::npos) {
      ++n;
      if ((long long)l.smem > most) most = (long long)l.smem;
    }
  if (most_smem) *most_smem = most;
  return n;
}

// ------------------------------------------------------------- registration
void** __cudaRegisterFatBinary(void*) {
  static void* h = nullptr;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names()[(const void*)host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

// ------------------------------------------------------------- launches
static dim3 g_grid, g_block;
static size_t g_smem;
static cudaStream_t g_stream;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* st) {
  g_grid = grid;
  g_block = block;
  g_smem = smem;
  g_stream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
  *grid = g_grid;
  *block = g_block;
  *smem = g_smem;
  *(cudaStream_t*)st = g_stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
  return launch((const void*)k, grid, block, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (v < 0 || (size_t)v > kSmemMost) return ret(cudaErrorInvalidValue);
    g_smem_limit[f] = (size_t)v;
  }
  return cudaSuccess;
}

// ------------------------------------------------------------- errors, device
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return g_last; }
const char* cudaGetErrorString(cudaError_t) { return "error of the host runtime"; }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
  return cudaSuccess;
}
static int encode_tiled() { return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *p = (void*)encode_tiled;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static void* a = calloc(1, 4 << 20);
  *p = a;
  return cudaSuccess;
}

// ------------------------------------------------------------- memory
cudaError_t cudaMalloc(void** p, size_t n) {
  ++g_mallocs;
  if (g_refuse && g_mallocs == g_refuse) {
    ++g_refusals;
    g_at_refusal = g_launches.size();
    return ret(cudaErrorMemoryAllocation);
  }
  void* m = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (m == MAP_FAILED) return ret(cudaErrorMemoryAllocation);
  *p = m;
  g_live[m] = n;
  g_bytes += n;
  if (g_bytes > g_peak) g_peak = g_bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  const auto it = g_live.find(p);
  if (it == g_live.end()) return p ? ret(cudaErrorInvalidValue) : cudaSuccess;
  munmap(p, it->second);
  g_bytes -= it->second;
  g_live.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  *p = calloc(1, n ? n : 1);
  g_pinned[n] = *p;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  if (bad(p)) return ret(cudaErrorInvalidValue);
  const auto it = g_live.find(p);
  if (v == 0 && it != g_live.end() && n == it->second) madvise(p, n, MADV_DONTNEED);
  else memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return g_capturing ? cudaSuccess : cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  if (bad(d) || bad(s)) return ret(cudaErrorInvalidValue);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  if (bad(d) || bad(s)) return ret(cudaErrorInvalidValue);
  return g_capturing ? cudaSuccess : cudaMemcpy(d, s, n, k);
}

// ------------------------------------------------------------- streams, events
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)malloc(8);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free((void*)s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)malloc(8);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free((void*)e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}

// ------------------------------------------------------------- graphs
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  g_capturing = true;
  g_captured = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*,
                                          size_t, cudaStreamCaptureMode) {
  return ret(cudaErrorNotSupported);
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  g_capturing = false;
  Graph* x = new Graph;
  x->kernels = g_captured;
  *g = (cudaGraph_t)x;
  return cudaSuccess;
}
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) {
  *g = (cudaGraph_t) new Graph;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete (Graph*)g;
  return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t* n, size_t* count) {
  if (!n) *count = (size_t)((Graph*)g)->kernels;
  return cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType* t) {
  *t = cudaGraphNodeTypeKernel;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t) new Graph;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete (Graph*)e;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphAddMemcpyNode1D(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, size_t, void*, const void*,
                                     size_t, cudaMemcpyKind) {
  return ret(cudaErrorNotSupported);
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                             cudaGraphNodeParams*) {
  return ret(cudaErrorNotSupported);
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle*, cudaGraph_t, unsigned, unsigned) {
  return ret(cudaErrorNotSupported);
}

}  // extern "C"
