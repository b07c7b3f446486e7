// A stand-in for the CUDA runtime, linked with the library's own object files
// (tests/fakecuda/__init__.py): device memory is host memory, kernels do not
// run, and every call is counted, so that the host side's decisions (what is
// allocated, waited for, launched, on which device, in what grid) can be
// checked without a GPU.
//   Devices: FAKE_DEVICES equal ones; a function's attributes belong to the
// device current when they are set, and a launch with more dynamic shared
// memory than the attribute (48 KB unless raised) fails, as on real devices.
//   Order: a copying call from (pageable) host memory may return before the
// device has the data, and the library's streams do not wait for the legacy
// stream: a launch on one of them after such a call is counted as
// "fake_unordered".
//   Time: a launch advances the clock by 1 ms, or by what fake_set_cost says
// for its number of blocks.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <utility>
#include <vector>

namespace {
constexpr int FAKE_DEVICES = 2, SMS = 100000, BLOCKS_PER_SM = 2;

struct Event {
  double at = 0.0;
};
struct Op {  // a launch, or an event record
  Event* ev;
  double ms;
};
struct Graph {
  std::vector<Op> ops;
};
struct Stream {
  Graph* capture = nullptr;
};
struct Launch {
  std::string name;
  unsigned grid[3];
  int device;
};

int g_device = 0;
cudaError_t g_last = cudaSuccess;
double g_now = 0.0;
std::map<const void*, std::string> g_names;
std::map<std::pair<int, const void*>, int> g_smem;
std::map<long long, double> g_cost;
std::map<std::string, long long> g_calls;
std::vector<Launch> g_launches;
std::map<void*, size_t> g_sizes;
long long g_bytes = 0;
bool g_copying = false;  // a copy from the host on the legacy stream may be under way
std::string g_fail;
Stream g_legacy;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
Stream* str(cudaStream_t s) { return s ? reinterpret_cast<Stream*>(s) : &g_legacy; }
void enqueue(cudaStream_t s, Op op) {
  if (Graph* g = str(s)->capture) {
    g->ops.push_back(op);
  } else if (op.ev) {
    op.ev->at = g_now;
  } else {
    g_now += op.ms;
  }
}
cudaError_t launch(const void* f, dim3 grid, size_t smem, cudaStream_t s) {
  const std::string& name = g_names[f];
  if (!g_fail.empty() && name.find(g_fail) != std::string::npos) return done(cudaErrorInvalidConfiguration);
  const auto it = g_smem.find({g_device, f});
  if (smem > (size_t)(it == g_smem.end() ? 48 * 1024 : it->second)) return done(cudaErrorInvalidValue);
  if (s && g_copying) ++g_calls["fake_unordered"];
  g_launches.push_back(Launch{name, {grid.x, grid.y, grid.z}, g_device});
  const auto c = g_cost.find((long long)grid.x * grid.y * grid.z);
  enqueue(s, Op{nullptr, c == g_cost.end() ? 1.0 : c->second});
  return cudaSuccess;
}
cudaError_t alloc(void** p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  if (!*p) return done(cudaErrorMemoryAllocation);
  g_sizes[*p] = n;
  g_bytes += (long long)n;
  return cudaSuccess;
}
cudaError_t release(void* p) {
  if (!p) return cudaSuccess;
  g_bytes -= (long long)g_sizes[p];
  g_sizes.erase(p);
  std::free(p);
  return cudaSuccess;
}
CUresult encode_tiled(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}
dim3 g_grid, g_block;
size_t g_dyn;
cudaStream_t g_stream;
}  // namespace

#define CALL ++g_calls[__func__]

extern "C" {
// ---- the test's side --------------------------------------------------------
void fake_reset() {
  g_calls.clear();
  g_launches.clear();
  g_cost.clear();
  g_fail.clear();
  g_last = cudaSuccess;
  g_device = 0;
  g_copying = false;
}
long long fake_calls(const char* name) { return g_calls[name]; }
long long fake_bytes() { return g_bytes; }
int fake_launches() { return (int)g_launches.size(); }
const char* fake_launch(int i, unsigned* grid, int* device) {
  for (int q = 0; q < 3; ++q) grid[q] = g_launches[i].grid[q];
  *device = g_launches[i].device;
  return g_launches[i].name.c_str();
}
void fake_set_cost(long long blocks, double ms) { g_cost[blocks] = ms; }
void fake_fail(const char* name) { g_fail = name; }  // launches of kernels whose name holds it fail

// ---- the runtime's side -----------------------------------------------------
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) {
  g_grid = g;
  g_block = b;
  g_dyn = smem;
  g_stream = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = g_grid;
  *b = g_block;
  *smem = g_dyn;
  *static_cast<cudaStream_t*>(s) = g_stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void**, size_t smem, cudaStream_t s) {
  return launch((const void*)k, g, smem, s);
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3, void**, size_t smem, cudaStream_t s) {
  return launch(f, g, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= FAKE_DEVICES) return done(cudaErrorInvalidDevice);
  g_device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = g_device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int) {
  *v = SMS;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  std::strcpy(p->name, "fake");
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_smem[{g_device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = BLOCKS_PER_SM;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
  *n = BLOCKS_PER_SM;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { CALL; return alloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { CALL; return alloc(p, n); }
cudaError_t cudaFree(void* p) {
  if (p) CALL;
  return release(p);
}
cudaError_t cudaFreeHost(void* p) { CALL; return release(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
  CALL;
  g_copying = k == cudaMemcpyHostToDevice;  // (a copy to the host waits for those before it)
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind, cudaStream_t) {
  CALL;
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { CALL; std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { CALL; std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void*) {
  std::memset(a, 0, sizeof *a);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static double scratch[64];
  *p = scratch;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             enum cudaDriverEntryPointQueryResult* q) {
  *f = (void*)encode_tiled;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  CALL;
  g_copying = false;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  CALL;
  if (!s) g_copying = false;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(new Stream());
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete str(s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(new Event());
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  enqueue(s, Op{reinterpret_cast<Event*>(e), 0.0});
  return cudaSuccess;
}
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned) { return cudaEventRecord(e, s); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { CALL; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(reinterpret_cast<Event*>(b)->at - reinterpret_cast<Event*>(a)->at);
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode) {
  str(s)->capture = new Graph();
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t s, cudaGraph_t g, const cudaGraphNode_t*, const cudaGraphEdgeData*,
                                          size_t, enum cudaStreamCaptureMode) {
  str(s)->capture = reinterpret_cast<Graph*>(g);
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(str(s)->capture);
  str(s)->capture = nullptr;
  return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, enum cudaStreamCaptureStatus* st, unsigned long long* id,
                                     cudaGraph_t* g, const cudaGraphNode_t** deps, const cudaGraphEdgeData** edges,
                                     size_t* n) {
  *st = str(s)->capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  if (id) *id = 0;
  if (g) *g = reinterpret_cast<cudaGraph_t>(str(s)->capture);
  if (deps) *deps = nullptr;
  if (edges) *edges = nullptr;
  if (n) *n = 0;
  return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, const cudaGraphEdgeData*, size_t, unsigned) {
  return cudaSuccess;
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) {
  *h = 0;
  return cudaSuccess;
}
cudaError_t cudaGraphAddNode(cudaGraphNode_t* n, cudaGraph_t g, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                             struct cudaGraphNodeParams* p) {
  static cudaGraph_t body;  // the loop's body runs once: into the same list
  body = g;
  p->conditional.phGraph_out = &body;
  *n = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  *x = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph*>(g)));
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Graph*>(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete reinterpret_cast<Graph*>(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
  for (const Op& o : reinterpret_cast<Graph*>(x)->ops) {
    if (o.ev)
      o.ev->at = g_now;
    else
      g_now += o.ms;
  }
  return cudaSuccess;
}
}
