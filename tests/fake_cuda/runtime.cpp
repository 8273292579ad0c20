// A stand-in for the CUDA runtime with no device behind it, for tests of the library's host code.
// "Device" memory is host memory, copies and memsets happen at once, and kernels do not run: every
// launch, copy, synchronisation and event operation is reported to a hook (one C function), which may
// write what a kernel would have written and may answer with an error code.  Loaded with RTLD_GLOBAL before
// the library, its symbols take the place of libcudart's.
// Launches check what the runtime would: clusters of more than 8 CTAs need
// cudaFuncAttributeNonPortableClusterSizeAllowed on that very function.
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

extern "C" {

struct FakeOp {
  const char* kind;  // "launch", "memcpy", "memset", "sync", "record", "wait", "malloc", "free", "stream"
  const char* name;  // launch: the kernel's (mangled) name
  unsigned long long stream;  // 0: the legacy stream; else the number of the stream's creation
  void** args;       // launch: the kernel's arguments; copies: {dst, src}; malloc: {the block}
  unsigned long long size;    // bytes of a copy or block; event number of record and wait
  int grid, cluster, completion_event;
};
typedef int (*FakeHook)(const FakeOp*);
static FakeHook g_hook = nullptr;
void fake_set_hook(FakeHook h) { g_hook = h; }

}  // extern "C"

namespace {
std::mutex g_mu;
std::map<const void*, std::string> g_name;
std::map<const void*, std::map<int, int>> g_attr;
std::map<const void*, std::vector<char>> g_var;
std::atomic<unsigned long long> g_streams{0}, g_events{0};
thread_local cudaError_t t_last = cudaSuccess;
struct Config { dim3 grid, block; size_t smem; cudaStream_t stream; };
thread_local std::vector<Config> t_cfg;

unsigned long long id(const void* h) { return h ? *static_cast<const unsigned long long*>(h) : 0ull; }
void* handle(std::atomic<unsigned long long>& n) { return new unsigned long long(++n); }
cudaError_t ret(int e) {
  if (e) t_last = (cudaError_t)e;
  return (cudaError_t)e;
}
cudaError_t op(const char* kind, const char* name, cudaStream_t s, void** args, unsigned long long size, int grid = 0,
               int cluster = 0, int ev = 0) {
  const FakeOp o{kind, name, id(s), args, size, grid, cluster, ev};
  return ret(g_hook ? g_hook(&o) : 0);
}
cudaError_t launch(const void* f, dim3 grid, void** args, cudaStream_t s, int cluster, int ev) {
  std::string name;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    name = g_name[f];
    if (cluster > 8 && !g_attr[f][cudaFuncAttributeNonPortableClusterSizeAllowed]) return ret(cudaErrorInvalidClusterSize);
  }
  return op("launch", name.c_str(), s, args, 0, (int)(grid.x * grid.y * grid.z), cluster, ev);
}
cudaError_t copy(const char* kind, void* d, const void* s, size_t n, cudaStream_t st) {
  void* a[2] = {d, const_cast<void*>(s)};
  const cudaError_t e = op(kind, "", st, a, n);
  if (e == cudaSuccess) memmove(d, s, n);
  return e;
}
int encode_tiled() { return 0; }
}  // namespace

extern "C" {

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_name[host] = name;
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t size, int, int) { g_var[host].resize(size); }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, void* st) {
  t_cfg.push_back({g, b, sm, (cudaStream_t)st});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sm, void* st) {
  const Config c = t_cfg.back();
  t_cfg.pop_back();
  *g = c.grid;
  *b = c.block;
  *sm = c.smem;
  *static_cast<cudaStream_t*>(st) = c.stream;
  return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3, void** args, size_t, cudaStream_t s) {
  return launch(f, g, args, s, 0, 0);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3, void** args, size_t, cudaStream_t s) {
  return launch(f, g, args, s, 0, 0);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
  int cluster = 0, ev = 0;
  for (unsigned i = 0; i < c->numAttrs; ++i) {
    if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = (int)c->attrs[i].val.clusterDim.x;
    if (c->attrs[i].id == cudaLaunchAttributeLaunchCompletionEvent)
      ev = (int)id(c->attrs[i].val.launchCompletionEvent.event);
  }
  return launch(f, c->gridDim, args, c->stream, cluster, ev);
}

cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> lk(g_mu);
  g_attr[f][a] = v;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f) {
  std::lock_guard<std::mutex> lk(g_mu);
  memset(a, 0, sizeof(*a));
  const int v = g_attr[f][cudaFuncAttributeMaxDynamicSharedMemorySize];
  a->maxDynamicSharedSizeBytes = v ? v : 48 * 1024;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = 1;
  return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  memset(p, 0, sizeof(*p));
  p->major = 10;
  p->multiProcessorCount = 148;
  p->sharedMemPerBlockOptin = 232448;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) {
  *least = 0;
  *greatest = -5;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *f = (void*)encode_tiled;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) {
  *p = g_var[sym].data();
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "an error of the stand-in runtime"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = t_last;
  t_last = cudaSuccess;
  return e;
}

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = calloc(1, n);
  return op("malloc", "", nullptr, p, n);
}
cudaError_t cudaFree(void* p) {
  const cudaError_t e = op("free", "", nullptr, &p, 0);
  free(p);
  return e;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return copy("memcpy", d, s, n, nullptr); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  return copy("memcpy", d, s, n, st);
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t st) {
  void* a[2] = {d, const_cast<void*>(s)};
  const cudaError_t e = op("memcpy", "", st, a, w * h);
  for (size_t i = 0; e == cudaSuccess && i < h; ++i) memmove((char*)d + i * dp, (const char*)s + i * sp, w);
  return e;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  void* a[2] = {d, nullptr};
  const cudaError_t e = op("memset", "", st, a, n);
  if (e == cudaSuccess) memset(d, v, n);
  return e;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaMemset2DAsync(void* d, size_t p, int v, size_t w, size_t h, cudaStream_t st) {
  void* a[2] = {d, nullptr};
  const cudaError_t e = op("memset", "", st, a, w * h);
  for (size_t i = 0; e == cudaSuccess && i < h; ++i) memset((char*)d + i * p, v, w);
  return e;
}

cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) {
  *s = (cudaStream_t)handle(g_streams);
  return op("stream", "", *s, nullptr, 0);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { return cudaStreamCreateWithPriority(s, f, 0); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return op("sync", "", s, nullptr, 0); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { return op("wait", "", s, nullptr, id(e)); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t)handle(g_events);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return op("record", "", s, nullptr, id(e)); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }

}  // extern "C"
