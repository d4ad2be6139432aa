// A stand-in for the CUDA runtime under which the library's host code runs without a GPU (LD_PRELOAD).
//
// Device memory is host memory, kernels do nothing, and work on a stream is put off until something waits for
// it.  That is the latest the real runtime may do it: a copy between device and pageable memory may still read
// or write the caller's buffer after the call that issued it, and neither a device memset nor the end of a
// synchronous copy from pageable memory is ordered before work on a non-blocking stream.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

namespace {

struct Op {
  bool host;  // reads or writes pageable host memory
  std::function<void()> run;
};

std::map<const void*, size_t> g_device, g_pinned;
std::map<uintptr_t, std::vector<Op>> g_streams;  // 0: the legacy stream
std::map<std::string, int> g_calls, g_fail;
size_t g_total = (size_t)280 << 30, g_used = 0;
int g_status = 0, g_unsettled = 0;
bool g_capturing = false;
cudaError_t g_last = cudaSuccess;
uintptr_t g_next = 16;

uintptr_t id(cudaStream_t s) { return (uintptr_t)s <= 2 ? 0 : (uintptr_t)s; }

bool within(const std::map<const void*, size_t>& m, const void* p) {
  auto it = m.upper_bound(p);
  if (it == m.begin()) return false;
  --it;
  return (const char*)p < (const char*)it->first + it->second;
}
bool pageable(const void* p) { return !within(g_device, p) && !within(g_pinned, p); }

cudaError_t called(const char* name) {
  ++g_calls[name];
  auto it = g_fail.find(name);
  if (it == g_fail.end() || --it->second > 0) return cudaSuccess;
  g_fail.erase(it);
  return g_last = cudaErrorUnknown;
}

void drain(uintptr_t s) {
  std::vector<Op> ops;
  ops.swap(g_streams[s]);
  for (Op& o : ops) o.run();
}
void drain_all() {
  for (auto& s : g_streams) drain(s.first);
}

cudaError_t take(void** p, size_t n, bool device) {
  if (device && g_used + n > g_total) return g_last = cudaErrorMemoryAllocation;
  void* q = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  if (q == MAP_FAILED) return cudaErrorMemoryAllocation;
  (device ? g_device : g_pinned)[q] = n;
  if (device) g_used += n;
  *p = q;
  return cudaSuccess;
}
cudaError_t give(void* p, bool device) {
  if (!p) return cudaSuccess;
  drain_all();
  auto& m = device ? g_device : g_pinned;
  auto it = m.find(p);
  if (it == m.end()) return cudaErrorInvalidValue;
  if (device) g_used -= it->second;
  munmap(p, it->second ? it->second : 1);
  m.erase(it);
  return cudaSuccess;
}

void copy(void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
  std::memcpy(dst, src, n);
  // the status word that a kernel sets when one of its waits expires: by itself, or at the end of the sums
  if (kind == cudaMemcpyDeviceToHost && g_status) {
    if (n == sizeof(int)) std::memcpy(dst, &g_status, sizeof(int));
    else if (within(g_pinned, dst)) std::memcpy((char*)dst + n - 8, &g_status, sizeof(int));
  }
}

}  // namespace

extern "C" {

// ---- what a test sets and reads ----
void fake_set_memory(size_t total) { g_total = total; }
size_t fake_used() { return g_used; }
void fake_status(int s) { g_status = s; }
void fake_fail(const char* name, int nth) {  // the nth call from now on fails (0: none does)
  if (nth > 0) g_fail[name] = nth;
  else g_fail.erase(name);
}
int fake_calls(const char* name) { return g_calls[name]; }
int fake_unsettled() { return g_unsettled; }  // launches that found writes of the legacy stream not ordered before
int fake_host_copies() {                      // copies from or into pageable memory still to be done
  int n = 0;
  for (auto& s : g_streams)
    for (Op& o : s.second) n += o.host;
  return n;
}

// ---- the runtime ----
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return called("cudaGetDeviceCount"); }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof(*p));
  p->major = 10;
  p->minor = 3;
  p->multiProcessorCount = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return called("cudaFuncSetAttribute"); }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return cudaErrorInvalidSymbol; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = g_total - g_used;
  *t = g_total;
  return called("cudaMemGetInfo");
}
cudaError_t cudaMalloc(void** p, size_t n) {
  const cudaError_t e = called("cudaMalloc");
  return e != cudaSuccess ? g_last = cudaErrorMemoryAllocation : take(p, n, true);
}
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n, false); }
cudaError_t cudaFree(void* p) { called("cudaFree"); return give(p, true); }
cudaError_t cudaFreeHost(void* p) { return give(p, false); }

cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t s) {
  if (cudaError_t e = called("cudaMemcpyAsync")) return e;
  g_streams[id(s)].push_back({pageable(dst) || pageable(src), [=] { copy(dst, src, n, kind); }});
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
  if (cudaError_t e = called("cudaMemcpy")) return e;
  drain(0);
  if (kind == cudaMemcpyDeviceToHost) {
    copy(dst, src, n, kind);
  } else {  // from pageable memory: staged, the last part of the way not waited for
    auto staged = std::make_shared<std::vector<char>>((const char*)src, (const char*)src + n);
    g_streams[0].push_back({false, [=] { std::memcpy(dst, staged->data(), n); }});
  }
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
  if (cudaError_t e = called("cudaMemsetAsync")) return e;
  g_streams[id(s)].push_back({false, [=] { std::memset(p, v, n); }});
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  if (cudaError_t e = called("cudaMemset")) return e;
  g_streams[0].push_back({false, [=] { std::memset(p, v, n); }});
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)(g_next += 16);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { drain(id(s)); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (cudaError_t e = called("cudaStreamSynchronize")) return e;
  drain(id(s));
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  drain_all();
  return called("cudaDeviceSynchronize");
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
  *c = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  drain(id(s));
  g_capturing = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  g_capturing = false;
  g_streams[id(s)].clear();
  *g = (cudaGraph_t)(g_next += 16);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) {
  *g = (cudaGraphExec_t)(g_next += 16);
  return called("cudaGraphInstantiate");
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return called("cudaGraphExecDestroy"); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return called("cudaGraphLaunch"); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)(g_next += 16); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 0.f; return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}

// ---- what nvcc's host stubs call ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static dim3 g_grid, g_block;
static size_t g_smem;
static cudaStream_t g_st;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  g_grid = grid; g_block = block; g_smem = smem; g_st = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
  *grid = g_grid; *block = g_block; *smem = g_smem; *(cudaStream_t*)s = g_st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t s) {
  if (id(s) && !g_streams[0].empty()) ++g_unsettled;
  g_streams[id(s)].push_back({false, [] {}});
  return called("cudaLaunchKernel");
}
}
