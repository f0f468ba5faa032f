// A CUDA runtime without a GPU for tests of the library's host side: device
// memory is host memory with bounds, copies and clears are checked against
// them, kernel launches are counted by name and do nothing, and allocations
// fail past a budget.  Linked with the library's objects in place of the real
// runtime.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <utility>

namespace {

std::recursive_mutex g_mu;
std::map<uintptr_t, size_t> g_dev, g_pinned;  // base -> bytes
size_t g_live = 0, g_budget = SIZE_MAX;
unsigned g_coop_blocks = 0;  // of the last cooperative launch
int g_refused = 0, g_violations = 0, g_device = 0, g_pinned_calls = 0, g_dev_calls = 0;
std::map<const void*, std::string> g_name;
std::map<std::string, int> g_launches;
std::set<std::pair<int, const void*>> g_opted;  // (device, kernel) with a shared-memory limit set
cudaError_t g_last = cudaSuccess;

using Lock = std::lock_guard<std::recursive_mutex>;

cudaError_t fail(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}

// Device addresses come from one reserved range, with gaps, and none is used
// again.
constexpr size_t kRange = size_t(1) << 38;
uintptr_t range() {
  static const uintptr_t base = reinterpret_cast<uintptr_t>(
      mmap(nullptr, kRange, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0));
  return base;
}
uintptr_t g_next = 0;

// Whether [p, p + bytes) is a device range outside every allocation.
bool leaves(const void* p, size_t bytes) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  if (a < range() || a >= range() + kRange) return p == nullptr && bytes > 0;  // host memory
  auto it = g_dev.upper_bound(a);
  if (it == g_dev.begin()) return true;
  --it;
  return a + bytes > it->first + it->second;
}

cudaError_t copy(void* d, const void* s, size_t bytes) {
  Lock l(g_mu);
  if (leaves(d, bytes) || leaves(s, bytes)) {
    ++g_violations;
    return cudaSuccess;
  }
  if (bytes) std::memmove(d, s, bytes);
  return cudaSuccess;
}

cudaError_t launch(const void* f, size_t smem) {
  Lock l(g_mu);
  // (Every kernel that asks for as much has some static shared memory too.)
  if (smem >= 48 * 1024 && !g_opted.count({g_device, f})) return fail(cudaErrorInvalidValue);
  ++g_launches[g_name.count(f) ? g_name[f] : std::string("?")];
  return cudaSuccess;
}

struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local Config g_cfg;

}  // namespace

extern "C" {

// ---- the test's side ----
void fake_reset() {
  Lock l(g_mu);
  g_budget = SIZE_MAX;
  g_refused = g_violations = g_device = g_pinned_calls = g_dev_calls = 0;
  g_launches.clear();
  g_last = cudaSuccess;
}
void fake_set_budget(unsigned long long bytes) { g_budget = bytes; }
unsigned long long fake_live() { return g_live; }
int fake_refused() { return g_refused; }
int fake_violations() { return g_violations; }
int fake_pinned_calls() { return g_pinned_calls; }
int fake_device_calls() { return g_dev_calls; }
unsigned fake_cooperative_blocks() { return g_coop_blocks; }
void fake_set_device(int d) { g_device = d; }
int fake_launches(const char* part) {
  Lock l(g_mu);
  int n = 0;
  for (auto& k : g_launches)
    if (k.first.find(part) != std::string::npos) n += k.second;
  return n;
}
// Fills bytes [offset, offset + 4) of every `stride` bytes of page-locked memory with `v`.
void fake_poke_pinned(unsigned long long offset, unsigned long long stride, uint32_t v) {
  Lock l(g_mu);
  for (auto& p : g_pinned)
    for (size_t at = offset; at + 4 <= p.second; at += stride)
      std::memcpy(reinterpret_cast<void*>(p.first + at), &v, 4);
}

// ---- the runtime's side ----
void** __cudaRegisterFatBinary(void*) {
  static void* h = nullptr;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_name[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* s) {
  g_cfg = {grid, block, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
  *grid = g_cfg.grid;
  *block = g_cfg.block;
  *smem = g_cfg.smem;
  *static_cast<cudaStream_t*>(s) = g_cfg.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3, void**, size_t smem, cudaStream_t) {
  g_coop_blocks = grid.x;
  return launch(f, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->dynamicSmemBytes);
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
  Lock l(g_mu);
  ++g_dev_calls;
  *p = nullptr;
  if (g_live + bytes > g_budget) {
    ++g_refused;
    return fail(cudaErrorMemoryAllocation);
  }
  *p = reinterpret_cast<void*>(range() + g_next);
  g_next += (bytes + (2u << 20)) >> 20 << 20;
  g_dev[reinterpret_cast<uintptr_t>(*p)] = bytes;
  g_live += bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  Lock l(g_mu);
  auto it = g_dev.find(reinterpret_cast<uintptr_t>(p));
  if (it == g_dev.end()) return p ? fail(cudaErrorInvalidValue) : cudaSuccess;
  g_live -= it->second;
  madvise(p, it->second, MADV_DONTNEED);
  g_dev.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t bytes) {
  Lock l(g_mu);
  ++g_pinned_calls;
  *p = std::calloc(1, bytes + 64);
  g_pinned[reinterpret_cast<uintptr_t>(*p)] = bytes;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  Lock l(g_mu);
  g_pinned.erase(reinterpret_cast<uintptr_t>(p));
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *t = *f = size_t(1) << 34;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t b, cudaMemcpyKind) { return copy(d, s, b); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t b, cudaMemcpyKind, cudaStream_t) { return copy(d, s, b); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t b, cudaStream_t) {
  Lock l(g_mu);
  if (leaves(d, b))
    ++g_violations;
  else
    std::memset(d, v, b);
  return cudaSuccess;
}

cudaError_t cudaGetDevice(int* d) {
  *d = g_device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int) {
  Lock l(g_mu);
  g_opted.insert({g_device, f});
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  *p = nullptr;
  return fail(cudaErrorInvalidSymbol);
}
cudaError_t cudaGetLastError() {
  Lock l(g_mu);
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(1);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(1);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaHostRegister(void*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }

}  // extern "C"
