// A CUDA runtime without a device, for tests of the library's host code: device
// memory is host memory that starts as garbage, copies and clears happen at once,
// kernels are written down and not run, and every operation that touches memory
// or launches is a line of a log with the stream it was issued on.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <utility>
#include <vector>

namespace {
struct State {
  std::string log;
  std::map<const void *, std::string> kernel;     // by host function
  std::map<const void *, int> dynamic_smem;       // by host function, what was allowed
  std::map<void *, size_t> device;                // allocations
  std::map<cudaStream_t, int> stream;
  std::set<cudaMemPool_t> pools;                  // alive
  std::vector<int> result;                        // what the next copy to the host brings
  std::map<std::string, void *> symbol;
  std::map<const void *, std::pair<std::string, size_t>> variable;
  size_t capacity = SIZE_MAX;
  int sms = 152;
  int streams = 0;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
  bool capturing = false, spoilt = false;  // some stream; by a call it does not take
  unsigned long long context = 1;
};
State &st() {
  static State s;
  return s;
}
std::string name(cudaStream_t s) {
  auto it = st().stream.find(s);
  return it == st().stream.end() ? "default" : "s" + std::to_string(it->second);
}
void note(const std::string &line) { st().log += line + "\n"; }
size_t used() {
  size_t n = 0;
  for (auto &d : st().device) n += d.second;
  return n;
}
cudaError_t take(void **p, size_t n) {
  if (used() + n > st().capacity) return cudaErrorMemoryAllocation;
  *p = std::malloc(n ? n : 1);
  std::memset(*p, 0xa5, n);
  st().device[*p] = n;
  return cudaSuccess;
}
cudaError_t give(void *p) {
  if (!p) return cudaSuccess;
  if (!st().device.erase(p)) return cudaErrorInvalidValue;
  std::free(p);
  return cudaSuccess;
}
cudaError_t copy(void *d, const void *s, size_t n, cudaMemcpyKind kind, const std::string &where) {
  static const char *const kinds[] = {"h2h", "h2d", "d2h", "d2d", "any"};
  note(std::string("copy ") + kinds[kind] + " " + std::to_string(n) + " " + where);
  std::memcpy(d, s, n);
  if (kind == cudaMemcpyDeviceToHost && !st().result.empty()) {
    std::memcpy(d, st().result.data(), std::min(n, 4 * st().result.size()));
    st().result.clear();
  }
  return cudaSuccess;
}
cudaError_t launch(const char *how, const void *f, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
  const int allowed = st().dynamic_smem.count(f) ? st().dynamic_smem[f] : 48 << 10;
  if (smem > static_cast<size_t>(allowed)) return cudaErrorInvalidValue;
  note(std::string(how) + " " + st().kernel[f] + " " + std::to_string(grid.x) + " " + std::to_string(block.x) + " " +
       name(s));
  return cudaSuccess;
}
}  // namespace

extern "C" {

// ---- for the test
const char *fake_log() { return st().log.c_str(); }
void fake_clear_log() { st().log.clear(); }
// The first `n` words of the next copy to the host.
void fake_result(const int *words, int n) { st().result.assign(words, words + n); }
void fake_capacity(size_t bytes) { st().capacity = bytes; }
void fake_multiprocessors(int n) { st().sms = n; }
void fake_begin_capture() {
  st().capturing = true;
  st().spoilt = false;
}
int fake_end_capture() {
  st().capturing = false;
  return st().spoilt ? 1 : 0;
}
size_t fake_used() { return used(); }
size_t fake_variable_bytes() {  // of the library's device variables
  size_t n = 0;
  for (auto &v : st().variable) n += v.second.second;
  return n;
}

// ---- the runtime
cudaError_t cudaDeviceReset() {  // every allocation, pool and attribute is gone
  st().device.clear();
  st().pools.clear();
  st().dynamic_smem.clear();
  st().symbol.clear();
  ++st().context;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *p) { return static_cast<void **>(p); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *device, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  st().kernel[host] = device;
}
void __cudaRegisterVar(void **, char *host, char *, const char *device, int, size_t size, int, int) {
  st().variable[host] = {device, size};
}
namespace {
struct Call {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_call;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) {
  g_call = {g, b, m, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s) {
  *g = g_call.grid;
  *b = g_call.block;
  *m = g_call.smem;
  *static_cast<cudaStream_t *>(s) = g_call.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(f));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **, size_t m, cudaStream_t s) {
  return launch("launch", k, g, b, m, s);
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t m, cudaStream_t s) {
  return launch("launch", f, g, b, m, s);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3 g, dim3 b, void **, size_t m, cudaStream_t s) {
  return launch("cooperative", f, g, b, m, s);
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  switch (a) {
    case cudaDevAttrMultiProcessorCount: *v = st().sms; break;
    case cudaDevAttrMaxSharedMemoryPerBlockOptin: *v = 232448; break;
    case cudaDevAttrMaxSharedMemoryPerMultiprocessor: *v = 233472; break;
    case cudaDevAttrReservedSharedMemoryPerBlock: *v = 1024; break;
    case cudaDevAttrComputeCapabilityMajor: *v = 10; break;
    case cudaDevAttrComputeCapabilityMinor: *v = 3; break;
    default: *v = 0;
  }
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int block, size_t) {
  *n = block >= 1024 ? 1 : 1024 / block;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *f) {
  std::memset(a, 0, sizeof *a);
  a->sharedSizeBytes = 10240;
  a->maxDynamicSharedSizeBytes = st().dynamic_smem.count(f) ? st().dynamic_smem[f] : 48 << 10;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) st().dynamic_smem[f] = v;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
  std::memset(p, 0, sizeof *p);
  return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(std::malloc(1));
  st().stream[*s] = st().streams++;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  st().stream.erase(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  note("wait " + name(s));
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t n) {
  note("malloc " + std::to_string(n));
  return take(p, n);
}
cudaError_t cudaFree(void *p) {
  if (p) note("free " + std::to_string(st().device[p]));
  return give(p);
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t pool, cudaStream_t) {
  return st().pools.count(pool) ? take(p, n) : cudaErrorInvalidValue;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return give(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const cudaMemPoolProps *) {
  if (st().capturing && st().mode != cudaStreamCaptureModeRelaxed) {
    st().spoilt = true;
    return cudaErrorStreamCaptureUnsupported;
  }
  *pool = reinterpret_cast<cudaMemPool_t>(std::malloc(1));
  st().pools.insert(*pool);
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t pool) {
  return st().pools.erase(pool) ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) {
  std::swap(*m, st().mode);
  return cudaSuccess;
}
static CUresult fake_context_id(CUcontext, unsigned long long *id) {
  *id = st().context;
  return CUDA_SUCCESS;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *found) {
  *p = reinterpret_cast<void *>(&fake_context_id);
  *found = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
  *p = std::calloc(1, n ? n : 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, k, "default"); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t q) {
  return copy(d, s, n, k, name(q));
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
  note("clear " + std::to_string(n) + " default");
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s) {
  note("clear " + std::to_string(n) + " " + name(s));
  auto block = st().device.upper_bound(p);  // what a lost context had is no memory
  if (block == st().device.begin() ||
      static_cast<char *>(p) + n > static_cast<char *>((--block)->first) + block->second)
    return cudaErrorIllegalAddress;
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *symbol) {
  auto &v = st().variable[symbol];
  void *&at = st().symbol[v.first];
  if (!at) take(&at, v.second);
  *p = at;
  return cudaSuccess;
}

}  // extern "C"
