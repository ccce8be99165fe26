// A CUDA runtime without a GPU, for the host side of the library: two devices,
// memory from the heap, kernels that are only noted. A launch with more than 48
// KiB of dynamic shared memory is refused, as by the CUDA runtime, unless the
// function was given that much on the current device.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <utility>

namespace {
int g_dev = 0;
cudaError_t g_last = cudaSuccess;
std::map<const void*, std::string> g_name;                  // host stub -> kernel
std::map<std::pair<int, const void*>, size_t> g_allowed;    // per device
std::map<std::pair<int, std::string>, int> g_launched;      // per device
std::string g_rejected;
char g_symbol[8 << 20];
size_t g_free = (size_t)-1;  // largest allocation that succeeds
struct Call {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_call;

cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
bool fits(const void* f, size_t smem) {
  if (smem <= 48 * 1024) return true;
  const auto it = g_allowed.find({g_dev, f});
  return it != g_allowed.end() && smem <= it->second;
}
cudaError_t launch(const void* f, size_t smem) {
  if (!fits(f, smem)) {
    g_rejected += g_name[f] + "\n";
    return set(cudaErrorInvalidValue);
  }
  ++g_launched[{g_dev, g_name[f]}];
  return cudaSuccess;
}
}  // namespace

extern "C" {
// For the test.
void fake_set_device(int d) { g_dev = d; }
void fake_set_free(size_t bytes) { g_free = bytes; }
const char* fake_rejected() { return g_rejected.c_str(); }
int fake_launches(const char* part) {
  int n = 0;
  for (const auto& l : g_launched)
    if (l.first.first == g_dev && l.first.second.find(part) != std::string::npos) n += l.second;
  return n;
}

void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
  g_name[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) {
  g_call = Call{g, b, smem, (cudaStream_t)st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = g_call.grid;
  *b = g_call.block;
  *smem = g_call.smem;
  *(cudaStream_t*)st = g_call.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) {
  return launch(f, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_allowed[{g_dev, f}] = (size_t)v;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof *a);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t smem, unsigned) {
  *n = fits(f, smem) ? 1 : 0;
  return cudaSuccess;
}
// The second device holds one cluster less (but one).
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
  if (!fits(f, c->dynamicSmemBytes)) return set(cudaErrorInvalidValue);
  const int most = (int)(c->gridDim.x / c->attrs[0].val.clusterDim.x);
  *n = most > 1 ? most - g_dev : most;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = g_dev;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorName(cudaError_t) { return "error"; }
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = n > g_free ? nullptr : std::calloc(n ? n : 1, 1);
  return *p ? cudaSuccess : set(cudaErrorMemoryAllocation);
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  for (size_t i = 0; i < h; ++i) std::memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  *p = g_symbol;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *fn = nullptr;
  *q = cudaDriverEntryPointSymbolNotFound;
  return set(cudaErrorSymbolNotFound);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)std::malloc(8);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)std::malloc(8);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) {
  *t = 1.0f;
  return cudaSuccess;
}
}
