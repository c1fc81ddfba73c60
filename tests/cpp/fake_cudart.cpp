// fake_cudart.cpp -- a CUDA runtime without a GPU, for tests of the engine's
// host code: memory is host memory, kernels do nothing, every call on a device
// is held to that device's limits.  A launch fails where a real one would: more
// dynamic shared memory than the kernel was allowed on the current device.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>

namespace {

constexpr int kDevices = 2, kSms = 148;
constexpr size_t kStatic = 4096;  // of every kernel
std::mutex g_mu;
thread_local int t_dev = 0;
thread_local cudaError_t t_err = cudaSuccess;
int g_optin[kDevices] = {232448, 232448};
std::map<const void*, std::string> g_name;
std::map<std::pair<int, const void*>, size_t> g_limit;  // dynamic shared memory
std::map<std::string, int> g_launches;                  // by name
std::map<std::string, double> g_cost;                   // ms of the launches whose name holds the key
std::map<void*, size_t> g_pool;                         // stream-ordered blocks
size_t g_pool_bytes = 0;
double g_clock = 0.0;
bool g_no_memory = false;
int g_frees = 0;
struct Event {
  double at;
};
struct Call {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
};
thread_local Call t_call;

cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) t_err = e;
  return e;
}
size_t limit_of(const void* f) {
  auto it = g_limit.find({t_dev, f});
  return it == g_limit.end() ? 49152 - kStatic : it->second;
}
cudaError_t launch(const void* f, size_t smem) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (smem > limit_of(f)) return set(cudaErrorInvalidValue);
  const std::string& n = g_name[f];
  ++g_launches[n];
  for (const auto& c : g_cost)
    if (n.find(c.first) != std::string::npos) g_clock += c.second;
  return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- what a test sets and reads ---------------------------------------------
void fake_set_optin(int dev, int bytes) { g_optin[dev] = bytes; }
void fake_set_cost(const char* part, double ms) { g_cost[part] = ms; }
size_t fake_pool_bytes() { return g_pool_bytes; }
void fake_no_memory(int on) { g_no_memory = on != 0; }
int fake_frees() { return g_frees; }  // blocks given back by cudaFree
int fake_launches(const char* part) {
  std::lock_guard<std::mutex> lk(g_mu);
  int n = 0;
  for (const auto& l : g_launches)
    if (l.first.find(part) != std::string::npos) n += l.second;
  return n;
}

// ---- registration and launches ------------------------------------------------
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  g_name[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, CUstream_st* stream) {
  t_call = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = t_call.grid;
  *block = t_call.block;
  *smem = t_call.smem;
  *(cudaStream_t*)stream = t_call.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->dynamicSmemBytes);
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof *a);
  a->sharedSizeBytes = kStatic;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || v < 0 || v + (int)kStatic > g_optin[t_dev])
    return set(cudaErrorInvalidValue);
  g_limit[{t_dev, f}] = (size_t)v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int threads, size_t smem,
                                                                   unsigned) {
  const size_t by_smem = ((size_t)g_optin[t_dev] + 1024) / (smem + kStatic + 1024);
  *n = (int)(by_smem < (size_t)(2048 / threads) ? by_smem : (size_t)(2048 / threads));
  return cudaSuccess;
}

// ---- devices, errors, memory ----------------------------------------------------
cudaError_t cudaGetDeviceCount(int* n) {
  *n = kDevices;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = t_dev;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= kDevices) return set(cudaErrorInvalidDevice);
  t_dev = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int dev) {
  *v = a == cudaDevAttrMultiProcessorCount ? kSms : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? g_optin[dev] : 0;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake CUDA error"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = t_err;
  t_err = cudaSuccess;
  return e;
}
static cudaError_t host_alloc(void** p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  return *p ? cudaSuccess : set(cudaErrorMemoryAllocation);
}
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = nullptr;
  return g_no_memory ? set(cudaErrorMemoryAllocation) : host_alloc(p, n);
}
cudaError_t cudaFree(void* p) {
  ++g_frees;
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return host_alloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return host_alloc(p, n); }
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) {
  const cudaError_t e = cudaMalloc(p, n);
  std::lock_guard<std::mutex> lk(g_mu);
  if (e == cudaSuccess) g_pool_bytes += g_pool[*p] = n;
  return e;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  {
    std::lock_guard<std::mutex> lk(g_mu);
    g_pool_bytes -= g_pool[p];
    g_pool.erase(p);
  }
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* fr, size_t* tot) {
  *fr = *tot = (size_t)180 << 30;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) {
  *p = const_cast<void*>(s);
  return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) {
  *p = nullptr;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }

// ---- streams, events (a clock of the launches' costs), graphs --------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  std::free((void*)s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t) new Event{0.0};
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete (Event*)e;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
  ((Event*)e)->at = g_clock;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(((Event*)b)->at - ((Event*)a)->at);
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  *x = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"
