// A CUDA runtime without a GPU for tests of the host paths: preloaded before
// libemd_gb300.so, it keeps "device" memory on the host, runs no kernel (what a kernel
// would write stays zero), and checks what the real one would check of a call: the
// launch's shared memory against the kernel's limit, streams and memory against the
// current device.  fake_* set failures and read counts.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
struct Fake {
  std::mutex mu;
  std::map<const void*, int> limit;        // kernel -> dynamic shared memory it may use
  std::map<void*, std::pair<size_t, int>> mem;  // allocation -> size, device
  size_t held = 0, budget = ~size_t(0);
  int wrong_device = 0, launches = 0, fail_end_capture = 0;
  cudaError_t last = cudaSuccess;
  std::map<const void*, std::string> names;
  std::string watched;       // argument `arg` of the last launch of the kernel of this name
  int arg = 0, count = 0;
  unsigned long long seen = 0;
  std::string failing;       // the kernel whose next launch fails
} F;
thread_local int device = 0;
thread_local struct {
  dim3 g, b;
  size_t sm;
  cudaStream_t st;
} cfg;
cudaError_t err(cudaError_t e) {
  if (e != cudaSuccess) F.last = e;
  return e;
}
int device_of(cudaStream_t s) { return s ? *reinterpret_cast<int*>(s) : device; }
cudaError_t launch(const void* k, dim3 g, dim3 b, void** args, size_t sm, cudaStream_t s) {
  std::lock_guard<std::mutex> l(F.mu);
  if (device_of(s) != device) {
    F.wrong_device++;
    return err(cudaErrorInvalidResourceHandle);
  }
  const auto it = F.limit.find(k);
  const size_t most = it == F.limit.end() ? 48 * 1024 : size_t(it->second);
  if (sm > most || g.x == 0 || b.x * b.y * b.z > 1024) return err(cudaErrorInvalidValue);
  const std::string& name = F.names[k];
  if (!F.failing.empty() && name.find(F.failing) != std::string::npos) {
    F.failing.clear();
    return err(cudaErrorLaunchOutOfResources);
  }
  F.launches++;
  if (!F.watched.empty() && name.find(F.watched) != std::string::npos) {
    memcpy(&F.seen, args[F.arg], sizeof F.seen);
    F.count++;
  }
  return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_set_budget(size_t bytes) { F.budget = bytes; }
size_t fake_held() { return F.held; }
int fake_wrong_device() { return F.wrong_device; }
int fake_launches() { return F.launches; }
void fake_watch(const char* kernel, int arg) { F.watched = kernel, F.arg = arg, F.count = 0; }
int fake_count() { return F.count; }
void fake_fail_launch(const char* kernel) { F.failing = kernel; }
unsigned long long fake_seen() { return F.seen; }
void fake_fail_end_capture(int n) { F.fail_end_capture = n; }

cudaError_t cudaGetDeviceCount(int* n) { return *n = 2, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return device = d, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = device, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { return memset(p, 0, sizeof *p), cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = F.last;
  F.last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }

cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> l(F.mu);
  *p = nullptr;
  if (F.held + n > F.budget) return err(cudaErrorMemoryAllocation);
  *p = calloc(n ? n : 1, 1);
  F.mem[*p] = {n, device};
  F.held += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> l(F.mu);
  const auto it = F.mem.find(p);
  if (it == F.mem.end()) return p ? err(cudaErrorInvalidValue) : cudaSuccess;
  F.held -= it->second.first;
  F.mem.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = calloc(n, 1), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return memmove(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
  for (size_t i = 0; i < h; ++i) memmove(static_cast<char*>(d) + i * dp, static_cast<const char*>(s) + i * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return memset(d, v, n), cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  int* d = static_cast<int*>(malloc(sizeof(int)));
  *d = device;
  *s = reinterpret_cast<cudaStream_t>(d);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = static_cast<cudaEvent_t>(malloc(1));
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = nullptr;
  if (F.fail_end_capture > 0 && F.fail_end_capture--) return err(cudaErrorStreamCaptureInvalidated);
  *g = static_cast<cudaGraph_t>(malloc(1));
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = static_cast<cudaGraphExec_t>(malloc(1));
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return free(e), cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return free(g), cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> l(F.mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) F.limit[f] = v;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, struct CUstream_st* s) {
  cfg.g = g, cfg.b = b, cfg.sm = sm, cfg.st = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sm, void* s) {
  *g = cfg.g, *b = cfg.b, *sm = cfg.sm, *static_cast<cudaStream_t*>(s) = cfg.st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void** a, size_t sm, cudaStream_t s) {
  return launch(k, g, b, a, sm, s);
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t sm, cudaStream_t s) {
  return launch(f, g, b, a, sm, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
  return launch(f, c->gridDim, c->blockDim, a, c->dynamicSmemBytes, c->stream);
}
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  F.names[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
}
