// A stand-in for the CUDA runtime, preloaded in front of the real one, so that the library's host code runs on a machine
// without a GPU: device memory is host memory, copies are memcpy, kernels are not run (their launches are counted). It
// keeps count of what is alive and can let a call fail, which no real device does on request.
//   fake_live(kind), fake_calls(kind) ... objects of a kind that are alive, calls that made one so far
//   fake_bytes(kind) .................... bytes of those alive
//   fake_fail(kind, n) .................. the n-th call from now (1: the next) that makes one fails, once
//   fake_launches(part) ................. launches so far of kernels whose (mangled) name contains `part`
//   fake_raise(part, value) ............. kernels whose name contains `part` store `value` at their second argument, an int*
// With FAKE_NO_MANAGED_ACCESS in the environment the host may not touch managed memory while kernels run.
// Kinds: "malloc" (device), "host" (pinned), "stream", "event", "graph", "exec", "capture".
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace {
struct Kind {
  std::map<void*, std::size_t> live;
  int calls = 0, fail_in = 0;
};
std::recursive_mutex mutex;
std::map<std::string, Kind>& kinds() {
  static std::map<std::string, Kind> k;
  return k;
}
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> n;
  return n;
}
std::map<std::string, long>& launches() {
  static std::map<std::string, long> n;
  return n;
}
std::string raise_part;
int raise_value = 0;

cudaError_t make(const char* kind, std::size_t bytes, void** out) {
  std::lock_guard<std::recursive_mutex> lock(mutex);
  Kind& k = kinds()[kind];
  ++k.calls;
  if (k.fail_in > 0 && --k.fail_in == 0) return cudaErrorMemoryAllocation;
  *out = std::calloc(1, bytes < 16 ? 16 : bytes);
  k.live[*out] = bytes;
  return cudaSuccess;
}
cudaError_t drop(const char* kind, void* p) {
  std::lock_guard<std::recursive_mutex> lock(mutex);
  if (!p) return cudaSuccess;
  if (kinds()[kind].live.erase(p) == 0) return cudaErrorInvalidValue;
  std::free(p);
  return cudaSuccess;
}
template <typename H>
cudaError_t make_handle(const char* kind, H* out) {
  void* p = nullptr;
  const cudaError_t e = make(kind, 16, &p);
  if (e == cudaSuccess) *out = static_cast<H>(p);
  return e;
}
}  // namespace

extern "C" {

int fake_live(const char* kind) { return static_cast<int>(kinds()[kind].live.size()); }
long long fake_bytes(const char* kind) {
  long long n = 0;
  for (const auto& l : kinds()[kind].live) n += static_cast<long long>(l.second);
  return n;
}
int fake_calls(const char* kind) { return kinds()[kind].calls; }
void fake_fail(const char* kind, int n) { kinds()[kind].fail_in = n; }
long fake_launches(const char* part) {
  long n = 0;
  for (const auto& l : launches())
    if (l.first.find(part) != std::string::npos) n += l.second;
  return n;
}
void fake_raise(const char* part, int value) {
  raise_part = part;
  raise_value = value;
}

cudaError_t cudaMalloc(void** p, size_t n) { return make("malloc", n, p); }
cudaError_t cudaMallocManaged(void** p, size_t n, unsigned int) { return make("malloc", n, p); }
cudaError_t cudaMemAdvise(const void*, size_t, cudaMemoryAdvise, int) { return cudaSuccess; }
cudaError_t cudaFree(void* p) { return drop("malloc", p); }
cudaError_t cudaMallocHost(void** p, size_t n) { return make("host", n, p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) { return make("host", n, p); }
cudaError_t cudaFreeHost(void* p) { return drop("host", p); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) { return make_handle("stream", s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop("stream", s); }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return make_handle("event", e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) { return make_handle("event", e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop("event", e); }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  Kind& k = kinds()["capture"];
  ++k.calls;
  return k.fail_in > 0 && --k.fail_in == 0 ? cudaErrorStreamCaptureUnsupported : cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return make_handle("graph", g); }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return drop("graph", g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { return make_handle("exec", x); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return drop("exec", x); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
  ++launches()["graph"];
  return cudaSuccess;
}

cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
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
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t, cudaStream_t) {
  std::lock_guard<std::recursive_mutex> lock(mutex);
  const std::string& name = names()[f];
  ++launches()[name];
  if (!raise_part.empty() && name.find(raise_part) != std::string::npos) **static_cast<int**>(args[1]) = raise_value;
  return cudaSuccess;
}

cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448
       : a == cudaDevAttrComputeCapabilityMajor ? 10
       : a == cudaDevAttrConcurrentManagedAccess ? std::getenv("FAKE_NO_MANAGED_ACCESS") == nullptr : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned int) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof *a);
  a->type = cudaMemoryTypeUnregistered;
  if (kinds()["host"].live.count(const_cast<void*>(p))) a->type = cudaMemoryTypeHost;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  static std::vector<char> memory(1 << 20);
  *p = memory.data();
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }

// What the compiler emits for kernels and their launches.
static thread_local struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} pushed;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  pushed = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = pushed.grid;
  *block = pushed.block;
  *smem = pushed.smem;
  *static_cast<cudaStream_t*>(stream) = pushed.stream;
  return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) {
  static void* handle = nullptr;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  std::lock_guard<std::recursive_mutex> lock(mutex);
  names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

}  // extern "C"
