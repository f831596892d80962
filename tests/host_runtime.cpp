// A CUDA runtime for tests of the library's host code without a GPU: device memory is host memory,
// copies are made at once, kernels do not run.  Every enqueued operation is recorded with its
// stream, so that a test can ask what is ordered before what (host_runtime.py), and a call can be
// made to fail.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

namespace {

std::mutex mu;
std::string text;                       // the record, one operation per line
std::map<const void*, std::string> kernels;
std::map<std::string, std::pair<int, int>> failures;   // call -> (calls until it fails, status)
std::map<const void*, int> streams, events;
const void* capturing = nullptr;
thread_local int new_fails_in = -1;     // operator new of this thread (-1: never)

int id_of(std::map<const void*, int>& m, const void* p) {
  std::lock_guard<std::mutex> lk(mu);
  return m.emplace(p, (int)m.size()).first->second;
}
struct Quiet {   // allocations of this runtime do not count
  int fails_in = new_fails_in;
  Quiet() { new_fails_in = -1; }
  ~Quiet() { new_fails_in = fails_in; }
};
void log_line(const std::string& line) {
  std::lock_guard<std::mutex> lk(mu);
  text += line + "\n";
}
#define log(line)   \
  do {              \
    Quiet quiet;    \
    log_line(line); \
  } while (0)
std::string at(cudaStream_t s) { return std::to_string(id_of(streams, s)); }
std::string ev(cudaEvent_t e) { return std::to_string(id_of(events, e)); }
std::string hex(const void* p) { return std::to_string((unsigned long long)p); }
cudaError_t status(const char* call) {
  Quiet quiet;
  std::lock_guard<std::mutex> lk(mu);
  auto it = failures.find(call);
  if (it == failures.end()) return cudaSuccess;
  if (it->second.first-- > 0) return cudaSuccess;
  const cudaError_t e = (cudaError_t)it->second.second;
  failures.erase(it);
  return e;
}
void* handle() { return std::malloc(16); }

}  // namespace

// ------------------------------------------------------------------ for the test
extern "C" const char* host_record() { return text.c_str(); }
extern "C" void host_forget() { text.clear(); }
extern "C" void host_fail(const char* call, int after, int code) { failures[call] = {after, code}; }
extern "C" void host_fail_new(int after) { new_fails_in = after; }
extern "C" void host_capture(void* stream, int on) { capturing = on ? stream : nullptr; }

void* operator new(size_t n) {
  if (new_fails_in >= 0 && new_fails_in-- == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

// ------------------------------------------------------------------ the runtime
extern "C" {

void** __cudaRegisterFatBinary(void*) {
  static void* none;
  return &none;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

static thread_local struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} pushed;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
  pushed = {g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  *g = pushed.grid;
  *b = pushed.block;
  *smem = pushed.smem;
  *(cudaStream_t*)st = pushed.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t st) {
  log("kernel " + at(st) + " " + kernels[f]);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  log("kernel " + at(c->stream) + " " + kernels[f]);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) {
  const cudaError_t e = status("cudaMallocAsync");
  return e == cudaSuccess ? cudaMalloc(p, n) : e;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *f = *t = (size_t)180 << 30;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
  const char* const names[] = {"copy", "upload", "download", "copy", "copy"};
  const cudaError_t e = status(names[kind]);
  if (e != cudaSuccess) return e;
  log(names[kind] + (" " + at(st)) + " " + hex(d) + " " + hex(s) + " " + std::to_string(n));
  std::memmove(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
  log("set " + at(st) + " " + hex(p) + " " + std::to_string(n));
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  std::memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorInvalidSymbol; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) {
  return cudaErrorNotSupported;
}

cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof(*p));
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) {
  *lo = *hi = 0;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
  *n = 1;
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = (cudaStream_t)handle();
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  log("wait_stream " + at(s));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  log("wait " + at(s) + " " + ev(e));
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t)handle();
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  log("record " + at(s) + " " + ev(e));
  return cudaSuccess;
}
cudaError_t cudaEventRecordWithFlags(cudaEvent_t e, cudaStream_t s, unsigned) { return cudaEventRecord(e, s); }
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  log("wait_event " + ev(e));
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.f;
  return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  if (capturing) return cudaErrorIllegalState;
  capturing = s;
  log("capture " + at(s));
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  capturing = nullptr;
  *g = (cudaGraph_t)handle();
  log("captured " + at(s));
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
  *st = capturing == s ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)handle();
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
  log("graph " + at(s));
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }

}  // extern "C"
