// A CUDA runtime without a GPU, for tests of what the library asks of the runtime: device and
// pinned memory are host memory, copies and clears happen at once (or, on a stream that is
// capturing, not at all), kernels do nothing.  Kernel launches and function attributes are
// written to a log with the kernel's name and whether a capture was open.  Linked first: the
// objects' constructors register their kernels here.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<const void*, std::string> names;
std::map<const void*, size_t> smem;  // kernels' dynamic shared-memory limits, where set
std::map<void*, size_t> device, pinned;
std::string log_text;
cudaStream_t capturing = nullptr;
bool open_capture = false;
struct Call {
  dim3 grid, block;
  size_t bytes;
  cudaStream_t stream;
} pushed;
char handle;  // something for streams, events and graphs to point to

void* take(std::map<void*, size_t>& live, size_t n) {
  void* p = calloc(n ? n : 1, 1);
  live[p] = n;
  return p;
}
cudaError_t give(std::map<void*, size_t>& live, void* p) {
  if (p && !live.erase(p)) return cudaErrorInvalidValue;
  free(p);
  return cudaSuccess;
}
size_t total(const std::map<void*, size_t>& live) {
  size_t s = 0;
  for (const auto& x : live) s += x.second;
  return s;
}
bool in_capture(cudaStream_t st) { return open_capture && st == capturing; }
}  // namespace

extern "C" {
const char* fake_log() { return log_text.c_str(); }
void fake_clear() { log_text.clear(); }
size_t fake_pinned() { return total(pinned); }
size_t fake_device() { return total(device); }

void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*,
                            int*) {
  names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t n, struct CUstream_st* st) {
  pushed = Call{g, b, n, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* n, void* st) {
  *g = pushed.grid;
  *b = pushed.block;
  *n = pushed.bytes;
  *static_cast<cudaStream_t*>(st) = pushed.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t n, cudaStream_t st) {
  log_text += std::string(in_capture(st) ? "captured " : "launched ") + names[f] + "\n";
  return n <= 48 << 10 || (smem.count(f) && n <= smem[f]) ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem[f] = v;
  log_text += std::string(open_capture ? "attribute-in-capture " : "attribute ") + names[f] + "\n";
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void*) {
  memset(a, 0, sizeof(*a));
  a->maxThreadsPerBlock = 1024;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) { return *p = take(device, n), cudaSuccess; }
cudaError_t cudaFree(void* p) { return give(device, p); }
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = take(pinned, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return give(pinned, p); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = *t = 1ull << 30, cudaSuccess; }
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, enum cudaMemcpyKind) {
  return memcpy(to, from, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, enum cudaMemcpyKind, cudaStream_t st) {
  if (!in_capture(st)) memcpy(to, from, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
  if (!in_capture(st)) memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = take(device, 1 << 20), cudaSuccess; }

cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaSetDeviceFlags(unsigned) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int) {
  memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 2;
  p->warpSize = 32;
  return cudaSuccess;
}
cudaError_t cudaDriverGetVersion(int* v) { return *v = 12090, cudaSuccess; }
cudaError_t cudaRuntimeGetVersion(int* v) { return *v = 12090, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error of the test's runtime"; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  return *s = reinterpret_cast<cudaStream_t>(new char), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode) {
  capturing = s;
  open_capture = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  open_capture = false;
  return *g = reinterpret_cast<cudaGraph_t>(&handle), cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, enum cudaStreamCaptureStatus* c) {
  return *c = in_capture(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  return *e = reinterpret_cast<cudaGraphExec_t>(&handle), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = reinterpret_cast<cudaEvent_t>(&handle), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
}  // extern "C"
