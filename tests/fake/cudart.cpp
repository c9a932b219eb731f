// A CUDA runtime without a GPU, linked with the library's objects in place of the
// real one (tests/fake/__init__.py): device memory is host memory under a limit,
// kernels do nothing, copies and fills are done at once, a launch can be made to
// fail, and the operations on streams and events are listed in order.  It covers
// the calls the library makes; tests use it for the host code's failure paths.
#include <cuda_runtime_api.h>

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<char *, size_t> mem;
std::map<const void *, std::string> kernels;
size_t limit_ = ~(size_t)0, used_ = 0;
std::string fail_kernel, log_;
cudaError_t last = cudaSuccess;
long ids = 0;
struct Config {
  dim3 g, b;
  size_t smem;
  cudaStream_t st;
} config;

cudaError_t note(cudaError_t e) { return e == cudaSuccess ? e : last = e; }
void line(const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  log_ += buf;
  log_ += '\n';
}
bool device(const void *p) {
  auto it = mem.upper_bound((char *)p);
  if (it == mem.begin()) return false;
  --it;
  return (const char *)p < it->first + it->second;
}
int unsupported(...) { return 0; }  // the linear algebra libraries' calls
}  // namespace

extern "C" {
// ---- control
void fake_limit(size_t bytes) { limit_ = bytes; }
size_t fake_used() { return used_; }
void fake_fail(const char *kernel) { fail_kernel = kernel ? kernel : ""; }
const char *fake_log() { return log_.c_str(); }
void fake_clear_log() { log_.clear(); }

// ---- memory
cudaError_t cudaMalloc(void **p, size_t n) {
  if (used_ + n > limit_) return note(cudaErrorMemoryAllocation);
  char *q = (char *)calloc(n ? n : 1, 1);
  mem[q] = n;
  used_ += n;
  *p = q;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  auto it = mem.find((char *)p);
  if (!p) return cudaSuccess;
  if (it == mem.end()) return note(cudaErrorInvalidValue);
  used_ -= it->second;
  mem.erase(it);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
  *p = calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaHostRegister(void *, size_t, unsigned) { return note(cudaErrorNotSupported); }
cudaError_t cudaHostUnregister(void *) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  line("copy %p", (void *)st);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h,
                              cudaMemcpyKind, cudaStream_t) {
  for (size_t r = 0; r < h; r++) memcpy((char *)d + r * dp, (const char *)s + r * sp, w);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
  memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
  memset(a, 0, sizeof *a);
  a->type = device(p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *s) {
  *p = const_cast<void *>(s);
  return cudaSuccess;
}

// ---- device
cudaError_t cudaGetDeviceCount(int *n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
  memset(p, 0, sizeof *p);
  p->major = 10;
  p->minor = 3;
  p->multiProcessorCount = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) {
  *lo = 0;
  *hi = -5;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
  memset(a, 0, sizeof *a);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)(++ids);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned f, int) {
  return cudaStreamCreateWithFlags(s, f);
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  line("sync %p", (void *)s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  line("wait %p %p", (void *)s, (void *)e);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t)(++ids);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  line("record %p %p", (void *)s, (void *)e);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
  *g = (cudaGraph_t)(++ids);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)(++ids);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
  line("graph %p", (void *)s);
  return cudaSuccess;
}

// ---- kernels (the calls that nvcc's host code makes)
void **__cudaRegisterFatBinary(void *) { return (void **)&config; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *fun, char *, const char *name, int, uint3 *,
                            uint3 *, dim3 *, dim3 *, int *) {
  kernels[fun] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
  config = {g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
  *g = config.g;
  *b = config.b;
  *smem = config.smem;
  *(cudaStream_t *)st = config.st;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fun) {
  *k = (cudaKernel_t)fun;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *fun, dim3, dim3, void **, size_t, cudaStream_t s) {
  const std::string &name = kernels[fun];
  if (!fail_kernel.empty() && name.find(fail_kernel) != std::string::npos)
    return note(cudaErrorLaunchOutOfResources);
  line("launch %p %s", (void *)s, name.c_str());
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **a, size_t n,
                               cudaStream_t s) {
  return cudaLaunchKernel((const void *)k, g, b, a, n, s);
}

// ---- the linear algebra libraries are not loaded
void *__wrap_dlopen(const char *, int) { return &config; }
void *__wrap_dlsym(void *, const char *) { return (void *)&unsupported; }
}
