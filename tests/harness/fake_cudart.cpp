// A CUDA runtime of the host for CPU tests of the library's host code,
// preloaded before it: device memory is host memory, kernels do not run.
// Kernel attributes are kept per device, as the runtime keeps them, and a
// launch that wants more dynamic shared memory than the current device's
// limit for that kernel fails.  fake_expire_waits makes the sliced products
// report what they report when a bounded wait runs out: a 1 in the error word
// their arguments point to.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <utility>

namespace {
std::mutex mu;
std::map<const void *, std::string> names;                  // host stub -> kernel
std::map<std::pair<const void *, int>, size_t> smem_limit;  // (kernel, device)
std::set<const void *> words;                               // live allocations of one int
int expire = 0;
long long launched = 0;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
struct Config {
  dim3 grid, block;
  size_t smem;
  void *stream;
};
thread_local Config config;

int encode_stub() { return 0; }
}  // namespace

extern "C" {
void fake_expire_waits(int on) { expire = on; }
long long fake_launches() { return launched; }

void **__cudaRegisterFatBinary(void *) {
  static void *h = nullptr;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *fun, char *, const char *name, int, void *, void *, void *, void *,
                            int *) {
  std::lock_guard<std::mutex> lk(mu);
  names[fun] = name;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fun) {
  *k = (cudaKernel_t)fun;
  return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *st) {
  config = {g, b, smem, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
  *g = config.grid;
  *b = config.block;
  *smem = config.smem;
  *(void **)st = config.stream;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **args, size_t smem, cudaStream_t) {
  std::lock_guard<std::mutex> lk(mu);
  launched++;
  auto it = smem_limit.find({(const void *)k, device});
  if (smem > (it == smem_limit.end() ? (size_t)48 * 1024 : it->second)) return last = cudaErrorInvalidValue;
  if (expire && names[(const void *)k].find("k_ozaki") != std::string::npos) {
    const char *a = (const char *)args[2];  // (tensor map, tensor map, arguments)
    for (int o = 0; o < 2048; o += 8) {
      void *p;
      memcpy(&p, a + o, 8);
      if (words.count(p)) {
        *(int *)p = 1;
        break;
      }
    }
  }
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::mutex> lk(mu);
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_limit[{f, device}] = (size_t)v;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
  *v = 152;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : "error"; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = calloc(1, n ? n : 1);
  std::lock_guard<std::mutex> lk(mu);
  if (n == sizeof(int)) words.insert(*p);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  {
    std::lock_guard<std::mutex> lk(mu);
    words.erase(p);
  }
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  *s = (cudaStream_t)calloc(1, 8);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
  *e = (cudaEvent_t)calloc(1, 8);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) {
  *p = (cudaMemPool_t)calloc(1, 8);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *r) {
  *f = (void *)encode_stub;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}
