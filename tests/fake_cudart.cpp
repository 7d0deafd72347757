// A stand-in for the CUDA runtime in which nothing runs: it keeps what the library asks of
// it - shared-memory limits per (device, kernel), launches - and refuses a launch as the
// runtime does, with cudaErrorInvalidValue, when its dynamic shared memory is above the limit
// in force for that kernel on the current device.  Linked with the library's own objects it
// lets a CPU test see every launch shape the host code makes, on any number of devices.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <utility>
#include <vector>

namespace {
constexpr int kDevices = 4;
constexpr size_t kDefaultSmem = 48 * 1024, kOptinSmem = 227 * 1024;
int g_dev = 0;
cudaError_t g_last = cudaSuccess;
std::map<std::pair<int, const void *>, size_t> g_limit;
long long g_launches = 0, g_refused = 0, g_fail_at = -1;
size_t g_next = 1 << 20, g_max_smem = 0;
std::vector<std::vector<double>> g_copies;  // small synchronous uploads, in order
struct Config { dim3 grid, block; size_t smem; cudaStream_t st; } g_cfg;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
cudaError_t launch(const void *f, dim3 g, dim3 b, size_t smem) {
  const auto it = g_limit.find({g_dev, f});
  const size_t lim = it == g_limit.end() ? kDefaultSmem : it->second;
  const bool ok = smem <= lim && g.x && g.y && g.z && b.x && b.x * b.y * b.z <= 1024;
  if (g_launches++ == g_fail_at) return done(cudaErrorLaunchOutOfResources);
  if (smem > g_max_smem) g_max_smem = smem;
  if (!ok) ++g_refused;
  return done(ok ? cudaSuccess : cudaErrorInvalidValue);
}
}  // namespace

extern "C" {

// what the test reads
void fake_fail_at(long long n) { g_fail_at = n; g_launches = 0; }  // launch n from now on fails, -1: none
long long fake_launches() { return g_launches; }
long long fake_refused() { return g_refused; }
size_t fake_max_smem() { return g_max_smem; }
int fake_copies() { return (int)g_copies.size(); }
const double *fake_copy(int k, long long *n) {
  *n = (long long)g_copies[k].size();
  return g_copies[k].data();
}
void fake_reset() { g_launches = g_refused = 0; g_max_smem = 0; g_last = cudaSuccess; g_copies.clear(); }

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void *st) {
  g_cfg = {g, b, smem, (cudaStream_t)st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
  *g = g_cfg.grid; *b = g_cfg.block; *smem = g_cfg.smem; *(cudaStream_t *)st = g_cfg.st;
  return cudaSuccess;
}

cudaError_t cudaGetDevice(int *d) { *d = g_dev; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d >= kDevices) return done(cudaErrorInvalidDevice);
  g_dev = d;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? (int)kOptinSmem : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if ((size_t)v > kOptinSmem) return done(cudaErrorInvalidValue);
    g_limit[{g_dev, f}] = (size_t)v;
  }
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t smem, cudaStream_t) {
  return launch(f, g, b, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "refused by the stand-in"; }

// device memory is an address that nothing touches
cudaError_t cudaMalloc(void **p, size_t n) { *p = (void *)g_next; g_next += (n + 255) & ~(size_t)255; return cudaSuccess; }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = calloc(1, n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void *, const void *src, size_t n, cudaMemcpyKind k) {
  if (k == cudaMemcpyHostToDevice && n <= 65536 && n % 8 == 0) {
    g_copies.emplace_back(n / 8);
    memcpy(g_copies.back().data(), src, n);
  }
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { *p = (void *)g_next; return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

// cuTensorMapEncodeTiled is the only driver entry point asked for: it succeeds
static int encode_ok() { return 0; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **p, unsigned long long, cudaDriverEntryPointQueryResult *r) {
  *p = (void *)&encode_ok;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

}  // extern "C"
