// A stand-in for the CUDA runtime, preloaded into a process without a GPU, for
// tests of the library's host side: what it launches, what it uploads, and
// what it does when a call of the runtime fails.  "Device" memory is host
// memory, copies are memmove, kernels do not run.
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime_api.h>

namespace {
int g_device = 0;
int g_fail_launches = 0;  // kernels to refuse
int g_mallocs_left = -1;  // device allocations until one fails, and all after it (-1: none fails)
int g_err_bits = 0;       // written by the next cooperative kernel ...
int* g_err_word = nullptr;  // ... to the int cleared last by an asynchronous memset
cudaError_t g_last = cudaSuccess;
long long g_launches = 0;
std::vector<unsigned char> g_uploads;  // bytes of host-to-device copies, in order
std::set<std::pair<int, const void*>> g_smem_set;
int g_smem_refused = 0;  // kernels launched with more dynamic shared memory than their device allows
struct Config { dim3 g, b; size_t smem; cudaStream_t st; };
std::vector<Config> g_cfg;

cudaError_t launch(const void* f, size_t smem, bool coop) {
  if (g_fail_launches > 0) {
    --g_fail_launches;
    return g_last = cudaErrorLaunchOutOfResources;
  }
  if (smem > 48 * 1024 && !g_smem_set.count({g_device, f})) {
    ++g_smem_refused;
    return g_last = cudaErrorInvalidValue;
  }
  ++g_launches;
  if (coop && g_err_bits && g_err_word) {
    *g_err_word |= g_err_bits;
    g_err_bits = 0;
  }
  return cudaSuccess;
}
void copy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  if (k == cudaMemcpyHostToDevice) {
    const unsigned char* p = static_cast<const unsigned char*>(s);
    g_uploads.insert(g_uploads.end(), p, p + n);
  }
  std::memmove(d, s, n);
}
}  // namespace

extern "C" {
// ---- control -------------------------------------------------------------------
void fake_set_device(int d) { g_device = d; }
void fake_fail_launches(int n) { g_fail_launches = n; }
void fake_fail_malloc_after(int n) { g_mallocs_left = n; }
void fake_next_error(int bits) { g_err_bits = bits; }
long long fake_launches() { return g_launches; }
int fake_smem_refused() { return g_smem_refused; }
// Bytes uploaded since the last call (up to cap of them to out).
size_t fake_uploads(unsigned char* out, size_t cap) {
  const size_t n = g_uploads.size();
  std::memcpy(out, g_uploads.data(), n < cap ? n : cap);
  g_uploads.clear();
  return n;
}

// ---- runtime -------------------------------------------------------------------
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* st) {
  g_cfg.push_back({g, b, smem, st});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  const Config c = g_cfg.back();
  g_cfg.pop_back();
  *g = c.g; *b = c.b; *smem = c.smem;
  *static_cast<cudaStream_t*>(st) = c.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem, false); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  bool coop = false;
  for (unsigned k = 0; k < c->numAttrs; ++k) coop |= c->attrs[k].id == cudaLaunchAttributeCooperative;
  return launch(f, c->dynamicSmemBytes, coop);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int) {
  g_smem_set.insert({g_device, f});
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "an error of the stand-in runtime"; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_mallocs_left == 0) return g_last = cudaErrorMemoryAllocation;
  if (g_mallocs_left > 0) --g_mallocs_left;
  *p = std::calloc(1, n ? n : 1);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(1, n ? n : 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { copy(d, s, n, k); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  copy(d, s, n, k);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  if (n == sizeof(int) && v == 0) g_err_word = static_cast<int*>(d);
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return g_last = cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return g_last = cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return g_last = cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return g_last = cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return g_last = cudaErrorInvalidSymbol; }
}
