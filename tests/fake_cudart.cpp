// A CUDA runtime that runs nothing, for host-side tests of the library's
// launch and allocation logic: device memory is host memory that no kernel
// touches, every call goes into a log, and a chosen launch fails.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <map>
#include <string>

namespace {
// (kernels register before this file's globals would be made)
std::map<const void*, std::string>& names() {
  static std::map<const void*, std::string> m;
  return m;
}
std::string calls, fail_kernel;
cudaError_t last = cudaSuccess;

void log(const char* what, const void* p, size_t bytes) {
  char line[96];
  snprintf(line, sizeof line, "%s %p %zu\n", what, p, bytes);
  calls += line;
}

cudaError_t launched(const void* fn) {
  const std::string& name = names()[fn];
  if (!fail_kernel.empty() && name.find(fail_kernel) != std::string::npos) {
    calls += "failed " + name + "\n";
    return last = cudaErrorMemoryAllocation;  // what a kernel loaded on first use returns on a full GPU
  }
  calls += "launch " + name + "\n";
  return cudaSuccess;
}
}  // namespace

extern "C" {

// ---- the test's side
const char* fake_calls() { return calls.c_str(); }
void fake_clear() { calls.clear(); }
void fake_fail(const char* kernel) { fail_kernel = kernel; }  // launches of kernels with this in their name fail

// ---- what compiled CUDA code calls to register its kernels
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* fn, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names()[fn] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 0; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }

// ---- the runtime
cudaError_t cudaLaunchKernel(const void* fn, dim3, dim3, void**, size_t, cudaStream_t) { return launched(fn); }
cudaError_t __cudaLaunchKernel(void* fn, dim3, dim3, void**, size_t, cudaStream_t) { return launched(fn); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* fn, void**) { return launched(fn); }
cudaError_t cudaMalloc(void** p, size_t bytes) {
  *p = calloc(1, bytes);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int, size_t bytes) {
  log("memset", p, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int, size_t bytes, cudaStream_t) {
  log("memset", p, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void*, size_t bytes, cudaMemcpyKind) {
  log("memcpy", dst, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void*, size_t bytes, cudaMemcpyKind, cudaStream_t) {
  log("memcpy", dst, bytes);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  calls += "synchronize\n";
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "an error of the fake runtime"; }
cudaError_t cudaGetDevice(int* device) {
  *device = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.f;
  return cudaSuccess;
}
}
