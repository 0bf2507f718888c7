// A CUDA runtime without a GPU, for the host code of the kernel library: the objects of its .cu files are linked against this
// file, every call succeeds and launches are taken down instead of executed.
// Like the real one it refuses a launch whose dynamic shared memory was not allowed on the current device.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <stdlib.h>

#include <atomic>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "operators.h"

namespace {

std::mutex lock;
std::map<const void*, std::string> names;                // kernels by the address that launches name
std::map<const void*, std::string> arrays;               // __device__ arrays likewise
std::set<std::pair<const void*, int>> allowed;           // (kernel, device) with a raised shared-memory limit
std::map<const void*, unsigned long long> borrowed;      // the words of a pool that launches were handed -> how often
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
int refuse_allowing = 0;
std::atomic<int> recording{0};
char words[1 << 20] __attribute__((aligned(256)));       // stands for every __device__ array

CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

// ---------------------------------------------------------------- what a test asks and sets
void fake_set_device(int d) { device = d; }
void fake_record(int on) { recording = on; }  // every stream is being captured
void fake_refuse_allowing(int n) { refuse_allowing = n; }  // the next n raises of a limit fail
// How many different places of a pool were handed out, the smallest and largest number of times that one was, and the first and the last.
void fake_borrowed(unsigned long long* out5) {
  std::lock_guard<std::mutex> hold(lock);
  out5[0] = borrowed.size();
  out5[1] = ~0ull, out5[2] = 0;
  for (const auto& [at, n] : borrowed) {
    if (n < out5[1]) out5[1] = n;
    if (n > out5[2]) out5[2] = n;
  }
  out5[3] = borrowed.empty() ? 0 : static_cast<const char*>(borrowed.begin()->first) - words;
  out5[4] = borrowed.empty() ? 0 : static_cast<const char*>(borrowed.rbegin()->first) - words;
  borrowed.clear();
}

// `threads` threads, each with `each` split products (768 x 768 x 8192) or column sums (300 x 768); the number of refused calls.
int fake_threads(int threads, int each, int products) {
  std::vector<std::thread> all;
  std::atomic<int> refused{0};
  void* p = reinterpret_cast<void*>(1 << 20);  // never followed
  const long long need = tb_gemm_workspace_bytes(768, 768, 8192);
  for (int t = 0; t < threads; ++t)
    all.emplace_back([&] {
      for (int i = 0; i < each; ++i)
        if (products ? need == 0 || tb_gemm_bf16(p, p, p, 768, 768, 8192, 768, 768, 768, 1, 1, 0, nullptr, nullptr, nullptr, 0, p, need, nullptr)
                     : tb_col_sum(p, 300, 768, 768, p, static_cast<float*>(p), nullptr))
          ++refused;
    });
  for (auto& t : all) t.join();
  return refused;
}

void tb_note_launch(int) {}

// ---------------------------------------------------------------- the runtime
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names[host] = name;
}
void __cudaRegisterVar(void**, char* host, char*, const char* name, int, size_t, int, int) { arrays[host] = name; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }

cudaError_t cudaGetDevice(int* out) { *out = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* out, cudaDeviceAttr, int) { *out = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaHostAlloc(void** out, size_t size, unsigned) { *out = calloc(1, size); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** out, void* p, unsigned) { *out = p; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** out, const void*) { *out = words; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** out, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *out = (void*)encode;
  if (q != nullptr) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* out) {
  *out = recording ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 74; return cudaSuccess; }

cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute what, int) {
  std::lock_guard<std::mutex> hold(lock);
  if (refuse_allowing > 0) return --refuse_allowing, last = cudaErrorInvalidValue;
  if (what == cudaFuncAttributeMaxDynamicSharedMemorySize) allowed.insert({kernel, device});
  return cudaSuccess;
}

static cudaError_t launched(const void* kernel, size_t smem, void** args) {
  std::lock_guard<std::mutex> hold(lock);
  if (smem > 48 * 1024 && !allowed.count({kernel, device})) return last = cudaErrorInvalidValue;
  // Pool words among the arguments: the eight-byte values that point into the array.  The one structure that carries such a
  // pointer, the GEMM's, is its sixth argument and at least 96 bytes long; the column sums' sixth is the pointer itself.
  const std::string& name = names[kernel];
  const int bytes = name.find("k_gemm") != std::string::npos ? 96 : name.find("k_col_sum") != std::string::npos ? 8 : 0;
  for (int at = 0; at < bytes; at += 8) {
    const char* value = *reinterpret_cast<const char* const*>(static_cast<const char*>(args[5]) + at);
    if (value >= words && value < words + sizeof(words)) ++borrowed[value];
  }
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* kernel, void** args) {
  return launched(kernel, config->dynamicSmemBytes, args);
}
cudaError_t cudaLaunchKernel(const void* kernel, dim3, dim3, void** args, size_t smem, cudaStream_t) { return launched(kernel, smem, args); }
cudaError_t cudaLaunchCooperativeKernel(const void* kernel, dim3, dim3, void** args, size_t smem, cudaStream_t) {
  return launched(kernel, smem, args);
}

}  // extern "C"
