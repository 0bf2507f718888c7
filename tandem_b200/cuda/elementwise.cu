// Fused element-wise kernels: multi-tensor AdamW and bucket pack/unpack.
//
// adamw: one pass over {param, grad, exp_avg, exp_avg_sq} instead of the nine
// ATen kernels of torch's single-tensor AdamW (the reference's ShardedAdamW,
// tandem/optim.py:28-37, and torch.optim.AdamW(foreach=False) used by its DDP
// path); the arithmetic is in adam.cuh.  Optionally also writes a bf16 copy of
// the updated parameter (the compute copy under mixed precision).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "adam.cuh"
#include "launch.cuh"

namespace {

template <typename G>
__device__ __forceinline__ float grad_of(G g);
template <>
__device__ __forceinline__ float grad_of<float>(float g) { return g; }
template <>
__device__ __forceinline__ float grad_of<__nv_bfloat16>(__nv_bfloat16 g) { return __bfloat162float(g); }

// Four consecutive gradients as floats.
__device__ __forceinline__ float4 grad4(const float* g) { return *reinterpret_cast<const float4*>(g); }
__device__ __forceinline__ float4 grad4(const __nv_bfloat16* g) {
  const uint2 v = *reinterpret_cast<const uint2*>(g);
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}

// Elements [from, n) one by one.
template <typename G>
__device__ __forceinline__ void adam_elements(float* __restrict__ param, const G* __restrict__ grad, float* __restrict__ exp_avg,
                                              float* __restrict__ exp_avg_sq, __nv_bfloat16* __restrict__ shadow, long long from, long long n,
                                              const AdamScalars& s, float grad_scale) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = from + (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    float g = grad_of<G>(grad[i]);
    if (grad_scale != 1.f) g = __fmul_rn(g, grad_scale);
    float p = param[i], m = exp_avg[i], v = exp_avg_sq[i];
    adam_update(p, m, v, g, s);
    param[i] = p;
    exp_avg[i] = m;
    exp_avg_sq[i] = v;
    if (shadow != nullptr) shadow[i] = __float2bfloat16_rn(p);
  }
}

// One pass over all elements.  28 bytes per element for 15 operations: memory bounds it.  Where every array is aligned for it
// (adam_vectors), a thread moves four elements per access and keeps two such groups in flight (with 4-byte accesses, one element at
// a time, 42.9 M fp32 elements took 205 us and 50 M with bf16 gradients 291 us), and the last n % 4 go one by one; else all do.
// Separate kernels: the loop over elements lives on resident warps, and the vectors' 64 registers make it a fifth slower
// (42.9 M: 308 us, 242 by itself with 32).
template <typename G, bool SCALED>
__device__ __forceinline__ void adam_quads(float* __restrict__ param, const G* __restrict__ grad, float* __restrict__ exp_avg,
                                          float* __restrict__ exp_avg_sq, __nv_bfloat16* __restrict__ shadow, long long n, const AdamScalars& s,
                                          float grad_scale) {
  const long long stride = (long long)gridDim.x * blockDim.x, first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long quads = n / 4;
  for (long long i = first; i < quads; i += 2 * stride) {
    float4 g[2], p[2], m[2], v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long at = 4 * (i + u * stride);
      if (at < 4 * quads) {
        g[u] = grad4(grad + at);
        p[u] = *reinterpret_cast<const float4*>(param + at);
        m[u] = *reinterpret_cast<const float4*>(exp_avg + at);
        v[u] = *reinterpret_cast<const float4*>(exp_avg_sq + at);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long at = 4 * (i + u * stride);
      if (at < 4 * quads) {
        if (SCALED) g[u] = make_float4(__fmul_rn(g[u].x, grad_scale), __fmul_rn(g[u].y, grad_scale), __fmul_rn(g[u].z, grad_scale), __fmul_rn(g[u].w, grad_scale));
        adam_update(p[u].x, m[u].x, v[u].x, g[u].x, s);
        adam_update(p[u].y, m[u].y, v[u].y, g[u].y, s);
        adam_update(p[u].z, m[u].z, v[u].z, g[u].z, s);
        adam_update(p[u].w, m[u].w, v[u].w, g[u].w, s);
        *reinterpret_cast<float4*>(param + at) = p[u];
        *reinterpret_cast<float4*>(exp_avg + at) = m[u];
        *reinterpret_cast<float4*>(exp_avg_sq + at) = v[u];
        if (shadow != nullptr) {
          const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(p[u].x, p[u].y), __floats2bfloat162_rn(p[u].z, p[u].w)};
          *reinterpret_cast<uint2*>(shadow + at) = *reinterpret_cast<const uint2*>(h);
        }
      }
    }
  }
  adam_elements<G>(param, grad, exp_avg, exp_avg_sq, shadow, 4 * quads, n, s, SCALED ? grad_scale : 1.f);
}

// (A hundred elements take 1.5 us in the larger kernel, 1.3 in the smaller one; from about 1000 on they are equal.)
template <typename G>
bool adam_vectors(const void* param, const void* grad, const void* exp_avg, const void* exp_avg_sq, const void* shadow, long long n) {
  return n >= 512 && (((uintptr_t)param | (uintptr_t)exp_avg | (uintptr_t)exp_avg_sq) & 15) == 0 && ((uintptr_t)grad & (4 * sizeof(G) - 1)) == 0 &&
         ((uintptr_t)shadow & 7) == 0;
}

template <typename G, bool VECTORS>
__global__ void __launch_bounds__(256)
k_adamw(float* __restrict__ param, const G* __restrict__ grad, float* __restrict__ exp_avg, float* __restrict__ exp_avg_sq,
        __nv_bfloat16* __restrict__ shadow, long long n, AdamScalars s, float grad_scale) {
  tb::pdl_enter();
  if (!VECTORS) adam_elements<G>(param, grad, exp_avg, exp_avg_sq, shadow, 0, n, s, grad_scale);
  else if (grad_scale != 1.f) adam_quads<G, true>(param, grad, exp_avg, exp_avg_sq, shadow, n, s, grad_scale);
  else adam_quads<G, false>(param, grad, exp_avg, exp_avg_sq, shadow, n, s, 1.f);
}

// Same update with the step-dependent scalars read from device memory, so the launch can sit in a
// CUDA graph and still see a new bias correction on every replay.
template <typename G, bool VECTORS>
__global__ void __launch_bounds__(256)
k_adamw_dev(float* __restrict__ param, const G* __restrict__ grad, float* __restrict__ exp_avg, float* __restrict__ exp_avg_sq,
            __nv_bfloat16* __restrict__ shadow, long long n, const AdamScalars* __restrict__ scalars) {
  tb::pdl_enter();
  const AdamScalars s = *scalars;
  if (!VECTORS) adam_elements<G>(param, grad, exp_avg, exp_avg_sq, shadow, 0, n, s, 1.f);
  else adam_quads<G, false>(param, grad, exp_avg, exp_avg_sq, shadow, n, s, 1.f);
}

// One thread: step += 1, then the scalars of that step, in double precision as the host would.
__global__ void k_adam_prepare(double* step, double lr, double beta1, double beta2, double eps, double wd, AdamScalars* out) {
  tb::pdl_enter();
  const double t = *step + 1.0;
  *step = t;
  const double bc1 = 1.0 - pow(beta1, t), bc2 = 1.0 - pow(beta2, t);
  AdamScalars s;
  s.decay = (float)(1.0 - lr * wd);
  s.w1 = (float)(1.0 - beta1);
  s.b2 = (float)beta2;
  s.w2 = (float)(1.0 - beta2);
  s.inv_bias2_sqrt = 1.0f / (float)sqrt(bc2);
  s.eps = (float)eps;
  s.neg_step = (float)(-(lr / bc1));
  s.do_decay = wd != 0.0;
  *out = s;
}

// ---------------------------------------------------------------- multi-tensor copy
#define TB_COPY_MAX 48
struct CopyTable {
  const char* src[TB_COPY_MAX];
  char* dst[TB_COPY_MAX];
  long long bytes[TB_COPY_MAX];
  int count;
};

// blockIdx.y picks the tensor, blockIdx.x strides over it.
__global__ void __launch_bounds__(256) k_multi_copy(CopyTable t) {
  tb::pdl_enter();
  const int k = blockIdx.y;
  const char* s = t.src[k];
  char* d = t.dst[k];
  const long long n = t.bytes[k];
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nth = (long long)gridDim.x * blockDim.x;
  const bool aligned = ((((uintptr_t)s) | ((uintptr_t)d)) & 15) == 0;
  const long long nvec = aligned ? n / 16 : 0;
  for (long long v = tid; v < nvec; v += 4 * nth) {  // four 16-byte loads in flight per thread
    uint4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v + u * nth < nvec) x[u] = reinterpret_cast<const uint4*>(s)[v + u * nth];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v + u * nth < nvec) reinterpret_cast<uint4*>(d)[v + u * nth] = x[u];
  }
  for (long long i = nvec * 16 + tid; i < n; i += nth) d[i] = s[i];
}

}  // namespace

extern "C" void tb_note_launch(int n);

extern "C" {

// 1 (default): kernels are launched with programmatic dependent launch; 0: plain launches (for A/B measurements).
void tb_set_pdl(int on) { tb::pdl_enabled() = on ? 1 : 0; }

// scalars: {1-lr*wd, 1-beta1, beta2, 1-beta2, sqrt(bias_correction2), eps, -lr/bias_correction1}
int tb_adamw(void* param, const void* grad, int grad_is_bf16, void* exp_avg, void* exp_avg_sq, void* shadow_bf16, long long n,
             const float* scalars, int do_decay, float grad_scale, cudaStream_t stream) {
  if (n <= 0) return 0;
  AdamScalars s{scalars[0], scalars[1], scalars[2], scalars[3], 1.0f / scalars[4], scalars[5], scalars[6], do_decay};
  long long want = (n + 256 * 4 - 1) / (256 * 4);
  int blocks = (int)(want > 148 * 8 ? 148 * 8 : want);
  tb_note_launch(1);
#define ADAMW(G) \
  tb::launch(adam_vectors<G>(param, grad, exp_avg, exp_avg_sq, shadow_bf16, n) ? k_adamw<G, true> : k_adamw<G, false>, dim3(blocks), dim3(256), 0, \
             stream, (float*)param, (const G*)grad, (float*)exp_avg, (float*)exp_avg_sq, (__nv_bfloat16*)shadow_bf16, n, s, grad_scale)
  if (grad_is_bf16) ADAMW(__nv_bfloat16);
  else ADAMW(float);
#undef ADAMW
  return (int)cudaGetLastError();
}

// Advances the device-resident step counter (a double) and writes that step's AdamScalars (32 bytes) to `scalars`.
int tb_adam_prepare(void* step_counter, double lr, double beta1, double beta2, double eps, double wd, void* scalars,
                    cudaStream_t stream) {
  tb_note_launch(1);
  tb::launch(k_adam_prepare, dim3(1), dim3(1), 0, stream, (double*)step_counter, lr, beta1, beta2, eps, wd, (AdamScalars*)scalars);
  return (int)cudaGetLastError();
}

// tb_adamw with the scalars taken from device memory (written by tb_adam_prepare).
int tb_adamw_dev(void* param, const void* grad, int grad_is_bf16, void* exp_avg, void* exp_avg_sq, void* shadow_bf16, long long n,
                 const void* scalars, cudaStream_t stream) {
  if (n <= 0) return 0;
  long long want = (n + 256 * 4 - 1) / (256 * 4);
  int blocks = (int)(want > 148 * 8 ? 148 * 8 : want);
  tb_note_launch(1);
#define ADAMW(G) \
  tb::launch(adam_vectors<G>(param, grad, exp_avg, exp_avg_sq, shadow_bf16, n) ? k_adamw_dev<G, true> : k_adamw_dev<G, false>, dim3(blocks), \
             dim3(256), 0, stream, (float*)param, (const G*)grad, (float*)exp_avg, (float*)exp_avg_sq, (__nv_bfloat16*)shadow_bf16, n, \
             (const AdamScalars*)scalars)
  if (grad_is_bf16) ADAMW(__nv_bfloat16);
  else ADAMW(float);
#undef ADAMW
  return (int)cudaGetLastError();
}

// Copies count tensors (src[k] -> dst[k], bytes[k] each) with ceil(count / 48) launches.
int tb_multi_copy(const void* const* src, void* const* dst, const long long* bytes, int count, cudaStream_t stream) {
  for (int base = 0; base < count; base += TB_COPY_MAX) {
    CopyTable t{};
    long long most = 0;
    t.count = count - base < TB_COPY_MAX ? count - base : TB_COPY_MAX;
    for (int k = 0; k < t.count; ++k) {
      t.src[k] = (const char*)src[base + k];
      t.dst[k] = (char*)dst[base + k];
      t.bytes[k] = bytes[base + k];
      if (t.bytes[k] > most) most = t.bytes[k];
    }
    long long want = (most + 256 * 16 * 4 - 1) / (256 * 16 * 4);
    // a few large tensors (a vocabulary's 100 MB: 132 us on 64 blocks) get the whole GPU, many small ones 64 blocks each
    const long long cap = 148 * 8 / t.count > 64 ? 148 * 8 / t.count : 64;
    dim3 grid((unsigned)(want < 1 ? 1 : (want > cap ? cap : want)), t.count);
    tb_note_launch(1);
    tb::launch(k_multi_copy, grid, dim3(256), 0, stream, t);
  }
  return (int)cudaGetLastError();
}

}  // extern "C"
