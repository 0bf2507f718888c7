// Memory-bound layer kernels around the GEMMs, bf16 in / bf16 out with fp32 math:
// LayerNorm forward/backward, fused softmax-cross-entropy forward/backward, token+position
// embedding forward/backward and column sums (bias gradients).  Each reads its input once and
// writes its output once.  The reference runs these as separate ATen calls
// (nn.LayerNorm, F.cross_entropy, nn.Embedding, autograd's bias reductions: tandem/model.py:50-116).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>
#include <mutex>

#include "launch.cuh"
#include "noalloc.h"

extern "C" void tb_note_launch(int n);

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* f) {
  uint4 v = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ void store8(__nv_bfloat16* p, const float* f) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = v;
}

// ------------------------------------------------------------------------------------ LayerNorm
// One warp per row; D is a multiple of 8.  MAXV 16-byte vectors per lane cover D <= 32*8*MAXV.
template <int MAXV>
__global__ void __launch_bounds__(256)
k_ln_fwd(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
         __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, int M, int D, float eps) {
  tb::pdl_enter();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= M) return;
  const int nvec = D >> 3;
  float v[MAXV][8];
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    const int vi = lane + 32 * j;
    if (vi < nvec) {
      load8(x + (size_t)row * D + vi * 8, v[j]);
#pragma unroll
      for (int e = 0; e < 8; ++e) sum += v[j][e];
    }
  }
  const float mean = warp_sum(sum) / D;
  float sq = 0.f;
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    if (lane + 32 * j < nvec) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float d = v[j][e] - mean;
        sq += d * d;
      }
    }
  }
  const float rstd = rsqrtf(warp_sum(sq) / D + eps);
  if (lane == 0) {
    mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    const int vi = lane + 32 * j;
    if (vi < nvec) {
      float wv[8], bv[8], o[8];
      load8(w + vi * 8, wv);
      load8(b + vi * 8, bv);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = (v[j][e] - mean) * rstd * wv[e] + bv[e];
      store8(y + (size_t)row * D + vi * 8, o);
    }
  }
}

// dx for each row, and per-block partial sums of dw = sum dy*xhat and db = sum dy into
// part[blockIdx.x][2][D] (fp32).  A second kernel adds the partials in a fixed order.
// add (optional): a second gradient of the same input, summed into dx in fp32 before the one rounding
// -- the residual branch's gradient in a pre-LayerNorm block, which autograd would otherwise add with a
// separate pass over the activations.
// Rows are software-pipelined: while a warp works on one row, the 16-byte loads of its next row (dy and x, kept
// packed as bf16 so that they cost half the registers) are already in flight, and the residual gradient of the
// current row is requested before the row's reductions start.  With one row per warp in flight the kernel ran at
// the pace of one memory round trip per row (0.42 of the copy bandwidth); two rows per warp and two blocks per SM
// keep about 100 KB per SM on the way.
template <int MAXV>
__global__ void __launch_bounds__(256, MAXV <= 4 ? 2 : 1)
k_ln_bwd(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
         const float* __restrict__ mean_in, const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ add,
         __nv_bfloat16* __restrict__ dx, float* __restrict__ part, int M, int D) {
  tb::pdl_enter();
  extern __shared__ __align__(16) float sh[];  // [warps][2][D]
  const int warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = D >> 3;
  float dw[MAXV][8], db[MAXV][8];
#pragma unroll
  for (int j = 0; j < MAXV; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) dw[j][e] = db[j][e] = 0.f;
  const int stride = gridDim.x * warps;
  int row = blockIdx.x * warps + warp;
  constexpr bool AHEAD = MAXV <= 4;  // wider rows have no registers left for a second row
  uint4 ndy[MAXV], nx[MAXV];  // the next row, packed
  float nmean = 0.f, nrstd = 0.f;
  auto fetch = [&](int r) {
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int vi = lane + 32 * j;
      if (vi < nvec) {
        ndy[j] = __ldg(reinterpret_cast<const uint4*>(dy + (size_t)r * D + vi * 8));
        nx[j] = __ldg(reinterpret_cast<const uint4*>(x + (size_t)r * D + vi * 8));
      }
    }
    nmean = mean_in[r];
    nrstd = rstd_in[r];
  };
  if (AHEAD && row < M) fetch(row);
  for (; row < M; row += stride) {
    if (!AHEAD) fetch(row);
    uint4 cdy[MAXV], cx[MAXV], cadd[MAXV];
    const float mean = nmean, rstd = nrstd;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      cdy[j] = ndy[j];
      cx[j] = nx[j];
    }
    if (AHEAD && row + stride < M) fetch(row + stride);
    if (add != nullptr) {  // may alias dx: this row's dx is written only after these loads have been consumed
#pragma unroll
      for (int j = 0; j < MAXV; ++j) {
        const int vi = lane + 32 * j;
        if (vi < nvec) cadd[j] = *reinterpret_cast<const uint4*>(add + (size_t)row * D + vi * 8);
      }
    }
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int vi = lane + 32 * j;
      if (vi < nvec) {
        float dyv[8], xv[8], wv[8];
        unpack8(cdy[j], dyv);
        unpack8(cx[j], xv);
        load8(w + vi * 8, wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = (xv[e] - mean) * rstd;
          const float gv = dyv[e] * wv[e];
          s1 += gv;
          s2 += gv * xh;
          dw[j][e] += dyv[e] * xh;
          db[j][e] += dyv[e];
        }
      }
    }
    s1 = warp_sum(s1) / D;
    s2 = warp_sum(s2) / D;
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int vi = lane + 32 * j;
      if (vi < nvec) {
        float dyv[8], xv[8], wv[8], o[8];
        unpack8(cdy[j], dyv);
        unpack8(cx[j], xv);
        load8(w + vi * 8, wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = (xv[e] - mean) * rstd;  // the same operations as above: the same values
          o[e] = rstd * (dyv[e] * wv[e] - s1 - xh * s2);
        }
        if (add != nullptr) {
          float a[8];
          unpack8(cadd[j], a);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += a[e];
        }
        store8(dx + (size_t)row * D + vi * 8, o);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    const int vi = lane + 32 * j;
    if (vi < nvec) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {  // 16-byte stores: scalar ones, 32 bytes apart from lane to lane, meet in the same bank eight at a time
        *reinterpret_cast<float4*>(sh + (warp * 2 + 0) * D + vi * 8 + 4 * q) = *reinterpret_cast<const float4*>(&dw[j][4 * q]);
        *reinterpret_cast<float4*>(sh + (warp * 2 + 1) * D + vi * 8 + 4 * q) = *reinterpret_cast<const float4*>(&db[j][4 * q]);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) {
    float acc = 0.f;
    for (int wv = 0; wv < warps; ++wv) acc += sh[wv * 2 * D + i];
    part[(size_t)blockIdx.x * 2 * D + i] = acc;
  }
}

// out[c] = sum over p of part[p][c], written as bf16.  32 columns x 8 row lanes per block: each lane adds
// every 8th partial, then the 8 lanes are combined in a fixed order (deterministic).
__global__ void __launch_bounds__(256)
k_reduce_partials(const float* __restrict__ part, int parts, int width, __nv_bfloat16* __restrict__ out0,
                  __nv_bfloat16* __restrict__ out1, int split) {
  tb::pdl_enter();
  __shared__ float sh[8][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float acc = 0.f;
  if (c < width && parts <= 64) {  // up to eight per lane: the long body below costs more than it saves (512 x 256 backward: 4.5 / 4.9 us)
    for (int p = ry; p < parts; p += 8) acc += part[(size_t)p * width + c];
  } else if (c < width) {
    constexpr int U = 40;  // loads in flight, added in order: one trip to L2 for up to 320 partials
    for (int p = ry; p < parts; p += 8 * U) {
      float v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (p + 8 * u < parts) v[u] = part[(size_t)(p + 8 * u) * width + c];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (p + 8 * u < parts) acc += v[u];
    }
  }
  sh[ry][cx] = acc;
  __syncthreads();
  if (ry == 0 && c < width) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += sh[k][cx];
    if (c < split) out0[c] = __float2bfloat16_rn(t);
    else out1[c - split] = __float2bfloat16_rn(t);
  }
}

// ------------------------------------------------------------------------------------ column sums
// Ticket words for k_col_sum's single-launch mode: all zero between launches.
__device__ unsigned g_col_sum_tickets[8192];

// part[blockIdx.y][c] = sum of x[r, c] over the block's row slice; 32 columns x 32 row lanes.
// With `tickets` (one zero word per column group) the kernel also finishes the job: the last row slice of a
// column group to arrive adds the group's partials -- in slice order, with the same grouping as
// k_reduce_partials, so the result does not depend on which block came last -- writes out[c] and leaves the
// ticket at zero for the next launch.
__global__ void __launch_bounds__(1024)
k_col_sum(const __nv_bfloat16* __restrict__ x, int M, int N, int ld, float* __restrict__ part, unsigned* tickets,
          __nv_bfloat16* __restrict__ out) {
  tb::pdl_enter();
  __shared__ float sh[32][33];
  __shared__ int is_last;
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + cx;
  const int rows_per = (M + gridDim.y - 1) / gridDim.y;
  const int r0 = blockIdx.y * rows_per, r1 = min(M, r0 + rows_per);
  float acc = 0.f;
  if (col < N)
    for (int r = r0 + ry; r < r1; r += 32) acc += __bfloat162float(x[(size_t)r * ld + col]);
  sh[ry][cx] = acc;
  __syncthreads();
  if (ry == 0 && col < N) {
    float t = 0.f;
    for (int k = 0; k < 32; ++k) t += sh[k][cx];
    part[(size_t)blockIdx.y * N + col] = t;
  }
  if (tickets == nullptr) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = atomicAdd(&tickets[blockIdx.x], 1u) == gridDim.y - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  float lane_sum = 0.f;
  if (ry < 8 && col < N)
    for (int p = ry; p < (int)gridDim.y; p += 8) lane_sum += __ldcg(part + (size_t)p * N + col);
  if (ry < 8) sh[ry][cx] = lane_sum;
  __syncthreads();
  if (ry == 0 && col < N) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += sh[k][cx];
    out[col] = __float2bfloat16_rn(t);
  }
  if (threadIdx.x == 0) tickets[blockIdx.x] = 0;
}

// The same job for matrices whose rows are 16-byte aligned (N, ld multiples of 8).  256 threads per 64 columns and row slice:
// they fetch 256 rows at a time as 16-byte vectors, all in flight together, into shared memory, and then add them up in
// eight row lanes, two columns per thread.  What bounds it is loads in flight and the chain of additions that each
// lane makes in row order: with the lanes reading global memory themselves, four vectors at a time, 8192 x 768 took 11.3 us.
// Partials over row lanes 0 .. 7 in order; the slices are grouped as in k_reduce_partials.
__global__ void __launch_bounds__(256)
k_col_sum_vec(const __nv_bfloat16* __restrict__ x, int M, int N, int ld, float* __restrict__ part, unsigned* tickets,
              __nv_bfloat16* __restrict__ out) {
  tb::pdl_enter();
  __shared__ __align__(16) uint32_t tile[256][32];  // bf16 pairs
  __shared__ float sh[8][64];
  __shared__ int is_last;
  const int rows_per = (M + gridDim.y - 1) / gridDim.y;
  const int r0 = blockIdx.y * rows_per, r1 = min(M, r0 + rows_per);
  const int vec = threadIdx.x & 7, first = threadIdx.x >> 3;  // fetching: 8 vectors x 32 rows
  const int cp = threadIdx.x & 31, lane = threadIdx.x >> 5;    // adding: 32 column pairs x 8 row lanes
  const bool inside = blockIdx.x * 64 + vec * 8 < N;
  const __nv_bfloat16* src = x + blockIdx.x * 64 + vec * 8;
  float acc0 = 0.f, acc1 = 0.f;
  for (int base = r0; base < r1; base += 256) {
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (inside && base + first + 32 * u < r1) v[u] = *reinterpret_cast<const uint4*>(src + (size_t)(base + first + 32 * u) * ld);
    if (base > r0) __syncthreads();  // the previous rows have been added
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (inside && base + first + 32 * u < r1) *reinterpret_cast<uint4*>(&tile[first + 32 * u][vec * 4]) = v[u];
    __syncthreads();
    const int rows = min(256, r1 - base);
    if (blockIdx.x * 64 + 2 * cp < N) {
#pragma unroll 8
      for (int r = lane; r < rows; r += 8) {
        const uint32_t w = tile[r][cp];
        acc0 += __uint_as_float(w << 16);
        acc1 += __uint_as_float(w & 0xffff0000u);
      }
    }
  }
  sh[lane][2 * cp] = acc0;
  sh[lane][2 * cp + 1] = acc1;
  __syncthreads();
  const int c = blockIdx.x * 64 + threadIdx.x;
  const bool mine = threadIdx.x < 64 && c < N;
  if (mine) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += sh[k][threadIdx.x];
    part[(size_t)blockIdx.y * N + c] = t;
  }
  if (tickets == nullptr) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = atomicAdd(&tickets[blockIdx.x], 1u) == gridDim.y - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // eight lanes of every-eighth slice, combined in lane order: the grouping of k_reduce_partials
  const int lx = threadIdx.x & 63;
  for (int k = threadIdx.x >> 6; k < 8; k += 4) {
    float t = 0.f;
    if (blockIdx.x * 64 + lx < N)
      for (int p = k; p < (int)gridDim.y; p += 8) t += __ldcg(part + (size_t)p * N + blockIdx.x * 64 + lx);
    sh[k][lx] = t;
  }
  __syncthreads();
  if (mine) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += sh[k][threadIdx.x];
    out[c] = __float2bfloat16_rn(t);
  }
  if (threadIdx.x == 0) tickets[blockIdx.x] = 0;
}

// The same sums with 256 columns per block: 32 column vectors x 8 row lanes, each lane reading four rows at a time by itself.
// Fewer and longer blocks, whose reads of a row are 512 bytes long: for wide matrices (tb_col_sum).
__global__ void __launch_bounds__(256)
k_col_sum_wide(const __nv_bfloat16* __restrict__ x, int M, int N, int ld, float* __restrict__ part, unsigned* tickets,
              __nv_bfloat16* __restrict__ out) {
  tb::pdl_enter();
  __shared__ float sh[8][256 + 8];
  __shared__ int is_last;
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int col = blockIdx.x * 256 + cx * 8;
  const int rows_per = (M + gridDim.y - 1) / gridDim.y;
  const int r0 = blockIdx.y * rows_per, r1 = min(M, r0 + rows_per);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < N) {
    int r = r0 + ry;
    for (; r + 24 < r1; r += 32) {
      float v[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) load8(x + (size_t)(r + 8 * u) * ld + col, v[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += v[u][e];
    }
    for (; r < r1; r += 8) {
      float v[8];
      load8(x + (size_t)r * ld + col, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += v[e];
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) sh[ry][cx * 8 + e] = acc[e];
  __syncthreads();
  {
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c < N) {
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) t += sh[k][threadIdx.x];
      part[(size_t)blockIdx.y * N + c] = t;
    }
  }
  if (tickets == nullptr) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = atomicAdd(&tickets[blockIdx.x], 1u) == gridDim.y - 1;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  {
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c < N) {
      // eight lanes of every-eighth slice, combined in lane order: the grouping of k_reduce_partials
      float lanes[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int p = 0; p < (int)gridDim.y; ++p) lanes[p & 7] += __ldcg(part + (size_t)p * N + c);
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) t += lanes[k];
      out[c] = __float2bfloat16_rn(t);
    }
  }
  if (threadIdx.x == 0) tickets[blockIdx.x] = 0;
}

// ------------------------------------------------------------------------------------ cross-entropy
// One block per row.  Forward: lse[row] and loss[row] = lse - logit[target].
__global__ void __launch_bounds__(256)
k_xent_fwd(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ lse_out,
           float* __restrict__ loss_out, int V, int ld) {
  tb::pdl_enter();
  __shared__ float red[8];
  const int row = blockIdx.x;
  const __nv_bfloat16* z = logits + (size_t)row * ld;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  // Both passes keep eight loads in flight per thread: at a 50304-wide vocabulary one load at a time ran at a tenth of the
  // memory rate (4096 rows: 666 us).  The order of the sum is one column per thread and step.
  float m = -INFINITY;
  {
    int i = threadIdx.x;
    const int vectors = ((uintptr_t)z & 15) == 0 ? V / 8 : 0;  // 16-byte loads where the row allows
    int v = threadIdx.x;
    for (; v < vectors; v += 4 * blockDim.x) {
      uint4 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (v + u * (int)blockDim.x < vectors) x[u] = *reinterpret_cast<const uint4*>(z + 8 * (v + u * blockDim.x));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (v + u * (int)blockDim.x < vectors) {
          float f[8];
          unpack8(x[u], f);
#pragma unroll
          for (int e = 0; e < 8; ++e) m = fmaxf(m, f[e]);
        }
      }
    }
    for (i += 8 * vectors; i < V; i += blockDim.x) m = fmaxf(m, __bfloat162float(z[i]));
  }
  m = warp_max(m);
  if (lane == 0) red[warp] = m;
  __syncthreads();
  m = red[0];
  for (int k = 1; k < warps; ++k) m = fmaxf(m, red[k]);
  __syncthreads();
  float s = 0.f;
  {
    int i = threadIdx.x;
    for (; i + 7 * (int)blockDim.x < V; i += 8 * blockDim.x) {
      __nv_bfloat16 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = z[i + u * blockDim.x];
#pragma unroll
      for (int u = 0; u < 8; ++u) s += __expf(__bfloat162float(x[u]) - m);
    }
    for (; i < V; i += blockDim.x) s += __expf(__bfloat162float(z[i]) - m);
  }
  s = warp_sum(s);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int k = 0; k < warps; ++k) t += red[k];
    const float lse = m + logf(t);
    lse_out[row] = lse;
    loss_out[row] = lse - __bfloat162float(z[targets[row]]);
  }
}

// Backward, in place: logits[row, i] <- (softmax_i - [i == target]) * scale.  Columns [V, width) <- 0
// (row padding, when the caller owns it).
__global__ void __launch_bounds__(256)
k_xent_bwd(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, const float* __restrict__ lse,
           const float* __restrict__ grad_scale, float inv_rows, int V, int ld, int width) {
  tb::pdl_enter();
  const int row = blockIdx.x;
  __nv_bfloat16* z = logits + (size_t)row * ld;
  const float l = lse[row];
  const float scale = grad_scale[0] * inv_rows;
  const int t = (int)targets[row];
  for (int i = threadIdx.x; i < width; i += blockDim.x) {
    float g = 0.f;
    if (i < V) g = (__expf(__bfloat162float(z[i]) - l) - (i == t ? 1.f : 0.f)) * scale;
    z[i] = __float2bfloat16_rn(g);
  }
}

// The same for rows that start on 16-byte boundaries and are long enough for at least half of the threads to have a vector: 16-byte
// vectors, four in flight per thread.  4096 x 50304 in 152 us, 431 by elements; 4096 x 512 in 6.7, 7.6; but 4096 x 256 in 6.5, 5.3.
// A kernel of its own: its registers would cost the loop above, which lives on resident warps, a third of its speed (16384 x 1003:
// 58 us, 43 by itself).
__global__ void __launch_bounds__(256)
k_xent_bwd_vec(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, const float* __restrict__ lse,
               const float* __restrict__ grad_scale, float inv_rows, int V, int ld, int width) {
  tb::pdl_enter();
  const int row = blockIdx.x;
  __nv_bfloat16* z = logits + (size_t)row * ld;
  const float l = lse[row];
  const float scale = grad_scale[0] * inv_rows;
  const int t = (int)targets[row];
  auto grad = [&](float x, int i) { return i < V ? (__expf(x - l) - (i == t ? 1.f : 0.f)) * scale : 0.f; };
  const int vectors = width / 8;
  for (int v = threadIdx.x; v < vectors; v += 4 * blockDim.x) {
    uint4 x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v + u * (int)blockDim.x < vectors) x[u] = *reinterpret_cast<const uint4*>(z + 8 * (v + u * blockDim.x));
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int at = 8 * (v + u * blockDim.x);
      if (v + u * (int)blockDim.x < vectors) {
        float f[8];
        unpack8(x[u], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = grad(f[e], at + e);
        store8(z + at, f);
      }
    }
  }
  const int i = 8 * vectors + threadIdx.x;
  if (i < width) z[i] = __float2bfloat16_rn(grad(__bfloat162float(z[i]), i));
}

// loss = mean(per_row) in a fixed order (one block).
__global__ void __launch_bounds__(1024) k_mean(const float* __restrict__ v, int n, float* __restrict__ out) {
  tb::pdl_enter();
  __shared__ float red[32];
  float acc = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += v[i];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    t = warp_sum(t);
    if (threadIdx.x == 0) out[0] = t / n;
  }
}

// ------------------------------------------------------------------------------------ embedding
__global__ void __launch_bounds__(256)
k_embed_fwd(const long long* __restrict__ idx, const __nv_bfloat16* __restrict__ tok, const __nv_bfloat16* __restrict__ pos,
            __nv_bfloat16* __restrict__ out, int rows, int T, int D) {
  tb::pdl_enter();
  const int nvec = D >> 3;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)rows * nvec; i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(i / nvec), v = (int)(i % nvec);
    float a[8], b[8];
    load8(tok + (size_t)idx[row] * D + v * 8, a);
    load8(pos + (size_t)(row % T) * D + v * 8, b);
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] += b[e];
    store8(out + (size_t)row * D + v * 8, a);
  }
}

// dtok32[idx[row]] += dy[row] (fp32 atomics, four columns each); dpos[t] = sum over batch of dy[b, t] (fixed order).
__device__ __forceinline__ void add4(float* p, float a, float b, float c, float d) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

__global__ void __launch_bounds__(256)
k_embed_bwd_tok(const long long* __restrict__ idx, const __nv_bfloat16* __restrict__ dy, float* __restrict__ dtok32, int rows, int D) {
  tb::pdl_enter();
  const int nvec = D >> 3;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < (long long)rows * nvec; i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(i / nvec), v = (int)(i % nvec);
    float f[8];
    load8(dy + (size_t)row * D + v * 8, f);
    float* dst = dtok32 + (size_t)idx[row] * D + v * 8;
    add4(dst, f[0], f[1], f[2], f[3]);
    add4(dst + 4, f[4], f[5], f[6], f[7]);
  }
}

__global__ void __launch_bounds__(256)
k_embed_bwd_pos(const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dpos, int B, int T, int D) {
  tb::pdl_enter();
  const long long vectors = (long long)T * D / 8;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < vectors; i += (long long)gridDim.x * blockDim.x) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int b = 0; b < B; ++b) {
      float f[8];
      load8(dy + (size_t)b * T * D + i * 8, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += f[e];
    }
    store8(dpos + i * 8, acc);
  }
}

// n is a multiple of 8 (whole embedding rows).
__global__ void __launch_bounds__(256) k_f32_to_bf16(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, long long n) {
  tb::pdl_enter();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n / 8; i += 2 * stride) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + (u >> 1) * stride < n / 8) v[u] = *reinterpret_cast<const float4*>(in + (i + (u >> 1) * stride) * 8 + 4 * (u & 1));
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float f[8] = {v[2 * u].x, v[2 * u].y, v[2 * u].z, v[2 * u].w, v[2 * u + 1].x, v[2 * u + 1].y, v[2 * u + 1].z, v[2 * u + 1].w};
      if (i + u * stride < n / 8) store8(out + (i + u * stride) * 8, f);
    }
  }
}

constexpr int DEVICES = 64, IDLE_EVENTS = 32;
std::mutex g_events_lock;
cudaEvent_t g_idle_events[DEVICES][IDLE_EVENTS];
int g_idle_count[DEVICES];
std::atomic<int> g_events_made{0};

int grid_for(long long work, int per_block, int cap) {
  long long b = (work + per_block - 1) / per_block;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

extern "C" {

// Work queued on `waiter` from here on starts after everything now queued on `signaller`.  A wait refers to the record before
// it, so an event is free again as soon as this returns: up to IDLE_EVENTS of them wait per device for the next call, on
// whatever thread, and the rest are given back.
int tb_stream_wait(cudaStream_t waiter, cudaStream_t signaller) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev >= DEVICES) return (int)cudaErrorInvalidDevice;
  cudaEvent_t event = nullptr;
  {
    std::lock_guard<std::mutex> hold(g_events_lock);
    if (g_idle_count[dev] > 0) event = g_idle_events[dev][--g_idle_count[dev]];
  }
  if (event == nullptr) {
    e = cudaEventCreateWithFlags(&event, cudaEventDisableTiming);
    if (e != cudaSuccess) return (int)e;
    ++g_events_made;
  }
  e = cudaEventRecord(event, signaller);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(waiter, event, 0);
  {
    std::lock_guard<std::mutex> hold(g_events_lock);
    if (g_idle_count[dev] < IDLE_EVENTS) {
      g_idle_events[dev][g_idle_count[dev]++] = event;
      event = nullptr;
    }
  }
  if (event != nullptr) cudaEventDestroy(event);
  return (int)e;
}

// Events that tb_stream_wait has made so far in this process.
int tb_stream_wait_events() { return g_events_made; }

int tb_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, int M, int D, float eps,
                     cudaStream_t s) {
  if (D % 8 || D > 32 * 8 * 8) return -20;
  const int blocks = (M + 7) / 8;
  tb_note_launch(1);
#define LN(V) tb::launch(k_ln_fwd<V>, dim3(blocks), dim3(256), 0, s, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)b, (__nv_bfloat16*)y, mean, rstd, M, D, eps)
  if (D <= 256 * 1) LN(1);
  else if (D <= 256 * 2) LN(2);
  else if (D <= 256 * 4) LN(4);
  else LN(8);
#undef LN
  return (int)cudaGetLastError();
}

// scratch: fp32 [blocks * 2 * D] with blocks = tb_layernorm_bwd_blocks(M).
// Few rows: one row per warp on as many SMs as it takes (at 1024 rows four rows per warp would leave 116 SMs idle);
// many rows: several rows per warp, so that the row look-ahead has something to fetch.
int tb_layernorm_bwd_blocks(int M) { return M < 8192 ? grid_for(M, 8, 296) : grid_for(M, 8 * 4, 592); }

int tb_layernorm_bwd_add(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, const void* add, void* dx,
                         void* dw, void* db, float* scratch, int M, int D, cudaStream_t s);

int tb_layernorm_bwd(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, void* dx, void* dw,
                     void* db, float* scratch, int M, int D, cudaStream_t s) {
  return tb_layernorm_bwd_add(dy, x, w, mean, rstd, nullptr, dx, dw, db, scratch, M, D, s);
}

// The same with `add` ([M, D] bf16, may be null; may alias dx) summed into dx.
int tb_layernorm_bwd_add(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, const void* add, void* dx,
                         void* dw, void* db, float* scratch, int M, int D, cudaStream_t s) {
  if (D % 8 || D > 32 * 8 * 8) return -20;
  const int blocks = tb_layernorm_bwd_blocks(M);
  const size_t smem = (size_t)8 * 2 * D * sizeof(float);
  tb_note_launch(2);
#define LN(V)                                                                                                          \
  do {                                                                                                                 \
    if (smem > 48 * 1024) cudaFuncSetAttribute(k_ln_bwd<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    tb::launch(k_ln_bwd<V>, dim3(blocks), dim3(256), smem, s, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,          \
               (const __nv_bfloat16*)w, mean, rstd, (const __nv_bfloat16*)add, (__nv_bfloat16*)dx, scratch, M, D);          \
  } while (0)
  if (D <= 256 * 1) LN(1);
  else if (D <= 256 * 2) LN(2);
  else if (D <= 256 * 3) LN(3);
  else if (D <= 256 * 4) LN(4);
  else LN(8);
#undef LN
  tb::launch(k_reduce_partials, dim3((2 * D + 31) / 32), dim3(256), 0, s, (const float*)scratch, blocks, 2 * D, (__nv_bfloat16*)dw, (__nv_bfloat16*)db, D);
  return (int)cudaGetLastError();
}

// out[c] = sum_r x[r, c]; scratch: fp32 [32 * N].
int tb_col_sum(const void* x, int M, int N, int ld, void* out_bf16, float* scratch, cudaStream_t s) {
  const int slices = M >= 2048 ? 32 : (M >= 256 ? 8 : 1);
  const bool vectors = (N & 7) == 0 && (ld & 7) == 0 && ((uintptr_t)x & 15) == 0;
  // Wide matrices with few rows per slice take the kernel of 256 columns per block: the other one has four times as many
  // blocks, more than the 592 that fit at a time, and little to fetch in each.  Measured (us, 256 / 64 columns): 2048 x 2304
  // 11.1 / 10.3, x 3072 11.1 / 12.4, x 50304 52 / 126; 4096 x 3072 14.2 / 13.6, x 4096 15.3 / 16.2, x 8192 23.9 / 27.1;
  // 1024 x 4096 7.7 / 7.2, x 6144 8.5 / 9.3; 1536 x 6144 10.5 / 10.3, x 8192 10.9 / 11.4; 100 x 8192 5.9 / 4.5, 64 x 50304
  // 5.8 / 9.2; from 256 rows per slice on within 8 % of one another up to 16384 columns, 16384 x 50304 258 / 279.
  const int rows_per = (M + slices - 1) / slices;
  int wide_from = 16385;
  if (slices == 1 && rows_per <= 64) wide_from = 8192;
  if (slices == 8) wide_from = rows_per < 192 ? 5120 : 8192;
  if (slices == 32 && rows_per <= 192) wide_from = rows_per < 128 ? 3072 : 4096;
  const bool wide = vectors && N >= wide_from;
  dim3 grid(wide ? (N + 255) / 256 : vectors ? (N + 63) / 64 : (N + 31) / 32, slices);
  // One launch: each column group's last block finishes the sum.  The ticket words come from a fixed pool handed
  // out round-robin, so launches in flight at the same time never share one (a pool's worth of launches would
  // have to overlap); matrices wider than the pool take the two-kernel path.
  constexpr int POOL = 8192;
  static unsigned* pool = nullptr;
  static int pool_device = -1, next = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (pool == nullptr || pool_device != dev) {
    if (cudaGetSymbolAddress((void**)&pool, g_col_sum_tickets) != cudaSuccess) return (int)cudaGetLastError();
    pool_device = dev;
  }
  if ((int)grid.x <= POOL) {
    if (next + (int)grid.x > POOL) next = 0;
    unsigned* tickets = pool + next;
    next += grid.x;
    tb_note_launch(1);
    if (wide)
      tb::launch(k_col_sum_wide, grid, dim3(256), 0, s, (const __nv_bfloat16*)x, M, N, ld, scratch, tickets, (__nv_bfloat16*)out_bf16);
    else if (vectors)
      tb::launch(k_col_sum_vec, grid, dim3(256), 0, s, (const __nv_bfloat16*)x, M, N, ld, scratch, tickets, (__nv_bfloat16*)out_bf16);
    else
      tb::launch(k_col_sum, grid, dim3(1024), 0, s, (const __nv_bfloat16*)x, M, N, ld, scratch, tickets, (__nv_bfloat16*)out_bf16);
    return (int)cudaGetLastError();
  }
  grid = dim3((N + 31) / 32, slices);
  tb_note_launch(2);
  tb::launch(k_col_sum, grid, dim3(1024), 0, s, (const __nv_bfloat16*)x, M, N, ld, scratch, (unsigned*)nullptr, (__nv_bfloat16*)nullptr);
  tb::launch(k_reduce_partials, dim3((N + 31) / 32), dim3(256), 0, s, (const float*)scratch, slices, N, (__nv_bfloat16*)out_bf16,
             (__nv_bfloat16*)nullptr, N);
  return (int)cudaGetLastError();
}

int tb_xent_fwd(const void* logits, const long long* targets, float* lse, float* row_loss, float* loss, int rows, int V, int ld,
                cudaStream_t s) {
  const int threads = V <= 128 ? 32 : (V <= 2048 ? 128 : 256);
  tb_note_launch(2);
  tb::launch(k_xent_fwd, dim3(rows), dim3(threads), 0, s, (const __nv_bfloat16*)logits, targets, lse, row_loss, V, ld);
  tb::launch(k_mean, dim3(1), dim3(1024), 0, s, (const float*)row_loss, rows, loss);
  return (int)cudaGetLastError();
}

int tb_xent_bwd(void* logits, const long long* targets, const float* lse, const float* grad_scale, int rows, int V, int ld,
                int width, cudaStream_t s) {
  const int threads = ld <= 128 ? 32 : (ld <= 2048 ? 128 : 256);
  tb_note_launch(1);
  const bool vectors = (ld & 7) == 0 && ((uintptr_t)logits & 15) == 0 && width / 8 >= threads / 2;
  tb::launch(vectors ? k_xent_bwd_vec : k_xent_bwd, dim3(rows), dim3(threads), 0, s, (__nv_bfloat16*)logits, targets, lse, grad_scale, 1.f / rows, V, ld, width);
  return (int)cudaGetLastError();
}

int tb_embed_fwd(const long long* idx, const void* tok, const void* pos, void* out, int rows, int T, int D, cudaStream_t s) {
  if (D % 8) return -20;
  tb_note_launch(1);
  tb::launch(k_embed_fwd, dim3(grid_for((long long)rows * (D / 8), 256, 148 * 8)), dim3(256), 0, s, idx, (const __nv_bfloat16*)tok,
             (const __nv_bfloat16*)pos, (__nv_bfloat16*)out, rows, T, D);
  return (int)cudaGetLastError();
}

// dtok32: zeroed fp32 [V, D] scratch; dtok / dpos: bf16 outputs.
int tb_embed_bwd(const long long* idx, const void* dy, float* dtok32, void* dtok, void* dpos, int B, int T, int D, int V,
                 cudaStream_t s) {
  if (D % 8) return -20;
  tb_note_launch(3);
  tb::launch(k_embed_bwd_tok, dim3(grid_for((long long)B * T * (D / 8), 256, 148 * 8)), dim3(256), 0, s, idx, (const __nv_bfloat16*)dy, dtok32, B * T, D);
  tb::launch(k_f32_to_bf16, dim3(grid_for((long long)V * D / 8, 256, 148 * 8)), dim3(256), 0, s, (const float*)dtok32, (__nv_bfloat16*)dtok, (long long)V * D);
  tb::launch(k_embed_bwd_pos, dim3(grid_for((long long)T * D / 8, 256, 148 * 8)), dim3(256), 0, s, (const __nv_bfloat16*)dy, (__nv_bfloat16*)dpos, B, T, D);
  return (int)cudaGetLastError();
}

}  // extern "C"

// ------------------------------------------------------------------------------------ no-allocation variant
// See noalloc.h.  The scratch lives in this file so that both host and device code here can
// name it; host code must not pass the name itself to a kernel (on the host it is only a
// stand-in for the symbol), so the device address is looked up once per device.
static __device__ __align__(256) float g_colsum_scratch[32 * TB_COLSUM_NOALLOC_MAX_N];
static float* g_colsum_scratch_addr[64] = {nullptr};
static char g_noalloc_error[160] = "";

extern "C" const char* tb_noalloc_last_error() { return g_noalloc_error; }

extern "C" int tb_col_sum_noalloc(const void* x_bf16, int M, int N, int ld, void* out_bf16, cudaStream_t stream) {
  if (N <= 0) return 0;
  if (M <= 0) return (int)cudaMemsetAsync(out_bf16, 0, (size_t)N * sizeof(__nv_bfloat16), stream);  // the sum over no rows
  if (N > TB_COLSUM_NOALLOC_MAX_N) {
    snprintf(g_noalloc_error, sizeof(g_noalloc_error), "tb_col_sum_noalloc: N = %d exceeds the built-in scratch (max %d columns)",
             N, TB_COLSUM_NOALLOC_MAX_N);
    return TB_NOALLOC_TOO_WIDE;
  }
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    snprintf(g_noalloc_error, sizeof(g_noalloc_error), "tb_col_sum_noalloc: no usable current device");
    return TB_NOALLOC_SETUP_FAILED;
  }
  if (g_colsum_scratch_addr[dev] == nullptr) {  // first call on this device: resolve the symbol here, with it current
    float* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&p, g_colsum_scratch);
    if (e != cudaSuccess || p == nullptr) {
      snprintf(g_noalloc_error, sizeof(g_noalloc_error), "tb_col_sum_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return TB_NOALLOC_SETUP_FAILED;
    }
    g_colsum_scratch_addr[dev] = p;
  }
  float* scratch = g_colsum_scratch_addr[dev];
  const int slices = M >= 2048 ? 32 : (M >= 256 ? 8 : 1);
  dim3 grid((N + 31) / 32, slices);
  tb_note_launch(2);
  k_col_sum<<<grid, 1024, 0, stream>>>((const __nv_bfloat16*)x_bf16, M, N, ld, scratch, nullptr, nullptr);
  k_reduce_partials<<<(N + 31) / 32, 256, 0, stream>>>(scratch, slices, N, (__nv_bfloat16*)out_bf16, nullptr, N);
  return (int)cudaGetLastError();
}
