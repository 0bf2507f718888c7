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

#include "f32x2.cuh"
#include "host_state.h"
#include "launch.cuh"
#include "noalloc.h"
#include "operators.h"

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

__device__ __forceinline__ void named_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void named_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// ------------------------------------------------------------------------------------ LayerNorm
// One warp per row; D is a multiple of 8.  MAXV 16-byte vectors per lane cover D <= 32*8*MAXV.  It is bound by the rows on their
// way to an SM, so a row waits for its reductions as it came, in bf16 pairs (unpacked, 2048 columns took 64 registers a lane
// and left 16 warps on an SM: 16384 x 2048 in 34.9 us, now 25.1, 21 at the copy rate).  EARLY also fetches the gain and bias before the
// reductions, for another 8 * MAXV registers: where all rows are resident at once even so (tb_layernorm_fwd), a trip to L2 is
// what counts (2048 x 2048: 5.3 us, 7.4 without), elsewhere the resident warps (16384 x 1024: 13.9 us without, 15.0 with).
template <int MAXV, bool EARLY>
__global__ void __launch_bounds__(256, EARLY && MAXV == 4 ? 4 : 1)
k_ln_fwd(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
         __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, int M, int D, float eps) {
  tb::pdl_enter();
  using namespace tc;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= M) return;
  const int nvec = D >> 3;
  uint4 v[MAXV];
#pragma unroll
  for (int j = 0; j < MAXV; ++j)
    if (lane + 32 * j < nvec) v[j] = *reinterpret_cast<const uint4*>(x + (size_t)row * D + (lane + 32 * j) * 8);
  uint4 wv[MAXV], bv[MAXV];
  auto gains = [&](int j) {
    if (lane + 32 * j < nvec) {
      wv[j] = __ldg(reinterpret_cast<const uint4*>(w + (lane + 32 * j) * 8));
      bv[j] = __ldg(reinterpret_cast<const uint4*>(b + (lane + 32 * j) * 8));
    }
  };
  if (EARLY) {
#pragma unroll
    for (int j = 0; j < MAXV; ++j) gains(j);
  }
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    if (lane + 32 * j < nvec) {
      const uint32_t xp[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        sum += __uint_as_float(xp[p] << 16);
        sum += __uint_as_float(xp[p] & 0xffff0000u);
      }
    }
  }
  const float mean = warp_sum(sum) / D;
  const f32x2 minus_mean2 = pair2(-mean, -mean);
  float sq = 0.f;
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    if (lane + 32 * j < nvec) {
      const uint32_t xp[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        float d0, d1;
        split2(add2(from_bf16_pair(xp[p]), minus_mean2), &d0, &d1);
        sq = fmaf(d0, d0, sq);
        sq = fmaf(d1, d1, sq);
      }
    }
  }
  const float rstd = rsqrtf(warp_sum(sq) / D + eps);
  if (lane == 0) {
    mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
  const f32x2 rstd2 = pair2(rstd, rstd);
#pragma unroll
  for (int j = 0; j < MAXV; ++j) {
    const int vi = lane + 32 * j;
    if (vi < nvec) {
      if (!EARLY) gains(j);
      const uint32_t xp[4] = {v[j].x, v[j].y, v[j].z, v[j].w}, wp[4] = {wv[j].x, wv[j].y, wv[j].z, wv[j].w},
                     bp[4] = {bv[j].x, bv[j].y, bv[j].z, bv[j].w};
      uint32_t o[4];
#pragma unroll
      for (int p = 0; p < 4; ++p)
        o[p] = bf16_pair(fma2(mul2(add2(from_bf16_pair(xp[p]), minus_mean2), rstd2), from_bf16_pair(wp[p]), from_bf16_pair(bp[p])));
      *reinterpret_cast<uint4*>(y + (size_t)row * D + vi * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// dx for each row, and partial sums of dw = sum dy*xhat and db = sum dy into part[slice][2][D] (fp32).  A second
// kernel adds the partials in a fixed order.  Rows are dealt to the `slices` eight at a time, round-robin; within a slice
// warp w sums row w of every eight in order, and the eight warps' sums are added in order, whatever the grid.
// add (optional): a second gradient of the same input, summed into dx in fp32 before the one rounding
// -- the residual branch's gradient in a pre-LayerNorm block, which autograd would otherwise add with a
// separate pass over the activations.  It may alias dx: a row's dx is written only after its `add` has been read.
//
// What bounds it is bytes on the way to an SM.  dw and db of a warp's columns take 16 * MAXV registers, which leaves none for
// rows that have not arrived yet.  So rows travel by cp.async into a ring of `stages` rows per warp in shared memory; each
// lane fetches the vectors that it alone reads, so the ring needs no barrier.  With the next row held in registers, and
// spills, 4096 x 1024 took 17.7 us, now 9.1 (5.1 at the copy rate); 8192 x 768 14.2, now 10.2 (7.7); 16384 x 2048 88, now 50 (41);
// 1024 x 768 5.2, now 3.8.
// A block with one slice adds its warps' sums side by side, in the shared memory of the ring.  A block with several keeps the ring
// busy: the sums meet in one [2][D] array, warp after warp (each adds its own and hands the array on through a named
// barrier), so that the first warps are on their next rows while the last ones add.
template <int MAXV>
struct LnBwd {
  static constexpr int STAGES = MAXV <= 2 ? 4 : 2;
  static constexpr int VEC_ROW = 32 * MAXV;  // 16-byte vectors of a row, padded to whole warps
  static constexpr int SUMS = 2 * 2 * VEC_ROW * 16;  // the array: fp32 dw and db
  static constexpr int STATS = 8 * STAGES * 2 * 4;   // mean and 1/std of every row in the ring
  static int smem(int stages, bool add, bool one_slice) {
    const int ring = SUMS + STATS + 8 * stages * (add ? 3 : 2) * VEC_ROW * 16;
    return one_slice && ring < 8 * SUMS ? 8 * SUMS : ring;
  }
};

template <int MAXV, bool ADD>
__global__ void __launch_bounds__(256, MAXV <= 4 ? 2 : 1)
k_ln_bwd(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
         const float* __restrict__ mean_in, const float* __restrict__ rstd_in, const __nv_bfloat16* add,
         __nv_bfloat16* dx, float* __restrict__ part, int M, int D, int slices, int stages) {
  tb::pdl_enter();
  using namespace tc;
  using L = LnBwd<MAXV>;
  extern __shared__ __align__(16) uint8_t ln_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = D >> 3;
  float4* sums = reinterpret_cast<float4*>(ln_smem);  // [dw, db][MAXV][two halves of a lane's vector][32 lanes]
  float* stats = reinterpret_cast<float*>(ln_smem + L::SUMS) + warp * L::STAGES * 2;
  constexpr int TENSORS = ADD ? 3 : 2;
  uint4* ring = reinterpret_cast<uint4*>(ln_smem + L::SUMS + L::STATS) + (size_t)warp * stages * TENSORS * L::VEC_ROW + lane;

  uint4 wv[MAXV];
  f32x2 dw[MAXV][4], db[MAXV][4];
#pragma unroll
  for (int j = 0; j < MAXV; ++j)
    if (lane + 32 * j < nvec) wv[j] = *reinterpret_cast<const uint4*>(w + (lane + 32 * j) * 8);

  // the warp's rows in the order in which it works on them: (slice, turn) -> row
  auto row_of = [&](int slice, int turn) { return (slice + turn * slices) * 8 + warp; };
  int f_slice = blockIdx.x, f_turn = 0, f_stage = 0;  // the next row to fetch
  auto fetch = [&]() {
    const int row = row_of(f_slice, f_turn);
    if (f_slice < slices && row < M) {
      uint4* slot = ring + (size_t)f_stage * TENSORS * L::VEC_ROW;
#pragma unroll
      for (int j = 0; j < MAXV; ++j) {
        const int vi = lane + 32 * j;
        if (vi < nvec) {
          const size_t at = (size_t)row * D + vi * 8;
          cp_async16(slot + 32 * j, dy + at);
          cp_async16(slot + L::VEC_ROW + 32 * j, x + at);
          if (ADD) cp_async16(slot + 2 * L::VEC_ROW + 32 * j, add + at);
        }
      }
      if (lane < 2) cp_async4(stats + 2 * f_stage + lane, (lane == 0 ? mean_in : rstd_in) + row);
      if (++f_stage == stages) f_stage = 0;
      ++f_turn;
      if (row_of(f_slice, f_turn) >= M) f_turn = 0, f_slice += gridDim.x;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int stage = 0;
  for (int i = 0; i < stages - 1; ++i) fetch();

  for (int slice = blockIdx.x; slice < slices; slice += gridDim.x) {
#pragma unroll
    for (int j = 0; j < MAXV; ++j)
#pragma unroll
      for (int p = 0; p < 4; ++p) dw[j][p] = db[j][p] = pair2(0.f, 0.f);
    for (int turn = 0, row; (row = row_of(slice, turn)) < M; ++turn) {
      __syncwarp();  // the slot that is filled next has been read by every lane
      fetch();
      if (stages == 1) asm volatile("cp.async.wait_group 0;" ::: "memory");
      else if (stages == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else if (stages == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
      else asm volatile("cp.async.wait_group 3;" ::: "memory");
      __syncwarp();
      const uint4* slot = ring + (size_t)stage * TENSORS * L::VEC_ROW;
      const float mean = stats[2 * stage], rstd = stats[2 * stage + 1];
      if (++stage == stages) stage = 0;
      const f32x2 minus_mean2 = pair2(-mean, -mean), rstd2 = pair2(rstd, rstd);
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int j = 0; j < MAXV; ++j) {
        if (lane + 32 * j < nvec) {
          const uint4 a = slot[32 * j], b = slot[L::VEC_ROW + 32 * j];
          const uint32_t dyp[4] = {a.x, a.y, a.z, a.w}, xp[4] = {b.x, b.y, b.z, b.w}, wp[4] = {wv[j].x, wv[j].y, wv[j].z, wv[j].w};
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const f32x2 dy2 = from_bf16_pair(dyp[p]);
            const f32x2 xh2 = mul2(add2(from_bf16_pair(xp[p]), minus_mean2), rstd2);
            const f32x2 g2 = mul2(dy2, from_bf16_pair(wp[p]));
            float h0, h1, g0, g1;
            split2(xh2, &h0, &h1);
            split2(g2, &g0, &g1);
            s1 += g0;
            s2 = fmaf(g0, h0, s2);
            s1 += g1;
            s2 = fmaf(g1, h1, s2);
            dw[j][p] = fma2(dy2, xh2, dw[j][p]);
            db[j][p] = add2(db[j][p], dy2);
          }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {  // warp_sum of both, side by side
        const float t1 = __shfl_xor_sync(0xffffffffu, s1, o), t2 = __shfl_xor_sync(0xffffffffu, s2, o);
        s1 += t1;
        s2 += t2;
      }
      s1 /= D;
      s2 /= D;
      const f32x2 minus_s1 = pair2(-s1, -s1), minus_s2 = pair2(-s2, -s2);
#pragma unroll
      for (int j = 0; j < MAXV; ++j) {
        const int vi = lane + 32 * j;
        if (vi < nvec) {
          const uint4 a = slot[32 * j], b = slot[L::VEC_ROW + 32 * j];
          const uint4 c = ADD ? slot[2 * L::VEC_ROW + 32 * j] : make_uint4(0, 0, 0, 0);
          const uint32_t dyp[4] = {a.x, a.y, a.z, a.w}, xp[4] = {b.x, b.y, b.z, b.w}, wp[4] = {wv[j].x, wv[j].y, wv[j].z, wv[j].w},
                         ap[4] = {c.x, c.y, c.z, c.w};
          uint32_t o[4];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const f32x2 xh2 = mul2(add2(from_bf16_pair(xp[p]), minus_mean2), rstd2);  // the same operations as above: the same values
            f32x2 t = fma2(xh2, minus_s2, fma2(from_bf16_pair(dyp[p]), from_bf16_pair(wp[p]), minus_s1));
            t = mul2(rstd2, t);
            float o0, o1;
            split2(t, &o0, &o1);
            if (ADD) {  // scalar: the assembler would make one fma of a packed product and sum, and round once less
              o0 = __fadd_rn(o0, __uint_as_float(ap[p] << 16));
              o1 = __fadd_rn(o1, __uint_as_float(ap[p] & 0xffff0000u));
            }
            o[p] = bf16_pair(pair2(o0, o1));
          }
          *reinterpret_cast<uint4*>(dx + (size_t)row * D + vi * 8) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
    }
    float* out = part + (size_t)slice * 2 * D;
    // value q of vector j: dw's or db's (q >> 1) columns 4 * (q & 1) .. + 3 of the lane's eight
    auto mine = [&](int j, int q) {
      float4 t;
      const f32x2* v = (q < 2 ? dw[j] : db[j]) + 2 * (q & 1);
      split2(v[0], &t.x, &t.y);
      split2(v[1], &t.z, &t.w);
      return t;
    };
    auto place = [&](int j, int q, int l) { return ((q >> 1) * MAXV + j) * 64 + (q & 1) * 32 + l; };
    if (gridDim.x == slices) {  // the block's only slice: the ring is free, and all columns are added side by side
      __syncthreads();
      float4* all = sums + warp * 128 * MAXV;
#pragma unroll
      for (int j = 0; j < MAXV; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) all[place(j, q, lane)] = mine(j, q);
      __syncthreads();
      for (int i = threadIdx.x; i < 128 * MAXV; i += 256) {
        const int q = (i >> 5) & 1, j = (i >> 6) % MAXV, half = (i >> 6) / MAXV, vi = (i & 31) + 32 * j;
        if (vi >= nvec) continue;
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float4 v = sums[k * 128 * MAXV + i];
          t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
        }
        *reinterpret_cast<float4*>(out + half * D + vi * 8 + 4 * q) = t;
      }
      return;
    }
    // warp 0 waits until the last warp has read the previous slice's sums, every other one for the warp before it
    if (warp > 0 || slice != (int)blockIdx.x) named_sync(1 + (warp + 7) % 8, 64);
#pragma unroll
    for (int j = 0; j < MAXV; ++j) {
      const int vi = lane + 32 * j;
      if (vi < nvec) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 m = mine(j, q);
          float4 t = warp == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : sums[place(j, q, lane)];
          t.x += m.x; t.y += m.y; t.z += m.z; t.w += m.w;
          if (warp < 7) sums[place(j, q, lane)] = t;
          else *reinterpret_cast<float4*>(out + (q >> 1) * D + vi * 8 + 4 * (q & 1)) = t;
        }
      }
    }
    if (warp < 7 || slice + (int)gridDim.x < slices) named_arrive(1 + warp, 64);
  }
}

// out[c] = sum over p of part[p][c], written as bf16.  16 columns x 8 row lanes per block: each lane adds
// every 8th partial, then the 8 lanes are combined in a fixed order (deterministic).  It is bound by the loads that an SM can
// have under way, so narrow blocks on many SMs: 296 x 2048 partials 3.7 us with 32 columns, 2.65 with 16, 2.7 with 8.
constexpr int PARTIAL_COLS = 16;
__global__ void __launch_bounds__(128)
k_reduce_partials(const float* __restrict__ part, int parts, int width, __nv_bfloat16* __restrict__ out0,
                  __nv_bfloat16* __restrict__ out1, int split) {
  tb::pdl_enter();
  constexpr int COLS = PARTIAL_COLS;
  __shared__ float sh[8][COLS + 1];
  const int cx = threadIdx.x % COLS, ry = threadIdx.x / COLS;
  const int c = blockIdx.x * COLS + cx;
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
// Ticket words for k_col_sum's single-launch mode.
constexpr int TICKET_POOL = 8192;
__device__ unsigned g_col_sum_tickets[2 * TICKET_POOL];
tb::WordPool g_ticket_pool(TICKET_POOL);

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
#define LN1(V, EARLY) tb::launch(k_ln_fwd<V, EARLY>, dim3(blocks), dim3(256), 0, s, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)b, (__nv_bfloat16*)y, mean, rstd, M, D, eps)
#define LN(V)                              \
  do {                                     \
    if (blocks <= 148 * (V <= 4 ? 4 : 2)) LN1(V, true); \
    else LN1(V, false);                    \
  } while (0)
  if (D <= 256 * 1) LN(1);
  else if (D <= 256 * 2) LN(2);
  else if (D <= 256 * 3) LN(3);
  else if (D <= 256 * 4) LN(4);
  else if (D <= 256 * 6) LN(6);
  else LN(8);
#undef LN1
#undef LN
  return (int)cudaGetLastError();
}

// scratch: fp32 [slices * 2 * D] with slices = tb_layernorm_bwd_blocks(M), 16-byte aligned.
// Few rows: one row per warp on as many SMs as it takes (at 1024 rows four rows per warp would leave 116 SMs idle);
// many rows: several rows per warp, so that the row look-ahead has something to fetch.
int tb_layernorm_bwd_blocks(int M) { return M < 8192 ? grid_for(M, 8, 296) : grid_for(M, 8 * 4, 592); }

int tb_layernorm_bwd(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, void* dx, void* dw,
                     void* db, float* scratch, int M, int D, cudaStream_t s) {
  return tb_layernorm_bwd_add(dy, x, w, mean, rstd, nullptr, dx, dw, db, scratch, M, D, s);
}

// The same with `add` ([M, D] bf16, may be null; may alias dx) summed into dx.
int tb_layernorm_bwd_add(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, const void* add, void* dx,
                         void* dw, void* db, float* scratch, int M, int D, cudaStream_t s) {
  if (D % 8 || D > 32 * 8 * 8) return -20;
  // as many blocks as are resident (registers allow two on an SM up to 1024 columns); rows: the most that a warp works on
  const int slices = tb_layernorm_bwd_blocks(M), per_warp = (M + slices * 8 - 1) / (slices * 8);
  tb_note_launch(2);
#define LN1(V, ADD)                                                                                                              \
  do {                                                                                                                           \
    const int resident = 148 * (V <= 4 ? 2 : 1), grid = slices < resident ? slices : resident;                                  \
    const int rows = per_warp * ((slices + grid - 1) / grid), stages = rows < LnBwd<V>::STAGES ? rows : LnBwd<V>::STAGES;       \
    const int smem = LnBwd<V>::smem(stages, ADD, grid == slices);                                                                               \
    static tb::SharedMemoryLimit limit;                                                                                         \
    const cudaError_t allowed = limit.raise(k_ln_bwd<V, ADD>, LnBwd<V>::smem(LnBwd<V>::STAGES, ADD, true));                     \
    if (allowed != cudaSuccess) return (int)allowed;                                                                            \
    tb::launch(k_ln_bwd<V, ADD>, dim3(grid), dim3(256), (size_t)smem, s, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,     \
               (const __nv_bfloat16*)w, mean, rstd, (const __nv_bfloat16*)add, (__nv_bfloat16*)dx, scratch, M, D, slices, stages); \
  } while (0)
#define LN(V)                        \
  do {                               \
    if (add != nullptr) LN1(V, true); \
    else LN1(V, false);              \
  } while (0)
  if (D <= 256 * 1) LN(1);
  else if (D <= 256 * 2) LN(2);
  else if (D <= 256 * 3) LN(3);
  else if (D <= 256 * 4) LN(4);
  else if (D <= 256 * 6) LN(6);
  else LN(8);
#undef LN
#undef LN1
  tb::launch(k_reduce_partials, dim3((2 * D + PARTIAL_COLS - 1) / PARTIAL_COLS), dim3(8 * PARTIAL_COLS), 0, s, (const float*)scratch, slices, 2 * D, (__nv_bfloat16*)dw, (__nv_bfloat16*)db, D);
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
  // One launch: each column group's last block finishes the sum.  Matrices wider than the pool of ticket words take the
  // two-kernel path.
  if ((int)grid.x <= TICKET_POOL) {
    unsigned* tickets = nullptr;
    const cudaError_t e = g_ticket_pool.take(grid.x, s, &tickets, [](void** at) { return cudaGetSymbolAddress(at, g_col_sum_tickets); });
    if (e != cudaSuccess) return (int)e;
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
  tb::launch(k_reduce_partials, dim3((N + PARTIAL_COLS - 1) / PARTIAL_COLS), dim3(8 * PARTIAL_COLS), 0, s, (const float*)scratch, slices, N, (__nv_bfloat16*)out_bf16,
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
  k_reduce_partials<<<(N + PARTIAL_COLS - 1) / PARTIAL_COLS, 8 * PARTIAL_COLS, 0, stream>>>(scratch, slices, N, (__nv_bfloat16*)out_bf16, nullptr, N);
  return (int)cudaGetLastError();
}
