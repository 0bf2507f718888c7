// bf16 GEMM on the 5th-generation tensor cores: D[M,N] = A . B (+ epilogue), fp32 accumulation in TMEM.
//
// Two kernels share the epilogue code: k_gemm (below: one persistent CTA per SM) and k_gemm_pair (further down: CTA
// pairs driving tcgen05.mma.cta_group::2).  Neither uses TMA multicast.  Outputs in bf16 leave through TMA stores.
//
// Structure of k_gemm (one persistent CTA per SM, 320 threads, no cluster):
//   warp 0      TMA producer: cp.async.bulk.tensor.2d loads A and B tiles (128B swizzle) into a
//               3- to 6-stage shared-memory ring, signalling `full[s]` by transaction bytes.
//   warp 1      MMA issuer: one elected lane issues tcgen05.mma.cta_group::1.kind::f16
//               (128 x BN x 16 per instruction, 4 per stage), releases stages with
//               tcgen05.commit -> `empty[s]`, and hands a finished accumulator to the epilogue
//               with tcgen05.commit -> `acc_full[b]`.  TMEM holds two accumulators (2 x BN
//               columns), so the next tile's MMAs overlap this tile's epilogue.
//   warps 2-9   epilogue: tcgen05.ld 32 lanes x 32 columns at a time, then bias / GELU / residual /
//               dGELU / accumulate in registers; a bf16 block is staged in shared memory (64-byte
//               swizzle) and written by one cp.async.bulk.tensor store, fp32 outputs by 16-byte stores.
// Tile shapes: 256x256, 128x256, 128x192, 128x128 and pair 256x256, 256x128 (plan_gemm); split-K of the last round.
//
// Operand layouts.  Each operand is either K-major (the reduction dimension is contiguous in
// global memory) or MN-major (the other dimension is).  That covers all three GEMMs of a linear
// layer without transposing anything in memory:
//   forward   Y[M,N]  = X[M,K] . W[N,K]^T          A K-major,  B K-major
//   dX        dX[M,K] = dY[M,N] . W[N,K]            A K-major,  B MN-major   (reduction over N)
//   dW        dW[N,K] = dY[M,N]^T . X[M,K]          A MN-major, B MN-major   (reduction over M)
// MN-major tiles are loaded as 64-element-wide (128-byte) column strips so the same 128B
// swizzle applies; the shared-memory descriptors carry the strip stride (LBO) and the 8-row
// group stride (SBO).
//
// Every mbarrier wait is bounded; a wait that runs out sets a host-visible error word and the CTA
// winds down (frees its TMEM, returns).  The reference has no GEMM of its own: its Linear layers
// call cuBLAS through torch (tandem/model.py:36-37,53-54,75).
#include <atomic>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "f32x2.cuh"
#include "host_state.h"
#include "launch.cuh"
#include "operators.h"
#include "tcgen05.cuh"

namespace {

constexpr int BK = 64;
constexpr int SMEM_BUDGET = 224 * 1024;  // operand ring and staging blocks
constexpr int BLOCK_BYTES = 2048;        // a staging block: 32 rows x 32 columns of bf16 on their way in (aux_in) or out

enum EpilogueFlags {
  EPI_BIAS = 1,        // + bias[col]
  EPI_GELU = 2,        // out = gelu(v); with aux_out: also write gelu'(v) there (what backward multiplies by)
  EPI_RESIDUAL = 4,    // + aux_in[row, col]
  EPI_DGELU = 8,       // out = v * aux_in[row, col]  (aux_in = the gelu'(.) that the forward GEMM saved)
  EPI_ACCUMULATE = 16, // out += v  (gradient accumulation)
  EPI_OUT_F32 = 32,    // out is fp32 (else bf16)
};

struct GemmArgs {
  int M, N, K;
  int ldc;            // leading dimension of out / aux (elements)
  int flags;
  void* out;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* aux_in;   // residual, or the saved gelu' factors, [M, ldc]
  __nv_bfloat16* aux_out;        // gelu'(pre-activation) out for EPI_GELU, [M, ldc]
  int* error;                    // host-mapped; set to 1 when a wait runs out
  // Split-K of the last wave.  Output tiles [0, whole_tiles) -- as many full rounds of one tile per CTA as there are --
  // are computed whole.  The remaining tiles, too few to occupy the SMs, have their reduction cut into `splits`
  // parts and each (tile, part) is a work item: parts 1 .. splits-1 ("producers") park their raw fp32 accumulator
  // tile in `partials` and raise one flag per epilogue warp; part 0 ("consumer") adds the parked tiles to its own
  // accumulator, in part order, and runs the ordinary epilogue (bias, GELU, residual, TMA store ...).  Items are
  // ordered whole tiles, producers, consumers; every CTA works through its items in that order and a producer
  // never waits, so the scheme cannot deadlock whatever the grid.  One kernel, no reduction pass, and the result
  // does not depend on scheduling.
  int splits;             // 1: nothing is split
  int whole_tiles;        // tiles computed by one item each (0 when every tile is split)
  float* partials;        // [split tile][splits - 1][column quad][row][4] floats
  unsigned* split_flags;  // [split tile][splits - 1][8 epilogue warps], zero between launches (the consumer resets them)
  int group_m;            // rows of tiles per raster group (tile_coords)
  int kind;               // EpilogueKind; all but KIND_DIRECT leave through TMA stores (map_out and map_pre are valid)
};

// Output tile `tile` -> its tile row and column.  The first `whole` tiles are swept in groups of `group_m` tile rows, column
// by column within a group, so that the tiles in flight at one time cover a block of the output that is roughly square and
// each operand panel is read by several of them; the tiles of an unfinished column and the split ones behind
// them come in column order.  Sweeping all of it by columns lets every tile in flight read an A panel of its own, and A,
// larger than L2 at 16384 tokens, comes from memory once per column of tiles.  Measured at 16384 x 2048 x 8192 (bf16, cold
// L2): 1245 -> 1515 TFLOP/s on 128 x 256 tiles, 1420 -> 1600 on 256 x 256 tiles; groups of 4 to 16 rows of tiles
// are within 3 % of one another.
__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int whole, int group_m, int* mi, int* ni) {
  const int columns = whole / tiles_m;
  if (tile >= columns * tiles_m) {
    *mi = tile % tiles_m;
    *ni = tile / tiles_m;
    return;
  }
  const int per_group = group_m * columns;
  const int first = tile / per_group * group_m, in = tile % per_group;
  const int size = tiles_m - first < group_m ? tiles_m - first : group_m;
  *mi = first + in % size;
  *ni = in / size;
}

// All-gather fused into the GEMM (B operand = a weight whose flat bytes are sharded over the ranks).
// Two extra warps per CTA pull the weight, chunk by chunk, from the owners' shard memory (plain 16-byte
// loads over NVLink from peer pointers) into this GPU's buffer and publish one flag per chunk; the TMA
// producer waits for the flags that cover a tile's weight panel before it loads it -- from local memory,
// never from the peer, and without multicast.  Transfer and math overlap panel by panel inside ONE
// kernel, launched cooperatively so that every CTA (hence every chunk's fetcher) is resident.
struct GatherArgs {
  const char* shard[8];   // shard[q]: rank q's shard as mapped here; its byte 0 is byte shard_lo[q] of the unit's flat buffer
  long long shard_lo[8];  // byte ranges of the shards within the unit's flat buffer
  long long shard_hi[8];
  char* full;             // this GPU's copy of the unit's flat buffer; the weight occupies [w_off, w_off + N*K*2)
  long long w_off, w_bytes;  // w_bytes: everything fetched = the weight plus tail_bytes
  long long tail_bytes;   // bytes right behind the weight that are fetched with it (the layer's bias)
  uint32_t* ready;        // one word per chunk of the weight; chunk c is complete once ready[c] == epoch
  uint32_t epoch;
  int n;                  // ranks
  int chunk_bytes;
  int n_start;            // the n-panel this rank visits first (the one its own shard feeds)
};

using namespace tc;

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_release_gpu(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Bounded wait for chunk flags [c_lo, c_hi] to reach `epoch`.
__device__ __forceinline__ bool wait_chunks(const uint32_t* ready, int c_lo, int c_hi, uint32_t epoch, int* error) {
  const long long start = clock64();
  for (int c = c_lo; c <= c_hi; ++c) {
    while (ld_acquire_gpu(ready + c) != epoch) {
      if (clock64() - start > (1ll << WAIT_LIMIT_CYCLES_SHIFT)) {
        *error = 1;
        __threadfence_system();
        return false;
      }
    }
  }
  return true;
}

// 1 / d of two values given as -d, 1 <= d: the special-function unit's approximation and one Newton step on the residual that an
// FMA leaves exact.  From an approximation within one unit in the last place that is the correctly rounded result (Markstein,
// IBM J. Res. Dev. 34, 1990), except that the theorem leaves out the significand of all ones, where the last place may be
// off by one; compared with a division over every significand, this unit's results were correct for that one too.  Above
// 1e30 it answers 1e-30, which the caller multiplies by exp(-x^2 / 2) = 0.  __frcp_rn's range checks cost a third of the GELU
// epilogue.
template <int N>
__device__ __forceinline__ void reciprocal2(const f32x2 (&minus_d)[N], f32x2 (&out)[N]) {
  float d[2 * N], r[2 * N];
#pragma unroll
  for (int i = 0; i < N; ++i) split2(minus_d[i], &d[2 * i], &d[2 * i + 1]);
#pragma unroll
  for (int i = 0; i < 2 * N; ++i) {
    d[i] = fmaxf(d[i], -1e30f);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r[i]) : "f"(-d[i]));
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const f32x2 r2 = pair2(r[2 * i], r[2 * i + 1]);
    out[i] = fma2(r2, fma2(pair2(d[2 * i], d[2 * i + 1]), r2, pair2(1.f, 1.f)), r2);
  }
}

// Exact (erf) GELU, in place, and its derivative from one evaluation of 2 * N values:  erf through Abramowitz & Stegun 7.1.26
// (absolute error below 1.5e-7, far inside a bf16 rounding), whose exp(-z^2) with z = |x| / sqrt(2) is the very
// exp(-x^2 / 2) that the density needs.  Everything but the special-function unit's part is packed, and the N pairs take each step
// together (one, two, four and eight at a time: 56, 47.4, 48.0 and 52 us for 8192 x 3072 x 768, where eight spill).
//   gelu(x)  = x * Phi(x)          Phi(x) = (1 + erf(x / sqrt 2)) / 2
//   gelu'(x) = Phi(x) + x * phi(x)  phi(x) = exp(-x^2 / 2) / sqrt(2 pi)
template <int N>
__device__ __forceinline__ void gelu_and_grad2(f32x2 (&x)[N], f32x2 (&slope)[N]) {
  auto both = [](float v) { return pair2(v, v); };
  f32x2 t[N], e[N], p[N];
  float v[2 * N], r[2 * N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    split2(x[i], &v[2 * i], &v[2 * i + 1]);
    const f32x2 z = mul2(pair2(fabsf(v[2 * i]), fabsf(v[2 * i + 1])), both(0.70710678118654752440f));
    p[i] = fma2(both(-0.3275911f), z, both(-1.f));
  }
  reciprocal2(p, t);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float a0, a1;
    split2(mul2(mul2(both(-0.72134752044448170368f), x[i]), x[i]), &a0, &a1);  // log2 of exp(-x^2 / 2)
    e[i] = pair2(ex2_approx(a0), ex2_approx(a1));
  }
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = fma2(t[i], both(-1.061405429f), both(1.453152027f));  // the polynomial with its sign turned
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = fma2(t[i], p[i], both(-1.421413741f));
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = fma2(t[i], p[i], both(0.284496736f));
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = fma2(t[i], p[i], both(-0.254829592f));
#pragma unroll
  for (int i = 0; i < N; ++i) split2(fma2(mul2(t[i], p[i]), e[i], both(1.f)), &r[2 * i], &r[2 * i + 1]);  // erf(|x| / sqrt 2)
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const f32x2 cdf = mul2(both(0.5f), add2(both(1.f), pair2(copysignf(r[2 * i], v[2 * i]), copysignf(r[2 * i + 1], v[2 * i + 1]))));
    slope[i] = fma2(mul2(x[i], both(0.39894228040143267794f)), e[i], cdf);
    x[i] = mul2(x[i], cdf);
  }
}
__device__ __forceinline__ void gelu_and_grad(float x, float* g, float* dg) {
  f32x2 g2[1] = {pair2(x, x)}, d2[1];
  gelu_and_grad2(g2, d2);
  float unused;
  split2(g2[0], g, &unused);
  split2(d2[0], dg, &unused);
}

// ------------------------------------------------------------------------------------------ kernel
// One 32-column chunk of one accumulator row: the general path (tile edges, padded rows, any flags).
__device__ __forceinline__ void epilogue_chunk_generic(const uint32_t (&raw)[32], int row, int col0, const GemmArgs& g, void* out,
                                                       bool out_f32) {
  if (row < g.M && col0 < g.N) {
    const size_t base = (size_t)row * g.ldc + col0;
#pragma unroll
    for (int v8 = 0; v8 < 4; ++v8) {  // 8 columns at a time
      const int col = col0 + v8 * 8;
      if (col >= g.N) break;
      float x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(raw[v8 * 8 + j]);
      if (g.flags & EPI_BIAS) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (col + j < g.N) x[j] += __bfloat162float(g.bias[col + j]);
      }
      const bool full8 = col + 8 <= g.ldc;  // the padded row has room for a whole vector
      if (g.flags & (EPI_RESIDUAL | EPI_DGELU)) {
        __nv_bfloat16 aux[8];
        if (full8) {
          *reinterpret_cast<uint4*>(aux) = *reinterpret_cast<const uint4*>(g.aux_in + base + v8 * 8);
        } else {
          for (int j = 0; j < 8; ++j) aux[j] = col + j < g.N ? g.aux_in[base + v8 * 8 + j] : __float2bfloat16(0.f);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float a = __bfloat162float(aux[j]);
          x[j] = (g.flags & EPI_RESIDUAL) ? x[j] + a : x[j] * a;
        }
      }
      if (g.flags & EPI_GELU) {
        float dg[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) gelu_and_grad(x[j], &x[j], &dg[j]);
        if (g.aux_out != nullptr) {
          __nv_bfloat16 pre[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) pre[j] = __float2bfloat16_rn(dg[j]);
          if (full8) {
            *reinterpret_cast<uint4*>(g.aux_out + base + v8 * 8) = *reinterpret_cast<const uint4*>(pre);
          } else {
            for (int j = 0; j < 8; ++j)
              if (col + j < g.N) g.aux_out[base + v8 * 8 + j] = pre[j];
          }
        }
      }
      if (out_f32) {
        float* o = reinterpret_cast<float*>(out) + base + v8 * 8;
        if (full8) {
          float4 lo = make_float4(x[0], x[1], x[2], x[3]), hi = make_float4(x[4], x[5], x[6], x[7]);
          if (g.flags & EPI_ACCUMULATE) {
            const float4 a = *reinterpret_cast<const float4*>(o), b = *reinterpret_cast<const float4*>(o + 4);
            lo.x += a.x; lo.y += a.y; lo.z += a.z; lo.w += a.w;
            hi.x += b.x; hi.y += b.y; hi.z += b.z; hi.w += b.w;
          }
          *reinterpret_cast<float4*>(o) = lo;
          *reinterpret_cast<float4*>(o + 4) = hi;
        } else {
          for (int j = 0; j < 8; ++j)
            if (col + j < g.N) o[j] = (g.flags & EPI_ACCUMULATE) ? o[j] + x[j] : x[j];
        }
      } else {
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(out) + base + v8 * 8;
        __nv_bfloat16 y[8];
        if (g.flags & EPI_ACCUMULATE) {
          if (full8) {
            *reinterpret_cast<uint4*>(y) = *reinterpret_cast<const uint4*>(o);
          } else {
            for (int j = 0; j < 8; ++j) y[j] = col + j < g.N ? o[j] : __float2bfloat16(0.f);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) x[j] += __bfloat162float(y[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = __float2bfloat16_rn(x[j]);
        if (full8) {
          *reinterpret_cast<uint4*>(o) = *reinterpret_cast<const uint4*>(y);
        } else {
          for (int j = 0; j < 8; ++j)
            if (col + j < g.N) o[j] = y[j];
        }
      }
    }
  }
}

// What a tile's accumulators become on the way out (chosen by the host).
enum EpilogueKind {
  KIND_DIRECT = 0,  // anything else: each thread stores its row (fp32 outputs, unaligned rows, rare flag combinations)
  KIND_PLAIN = 1,   // (+ bias)
  KIND_ADD = 2,     // (+ bias) + aux_in
  KIND_MUL = 3,     // (+ bias) * aux_in
  KIND_GELU = 4,    // gelu(+ bias), and gelu' to aux_out if it is wanted
};

// Eight columns of a lane's row of a 32-row x 32-column bf16 block in shared memory: rows of 64 bytes, 16-byte slots
// XOR-swizzled as TMA's 64-byte swizzle does, which also spreads a warp's writes (lane = row) over all banks.
__device__ __forceinline__ void put8(uint8_t* block, int lane, int slot, uint4 v) {
  *reinterpret_cast<uint4*>(block + lane * 64 + ((slot ^ ((lane >> 1) & 3)) << 4)) = v;
}

__device__ __forceinline__ void bulk_store_2d(const CUtensorMap* map, const uint8_t* block, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(smem_u32(block)), "r"(x), "r"(y)
               : "memory");
}

// One epilogue warp's way out of a tile: 32 rows x columns [32 * c_begin, 32 * c_end), 32 columns at a time.
// TMEM -> registers -> element-wise work -> a swizzled 2 KB block in shared memory -> one bulk tensor store, which clips
// rows >= M and columns >= N.  The stores never pass through the load/store unit, whose
// global stores (measured on B200) slow the MMA/TMA traffic of the main loop several times more than their size
// would suggest.  There is one body per kind, the loop over chunks stays rolled (with every flag tested in one body
// unrolled over 64 columns it cost 1100 cycles per 64 columns to fetch the instructions of plain results, 12000 of GELU), and the bias passes
// through shared memory (one coalesced load per chunk instead of a load per column).
// What bounded it was waiting: for a chunk's aux_in, fetched by the lanes one chunk ahead and row by row, for the first bias, and
// for the stores to release the blocks.  So begin(), called before the accumulator is complete, fetches the tile's bias and starts TMA
// loads of aux_in into the blocks that the results will leave from (a lane replaces the values of its own row), and there are
// BLOCKS blocks per warp, four where the ring keeps enough stages without their memory.  Before and after (with what this file gained
// since: the deeper ring, the late trigger, the relaxed arrival), us, one after the other in a graph: bias + residual 3072 x 384 x 384 6.3, 4.9;
// 1024 x 768 x 768 7.3, 5.9; 4096 x 1024 x 1024 14.2, 10.7; 8192 x 768 x 3072 46.1, 35.8; times gelu' 8192 x 3072 x 768 44.9, 37.5; GELU
// at that size 55.9, 44.4.  What bounds GELU beside a main loop of twelve k-blocks is a warp's own chain (TMEM, special functions,
// packed arithmetic, block; two warps per scheduler): the tensor pipe is active for 34 %, shared memory's pipes for 32 % and its banks for 12 %.
template <int BLOCKS, int CHUNKS, int GELU_PAIRS = 2>
struct Epilogue {
  uint8_t* staging;    // of all eight warps: blocks [8][BLOCKS][BLOCK_BYTES], bias values [8][32], barriers of the loads [8][BLOCKS]
  int warp;            // 0 .. 7
  uint32_t aux_phase;  // bit b: parity of the next completion of block b's barrier
  uint32_t stored;     // chunks stored so far
  uint32_t bias[(CHUNKS + 1) / 2];  // a lane's column of each chunk: bf16, two to a register

  static constexpr int BIAS_AT = 8 * BLOCKS * BLOCK_BYTES, BARRIERS_AT = BIAS_AT + 8 * 128, BYTES = BARRIERS_AT + 8 * BLOCKS * 8;
  // Worked out where they are used: the compiler would keep them through fold_tile, which needs every register.
  __device__ __forceinline__ int here() const {
    int w = warp;
    asm volatile("" : "+r"(w));
    return w;
  }
  __device__ __forceinline__ uint8_t* blocks() const { return staging + here() * BLOCKS * BLOCK_BYTES; }
  __device__ __forceinline__ float* bias_sm() const { return reinterpret_cast<float*>(staging + BIAS_AT + here() * 128); }
  __device__ __forceinline__ uint64_t* aux_full() const { return reinterpret_cast<uint64_t*>(staging + BARRIERS_AT) + here() * BLOCKS; }

  __device__ __forceinline__ void init() {
#pragma unroll
    for (int b = 0; b < BLOCKS; ++b) mbar_init(&aux_full()[b], 1);
  }

  static __device__ __forceinline__ void wait_stores_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

  // The chunks that lie in the matrix: none if the warp's rows do not.
  static __device__ __forceinline__ int clip(const GemmArgs& g, int c_end, int n0, int row0) {
    const int in = (g.N - n0 + 31) / 32;
    return row0 >= g.M ? 0 : c_end < in ? c_end : in;
  }

  __device__ __forceinline__ void load_aux(const CUtensorMap* map, int block, int x, int y) {
    mbar_expect_tx(&aux_full()[block], BLOCK_BYTES);
    tma_load_2d(blocks() + block * BLOCK_BYTES, map, &aux_full()[block], x, y);
  }

  __device__ __forceinline__ void begin(const GemmArgs& g, const CUtensorMap* aux_map, int c_begin, int c_end, int n0, int row0, int lane) {
    c_end = clip(g, c_end, n0, row0);
    if ((g.kind == KIND_ADD || g.kind == KIND_MUL) && c_begin < c_end && elect_one()) {
      wait_stores_read();
#pragma unroll
      for (int i = 0; i < BLOCKS; ++i)
        if (c_begin + i < c_end) load_aux(aux_map, i, n0 + (c_begin + i) * 32, row0);
    }
    if (g.kind != KIND_DIRECT && (g.flags & EPI_BIAS)) {
      const unsigned short* b = reinterpret_cast<const unsigned short*>(g.bias);
      auto value = [&](int i) {
        const int col = n0 + (c_begin + i) * 32 + lane;
        return i < CHUNKS && c_begin + i < c_end && col < g.N ? (uint32_t)b[col] : 0u;
      };
#pragma unroll
      for (int i = 0; i < CHUNKS; i += 2) bias[i / 2] = value(i) | value(i + 1) << 16;
    }
  }

  // False (and the error word raised) if a load did not arrive.
  template <int KIND, typename Release>
  __device__ __forceinline__ bool store(uint32_t taddr, int c_begin, int c_end, int n0, int row0, int lane, const GemmArgs& g,
                                        const CUtensorMap* aux_map, const CUtensorMap* out_map, const CUtensorMap* pre_map, Release release) {
    c_end = clip(g, c_end, n0, row0);
    if (c_begin >= c_end) {
      release();
      return true;
    }
    const bool has_bias = g.flags & EPI_BIAS, keep_pre = KIND == KIND_GELU && g.aux_out != nullptr;
    constexpr bool HAS_AUX = KIND == KIND_ADD || KIND == KIND_MUL;
    constexpr int PER_CHUNK = KIND == KIND_GELU ? 2 : 1, TURNS = BLOCKS / PER_CHUNK;  // blocks per chunk; chunks in flight
    uint8_t* const blocks = this->blocks();
    float* const bias_sm = this->bias_sm();
    bool ok = true;
#pragma unroll 1
    for (int c = c_begin; c < c_end; ++c) {
      uint32_t raw[32];
      tmem_ld32(taddr + c * 32, raw);
      if (has_bias) {
        __syncwarp();  // the previous chunk's values have been read
        bias_sm[lane] = __uint_as_float(bias[0] << 16);
        constexpr int LAST = (CHUNKS + 1) / 2 - 1;
#pragma unroll
        for (int i = 0; i < LAST; ++i) bias[i] = __funnelshift_r(bias[i], bias[i + 1], 16);
        bias[LAST] >>= 16;
      }
      const int turn = HAS_AUX ? (c - c_begin) % TURNS : (int)(stored % TURNS);
      uint8_t* block = blocks + turn * PER_CHUNK * BLOCK_BYTES;
      uint4 aux[4];
      if (HAS_AUX) {
        if (!(ok = mbar_wait_all(&aux_full()[turn], (aux_phase >> turn) & 1, g.error))) break;
        aux_phase ^= 1u << turn;
#pragma unroll
        for (int v = 0; v < 4; ++v) aux[v] = *reinterpret_cast<const uint4*>(block + lane * 64 + ((v ^ ((lane >> 1) & 3)) << 4));
      } else if (elect_one()) {  // the store that last used this block has read it
        asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(TURNS - 1) : "memory");
      }
      __syncwarp();
      tmem_ld_wait();
      if (c + 1 == c_end) release();  // the accumulator is in registers
      f32x2 x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] = pair2(__uint_as_float(raw[2 * j]), __uint_as_float(raw[2 * j + 1]));
      if (has_bias) {
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const float4 b = *reinterpret_cast<const float4*>(bias_sm + 4 * v);
          x[2 * v] = add2(x[2 * v], pair2(b.x, b.y));
          x[2 * v + 1] = add2(x[2 * v + 1], pair2(b.z, b.w));
        }
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        uint32_t y[4], dy[4];
        const uint32_t a[4] = {aux[v].x, aux[v].y, aux[v].z, aux[v].w};
        if (KIND == KIND_GELU) {
          f32x2 slope[4];
#pragma unroll
          for (int j = 0; j < 4; j += GELU_PAIRS)
            gelu_and_grad2(*reinterpret_cast<f32x2(*)[GELU_PAIRS]>(x + 4 * v + j), *reinterpret_cast<f32x2(*)[GELU_PAIRS]>(slope + j));
#pragma unroll
          for (int j = 0; j < 4; ++j) dy[j] = bf16_pair(slope[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          f32x2 w = x[4 * v + j];
          if (KIND == KIND_ADD) w = add2(w, from_bf16_pair(a[j]));
          if (KIND == KIND_MUL) w = mul2(w, from_bf16_pair(a[j]));
          y[j] = bf16_pair(w);
        }
        put8(block, lane, v, make_uint4(y[0], y[1], y[2], y[3]));
        if (keep_pre) put8(block + BLOCK_BYTES, lane, v, make_uint4(dy[0], dy[1], dy[2], dy[3]));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy accesses, then the async proxy's
      __syncwarp();
      if (elect_one()) {
        bulk_store_2d(out_map, block, n0 + c * 32, row0);
        if (keep_pre) bulk_store_2d(pre_map, block + BLOCK_BYTES, n0 + c * 32, row0);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        if (HAS_AUX && c + TURNS < c_end) {  // fewer blocks than chunks: the next load into this one
          wait_stores_read();
          load_aux(aux_map, turn, n0 + (c + TURNS) * 32, row0);
        }
      }
      ++stored;
    }
    if (!ok) release();
    return ok;
  }

  template <typename Release>
  __device__ __forceinline__ bool finish(uint32_t taddr, int c_begin, int c_end, int n0, int row0, int lane, const GemmArgs& g,
                                         const CUtensorMap* aux_map, const CUtensorMap* out_map, const CUtensorMap* pre_map, Release release) {
    switch (g.kind) {
      case KIND_PLAIN: return store<KIND_PLAIN>(taddr, c_begin, c_end, n0, row0, lane, g, aux_map, out_map, pre_map, release);
      case KIND_ADD: return store<KIND_ADD>(taddr, c_begin, c_end, n0, row0, lane, g, aux_map, out_map, pre_map, release);
      case KIND_MUL: return store<KIND_MUL>(taddr, c_begin, c_end, n0, row0, lane, g, aux_map, out_map, pre_map, release);
      case KIND_GELU: return store<KIND_GELU>(taddr, c_begin, c_end, n0, row0, lane, g, aux_map, out_map, pre_map, release);
      default: {
#pragma unroll 1
        for (int c = c_begin; c < c_end; ++c) {
          uint32_t raw[32];
          tmem_ld32(taddr + c * 32, raw);
          tmem_ld_wait();
          epilogue_chunk_generic(raw, row0 + lane, n0 + c * 32, g, g.out, g.flags & EPI_OUT_F32);
        }
        release();
        return true;
      }
    }
  }
};

// Split-K (GemmArgs): a producer's warp parks its 32 rows x columns [32 * c_begin, 32 * c_end) of raw accumulator; the
// consumer's matching warp folds the parked parts, in part order, into its own accumulator in TMEM.
// Layout of a parked tile of ROWS rows: [column quad][row][4 floats].  A lane's four consecutive columns are one 16-byte
// vector and consecutive lanes (rows) are consecutive vectors, so a warp moves 512 contiguous bytes per instruction.
template <int ROWS>
__device__ __forceinline__ void park_tile(uint32_t taddr, int c_begin, int c_end, float* tile, int tile_row) {
#pragma unroll 1
  for (int c = c_begin; c < c_end; ++c) {
    uint32_t raw[32];
    tmem_ld32(taddr + c * 32, raw);
    tmem_ld_wait();
    float4* dst = reinterpret_cast<float4*>(tile) + (size_t)c * 8 * ROWS + tile_row;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      __stcg(dst + (size_t)q * ROWS, make_float4(__uint_as_float(raw[4 * q]), __uint_as_float(raw[4 * q + 1]),
                                                 __uint_as_float(raw[4 * q + 2]), __uint_as_float(raw[4 * q + 3])));
  }
}

template <int ROWS, int TILE_FLOATS>
__device__ __forceinline__ void fold_tile(uint32_t taddr, int c_begin, int c_end, const float* tiles, int parts, int tile_row) {
#pragma unroll 1
  for (int c = c_begin; c < c_end; c += 2) {
    const bool two = c + 1 < c_end;
    uint32_t raw[2][32];
    tmem_ld32(taddr + c * 32, raw[0]);
    if (two) tmem_ld32(taddr + (c + 1) * 32, raw[1]);
    tmem_ld_wait();
    for (int p = 0; p < parts; ++p) {
      const float4* src = reinterpret_cast<const float4*>(tiles + (size_t)p * TILE_FLOATS) + (size_t)c * 8 * ROWS + tile_row;
      // all sixteen loads of a part are issued before the first add: one trip to L2 per part, not one per batch
      // the compiler happens to pick (volatile asm statements keep their order)
      float4 v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (q < 8 || two)
          asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v[q].x), "=f"(v[q].y), "=f"(v[q].z), "=f"(v[q].w)
                       : "l"(src + (size_t)q * ROWS)
                       : "memory");
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        if (q < 8 || two) {
          uint32_t* r = raw[q >> 3] + 4 * (q & 7);
          r[0] = __float_as_uint(__uint_as_float(r[0]) + v[q].x);
          r[1] = __float_as_uint(__uint_as_float(r[1]) + v[q].y);
          r[2] = __float_as_uint(__uint_as_float(r[2]) + v[q].z);
          r[3] = __float_as_uint(__uint_as_float(r[3]) + v[q].w);
        }
      }
    }
    tmem_st32(taddr + c * 32, raw[0]);
    if (two) tmem_st32(taddr + (c + 1) * 32, raw[1]);
  }
  tmem_st_wait();
}

// The flag a producer's warp raises once its share is parked, and the consumer's bounded wait for the same warp's flags
// of all parts (`stride` words apart).  The flags are zero again afterwards, for the next launch that is handed these words.
__device__ __forceinline__ void raise_flag(unsigned* flag, int lane) {
  __syncwarp();  // every lane's stores come before lane 0's release, which is cumulative: it covers them all
  if (lane == 0) st_release_gpu(flag, 1u);
}
__device__ __forceinline__ bool wait_flags(unsigned* flags, int parts, int stride, int lane, int* error) {
  bool seen = true;
  if (lane < parts) {
    const long long start = clock64();
    while (ld_acquire_gpu(flags + lane * stride) == 0u) {
      if (clock64() - start > (1ll << WAIT_LIMIT_CYCLES_SHIFT)) {
        *error = 1;
        __threadfence_system();
        seen = false;
        break;
      }
    }
    flags[lane * stride] = 0u;
  }
  seen = __all_sync(0xffffffffu, seen);
  __syncwarp();  // every lane reads the parked parts next: behind what the polling lanes acquired (a vote orders no memory)
  return seen;
}

// Work items of a split problem: whole tiles, then the tail's producers (parts 1 .. splits-1), then its consumers (part 0).
struct Items {
  int whole, tail, splits, k_blocks, k_per, count;
  __device__ Items(const GemmArgs& g, int out_tiles) {
    splits = g.splits > 1 ? g.splits : 1;
    whole = splits > 1 ? g.whole_tiles : out_tiles;
    tail = out_tiles - whole;
    count = whole + tail * splits;
    k_blocks = (g.K + BK - 1) / BK;
    k_per = (k_blocks + splits - 1) / splits;
  }
  __device__ int tile(int item) const { return item < whole ? item : whole + (item - whole) % tail; }
  __device__ int part(int item) const {  // -1: the whole reduction
    return item < whole ? -1 : (item - whole < tail * (splits - 1) ? 1 + (item - whole) / tail : 0);
  }
  __device__ void k_range(int item, int* kb0, int* kb1) const {
    const int p = part(item);
    *kb0 = p < 0 ? 0 : p * k_per;
    *kb1 = p < 0 || (p + 1) * k_per > k_blocks ? k_blocks : (p + 1) * k_per;
  }
};

// Before an epilogue warp leaves: its bulk stores have read their shared-memory blocks (the writes themselves
// complete with the grid).
__device__ __forceinline__ void drain_stores() {
  if (elect_one()) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
}

// Tile shapes.  BM = 128: one 128-row accumulator per tile, two of them in TMEM so the next tile's
// MMAs overlap this tile's epilogue.  BM = 256: two 128-row MMAs per k-step share one B tile (a
// third less operand traffic per flop and twice the work per pipeline stage, which is what hides
// the load latency); its two accumulators fill TMEM, so only the halves overlap.
template <int BM, int BN>
struct SmemLayout {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int BLOCKS = BM == 128 && BN == 192 ? 4 : 2;  // staging blocks per epilogue warp
  static constexpr int STAGING = Epilogue<BLOCKS, 1>::BYTES;
  static constexpr int FIT = (SMEM_BUDGET - 8 * BLOCKS * BLOCK_BYTES) / STAGE_BYTES, STAGES = FIT > 8 ? 8 : FIT;
  static constexpr int TOTAL = STAGES * STAGE_BYTES + STAGING + 1024 /* alignment slack */ + 256 /* barriers */;
  static_assert(TOTAL <= 227 * 1024, "shared memory of one SM");
  static constexpr int THREADS = 64 + 256;  // producer warp, MMA warp, eight epilogue warps
};

template <int BM, int BN, bool A_MN, bool B_MN, bool GATHER = false>
__global__ void __launch_bounds__(GATHER ? 448 : 320, 1)
k_gemm(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_out,
       const __grid_constant__ CUtensorMap map_pre, const __grid_constant__ CUtensorMap map_aux, const GemmArgs g, const GatherArgs ga) {
  extern __shared__ uint8_t smem_raw[];
  using L = SmemLayout<BM, BN>;
  constexpr int STAGES = L::STAGES;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + STAGES * L::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + L::STAGING);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // warp: known to be uniform
  const int tiles_m = (g.M + BM - 1) / BM, tiles_n = (g.N + BN - 1) / BN;
  const Items items(g, tiles_m * tiles_n);
  constexpr uint32_t ACC_COLS = BN == 192 ? 256 : BN;  // column stride between the two accumulators
  constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;         // 256 or 512: a power of two
  // Item -> (m0, n0).  With GATHER m runs fastest, so the CTAs sweep one weight panel at a time, starting from the one
  // this rank's own shard feeds: the order in which the chunks arrive.
  auto tile_origin = [&](int item, int* m0, int* n0) {
    int m_idx, n_idx;
    tile_coords(items.tile(item), tiles_m, items.whole, GATHER ? tiles_m : g.group_m, &m_idx, &n_idx);
    if (GATHER) n_idx = (n_idx + ga.n_start) % tiles_n;
    *m0 = m_idx * BM;
    *n0 = n_idx * BN;
  };

  if (warp == 0) {  // one lane per barrier; warp 1 allocates TMEM meanwhile
    if (lane < STAGES) {
      mbar_init(&full[lane], 1);
      mbar_init(&empty[lane], 1);
    } else if (lane < STAGES + 2) {
      mbar_init(&acc_full[lane - STAGES], 1);
      mbar_init(&acc_empty[lane - STAGES], BM == 128 ? 8 : 4);  // one arrival per epilogue warp that drains it
    } else if (lane < STAGES + 2 + 8) {
      Epilogue<L::BLOCKS, 1>{staging, lane - STAGES - 2}.init();
    } else if (lane == STAGES + 2 + 8) {
      prefetch_tensormap(&map_a);
      prefetch_tensormap(&map_b);
      if (g.kind != KIND_DIRECT) prefetch_tensormap(&map_out);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  tb::pdl_wait();  // barriers and TMEM are ready; from here on global memory written by earlier kernels is read

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    uint32_t s = 0, phase = 1;  // ring slot and the parity of its next `empty`
    bool ok = true;
    for (int tile = blockIdx.x; tile < items.count && ok; tile += gridDim.x) {
      int m0, n0;
      tile_origin(tile, &m0, &n0);
      if (GATHER) {  // the panel's bytes must have arrived (they are row-contiguous: rows n0 .. n0+BN of [N, K])
        const long long lo = (long long)n0 * g.K * 2;
        long long hi = (long long)(n0 + BN < g.N ? n0 + BN : g.N) * g.K * 2;
        ok = wait_chunks(ga.ready, (int)(lo / ga.chunk_bytes), (int)((hi - 1) / ga.chunk_bytes), ga.epoch, g.error);
        if (!(ok = __all_sync(0xffffffffu, ok))) break;
        asm volatile("fence.proxy.async;" ::: "memory");  // the fetchers' generic-proxy stores, then TMA's async-proxy loads
      }
      int kb0, kb1;
      items.k_range(tile, &kb0, &kb1);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!(ok = mbar_wait_all(&empty[s], phase, g.error))) break;
        if (elect_one()) {
          uint8_t* a_dst = smem + s * L::STAGE_BYTES;
          uint8_t* b_dst = a_dst + L::A_BYTES;
          mbar_expect_tx(&full[s], L::STAGE_BYTES);
          const int k0 = kb * BK;
          if (!A_MN) {
            tma_load_2d(a_dst, &map_a, &full[s], k0, m0);  // box {64 k, BM rows}
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d(a_dst + j * 8192, &map_a, &full[s], m0 + j * 64, k0);  // box {64 mn, 64 k}
          }
          if (!B_MN) {
            tma_load_2d(b_dst, &map_b, &full[s], k0, n0);  // box {64 k, BN rows}
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_2d(b_dst + j * 8192, &map_b, &full[s], n0 + j * 64, k0);
          }
        }
        if (++s == STAGES) s = 0, phase ^= 1;
      }
    }
    tb::pdl_launch_dependents();  // all loads are under way: the next kernel may set itself up while the last tile is finished
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc = instr_desc(128, BN, A_MN, B_MN);
    constexpr int HALVES = BM / 128;
    uint32_t s = 0, phase = 0, local_tile = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < items.count && ok; tile += gridDim.x, ++local_tile) {
      // BM = 128: accumulators alternate between the two TMEM regions.  BM = 256: region h holds rows [128h, 128h+128).
      const uint32_t first_buf = HALVES == 1 ? (local_tile & 1) : 0;
      const uint32_t acc_phase = HALVES == 1 ? ((local_tile >> 1) & 1) : (local_tile & 1);
      int kb0, kb1;
      items.k_range(tile, &kb0, &kb1);
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        if (!(ok = mbar_wait_all(&full[s], phase, g.error))) break;
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + s * L::STAGE_BYTES);
        const uint32_t b_addr = a_addr + L::A_BYTES;
        // K-major: rows of 128 B, 8-row groups 1024 B apart; one K=16 step is 32 B along the row.
        // MN-major: 64-wide strips 8192 B apart (LBO), 8 k-rows 1024 B apart (SBO); one K=16 step is 16 rows = 2048 B.
        const uint64_t b_desc = B_MN ? smem_desc(b_addr, 8192, 1024) : smem_desc(b_addr, 16, 1024);
#pragma unroll
        for (int h = 0; h < HALVES; ++h) {
          const uint32_t buf = first_buf + h;
          if (kb == kb0) {  // the epilogue has drained this accumulator
            if (!(ok = mbar_wait_all(&acc_empty[buf], acc_phase ^ 1, g.error))) break;
            tc_fence_after();
          }
          const uint32_t d_tmem = tmem_base + buf * ACC_COLS;
          const uint32_t a_half = a_addr + h * 16384;  // 128 rows x 128 B, or two 64-wide strips
          const uint64_t a_desc = A_MN ? smem_desc(a_half, 8192, 1024) : smem_desc(a_half, 16, 1024);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) {
              const uint64_t a_k = a_desc + (uint64_t)((A_MN ? 2048 : 32) * k >> 4);
              const uint64_t b_k = b_desc + (uint64_t)((B_MN ? 2048 : 32) * k >> 4);
              mma_bf16(d_tmem, a_k, b_k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
            }
          }
        }
        if (ok && elect_one()) mma_commit(&empty[s]);  // the stage may be refilled once these MMAs have read it
        if (++s == STAGES) s = 0, phase ^= 1;
      }
      if (ok && elect_one()) {
#pragma unroll
        for (int h = 0; h < HALVES; ++h) mma_commit(&acc_full[first_buf + h]);
      }
    }
  } else if (GATHER && warp >= 10) {
    // ------------------------------------------------------------------ weight fetchers (warps 10 - 13)
    const int ft = threadIdx.x - 320;  // 0..127: four fetch warps
    constexpr int FT = 128, DEPTH = 8;  // eight independent 16-byte loads in flight per thread: 16 KB per CTA, ~2.4 MB per GPU
    const int nchunks = (int)((ga.w_bytes + ga.chunk_bytes - 1) / ga.chunk_bytes);
    const int first = (int)(((long long)ga.n_start * BN * g.K * 2) / ga.chunk_bytes);
    __threadfence_system();  // observe the owners' latest stores to their shards
    for (int ci = blockIdx.x; ci < nchunks; ci += gridDim.x) {
      const int c = (first + ci) % nchunks;
      const long long c0 = ga.w_off + (long long)c * ga.chunk_bytes;
      const long long c1 = ga.w_off + ((long long)(c + 1) * ga.chunk_bytes < ga.w_bytes ? (long long)(c + 1) * ga.chunk_bytes : ga.w_bytes);
      for (int q = 0; q < ga.n; ++q) {
        const long long lo = c0 > ga.shard_lo[q] ? c0 : ga.shard_lo[q];
        const long long hi = c1 < ga.shard_hi[q] ? c1 : ga.shard_hi[q];
        if (lo >= hi) continue;
        const char* src = ga.shard[q] + (lo - ga.shard_lo[q]);
        char* dst = ga.full + lo;
        const long long len = hi - lo;
        const bool al = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
        const long long nv = al ? len / 16 : 0;
        for (long long v = ft; v < nv; v += FT * DEPTH) {
          uint4 x[DEPTH];
#pragma unroll
          for (int u = 0; u < DEPTH; ++u)
            if (v + u * FT < nv)
              asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                           : "=r"(x[u].x), "=r"(x[u].y), "=r"(x[u].z), "=r"(x[u].w) : "l"(src + (v + u * FT) * 16));
#pragma unroll
          for (int u = 0; u < DEPTH; ++u)
            if (v + u * FT < nv) *reinterpret_cast<uint4*>(dst + (v + u * FT) * 16) = x[u];
        }
        for (long long i = nv * 16 + ft; i < len; i += FT) dst[i] = *reinterpret_cast<volatile const char*>(src + i);
      }
      __threadfence();
      asm volatile("bar.sync 1, 128;" ::: "memory");  // the fetch warps only
      if (ft == 0) st_release_gpu(ga.ready + c, ga.epoch);
    }
  } else if (warp < 10) {
    // ------------------------------------------------------------------ epilogue (warps 2 .. 9)
    // Eight epilogue warps in two groups of four (one warp per TMEM lane quarter in each group).
    // BM = 128: both groups drain the same accumulator, each taking half of its columns.
    // BM = 256: group h drains the accumulator of rows [128h, 128h + 128).
    const int quarter = warp & 3;        // TMEM lanes [32*quarter, 32*quarter + 32) belong to this warp
    const int group = (warp - 2) >> 2;
    const int half = BM == 128 ? 0 : group;
    uint32_t local_tile = 0;
    bool ok = true;
    constexpr int CHUNKS = BN / 32, MINE = BM == 128 ? CHUNKS / 2 : CHUNKS;  // BM = 128: the two warp groups split the columns
    Epilogue<L::BLOCKS, MINE> epilogue{staging, warp - 2, 0, 0, {}};
    const int c_begin = BM == 128 ? group * MINE : 0, c_end = c_begin + MINE;
    if (GATHER && (g.flags & EPI_BIAS) && ga.tail_bytes > 0) {
      // the bias sits right behind the weight in the flat buffer and is fetched with it: wait for its chunks
      const long long lo = (long long)g.N * g.K * 2, hi = lo + ga.tail_bytes;
      ok = wait_chunks(ga.ready, (int)(lo / ga.chunk_bytes), (int)((hi - 1) / ga.chunk_bytes), ga.epoch, g.error);
      ok = __all_sync(0xffffffffu, ok);
    }
    for (int tile = blockIdx.x; tile < items.count && ok; tile += gridDim.x, ++local_tile) {
      int m0, n0;
      tile_origin(tile, &m0, &n0);
      const int part = items.part(tile), split_tile = items.tile(tile) - items.whole, parts = items.splits - 1;
      // the parked parts of its output tile, and this warp's flag for the first of them
      float* parked = part >= 0 ? g.partials + (size_t)split_tile * parts * (BM * BN) : nullptr;
      unsigned* my_flags = part >= 0 ? g.split_flags + (size_t)split_tile * parts * 8 + (warp - 2) : nullptr;
      const int tile_row = half * 128 + quarter * 32 + lane;
      const uint32_t buf = BM == 128 ? (local_tile & 1) : half;
      const uint32_t acc_phase = BM == 128 ? ((local_tile >> 1) & 1) : (local_tile & 1);
      const int row0 = m0 + half * 128 + quarter * 32;  // first row of this warp's block
      if (part <= 0) epilogue.begin(g, &map_aux, c_begin, c_end, n0, row0, lane);
      ok = mbar_wait_all(&acc_full[buf], acc_phase, g.error);
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * ACC_COLS;
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      };
      if (part > 0) {
        park_tile<BM>(taddr, c_begin, c_end, parked + (size_t)(part - 1) * (BM * BN), tile_row);
        release();
        raise_flag(my_flags + (part - 1) * 8, lane);
        continue;
      }
      if (part == 0) {
        if (!(ok = wait_flags(my_flags, parts, 8, lane, g.error))) break;
        fold_tile<BM, BM * BN>(taddr, c_begin, c_end, parked, parts, tile_row);
      }
      ok = epilogue.finish(taddr, c_begin, c_end, n0, row0, lane, g, &map_aux, &map_out, &map_pre, release);
    }
    drain_stores();
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}


// ------------------------------------------------------------------------------------------ CTA-pair kernel
// The same GEMM with tcgen05.mma.cta_group::2: two CTAs of a cluster, on neighbouring SMs, compute one
// 256 x BN tile together.  Each CTA loads its own 128 rows of A and HALF of the B tile (BN/2 rows), and the
// leader's MMA instructions read B from both CTAs' shared memory, so per flop each SM moves a third less
// operand data through TMA and reads a third less of it from shared memory than the 128 x 256 single-CTA
// tile -- the resource that bounds the single-CTA kernel.  Roles per CTA are the same as above (warp 0 TMA
// producer, warp 1 MMA issuer in the leader only, warps 2-9 epilogue of this CTA's 128 accumulator rows).
//   full[s]       leader's barrier: one arrive.expect_tx by the leader's producer + the bytes of BOTH CTAs' loads
//   empty[s]      each CTA's own barrier, signalled in both by one multicast tcgen05.commit
//   acc_full[b]   each CTA's own barrier, signalled in both by one multicast tcgen05.commit
//   acc_empty[b]  leader's barrier: 16 arrivals, one per epilogue warp of either CTA
// No TMA load uses multicast: each CTA reads its own tiles from global memory.
// DEEP: a ring of six stages (BN = 256) and two staging blocks per warp, instead of five and four.  With few k-blocks per tile the epilogue and
// its blocks count, with many the ring (us, deep / not: 16384 x 4096 x 1024 times gelu' 128 / 119, with GELU 144 / 136;
// 16384 x 8192 x 2048 444 / 453 and 475 / 496; 3072 x 768 x 8192 in two parts 34.2 / 34.9).
template <int BN, bool DEEP>
struct PairLayout {
  static constexpr int A_BYTES = 128 * BK * 2;       // this CTA's 128 rows of the 256-row A tile
  static constexpr int B_BYTES = (BN / 2) * BK * 2;  // this CTA's half of the B tile
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int BLOCKS = DEEP ? 2 : 4;  // staging blocks per epilogue warp
  static constexpr int STAGING = Epilogue<BLOCKS, 1>::BYTES;
  static constexpr int FIT = (SMEM_BUDGET - 8 * BLOCKS * BLOCK_BYTES) / STAGE_BYTES, STAGES = FIT > 8 ? 8 : FIT;
  static constexpr int TOTAL = STAGES * STAGE_BYTES + STAGING + 1024 /* alignment slack */ + 256 /* barriers */;
  static_assert(TOTAL <= 227 * 1024, "shared memory of one SM");
  static constexpr int THREADS = 64 + 256;
};

template <int BN, bool A_MN, bool B_MN, bool DEEP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320, 1)
k_gemm_pair(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_out,
            const __grid_constant__ CUtensorMap map_pre, const __grid_constant__ CUtensorMap map_aux, const GemmArgs g) {
  extern __shared__ uint8_t smem_raw[];
  using L = PairLayout<BN, DEEP>;
  constexpr int STAGES = L::STAGES;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + STAGES * L::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + L::STAGING);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;  // warp: known to be uniform
  const uint32_t rank = cluster_ctarank();  // 0: the leader
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int tiles_m = (g.M + 255) / 256, tiles_n = (g.N + BN - 1) / BN;
  const Items items(g, tiles_m * tiles_n);
  constexpr uint32_t TMEM_COLS = 2 * BN;  // two accumulators of BN fp32 columns

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 16);
    }
    for (int w = 0; w < 8; ++w) Epilogue<L::BLOCKS, 1>{staging, w}.init();
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_holder, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();  // both CTAs' barriers are initialised before either one signals the other's
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  tb::pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    uint32_t s = 0, phase = 1;
    bool ok = true;
    for (int tile = pair; tile < items.count && ok; tile += num_pairs) {
      int m_idx, n_idx;
      tile_coords(items.tile(tile), tiles_m, items.whole, g.group_m, &m_idx, &n_idx);
      const int m0 = m_idx * 256 + (int)rank * 128;
      const int n0 = n_idx * BN + (int)rank * (BN / 2);
      int kb0, kb1;
      items.k_range(tile, &kb0, &kb1);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!(ok = mbar_wait_all(&empty[s], phase, g.error))) break;
        if (elect_one()) {
          uint8_t* a_dst = smem + s * L::STAGE_BYTES;
          uint8_t* b_dst = a_dst + L::A_BYTES;
          if (rank == 0) mbar_expect_tx(&full[s], 2 * L::STAGE_BYTES);
          const uint32_t bar = map_to_cta(smem_u32(&full[s]), 0);
          const int k0 = kb * BK;
          if (!A_MN) {
            tma_load_2d_pair(a_dst, &map_a, bar, k0, m0);  // box {64 k, 128 rows}
          } else {
#pragma unroll
            for (int j = 0; j < 2; ++j) tma_load_2d_pair(a_dst + j * 8192, &map_a, bar, m0 + j * 64, k0);  // box {64 m, 64 k}
          }
          if (!B_MN) {
            tma_load_2d_pair(b_dst, &map_b, bar, k0, n0);  // box {64 k, BN/2 rows}
          } else {
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tma_load_2d_pair(b_dst + j * 8192, &map_b, bar, n0 + j * 64, k0);
          }
        }
        if (++s == STAGES) s = 0, phase ^= 1;
      }
    }
    tb::pdl_launch_dependents();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    if (rank == 0) {
      constexpr uint32_t idesc = instr_desc(256, BN, A_MN, B_MN);
      uint32_t s = 0, phase = 0, local_tile = 0;
      bool ok = true;
      for (int tile = pair; tile < items.count && ok; tile += num_pairs, ++local_tile) {
        const uint32_t buf = local_tile & 1;
        const uint32_t acc_phase = (local_tile >> 1) & 1;
        int kb0, kb1;
        items.k_range(tile, &kb0, &kb1);
        for (int kb = kb0; kb < kb1 && ok; ++kb) {
          if (!(ok = mbar_wait_all(&full[s], phase, g.error))) break;
          tc_fence_after();
          if (kb == kb0) {  // both CTAs' epilogues have drained this accumulator
            if (!(ok = mbar_wait_all(&acc_empty[buf], acc_phase ^ 1, g.error))) break;
            tc_fence_after();
          }
          const uint32_t a_addr = smem_u32(smem + s * L::STAGE_BYTES);
          const uint32_t b_addr = a_addr + L::A_BYTES;
          const uint64_t a_desc = A_MN ? smem_desc(a_addr, 8192, 1024) : smem_desc(a_addr, 16, 1024);
          const uint64_t b_desc = B_MN ? smem_desc(b_addr, 8192, 1024) : smem_desc(b_addr, 16, 1024);
          const uint32_t d_tmem = tmem_base + buf * BN;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) {
              const uint64_t a_k = a_desc + (uint64_t)((A_MN ? 2048 : 32) * k >> 4);
              const uint64_t b_k = b_desc + (uint64_t)((B_MN ? 2048 : 32) * k >> 4);
              mma_bf16_pair(d_tmem, a_k, b_k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
            }
            mma_commit_pair(&empty[s], 3);  // both CTAs may refill the stage once these MMAs have read it
          }
          if (++s == STAGES) s = 0, phase ^= 1;
        }
        if (ok && elect_one()) mma_commit_pair(&acc_full[buf], 3);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2 .. 9, both CTAs)
    const int quarter = warp & 3;
    const int group = (warp - 2) >> 2;
    uint32_t local_tile = 0;
    bool ok = true;
    constexpr int MINE = BN / 64;  // chunks of 32 columns: the two warp groups split them
    Epilogue<L::BLOCKS, MINE, 4> epilogue{staging, warp - 2, 0, 0, {}};
    const int c_begin = group * MINE, c_end = c_begin + MINE;
    for (int tile = pair; tile < items.count && ok; tile += num_pairs, ++local_tile) {
      int m_idx, n_idx;
      tile_coords(items.tile(tile), tiles_m, items.whole, g.group_m, &m_idx, &n_idx);
      const int m0 = m_idx * 256 + (int)rank * 128;
      const int n0 = n_idx * BN;
      const uint32_t buf = local_tile & 1;
      const uint32_t acc_phase = (local_tile >> 1) & 1;
      const int part = items.part(tile), row0 = m0 + quarter * 32;
      if (part <= 0) epilogue.begin(g, &map_aux, c_begin, c_end, n0, row0, lane);
      ok = mbar_wait_all(&acc_full[buf], acc_phase, g.error);
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * BN;
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[buf]), 0));
      };
      if (part >= 0) {  // 16 flags per part: the eight epilogue warps of either CTA
        const int split_tile = items.tile(tile) - items.whole, parts = items.splits - 1, tile_row = (int)rank * 128 + quarter * 32 + lane;
        float* parked = g.partials + (size_t)split_tile * parts * (256 * BN);
        unsigned* my_flags = g.split_flags + (size_t)split_tile * parts * 16 + rank * 8 + (warp - 2);
        if (part > 0) {
          park_tile<256>(taddr, c_begin, c_end, parked + (size_t)(part - 1) * (256 * BN), tile_row);
          release();
          raise_flag(my_flags + (part - 1) * 16, lane);
          continue;
        }
        if (!(ok = wait_flags(my_flags, parts, 16, lane, g.error))) break;
        fold_tile<256, 256 * BN>(taddr, c_begin, c_end, parked, parts, tile_row);
      }
      ok = epilogue.finish(taddr, c_begin, c_end, n0, row0, lane, g, &map_aux, &map_out, &map_pre, release);
    }
    drain_stores();
  }

  // ------------------------------------------------------------------ teardown
  // Neither CTA may leave (or free TMEM) while its partner can still signal its barriers or read its tiles.
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}


// ------------------------------------------------------------------------------------------ host
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encoder() {
  static std::atomic<EncodeTiled> known{nullptr};
  EncodeTiled fn = known.load(std::memory_order_relaxed);
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      known.store(fn = (EncodeTiled)p, std::memory_order_relaxed);
  }
  return fn;
}

thread_local char g_map_error[256] = "";

// A 2-D bf16 tensor map: `inner` contiguous elements per row, `outer` rows of `row_stride` elements.
int make_map(CUtensorMap* map, const void* ptr, long long inner, long long outer, long long row_stride, int box_inner, int box_outer,
             CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  // cuTensorMapEncodeTiled is a driver entry point: it needs this thread to have a current context, which a
  // thread that has so far only been handed cached allocations (an autograd worker) may not have yet.
  static thread_local bool context_ready = false;
  if (!context_ready) {
    cudaFree(nullptr);
    context_ready = true;
  }
  EncodeTiled enc = encoder();
  if (enc == nullptr) return -10;
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  cuuint64_t strides[1] = {(cuuint64_t)row_stride * 2};
  cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
  cuuint32_t elem[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    snprintf(g_map_error, sizeof(g_map_error), "cuTensorMapEncodeTiled -> %d (ptr %p, dims %lld x %lld, row stride %lld el, box %d x %d)",
             (int)r, ptr, inner, outer, row_stride, box_inner, box_outer);
  return r == CUDA_SUCCESS ? 0 : -11;
}

// The epilogue of this call, with the tensor maps of its TMA stores and loads: 32-row x 32-column bf16 blocks of out, of the kept
// gelu' factors and of what is added or multiplied (when gradients are accumulated, the output's old values).
int g_tma_store_enabled = 1;
int plan_epilogue(CUtensorMap* mo, CUtensorMap* mp, CUtensorMap* mx, void* out, void* aux_out, const void* aux_in, int M, int N, int ldc, int flags) {
  memset(mo, 0, sizeof(*mo));
  memset(mp, 0, sizeof(*mp));
  memset(mx, 0, sizeof(*mx));
  const int work = flags & (EPI_GELU | EPI_RESIDUAL | EPI_DGELU | EPI_ACCUMULATE);
  const int kind = work == 0 ? KIND_PLAIN : work == EPI_RESIDUAL || work == EPI_ACCUMULATE ? KIND_ADD : work == EPI_DGELU ? KIND_MUL
                   : work == EPI_GELU ? KIND_GELU : KIND_DIRECT;
  if (!g_tma_store_enabled || (flags & EPI_OUT_F32) || (ldc & 7) || ((uintptr_t)out & 15) || N < 64 || M < 32) return KIND_DIRECT;
  const bool keep_pre = (flags & EPI_GELU) && aux_out != nullptr;
  if (keep_pre && ((uintptr_t)aux_out & 15)) return KIND_DIRECT;
  if (make_map(mo, out, N, M, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B)) return KIND_DIRECT;
  if (keep_pre && make_map(mp, aux_out, N, M, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B)) return KIND_DIRECT;
  if ((kind == KIND_ADD || kind == KIND_MUL) &&
      make_map(mx, flags & EPI_ACCUMULATE ? out : aux_in, N, M, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B))
    return KIND_DIRECT;
  return kind;
}

tb::ErrorWord g_error;

template <int BM, int BN, bool A_MN, bool B_MN>
int launch_gemm(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo, const CUtensorMap& mp, const CUtensorMap& mx, const GemmArgs& g, int max_ctas,
                cudaStream_t stream) {
  auto kernel = k_gemm<BM, BN, A_MN, B_MN>;
  using L = SmemLayout<BM, BN>;
  static tb::SharedMemoryLimit limit;
  const cudaError_t e = limit.raise(kernel, L::TOTAL);
  if (e != cudaSuccess) return (int)e;
  const int out_tiles = ((g.M + BM - 1) / BM) * ((g.N + BN - 1) / BN);
  const int tiles = g.splits > 1 ? g.whole_tiles + (out_tiles - g.whole_tiles) * g.splits : out_tiles;
  const int sms = tb::sm_count();
  int ctas = tiles < sms ? tiles : sms;
  if (max_ctas > 0 && ctas > max_ctas) ctas = max_ctas;
  return (int)tb::launch(kernel, dim3(ctas), dim3(L::THREADS), L::TOTAL, stream, ma, mb, mo, mp, mx, g, GatherArgs{});
}


template <int BN, bool A_MN, bool B_MN, bool DEEP>
int launch_gemm_pair(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo, const CUtensorMap& mp, const CUtensorMap& mx, const GemmArgs& g,
                     int max_ctas, cudaStream_t stream) {
  auto kernel = k_gemm_pair<BN, A_MN, B_MN, DEEP>;
  using L = PairLayout<BN, DEEP>;
  static tb::SharedMemoryLimit limit;
  const cudaError_t e = limit.raise(kernel, L::TOTAL);
  if (e != cudaSuccess) return (int)e;
  static std::atomic<int> known_pairs{0};
  int max_pairs = known_pairs.load(std::memory_order_relaxed);
  if (max_pairs == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tb::sm_count() & ~1);
    cfg.blockDim = dim3(L::THREADS);
    cfg.dynamicSmemBytes = L::TOTAL;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = tb::sm_count() / 2;
    }
    max_pairs = n < tb::sm_count() / 2 ? n : tb::sm_count() / 2;
    known_pairs.store(max_pairs, std::memory_order_relaxed);
  }
  const int out_tiles = ((g.M + 255) / 256) * ((g.N + BN - 1) / BN);
  const int tiles = g.splits > 1 ? g.whole_tiles + (out_tiles - g.whole_tiles) * g.splits : out_tiles;
  int pairs = tiles < max_pairs ? tiles : max_pairs;
  if (max_ctas > 1 && pairs > max_ctas / 2) pairs = max_ctas / 2;
  return (int)tb::launch(kernel, dim3(2 * pairs), dim3(L::THREADS), L::TOTAL, stream, ma, mb, mo, mp, mx, g);
}

// Plans.  The CTAs (or CTA pairs) take output tiles round-robin; the last, partial round leaves SMs idle, so the tiles of
// that round ("tail") may have their reduction cut into parts that are spread over the idle SMs (GemmArgs).  A plan is made
// in two steps.
//
// 1. Which sums are cut, and where (plan_cut).  That order of summation is part of a product's result: single bf16 roundings
//    flip with it, and after 24 layers every gradient differs by about 1 %.  So it depends on the product's sizes and the
//    number of SMs alone, by a model that stays as it is when kernels get faster: a run gives the same bits before and after.
//
// 2. Tile shape (plan_gemm): among all shapes that make those very sums, the one with the least estimated time.  The estimate,
//    in microseconds, is
//        start-up + full rounds x (k-blocks x per-k-block + per-tile) + [tail: k-blocks per part x per-k-block + per-tile + fold]
//    with constants fitted to sweeps on B200 (bench/bench_gemm.py --sweep, CUDA-graph timing, cold L2) over 1024 - 16384
//    tokens and widths 768 - 2048.  What a k-block costs: a 256 x 256 pair tile feeds 256 x 256 x 64 multiply-adds to two tensor
//    pipes per 64 KB of operands and runs at the power limit (1620 - 1680 TFLOP/s from 10^11 flops on, cuBLAS 1450 - 1640);
//    the 128-row tiles move up to twice the bytes per flop and pay 0.22 - 0.37 us; the one-CTA 256 x 256 tile fills TMEM, so that
//    its epilogue cannot overlap the next tile.  Narrow tiles win where rounds are few: 1024 x 768 x 2304 takes 12.5 us on
//    pair 256 x 128 tiles, 17 on pair 256 x 256.  Folding parked partial tiles costs about 4 us for two parts, 1 us per part more
//    and 0.2 us per parked megabyte.
struct TileShape { int id, bm, bn; double start, per_kblock, per_tile; };
constexpr int PAIR = 512;  // bm of the CTA-pair kernel's 256-row tiles
constexpr TileShape SHAPES[6] = {{0, 256, 256, 4.5, 0.64, 3.3}, {1, 128, 256, 4.3, 0.37, 0.9},   {2, 128, 128, 4.3, 0.205, 0.7},
                                 {5, 128, 192, 4.3, 0.335, 0.8}, {3, PAIR, 256, 6.0, 0.345, 0.7}, {4, PAIR, 128, 4.8, 0.19, 0.9}};
constexpr int MAX_SPLITS = 8;
constexpr double FOLD_US = 3.0, FOLD_PART_US = 1.0, FOLD_US_PER_MB = 0.2;

// Tuning and test hooks (tb_gemm_force_tile / tb_gemm_force_splits): process-wide, read once per call into locals.
// Atomic so that a setter racing with a launch on another thread (an autograd worker) yields one value or the other.
std::atomic<int> g_forced_tile{-1};   // 0: 256x256, 1: 128x256, 2: 128x128, 3 / 4: CTA pair 256x256 / 256x128, 5: 128x192; -1: planned
std::atomic<int> g_forced_splits{0};  // > 0: that many k-parts for the tail (where the reduction is long enough); 0: planned

struct GemmPlan {
  int bm, bn, splits, whole_tiles;
  int rows() const { return bm == PAIR ? 256 : bm; }
  long long tiles(int M, int N) const { return (long long)((M + rows() - 1) / rows()) * ((N + bn - 1) / bn); }
  long long tail(int M, int N) const { return tiles(M, N) - whole_tiles; }
  long long workspace_bytes(int M, int N) const { return splits <= 1 ? 0 : tail(M, N) * (splits - 1) * rows() * bn * 4; }
  long long flag_words(int M, int N) const { return tail(M, N) * (splits - 1) * (bm == PAIR ? 16 : 8); }
};

// Every part gets at least two k-blocks and none is empty.
bool valid_splits(int k_blocks, int s) {
  const int per = (k_blocks + s - 1) / s;
  return s == 1 || (per >= 2 && (s - 1) * per < k_blocks);
}

// The plan whose sums every plan of this product makes: the tail of a one-CTA shape's tiles is cut where one round takes much
// longer than folding its parts.  The prices, fitted to early kernels, no longer say how long anything takes: they fix where
// the cuts are.
GemmPlan plan_cut(int M, int N, int K, int ctas) {
  struct { int bm, bn; double per_kblock, per_tile; } constexpr shapes[] = {{256, 256, 0.77, 5.3}, {128, 256, 0.43, 0.5}, {128, 128, 0.34, 0.6}, {128, 192, 0.41, 0.6}};
  const int k_blocks = (K + BK - 1) / BK;
  GemmPlan best{128, 128, 1, 0};
  double best_us = 1e300;
  for (const auto& t : shapes) {
    if (t.bn > 128 && N <= 128) continue;
    const long long tiles = GemmPlan{t.bm, t.bn, 1, 0}.tiles(M, N);
    const long long rounds = tiles / ctas, tail = tiles % ctas;
    for (int sp = 1; sp <= MAX_SPLITS; ++sp) {
      if (!valid_splits(k_blocks, sp) || (sp > 1 && (tail == 0 || tail * sp > ctas))) continue;
      double us = 5.0 + rounds * (k_blocks * t.per_kblock + t.per_tile);
      if (tail > 0) {
        const int per = (k_blocks + sp - 1) / sp;
        us += per * t.per_kblock + t.per_tile;
        if (sp > 1) us += 2.5 + 1.7 * (sp - 1) + 0.3 * (double)tail * (sp - 1) * t.bm * t.bn * 4 / 1e6;
      }
      if (us < best_us - 1e-9) {
        best_us = us;
        best = {t.bm, t.bn, sp, sp > 1 ? (int)(rounds * ctas) : 0};
      }
    }
  }
  return best;
}

// Do two plans add up every output element in the same order?  Whole tiles come first, column by column of tiles, so the uncut
// region is some full columns of the matrix and the upper rows of the tiles' next column.
bool same_sums(const GemmPlan& a, const GemmPlan& b, int M, int N) {
  if (a.splits != b.splits) return false;
  if (a.splits == 1) return true;
  struct Region { long long columns, rows, columns_with_rows; };
  auto region = [&](const GemmPlan& p) {
    const int tiles_m = (M + p.rows() - 1) / p.rows();
    const long long columns = (long long)(p.whole_tiles / tiles_m) * p.bn, rows = (long long)(p.whole_tiles % tiles_m) * p.rows();
    return Region{columns, rows, rows == 0 ? columns : columns + p.bn < N ? columns + p.bn : N};
  };
  const Region x = region(a), y = region(b);
  return x.columns == y.columns && x.rows == y.rows && x.columns_with_rows == y.columns_with_rows;
}

GemmPlan plan_gemm(int M, int N, int K, int ctas) {
  const int k_blocks = (K + BK - 1) / BK;
  const int forced_tile = g_forced_tile.load(std::memory_order_relaxed), forced_splits = g_forced_splits.load(std::memory_order_relaxed);
  const bool pinned = forced_tile >= 0 || forced_splits > 0;
  const GemmPlan cut = plan_cut(M, N, K, ctas);
  GemmPlan best{128, 128, 1, 0};
  double best_us = 1e300;
  for (const TileShape& t : SHAPES) {
    if (forced_tile >= 0 && forced_tile != t.id) continue;
    if (forced_tile < 0 && (t.bn > 128 && N <= 128)) continue;
    const int units = t.bm == PAIR ? ctas / 2 : ctas;
    if (units < 1) continue;
    const GemmPlan shape{t.bm, t.bn, 1, 0};
    const long long tiles = shape.tiles(M, N);
    const long long rounds = tiles / units, tail = tiles % units;
    const double whole_us = rounds * (k_blocks * t.per_kblock + t.per_tile);
    for (int sp = 1; sp <= MAX_SPLITS; ++sp) {
      if (!valid_splits(k_blocks, sp) || (sp > 1 && (tail == 0 || tail * sp > units))) continue;
      if (forced_splits > 0 && sp != forced_splits && tail > 0 && valid_splits(k_blocks, forced_splits) && tail * forced_splits <= units) continue;
      const GemmPlan plan{t.bm, t.bn, sp, sp > 1 ? (int)(rounds * units) : 0};
      if (!pinned && !same_sums(plan, cut, M, N)) continue;
      double us = t.start + whole_us;
      if (tail > 0) {
        const int per = (k_blocks + sp - 1) / sp;
        us += per * t.per_kblock + t.per_tile;
        if (sp > 1) us += FOLD_US + FOLD_PART_US * (sp - 1) + FOLD_US_PER_MB * (double)tail * (sp - 1) * shape.rows() * t.bn * 4 / 1e6;
      }
      if (us < best_us - 1e-9) {
        best_us = us;
        best = plan;
      }
    }
  }
  return best;
}

// Without a device (a build machine) the plan is the one a B200's 148 SMs would get.
int planned_sms() {
  const int n = tb::sm_count();
  return n > 0 ? n : 148;
}

// reciprocal2 as the GELU epilogue uses it, for comparisons with a division.
__global__ void k_reciprocals(const float* d, float* out, long long pairs) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pairs) return;
  const f32x2 minus_d[1] = {pair2(-d[2 * i], -d[2 * i + 1])};
  f32x2 r[1];
  reciprocal2(minus_d, r);
  split2(r[0], &out[2 * i], &out[2 * i + 1]);
}

// Flag words for split-K.
constexpr int SPLIT_FLAG_POOL = 1 << 16;
__device__ unsigned g_split_flags[2 * SPLIT_FLAG_POOL];
tb::WordPool g_flag_pool(SPLIT_FLAG_POOL);

}  // namespace

extern "C" void tb_note_launch(int n);

extern "C" {

// 0 while every GEMM wait so far has completed; 1 after one ran out.
int tb_gemm_error() { return g_error.raised(); }

// D[M,N] = op(A) . op(B) with bf16 operands, then the epilogue selected by `flags` (EpilogueFlags).
//   a_mn == 0: A is [M, K] with leading dimension lda (K contiguous); a_mn == 1: A is [K, M], lda (M contiguous).
//   b_mn == 0: B is [N, K] with leading dimension ldb (K contiguous); b_mn == 1: B is [K, N], ldb (N contiguous).
// Leading dimensions must be multiples of 8 elements and base pointers 16-byte aligned (TMA).
int tb_gemm_bf16(const void* A, const void* B, void* out, int M, int N, int K, int lda, int ldb, int ldc, int a_mn, int b_mn, int flags,
                 const void* bias, const void* aux_in, void* aux_out, int max_ctas, void* workspace, long long workspace_bytes,
                 cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda & 7) || (ldb & 7) || (((uintptr_t)A | (uintptr_t)B) & 15)) return -12;
  int* const error = g_error.device();
  if (error == nullptr) return -13;
  const int sms = tb::sm_count();
  const int ctas = max_ctas > 0 && max_ctas < sms ? max_ctas : sms;
  const GemmPlan plan = plan_gemm(M, N, K, ctas);
  const int BM = plan.bm, BN = plan.bn;
  int splits = plan.splits;
  const bool paired = BM == PAIR;  // a 256 x BN tile shared by a CTA pair: per CTA 128 rows of A, BN/2 rows of B
  unsigned* split_flags = nullptr;
  if (splits > 1) {
    const long long need = plan.workspace_bytes(M, N), words = plan.flag_words(M, N);
    if (workspace == nullptr || workspace_bytes < need || ((uintptr_t)workspace & 15) || words > SPLIT_FLAG_POOL) {
      splits = 1;  // no room to park partial tiles: compute unsplit (same result up to summation order)
    } else {
      const cudaError_t e = g_flag_pool.take(words, stream, &split_flags, [](void** at) { return cudaGetSymbolAddress(at, g_split_flags); });
      if (e != cudaSuccess) return (int)e;
    }
  }
  CUtensorMap ma, mb;
  int rc;
  if (!a_mn) rc = make_map(&ma, A, K, M, lda, 64, paired ? 128 : BM);
  else rc = make_map(&ma, A, M, K, lda, 64, 64);
  if (rc) return rc;
  if (!b_mn) rc = make_map(&mb, B, K, N, ldb, 64, paired ? BN / 2 : BN);
  else rc = make_map(&mb, B, N, K, ldb, 64, 64);
  if (rc) return rc;
  CUtensorMap mo, mp, mx;
  const int kind = plan_epilogue(&mo, &mp, &mx, out, aux_out, aux_in, M, N, ldc, flags);
  const int group_m = BM == 128 ? 8 : 4;  // 1024 rows
  GemmArgs g{M, N, K, ldc, flags, out, (const __nv_bfloat16*)bias, (const __nv_bfloat16*)aux_in, (__nv_bfloat16*)aux_out, error,
             splits, splits > 1 ? plan.whole_tiles : 0, (float*)workspace, split_flags, group_m, kind};
  tb_note_launch(1);
  const bool deep = K >= 32 * BK;
#define GO2(BN_) \
  do { \
    if (a_mn && b_mn) return launch_gemm_pair<BN_, true, true, true>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
    if (a_mn) return launch_gemm_pair<BN_, true, false, true>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
    if (!b_mn && deep) return launch_gemm_pair<BN_, false, false, true>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
    if (!b_mn) return launch_gemm_pair<BN_, false, false, false>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
    if (deep) return launch_gemm_pair<BN_, false, true, true>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
    return launch_gemm_pair<BN_, false, true, false>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
  } while (0)
  if (paired && BN == 256) GO2(256);
  if (paired) GO2(128);
#undef GO2
#define GO(BM_, BN_) \
  do { \
    if (!a_mn && !b_mn) return launch_gemm<BM_, BN_, false, false>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
    if (!a_mn && b_mn) return launch_gemm<BM_, BN_, false, true>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
    if (a_mn && b_mn) return launch_gemm<BM_, BN_, true, true>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
    return launch_gemm<BM_, BN_, true, false>(ma, mb, mo, mp, mx, g, max_ctas, stream); \
  } while (0)
  if (BM == 256) GO(256, 256);
  if (BN == 256) GO(128, 256);
  if (BN == 192) GO(128, 192);
  GO(128, 128);
#undef GO
}

// Bytes of workspace tb_gemm_bf16 wants for this problem (0: it will not split the reduction).  The caller allocates
// at least that much (any stream-ordered allocator will do: the kernel is done with it when it completes) and passes it.
long long tb_gemm_workspace_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  return plan_gemm(M, N, K, planned_sms()).workspace_bytes(M, N);
}

// What the planner picks: writes {BM (512: CTA pair), BN, parts the tail tiles are cut into, tiles computed whole}.
void tb_gemm_plan(int M, int N, int K, int* out4) {
  const GemmPlan plan = plan_gemm(M, N, K, planned_sms());
  out4[0] = plan.bm;
  out4[1] = plan.bn;
  out4[2] = plan.splits;
  out4[3] = plan.whole_tiles;
}

// Pins the number of k-parts (0: planned) / the tile shape (-1: planned) for every later call.  For tuning and tests.
void tb_gemm_force_splits(int n) { g_forced_splits.store(n, std::memory_order_relaxed); }

// out[M, N] = A[M, K] . W[N, K]^T (+ epilogue) where W is gathered by the kernel itself: rank q's shard (peer
// address shards[q]) holds bytes [shard_lo[q], shard_hi[q]) of the unit's flat buffer; W is the byte range
// [w_off, w_off + N*K*2) of it and is assembled in `full` (this GPU's copy) while the GEMM runs.
// tail_bytes: bytes right behind W in the flat buffer to fetch as well (the layer's bias; pass bias = full + w_off +
// N*K*2 then).  ready: one zero-initialised word per chunk (ceil((N*K*2 + tail_bytes) / chunk_bytes)); epoch: a value not used by an earlier
// call on the same words.  One cooperative launch; returns a CUDA error if the grid cannot be co-resident.
int tb_gemm_gathered(const void* A, void* out, int M, int N, int K, int lda, int ldc, int flags, const void* bias, const void* aux_in,
                     void* aux_out, void* const* shards, const long long* shard_lo, const long long* shard_hi, int n_ranks, void* full,
                     long long w_off, long long tail_bytes, void* ready, unsigned epoch, int chunk_bytes, int n_start,
                     cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda & 7) || (K & 7) || (w_off & 15) || (((uintptr_t)A | (uintptr_t)full) & 15) || n_ranks < 1 || n_ranks > 8) return -12;
  int* const error = g_error.device();
  if (error == nullptr) return -13;
  const int sms = tb::sm_count();
  // 256-row tiles (two MMAs per weight panel in shared memory: a third less operand traffic per flop) once the problem
  // has enough of them for every SM; 128-row tiles otherwise.  The weight panel is 256 columns wide in both.
  constexpr int BN = 256;
  const int tiles_n = (N + BN - 1) / BN;
  const bool tall = (long long)((M + 255) / 256) * tiles_n >= sms;
  const int BM = tall ? 256 : 128;
  CUtensorMap ma, mb;
  int rc = make_map(&ma, A, K, M, lda, 64, BM);
  if (rc) return rc;
  rc = make_map(&mb, (const char*)full + w_off, K, N, K, 64, BN);
  if (rc) return rc;
  CUtensorMap mo, mp, mx;
  const int kind = plan_epilogue(&mo, &mp, &mx, out, aux_out, aux_in, M, N, ldc, flags);
  GemmArgs g{M, N, K, ldc, flags, out, (const __nv_bfloat16*)bias, (const __nv_bfloat16*)aux_in, (__nv_bfloat16*)aux_out, error,
             1, 0, nullptr, nullptr, 1, kind};
  GatherArgs ga{};
  for (int q = 0; q < n_ranks; ++q) {
    ga.shard[q] = (const char*)shards[q];
    ga.shard_lo[q] = shard_lo[q];
    ga.shard_hi[q] = shard_hi[q];
  }
  ga.full = (char*)full;
  ga.w_off = w_off;
  ga.w_bytes = (long long)N * K * 2 + tail_bytes;
  ga.tail_bytes = tail_bytes;
  ga.ready = (uint32_t*)ready;
  ga.epoch = epoch;
  ga.n = n_ranks;
  ga.chunk_bytes = chunk_bytes;
  ga.n_start = ((n_start % tiles_n) + tiles_n) % tiles_n;
  const auto kernel = tall ? k_gemm<256, BN, false, false, true> : k_gemm<128, BN, false, false, true>;
  const int smem = tall ? SmemLayout<256, BN>::TOTAL : SmemLayout<128, BN>::TOTAL;
  static tb::SharedMemoryLimit limits[2];
  const cudaError_t e = limits[tall].raise(kernel, smem);
  if (e != cudaSuccess) return (int)e;
  const int tiles = ((M + BM - 1) / BM) * tiles_n;
  int ctas = tiles < sms ? tiles : sms;
  void* params[] = {(void*)&ma, (void*)&mb, (void*)&mo, (void*)&mp, (void*)&mx, (void*)&g, (void*)&ga};
  tb_note_launch(1);
  return (int)cudaLaunchCooperativeKernel((const void*)kernel, dim3(ctas), dim3(448), params, smem, stream);
}

void tb_gemm_force_tile(int which) { g_forced_tile.store(which, std::memory_order_relaxed); }

// 1 (default): bf16 outputs leave through TMA stores; 0: the epilogue warps store them.  For measurements.
void tb_gemm_tma_store(int on) { g_tma_store_enabled = on; }

// out[i] = 1 / d[i], i < n (even), by the GELU epilogue's own reciprocal.  For tests.
int tb_gemm_reciprocals(const float* d, float* out, long long n, cudaStream_t stream) {
  if (n < 2) return 0;
  k_reciprocals<<<(unsigned)((n / 2 + 255) / 256), 256, 0, stream>>>(d, out, n / 2);
  return (int)cudaGetLastError();
}

const char* tb_gemm_last_error() { return g_map_error; }

}  // extern "C"
