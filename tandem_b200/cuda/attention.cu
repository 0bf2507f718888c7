// Causal self-attention on tcgen05 / TMEM, forward and backward, over a packed qkv tensor.
//
// qkv is [B*T, 3*d] bf16 (q | k | v along the row, head h at columns h*HD .. h*HD+HD of each part), T a
// multiple of 128, HD 64 or 128.  One TMA tensor map over that matrix serves every tile load
// (cp.async.bulk.tensor.2d, 128-byte swizzle, no multicast): a 128-row x 64-column box is a K-major
// operand when the reduction runs over the head dimension (Q.K^T, dO.V^T) and, with the same bytes,
// an MN-major operand when it runs over the rows (P.V, P^T.dO, dS^T.Q, dS.K).
//
// Three warp-specialised kernels (one TMA producer warp, one MMA-issuing warp, four or eight element-wise warps):
//   k_attn_fwd_ws    two 128-query tiles per SM alternate on the tensor pipe; single pass, online softmax with a lazy
//                    rescale of the accumulator in TMEM; P stays in TMEM as the A operand of P.V
//   k_attn_bwd_dq    per query tile: S, dP -> dS (TMEM) -> dQ += dS.K; also produces delta = rowsum(dO * O)
//   k_attn_bwd_dkv   per key tile, transposed scores: P^T, dS^T (TMEM) -> dV += P^T.dO, dK += dS^T.Q
// Probabilities and score gradients never pass through shared memory, nothing is accumulated with atomics, and
// the results do not depend on scheduling.  Consecutive CTAs work on the same head so its K and V stay in L2.
//
// Every wait is bounded (tcgen05.cuh); on expiry the CTA raises the host-visible error word, frees its
// TMEM and returns.  The reference calls torch's scaled_dot_product_attention (tandem/model.py:43).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <atomic>

#include "f32x2.cuh"
#include "host_state.h"
#include "launch.cuh"
#include "operators.h"
#include "tcgen05.cuh"

extern "C" void tb_note_launch(int n);

namespace {

using namespace tc;

constexpr int TILE = 128;           // queries per CTA, keys per step
constexpr int STRIP = TILE * 128;   // bytes of one 128-row x 64-column bf16 strip (128-byte rows)

// Loads one [128 rows x HD cols] operand tile (HD/64 strips) whose first element is (row, col) of qkv.
template <int HD>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col, int row) {
#pragma unroll
  for (int s = 0; s < HD / 64; ++s) tma_load_2d(dst + s * STRIP, map, bar, col + s * 64, row);
}

// D[128, N] (+)= A[128, K=HD] . B[N=128, K=HD]^T with both operands K-major strips.
template <int HD>
__device__ __forceinline__ void mma_kmajor(uint32_t d_tmem, const uint8_t* a, const uint8_t* b, uint32_t idesc, bool accumulate) {
  const uint64_t a_desc = smem_desc(smem_u32(a), 16, 1024), b_desc = smem_desc(smem_u32(b), 16, 1024);
#pragma unroll
  for (int s = 0; s < HD / 64; ++s)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      mma_bf16(d_tmem, a_desc + ((s * STRIP + k * 32) >> 4), b_desc + ((s * STRIP + k * 32) >> 4), idesc,
               (accumulate || s > 0 || k > 0) ? 1u : 0u);
}

// ------------------------------------------------------------------------------------------ work lists
// Head dim 64 leaves shared memory and TMEM for the next tile's operands and accumulators, so its kernels run one CTA per place on the
// GPU, which takes item after item: the loads of the next item, its barriers' turns and its first scores are under way while the last one is
// finished.  (A CTA per item spent 2 to 3.5 us of its 5 to 6 outside the loop over tiles; dQ and dK/dV, us: 16 x 512, 12 heads
// 40.4 -> 29.5 and 47.1 -> 38.9; 32 x 1024, 16 heads 251 -> 176 and 296 -> 243.)  Head dim 128 fills an SM with one item; its
// grid has a CTA for each.
// An item is a tile of a head (NT = 2: two query tiles).  The tiles of a head take from one step to as many as it has tiles, so their order decides how evenly the
// GPU ends.  MANY: items come in groups of `per_group` heads, the longest tiles of all heads of a group first, so that the rounds end together, and few enough
// heads that what they share stays in L2; CTA c takes the c-th item of even rounds and the c-th from the end of odd ones.
// Otherwise CTA c has the c-th item: head by head, so that a head's K and V are read once from memory, but for the last group of
// heads, whose longest tiles come first (head by head to the end, the last CTAs ran alone for as long as a whole
// head takes: forward, dQ, dK/dV of 2 x 4096, 16 heads of 128 157, 212 and 252 us, now 131, 200 and 232; 3 x 2048 82, 118 and 130, now 68, 112
// and 120).
// Finding an item takes a few hundred cycles of divisions: the first is found while the CTA sets itself up, the next one by prefetch(), which
// every role calls where it would wait anyway.
struct WorkItem {
  int rank, head, b, h;  // rank 0: the longest tile of its head; head = b * H + h; head < 0: none
};
template <bool MANY>
struct WorkList {
  int tiles, all, per_group, H, round;  // tiles per head; heads in all, per group and per batch row
  WorkItem now, then;

  __device__ __forceinline__ WorkItem find(int at) const {
    WorkItem w;
    int first = all - per_group, size = per_group;  // the group's heads
    if (MANY) {
      if (at >= tiles * all) return {0, -1, 0, 0};
      first = at / (per_group * tiles) * per_group;
      size = all - first < per_group ? all - first : per_group;
    }
    if (MANY || at >= first * tiles) {
      const int in = at - first * tiles;
      w.rank = in / size;
      w.head = first + in - w.rank * size;
    } else {
      w.head = at / tiles;
      w.rank = at - w.head * tiles;
    }
    w.b = w.head / H;
    w.h = w.head - w.b * H;
    return w;
  }
  __device__ __forceinline__ WorkList(int tiles_, int heads, int H_, int heads_per_group) : tiles(tiles_), all(heads), per_group(heads_per_group), H(H_), round(0) {
    now = find(blockIdx.x);
  }
  __device__ __forceinline__ void prefetch() {
    if (!MANY) return;
    ++round;
    then = find(round * (int)gridDim.x + (round & 1 ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x));
  }
  __device__ __forceinline__ bool advance() {  // after prefetch(); false: that was the last item
    if (!MANY) return false;
    now = then;
    return now.head >= 0;
  }
};

// ------------------------------------------------------------------------------------------ forward, warp-specialised
// A CTA owns NT 128-query tiles of one head: two with head dim 128; one with head dim 64, where two such CTAs share an SM.
//   warp 0       TMA producer: the Q tiles once, then K_0, V_0, K_1, V_1, ... through a ring of tile slots
//   warp 1       MMA issuer (one elected thread): S_i = Q_i.K_j^T and O_i += P_i.V_j for the query tiles i in turn
//   warps 2-5    softmax of query tile 0: one thread per query row (= TMEM lane)
//   warps 6-9    softmax of query tile 1
// Single pass with an online softmax: a row keeps the maximum it is currently scaled by (m_used) and only rescales its
// accumulator row in TMEM (tcgen05.ld, multiply, tcgen05.st) when a new maximum exceeds it by more than 2^8; otherwise
// the probabilities simply run up to 256, which fp32 accumulation and bf16 probabilities absorb.
// Two tiles alternate on the tensor pipe: while the softmax threads of one tile work on S_i(j) (exponentials), the
// MMAs of the other tile run.  P stays in TMEM, as bf16 pairs, and is the A operand of a TMEM-sourced MMA (measured
// against staging P in shared memory: 198 vs 223 us at T = 2048, head dim 128).
// Head dim 128.  TMEM: S_0 [0,128)  S_1 [128,256)  O_0 [256,384)  O_1 [384,512); P_i lies over the first 64 columns of S_i.
//   The rescale needs no barrier of its own: S_i(j) is committed after O_i += P.V of step j-1 on the in-order tensor
//   pipe, and the next one is only issued after this row's thread has arrived on p_full.
// Head dim 64.  TMEM: S [0,128)  O [128,192)  P [192,256).  With a P of its own, S(j+1) is issued as soon as the softmax threads
//   have S(j) in registers, so that they never wait for scores; P(j) and the rescale of O wait for P.V of step j-1 (pv_done),
//   which is long over by the time the maxima are known.  256 columns and 113 KB let two CTAs share an SM.
//   Items follow one another in a CTA (WorkList): Q of the next one is on its way and its first scores are issued ahead of this one's
//   last P.V (us: 16 x 512, 12 heads 27.6 -> 23.5; 4 x 1024, 16 heads 28.5 -> 21.5; 1 x 8192, 16 heads 240 -> 195).
template <int HD, bool MANY>
struct Fwd2Smem {
  static constexpr int TILE_BYTES = (HD / 64) * STRIP;
  static constexpr int NT = HD == 64 ? 1 : 2;                        // query tiles
  static constexpr int THREADS = 64 + 128 * NT;
  static constexpr int BUFS = MANY ? 2 : 1;                         // sets of Q tiles
  static constexpr int Q = 0;
  static constexpr int RING = Q + BUFS * NT * TILE_BYTES;
  static constexpr int SLOTS = 5;                                   // K and V tiles in flight
  static constexpr int BARS = RING + SLOTS * TILE_BYTES;
  static constexpr int TOTAL = BARS + 256;
  static_assert(TOTAL <= (HD == 64 ? 113 : 227) * 1024, "shared memory of one SM");
};

template <int HD, bool MANY>
__global__ void __launch_bounds__(Fwd2Smem<HD, MANY>::THREADS, HD == 64 ? 2 : 1)
k_attn_fwd_ws(const __grid_constant__ CUtensorMap map, __nv_bfloat16* __restrict__ out, float* __restrict__ lse, int B, int T, int H,
              int d, float scale_log2e, int group_heads, int* error) {
  extern __shared__ __align__(1024) uint8_t fwd2_smem[];
  uint8_t* smem = fwd2_smem;
  if (smem_u32(smem) & 1023) {  // the swizzled tiles need 1024-byte alignment; nothing is allocated yet
    if (threadIdx.x == 0) {
      *error = 1;
      __threadfence_system();
    }
    return;
  }
  using L = Fwd2Smem<HD, MANY>;
  static_assert(!MANY || HD == 64, "two query tiles of head dim 128 leave no room for the next item");
  constexpr int TILE_BYTES = L::TILE_BYTES, SLOTS = L::SLOTS, BUFS = L::BUFS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t *q_full = bars, *s_full = bars + 2, *p_full = bars + 4, *o_full = bars + 6, *kv_full = bars + 8, *kv_empty = bars + 8 + SLOTS;
  uint64_t *s_read = bars + 8 + 2 * SLOTS, *pv_done = s_read + 2, *q_empty = pv_done + 2, *o_empty = q_empty + 2;
  uint32_t* holder = reinterpret_cast<uint32_t*>(o_empty + 1);
  constexpr bool OWN_P = HD == 64;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;  // warp: known to be uniform
  constexpr int NT = L::NT;
  // An item: NT query tiles of one head (NT = 2: always a CTA's only one).  Query tile i visits n_i key tiles.
  const int n_qt = T / TILE, n_groups = (n_qt + NT - 1) / NT;
  WorkList<MANY> work(n_groups, B * H, H, group_heads);
  const int qt0 = NT * (n_groups - 1 - work.now.rank), qt1 = qt0 + 1;
  const int n0 = qt0 + 1, n1 = NT == 2 && qt1 < n_qt ? qt1 + 1 : 0;
  const int n_steps = n1 > n0 ? n1 : n0;
  constexpr uint32_t TMEM_COLS = HD == 64 ? 256 : 512;
  constexpr uint32_t C_O = HD == 64 ? 128 : 256, C_P = 192;  // S_i at 128 * i; C_P: with OWN_P

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);  // one arrival per softmax warp of the tile
      mbar_init(&o_full[i], 1);
      mbar_init(&s_read[i], 4);
      mbar_init(&pv_done[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    mbar_init(o_empty, 4);
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tensormap(&map);
  }
  if (warp == 1) {
    tmem_alloc(holder, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *holder;
  tb::pdl_wait();  // set-up is done; everything below reads what earlier kernels wrote

  // Item number `it` of this CTA uses Q buffer it % BUFS for the (it / BUFS)-th time; steps (key tiles) are counted through all items.
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    bool ok = true;
    int it = 0, ld = 0;
    do {
      const int b = work.now.b, h = work.now.h, q0 = NT * (n_groups - 1 - work.now.rank), buf = it % BUFS;
      const int steps = MANY ? q0 + 1 : n_steps;
      if (MANY && !(ok = mbar_wait_all(&q_empty[buf], ((it / BUFS) & 1) ^ 1, error))) break;
      if (elect_one()) {
        mbar_expect_tx(&q_full[buf], TILE_BYTES);
        load_tile<HD>(smem + L::Q + buf * TILE_BYTES, &map, &q_full[buf], h * HD, b * T + q0 * TILE);
        if (n1) {
          mbar_expect_tx(&q_full[1], TILE_BYTES);
          load_tile<HD>(smem + L::Q + TILE_BYTES, &map, &q_full[1], h * HD, b * T + qt1 * TILE);
        }
      }
      work.prefetch();
      for (int end = ld + 2 * steps, first = ld; ld < end; ++ld) {  // load 2j: K_j, load 2j+1: V_j
        const int s = ld % SLOTS, j = (ld - first) >> 1, part = ld & 1;
        if (!(ok = mbar_wait_all(&kv_empty[s], ((ld / SLOTS) & 1) ^ 1, error))) break;
        if (elect_one()) {
          mbar_expect_tx(&kv_full[s], TILE_BYTES);
          load_tile<HD>(smem + L::RING + s * TILE_BYTES, &map, &kv_full[s], (1 + part) * d + h * HD, b * T + j * TILE);
        }
      }
      ++it;
    } while (ok && work.advance());
    tb::pdl_launch_dependents();  // all loads are under way
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc_s = instr_desc(128, 128, false, false);
    constexpr uint32_t idesc_o = instr_desc(128, HD, false, true);
    auto slot_of = [&](int ld) { return smem + L::RING + (ld % SLOTS) * TILE_BYTES; };
    auto wait_slot = [&](int ld) { return mbar_wait_all(&kv_full[ld % SLOTS], (ld / SLOTS) & 1, error); };
    auto issue_s = [&](int i, int j, int q) {  // S_i = Q_i . K_j^T, Q_i in place q
      mma_kmajor<HD>(tmem + i * 128, smem + L::Q + q * TILE_BYTES, slot_of(2 * j), idesc_s, false);
      mma_commit(&s_full[i]);
    };
    auto issue_pv = [&](int i, int j, bool first) {  // O_i (+)= P_i . V_j: eight steps of 16 keys; V is MN-major (head dim contiguous)
      const uint32_t tO = tmem + C_O + i * HD;
      const uint64_t v_desc = smem_desc(smem_u32(slot_of(2 * j + 1)), STRIP, 1024);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        mma_bf16_ts(tO, (OWN_P ? tmem + C_P : tmem + i * 128) + kk * 8, v_desc + kk * (2048 >> 4), idesc_o, (!first || kk > 0) ? 1u : 0u);  // 16 keys = 8 TMEM columns of P
    };
    bool ok = mbar_wait_all(&q_full[0], 0, error) && (!n1 || mbar_wait_all(&q_full[1], 0, error)) && wait_slot(0);
    if (ok) {
      tc_fence_after();
      if (elect_one()) {
        issue_s(0, 0, 0);
        if (n1) issue_s(1, 0, 1);
        mma_commit(&kv_empty[0]);  // K_0 is free once these have read it
        if (MANY && n0 == 1) mma_commit(&q_empty[0]);
      }
    }
    if constexpr (OWN_P) {
      int it = 0, step = 0, n = n0;
      while (ok) {
        const int buf = it % BUFS;
        work.prefetch();
        for (int j = 0; j < (MANY ? n - 1 : n); ++j, ++step) {
          if (MANY || j + 1 < n) {
            if (!(ok = wait_slot(2 * step + 2) && mbar_wait_all(&s_read[0], step & 1, error))) break;  // K_{j+1}; S(j) is in registers
            tc_fence_after();
            if (elect_one()) {
              issue_s(0, step + 1, buf);
              mma_commit(&kv_empty[(2 * step + 2) % SLOTS]);
              if (MANY && j + 2 == n) mma_commit(&q_empty[buf]);
            }
          }
          if (!(ok = wait_slot(2 * step + 1) && mbar_wait_all(&p_full[0], step & 1, error))) break;  // V_j; P(j) is in place, O rescaled if it had to be
          if (MANY && j == 0 && !(ok = mbar_wait_all(o_empty, (it & 1) ^ 1, error))) break;          // the last item's O has been read
          tc_fence_after();
          if (elect_one()) {
            issue_pv(0, step, j == 0);
            mma_commit(!MANY && j + 1 == n ? &o_full[0] : &pv_done[0]);
            mma_commit(&kv_empty[(2 * step + 1) % SLOTS]);
          }
        }
        if (!MANY || !ok) break;
        // the item's last step: ahead of its P.V the first scores of the next item
        const bool more = work.advance(), only = n == 1;
        if (more) {
          n = n_groups - work.now.rank;
          const int next = (it + 1) % BUFS;
          if (!(ok = mbar_wait_all(&q_full[next], ((it + 1) / BUFS) & 1, error) && wait_slot(2 * step + 2) && mbar_wait_all(&s_read[0], step & 1, error))) break;
          tc_fence_after();
          if (elect_one()) {
            issue_s(0, step + 1, next);
            mma_commit(&kv_empty[(2 * step + 2) % SLOTS]);
            if (n == 1) mma_commit(&q_empty[next]);
          }
        }
        if (!(ok = wait_slot(2 * step + 1) && mbar_wait_all(&p_full[0], step & 1, error))) break;
        if (only && !(ok = mbar_wait_all(o_empty, (it & 1) ^ 1, error))) break;
        tc_fence_after();
        if (elect_one()) {
          issue_pv(0, step, only);
          mma_commit(&o_full[0]);
          mma_commit(&kv_empty[(2 * step + 1) % SLOTS]);
        }
        if (!more) break;
        ++it, ++step;
      }
    } else {
      for (int j = 0; j < n_steps && ok; ++j) {
        if (!(ok = wait_slot(2 * j + 1))) break;                       // V_j
        if (j + 1 < n_steps && !(ok = wait_slot(2 * j + 2))) break;    // K_{j+1}
        tc_fence_after();
        for (int i = 0; i < NT && ok; ++i) {
          const int n_i = i == 0 ? n0 : n1;
          if (j >= n_i) continue;
          if (!(ok = mbar_wait_all(&p_full[i], j & 1, error))) break;  // P_i(j) is in place, O_i rescaled if it had to be
          tc_fence_after();
          if (elect_one()) {
            issue_pv(i, j, j == 0);
            if (j == n_i - 1) mma_commit(&o_full[i]);
            else issue_s(i, j + 1, i);
          }
        }
        if (!ok) break;
        if (elect_one()) {
          mma_commit(&kv_empty[(2 * j + 1) % SLOTS]);                      // V_j
          if (j + 1 < n_steps) mma_commit(&kv_empty[(2 * j + 2) % SLOTS]);  // K_{j+1}
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax (warps 2-5: tile 0, warps 6-9: tile 1)
    const int i = (warp - 2) >> 2;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;                      // query row within the tile = TMEM lane
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem + i * 128 + lane_base;
    const uint32_t tO = tmem + C_O + i * HD + lane_base;
    const uint32_t tP = OWN_P ? tmem + C_P + lane_base : tS;  // bf16: keys 2c, 2c+1 in column c
    bool ok = true;
    int it = 0, step = 0, pv = 0;  // pv: P.V products waited for
    do {
      const int n_i = MANY ? n_groups - work.now.rank : i == 0 ? n0 : n1;
      const int qt = MANY ? n_i - 1 : i == 0 ? qt0 : qt1;
      const int b = work.now.b, h = work.now.h;
      float m_used = -INFINITY, l = 0.f;  // m_used in raw score units
      for (int j = 0; j < n_i && ok; ++j, ++step) {
        if (!(ok = mbar_wait_all(&s_full[i], step & 1, error))) break;
        tc_fence_after();
        uint32_t raw[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, raw[c]);
        tmem_ld_wait();
        if (OWN_P) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_read[i]);
        }
        float mx = -INFINITY;
        if (j == qt) {  // the diagonal tile: keys beyond the query are masked
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (c * 32 + e > r) raw[c][e] = 0xff800000u;  // -inf
        }
        {
          // eight independent running maxima, two elements at a time: a single chain of dependent maxima would cost ~5 cycles each
          float part[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) part[e] = __uint_as_float(raw[0][e]);
#pragma unroll
          for (int e = 8; e < 120; e += 16)
#pragma unroll
            for (int u = 0; u < 8; ++u)
              part[u] = max3(part[u], __uint_as_float(raw[(e + u) >> 5][(e + u) & 31]), __uint_as_float(raw[(e + 8 + u) >> 5][(e + 8 + u) & 31]));
#pragma unroll
          for (int u = 0; u < 8; ++u) part[u] = fmaxf(part[u], __uint_as_float(raw[3][24 + u]));
          mx = max3(max3(part[0], part[1], part[2]), max3(part[3], part[4], part[5]), fmaxf(part[6], part[7]));
        }
        if (OWN_P && j > 0) {
          if (!(ok = mbar_wait_all(&pv_done[i], pv & 1, error))) break;
          ++pv;
          tc_fence_after();
        }
        if (j == 0) {
          m_used = mx;
        } else {
          const bool need = (mx - m_used) * scale_log2e > 8.f;
          if (__any_sync(0xffffffffu, need)) {  // rare after the first tiles: rescale this warp's accumulator rows
            const float f = need ? ex2_approx((m_used - mx) * scale_log2e) : 1.f;
            if (need) m_used = mx;
            l *= f;
#pragma unroll 1
            for (int c = 0; c < HD / 32; ++c) {
              uint32_t o[32];
              tmem_ld32(tO + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
              tmem_st32(tO + c * 32, o);
            }
            tmem_st_wait();
          }
        }
        const float mc = m_used * scale_log2e;
        const f32x2 scale2 = pair2(scale_log2e, scale_log2e), shift2 = pair2(-mc, -mc);
        f32x2 sums01 = pair2(0.f, 0.f), sums23 = sums01;  // four running sums: columns 0, 1, 2, 3 modulo 4
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {  // 64 keys at a time: 32 registers of bf16 pairs
          uint32_t pk[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int col = hh * 64 + 2 * e;
            float p0, p1;
            split2(fma2(pair2(__uint_as_float(raw[col >> 5][col & 31]), __uint_as_float(raw[col >> 5][(col & 31) + 1])), scale2, shift2), &p0, &p1);
            const f32x2 p = pair2(ex2_approx(p0), ex2_approx(p1));
            if (e & 1) sums23 = add2(sums23, p);
            else sums01 = add2(sums01, p);
            pk[e] = bf16_pair(p);
          }
          tmem_st32(tP + hh * 32, pk);  // head dim 128: over the first 64 columns of S
        }
        float sums[4];
        split2(sums01, &sums[0], &sums[1]);
        split2(sums23, &sums[2], &sums[3]);
        l += (sums[0] + sums[1]) + (sums[2] + sums[3]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[i]);
        if (j == 0) work.prefetch();
      }
      if (ok && n_i > 0) ok = mbar_wait_all(&o_full[i], it & 1, error);
      if (ok && n_i > 0) {
        tc_fence_after();
        const float inv_l = 1.f / l;
        const int q_idx = qt * TILE + r;
        __nv_bfloat16* o_row = out + (size_t)(b * T + q_idx) * d + h * HD;
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + c * 32, o);
          tmem_ld_wait();
          if (MANY && c + 1 == HD / 32) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_empty);
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            __nv_bfloat162 y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              y[e] = __floats2bfloat162_rn(__uint_as_float(o[v * 8 + 2 * e]) * inv_l, __uint_as_float(o[v * 8 + 2 * e + 1]) * inv_l);
            *reinterpret_cast<uint4*>(o_row + c * 32 + v * 8) = *reinterpret_cast<const uint4*>(y);
          }
        }
        lse[((size_t)b * H + h) * T + q_idx] = (m_used * scale_log2e + log2f(l)) * 0.69314718055994530942f;  // natural log
      }
      ++it;
    } while (ok && work.advance());
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------ backward, warp-specialised
// Two kernels, no atomics: k_attn_bwd_dq owns a tile of 128 queries and walks the key tiles at or below the
// diagonal (dQ accumulates in TMEM); k_attn_bwd_dkv owns a tile of 128 keys and walks the query tiles at or above it
// (dK and dV accumulate in TMEM).  Both recompute S and dP; results are deterministic.  Roles per CTA (320 threads):
// warp 0 TMA producer, warp 1 MMA issuer (one elected lane), warps 2-9 element-wise work, two threads per TMEM lane (warps
// w and w + 4 share a lane quarter and split the 128 columns).  Probabilities and dS never touch shared memory: they
// are written back to TMEM as bf16 pairs and feed the next MMA as its A operand.

__device__ __forceinline__ void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// ---- dQ.  Per key tile j <= qt:  S = Q.K_j^T, dP = dO.V_j^T (TMEM) -> dS = P * (dP - delta) * scale as bf16 in TMEM
// (two buffers) -> dQ += dS.K_j.  The S / dP MMAs of tile j+1 are issued as soon as the element-wise warps have pulled
// tile j into registers, so the tensor pipe works on j+1 while they compute dS(j).  The kernel also produces
// delta[row] = sum_c dO[row, c] * O[row, c] for its queries (needed here and by the dK/dV kernel, which runs after it).
// Head dim 64: items follow one another (WorkList); Q, dO, O and lse of the next one arrive meanwhile, and dQ alternates between two
// accumulators.  TMEM: S [0,128)  dP [128,256)  dQ [256,256+BUFS*HD)  dS buffers behind it, 64 columns each.
template <int HD, bool MANY>
struct BwdDqSmem {
  static constexpr int TILE_BYTES = (HD / 64) * STRIP;
  static constexpr int BUFS = MANY ? 2 : 1;
  static constexpr bool O_TILE = HD == 64;  // O and lse come with Q and dO; else the threads read them
  static constexpr int ITEM_BYTES = (O_TILE ? 3 : 2) * TILE_BYTES;  // Q, dO (, O)
  static constexpr int RING = BUFS * ITEM_BYTES;
  // K_j is read again by dQ += dS.K_j, V_j only by dP: with rings of their own V_j+2 is on its way as soon as the scores of
  // tile j are done.  In one ring of five slots (head dim 128) it waited for K_j's slot, 1500 of 3350 cycles per tile.
  static constexpr int K_SLOTS = HD == 128 ? 3 : 4, V_SLOTS = HD == 128 ? 2 : 3, SLOTS = K_SLOTS + V_SLOTS;
  static constexpr int DELTA = RING + SLOTS * TILE_BYTES;  // [2 halves][128 rows] floats
  static constexpr int LSE = DELTA + 1024;                 // [BUFS][128] floats
  static constexpr int BARS = LSE + BUFS * 512;
  static constexpr int TOTAL = BARS + 256;
  static_assert(TOTAL <= 227 * 1024, "shared memory of one SM");
};

template <int HD, bool MANY>
__global__ void __launch_bounds__(320, 1)
k_attn_bwd_dq(const __grid_constant__ CUtensorMap map_qkv, const __grid_constant__ CUtensorMap map_do, const __grid_constant__ CUtensorMap map_o,
              const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, const float* __restrict__ lse, float* __restrict__ delta_out,
              __nv_bfloat16* __restrict__ dqkv, int B, int T, int H, int d, float scale, int group_heads, int* error) {
  extern __shared__ __align__(1024) uint8_t dq_smem[];
  uint8_t* smem = dq_smem;
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) {
      *error = 1;
      __threadfence_system();
    }
    return;
  }
  using L = BwdDqSmem<HD, MANY>;
  constexpr int TILE_BYTES = L::TILE_BYTES, SLOTS = L::SLOTS, K_SLOTS = L::K_SLOTS, V_SLOTS = L::V_SLOTS;  // K's slots, then V's
  constexpr int BUFS = L::BUFS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t *item_full = bars /* [2] */, *item_empty = bars + 2 /* [2] */, *dq_full = bars + 4 /* [2] */, *dq_empty = bars + 6 /* [2] */,
           *sdp_full = bars + 8, *sdp_read = bars + 9, *ds_full = bars + 10 /* [2] */, *delta_full = bars + 12, *kv_full = bars + 13,
           *kv_empty = bars + 13 + SLOTS;
  uint32_t* holder = reinterpret_cast<uint32_t*>(bars + 13 + 2 * SLOTS);
  float* delta_sm = reinterpret_cast<float*>(smem + L::DELTA);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;  // warp: known to be uniform
  const int n_qt = T / TILE;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t C_S = 0, C_DP = 128, C_DQ = 256, C_DS = 256 + BUFS * HD;
  WorkList<MANY> work(T / TILE, B * H, H, group_heads);

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&item_full[i], 1);
      mbar_init(&item_empty[i], 1 + 8);  // the last MMA that reads Q and dO, and the element-wise warps
      mbar_init(&dq_full[i], 1);
      mbar_init(&dq_empty[i], 8);
      mbar_init(&ds_full[i], 8);
    }
    mbar_init(sdp_full, 1);
    mbar_init(sdp_read, 8);
    mbar_init(delta_full, 8);
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&kv_full[s], 1);
      mbar_init(&kv_empty[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tensormap(&map_qkv);
    prefetch_tensormap(&map_do);
    if (L::O_TILE) prefetch_tensormap(&map_o);
  }
  if (warp == 1) {
    tmem_alloc(holder, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *holder;
  tb::pdl_wait();  // set-up is done; everything below reads what earlier kernels wrote
  // Item number `it` of this CTA uses buffer it % BUFS for the (it / BUFS)-th time; steps (key tiles) are counted through all items.

  if (warp == 0) {
    bool ok = true;
    int step = 0, it = 0;
    do {
      const int qt = n_qt - 1 - work.now.rank, n = qt + 1, head = work.now.head, b = work.now.b, h = work.now.h, buf = it % BUFS;
      if (!(ok = mbar_wait_all(&item_empty[buf], ((it / BUFS) & 1) ^ 1, error))) break;
      if (elect_one()) {
        uint8_t* item = smem + buf * L::ITEM_BYTES;
        const int row = b * T + qt * TILE;
        mbar_expect_tx(&item_full[buf], L::ITEM_BYTES + (L::O_TILE ? 512 : 0));
        load_tile<HD>(item, &map_qkv, &item_full[buf], h * HD, row);
        load_tile<HD>(item + TILE_BYTES, &map_do, &item_full[buf], h * HD, row);
        if (L::O_TILE) {
          load_tile<HD>(item + 2 * TILE_BYTES, &map_o, &item_full[buf], h * HD, row);
          bulk_load_1d(smem + L::LSE + buf * 512, lse + (size_t)head * T + qt * TILE, 512, &item_full[buf]);
        }
      }
      work.prefetch();
      for (int j = 0; j < n && ok; ++j, ++step) {
        for (int part = 0; part < 2; ++part) {  // K_j, V_j: the order in which the slots come free
          const int s = part == 0 ? step % K_SLOTS : K_SLOTS + step % V_SLOTS, turn = part == 0 ? step / K_SLOTS : step / V_SLOTS;
          if (!(ok = mbar_wait_all(&kv_empty[s], (turn & 1) ^ 1, error))) break;
          if (elect_one()) {
            mbar_expect_tx(&kv_full[s], TILE_BYTES);
            load_tile<HD>(smem + L::RING + s * TILE_BYTES, &map_qkv, &kv_full[s], (1 + part) * d + h * HD, b * T + j * TILE);
          }
        }
      }
      ++it;
    } while (ok && work.advance());
    tb::pdl_launch_dependents();  // all loads are under way
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = instr_desc(128, 128, false, false);
    constexpr uint32_t idesc_dq = instr_desc(128, HD, false, true);
    auto k_of = [&](int step) { return smem + L::RING + (step % K_SLOTS) * TILE_BYTES; };
    auto v_of = [&](int step) { return smem + L::RING + (K_SLOTS + step % V_SLOTS) * TILE_BYTES; };
    auto wait_tiles = [&](int step) {
      return mbar_wait_all(&kv_full[step % K_SLOTS], (step / K_SLOTS) & 1, error) &&
             mbar_wait_all(&kv_full[K_SLOTS + step % V_SLOTS], (step / V_SLOTS) & 1, error);
    };
    auto issue_scores = [&](int step, int buf) {
      const uint8_t* item = smem + buf * L::ITEM_BYTES;
      mma_kmajor<HD>(tmem + C_S, item, k_of(step), idesc_s, false);                // S  = Q . K_j^T
      mma_kmajor<HD>(tmem + C_DP, item + TILE_BYTES, v_of(step), idesc_s, false);  // dP = dO . V_j^T
      mma_commit(sdp_full);
      mma_commit(&kv_empty[K_SLOTS + step % V_SLOTS]);  // V_j has no other reader
    };
    auto issue_dq = [&](int step, int buf, bool first) {  // dQ += dS . K_j: dS from TMEM (16 keys = 8 columns per step), K_j MN-major over the keys
      const uint64_t k_desc = smem_desc(smem_u32(k_of(step)), STRIP, 1024);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        mma_bf16_ts(tmem + C_DQ + buf * HD, tmem + C_DS + (step & 1) * 64 + kk * 8, k_desc + kk * (2048 >> 4), idesc_dq, (!first || kk > 0) ? 1u : 0u);
      mma_commit(&kv_empty[step % K_SLOTS]);
    };
    int it = 0, step = 0, n = n_qt - work.now.rank;
    bool ok = mbar_wait_all(&item_full[0], 0, error) && wait_tiles(0);
    if (ok) {
      tc_fence_after();
      if (elect_one()) {
        issue_scores(0, 0);
        if (n == 1) mma_commit(&item_empty[0]);
      }
    }
    // The scores of a step are issued ahead of dQ of the step before; across items, too.  (Steps within an item have a loop of their own: with one
    // loop for both, whose counters run through the items, head dim 128 took 9 % longer.)
    while (ok) {
      const int buf = it % BUFS;
      work.prefetch();
      for (int j = 0; j < (MANY ? n - 1 : n); ++j, ++step) {
        if (MANY || j + 1 < n) {
          if (!(ok = mbar_wait_all(sdp_read, step & 1, error))) break;  // this step's S and dP are in registers
          if (!(ok = wait_tiles(step + 1))) break;
          tc_fence_after();
          if (elect_one()) {
            issue_scores(step + 1, buf);
            if (MANY && j + 2 == n) mma_commit(&item_empty[buf]);
          }
        }
        if (!(ok = mbar_wait_all(&ds_full[step & 1], (step >> 1) & 1, error))) break;
        if (MANY && j == 0 && !(ok = mbar_wait_all(&dq_empty[buf], ((it / BUFS) & 1) ^ 1, error))) break;
        tc_fence_after();
        if (elect_one()) issue_dq(step, buf, j == 0);
      }
      if (!ok) break;
      if (!MANY) {
        if (elect_one()) mma_commit(&dq_full[0]);
        break;
      }
      const bool more = work.advance(), only = n == 1;
      if (more) {
        n = n_qt - work.now.rank;
        const int next = (it + 1) % BUFS;
        if (!(ok = mbar_wait_all(sdp_read, step & 1, error))) break;
        if (!(ok = mbar_wait_all(&item_full[next], ((it + 1) / BUFS) & 1, error) && wait_tiles(step + 1))) break;
        tc_fence_after();
        if (elect_one()) {
          issue_scores(step + 1, next);
          if (n == 1) mma_commit(&item_empty[next]);
        }
      }
      if (!(ok = mbar_wait_all(&ds_full[step & 1], (step >> 1) & 1, error))) break;
      if (only && !(ok = mbar_wait_all(&dq_empty[buf], ((it / BUFS) & 1) ^ 1, error))) break;
      tc_fence_after();
      if (elect_one()) {
        issue_dq(step, buf, only);
        mma_commit(&dq_full[buf]);
      }
      if (!more) break;
      ++it, ++step;
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const float c2 = scale * 1.4426950408889634f;
    bool ok = true;
    int step = 0, it = 0;
    do {
      const int qt = n_qt - 1 - work.now.rank, n = qt + 1, head = work.now.head, b = work.now.b, h = work.now.h, buf = it % BUFS;
      const int q_idx = qt * TILE + r;
      const size_t row = (size_t)b * T + q_idx;
      float neg_lse2;
      // delta for this row: each of the row's two threads sums half of the head dimension
      {
        constexpr int COLS = HD / 2;
        const __nv_bfloat16* a = o + row * d + h * HD + half * COLS;
        const __nv_bfloat16* g = d_o + row * d + h * HD + half * COLS;
        const uint8_t* item = smem + buf * L::ITEM_BYTES + r * 128;  // rows of 128 bytes, 16-byte chunks swizzled
        if (L::O_TILE) {
          if (!(ok = mbar_wait_all(&item_full[buf], (it / BUFS) & 1, error))) break;
          neg_lse2 = -reinterpret_cast<const float*>(smem + L::LSE + buf * 512)[r] * 1.4426950408889634f;
        } else {
          neg_lse2 = -lse[(size_t)head * T + q_idx] * 1.4426950408889634f;
        }
        float acc = 0.f;
#pragma unroll
        for (int c = 0; c < COLS; c += 8) {
          const int chunk = ((half * COLS + c) / 8) ^ (r & 7);
          const uint4 av = L::O_TILE ? *reinterpret_cast<const uint4*>(item + 2 * TILE_BYTES + chunk * 16) : *reinterpret_cast<const uint4*>(a + c);
          const uint4 gv = L::O_TILE ? *reinterpret_cast<const uint4*>(item + TILE_BYTES + chunk * 16) : *reinterpret_cast<const uint4*>(g + c);
          const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&av);
          const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&gv);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 x = __bfloat1622float2(a2[e]), y = __bfloat1622float2(g2[e]);
            acc = fmaf(x.x, y.x, acc);
            acc = fmaf(x.y, y.y, acc);
          }
        }
        delta_sm[half * TILE + r] = acc;
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(delta_full);
        if (L::O_TILE) mbar_arrive(&item_empty[buf]);
      }
      // The row's other thread has added its half.  (No warp writes again before all have read: a step takes an arrival of every one.)
      if (!(ok = mbar_wait_all(delta_full, it & 1, error))) break;
      const float delta = delta_sm[r] + delta_sm[TILE + r];
      if (half == 0) delta_out[(size_t)head * T + q_idx] = delta;
      for (int j = 0; j < n && ok; ++j, ++step) {
        if (!(ok = mbar_wait_all(sdp_full, step & 1, error))) break;
        tc_fence_after();
        uint32_t s[2][32], dp[2][32];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tmem_ld32(tmem + C_S + lane_base + half * 64 + c * 32, s[c]);
          tmem_ld32(tmem + C_DP + lane_base + half * 64 + c * 32, dp[c]);
        }
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(sdp_read);
        uint32_t pk[32];
        if (j == qt) {  // the diagonal tile: exp2(-inf) = 0 for keys beyond the query
#pragma unroll
          for (int col = 0; col < 64; ++col)
            if (half * 64 + col > r) s[col >> 5][col & 31] = 0xff800000u;
        }
        const f32x2 scale_log2e2 = pair2(c2, c2), shift2 = pair2(neg_lse2, neg_lse2), minus_delta2 = pair2(-delta, -delta), scale2 = pair2(scale, scale);
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const int c = (2 * e) >> 5, i = (2 * e) & 31;  // within this thread's 64 columns
          float p0, p1;
          split2(fma2(pair2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), scale_log2e2, shift2), &p0, &p1);
          const f32x2 over = add2(pair2(__uint_as_float(dp[c][i]), __uint_as_float(dp[c][i + 1])), minus_delta2);
          pk[e] = bf16_pair(mul2(mul2(pair2(ex2_approx(p0), ex2_approx(p1)), over), scale2));
        }
        tmem_st32(tmem + C_DS + (step & 1) * 64 + lane_base + half * 32, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ds_full[step & 1]);
        if (j == 0) work.prefetch();
      }
      if (!ok || !(ok = mbar_wait_all(&dq_full[buf], (it / BUFS) & 1, error))) break;
      tc_fence_after();
      constexpr int COLS = HD / 2;
      __nv_bfloat16* dq_row = dqkv + row * 3 * d + h * HD + half * COLS;
#pragma unroll 1
      for (int c = 0; c < COLS / 32; ++c) {
        uint32_t raw[32];
        tmem_ld32(tmem + C_DQ + buf * HD + lane_base + half * COLS + c * 32, raw);
        tmem_ld_wait();
        if (c + 1 == COLS / 32) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&dq_empty[buf]);
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint32_t y[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) y[e] = pack_bf16(__uint_as_float(raw[v * 8 + 2 * e]), __uint_as_float(raw[v * 8 + 2 * e + 1]));
          *reinterpret_cast<uint4*>(dq_row + c * 32 + v * 8) = *reinterpret_cast<const uint4*>(y);
        }
      }
      ++it;
    } while (work.advance());
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// ---- dK, dV.  Transposed scores, so that the thread that owns a KEY row produces P^T and dS^T rows, which are the A
// operands (M = keys) of the accumulating MMAs:  S^T = K.Q_i^T, dP^T = V.dO_i^T  ->  P^T = exp(S^T*scale - lse[q]) to
// TMEM (bf16)  ->  dV += P^T.dO_i;  dS^T = P^T * (dP^T - delta[q]) * scale to TMEM  ->  dK += dS^T.Q_i.
// lse and delta of the query tile travel with Q_i and dO_i in a stage (plain bulk copies onto the same barrier).
// Each half-warp pair of a lane writes its bf16 result over the first 32 columns of ITS OWN half of the fp32 tile it
// has just consumed (columns [0,32) and [64,96)), so no thread overwrites columns the other has yet to read.
// Head dim 64: items follow one another (WorkList), with K and V of the next one on their way and two sets of accumulators.
// TMEM: S^T [0,128)  dP^T [128,256)  dV and dK [256, 256 + BUFS * 2 * HD).
template <int HD, bool MANY>
struct BwdDkvSmem {
  static constexpr int TILE_BYTES = (HD / 64) * STRIP;
  static constexpr int BUFS = MANY ? 2 : 1;
  static constexpr int ITEM_BYTES = 2 * TILE_BYTES, STAGES_AT = BUFS * ITEM_BYTES;  // K, V
  static constexpr int STAGE_BYTES = 2 * TILE_BYTES + 1024;  // Q_i, dO_i, lse[128], delta[128]
  static constexpr int STAGES_FIT = (223 * 1024 - STAGES_AT) / STAGE_BYTES;
  static constexpr int STAGES = STAGES_FIT > 4 ? 4 : STAGES_FIT;
  static constexpr int BARS = STAGES_AT + STAGES * STAGE_BYTES;
  static constexpr int TOTAL = BARS + 256;
  static_assert(STAGES >= 2, "two query tiles must be in flight");
};

template <int HD, bool MANY>
__global__ void __launch_bounds__(320, 1)
k_attn_bwd_dkv(const __grid_constant__ CUtensorMap map_qkv, const __grid_constant__ CUtensorMap map_do, const float* __restrict__ lse,
               const float* __restrict__ delta, __nv_bfloat16* __restrict__ dqkv, int B, int T, int H, int d, float scale, int group_heads, int* error) {
  extern __shared__ __align__(1024) uint8_t dkv_smem[];
  uint8_t* smem = dkv_smem;
  if (smem_u32(smem) & 1023) {
    if (threadIdx.x == 0) {
      *error = 1;
      __threadfence_system();
    }
    return;
  }
  using L = BwdDkvSmem<HD, MANY>;
  constexpr int TILE_BYTES = L::TILE_BYTES, STAGES = L::STAGES, STAGE_BYTES = L::STAGE_BYTES;
  constexpr int BUFS = L::BUFS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t *kv_full = bars /* [2] */, *kv_empty = bars + 2 /* [2] */, *acc_full = bars + 4 /* [2] */, *acc_empty = bars + 6 /* [2] */, *s_full = bars + 8,
           *dp_full = bars + 9, *p_full = bars + 10, *ds_full = bars + 11, *st_full = bars + 12, *st_empty = bars + 12 + STAGES;
  uint32_t* holder = reinterpret_cast<uint32_t*>(bars + 12 + 2 * STAGES);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;  // warp: known to be uniform
  const int n_tiles = T / TILE;
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t C_S = 0, C_DP = 128, C_ACC = 256;  // dV of buffer i at C_ACC + i * 2 * HD, dK behind it
  WorkList<MANY> work(T / TILE, B * H, H, group_heads);

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 8);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, 8);
    mbar_init(ds_full, 8);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&st_full[s], 1);
      mbar_init(&st_empty[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tensormap(&map_qkv);
    prefetch_tensormap(&map_do);
  }
  if (warp == 1) {
    tmem_alloc(holder, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *holder;
  tb::pdl_wait();  // set-up is done; everything below reads what earlier kernels wrote
  auto stage_at = [&](int step) { return smem + L::STAGES_AT + (step % STAGES) * STAGE_BYTES; };
  // Item number `it` of this CTA uses buffer it % BUFS for the (it / BUFS)-th time; steps (query tiles) are counted through all items.
  // The longest tile of a head is key tile 0, which visits every query tile.

  if (warp == 0) {
    bool ok = true;
    int step = 0, it = 0;
    do {
      const int kt = work.now.rank, head = work.now.head, b = work.now.b, h = work.now.h, buf = it % BUFS;
      if (!(ok = mbar_wait_all(&kv_empty[buf], ((it / BUFS) & 1) ^ 1, error))) break;
      if (elect_one()) {
        uint8_t* item = smem + buf * L::ITEM_BYTES;
        mbar_expect_tx(&kv_full[buf], L::ITEM_BYTES);
        load_tile<HD>(item, &map_qkv, &kv_full[buf], d + h * HD, b * T + kt * TILE);
        load_tile<HD>(item + TILE_BYTES, &map_qkv, &kv_full[buf], 2 * d + h * HD, b * T + kt * TILE);
      }
      work.prefetch();
      for (int i = kt; i < n_tiles; ++i, ++step) {
        const int s = step % STAGES;
        if (!(ok = mbar_wait_all(&st_empty[s], ((step / STAGES) & 1) ^ 1, error))) break;
        if (elect_one()) {
          uint8_t* st = stage_at(step);
          mbar_expect_tx(&st_full[s], STAGE_BYTES);
          load_tile<HD>(st, &map_qkv, &st_full[s], h * HD, b * T + i * TILE);
          load_tile<HD>(st + TILE_BYTES, &map_do, &st_full[s], h * HD, b * T + i * TILE);
          const size_t stat0 = (size_t)head * T + (size_t)i * TILE;
          bulk_load_1d(st + 2 * TILE_BYTES, lse + stat0, 512, &st_full[s]);
          bulk_load_1d(st + 2 * TILE_BYTES + 512, delta + stat0, 512, &st_full[s]);
        }
      }
      ++it;
    } while (ok && work.advance());
    tb::pdl_launch_dependents();  // all loads are under way
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = instr_desc(128, 128, false, false);
    constexpr uint32_t idesc_acc = instr_desc(128, HD, false, true);
    // bf16 A operand written over an fp32 tile: keys k-step kk sits at columns (kk / 4) * 64 + (kk % 4) * 8
    auto a_cols = [](int kk) { return (uint32_t)((kk >> 2) * 64 + (kk & 3) * 8); };
    auto issue_s = [&](int step, int buf) {  // S^T = K . Q_i^T
      mma_kmajor<HD>(tmem + C_S, smem + buf * L::ITEM_BYTES, stage_at(step), idesc_s, false);
      mma_commit(s_full);
    };
    auto issue_dp = [&](int step, int buf) {  // dP^T = V . dO_i^T
      mma_kmajor<HD>(tmem + C_DP, smem + buf * L::ITEM_BYTES + TILE_BYTES, stage_at(step) + TILE_BYTES, idesc_s, false);
      mma_commit(dp_full);
    };
    auto issue_dv = [&](int step, int buf, bool first) {  // dV += P^T . dO_i (16 queries per step; dO_i MN-major over the queries)
      const uint64_t do_desc = smem_desc(smem_u32(stage_at(step)) + TILE_BYTES, STRIP, 1024);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        mma_bf16_ts(tmem + C_ACC + buf * 2 * HD, tmem + C_S + a_cols(kk), do_desc + kk * (2048 >> 4), idesc_acc, (!first || kk > 0) ? 1u : 0u);
    };
    auto issue_dk = [&](int step, int buf, bool first) {  // dK += dS^T . Q_i
      const uint64_t q_desc = smem_desc(smem_u32(stage_at(step)), STRIP, 1024);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        mma_bf16_ts(tmem + C_ACC + buf * 2 * HD + HD, tmem + C_DP + a_cols(kk), q_desc + kk * (2048 >> 4), idesc_acc, (!first || kk > 0) ? 1u : 0u);
      mma_commit(&st_empty[step % STAGES]);  // Q_i, dO_i (and its lse / delta, read before ds_full) are done with
    };
    auto wait_stage = [&](int step) { return mbar_wait_all(&st_full[step % STAGES], (step / STAGES) & 1, error); };
    int it = 0, step = 0, n = n_tiles - work.now.rank;
    bool ok = mbar_wait_all(&kv_full[0], 0, error) && wait_stage(0);
    if (ok) {
      tc_fence_after();
      if (elect_one()) {
        issue_s(0, 0);
        issue_dp(0, 0);
        if (n == 1) mma_commit(&kv_empty[0]);
      }
    }
    // S^T of the next step is issued behind dV of this one and dP^T behind its dK; across items, too.
    while (ok) {
      const int buf = it % BUFS;
      work.prefetch();
      for (int t = 0; t < (MANY ? n - 1 : n); ++t, ++step) {
        if (!(ok = mbar_wait_all(p_full, step & 1, error))) break;
        if (MANY && t == 0 && !(ok = mbar_wait_all(&acc_empty[buf], ((it / BUFS) & 1) ^ 1, error))) break;
        tc_fence_after();
        if (elect_one()) issue_dv(step, buf, t == 0);
        if (MANY || t + 1 < n) {
          if (!(ok = wait_stage(step + 1))) break;
          tc_fence_after();
          if (elect_one()) issue_s(step + 1, buf);
        }
        if (!(ok = mbar_wait_all(ds_full, step & 1, error))) break;
        tc_fence_after();
        if (elect_one()) {
          issue_dk(step, buf, t == 0);
          if (MANY || t + 1 < n) issue_dp(step + 1, buf);
          if (MANY && t + 2 == n) mma_commit(&kv_empty[buf]);
        }
      }
      if (!ok) break;
      if (!MANY) {
        if (elect_one()) mma_commit(&acc_full[0]);
        break;
      }
      const bool more = work.advance(), only = n == 1;
      const int next = (it + 1) % BUFS;
      if (!(ok = mbar_wait_all(p_full, step & 1, error))) break;
      if (only && !(ok = mbar_wait_all(&acc_empty[buf], ((it / BUFS) & 1) ^ 1, error))) break;
      tc_fence_after();
      if (elect_one()) issue_dv(step, buf, only);
      if (more) {
        n = n_tiles - work.now.rank;
        if (!(ok = mbar_wait_all(&kv_full[next], ((it + 1) / BUFS) & 1, error) && wait_stage(step + 1))) break;
        tc_fence_after();
        if (elect_one()) issue_s(step + 1, next);
      }
      if (!(ok = mbar_wait_all(ds_full, step & 1, error))) break;
      tc_fence_after();
      if (elect_one()) {
        issue_dk(step, buf, only);
        mma_commit(&acc_full[buf]);
        if (more) {
          issue_dp(step + 1, next);
          if (n == 1) mma_commit(&kv_empty[next]);
        }
      }
      if (!more) break;
      ++it, ++step;
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;  // key row within the tile
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const float c2 = scale * 1.4426950408889634f;
    bool ok = true;
    int step = 0, it = 0;
    do {
      const int kt = work.now.rank, b = work.now.b, h = work.now.h, buf = it % BUFS;
      for (int i = kt; i < n_tiles && ok; ++i, ++step) {
        const float* stat = reinterpret_cast<const float*>(stage_at(step) + 2 * TILE_BYTES) + half * 64;  // lse, then (+128) delta
        if (!(ok = mbar_wait_all(&st_full[step % STAGES], (step / STAGES) & 1, error))) break;  // lse / delta have landed
        if (!(ok = mbar_wait_all(s_full, step & 1, error))) break;
        tc_fence_after();
        const float4* lse4 = reinterpret_cast<const float4*>(stat);
        const float4* delta4 = reinterpret_cast<const float4*>(stat + 128);
        const f32x2 minus_log2e2 = pair2(-1.4426950408889634f, -1.4426950408889634f), scale_log2e2 = pair2(c2, c2);
        f32x2 p[32];
        {
          uint32_t s[2][32], pk[32];
          tmem_ld32(tmem + C_S + lane_base + half * 64, s[0]);
          tmem_ld32(tmem + C_S + lane_base + half * 64 + 32, s[1]);
          tmem_ld_wait();
          auto probabilities = [&](bool diagonal) {
  #pragma unroll
            for (int q = 0; q < 16; ++q) {
              const float4 l4 = lse4[q];
  #pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int e = 2 * q + u, c = (2 * e) >> 5, k = (2 * e) & 31;
                const f32x2 shift = mul2(minus_log2e2, u == 0 ? pair2(l4.x, l4.y) : pair2(l4.z, l4.w));
                float x0, x1;
                split2(fma2(pair2(__uint_as_float(s[c][k]), __uint_as_float(s[c][k + 1])), scale_log2e2, shift), &x0, &x1);
                x0 = ex2_approx(x0), x1 = ex2_approx(x1);
                if (diagonal) {
                  x0 = r > half * 64 + 2 * e ? 0.f : x0;
                  x1 = r > half * 64 + 2 * e + 1 ? 0.f : x1;
                }
                p[e] = pair2(x0, x1);
                pk[e] = bf16_pair(p[e]);
              }
            }
          };
          // In the diagonal tile nothing of a query reaches the keys after it, not even the NaN of one whose sum is NaN.
          if (i == kt) probabilities(true);
          else probabilities(false);
          tmem_st32(tmem + C_S + lane_base + half * 64, pk);
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
        if (i == kt) work.prefetch();
        if (!(ok = mbar_wait_all(dp_full, step & 1, error))) break;
        tc_fence_after();
        {
          uint32_t dp[2][32], pk[32];
          tmem_ld32(tmem + C_DP + lane_base + half * 64, dp[0]);
          tmem_ld32(tmem + C_DP + lane_base + half * 64 + 32, dp[1]);
          tmem_ld_wait();
          const f32x2 scale2 = pair2(scale, scale), minus_one2 = pair2(-1.f, -1.f);
  #pragma unroll
          for (int q = 0; q < 16; ++q) {
            const float4 d4 = delta4[q];
  #pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int e = 2 * q + u, c = (2 * e) >> 5, k = (2 * e) & 31;
              const f32x2 dp2 = pair2(__uint_as_float(dp[c][k]), __uint_as_float(dp[c][k + 1]));
              const f32x2 over = fma2(u == 0 ? pair2(d4.x, d4.y) : pair2(d4.z, d4.w), minus_one2, dp2);  // dP - delta
              pk[e] = bf16_pair(mul2(mul2(p[e], over), scale2));
            }
          }
          tmem_st32(tmem + C_DP + lane_base + half * 64, pk);
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full);
      }
      if (!ok || !(ok = mbar_wait_all(&acc_full[buf], (it / BUFS) & 1, error))) break;
      tc_fence_after();
      constexpr int COLS = HD / 2;
      __nv_bfloat16* dk = dqkv + ((size_t)b * T + kt * TILE + r) * 3 * d + d + h * HD + half * COLS;
      __nv_bfloat16* dv = dk + d;
#pragma unroll 1
      for (int part = 0; part < 2; ++part) {
        __nv_bfloat16* dst = part == 0 ? dv : dk;
        const uint32_t src = tmem + C_ACC + (buf * 2 + part) * HD + lane_base + half * COLS;
#pragma unroll 1
        for (int c = 0; c < COLS / 32; ++c) {
          uint32_t raw[32];
          tmem_ld32(src + c * 32, raw);
          tmem_ld_wait();
          if (part == 1 && c + 1 == COLS / 32) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
          }
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint32_t y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = pack_bf16(__uint_as_float(raw[v * 8 + 2 * e]), __uint_as_float(raw[v * 8 + 2 * e + 1]));
            *reinterpret_cast<uint4*>(dst + c * 32 + v * 8) = *reinterpret_cast<const uint4*>(y);
          }
        }
      }
      ++it;
    } while (work.advance());
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int make_map(CUtensorMap* map, const void* ptr, long long cols, long long rows, long long row_stride) {
  static thread_local bool context_ready = false;  // the driver entry point below needs a current context in this thread
  if (!context_ready) {
    cudaFree(nullptr);
    context_ready = true;
  }
  static std::atomic<EncodeTiled> known{nullptr};
  EncodeTiled enc = known.load(std::memory_order_relaxed);
  if (enc == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      return -10;
    known.store(enc = (EncodeTiled)p, std::memory_order_relaxed);
  }
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)row_stride * 2};
  cuuint32_t box[2] = {64, 128};
  cuuint32_t elem[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? 0 : -11;
}

tb::ErrorWord g_error;

// Places for one CTA per SM.
int sm_count() {
  const int n = tb::sm_count();
  return n > 0 ? n : 148;
}

// WorkList: heads per group.  CTAs that take many items take the same number each, so the groups are as long as L2 allows (eight
// rounds; 1 x 8192, 16 heads, dK/dV: four rounds 355 us, eight 329).  Of CTAs with one item the GPU starts another whenever one ends, so
// only the last items have to be sorted: three rounds' worth (one: 2 x 8192, 16 heads of 128, dK/dV 880 us, two 850, three 837, four 863).
int group_heads(int tiles, int heads, bool many) {
  if (!many && tiles * heads <= sm_count()) return 1;  // all start at once; neighbours that share a head read it once
  const int want = ((many ? 8 : 3) * sm_count() + tiles - 1) / tiles;
  return want < heads ? want : heads;
}

}  // namespace

extern "C" {

int tb_attn_error() { return g_error.raised(); }

// out[B*T, d] = causal softmax(q k^T / sqrt(HD)) v per head; lse[B, H, T] (fp32) kept for backward.
int tb_attn_fwd(const void* qkv, void* out, float* lse, int B, int T, int H, int HD, cudaStream_t stream) {
  if (T % TILE || (HD != 64 && HD != 128)) return -21;
  int* const error = g_error.device();
  if (error == nullptr) return -13;
  const int d = H * HD;
  CUtensorMap map;
  int rc = make_map(&map, qkv, 3LL * d, (long long)B * T, 3LL * d);
  if (rc) return rc;
  const float scale_log2e = 1.4426950408889634f / sqrtf((float)HD);
  const int tiles = HD == 64 ? 1 : 2;
  const long long items = (long long)((T / TILE + tiles - 1) / tiles) * H * B;
  const bool many = HD == 64 && items > 2 * sm_count();  // two CTAs share an SM
  const int group = group_heads((T / TILE + tiles - 1) / tiles, H * B, many);
  const unsigned ctas = (unsigned)(many ? 2 * sm_count() : items);
  tb_note_launch(1);
#define LAUNCH_FWD(HD_, MANY_) \
  do { \
    using L = Fwd2Smem<HD_, MANY_>; \
    static tb::SharedMemoryLimit limit; \
    const cudaError_t e = limit.raise(k_attn_fwd_ws<HD_, MANY_>, L::TOTAL); \
    if (e != cudaSuccess) return (int)e; \
    return (int)tb::launch(k_attn_fwd_ws<HD_, MANY_>, dim3(ctas), dim3(L::THREADS), L::TOTAL, stream, map, (__nv_bfloat16*)out, lse, B, T, H, d, scale_log2e, \
                           group, error); \
  } while (0)
  if (HD == 128) LAUNCH_FWD(128, false);
  if (many) LAUNCH_FWD(64, true);
  LAUNCH_FWD(64, false);
#undef LAUNCH_FWD
}

// dqkv[B*T, 3d] from qkv, out, d_out, lse.  delta: fp32 [B*H*T], written by the dQ kernel and read by the dK/dV kernel.
int tb_attn_bwd(const void* qkv, const void* out, const void* d_out, const float* lse, void* dqkv, float* delta, int B, int T, int H, int HD,
                cudaStream_t stream) {
  if (T % TILE || (HD != 64 && HD != 128)) return -21;
  int* const error = g_error.device();
  if (error == nullptr) return -13;
  const int d = H * HD;
  const long long rows = (long long)B * T;
  CUtensorMap map_qkv, map_do, map_o;
  int rc = make_map(&map_qkv, qkv, 3LL * d, rows, 3LL * d);
  if (rc) return rc;
  rc = make_map(&map_do, d_out, d, rows, d);
  if (rc) return rc;
  rc = make_map(&map_o, out, d, rows, d);
  if (rc) return rc;
  const float scale = 1.f / sqrtf((float)HD);
  const long long items = (long long)(T / TILE) * H * B;
  // Where every item has an SM to itself the kernel for one item is 0.3 to 0.8 us faster (2 x 512, 12 heads: dK/dV 10.7 / 11.5 us).
  const bool many = HD == 64 && items > sm_count();
  const int group = group_heads(T / TILE, H * B, many);
  const unsigned ctas = (unsigned)(many ? sm_count() : items);
  tb_note_launch(2);
#define LAUNCH_BWD(HD_, MANY_) \
  do { \
    static tb::SharedMemoryLimit dq_limit, dkv_limit; \
    cudaError_t e = dq_limit.raise(k_attn_bwd_dq<HD_, MANY_>, BwdDqSmem<HD_, MANY_>::TOTAL); \
    if (e == cudaSuccess) e = dkv_limit.raise(k_attn_bwd_dkv<HD_, MANY_>, BwdDkvSmem<HD_, MANY_>::TOTAL); \
    if (e != cudaSuccess) return (int)e; \
    e = tb::launch(k_attn_bwd_dq<HD_, MANY_>, dim3(ctas), dim3(320), BwdDqSmem<HD_, MANY_>::TOTAL, stream, map_qkv, map_do, map_o, \
                               (const __nv_bfloat16*)out, (const __nv_bfloat16*)d_out, lse, delta, (__nv_bfloat16*)dqkv, B, T, H, d, scale, group, error); \
    if (e != cudaSuccess) return (int)e; \
    return (int)tb::launch(k_attn_bwd_dkv<HD_, MANY_>, dim3(ctas), dim3(320), BwdDkvSmem<HD_, MANY_>::TOTAL, stream, map_qkv, map_do, lse, (const float*)delta, \
                           (__nv_bfloat16*)dqkv, B, T, H, d, scale, group, error); \
  } while (0)
  if (HD == 128) LAUNCH_BWD(128, false);
  if (many) LAUNCH_BWD(64, true);
  LAUNCH_BWD(64, false);
#undef LAUNCH_BWD
}

}  // extern "C"
