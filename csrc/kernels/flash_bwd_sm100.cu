// Flash attention backward for sm_100a (head_dim 128 or 64, bf16, causal or full, GQA), in three kernels:
//
//   delta   : delta[b,h,s] = sum_d dO * O                                   (row kernel)
//   dQ      : 128 query rows at a time; loops over key tiles:
//                S = Q K^T, dP = dO V^T (tcgen05, TMEM) -> dS = P o (dP - delta) (bf16, written over dP in TMEM) -> dQ += dS K
//   dK / dV : one CTA per 128 keys of one KV head; loops over the query heads of its group and 128-row query tiles:
//                S^T = K Q^T, dP^T = V dO^T -> P^T, dS^T (bf16, in TMEM) -> dV += P^T dO, dK += dS^T Q
// Both MMA kernels recompute the probabilities from the saved log-sum-exp, keep their output accumulators in tensor
// memory for the whole loop and never use atomics, so results are deterministic. A Q / dO / K / V tile sits in shared
// memory once and serves two products through two descriptors (K-major for the score products, MN-major for the
// gradient products). The gradient products read their A operand (P^T, dS^T, dS) from tensor memory, where the softmax
// threads leave it with tcgen05.st: with both operands in shared memory the operand fetch (about 95 bytes per cycle
// measured against 128 needed), not the tensor pipe, set the pace. No reduction crosses the softmax threads: the row statistics
// come from the forward pass and the delta kernel.
//
// Replaces the reference's attention template backward (src/dew/nn/kernels/templates/attention_mosaic_dkv.py,
// attention_mosaic_dq.py), which it records as 6-9x slower than cuDNN on B200 (src/dew/nn/attention_kernels.py:772-796).
#include "../common/ptx.cuh"
#include "../common/tmap.h"
#include "../common/attn_variant.cuh"

namespace dewb {
namespace flashbwd {

constexpr int SOFTMAX_WARPS = 16, THREADS = 640;       // four softmax threads per TMEM lane, a TMA warp, an MMA warp, two that only complete its group of four
constexpr int TMA_WARP = 16, MMA_WARP = 17;
constexpr int COLS = 32;                               // columns of a 128 x 128 tile that a softmax thread has
// Registers a thread: 96 at the launch (20 warps on four schedulers), then moved to the softmax.
constexpr int SOFTMAX_REGS = 104, ISSUE_REGS = 64;
static_assert(4 * SOFTMAX_REGS + ISSUE_REGS <= 5 * 96, "an increase past what the block was launched with never ends");
constexpr float LOG2E = 1.4426950408889634f;
using attn::Variant;

// A capped score is cap * tanh(x), x = score / cap.  With e = e^(-2 |x|) and u = 1 / (1 + e) the tangent is (1 - e) u with the sign of x, and its derivative 4 e u^2: one exponential
// and one reciprocal for both, and a derivative that is as good where it is small (with 1 - tanh^2 of a second pair in dK / dV the backward of 8192 tokens, 4 heads of 128 over
// one, took 1273 us, 995 now).  `twice`: 2 log2(e) x / score.
__device__ __forceinline__ float capped(uint32_t score, float twice, float& slope) {
  const float x = __uint_as_float(score) * twice, e = fast_exp2(-fabsf(x)), u = __fdividef(1.f, 1.f + e);
  slope = 4.f * e * u * u;
  return copysignf((1.f - e) * u, x);
}

// ---------------------------------------------------------------------------------------------------------------
// delta[b,h,s] = sum_d dO * O.  Bound by the read of dO and O.  A block takes ROWS consecutive positions of one head; D / 8 lanes share a row with one 16-byte
// load of each operand apiece, and every lane has ROWS_PER_LANE rows in flight.  One warp per row with 4-byte loads, rows ordered by head (each result four
// bytes of another sector), took 75 us for 2 x 4096 x 32 heads of 128 and 33 us for 8 x 512 x 32 heads of 64; this form takes 28 (4.8 TB/s) and 6.
constexpr int DELTA_THREADS = 256, ROWS_PER_LANE = 4;
template <int D>
__global__ void __launch_bounds__(DELTA_THREADS)
delta_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O, const float* __restrict__ lse, float* __restrict__ delta,
             float* __restrict__ lse2n, int S, int H, long long do_sb, long long do_ss, long long do_sh, long long o_sb, long long o_ss, long long o_sh,
             bool aligned) {
  constexpr int LANES = D / 8, PER_PASS = DELTA_THREADS / LANES;
  const int sub = threadIdx.x % LANES, first = blockIdx.x * (PER_PASS * ROWS_PER_LANE) + threadIdx.x / LANES;
  const int h = blockIdx.y, b = blockIdx.z;
  const __nv_bfloat16* a = dO + b * do_sb + h * do_sh + sub * 8;
  const __nv_bfloat16* c = O + b * o_sb + h * o_sh + sub * 8;
  uint4 x[ROWS_PER_LANE], y[ROWS_PER_LANE];
#pragma unroll
  for (int i = 0; i < ROWS_PER_LANE; ++i) {
    const long long s = min(first + i * PER_PASS, S - 1);
    if (aligned) {
      x[i] = *reinterpret_cast<const uint4*>(a + s * do_ss);
      y[i] = *reinterpret_cast<const uint4*>(c + s * o_ss);
    } else {                                          // rows on 4-byte boundaries only
      const uint32_t *xa = reinterpret_cast<const uint32_t*>(a + s * do_ss), *yc = reinterpret_cast<const uint32_t*>(c + s * o_ss);
      x[i] = make_uint4(xa[0], xa[1], xa[2], xa[3]);
      y[i] = make_uint4(yc[0], yc[1], yc[2], yc[3]);
    }
  }
#pragma unroll
  for (int i = 0; i < ROWS_PER_LANE; ++i) {
    const uint32_t xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, ys[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
    float acc = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) acc += bf16_lo(xs[w]) * bf16_lo(ys[w]) + bf16_hi(xs[w]) * bf16_hi(ys[w]);
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const int s = first + i * PER_PASS;
    if (sub == 0 && s < S) {
      const long long o = (static_cast<long long>(b) * H + h) * S + s;
      delta[o] = acc;
      lse2n[o] = -lse[o] * LOG2E;        // the log-sum-exp in log2 units, negative: the addend of both product kernels
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Both product kernels run sixteen softmax warps (four threads per TMEM lane, a quarter of a 128 x 128 tile's columns each), a TMA warp and an MMA warp.  What bounds
// them is the chain of a tile: scores to registers, exponentials, dP to registers, dS back to tensor memory, products, and a barrier between any two of these.  No unit
// is near its rate, so the chain is kept short: many warps with little each, and scores and dP handed over one by one, so that the tensor cores finish one while the
// other is worked on.  Two groups of four warps that took turns at 64-wide tiles, each handed scores and dP together, and a CTA for each item (before -> now, us):
//   2 x 4096 tokens, 32 / 8 heads of 128, causal    dQ 400 -> 366   dK / dV 557 -> 508
//   8 x 512 tokens, 32 / 8 heads of 64, causal      dQ  52 ->  39   dK / dV  58 ->  40
//   64 x 256 tokens, 12 heads of 64                 dQ  73 ->  55   dK / dV 109 ->  97
// (eight warps: 396 and 581 us of the first; with neither their exponentials nor their products still 261 and 419).

// This thread's 32 columns of its row of a [128 x 128] accumulator.
__device__ __forceinline__ void load_part(uint32_t addr, uint32_t (&v)[COLS]) {
  tmem_ld_32x32b_x32(addr, v);
  tmem_ld_wait();
}

// The same 32 values as bf16 over the first 16 of these columns (its neighbours may still be reading theirs).
__device__ __forceinline__ void store_part(uint32_t addr, const uint32_t (&pk)[COLS / 2]) {
  tmem_st_32x32b_x16(addr, pk);
  tmem_st_wait();
}

// The k-th 16 columns of a tile stored by store_part, as a tensor-memory A operand.
__device__ __forceinline__ uint32_t part_operand(uint32_t tile, int kk) { return tile + (kk >> 1) * COLS + (kk & 1) * 8; }

// Two tiles' rows of D bf16 from swizzled shared tiles of 128 rows to tensor memory (32-bit column w = features 2w, 2w + 1), 32 features a piece, by four threads a row.
template <int D>
__device__ __forceinline__ void rows_to_tmem(const uint8_t* a, const uint8_t* b, int r, int part, uint32_t to_a, uint32_t to_b) {
#pragma unroll
  for (int g = 0; g < 2 * D / 32; g += 4) {
    const int piece = g + part, c = piece % (D / 32);
    const uint8_t* from = (piece < D / 32 ? a : b) + (c >> 1) * (128 * 128) + r * 128;
    uint32_t w[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 x = *reinterpret_cast<const uint4*>(from + ((((c & 1) * 4 + q) ^ (r & 7)) << 4));
      w[q * 4] = x.x; w[q * 4 + 1] = x.y; w[q * 4 + 2] = x.z; w[q * 4 + 3] = x.w;
    }
    tmem_st_32x32b_x16((piece < D / 32 ? to_a : to_b) + c * 16, w);
  }
  tmem_st_wait();
}

// A quarter of this thread's row of a gradient accumulator, times `scale`, as bf16; zeros where nothing was accumulated.
template <int D>
__device__ __forceinline__ void write_quarter(uint32_t addr, bool any, float scale, __nv_bfloat16* to, bool real) {
  uint32_t v[32];
  if (any) {
    if constexpr (D == 128) {
      tmem_ld_32x32b_x32(addr, v);
    } else {
      uint32_t h[16];
      tmem_ld_32x32b_x16(addr, h);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = h[i];
    }
    tmem_ld_wait();
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0;
  }
  if (real) {
#pragma unroll
    for (int q = 0; q < D / 64; ++q) {
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = pack_bf16(__uint_as_float(v[q * 16 + 2 * i]) * scale, __uint_as_float(v[q * 16 + 2 * i + 1]) * scale);
      st_global_32_any(to + q * 16, w);
    }
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------------------------------------------
// dQ kernel: persistent, items of 128 query rows of one head; key tiles of 128 stream through one ring of K and V, from one item into the next.  Q and dO are the A
// operands of every score product of an item: the softmax threads copy them once from shared to tensor memory, so the score products fetch only K / V from shared
// memory, and the next item's Q and dO arrive while this one is worked on.  (With a CTA an item, 406 us instead of 366, and 51 instead of 39 for 8 x 512 tokens of 64-wide heads.)
//   softmax : scores into registers (the next ones may then be computed), P = exp2(S - lse), dS = P o (dP - delta) over dP in tensor memory
//   MMA     : S(j + 1) as soon as S(j) has been read; dQ += dS(j) K(j), then dP(j + 1)
template <int D>
struct DqCfg {
  static constexpr int BM = 128, BN = 128, RING = D == 128 ? 5 : 8;
  static constexpr int SUB = D / 64;
  static constexpr int TILE = 128 * D * 2;
  static constexpr int SMEM = (2 + RING) * TILE + 256;      // no slack to align by hand
  static constexpr int TM_S = 0, TM_DP = 128, TM_DQ = 256, TM_COLS = 512;
  static constexpr int TM_QA = 384, TM_DOA = 448;    // Q and dO as tensor-memory A operands (D / 2 packed columns each)
};

struct DqBars {
  uint64_t q_full;
  uint64_t kv_full[8], kv_empty[8];
  uint64_t s_full, s_free, dp_full, ds_full;
  uint64_t a_ready;                     // Q and dO copied to tensor memory (one arrival per softmax warp)
  uint64_t all_done;
  uint32_t tmem_base;
  int abort_flag;
  int poisoned;
};
static_assert(sizeof(DqBars) <= 256, "DqBars must fit its slot");

template <int D, bool CAUSAL, bool VAR>
__global__ void __launch_bounds__(THREADS, 1)
flash_dq_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tdo,
                const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                const float* __restrict__ lse2n, const float* __restrict__ delta, __nv_bfloat16* __restrict__ dq, int S,
                int T, int Hq, int Hkv, int B, long long dq_sb, long long dq_ss, long long dq_sh, float scale, Variant var,
                int* __restrict__ err) {
  using C = DqCfg<D>;
  constexpr int BM = C::BM, BN = C::BN, RING = C::RING;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // The 128-byte swizzle atoms need tiles on 1024-byte boundaries: refuse instead of overrunning.
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(err, 0, ERR_BAD_ARG);
    return;
  }
  uint8_t* sQ = smem_raw;
  uint8_t* sdO = sQ + C::TILE;
  uint8_t* sKV = sdO + C::TILE;              // RING stages: K(0), V(0), K(1), ...
  DqBars* bars = reinterpret_cast<DqBars*>(sKV + RING * C::TILE);
  {
    // An earlier launch reported a timed-out wait: leave at once instead of queueing more waits behind it. One
    // thread reads the status so the whole CTA takes the same branch.
    if (threadIdx.x == 0) bars->poisoned = *reinterpret_cast<volatile int*>(err);
    __syncthreads();
    if (bars->poisoned != 0) return;
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float scale_log2 = scale * LOG2E;
  const int q_tiles = (S + BM - 1) / BM, per = Hq * B, items = q_tiles * per;
  // The CTA's items, every other turn backwards over the CTAs, so that items sorted by length (causal: the longest first) come out even.  False: none this turn.
  struct Item { int q0, h, b, lo, iters; };
  auto item_of = [&](int turn, Item& w) -> bool {
    const int g = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
    const int index = turn * g + ((turn & 1) ? g - 1 - c : c);
    if (index >= items) return false;
    const int qi = index / per, rest = index - qi * per;
    w.q0 = (CAUSAL ? q_tiles - 1 - qi : qi) * BM;
    w.h = rest % Hq;
    w.b = rest / Hq;
    const int n_all = max(0, CAUSAL ? min((w.q0 + BM + (T - S) + BN - 1) / BN, (T + BN - 1) / BN) : (T + BN - 1) / BN);
    w.lo = VAR ? attn::first_key_tile_of_warp(var, w.b, w.q0, S, T, BN, n_all, lane) : 0;
    w.iters = n_all - w.lo;
    return true;
  };
  const int turns = (items + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int i = 0; i < RING; ++i) { mbar_init(&bars->kv_full[i], 1); mbar_init(&bars->kv_empty[i], 1); }
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->s_free, SOFTMAX_WARPS);
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->ds_full, SOFTMAX_WARPS);
    mbar_init(&bars->all_done, 1);
    mbar_init(&bars->a_ready, SOFTMAX_WARPS);
    bars->abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == MMA_WARP) { tmem_alloc(&bars->tmem_base, C::TM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;
  if (warp >= TMA_WARP) {
   regs_down<ISSUE_REGS>();
   if (warp == TMA_WARP) {
    // (the warp together, one lane issues)
    int slot = 0, n = 0;                                   // n: items begun
    uint32_t phase = 1;
    bool ok = true;
    for (int turn = 0; turn < turns && ok; ++turn) {
      Item w;
      if (!item_of(turn, w) || w.iters <= 0) continue;
      // the item before has Q and dO in tensor memory
      if (n > 0 && !mbar_wait_warp(&bars->a_ready, (n - 1) & 1, abort_flag)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
      ++n;
      if (lane == 0) {
        mbar_expect_tx(&bars->q_full, 2 * C::TILE);
#pragma unroll
        for (int t = 0; t < C::SUB; ++t) {
          tma_load_4d(sQ + t * (BM * 128), &tq, &bars->q_full, t * 64, w.h, w.q0, w.b);
          tma_load_4d(sdO + t * (BM * 128), &tdo, &bars->q_full, t * 64, w.h, w.q0, w.b);
        }
      }
      __syncwarp();
      const int hk = w.h / (Hq / Hkv);
      for (int it = 0; it < 2 * w.iters; ++it) {
        ok = mbar_wait_warp(&bars->kv_empty[slot], phase, abort_flag);
        if (!ok) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
        if (lane == 0) {
          mbar_expect_tx(&bars->kv_full[slot], C::TILE);
#pragma unroll
          for (int t = 0; t < C::SUB; ++t)
            tma_load_4d(sKV + slot * C::TILE + t * (BN * 128), (it & 1) ? &tv : &tk, &bars->kv_full[slot], t * 64, hk, (w.lo + (it >> 1)) * BN, w.b);
        }
        __syncwarp();
        if (++slot == RING) { slot = 0; phase ^= 1; }
      }
    }
   } else if (warp == MMA_WARP) {
    // The whole warp runs this loop and waits together; one elected lane issues (see mbar_wait_warp).
    constexpr uint32_t idesc_s = make_idesc(BM, BN, 1, 1, 0, 0);
    constexpr uint32_t idesc_dq = make_idesc(BM, D, 1, 1, 0, 1);
    auto await = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
      if (mbar_wait_warp(bar, parity, abort_flag)) return true;
      if (lane == 0) atomicCAS(err, 0, code);
      return false;
    };
    int slot = 0;
    uint32_t phase = 0;
    auto take = [&](int& at) -> bool {                    // wait for the ring's next tile
      at = slot;
      if (!await(&bars->kv_full[slot], phase, ERR_WAIT_FULL)) return false;
      if (++slot == RING) { slot = 0; phase ^= 1; }
      return true;
    };
    // a [128 x 128] product of a tensor-memory operand and a key or value tile over their features
    auto score_product = [&](uint32_t d, uint32_t a, int at) {
      const uint32_t ba = smem_u32(sKV + at * C::TILE);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)                 // 16 features = 8 packed 32-bit columns
        umma_bf16_ts(d, a + kk * 8, make_sdesc_sw128(ba + (kk >> 2) * (BN * 128) + (kk & 3) * 32, 16, 1024), idesc_s, kk > 0 ? 1u : 0u);
    };
    int n = 0;                                             // items begun
    uint32_t ph = 0;                                       // parity of the tile, counted over all items
    bool ok = true;
    for (int turn = 0; turn < turns && ok; ++turn) {
      Item w;
      if (!item_of(turn, w) || w.iters <= 0) continue;
      int k_at = 0, k_next = 0, v_at = 0;
      ok = await(&bars->a_ready, n & 1, ERR_WAIT_FULL) && take(k_at) && take(v_at);
      ++n;
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        score_product(tmem + C::TM_S, tmem + C::TM_QA, k_at);
        umma_commit(&bars->s_full);
        score_product(tmem + C::TM_DP, tmem + C::TM_DOA, v_at);
        umma_commit(&bars->dp_full);
        umma_commit(&bars->kv_empty[v_at]);
      }
      __syncwarp();
      for (int it = 0; it < w.iters; ++it, ph ^= 1) {
        const bool more = it + 1 < w.iters;
        if (more) {
          ok = take(k_next) && await(&bars->s_free, ph, ERR_WAIT_TMEM_EMPTY);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            score_product(tmem + C::TM_S, tmem + C::TM_QA, k_next);
            umma_commit(&bars->s_full);
          }
          __syncwarp();
          ok = take(v_at);
          if (!ok) break;
        }
        ok = await(&bars->ds_full, ph, ERR_WAIT_OTHER);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ka = smem_u32(sKV + k_at * C::TILE);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BN / 16; ++kk)
            umma_bf16_ts(tmem + C::TM_DQ, part_operand(tmem + C::TM_DP, kk), make_sdesc_sw128(ka + kk * 2048, BN * 128, 1024), idesc_dq,
                         (it > 0 || kk > 0) ? 1u : 0u);
          umma_commit(&bars->kv_empty[k_at]);
          if (more) {
            // over dS(it), which the product before has read by then: one thread's products run in order
            score_product(tmem + C::TM_DP, tmem + C::TM_DOA, v_at);
            umma_commit(&bars->dp_full);
            umma_commit(&bars->kv_empty[v_at]);
          } else {
            umma_commit(&bars->all_done);
          }
        }
        __syncwarp();
        k_at = k_next;
      }
    }
   }
  } else {
    regs_up<SOFTMAX_REGS>();
    const int q4 = warp & 3, part = warp >> 2;
    const int r = q4 * 32 + lane;                   // query row within the tile == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + C::TM_S + part * COLS, t_dp = tmem + lane_addr + C::TM_DP + part * COLS;
    const uint64_t factor = pair_of(scale_log2, scale_log2);
    int n = 0;                                      // items begun
    uint32_t ph = 0;                                // parity of the tile, counted over all items
    bool ok = true;
    for (int turn = 0; turn < turns && ok; ++turn) {
      Item w;
      if (!item_of(turn, w)) continue;
      const int row = w.q0 + r;
      const long long stat = (static_cast<long long>(w.b) * Hq + w.h) * S + row;
      const float nlse = row < S ? lse2n[stat] : 0.f;
      const float dl = row < S ? delta[stat] : 0.f;
      const int limit = min(CAUSAL ? row + (T - S) : T - 1, T - 1);
      // only tiles that reach past the warp's first row's last visible key need the comparisons: one branch per warp
      const int warp_limit = min(CAUSAL ? w.q0 + q4 * 32 + (T - S) : T - 1, T - 1);
      const uint64_t shift = pair_of(nlse, nlse), minus_delta = pair_of(-dl, -dl);
      if (w.iters > 0) {
        // (every product that read the Q and dO of the item before has completed: all_done)
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->q_full, n & 1, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_FULL); ok = false; break; }
        rows_to_tmem<D>(sQ, sdO, r, part, tmem + lane_addr + C::TM_QA, tmem + lane_addr + C::TM_DOA);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->a_ready);
      }
      for (int it = 0; it < w.iters; ++it, ph ^= 1) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->s_full, ph, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_TMEM_FULL); ok = false; break; }
        tc_fence_after();
        const int k0 = (w.lo + it) * BN + part * COLS;
        uint32_t v[COLS];
        float p[COLS];
        load_part(t_s, v);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->s_free);
#pragma unroll
        for (int i = 0; i < COLS; i += 2) {
          float x0, x1, f0 = 1.f, f1 = 1.f;           // f: d(capped score) / d(score)
          if (VAR && var.softcap > 0.f) {
            const float cap2 = var.softcap * LOG2E, twice = 2.f * scale / var.softcap * LOG2E;
            x0 = fmaf(cap2, capped(v[i], twice, f0), nlse);
            x1 = fmaf(cap2, capped(v[i + 1], twice, f1), nlse);
          } else {
            unpair(fma2(pair_of(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), factor, shift), x0, x1);
          }
          p[i] = fast_exp2(x0) * f0;
          p[i + 1] = fast_exp2(x1) * f1;
        }
        if (k0 + COLS - 1 > warp_limit) {
          const int past = limit - k0;
#pragma unroll
          for (int i = 0; i < COLS; ++i) if (i > past) p[i] = 0.f;
        }
        if (VAR && var.window > 0) {
          const int first = row + (T - S) - var.window + 1 - k0;       // first visible key of this row
          if (first > 0) {
#pragma unroll
            for (int i = 0; i < COLS; ++i) if (i < first) p[i] = 0.f;
          }
        }
        if (VAR && var.q_seg != nullptr) {
          const int* ks = var.k_seg + static_cast<long long>(w.b) * T;
          const int mine = var.q_seg[static_cast<long long>(w.b) * S + min(row, S - 1)];
#pragma unroll
          for (int i = 0; i < COLS; ++i) if (k0 + i < T && ks[k0 + i] != mine) p[i] = 0.f;
        }
        __syncwarp();
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->dp_full, ph, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_TMEM_FULL); ok = false; break; }
        tc_fence_after();
        uint32_t ds[COLS / 2];
        load_part(t_dp, v);
#pragma unroll
        for (int i = 0; i < COLS; i += 2) {
          float a, b2;
          unpair(mul2(pair_of(p[i], p[i + 1]), add2(pair_of(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), minus_delta)), a, b2);
          ds[i >> 1] = pack_bf16(a, b2);
        }
        store_part(t_dp, ds);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->ds_full);
      }
      if (ok && w.iters > 0) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->all_done, n & 1, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_OTHER); ok = false; }
        ++n;
      }
      if (!ok) break;
      tc_fence_after();
      write_quarter<D>(tmem + lane_addr + C::TM_DQ + part * (D / 4), w.iters > 0, scale,
                       dq + w.b * dq_sb + static_cast<long long>(row) * dq_ss + w.h * dq_sh + part * (D / 4), row < S);
      tc_fence_before();                            // the next item's products over this dQ are told of by its ds_full
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, C::TM_COLS); }
}

// ---------------------------------------------------------------------------------------------------------------
// dK / dV kernel: one CTA per 128 keys of one KV head; query tiles of 128 of the heads of its group stream through a ring of Q, dO and their statistics.
//   softmax : one key row, a quarter of the queries a thread: P^T = exp2(S^T - lse), dS^T = P^T o (dP^T - delta) over dP^T, both in tensor memory
//   MMA     : dV += P^T(j) dO(j);  dK += dS^T(j) Q(j), then dP^T(j + 1);  S^T(j + 1) as early as its place is free
// Heads of 64 leave room in tensor memory for P^T beside the scores, so that the next ones are computed while the exponentials are taken, and for K and V as A operands of
// the score products (8 x 512 tokens, 32 / 8 heads: 49.5 -> 39.6 us).  At 128 the accumulators and scores take all of it: P^T lies over the scores, and the next ones come
// behind its product.  (Through shared memory instead, with the scores early, the product's second operand from there cost more than that: 551 us against 500.)
template <int D>
struct DkvCfg {
  static constexpr int BKV = 128, BQ = 128, QSTAGES = D == 128 ? 2 : 4;
  static constexpr int SUB = D / 64;
  static constexpr bool KV_IN_TMEM = D == 64, P_APART = D == 64;
  static constexpr int TILE = 128 * D * 2;
  static constexpr int STAT_BYTES = 2 * BQ * 4;      // per stage: 128 log-sum-exps, 128 deltas
  static constexpr int SMEM = 2 * TILE + QSTAGES * (2 * TILE + STAT_BYTES) + 256;      // no slack to align by hand
  static constexpr int TM_S = 0, TM_DP = 128, TM_DV = 256, TM_DK = 256 + D, TM_COLS = 512;
  static constexpr int TM_KA = 384, TM_VA = 416, TM_P = 448;     // (at heads of 64)
};

struct DkvBars {
  uint64_t kv_full;
  uint64_t q_full[4], q_empty[4];
  uint64_t s_full, p_full, dp_full, ds_full;
  uint64_t s_free, p_free;              // (P_APART)
  uint64_t a_ready;
  uint64_t all_done;
  uint32_t tmem_base;
  int abort_flag;
  int q_end;                            // one past the last query tile that sees this key tile
  int poisoned;
};
static_assert(sizeof(DkvBars) <= 256, "DkvBars must fit its slot");

template <int D, bool CAUSAL, bool VAR>
__global__ void __launch_bounds__(THREADS, 1)
flash_dkv_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tdo,
                 const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                 const float* __restrict__ lse2n, const float* __restrict__ delta, __nv_bfloat16* __restrict__ dk,
                 __nv_bfloat16* __restrict__ dv, int S, int T, int Hq, int Hkv, long long dk_sb, long long dk_ss,
                 long long dk_sh, long long dv_sb, long long dv_ss, long long dv_sh, float scale, Variant var,
                 int* __restrict__ err) {
  using C = DkvCfg<D>;
  constexpr int BKV = C::BKV, BQ = C::BQ, QS = C::QSTAGES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // The 128-byte swizzle atoms need tiles on 1024-byte boundaries: refuse instead of overrunning.
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(err, 0, ERR_BAD_ARG);
    return;
  }
  uint8_t* sK = smem_raw;
  uint8_t* sV = sK + C::TILE;
  uint8_t* sQ = sV + C::TILE;                // QS stages
  uint8_t* sdO = sQ + QS * C::TILE;          // QS stages
  float* sStat = reinterpret_cast<float*>(sdO + QS * C::TILE);     // [QS stages][-lse2 128 | delta 128]
  DkvBars* bars = reinterpret_cast<DkvBars*>(reinterpret_cast<uint8_t*>(sStat) + QS * C::STAT_BYTES);
  {
    // An earlier launch reported a timed-out wait: leave at once instead of queueing more waits behind it. One
    // thread reads the status so the whole CTA takes the same branch.
    if (threadIdx.x == 0) bars->poisoned = *reinterpret_cast<volatile int*>(err);
    __syncthreads();
    if (bars->poisoned != 0) return;
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // 1-D grid ordered by key tile first, so that with causal masking the long CTAs (early key tiles see every later
  // query tile) of ALL heads start first and the short ones fill the tail: blocks are issued in index order.
  const int per_tile = static_cast<int>(gridDim.x) / ((T + BKV - 1) / BKV);      // = Hkv * batch
  const int kt = blockIdx.x / per_tile;
  const int hk = (blockIdx.x % per_tile) % Hkv, b = (blockIdx.x % per_tile) / Hkv;
  const int rep = Hq / Hkv;
  const int kv0 = kt * BKV;
  // first query tile that can see any key of this tile (causal, bottom-right aligned): q + (T - S) >= kv0
  const int q_first = CAUSAL ? max(0, kv0 - (T - S)) / BQ : 0;
  const float scale_log2 = scale * LOG2E;

  if (threadIdx.x == 0) {
    // one past the last query tile that sees this key tile (a window or packed documents end it early)
    bars->q_end = VAR ? attn::end_query_block(var, b, kv0, BKV, S, T, BQ) : (S + BQ - 1) / BQ;
    mbar_init(&bars->kv_full, 1);
    for (int i = 0; i < QS; ++i) { mbar_init(&bars->q_full[i], 1); mbar_init(&bars->q_empty[i], 1); }
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->s_free, SOFTMAX_WARPS);
    mbar_init(&bars->p_full, SOFTMAX_WARPS);
    mbar_init(&bars->p_free, 1);
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->ds_full, SOFTMAX_WARPS);
    mbar_init(&bars->a_ready, SOFTMAX_WARPS);
    mbar_init(&bars->all_done, 1);
    bars->abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == MMA_WARP) { tmem_alloc(&bars->tmem_base, C::TM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;
  const int nqb = bars->q_end - q_first;                // query tiles per head
  const int iters = nqb > 0 ? nqb * rep : 0;

  if (warp >= TMA_WARP) {
   regs_down<ISSUE_REGS>();
   if (warp == TMA_WARP) {
    if (lane == 0) {
      mbar_expect_tx(&bars->kv_full, 2 * C::TILE);
#pragma unroll
      for (int t = 0; t < C::SUB; ++t) {
        tma_load_4d(sK + t * (BKV * 128), &tk, &bars->kv_full, t * 64, hk, kv0, b);
        tma_load_4d(sV + t * (BKV * 128), &tv, &bars->kv_full, t * 64, hk, kv0, b);
      }
      for (int it = 0; it < iters; ++it) {
        const int qs = it % QS; const uint32_t ph = (it / QS) & 1;
        const int h = hk * rep + it / nqb;
        const int qb = (q_first + it % nqb) * BQ;
        if (!mbar_wait(&bars->q_empty[qs], ph ^ 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
        const uint32_t stat_bytes = static_cast<uint32_t>(min(BQ, S - qb)) * 4;        // S is a multiple of 64
        mbar_expect_tx(&bars->q_full[qs], 2 * C::TILE + 2 * stat_bytes);
#pragma unroll
        for (int t = 0; t < C::SUB; ++t) tma_load_4d(sQ + qs * C::TILE + t * (BQ * 128), &tq, &bars->q_full[qs], t * 64, h, qb, b);
        // the tile's per-query statistics ride the same barrier
        const long long stat = (static_cast<long long>(b) * Hq + h) * S + qb;
        bulk_load_1d(sStat + qs * 2 * BQ, lse2n + stat, stat_bytes, &bars->q_full[qs]);
        bulk_load_1d(sStat + qs * 2 * BQ + BQ, delta + stat, stat_bytes, &bars->q_full[qs]);
#pragma unroll
        for (int t = 0; t < C::SUB; ++t) tma_load_4d(sdO + qs * C::TILE + t * (BQ * 128), &tdo, &bars->q_full[qs], t * 64, h, qb, b);
      }
    }
   } else if (warp == MMA_WARP) {
    // The whole warp runs this loop and waits together; one elected lane issues (see mbar_wait_warp).
    constexpr uint32_t idesc_s = make_idesc(BKV, BQ, 1, 1, 0, 0);
    constexpr uint32_t idesc_acc = make_idesc(BKV, D, 1, 1, 0, 1);
    auto await = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
      if (mbar_wait_warp(bar, parity, abort_flag)) return true;
      if (lane == 0) atomicCAS(err, 0, code);
      return false;
    };
    // a [128 x 128] product over the features of K or V and a query tile
    auto score_product = [&](uint32_t d, const uint8_t* a, uint32_t a_tmem, const uint8_t* bt) {
      const uint32_t aa = smem_u32(a), ba = smem_u32(bt);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t off = (kk >> 2) * (128 * 128) + (kk & 3) * 32;
        if (C::KV_IN_TMEM) umma_bf16_ts(d, a_tmem + kk * 8, make_sdesc_sw128(ba + off, 16, 1024), idesc_s, kk > 0 ? 1u : 0u);
        else umma_bf16_ss(d, make_sdesc_sw128(aa + off, 16, 1024), make_sdesc_sw128(ba + off, 16, 1024), idesc_s, kk > 0 ? 1u : 0u);
      }
    };
    auto value_product = [&](const uint8_t* bt, bool fresh) {              // dV += P^T dO
      const uint32_t ba = smem_u32(bt);
#pragma unroll
      for (int kk = 0; kk < BQ / 16; ++kk)
        umma_bf16_ts(tmem + C::TM_DV, C::P_APART ? tmem + C::TM_P + kk * 8 : part_operand(tmem + C::TM_S, kk), make_sdesc_sw128(ba + kk * 2048, BQ * 128, 1024), idesc_acc,
                     (!fresh || kk > 0) ? 1u : 0u);
    };
    auto key_product = [&](const uint8_t* bt, bool fresh) {                // dK += dS^T Q
      const uint32_t ba = smem_u32(bt);
#pragma unroll
      for (int kk = 0; kk < BQ / 16; ++kk)
        umma_bf16_ts(tmem + C::TM_DK, part_operand(tmem + C::TM_DP, kk), make_sdesc_sw128(ba + kk * 2048, BQ * 128, 1024), idesc_acc, (!fresh || kk > 0) ? 1u : 0u);
    };
    bool ok = await(C::KV_IN_TMEM ? &bars->a_ready : &bars->kv_full, 0, ERR_WAIT_FULL);
    if (ok && iters > 0) {
      ok = await(&bars->q_full[0], 0, ERR_WAIT_FULL);
      tc_fence_after();
      if (ok && elect_one()) {
        score_product(tmem + C::TM_S, sK, tmem + C::TM_KA, sQ);
        umma_commit(&bars->s_full);
        score_product(tmem + C::TM_DP, sV, tmem + C::TM_VA, sdO);
        umma_commit(&bars->dp_full);
      }
      __syncwarp();
    }
    for (int it = 0; it < iters && ok; ++it) {
      const int qs = it % QS, qn = (it + 1) % QS; const uint32_t ph = it & 1;
      const bool more = it + 1 < iters;
      auto next_scores = [&]() -> bool {
        if (!more) return true;
        if (C::P_APART && !await(&bars->s_free, ph, ERR_WAIT_TMEM_EMPTY)) return false;
        if (!await(&bars->q_full[qn], ((it + 1) / QS) & 1, ERR_WAIT_FULL)) return false;
        tc_fence_after();
        if (elect_one()) {
          // (over P^T(it) where that is not apart, which the product before has read by then: one thread's products run in order)
          score_product(tmem + C::TM_S, sK, tmem + C::TM_KA, sQ + qn * C::TILE);
          umma_commit(&bars->s_full);
        }
        __syncwarp();
        return true;
      };
      if (C::P_APART) ok = next_scores();
      ok = ok && await(&bars->p_full, ph, ERR_WAIT_OTHER);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        value_product(sdO + qs * C::TILE, it == 0);
        if (C::P_APART) umma_commit(&bars->p_free);
      }
      __syncwarp();
      if (!C::P_APART) ok = next_scores();
      if (!ok) break;
      ok = await(&bars->ds_full, ph, ERR_WAIT_OTHER);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        key_product(sQ + qs * C::TILE, it == 0);
        umma_commit(&bars->q_empty[qs]);
        if (more) {
          // over dS^T(it), which the product before has read by then: one thread's products run in order
          score_product(tmem + C::TM_DP, sV, tmem + C::TM_VA, sdO + qn * C::TILE);
          umma_commit(&bars->dp_full);
        }
      }
      __syncwarp();
    }
    if (ok && elect_one()) umma_commit(&bars->all_done);        // every product issued above has completed when this fires
    __syncwarp();
   }
  } else {
    regs_up<SOFTMAX_REGS>();
    const int q4 = warp & 3, part = warp >> 2;
    const int r = q4 * 32 + lane;                   // key row within the tile == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(q4 * 32) << 16;
    const int key = kv0 + r;
    const uint32_t t_s = tmem + lane_addr + C::TM_S + part * COLS, t_dp = tmem + lane_addr + C::TM_DP + part * COLS;
    bool ok = true;
    if (C::KV_IN_TMEM) {
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->kv_full, 0, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_FULL); ok = false; }
      if (ok) {
        rows_to_tmem<D>(sK, sV, r, part, tmem + lane_addr + C::TM_KA, tmem + lane_addr + C::TM_VA);
        tc_fence_before();
      }
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(&bars->a_ready);
    }
    const uint64_t factor = pair_of(scale_log2, scale_log2), minus_one = pair_of(-1.f, -1.f);
    for (int it = 0; it < iters && ok; ++it) {
      const uint32_t ph = it & 1;
      const int qs = it % QS; const uint32_t phq = (it / QS) & 1;
      const int qb = (q_first + it % nqb) * BQ + part * COLS;     // this thread's first query
      // the tile's statistics arrived with its Q / dO
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->q_full[qs], phq, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_FULL); ok = false; break; }
      const float4* lse4 = reinterpret_cast<const float4*>(sStat + qs * 2 * BQ + part * COLS);
      const float4* dlt4 = reinterpret_cast<const float4*>(sStat + qs * 2 * BQ + BQ + part * COLS);
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->s_full, ph, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_TMEM_FULL); ok = false; break; }
      tc_fence_after();
      uint32_t v[COLS], pk[COLS / 2];
      float p[COLS];
      load_part(t_s, v);
      if (C::P_APART) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->s_free);
      }
#pragma unroll
      for (int i = 0; i < COLS; i += 4) {
        const float4 l4 = lse4[i >> 2];
        if (VAR && var.softcap > 0.f) {
          const float cap2 = var.softcap * LOG2E, twice = 2.f * scale / var.softcap * LOG2E;
          const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float slope;
            p[i + q] = fmaf(cap2, capped(v[i + q], twice, slope), l[q]);
            v[i + q] = __float_as_uint(slope);
          }
        } else {
          unpair(fma2(pair_of(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), factor, pair_of(l4.x, l4.y)), p[i], p[i + 1]);
          unpair(fma2(pair_of(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])), factor, pair_of(l4.z, l4.w)), p[i + 2], p[i + 3]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) p[i + q] = fast_exp2(p[i + q]);
      }
      // only query tiles that start before this warp's last key, or tiles with rows past the end of either, need the comparisons: one branch per warp; with a window
      // or packed documents every tile is compared
      const int warp_last_key = kv0 + q4 * 32 + 31;
      if ((VAR && (var.window > 0 || var.q_seg != nullptr)) || (CAUSAL && warp_last_key > qb + (T - S)) || warp_last_key >= T || qb + COLS > S) {
        const int before = CAUSAL ? key - (T - S) - qb : 0;       // queries in front of it do not see this key
        const int end = key < T ? S - qb : 0;                     // nor do those past the end
#pragma unroll
        for (int i = 0; i < COLS; ++i) if (i < before || i >= end) p[i] = 0.f;
        if (VAR && var.window > 0) {
          const int past = key + var.window - (T - S) - qb;       // key visible iff key > (query + T - S) - window
#pragma unroll
          for (int i = 0; i < COLS; ++i) if (i >= past) p[i] = 0.f;
        }
        if (VAR && var.q_seg != nullptr) {
          const int* qsp = var.q_seg + static_cast<long long>(b) * S + qb;
          const int mine = var.k_seg[static_cast<long long>(b) * T + min(key, T - 1)];
#pragma unroll
          for (int i = 0; i < COLS; i += 4) {
            if (qb + i + 3 < S) {                                 // (S is a multiple of 4 here)
              const int4 id = *reinterpret_cast<const int4*>(qsp + i);
              if (id.x != mine) p[i] = 0.f;
              if (id.y != mine) p[i + 1] = 0.f;
              if (id.z != mine) p[i + 2] = 0.f;
              if (id.w != mine) p[i + 3] = 0.f;
            }
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < COLS; i += 2) pk[i >> 1] = pack_bf16(p[i], p[i + 1]);
      if (VAR && var.softcap > 0.f) {
        // from here on the weight times d(capped score) / d(score)
#pragma unroll
        for (int i = 0; i < COLS; ++i) p[i] *= __uint_as_float(v[i]);
      }
      if (C::P_APART) {
        // the product before has read its P^T
        if (it > 0 && !__all_sync(0xffffffffu, mbar_wait(&bars->p_free, ph ^ 1, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_OTHER); ok = false; break; }
        tc_fence_after();
        store_part(tmem + lane_addr + C::TM_P + part * (COLS / 2), pk);
      } else {
        store_part(t_s, pk);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->p_full);
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->dp_full, ph, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_TMEM_FULL); ok = false; break; }
      tc_fence_after();
      load_part(t_dp, v);
#pragma unroll
      for (int i = 0; i < COLS; i += 4) {
        const float4 d4 = dlt4[i >> 2];
        float a[4];
        unpair(mul2(pair_of(p[i], p[i + 1]), fma2(pair_of(d4.x, d4.y), minus_one, pair_of(__uint_as_float(v[i]), __uint_as_float(v[i + 1])))), a[0], a[1]);
        unpair(mul2(pair_of(p[i + 2], p[i + 3]), fma2(pair_of(d4.z, d4.w), minus_one, pair_of(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])))), a[2], a[3]);
        pk[i >> 1] = pack_bf16(a[0], a[1]);
        pk[(i >> 1) + 1] = pack_bf16(a[2], a[3]);
      }
      if (qb + COLS > S) {
        // a weight past the end of the queries is zero, but what it was multiplied by may be anything: the statistics there are an earlier tile's.  (S is even)
#pragma unroll
        for (int i = 0; i < COLS; i += 2) if (qb + i >= S) pk[i >> 1] = 0;
      }
      store_part(t_dp, pk);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->ds_full);
    }
    if (ok && iters > 0) {
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->all_done, 0, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_OTHER); ok = false; }
    }
    if (ok) {
      tc_fence_after();
      write_quarter<D>(tmem + lane_addr + C::TM_DV + part * (D / 4), iters > 0, 1.f, dv + b * dv_sb + static_cast<long long>(key) * dv_ss + hk * dv_sh + part * (D / 4), key < T);
      write_quarter<D>(tmem + lane_addr + C::TM_DK + part * (D / 4), iters > 0, scale, dk + b * dk_sb + static_cast<long long>(key) * dk_ss + hk * dk_sh + part * (D / 4), key < T);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem, C::TM_COLS); }
}

static int make_map(CUtensorMap* m, const void* base, int B, int L, int H, int D, long long sb, long long sl, long long sh,
                    int box_rows) {
  const uint64_t dims[4] = {static_cast<uint64_t>(D), static_cast<uint64_t>(H), static_cast<uint64_t>(L), static_cast<uint64_t>(B)};
  const uint64_t strides[3] = {static_cast<uint64_t>(sh) * 2, static_cast<uint64_t>(sl) * 2, static_cast<uint64_t>(sb) * 2};
  const uint32_t box[4] = {64, 1, static_cast<uint32_t>(box_rows), 1};
  return make_tmap_nd(m, base, 4, dims, strides, box, 2, true);
}

static int multiprocessors() {
  static int n[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (n[dev] == 0) {
    int v = 0;
    n[dev] = cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0 ? v : 148;
  }
  return n[dev];
}

static_assert(DqCfg<128>::SMEM + 64 <= 232448 && DkvCfg<128>::SMEM + 64 <= 232448, "over the 227 KB a CTA may use");

template <int D, bool CAUSAL, bool VAR>
static int launch_bwd(const void* dO, const void* q, const void* k, const void* v, const float* lse2n, const float* delta,
                      void* dq, void* dk, void* dv, int B, int S, int T, int Hq, int Hkv, const long long* qs,
                      const long long* ks, const long long* vs, const long long* os, const long long* dos,
                      const long long* dqs, const long long* dks, const long long* dvs, float scale, const Variant& var,
                      int* err, cudaStream_t stream) {
  int r;
  CUtensorMap tq, tdo, tk, tv;
  if ((r = make_map(&tq, q, B, S, Hq, D, qs[0], qs[1], qs[2], 128))) return 1000 + r;
  if ((r = make_map(&tdo, dO, B, S, Hq, D, dos[0], dos[1], dos[2], 128))) return 1100 + r;
  if ((r = make_map(&tk, k, B, T, Hkv, D, ks[0], ks[1], ks[2], 128))) return 1200 + r;
  if ((r = make_map(&tv, v, B, T, Hkv, D, vs[0], vs[1], vs[2], 128))) return 1300 + r;
  {
    auto kern = flash_dq_kernel<D, CAUSAL, VAR>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, DqCfg<D>::SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    const long long items = static_cast<long long>((S + 127) / 128) * Hq * B;
    if (items > 0x3fffffff) return -3;
    const int sms = multiprocessors();
    kern<<<items < sms ? static_cast<int>(items) : sms, THREADS, DqCfg<D>::SMEM, stream>>>(tq, tdo, tk, tv, lse2n, delta, reinterpret_cast<__nv_bfloat16*>(dq), S, T,
                                                     Hq, Hkv, B, dqs[0], dqs[1], dqs[2], scale, var, err);
    if ((r = static_cast<int>(cudaGetLastError()))) return r;
  }
  {
    auto kern = flash_dkv_kernel<D, CAUSAL, VAR>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, DkvCfg<D>::SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    dim3 grid(((T + 127) / 128) * Hkv * B, 1, 1);
    kern<<<grid, THREADS, DkvCfg<D>::SMEM, stream>>>(tq, tdo, tk, tv, lse2n, delta, reinterpret_cast<__nv_bfloat16*>(dk),
                                                      reinterpret_cast<__nv_bfloat16*>(dv), S, T, Hq, Hkv, dks[0], dks[1],
                                                      dks[2], dvs[0], dvs[1], dvs[2], scale, var, err);
    if ((r = static_cast<int>(cudaGetLastError()))) return r;
  }
  return 0;
}

}  // namespace flashbwd
}  // namespace dewb

// Every tensor is [B, length, heads, D] bf16 with unit stride along D and its own (batch, sequence, head) element
// strides, so q / k / v may be views of one fused projection output and dq / dk / dv views of one fused gradient
// buffer. lse [B,Hq,S] comes from the forward; delta is scratch of 2 * B * Hq * S floats this call fills (delta, then
// the negative log-sum-exp in log2 units). S must be a multiple of 64 (the statistics travel by 256-byte bulk copies).
// `strides` holds 8 triples in the order q, k, v, out, dO, dq, dk, dv.
// Variants as in the forward (window, softcap, segment ids of packed documents); `lse` must come from a forward run with the
// same variants (and sinks, if any).
extern "C" int dewb_flash_bwd_var(const void* dO, const void* q, const void* k, const void* v, const void* out,
                                  const float* lse, float* delta, void* dq, void* dk, void* dv, int B, int S, int T, int Hq,
                                  int Hkv, int D, const long long* strides, float scale, int causal, int window, float softcap,
                                  const int* q_seg, const int* k_seg, int* err, void* stream_ptr) {
  using namespace dewb::flashbwd;
  if ((D != 128 && D != 64) || Hq % Hkv != 0 || S % 64 != 0) return -3;
  if ((q_seg != nullptr) != (k_seg != nullptr) || window < 0 || softcap < 0.f) return -3;
  if (q_seg != nullptr && ((S % 4) || (T % 4) || (reinterpret_cast<uintptr_t>(q_seg) & 15) || (reinterpret_cast<uintptr_t>(k_seg) & 15))) return -3;
  const long long *qs = strides, *ks = strides + 3, *vs = strides + 6, *os = strides + 9, *dos = strides + 12,
                  *dqs = strides + 15, *dks = strides + 18, *dvs = strides + 21;
  for (int i = 0; i < 24; ++i) if (strides[i] % 8) return -3;       // 16-byte rows for TMA and the uint4 stores
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  const bool wide = ((reinterpret_cast<uintptr_t>(dO) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  const int per_block = DELTA_THREADS / (D / 8) * ROWS_PER_LANE;
  auto delta_fn = D == 128 ? delta_kernel<128> : delta_kernel<64>;
  delta_fn<<<dim3((S + per_block - 1) / per_block, Hq, B), DELTA_THREADS, 0, stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(dO), reinterpret_cast<const __nv_bfloat16*>(out), lse, delta, delta + static_cast<long long>(B) * Hq * S, S, Hq,
      dos[0], dos[1], dos[2], os[0], os[1], os[2], wide);
  const float* lse2n = delta + static_cast<long long>(B) * Hq * S;
  // the sink logits reach the backward through the saved log-sum-exp alone
  const Variant var{window, softcap, nullptr, q_seg, k_seg, 0, 0, nullptr, nullptr, nullptr};
  const bool any = window > 0 || softcap > 0.f || q_seg != nullptr;
#define DEWB_BWD_GO(DD, CC, VV) launch_bwd<DD, CC, VV>(dO, q, k, v, lse2n, delta, dq, dk, dv, B, S, T, Hq, Hkv, qs, ks, vs, os, dos, dqs, dks, dvs, scale, var, err, stream)
  if (D == 128) {
    if (any) return causal ? DEWB_BWD_GO(128, true, true) : DEWB_BWD_GO(128, false, true);
    return causal ? DEWB_BWD_GO(128, true, false) : DEWB_BWD_GO(128, false, false);
  }
  if (any) return causal ? DEWB_BWD_GO(64, true, true) : DEWB_BWD_GO(64, false, true);
  return causal ? DEWB_BWD_GO(64, true, false) : DEWB_BWD_GO(64, false, false);
#undef DEWB_BWD_GO
}

extern "C" int dewb_flash_bwd(const void* dO, const void* q, const void* k, const void* v, const void* out,
                              const float* lse, float* delta, void* dq, void* dk, void* dv, int B, int S, int T, int Hq,
                              int Hkv, int D, const long long* strides, float scale, int causal, int* err,
                              void* stream_ptr) {
  return dewb_flash_bwd_var(dO, q, k, v, out, lse, delta, dq, dk, dv, B, S, T, Hq, Hkv, D, strides, scale, causal, 0, 0.f, nullptr,
                            nullptr, err, stream_ptr);
}
