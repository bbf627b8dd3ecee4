// Flash attention forward for sm_100a (bf16, causal or full, GQA, heads of 64 or 128): two query tiles a CTA against one stream of keys and values.
//
// Persistent, one CTA per SM, 12 warps; a work item is two query tiles of 128 rows that share a key head, or, where tiles are few, the two halves of one tile's keys
// (every second key tile each; the halves' outputs, maxima and sums are joined at the end, and a CTA has one item):
//   warps 0..3  softmax of tile 0, one thread per query row (all 128 key columns: no reduction crosses threads)
//   warps 4..7  softmax of tile 1
//   warp 8      TMA producer : the item's queries, then its keys and values in the order they are used, into one ring
//   warp 9      MMA issuer   (warps 10, 11 only complete its group for the move of registers) : per key tile P0 V, S0 = Q0 K(next), P1 V, S1 = Q1 K(next)
// Tensor memory holds both tiles' scores and outputs (4 x 128 columns); P is written over its scores and read from there.
//
// What bounds it: of a pair of 128 x 128 tiles the tensor cores need 2048 cycles at heads of 128 (1024 at 64), the exponentials 2048.  With one tile a CTA the
// two took turns: scores, exponentials and P V of a tile depend on one another, and a second score buffer hides only the first of the three.  With two tiles the
// tensor cores work on one while the other is exponentiated, and a key or value tile that is fetched serves both.  The next item's scores are issued behind the
// last products of this one, so that its outputs are written while the tensor cores have work.  Measured (one tile a CTA of its own -> this), causal: 2 x 4096 tokens,
// 32 / 8 heads of 128, 365 -> 264 us; 1 x 16384 2210 -> 1770; 8 x 512, 32 / 8 heads of 64, 55 -> 33; not causal, 64 x 256, 12 heads of 64, 75 -> 44.  A pair's step is
// 3550 cycles now: a tile's chain (280 to be told of its scores, 140 to load and compare them, 1570 of exponentials, 80 to deliver P, 210 to tell the issuer, 1260 of
// products) twice over, each tile's exponentials beside the other's products.  Two threads a row with half of the columns each, for shorter exponentials, took 291 us
// (they have to meet once a tile), P delivered in halves 274, a quarter of the exponentials as polynomials 270.
//
// A row's running maximum is applied lazily: O and the row sum are rescaled only when it has grown by more than 2^8 since the last time.  The scores of key tile
// j + 1 are issued behind P V of tile j by the same thread, and the tensor cores run one thread's products in order: a warp that has been told of its scores may
// read and write O, and P and the next scores of a tile need no barrier between them.
#include "../common/ptx.cuh"
#include "../common/tmap.h"
#include "../common/attn_variant.cuh"

namespace dewb {
namespace attnpair {

constexpr int BM = 128;        // query rows per tile
constexpr int BN = 128;        // keys per tile
constexpr int THREADS = 384;
// Registers a thread: 168 at the launch (12 warps on four schedulers), then moved to the softmax, whose threads hold a row of 128 scores.
constexpr int SOFTMAX_REGS = 208, ISSUE_REGS = 88;
static_assert(2 * SOFTMAX_REGS + ISSUE_REGS <= 3 * 168, "an increase past what the block was launched with never ends");
constexpr int TMA_WARP = 8, MMA_WARP = 9;
constexpr float RESCALE_THRESHOLD = 8.0f;   // log2 units
constexpr float LOG2E = 1.4426950408889634f;
constexpr int NEVER = 0x3fffffff;

using attn::Variant;

template <int D>
struct Cfg {
  static constexpr int SUB = D / 64;                 // 64-column (128-byte) sub-tiles per row
  static constexpr int Q_TILE = BM * D * 2;
  static constexpr int KV_TILE = BN * D * 2;
  static constexpr int QSTAGES = D == 128 ? 1 : 2;   // pairs of query tiles
  static constexpr int RING = D == 128 ? 5 : 8;      // keys and values alike
  static constexpr int SMEM = QSTAGES * 2 * Q_TILE + RING * KV_TILE + 2048;
  static constexpr int TM_S = 0, TM_O = 256, TM_COLS = 512;      // 128 columns a tile each
};

struct Bars {
  uint64_t q_full[2], q_empty[2];
  uint64_t kv_full[8], kv_empty[8];
  uint64_t s_full[2], p_full[2], o_full[2];          // per tile
  uint32_t tmem_base;
  int abort_flag;
  int poisoned;
  float2 half[BM];                                   // SPLIT: maximum and sum of tile 1's rows
};
static_assert(sizeof(Bars) <= 2048 && Cfg<128>::SMEM <= 232448 && Cfg<64>::SMEM <= 232448, "over the 227 KB a CTA may use");

// What a launch is about, and how its query tiles are paired.
enum : int { HEADS = 0, ROWS = 1, SPLIT = 2 };
struct Shape {
  int B, S, T, Hq, Hkv;
  int pairing;                     // HEADS: the same rows of two neighbouring query heads of a key head; ROWS: two neighbouring tiles of a head;
                                   // SPLIT: both the same rows, tile 0 against the first, third, ... of their key tiles, tile 1 against the others (one item a CTA)
  int items;
};

// One item: its tiles' rows, heads and key tiles [0, keep) and [lo, hi); an empty tile has hi = 0 and lo = NEVER.  SPLIT: the key tiles of its rows are counted, `to` of
// them: the first keep[0] ones, then those from lo[0] on.
struct Item {
  int b, hk, from, to;             // the walk is over the tiles of both: [0, kept) and [from, to)
  int kept;
  int q0[2], h[2], lo[2], hi[2], keep[2];
};

template <bool CAUSAL, bool VAR, bool HALVES>
__device__ __forceinline__ Item make_item(int index, const Shape& s, const Variant& var, int lane) {
  Item w;
  const int heads = s.pairing == HEADS ? s.Hq / 2 : s.Hq;
  const int per = heads * s.B;
  const int tiles = (s.S + BM - 1) / BM;
  const int rows = s.pairing == ROWS ? (tiles + 1) / 2 : tiles;
  int qi = index / per;
  const int rest = index - qi * per;
  if (CAUSAL) qi = rows - 1 - qi;                    // the longest first
  const int hp = rest % heads;
  w.b = rest / heads;
  w.from = NEVER;
  w.to = w.kept = 0;
  int first = 0;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int qt = s.pairing == ROWS ? 2 * qi + i : qi;
    w.h[i] = s.pairing == HEADS ? 2 * hp + i : hp;
    w.q0[i] = qt * BM;
    int hi = (s.T + BN - 1) / BN;
    // keys visible to this query tile: causal alignment is bottom-right (query i sees keys <= i + T - S)
    if (CAUSAL) hi = min(hi, (w.q0[i] + BM + (s.T - s.S) + BN - 1) / BN);
    if (qt >= tiles) {
      hi = 0;
      w.q0[i] = s.S;
    }
    if (i == 1 && (HALVES || s.pairing == HEADS)) {
      first = min(first, max(hi, 0));                // (the same rows)
    } else if (hi > 0) {
      first = VAR ? attn::first_key_tile_of_warp(var, w.b, w.q0[i], s.S, s.T, BN, hi, lane) : var.first != nullptr ? min(var.first[qt], hi) : 0;
    } else {
      first = 0;
    }
    int lo = first;
    if constexpr (HALVES) {
      w.lo[i] = lo;
      w.keep[i] = VAR ? min(lo, (var.keep + BN - 1) / BN) : 0;
      w.hi[i] = w.to = w.keep[i] + max(hi - lo, 0);
      w.from = 0;
      continue;
    }
    w.keep[i] = VAR ? min(lo, (var.keep + BN - 1) / BN) : 0;
    if (lo >= hi) {                                  // (kept tiles are before lo: a tile whose window is empty has none to add)
      hi = w.keep[i] > 0 ? min(w.keep[i], hi) : 0;
      w.keep[i] = hi;
      lo = NEVER;
      w.kept = max(w.kept, hi);
    } else {
      w.from = min(w.from, lo);
      w.to = max(w.to, hi);
      w.kept = max(w.kept, w.keep[i]);
    }
    w.lo[i] = lo;
    w.hi[i] = hi;
  }
  w.hk = w.h[0] / (s.Hq / s.Hkv);
  if constexpr (HALVES) return w;
  if (w.from < NEVER) w.to = max(w.to, w.kept);
  w.kept = min(w.kept, w.from);
  return w;
}

// (SPLIT) the key tile that is n-th of an item's
__device__ __forceinline__ int nth_tile(const Item& w, int n) { return n < w.keep[0] ? n : w.lo[0] + n - w.keep[0]; }
__device__ __forceinline__ bool active(const Item& w, int i, int j) { return j < w.hi[i] && (j >= w.lo[i] || j < w.keep[i]); }
__device__ __forceinline__ bool first_of(const Item& w, int i, int j) { return j == (w.keep[i] > 0 ? 0 : w.lo[i]); }
__device__ __forceinline__ int last_of(const Item& w, int i) { return w.hi[i] - 1; }
__device__ __forceinline__ bool empty(const Item& w) { return w.kept == 0 && w.to == 0; }
__device__ __forceinline__ int walk_begin(const Item& w) { return w.kept > 0 ? 0 : w.from; }
__device__ __forceinline__ int walk_last(const Item& w) { return w.to > 0 ? w.to - 1 : w.kept - 1; }
__device__ __forceinline__ int walk_next(const Item& w, int j) { return j + 1 == w.kept && j + 1 < w.from ? w.from : j + 1; }

// The items of a CTA: every other turn runs backwards over the CTAs, so that sorted items come out even.
__device__ __forceinline__ int item_index(int turn) {
  const int g = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
  return turn * g + ((turn & 1) ? g - 1 - c : c);
}

template <int D, bool CAUSAL, bool VAR, bool SIG, bool HALVES>
__global__ void __launch_bounds__(THREADS, 1)
flash_fwd_pair_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                      __nv_bfloat16* __restrict__ out, float* __restrict__ lse, Shape shape, long long o_stride_b, long long o_stride_s, long long o_stride_h,
                      float scale_log2, Variant var, int* __restrict__ err) {
  using C = Cfg<D>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // The 128-byte swizzle atoms need tiles on 1024-byte boundaries, and there is no room to align by hand: refuse instead of overrunning.
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(err, 0, ERR_BAD_ARG);
    return;
  }
  uint8_t* sQ = smem_raw;                                  // QSTAGES pairs
  uint8_t* sKV = sQ + C::QSTAGES * 2 * C::Q_TILE;          // RING stages
  Bars* bars = reinterpret_cast<Bars*>(sKV + C::RING * C::KV_TILE);
  {
    // An earlier launch reported a timed-out wait: leave at once instead of queueing more waits behind it. One
    // thread reads the status so the whole CTA takes the same branch.
    if (threadIdx.x == 0) bars->poisoned = *reinterpret_cast<volatile int*>(err);
    __syncthreads();
    if (bars->poisoned != 0) return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->q_full[i], 1); mbar_init(&bars->q_empty[i], 1);
      mbar_init(&bars->s_full[i], 1); mbar_init(&bars->p_full[i], 4); mbar_init(&bars->o_full[i], 1);
    }
    for (int i = 0; i < C::RING; ++i) { mbar_init(&bars->kv_full[i], 1); mbar_init(&bars->kv_empty[i], 1); }
    bars->abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == MMA_WARP) { tmem_alloc(&bars->tmem_base, C::TM_COLS); tmem_relinquish(); }
  if (warp == TMA_WARP && lane == 0) { tma_prefetch_desc(&tq); tma_prefetch_desc(&tk); tma_prefetch_desc(&tv); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  volatile int* abort_flag = &bars->abort_flag;

  if (warp >= TMA_WARP) {
   regs_down<ISSUE_REGS>();
   if (warp == TMA_WARP) {
    // ------------------------------------------------------------------ TMA producer (the warp together, one lane issues)
    int slot = 0, items = 0;
    uint32_t ring_phase = 1;                               // parity that a free slot has
    bool ok = true;
    for (int turn = 0; ok; ++turn) {
      const int index = item_index(turn);
      if (turn * static_cast<int>(gridDim.x) >= shape.items) break;
      if (index >= shape.items) continue;
      const Item w = make_item<CAUSAL, VAR, HALVES>(index, shape, var, lane);
      if (empty(w)) continue;
      const int qs = items % C::QSTAGES;
      if (!mbar_wait_warp(&bars->q_empty[qs], ((items / C::QSTAGES) & 1) ^ 1, abort_flag)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
      ++items;
      auto fetch = [&](const CUtensorMap* map, int key0) -> bool {
        if (!mbar_wait_warp(&bars->kv_empty[slot], ring_phase, abort_flag)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_EMPTY); return false; }
        if (lane == 0) {
          mbar_expect_tx(&bars->kv_full[slot], C::KV_TILE);
#pragma unroll
          for (int t = 0; t < C::SUB; ++t) tma_load_4d(sKV + slot * C::KV_TILE + t * (BN * 128), map, &bars->kv_full[slot], t * 64, w.hk, key0, w.b);
        }
        __syncwarp();
        if (++slot == C::RING) { slot = 0; ring_phase ^= 1; }
        return true;
      };
      if (lane == 0) {
        // (an empty tile's rows are those past the end: zeros, which nothing reads)
        mbar_expect_tx(&bars->q_full[qs], 2 * C::Q_TILE);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int t = 0; t < C::SUB; ++t) tma_load_4d(sQ + (qs * 2 + i) * C::Q_TILE + t * (BM * 128), &tq, &bars->q_full[qs], t * 64, w.h[i], w.q0[i], w.b);
      }
      __syncwarp();
      if constexpr (HALVES) {
        // in the order in which the issuer takes them
        const int end = w.to;
        ok = fetch(&tk, nth_tile(w, 0) * BN) && (1 >= end || fetch(&tk, nth_tile(w, 1) * BN));
        for (int n = 0; ok && n < end; ++n) ok = fetch(&tv, nth_tile(w, n) * BN) && (n + 2 >= end || fetch(&tk, nth_tile(w, n + 2) * BN));
        continue;
      }
      const int end = walk_last(w);
      for (int j = walk_begin(w); ok; j = walk_next(w, j)) {
        ok = fetch(&tk, j * BN) && fetch(&tv, j * BN);
        if (j == end) break;
      }
    }
   } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp runs this loop and waits together; one elected lane issues (see mbar_wait_warp).
    constexpr uint32_t idesc_qk = make_idesc(BM, BN, 1, 1, 0, 0);
    constexpr uint32_t idesc_pv = make_idesc(BM, D, 1, 1, 0, 1);
    int turn = 0, items = 0, slot = 0;                     // items: those begun; slot: the ring's next
    uint32_t ring_phase = 0, p_phase[2] = {0, 0};
    bool ok = true;
    Item w;
    auto next_item = [&]() -> bool {
      for (;; ++turn) {
        if (turn * static_cast<int>(gridDim.x) >= shape.items) return false;
        const int index = item_index(turn);
        if (index >= shape.items) continue;
        w = make_item<CAUSAL, VAR, HALVES>(index, shape, var, lane);
        if (!empty(w)) { ++turn; ++items; return true; }
      }
    };
    auto take = [&](int& at) -> bool {                     // wait for the ring's next slot
      at = slot;
      if (!mbar_wait_warp(&bars->kv_full[slot], ring_phase, abort_flag)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_FULL); return false; }
      if (++slot == C::RING) { slot = 0; ring_phase ^= 1; }
      return true;
    };
    auto scores = [&](int i, int qs, int at) {
      const uint32_t qa = smem_u32(sQ + (qs * 2 + i) * C::Q_TILE), ka = smem_u32(sKV + at * C::KV_TILE), ts = tmem + C::TM_S + i * 128;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk >> 2) * (BM * 128) + (kk & 3) * 32;
          umma_bf16_ss(ts, make_sdesc_sw128(qa + off, 16, 1024), make_sdesc_sw128(ka + off, 16, 1024), idesc_qk, kk > 0 ? 1u : 0u);
        }
        umma_commit(&bars->s_full[i]);
      }
      __syncwarp();
    };
    auto commit = [&](uint64_t* bar) { if (elect_one()) umma_commit(bar); __syncwarp(); };
    auto await_queries = [&](int qs) -> bool {
      if (mbar_wait_warp(&bars->q_full[qs], ((items - 1) / C::QSTAGES) & 1, abort_flag)) return true;
      if (lane == 0) atomicCAS(err, 0, ERR_WAIT_FULL);
      return false;
    };
    bool more = next_item();
    int j = 0, qs = 0, k_at = 0, v_at = 0;
    auto product = [&](int i, bool fresh, bool last) -> bool {      // P V of the tile, with the values in slot v_at
      if (!mbar_wait_warp(&bars->p_full[i], p_phase[i], abort_flag)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_OTHER); return false; }
      p_phase[i] ^= 1;
      tc_fence_after();
      const uint32_t va = smem_u32(sKV + v_at * C::KV_TILE), tp = tmem + C::TM_S + i * 128, to = tmem + C::TM_O + i * 128;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk)             // 16 keys of P = 8 packed 32-bit columns
          umma_bf16_ts(to, tp + kk * 8, make_sdesc_sw128(va + kk * 2048, BN * 128, 1024), idesc_pv, kk > 0 || !fresh ? 1u : 0u);
        if (last) umma_commit(&bars->o_full[i]);
      }
      __syncwarp();
      return true;
    };
    if constexpr (HALVES) {
      // One item: the tiles' scores are in front of each other's products, as with two tiles of rows.
      const int end = w.to;
      ok = more && await_queries(0);
      for (int i = 0; ok && i < 2 && i < end; ++i) {
        ok = take(k_at);
        tc_fence_after();
        if (ok) { scores(i, 0, k_at); commit(&bars->kv_empty[k_at]); }
      }
      for (int at = 0; ok && at < end; ++at) {
        const int i = at & 1;
        ok = take(v_at) && product(i, at < 2, at + 2 >= end);
        if (!ok) break;
        commit(&bars->kv_empty[v_at]);
        if (at + 2 >= end) continue;
        ok = take(k_at);
        tc_fence_after();
        if (ok) { scores(i, 0, k_at); commit(&bars->kv_empty[k_at]); }
      }
      more = false;
    }
    if (more) {
      j = walk_begin(w);
      qs = (items - 1) % C::QSTAGES;
      ok = await_queries(qs) && take(k_at);
      tc_fence_after();
      if (ok) {
        for (int i = 0; i < 2; ++i) if (active(w, i, j)) scores(i, qs, k_at);
        commit(&bars->kv_empty[k_at]);
        if (j == walk_last(w)) commit(&bars->q_empty[qs]);
      }
    }
    while (more && ok) {
      // what this step's products are about; the walk then moves one on
      const Item now = w;
      const int at = j;
      ok = take(v_at);
      if (!ok) break;
      const bool crosses = at == walk_last(w);
      if (crosses) {
        more = next_item();
        j = more ? walk_begin(w) : 0;
        qs = more ? (items - 1) % C::QSTAGES : 0;
      } else {
        j = walk_next(w, at);
      }
      auto values = [&](int i) -> bool {
        return !active(now, i, at) || product(i, first_of(now, i, at), at == last_of(now, i));
      };
      // At an item's end the other tile's products go first: the next item's queries may still be on their way.
      if (crosses) {
        ok = values(0) && values(1);
        if (ok && more) ok = await_queries(qs) && take(k_at);
        tc_fence_after();
        if (ok && more) for (int i = 0; i < 2; ++i) if (active(w, i, j)) scores(i, qs, k_at);
      } else {
        ok = values(0) && take(k_at);
        tc_fence_after();
        if (ok && active(w, 0, j)) scores(0, qs, k_at);
        ok = ok && values(1);
        if (ok && active(w, 1, j)) scores(1, qs, k_at);
      }
      if (!ok) break;
      commit(&bars->kv_empty[v_at]);
      if (more) {
        commit(&bars->kv_empty[k_at]);
        if (j == walk_last(w)) commit(&bars->q_empty[qs]);
      }
    }
   }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue (warps 0..7)
    regs_up<SOFTMAX_REGS>();
    const int i = warp >> 2, q4 = warp & 3;
    const int r = q4 * 32 + lane;                    // query row within the tile == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + C::TM_S + i * 128, t_o = tmem + lane_addr + C::TM_O + i * 128;
    const int S = shape.S, T = shape.T;
    uint32_t s_phase = 0, o_phase = 0;
    bool ok = true;
    for (int turn = 0; ok; ++turn) {
      const int index = item_index(turn);
      if (turn * static_cast<int>(gridDim.x) >= shape.items) break;
      if (index >= shape.items) continue;
      const Item w = make_item<CAUSAL, VAR, HALVES>(index, shape, var, lane);
      // (picked, not indexed: a row's tile is known when the kernel runs)
      const int q0 = i ? w.q0[1] : w.q0[0], h = i ? w.h[1] : w.h[0], b = w.b;
      const int lo = i ? w.lo[1] : w.lo[0], hi = i ? w.hi[1] : w.hi[0], kept = i ? w.keep[1] : w.keep[0];
      const int j_first = kept > 0 ? 0 : lo;
      if (q0 >= S) continue;
      const int row = q0 + r;
      const int limit = min(CAUSAL ? row + (T - S) : T - 1, T - 1);   // last visible key of this row
      const int warp_limit = min(CAUSAL ? q0 + q4 * 32 + (T - S) : T - 1, T - 1);   // (of the warp's first row)
      float m_used = -INFINITY, l = 0.f;
      const float gained = VAR && var.gain != nullptr ? scale_log2 * var.gain[h] : scale_log2;
      const float sig2 = SIG ? var.sig[h] * LOG2E : 0.f;
      const bool any = HALVES ? i < w.to : hi > 0;
      const bool packed = VAR && var.q_seg != nullptr;
      const int mine = packed ? var.q_seg[static_cast<long long>(b) * S + min(row, S - 1)] : 0;      // this row's document
      for (int j = HALVES ? nth_tile(w, i) : j_first, n = i; any && ok; ) {
        // which keys of the tile are of this row's document, bit l of word q for key 4 l + q: found once for each of the documents that the warp's rows are of, while the
        // scores are made (T is a multiple of 4 here)
        uint32_t same[4] = {0u, 0u, 0u, 0u};
        if (packed) {
          const int key = j * BN + lane * 4;
          const int4 id = key < T ? *reinterpret_cast<const int4*>(var.k_seg + static_cast<long long>(b) * T + key) : make_int4(0, 0, 0, 0);
          for (unsigned todo = 0xffffffffu; todo != 0; ) {
            const int doc = __shfl_sync(0xffffffffu, mine, __ffs(todo) - 1);
            const bool hit = mine == doc;
            const uint32_t v[4] = {__ballot_sync(0xffffffffu, id.x == doc), __ballot_sync(0xffffffffu, id.y == doc), __ballot_sync(0xffffffffu, id.z == doc),
                                   __ballot_sync(0xffffffffu, id.w == doc)};
#pragma unroll
            for (int q = 0; q < 4; ++q) same[q] = hit ? v[q] : same[q];
            todo &= ~__ballot_sync(0xffffffffu, hit);
          }
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->s_full[i], s_phase, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_TMEM_FULL); ok = false; break; }
        s_phase ^= 1;
        tc_fence_after();
        float s[BN];
        {
          uint32_t v[4][32];                          // every load is in flight before the single wait
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(t_s + c * 32, v[c]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int x = 0; x < 32; ++x) s[c * 32 + x] = VAR ? __uint_as_float(v[c][x]) * gained : __uint_as_float(v[c][x]);
        }
        const int k0 = j * BN;
        if (VAR && var.softcap > 0.f) {
          // cap * tanh(score / cap) = cap - 2 cap / (1 + e^(2 score / cap)), kept in the log2 domain; fp32 accurate relative to the cap
          const float cap2 = var.softcap * LOG2E, twice = 2.f * LOG2E / cap2;
#pragma unroll
          for (int x = 0; x < BN; ++x) s[x] = fmaf(-2.f * cap2, __fdividef(1.f, 1.f + fast_exp2(s[x] * twice)), cap2);
        }
        if (k0 + BN - 1 > warp_limit) {
          const int past = limit - k0;
#pragma unroll
          for (int x = 0; x < BN; ++x) if (x > past) s[x] = -INFINITY;
        }
        if (VAR) {
          if (var.window > 0 || var.chunk > 0) {
            const int at = row + (T - S);
            int first = var.window > 0 ? at - var.window + 1 : 0;   // first visible key of this row
            if (var.chunk > 0) first = max(first, at / var.chunk * var.chunk);
            if (k0 < first) {
#pragma unroll
              for (int x = 0; x < BN; ++x) if (k0 + x < first && k0 + x >= var.keep) s[x] = -INFINITY;
            }
          }
          if (packed && (same[0] & same[1] & same[2] & same[3]) != 0xffffffffu) {
#pragma unroll
            for (int x = 0; x < BN; ++x) if (!(same[x & 3] >> (x >> 2) & 1)) s[x] = -INFINITY;
          }
        }
        __syncwarp();                                  // the masks above branch by row; what follows takes whole warps
        if constexpr (SIG) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int x = 0; x < 16; ++x)
              pk[x] = pack_bf16(__fdividef(1.f, 1.f + fast_exp2(-(s[c * 32 + 2 * x] + sig2))), __fdividef(1.f, 1.f + fast_exp2(-(s[c * 32 + 2 * x + 1] + sig2))));
            tmem_st_32x32b_x16(t_s + c * 16, pk);
          }
        } else {
          // independent chains, not one of 128 dependent maxima
          float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
          for (int x = 4; x < BN; x += 8) {
#pragma unroll
            for (int q = 0; q < 4; ++q) mx[q] = x + 4 + q < BN ? fmaxf(fmaxf(mx[q], s[x + q]), s[x + 4 + q]) : fmaxf(mx[q], s[x + q]);
          }
          float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
          if (!VAR) mt *= scale_log2;                  // (scale > 0 here)
          const float m_new = fmaxf(m_used, mt);
          const bool need = (m_new - m_used > RESCALE_THRESHOLD) || (m_used == -INFINITY && m_new > -INFINITY);
          if (__any_sync(0xffffffffu, need)) {
            const float alpha = (need && m_used > -INFINITY) ? fast_exp2(m_used - m_new) : 1.f;
            if (need) { m_used = m_new; l *= alpha; }
            if (HALVES ? n != i : j != j_first) {
#pragma unroll
              for (int c = 0; c < D / 16; ++c) {
                uint32_t v[16];
                tmem_ld_32x32b_x16(t_o + c * 16, v);
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 16; ++x) v[x] = __float_as_uint(__uint_as_float(v[x]) * alpha);
                tmem_st_32x32b_x16(t_o + c * 16, v);
              }
            }
          }
          // P = exp2(s - m_used) -> bf16 over the scores, which this thread holds in registers; sums in fp32, before the rounding
          const float mu = (m_used == -INFINITY) ? 0.f : m_used;
          const uint64_t factor = pair_of(VAR ? 1.f : scale_log2, VAR ? 1.f : scale_log2), shift = pair_of(-mu, -mu);
          uint64_t sum0 = 0, sum1 = 0;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int x = 0; x < 16; ++x) {
              float a, b2;
              unpair(fma2(pair_of(s[c * 32 + 2 * x], s[c * 32 + 2 * x + 1]), factor, shift), a, b2);
              a = fast_exp2(a);
              b2 = fast_exp2(b2);
              pk[x] = pack_bf16(a, b2);
              if (x & 1) sum1 = add2(sum1, pair_of(a, b2)); else sum0 = add2(sum0, pair_of(a, b2));
            }
            tmem_st_32x32b_x16(t_s + c * 16, pk);
          }
          float a, b2;
          unpair(add2(sum0, sum1), a, b2);
          l += a + b2;
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_full[i]);
        if constexpr (HALVES) {
          n += 2;
          if (n >= w.to) break;
          j = nth_tile(w, n);
        } else {
          if (j == hi - 1) break;
          ++j;
          if (VAR && j >= kept && j < lo) j = lo;
        }
      }
      // epilogue: O / l -> bf16, lse
      if (ok && any) {
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->o_full[i], o_phase, abort_flag))) { atomicCAS(err, 0, ERR_WAIT_OTHER); ok = false; }
        o_phase ^= 1;
      }
      float own = 1.f, other = 0.f;                    // what the tiles' rows weigh in the result
      if constexpr (HALVES) {
        // (every warp passes here, whatever went wrong before; with one key tile there is nothing to join)
        if (i == 1 && w.to > 1) bars->half[r] = make_float2(m_used, l);
        tc_fence_before();
        if (w.to > 1) asm volatile("bar.sync 1, 256;" ::: "memory");
        if (i == 1) { if (ok) continue; break; }
        const float2 o = w.to > 1 ? bars->half[r] : make_float2(-INFINITY, 0.f);
        // (the other half's products are complete: its warps waited for them before they came here)
        if constexpr (SIG) {
          other = w.to > 1 ? 1.f : 0.f;
        } else {
          const float m = fmaxf(m_used, o.x);
          own = m_used > -INFINITY ? fast_exp2(m_used - m) : 0.f;
          other = o.x > -INFINITY ? fast_exp2(o.x - m) : 0.f;
          l = l * own + o.y * other;
          m_used = m;
        }
      }
      if (!ok) break;
      tc_fence_after();
      float lse_shift = 0.f;     // log2 of the factor the sink adds to the denominator's scale
      float inv = SIG ? 1.f : l > 0.f ? 1.f / l : 0.f;
      if (!SIG && var.sinks != nullptr) {
        // the sink joins the denominator only: softmax over [scores, sink] with the sink's value column dropped
        const float sink2 = var.sinks[h] * LOG2E;
        const float m_fin = fmaxf(m_used, sink2);
        const float a = m_used > -INFINITY ? fast_exp2(m_used - m_fin) : 0.f;
        const float l_fin = l * a + fast_exp2(sink2 - m_fin);
        inv = a / l_fin;
        lse_shift = m_fin + log2f(l_fin);
      }
      __nv_bfloat16* orow = out + b * o_stride_b + static_cast<long long>(row) * o_stride_s + h * o_stride_h;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t v[32];
        if (any) { tmem_ld_32x32b_x32(t_o + c * 32, v); tmem_ld_wait(); }
        else {
#pragma unroll
          for (int x = 0; x < 32; ++x) v[x] = 0;
        }
        if constexpr (HALVES) {
          if (w.to > 1) {
            uint32_t u[32];
            tmem_ld_32x32b_x32(t_o + 128 + c * 32, u);
            tmem_ld_wait();
#pragma unroll
            for (int x = 0; x < 32; ++x) v[x] = __float_as_uint(own * __uint_as_float(v[x]) + (other > 0.f ? other * __uint_as_float(u[x]) : 0.f));
          }
        }
        if (row < S) store_row_32<false>(orow + c * 32, v, inv);
        __syncwarp();
      }
      if (row < S && lse != nullptr) {
        float v = l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
        if (var.sinks != nullptr) v = lse_shift * 0.6931471805599453f;
        lse[(static_cast<long long>(b) * shape.Hq + h) * S + row] = v;
      }
      tc_fence_before();                               // the next item's products over this O are told of by its p_full
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, C::TM_COLS);
  }
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

// Few tiles: both halves of a CTA on one tile's keys, a CTA an item.  Up to a tile an SM always (pairs / halves, us: 11008 causal tokens of one head of 128, 86 tiles, 163 / 88;
// 3328 tokens, 4 heads of 64, 104 tiles, 50 / 27, with a soft cap 127 / 65, packed documents 24 / 16).  Up to two tiles an SM where pairs of odd numbers of rows take a second
// wave (6 x 384, 16 heads of 64, a window, 20.5 / 17.8; of one tile 2 x 128, 100 heads, 13.1 / 14.9), and where a row's keys are many: the longest items set the pace, and are half as long by halves, but setting an
// item up takes as long as a few key tiles.  The lines, in key tiles that a row sees:
//   causal 8 (5 up to four thirds of a tile an SM)   1 x 2048, 12 heads of 128, 37.5 / 23.8   1 x 1152, 32 heads, 26.6 / 24.8   2 x 768, 16 heads of 64, a window of 512, 20.5 / 17.2
//                                                    3 x 640, 16 heads of 64, 14.3 / 16.5   1 x 896, 32 / 8 heads of 128, a window of 256, 17.2 / 22.7
//   causal, soft caps and sigmoids 3                 2 x 384, 32 / 8 heads of 128, 22.9 / 21.3 and 18.4 / 18.6   8 x 512, 8 heads of 64, 27.2 / 24.4   1 x 256, 100 heads, 15.6 / 18.6
//   not causal, chunks and documents 9               1 x 1152, 18 heads of 128, 28.7 / 20.7 and 33.0 / 23.1   1 x 1024, 32 / 8 heads, 27.4 / 28.7 and 31.5 / 31.1
//   not causal, windows and soft caps 16             1 x 3200, 8 heads of 64, 60 / 37 and 140 / 123   1 x 1152, 18 heads of 128, 28.3 / 32.0 and 52 / 55
//   not causal, else never                           1 x 3200, 8 heads of 64, 50 / 52   1 x 1152, 18 heads of 128, 25 / 30
template <bool CAUSAL, bool VAR, bool SIG>
static bool by_halves(const Shape& s, const Variant& var, int sms) {
  const int tiles = (s.S + BM - 1) / BM;
  const long long singles = static_cast<long long>(tiles) * s.Hq * s.B;
  if (singles <= sms) return true;
  if (singles > 2 * sms) return false;
  if (tiles >= 3 && (s.Hq / s.Hkv) % 2 != 0 && static_cast<long long>((tiles + 1) / 2) * s.Hq * s.B > sms) return true;
  int keys = (s.T + BN - 1) / BN;
  if (!CAUSAL) return VAR && (var.chunk > 0 || var.q_seg != nullptr ? keys >= 9 : (var.window > 0 || var.softcap > 0.f) && keys >= 16);
  if (VAR && var.window > 0) keys = min(keys, var.window / BN + 1);
  if (VAR && var.chunk > 0) keys = min(keys, (var.chunk + BN - 1) / BN);
  return keys >= (SIG || (VAR && var.softcap > 0.f) ? 3 : 3 * singles <= 4 * sms ? 5 : 8);
}

template <int D, bool CAUSAL, bool VAR, bool SIG, bool HALVES = false>
static int launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, void* out, float* lse, Shape s, long long osb, long long oss, long long osh,
                  float scale_log2, const Variant& var, int* err, cudaStream_t stream) {
  auto kern = flash_fwd_pair_kernel<D, CAUSAL, VAR, SIG, HALVES>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<D>::SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int tiles = (s.S + BM - 1) / BM, sms = multiprocessors();
  const long long singles = static_cast<long long>(tiles) * s.Hq * s.B;
  if constexpr (!HALVES)
    if (by_halves<CAUSAL, VAR, SIG>(s, var, sms)) return launch<D, CAUSAL, VAR, SIG, true>(tq, tk, tv, out, lse, s, osb, oss, osh, scale_log2, var, err, stream);
  // pairs: heads of one key head before neighbouring rows, since their key tiles are the same
  s.pairing = HALVES ? SPLIT : (s.Hq / s.Hkv) % 2 == 0 ? HEADS : ROWS;
  const long long items = HALVES ? singles : s.pairing == HEADS ? singles / 2 : static_cast<long long>((tiles + 1) / 2) * s.Hq * s.B;
  if (items > 0x3fffffff) return -3;
  s.items = static_cast<int>(items);
  kern<<<HALVES || s.items < sms ? s.items : sms, THREADS, Cfg<D>::SMEM, stream>>>(tq, tk, tv, reinterpret_cast<__nv_bfloat16*>(out), lse, s, osb, oss, osh, scale_log2, var, err);
  return static_cast<int>(cudaGetLastError());
}

// Maps with boxes of 128 rows x 64 columns; the arguments have been checked.
int run(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, void* out, float* lse, int B, int S, int T, int Hq, int Hkv, int D, long long osb, long long oss,
        long long osh, float scale_log2, int causal, const Variant& var, int* err, cudaStream_t stream) {
  const Shape s{B, S, T, Hq, Hkv, HEADS, 0};
  // what changes single scores takes kernels of its own; a first key tile and sinks do not
  const bool any = var.window > 0 || var.chunk > 0 || var.softcap > 0.f || var.q_seg != nullptr || var.gain != nullptr || !(scale_log2 > 0.f);
#define DEWB_PAIR_GO(DD, CC, VV, SS) launch<DD, CC, VV, SS>(tq, tk, tv, out, lse, s, osb, oss, osh, scale_log2, var, err, stream)
  if (var.sig != nullptr) return D == 128 ? DEWB_PAIR_GO(128, true, true, true) : DEWB_PAIR_GO(64, true, true, true);
  if (D == 128) {
    if (any) return causal ? DEWB_PAIR_GO(128, true, true, false) : DEWB_PAIR_GO(128, false, true, false);
    return causal ? DEWB_PAIR_GO(128, true, false, false) : DEWB_PAIR_GO(128, false, false, false);
  }
  if (any) return causal ? DEWB_PAIR_GO(64, true, true, false) : DEWB_PAIR_GO(64, false, true, false);
  return causal ? DEWB_PAIR_GO(64, true, false, false) : DEWB_PAIR_GO(64, false, false, false);
#undef DEWB_PAIR_GO
}

}  // namespace attnpair
}  // namespace dewb
