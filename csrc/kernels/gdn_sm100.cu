// Gated delta rule (chunk 64, 128-wide keys and values) for sm_100a: three kernels.
//
//   gdn_prepare_kernel   one CTA per 128 tokens (two chunks) of one (batch, head).  TMA brings the K, Q and V rows;
//                        K K^T and Q K^T are two 128x128x128 tcgen05 products (only the two 64x64 diagonal blocks are
//                        used); the strictly lower system (I + A) [W | U] = [beta e^g K | beta V] is solved by forward
//                        substitution in fp32, one right-hand-side column per thread, the A row broadcast from shared
//                        memory.  Writes gc (cumulative log decay inside the chunk), W, U, P = scale * (Q K^T) e^{g_i-g_j}
//                        (lower triangle) and, for the backward, Qg = scale * e^g Q.
//   gdn_scan_fwd_kernel  one CTA per (batch, head), chunks in order.  The state is kept transposed (rows = value index):
//                        fp32 in the registers of 128 threads (one value row each) and bf16 as a K-major operand tile in
//                        shared memory, so every product has M = 128:
//                          acc1 = S^T W^T, o1 = S^T Q^T            (after the state tile is written)
//                          Vn^T = U^T - acc1 ;  o2 = Vn^T P^T ;  dS = (Vn e^{g_L - g})^T K
//                          O^T = scale e^{g} o1 + o2 ;  S^T <- e^{g_L} S^T + dS
//   gdn_scan_bwd_kernel  the same walk from the last chunk to the first for the state gradient G (also transposed):
//                          a = dO^T P, b = G^T K^T ;  dVn^T = a + e^{g_L - g} b
//                          G^T <- e^{g_L} G^T + dO^T Qg - dVn^T W
//                        and stores G as it stands on entry to each chunk (the gradient of that chunk's exit state).
//
// A scan is one chain of products and of the elementwise steps between them, on B * H of the SMs, and nothing in it is near the rate of any unit; what counts is what
// stands in the chain.  Warp roles: warps 0..15 hold the state (thread = TMEM lane = value index, a quarter of the keys each, a quarter of a chunk's tokens in the steps
// over tokens) and keep it as an operand in tensor memory; two warps fetch, what the start of a chunk needs apart from the rest; one issues the products, uniformly; in
// the forward scan four write O, whose accumulators are double, beside the chain; what the backward reads (Vn, the states and their gradients) leaves as whole tiles
// through shared memory, sent by one thread.  The backward's products that need no state are issued before the state is there.  Measured for 2 x 16 heads of 8192
// tokens: with eight warps, the state's operand in shared memory, two stages of everything and stores from registers the forward walk took 400 us with the output and
// 400 with what the backward reads, the reverse walk 275; now 279, 228 and 223.  Every wait is bounded; a timed-out wait records a status code, raises
// the CTA's abort flag, and all roles leave through the common exit that frees the tensor memory.
//
// Replaces the reference's fla-style kernels KktSolve / RecomputeWU / ChunkFwdH / ChunkFwdO / ChunkBwdDhu
// (src/dew/nn/kernels/fla_gdn.py:199-795) and the recurrence template's chunk_forward / mainloop
// (src/dew/nn/kernels/templates/recurrence/).
#include "../common/ptx.cuh"
#include "../common/tmap.h"

namespace dewb {
namespace gdn {

constexpr int HD = 128;           // key and value head dimension
constexpr int CH = 64;            // chunk length
constexpr int PT = 128;           // tokens per prepare CTA
constexpr uint32_t FULL = 0xffffffffu;

// Byte offset of the 16-byte piece `c16` (8 bf16) of row `r` inside a 128-byte-swizzled tile whose rows are 128 bytes.
__device__ __forceinline__ uint32_t swz(int r, int c16) { return static_cast<uint32_t>(r * 128 + ((c16 ^ (r & 7)) << 4)); }

// ------------------------------------------------------------------------------------------------------------------
// prepare

constexpr int PREP_THREADS = 256;
constexpr int PREP_TILE = PT * HD * 2;                 // 32 KiB: a [128 x 128] bf16 tile as two 64-column sub-tiles
constexpr int PREP_SMEM = 3 * PREP_TILE + 2048;

struct PrepTail {
  float g[PT];          // cumulative log decay inside the chunk
  float beta[PT];
  float eg[PT];         // e^{g}
  float warp_sum[4];
  uint64_t bar_load, bar_mma;
  uint32_t tmem_base;
  int poisoned, abort_flag;
};
static_assert(sizeof(PrepTail) <= 2048, "PrepTail must fit its slot");

__global__ void __launch_bounds__(PREP_THREADS, 2)
gdn_prepare_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                   const __grid_constant__ CUtensorMap tv, const float* __restrict__ g, const float* __restrict__ beta,
                   float* __restrict__ gc_out, __nv_bfloat16* __restrict__ W, __nv_bfloat16* __restrict__ U,
                   __nv_bfloat16* __restrict__ P, __nv_bfloat16* __restrict__ Qg, int T, int H, int rep, int Tp, float scale,
                   int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(err, 0, ERR_BAD_ARG);
    return;
  }
  uint8_t* sK = smem;
  uint8_t* sQ = smem + PREP_TILE;
  uint8_t* sV = smem + 2 * PREP_TILE;
  float* sA = reinterpret_cast<float*>(sQ);              // the Q tile's space is reused for A once Q has been consumed
  PrepTail* tail = reinterpret_cast<PrepTail*>(smem + 3 * PREP_TILE);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) tail->poisoned = *reinterpret_cast<volatile int*>(err);
  __syncthreads();
  if (tail->poisoned != 0) return;

  const int x = blockIdx.y, b = x / H, h = x % H;
  const int t0 = blockIdx.x * PT;
  if (tid == 0) {
    mbar_init(&tail->bar_load, 1);
    mbar_init(&tail->bar_mma, 1);
    tail->abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 0) { tmem_alloc(&tail->tmem_base, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tail->tmem_base;
  volatile int* abort_flag = &tail->abort_flag;

  if (tid == 0) {
    mbar_expect_tx(&tail->bar_load, 3 * PREP_TILE);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      tma_load_4d(sK + s * (PT * 128), &tk, &tail->bar_load, s * 64, h / rep, t0, b);      // `rep` value heads share a key head
      tma_load_4d(sQ + s * (PT * 128), &tq, &tail->bar_load, s * 64, h / rep, t0, b);
      tma_load_4d(sV + s * (PT * 128), &tv, &tail->bar_load, s * 64, h, t0, b);
    }
  }
  // cumulative log decay inside each chunk (tokens past the end: no decay, no write strength)
  if (tid < PT) {
    const int t = t0 + tid;
    const bool valid = t < T;
    float gi = valid ? g[(static_cast<long long>(b) * T + t) * H + h] : 0.f;
    const float bi = valid ? beta[(static_cast<long long>(b) * T + t) * H + h] : 0.f;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float up = __shfl_up_sync(FULL, gi, d);
      if (lane >= d) gi += up;
    }
    if (lane == 31) tail->warp_sum[warp] = gi;
    tail->beta[tid] = bi;
    tail->g[tid] = gi;     // finished below for the second warp of each chunk
  }
  __syncthreads();
  if (tid < PT) {
    float gi = tail->g[tid];
    if (warp & 1) gi += tail->warp_sum[warp - 1];
    tail->g[tid] = gi;
    tail->eg[tid] = __expf(gi);
    gc_out[static_cast<long long>(x) * Tp + t0 + tid] = gi;
  }
  __syncthreads();

  bool ok = true;
  if (tid == 0) {
    if (!mbar_wait(&tail->bar_load, 0, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_FULL); }
    else {
      tc_fence_after();
      constexpr uint32_t idesc = make_idesc(128, 128, 1, 1, 0, 0);
      const uint32_t ka = smem_u32(sK), qa = smem_u32(sQ);
#pragma unroll
      for (int kk = 0; kk < HD / 16; ++kk) {
        const uint32_t off = (kk >> 2) * (PT * 128) + (kk & 3) * 32;
        umma_bf16_ss(tmem, make_sdesc_sw128(ka + off, 16, 1024), make_sdesc_sw128(ka + off, 16, 1024), idesc, kk > 0 ? 1u : 0u);
      }
#pragma unroll
      for (int kk = 0; kk < HD / 16; ++kk) {
        const uint32_t off = (kk >> 2) * (PT * 128) + (kk & 3) * 32;
        umma_bf16_ss(tmem + 128, make_sdesc_sw128(qa + off, 16, 1024), make_sdesc_sw128(ka + off, 16, 1024), idesc, kk > 0 ? 1u : 0u);
      }
      umma_commit(&tail->bar_mma);
    }
  }
  // the other lanes of the issuing thread's warp park here instead of spinning on the barrier beside it
  if (warp == 0) __syncwarp();
  {
    // (half a row a thread of all eight warps: 213 -> 203 us for 2 x 8192 tokens of 16 heads; four warps did whole rows while four waited)
    // token row i of the 128, and 32 of its chunk's 64 columns of both score matrices (half of its row of Q) a thread
    const int i = tid & 127, c = i >> 6, il = i & 63, part = warp >> 2, j0 = part * 32;
    const bool got = mbar_wait(&tail->bar_mma, 0, abort_flag);
    if (!__all_sync(FULL, got)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_TMEM_FULL); ok = false; }
    const uint32_t from = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + c * 64 + j0;
    const float gi = tail->g[i], bi = tail->beta[i];
    const long long row = static_cast<long long>(x) * Tp + t0 + i;
    float a[32];
    if (ok) {
      tc_fence_after();
      uint32_t vp[32], va[32];
      tmem_ld_32x32b_x32(from + 128, vp);
      tmem_ld_32x32b_x32(from, va);
      tmem_ld_wait();
      // P row: scale * (q_i . k_j) * e^{g_i - g_j} for j <= i;  A row: beta_i * (k_i . k_j) * e^{g_i - g_j} for j < i
#pragma unroll
      for (int j16 = 0; j16 < 2; ++j16) {
        float p[16];
#pragma unroll
        for (int jj = 0; jj < 16; ++jj) {
          const int at = j16 * 16 + jj, j = j0 + at;
          const float decay = j <= il ? __expf(gi - tail->g[c * 64 + j]) : 0.f;
          p[jj] = j <= il ? scale * __uint_as_float(vp[at]) * decay : 0.f;
          a[at] = j < il ? bi * __uint_as_float(va[at]) * decay : 0.f;
        }
        uint32_t w[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) w[x] = pack_bf16(p[2 * x], p[2 * x + 1]);
        st_global_32_any(P + row * CH + j0 + j16 * 16, w);
      }
      if (Qg != nullptr) {
        const float m = scale * tail->eg[i];
#pragma unroll
        for (int c32 = 0; c32 < 4; ++c32) {
          const uint4 a = *reinterpret_cast<const uint4*>(sQ + part * (PT * 128) + swz(i, 2 * c32)), b = *reinterpret_cast<const uint4*>(sQ + part * (PT * 128) + swz(i, 2 * c32 + 1));
          const uint32_t in[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
          uint32_t w[8];
#pragma unroll
          for (int x = 0; x < 8; ++x) w[x] = pack_bf16(bf16_lo(in[x]) * m, bf16_hi(in[x]) * m);
          st_global_32_any(Qg + row * HD + part * 64 + c32 * 16, w);
        }
      }
    }
    // every row of Q has been read (by the tensor core and by its threads) before A overwrites the tile
    __syncthreads();
    if (ok) {
      // row i of chunk c at sA[c][il][.], its columns rotated by 4 * il so that neither these stores nor the broadcast
      // reads of the solve meet a bank conflict
      float4* arow = reinterpret_cast<float4*>(sA + c * (CH * CH) + il * CH);
#pragma unroll
      for (int j4 = 0; j4 < 8; ++j4)
        arow[(part * 8 + j4 + il) & 15] = make_float4(a[j4 * 4], a[j4 * 4 + 1], a[j4 * 4 + 2], a[j4 * 4 + 3]);
    }
    tc_fence_before();
  }
  __syncthreads();
  if (tail->abort_flag == 0) {
    // forward substitution: thread = one column of [W | U]; x_i = r_i - sum_{j < i} A_ij x_j
    const int col = tid & 127;
    const bool is_w = tid < 128;
    const uint8_t* src = (is_w ? sK : sV) + (col >> 6) * (PT * 128) + (col & 7) * 2;
    const int c16 = (col & 63) >> 3;
    __nv_bfloat16* dst = (is_w ? W : U) + (static_cast<long long>(x) * Tp + t0) * HD + col;
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
      float xv[CH];
#pragma unroll
      for (int i = 0; i < CH; ++i) xv[i] = 0.f;
      const float* Ac = sA + c * (CH * CH);
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int r = c * 64 + i;
        const float raw = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(src + swz(r, c16)));
        float acc = raw * tail->beta[r] * (is_w ? tail->eg[r] : 1.f), acc1 = 0.f;      // two chains per row
        const float4* arow = reinterpret_cast<const float4*>(Ac + i * CH);
#pragma unroll
        for (int j4 = 0; j4 < (i + 3) / 4; ++j4) {
          const float4 av = arow[(j4 + i) & 15];
          acc = fmaf(-av.x, xv[j4 * 4], acc);
          acc1 = fmaf(-av.y, xv[j4 * 4 + 1], acc1);
          acc = fmaf(-av.z, xv[j4 * 4 + 2], acc);
          acc1 = fmaf(-av.w, xv[j4 * 4 + 3], acc1);
        }
        acc += acc1;
        xv[i] = acc;
        dst[static_cast<long long>(r) * HD] = __float2bfloat16(acc);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// scans

constexpr int STATE_WARPS = 16, OUT_WARPS = 4;
constexpr int KEYS = HD * 4 / STATE_WARPS;             // of the state, held by one thread (32)
constexpr int TOKENS = CH * 4 / STATE_WARPS;           // of a chunk, in its steps over tokens (16)
constexpr int T16 = CH * HD * 2;                       // 16 KiB: a [64 x 128] bf16 tile (two 64-column sub-tiles)
constexpr int T8 = CH * CH * 2;                        // 8 KiB: P

// Backward: what the start of a chunk needs (dO, Qg, K, P, g) in two slots that are free early in the chunk, W in three.  With `SEND` the chunks' exit-state gradients and
// dVn leave as bf16 tiles that one thread sends to memory; without, the state gradients in fp32 by the threads that hold them.
template <bool SEND>
struct Bwd {
  static constexpr int A = 2, W = 3;
  static constexpr int A_SLOT = 3 * T16 + T8;
  static constexpr int OFF_A = 0, OFF_WT = A * A_SLOT, OFF_DVN = OFF_WT + W * T16;      // DVN: -dVn^T [128 x 64] as an operand
  static constexpr int OFF_OUT = OFF_DVN + T16, OFF_ST = OFF_OUT + (SEND ? T16 : 0);     // dVn [64 x 128] and the state gradient [key][value] on their way to memory
  static constexpr int OFF_G = OFF_ST + (SEND ? 2 * T16 : 0), OFF_BARS = OFF_G + A * CH * 4, OFF_W = OFF_BARS + 256;      // OFF_W: a warp's own copy of its tokens' decays
  static constexpr int SMEM = OFF_W + STATE_WARPS * TOKENS * 4;
  static constexpr int SEND_WARP = STATE_WARPS, TMA_WARP = STATE_WARPS + 1, TMA2_WARP = TMA_WARP + 1, MMA_WARP = TMA_WARP + 2, THREADS = 32 * (MMA_WARP + 1);
  static_assert(SMEM <= 232448, "scan kernels exceed the shared memory of an SM");
};

struct BwdBars {
  uint64_t a_full[2], a_empty[2], w_full[3], w_empty[3];
  uint64_t s_ready, acc_full, vn_ready, ds_full, tile_ready, state_sent, vn_sent;
  uint32_t tmem_base;
  int abort_flag, poisoned;
};
static_assert(sizeof(BwdBars) <= 256, "BwdBars must fit its slot");

// Forward: W, U and g in three slots, Q in three, K and P in as many as there is room for.  A chunk's share arrives some 2.3 us after its slot is free, and what the start
// of a chunk needs is free early in the one it was for, so a third slot there covers what two stages of everything did not: the walk waited for its tiles for two of
// every five cycles.  With `OUT` the output is written (by four warps); without, what the backward reads: the states in front of the chunks and Vn, as tiles that one
// thread sends to memory, since 48 scattered stores a thread and chunk stood in the chain for half of its time.
template <bool OUT>
struct Fwd {
  static constexpr int AB = 3, C = OUT ? 2 : 3;                        // slots
  static constexpr int A_SLOT = 2 * T16, C_SLOT = T16 + (OUT ? T8 : 0);
  static constexpr int OFF_A = 0, OFF_Q = AB * A_SLOT, OFF_C = OFF_Q + (OUT ? AB * T16 : 0), OFF_VD = OFF_C + C * C_SLOT;
  static constexpr int OFF_VN = OFF_VD + T16;                          // OUT: Vn^T [128 x 64] as an operand; else Vn [64 x 128] on its way to memory
  static constexpr int OFF_ST = OFF_VN + T16;                          // the state [128 x 128] on its way to memory
  static constexpr int OFF_G = OFF_ST + (OUT ? 0 : 2 * T16);
  static constexpr int OFF_BARS = OFF_G + AB * CH * 4, OFF_W = OFF_BARS + 256;
  static constexpr int SMEM = OFF_W + (STATE_WARPS * TOKENS + (OUT ? OUT_WARPS * CH : 0)) * 4;
  static constexpr int EXTRA = OUT ? OUT_WARPS : 1;                    // output warps, or the one that sends tiles off
  static constexpr int TMA_WARP = STATE_WARPS + EXTRA, TMA2_WARP = TMA_WARP + 1, MMA_WARP = TMA_WARP + 2, THREADS = 32 * (MMA_WARP + 1);
  static_assert(SMEM <= 232448, "scan kernels exceed the shared memory of an SM");
};

struct FwdBars {
  uint64_t a_full[3], a_empty[3], q_full[3], q_empty[3], c_full[3], c_empty[3];
  uint64_t s_ready, acc_full, vn_ready, ds_full, o_full[2], o_read[2], tile_ready, state_sent, vn_sent;
  uint32_t tmem_base;
  int abort_flag, poisoned;
};
static_assert(sizeof(FwdBars) <= 256, "FwdBars must fit its slot");

__device__ __forceinline__ uint4 pack8(const float* v) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}

// Writes this thread's part of a row of the transposed state as bf16 to the tensor-memory operand (two keys a 32-bit column).
__device__ __forceinline__ void write_state_row(uint32_t operand, const float (&S)[KEYS]) {
  uint32_t w[KEYS / 2];
#pragma unroll
  for (int d = 0; d < KEYS / 2; ++d) w[d] = pack_bf16(S[2 * d], S[2 * d + 1]);
  tmem_st_32x32b_x16(operand, w);
  tmem_st_wait();
}

// This thread's part of a row of a state [key][value] in memory, or zeros.
__device__ __forceinline__ void read_state(float (&S)[KEYS], const float* states, int x, int v, int part) {
  if (states == nullptr) {
#pragma unroll
    for (int d = 0; d < KEYS; ++d) S[d] = 0.f;
  } else {
    const float* src = states + (static_cast<long long>(x) * HD + part * KEYS) * HD + v;
#pragma unroll
    for (int d = 0; d < KEYS; ++d) S[d] = src[d * HD];
  }
}

struct ScanCommon {
  uint8_t* smem;
  uint32_t tmem;
  volatile int* abort_flag;
};

// Common prologue: status check, barriers (`init`, by one thread), tensor memory.  Returns false if the CTA must leave at once.
template <typename Bars, typename Init>
__device__ __forceinline__ bool scan_prologue(uint8_t* smem, Bars* bars, int* err, ScanCommon& sc, int alloc_warp, Init init) {
  if ((smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(err, 0, ERR_BAD_ARG);
    return false;
  }
  if (threadIdx.x == 0) bars->poisoned = *reinterpret_cast<volatile int*>(err);
  __syncthreads();
  if (bars->poisoned != 0) return false;
  if (threadIdx.x == 0) {
    init();
    mbar_init(&bars->s_ready, STATE_WARPS);
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->vn_ready, STATE_WARPS);
    mbar_init(&bars->ds_full, 1);
    bars->abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if ((threadIdx.x >> 5) == alloc_warp) { tmem_alloc(&bars->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  sc.smem = smem;
  sc.tmem = bars->tmem_base;
  sc.abort_flag = &bars->abort_flag;
  return true;
}

__device__ __forceinline__ void scan_epilogue(const ScanCommon& sc, int alloc_warp) {
  tc_fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == alloc_warp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(sc.tmem, 512);
  }
}

// Warp-uniform bounded wait.
__device__ __forceinline__ bool math_wait(uint64_t* bar, uint32_t parity, const ScanCommon& sc, int* err, int code) {
  const bool got = mbar_wait(bar, parity, sc.abort_flag);
  if (!__all_sync(FULL, got)) {
    if ((threadIdx.x & 31) == 0) atomicCAS(err, 0, code);
    return false;
  }
  return true;
}

template <bool OUT>
__global__ void __launch_bounds__(Fwd<OUT>::THREADS, 1)
gdn_scan_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                    const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap tu,
                    const __grid_constant__ CUtensorMap tp, const __grid_constant__ CUtensorMap tstates, const __grid_constant__ CUtensorMap tvn,
                    const float* __restrict__ gc, const float* __restrict__ initial, __nv_bfloat16* __restrict__ out, float* __restrict__ final_state,
                    __nv_bfloat16* __restrict__ states, __nv_bfloat16* __restrict__ vn_out, int T, int H, int rep, int Tp, int N, float scale, int* __restrict__ err) {
  using F = Fwd<OUT>;
  extern __shared__ __align__(1024) uint8_t smem[];
  FwdBars* bars = reinterpret_cast<FwdBars*>(smem + F::OFF_BARS);
  ScanCommon sc;
  if (!scan_prologue(smem, bars, err, sc, F::MMA_WARP, [&]() {
        for (int i = 0; i < 3; ++i) {
          mbar_init(&bars->a_full[i], 1); mbar_init(&bars->a_empty[i], STATE_WARPS + (OUT ? OUT_WARPS : 0) + 1);
          mbar_init(&bars->q_full[i], 1); mbar_init(&bars->q_empty[i], 1);
          mbar_init(&bars->c_full[i], 1); mbar_init(&bars->c_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) { mbar_init(&bars->o_full[i], 1); mbar_init(&bars->o_read[i], OUT_WARPS); }
        mbar_init(&bars->tile_ready, STATE_WARPS);
        mbar_init(&bars->state_sent, 1);
        mbar_init(&bars->vn_sent, 1);
      })) return;
  const uint32_t tmem = sc.tmem;
  volatile int* abort_flag = sc.abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int x = blockIdx.x, b = x / H, h = x % H;
  uint8_t* sVn = smem + F::OFF_VN;
  uint8_t* sVd = smem + F::OFF_VD;
  float* sG = reinterpret_cast<float*>(smem + F::OFF_G);
  constexpr int TM_ACC1 = 0, TM_O1 = 64, TM_O2 = 192, TM_ST = 320, TM_DS = 384;       // O1 and O2 by the parity of the chunk, 64 columns apart; ST: the state as an operand
  const int v = tid & 127;                               // value index == TMEM lane == row of the transposed state
  const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;

  if (warp == F::TMA_WARP) {
    // W, U, g and Q
    if (lane == 0) {
      tma_prefetch_desc(&tq); tma_prefetch_desc(&tw); tma_prefetch_desc(&tu);
      for (int n = 0; n < N; ++n) {
        const int s = n % F::AB; const uint32_t ph = (n / F::AB) & 1;
        const int row = x * Tp + n * CH;
        if (!mbar_wait(&bars->a_empty[s], ph ^ 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
        uint8_t* st = smem + F::OFF_A + s * F::A_SLOT;
        mbar_expect_tx(&bars->a_full[s], F::A_SLOT + CH * 4);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          tma_load_2d(st + t * (CH * 128), &tw, &bars->a_full[s], t * 64, row);
          tma_load_2d(st + T16 + t * (CH * 128), &tu, &bars->a_full[s], t * 64, row);
        }
        bulk_load_1d(sG + s * CH, gc + static_cast<long long>(x) * Tp + n * CH, CH * 4, &bars->a_full[s]);
        if (OUT) {
          if (!mbar_wait(&bars->q_empty[s], ph ^ 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
          mbar_expect_tx(&bars->q_full[s], T16);
#pragma unroll
          for (int t = 0; t < 2; ++t) tma_load_4d(smem + F::OFF_Q + s * T16 + t * (CH * 128), &tq, &bars->q_full[s], t * 64, h / rep, n * CH, b);
        }
      }
    }
  } else if (warp == F::TMA2_WARP) {
    // K and P
    if (lane == 0) {
      tma_prefetch_desc(&tk); tma_prefetch_desc(&tp);
      for (int n = 0; n < N; ++n) {
        const int s = n % F::C; const uint32_t ph = (n / F::C) & 1;
        if (!mbar_wait(&bars->c_empty[s], ph ^ 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
        uint8_t* st = smem + F::OFF_C + s * F::C_SLOT;
        mbar_expect_tx(&bars->c_full[s], F::C_SLOT);
#pragma unroll
        for (int t = 0; t < 2; ++t) tma_load_4d(st + t * (CH * 128), &tk, &bars->c_full[s], t * 64, h / rep, n * CH, b);
        if (OUT) tma_load_2d(st + T16, &tp, &bars->c_full[s], 0, x * Tp + n * CH);
      }
    }
  } else if (warp == F::MMA_WARP) {
    constexpr uint32_t idesc_n64 = make_idesc(128, 64, 1, 1, 0, 0);
    constexpr uint32_t idesc_ds = make_idesc(128, 128, 1, 1, 0, 1);
    const uint32_t vna = smem_u32(sVn), vda = smem_u32(sVd);
    for (int n = 0; n < N; ++n) {
      const int s = n & 1, sa = n % F::AB, sk = n % F::C; const uint32_t pa = (n / F::AB) & 1, pk = (n / F::C) & 1;
      const uint32_t wa = smem_u32(smem + F::OFF_A + sa * F::A_SLOT), qa = smem_u32(smem + F::OFF_Q + sa * T16), ka = smem_u32(smem + F::OFF_C + sk * F::C_SLOT);
      if (!math_wait(&bars->a_full[sa], pa, sc, err, ERR_WAIT_FULL)) break;
      if (!math_wait(&bars->s_ready, n & 1, sc, err, ERR_WAIT_OTHER)) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t boff = (kk >> 2) * (CH * 128) + (kk & 3) * 32;
          umma_bf16_ts(tmem + TM_ACC1, tmem + TM_ST + kk * 8, make_sdesc_sw128(wa + boff, 16, 1024), idesc_n64, kk > 0 ? 1u : 0u);
        }
        umma_commit(&bars->acc_full);
        umma_commit(&bars->a_empty[sa]);
      }
      __syncwarp();
      if (OUT) {
        if (!math_wait(&bars->q_full[sa], pa, sc, err, ERR_WAIT_FULL)) break;
        if (n > 1 && !math_wait(&bars->o_read[s], ((n >> 1) - 1) & 1, sc, err, ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) {
            const uint32_t boff = (kk >> 2) * (CH * 128) + (kk & 3) * 32;
            umma_bf16_ts(tmem + TM_O1 + s * 64, tmem + TM_ST + kk * 8, make_sdesc_sw128(qa + boff, 16, 1024), idesc_n64, kk > 0 ? 1u : 0u);
          }
          umma_commit(&bars->q_empty[sa]);
        }
        __syncwarp();
      }
      if (!math_wait(&bars->c_full[sk], pk, sc, err, ERR_WAIT_FULL)) break;
      if (!math_wait(&bars->vn_ready, n & 1, sc, err, ERR_WAIT_OTHER)) break;
      tc_fence_after();
      if (elect_one()) {
        // the state's product first: the chain waits for it (and for all before it, so that O1 is done with the state)
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk) {
          umma_bf16_ss(tmem + TM_DS, make_sdesc_sw128(vda + kk * 32, 16, 1024), make_sdesc_sw128(ka + kk * 2048, CH * 128, 1024), idesc_ds, kk > 0 ? 1u : 0u);
        }
        umma_commit(&bars->ds_full);
        if (OUT) {
#pragma unroll
          for (int kk = 0; kk < CH / 16; ++kk) {
            umma_bf16_ss(tmem + TM_O2 + s * 64, make_sdesc_sw128(vna + kk * 32, 16, 1024), make_sdesc_sw128(ka + T16 + kk * 32, 16, 1024),
                         idesc_n64, kk > 0 ? 1u : 0u);
          }
          umma_commit(&bars->o_full[s]);                 // Vn's tile is rewritten only after the next acc_full, which comes behind this product
        }
        umma_commit(&bars->c_empty[sk]);
      }
      __syncwarp();
    }
  } else if (warp >= STATE_WARPS) {
    if constexpr (OUT) {
      float* w = reinterpret_cast<float*>(smem + F::OFF_W) + STATE_WARPS * TOKENS + (warp - STATE_WARPS) * CH;
      for (int n = 0; n < N; ++n) {
        const int s = n & 1, sa = n % F::AB;
        const float* gs = sG + sa * CH;
        if (!math_wait(&bars->a_full[sa], (n / F::AB) & 1, sc, err, ERR_WAIT_FULL)) break;
        w[lane] = scale * __expf(gs[lane]);
        w[lane + 32] = scale * __expf(gs[lane + 32]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->a_empty[sa]);
        if (!math_wait(&bars->o_full[s], (n >> 1) & 1, sc, err, ERR_WAIT_TMEM_FULL)) break;
        tc_fence_after();
        // O^T row
        __nv_bfloat16* orow = out + ((static_cast<long long>(b) * T + n * CH) * H + h) * HD + v;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t o1[16], o2[16];
          tmem_ld_32x32b_x16(tmem + lane_addr + TM_O1 + s * 64 + q * 16, o1);
          tmem_ld_32x32b_x16(tmem + lane_addr + TM_O2 + s * 64 + q * 16, o2);
          tmem_ld_wait();
#pragma unroll
          for (int ii = 0; ii < 16; ++ii) {
            const int i = q * 16 + ii;
            const float o = w[i] * __uint_as_float(o1[ii]) + __uint_as_float(o2[ii]);
            if (out != nullptr && n * CH + i < T) orow[static_cast<long long>(i) * H * HD] = __float2bfloat16(o);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->o_read[s]);
      }
    } else if (lane == 0) {
      // the tiles on their way to memory
      for (int n = 0; n < N; ++n) {
        if (!mbar_wait(&bars->tile_ready, n & 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_OTHER); break; }
#pragma unroll
        for (int t = 0; t < 2; ++t) tma_store_2d(&tstates, smem + F::OFF_ST + t * (HD * 128), t * 64, (x * N + n) * HD);
        tma_store_commit();
        tma_store_wait_read<0>();
        mbar_arrive(&bars->state_sent);
        if (!mbar_wait(&bars->vn_ready, n & 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_OTHER); break; }
#pragma unroll
        for (int t = 0; t < 2; ++t) tma_store_2d(&tvn, smem + F::OFF_VN + t * (CH * 128), t * 64, x * Tp + n * CH);
        tma_store_commit();
        tma_store_wait_read<0>();
        mbar_arrive(&bars->vn_sent);
      }
      tma_store_wait<0>();
    }
  } else {
    const int part = warp >> 2, j0 = part * TOKENS;      // this thread's keys KEYS part .., and its tokens of a chunk
    float* w = reinterpret_cast<float*>(smem + F::OFF_W) + warp * TOKENS;
    const uint32_t operand = tmem + lane_addr + TM_ST + part * (KEYS / 2);
    uint8_t* srow = smem + F::OFF_ST + (part >> 1) * (HD * 128);
    float S[KEYS];
    // the state as the operand of the next products, then (not OUT) as a row of the tile that goes to memory
    auto deliver = [&](bool last) {
      write_state_row(operand, S);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->s_ready);
      if (!OUT && !last) {
#pragma unroll
        for (int c = 0; c < KEYS / 8; ++c) *reinterpret_cast<uint4*>(srow + swz(v, (part & 1) * 4 + c)) = pack8(S + c * 8);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->tile_ready);
      }
    };
    read_state(S, initial, x, v, part);
    deliver(false);
    bool ok = true;
    for (int n = 0; n < N && ok; ++n) {
      const int sa = n % F::AB;
      const uint8_t* st = smem + F::OFF_A + sa * F::A_SLOT;
      const float* gs = sG + sa * CH;
      if (!math_wait(&bars->a_full[sa], (n / F::AB) & 1, sc, err, ERR_WAIT_FULL)) { ok = false; break; }
      const float gl = gs[CH - 1];
      // Vn^T row: U[j][v] - acc1[j]; the copy for the state update carries e^{g_L - g_j}.  U and the decays are read while the product runs.
      const uint8_t* ucol = st + T16 + (v >> 6) * (CH * 128) + (v & 7) * 2;
      const int uc16 = (v & 63) >> 3;
      uint32_t u[TOKENS / 2];                            // U, then Vn
#pragma unroll
      for (int jj = 0; jj < TOKENS / 2; ++jj)
        u[jj] = *reinterpret_cast<const uint16_t*>(ucol + swz(j0 + 2 * jj, uc16)) |
                static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(ucol + swz(j0 + 2 * jj + 1, uc16))) << 16;
      if (lane < TOKENS) w[lane] = __expf(gl - gs[j0 + lane]);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->a_empty[sa]);
      if (!OUT && n > 0 && !math_wait(&bars->vn_sent, (n - 1) & 1, sc, err, ERR_WAIT_OTHER)) { ok = false; break; }
      if (!math_wait(&bars->acc_full, n & 1, sc, err, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      {
        uint32_t a[TOKENS];
        tmem_ld_32x32b_x16(tmem + lane_addr + TM_ACC1 + j0, a);
        tmem_ld_wait();
#pragma unroll
        for (int j8 = 0; j8 < TOKENS / 8; ++j8) {
          float vn[8], vd[8];
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) {
            const uint32_t pair = u[j8 * 4 + (jj >> 1)];
            vn[jj] = ((jj & 1) ? bf16_hi(pair) : bf16_lo(pair)) - __uint_as_float(a[j8 * 8 + jj]);
            vd[jj] = vn[jj] * w[j8 * 8 + jj];
          }
          const uint4 packed = pack8(vn);
          u[j8 * 4] = packed.x; u[j8 * 4 + 1] = packed.y; u[j8 * 4 + 2] = packed.z; u[j8 * 4 + 3] = packed.w;
          *reinterpret_cast<uint4*>(sVd + swz(v, part * (TOKENS / 8) + j8)) = pack8(vd);
          if (OUT) *reinterpret_cast<uint4*>(sVn + swz(v, part * (TOKENS / 8) + j8)) = packed;
        }
      }
      if (!OUT) {
        uint8_t* ncol = sVn + (v >> 6) * (CH * 128) + (v & 7) * 2;
#pragma unroll
        for (int jj = 0; jj < TOKENS; ++jj) *reinterpret_cast<uint16_t*>(ncol + swz(j0 + jj, uc16)) = static_cast<uint16_t>(u[jj >> 1] >> (jj & 1) * 16);
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->vn_ready);
      if (OUT && vn_out != nullptr) {
        uint16_t* dst = reinterpret_cast<uint16_t*>(vn_out) + (static_cast<long long>(x) * Tp + n * CH + j0) * HD + v;
#pragma unroll
        for (int jj = 0; jj < TOKENS; ++jj) dst[jj * HD] = static_cast<uint16_t>(u[jj >> 1] >> (jj & 1) * 16);
      }
      if (OUT && states != nullptr) {
        // the state on entry to this chunk, as the operand holds it (row v = 128 bf16)
        uint4* dst = reinterpret_cast<uint4*>(states + ((static_cast<long long>(x) * N + n) * HD + v) * HD + part * KEYS);
#pragma unroll
        for (int c16 = 0; c16 < KEYS / 8; ++c16) dst[c16] = pack8(S + c16 * 8);
      }
      if (!OUT && !math_wait(&bars->state_sent, n & 1, sc, err, ERR_WAIT_OTHER)) { ok = false; break; }
      if (!math_wait(&bars->ds_full, n & 1, sc, err, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      // S^T <- e^{g_L} S^T + dS
      const float dl = __expf(gl);
      {
        uint32_t d[KEYS];
        tmem_ld_32x32b_x32(tmem + lane_addr + TM_DS + part * KEYS, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < KEYS; ++i) S[i] = fmaf(S[i], dl, __uint_as_float(d[i]));
      }
      deliver(n + 1 == N);
    }
    if (ok && final_state != nullptr) {
      float* dst = final_state + (static_cast<long long>(x) * HD + part * KEYS) * HD + v;
#pragma unroll
      for (int d = 0; d < KEYS; ++d) dst[d * HD] = S[d];
    }
  }
  scan_epilogue(sc, F::MMA_WARP);
}

template <bool SEND>
__global__ void __launch_bounds__(Bwd<SEND>::THREADS, 1)
gdn_scan_bwd_kernel(const __grid_constant__ CUtensorMap tdo, const __grid_constant__ CUtensorMap tk,
                    const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap tqg,
                    const __grid_constant__ CUtensorMap tp, const __grid_constant__ CUtensorMap tstates, const __grid_constant__ CUtensorMap tvn,
                    const float* __restrict__ gc, const float* __restrict__ d_final, float* __restrict__ dstates, __nv_bfloat16* __restrict__ dstates_bf16,
                    __nv_bfloat16* __restrict__ dvn_out, float* __restrict__ d_initial, int T, int H, int rep,
                    int Tp, int N, int* __restrict__ err) {
  using F = Bwd<SEND>;
  extern __shared__ __align__(1024) uint8_t smem[];
  BwdBars* bars = reinterpret_cast<BwdBars*>(smem + F::OFF_BARS);
  ScanCommon sc;
  if (!scan_prologue(smem, bars, err, sc, F::MMA_WARP, [&]() {
        for (int i = 0; i < F::A; ++i) { mbar_init(&bars->a_full[i], 1); mbar_init(&bars->a_empty[i], STATE_WARPS + 1); }
        for (int i = 0; i < F::W; ++i) { mbar_init(&bars->w_full[i], 1); mbar_init(&bars->w_empty[i], 1); }
        mbar_init(&bars->tile_ready, STATE_WARPS);
        mbar_init(&bars->state_sent, 1);
        mbar_init(&bars->vn_sent, 1);
      })) return;
  const uint32_t tmem = sc.tmem;
  volatile int* abort_flag = sc.abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int x = blockIdx.x, b = x / H, h = x % H;
  uint8_t* sDvn = smem + F::OFF_DVN;                     // -dVn^T as bf16
  float* sG = reinterpret_cast<float*>(smem + F::OFF_G);
  constexpr int TM_A = 0, TM_B = 128, TM_ST = 192, TM_DD = 256;       // A and DD by the parity of the step, 64 and 128 columns apart; ST: G^T as an operand
  constexpr int B_DO = 0, B_QG = T16, B_K = 2 * T16, B_P = 3 * T16;   // in a slot

  if (warp == F::TMA_WARP) {
    if (lane == 0) {
      tma_prefetch_desc(&tdo); tma_prefetch_desc(&tk); tma_prefetch_desc(&tqg); tma_prefetch_desc(&tp);
      for (int it = 0; it < N; ++it) {
        const int n = N - 1 - it;
        const int s = it & 1; const uint32_t ph = (it >> 1) & 1;
        if (!mbar_wait(&bars->a_empty[s], ph ^ 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
        uint8_t* st = smem + F::OFF_A + s * F::A_SLOT;
        uint64_t* bar = &bars->a_full[s];
        mbar_expect_tx(bar, F::A_SLOT + CH * 4);
        const int row = x * Tp + n * CH;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          tma_load_4d(st + B_K + t * (CH * 128), &tk, bar, t * 64, h / rep, n * CH, b);
          tma_load_4d(st + B_DO + t * (CH * 128), &tdo, bar, t * 64, h, n * CH, b);
          tma_load_2d(st + B_QG + t * (CH * 128), &tqg, bar, t * 64, row);
        }
        tma_load_2d(st + B_P, &tp, bar, 0, row);
        bulk_load_1d(sG + s * CH, gc + static_cast<long long>(x) * Tp + n * CH, CH * 4, bar);
      }
    }
  } else if (warp == F::TMA2_WARP) {
    if (lane == 0) {
      tma_prefetch_desc(&tw);
      for (int it = 0; it < N; ++it) {
        const int s = it % F::W; const uint32_t ph = (it / F::W) & 1;
        if (!mbar_wait(&bars->w_empty[s], ph ^ 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); break; }
        mbar_expect_tx(&bars->w_full[s], T16);
#pragma unroll
        for (int t = 0; t < 2; ++t) tma_load_2d(smem + F::OFF_WT + s * T16 + t * (CH * 128), &tw, &bars->w_full[s], t * 64, x * Tp + (N - 1 - it) * CH);
      }
    }
  } else if (warp == F::MMA_WARP) {
    constexpr uint32_t idesc_a = make_idesc(128, 64, 1, 1, 1, 1);      // dO^T P: both operands MN-major
    constexpr uint32_t idesc_b = make_idesc(128, 64, 1, 1, 0, 0);      // G^T K^T: both K-major
    constexpr uint32_t idesc_dq = make_idesc(128, 128, 1, 1, 1, 1);    // dO^T Qg
    constexpr uint32_t idesc_dw = make_idesc(128, 128, 1, 1, 0, 1);    // (-dVn^T) W
    const uint32_t dva = smem_u32(sDvn);
    for (int it = 0; it < N; ++it) {
      const int s = it & 1, sw = it % F::W; const uint32_t ph = (it >> 1) & 1;
      const uint32_t st = smem_u32(smem + F::OFF_A + s * F::A_SLOT), wa = smem_u32(smem + F::OFF_WT + sw * T16);
      if (!math_wait(&bars->a_full[s], ph, sc, err, ERR_WAIT_FULL)) break;
      tc_fence_after();
      if (elect_one()) {
        // what needs no state, into the half of the accumulators that the step before last has left
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk) {
          umma_bf16_ss(tmem + TM_A + s * 64, make_sdesc_sw128(st + B_DO + kk * 2048, CH * 128, 1024),
                       make_sdesc_sw128(st + B_P + kk * 2048, CH * 128, 1024), idesc_a, kk > 0 ? 1u : 0u);
        }
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk) {
          umma_bf16_ss(tmem + TM_DD + s * 128, make_sdesc_sw128(st + B_DO + kk * 2048, CH * 128, 1024),
                       make_sdesc_sw128(st + B_QG + kk * 2048, CH * 128, 1024), idesc_dq, kk > 0 ? 1u : 0u);
        }
      }
      __syncwarp();
      if (!math_wait(&bars->s_ready, it & 1, sc, err, ERR_WAIT_OTHER)) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t boff = (kk >> 2) * (CH * 128) + (kk & 3) * 32;
          umma_bf16_ts(tmem + TM_B, tmem + TM_ST + kk * 8, make_sdesc_sw128(st + B_K + boff, 16, 1024), idesc_b, kk > 0 ? 1u : 0u);
        }
        umma_commit(&bars->acc_full);
        umma_commit(&bars->a_empty[s]);
      }
      __syncwarp();
      if (!math_wait(&bars->w_full[sw], (it / F::W) & 1, sc, err, ERR_WAIT_FULL)) break;
      if (!math_wait(&bars->vn_ready, it & 1, sc, err, ERR_WAIT_OTHER)) break;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < CH / 16; ++kk) {
          umma_bf16_ss(tmem + TM_DD + s * 128, make_sdesc_sw128(dva + kk * 32, 16, 1024),
                       make_sdesc_sw128(wa + kk * 2048, CH * 128, 1024), idesc_dw, 1u);
        }
        umma_commit(&bars->ds_full);
        umma_commit(&bars->w_empty[sw]);
      }
      __syncwarp();
    }
  } else if (warp == F::SEND_WARP) {
    if (SEND && lane == 0) {
      for (int it = 0; it < N; ++it) {
        const int n = N - 1 - it;
        if (!mbar_wait(&bars->tile_ready, it & 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_OTHER); break; }
#pragma unroll
        for (int t = 0; t < 2; ++t) tma_store_2d(&tstates, smem + F::OFF_ST + t * (HD * 128), t * 64, (x * N + n) * HD);
        tma_store_commit();
        tma_store_wait_read<0>();
        mbar_arrive(&bars->state_sent);
        if (!mbar_wait(&bars->vn_ready, it & 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_OTHER); break; }
#pragma unroll
        for (int t = 0; t < 2; ++t) tma_store_2d(&tvn, smem + F::OFF_OUT + t * (CH * 128), t * 64, x * Tp + n * CH);
        tma_store_commit();
        tma_store_wait_read<0>();
        mbar_arrive(&bars->vn_sent);
      }
      tma_store_wait<0>();
    }
  } else {
    const int v = tid & 127, part = warp >> 2, j0 = part * TOKENS;      // as in the forward scan
    float* w = reinterpret_cast<float*>(smem + F::OFF_W) + warp * TOKENS;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t operand = tmem + lane_addr + TM_ST + part * (KEYS / 2);
    const int c16 = (v & 63) >> 3;
    uint8_t* gcol = smem + F::OFF_ST + (v >> 6) * (HD * 128) + (v & 7) * 2;            // this value's column of both tiles
    uint8_t* ncol = smem + F::OFF_OUT + (v >> 6) * (CH * 128) + (v & 7) * 2;
    float G[KEYS];
    // the state gradient as the operand of the next products, then as it stands on entry to the next chunk of the walk (that chunk's exit state's gradient), for memory
    auto deliver = [&](int n) {
      write_state_row(operand, G);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->s_ready);
      if (n < 0) return;
      if (SEND) {
#pragma unroll
        for (int d = 0; d < KEYS; d += 2) {
          const uint32_t pair = pack_bf16(G[d], G[d + 1]);
          *reinterpret_cast<uint16_t*>(gcol + swz(part * KEYS + d, c16)) = static_cast<uint16_t>(pair);
          *reinterpret_cast<uint16_t*>(gcol + swz(part * KEYS + d + 1, c16)) = static_cast<uint16_t>(pair >> 16);
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->tile_ready);
      } else {
        // [Dk, Dv] with the value index contiguous
        const long long cell = ((static_cast<long long>(x) * N + n) * HD + part * KEYS) * HD + v;
        if (dstates != nullptr) {
#pragma unroll
          for (int d = 0; d < KEYS; ++d) dstates[cell + d * HD] = G[d];
        }
        if (dstates_bf16 != nullptr) {
#pragma unroll
          for (int d = 0; d < KEYS; ++d) dstates_bf16[cell + d * HD] = __float2bfloat16(G[d]);
        }
      }
    };
    read_state(G, d_final, x, v, part);
    deliver(N - 1);
    bool ok = true;
    for (int it = 0; it < N && ok; ++it) {
      const int n = N - 1 - it;
      const int s = it & 1; const uint32_t ph = (it >> 1) & 1;
      const float* gs = sG + s * CH;
      if (!math_wait(&bars->a_full[s], ph, sc, err, ERR_WAIT_FULL)) { ok = false; break; }
      const float gl = gs[CH - 1];
      if (lane < TOKENS) w[lane] = __expf(gl - gs[j0 + lane]);
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->a_empty[s]);
      if (SEND && it > 0 && !math_wait(&bars->vn_sent, (it - 1) & 1, sc, err, ERR_WAIT_OTHER)) { ok = false; break; }
      if (!math_wait(&bars->acc_full, it & 1, sc, err, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      {
        uint32_t a[TOKENS], bb[TOKENS];
        tmem_ld_32x32b_x16(tmem + lane_addr + TM_A + s * 64 + j0, a);
        tmem_ld_32x32b_x16(tmem + lane_addr + TM_B + j0, bb);
        tmem_ld_wait();
#pragma unroll
        for (int j8 = 0; j8 < TOKENS / 8; ++j8) {
          float nv[8];
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) nv[jj] = -(__uint_as_float(a[j8 * 8 + jj]) + w[j8 * 8 + jj] * __uint_as_float(bb[j8 * 8 + jj]));
          const uint4 packed = pack8(nv);                // -dVn
          *reinterpret_cast<uint4*>(sDvn + swz(v, part * (TOKENS / 8) + j8)) = packed;
          if (SEND) {
            const uint32_t pairs[4] = {packed.x ^ 0x80008000u, packed.y ^ 0x80008000u, packed.z ^ 0x80008000u, packed.w ^ 0x80008000u};      // the sign of both
#pragma unroll
            for (int j2 = 0; j2 < 4; ++j2) {
              *reinterpret_cast<uint16_t*>(ncol + swz(j0 + j8 * 8 + 2 * j2, c16)) = static_cast<uint16_t>(pairs[j2]);
              *reinterpret_cast<uint16_t*>(ncol + swz(j0 + j8 * 8 + 2 * j2 + 1, c16)) = static_cast<uint16_t>(pairs[j2] >> 16);
            }
          } else if (dvn_out != nullptr) {
            __nv_bfloat16* dst = dvn_out + (static_cast<long long>(x) * Tp + n * CH + j0 + j8 * 8) * HD + v;
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) dst[jj * HD] = __float2bfloat16(-nv[jj]);
          }
        }
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->vn_ready);
      if (SEND && !math_wait(&bars->state_sent, it & 1, sc, err, ERR_WAIT_OTHER)) { ok = false; break; }
      if (!math_wait(&bars->ds_full, it & 1, sc, err, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const float dl = __expf(gl);
      {
        uint32_t d[KEYS];
        tmem_ld_32x32b_x32(tmem + lane_addr + TM_DD + s * 128 + part * KEYS, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < KEYS; ++i) G[i] = fmaf(G[i], dl, __uint_as_float(d[i]));
      }
      deliver(n - 1);
    }
    if (ok && d_initial != nullptr) {
      float* dst = d_initial + (static_cast<long long>(x) * HD + part * KEYS) * HD + v;
#pragma unroll
      for (int d = 0; d < KEYS; ++d) dst[d * HD] = G[d];
    }
  }
  scan_epilogue(sc, F::MMA_WARP);
}

// A [B, T, H, 128] bf16 tensor with element strides (sb, st, sh), tiled [rows x 64 columns].
static int make_bthd_map(CUtensorMap* m, const void* base, int B, int T, int H, long long sb, long long st, long long sh,
                         int box_rows) {
  const uint64_t dims[4] = {static_cast<uint64_t>(HD), static_cast<uint64_t>(H), static_cast<uint64_t>(T), static_cast<uint64_t>(B)};
  const uint64_t strides[3] = {static_cast<uint64_t>(sh) * 2, static_cast<uint64_t>(st) * 2, static_cast<uint64_t>(sb) * 2};
  const uint32_t box[4] = {64, 1, static_cast<uint32_t>(box_rows), 1};
  return make_tmap_nd(m, base, 4, dims, strides, box, 2, true);
}

static bool strides_ok(long long sb, long long st, long long sh) { return (sb % 8) == 0 && (st % 8) == 0 && (sh % 8) == 0; }

}  // namespace gdn
}  // namespace dewb

// q, k: bf16 [B, T, H / rep, 128], v: bf16 [B, T, H, 128] (`rep` consecutive value heads share one key head; unit stride along
// the head dimension; the other strides in elements: batch, token, head);
// g, beta: fp32 [B, T, H] contiguous.  With X = B * H and Tp = T rounded up to 128:
// gc fp32 [X, Tp]; W, U bf16 [X, Tp, 128]; P bf16 [X, Tp, 64]; Qg bf16 [X, Tp, 128] or null.
extern "C" int dewb_gdn_prepare(const void* q, const void* k, const void* v, const float* g, const float* beta, float* gc,
                                void* W, void* U, void* P, void* Qg, int B, int T, int H, int rep, long long q_sb, long long q_st,
                                long long q_sh, long long k_sb, long long k_st, long long k_sh, long long v_sb,
                                long long v_st, long long v_sh, float scale, int* err, void* stream_ptr) {
  using namespace dewb::gdn;
  if (B <= 0 || T <= 0 || H <= 0 || rep <= 0 || H % rep != 0) return -3;
  if (!strides_ok(q_sb, q_st, q_sh) || !strides_ok(k_sb, k_st, k_sh) || !strides_ok(v_sb, v_st, v_sh)) return -3;
  const int Tp = (T + PT - 1) / PT * PT;
  CUtensorMap tq, tk, tv;
  int r;
  if ((r = make_bthd_map(&tq, q, B, T, H / rep, q_sb, q_st, q_sh, PT))) return 1000 + r;
  if ((r = make_bthd_map(&tk, k, B, T, H / rep, k_sb, k_st, k_sh, PT))) return 2000 + r;
  if ((r = make_bthd_map(&tv, v, B, T, H, v_sb, v_st, v_sh, PT))) return 3000 + r;
  cudaError_t e = cudaFuncSetAttribute(gdn_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP_SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  dim3 grid(Tp / PT, B * H);
  gdn_prepare_kernel<<<grid, PREP_THREADS, PREP_SMEM, reinterpret_cast<cudaStream_t>(stream_ptr)>>>(
      tq, tk, tv, g, beta, gc, reinterpret_cast<__nv_bfloat16*>(W), reinterpret_cast<__nv_bfloat16*>(U),
      reinterpret_cast<__nv_bfloat16*>(P), reinterpret_cast<__nv_bfloat16*>(Qg), T, H, rep, Tp, scale, err);
  return static_cast<int>(cudaGetLastError());
}

// out bf16 [B, T, H, 128] contiguous or null; initial / final_state fp32 [X, 128 (key), 128 (value)] (initial may be null);
// states bf16 [X, N, 128 (value), 128 (key)] or null: the state on entry to each chunk, transposed;
// vn_out bf16 [X, Tp, 128] or null: the corrected values Vn = U - W S of every chunk (the backward reads them).
extern "C" int dewb_gdn_scan_fwd(const void* q, const void* k, const float* gc, const void* W, const void* U, const void* P,
                                 const float* initial, void* out, float* final_state, void* states, void* vn_out, int B,
                                 int T, int H, int rep, int Tp, long long q_sb, long long q_st, long long q_sh, long long k_sb, long long k_st,
                                 long long k_sh, float scale, int* err, void* stream_ptr) {
  using namespace dewb::gdn;
  if (B <= 0 || T <= 0 || H <= 0 || Tp % PT != 0 || Tp < T) return -3;
  if (!strides_ok(q_sb, q_st, q_sh) || !strides_ok(k_sb, k_st, k_sh)) return -3;
  const int N = (T + CH - 1) / CH;
  const uint64_t rows = static_cast<uint64_t>(B) * H * Tp;
  CUtensorMap tq, tk, tw, tu, tp;
  int r;
  if (rep <= 0 || H % rep != 0) return -3;
  if ((r = make_bthd_map(&tq, q, B, T, H / rep, q_sb, q_st, q_sh, CH))) return 1000 + r;
  if ((r = make_bthd_map(&tk, k, B, T, H / rep, k_sb, k_st, k_sh, CH))) return 2000 + r;
  if ((r = dewb::make_tmap_2d(&tw, W, rows, HD, HD, CH, 64, 2, true))) return 3000 + r;
  if ((r = dewb::make_tmap_2d(&tu, U, rows, HD, HD, CH, 64, 2, true))) return 4000 + r;
  if ((r = dewb::make_tmap_2d(&tp, P, rows, CH, CH, CH, 64, 2, true))) return 5000 + r;
  // What the backward reads and nothing else, or any other selection, by the threads that hold it.
  const bool send = out == nullptr && states != nullptr && vn_out != nullptr;
  CUtensorMap ts = tu, tv = tu;                                            // (not read where nothing is sent)
  if (send) {
    if ((r = dewb::make_tmap_2d(&ts, states, static_cast<uint64_t>(B) * H * N * HD, HD, HD, HD, 64, 2, true))) return 6000 + r;
    if ((r = dewb::make_tmap_2d(&tv, vn_out, rows, HD, HD, CH, 64, 2, true))) return 7000 + r;
  }
  auto fn = send ? gdn_scan_fwd_kernel<false> : gdn_scan_fwd_kernel<true>;
  const int smem = send ? Fwd<false>::SMEM : Fwd<true>::SMEM, threads = send ? Fwd<false>::THREADS : Fwd<true>::THREADS;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  fn<<<B * H, threads, smem, reinterpret_cast<cudaStream_t>(stream_ptr)>>>(tq, tk, tw, tu, tp, ts, tv, gc, initial, reinterpret_cast<__nv_bfloat16*>(out), final_state,
                                                                           reinterpret_cast<__nv_bfloat16*>(states), reinterpret_cast<__nv_bfloat16*>(vn_out), T, H, rep, Tp, N, scale, err);
  return static_cast<int>(cudaGetLastError());
}

// d_out bf16 [B, T, H, 128] (strides in elements); d_final fp32 [X, 128, 128] or null; dstates fp32 [X, N, 128 (key),
// 128 (value)] (or null) and dstates_bf16 (same shape, bf16, or null): the gradient of each chunk's exit state;
// dvn_out bf16 [X, Tp, 128] or null: dVn of every chunk; d_initial fp32 [X, 128, 128].
extern "C" int dewb_gdn_scan_bwd(const void* d_out, const void* k, const float* gc, const void* W, const void* P,
                                 const void* Qg, const float* d_final, float* dstates, void* dstates_bf16, void* dvn_out,
                                 float* d_initial, int B, int T, int H, int rep, int Tp, long long do_sb, long long do_st, long long do_sh, long long k_sb,
                                 long long k_st, long long k_sh, int* err, void* stream_ptr) {
  using namespace dewb::gdn;
  if (B <= 0 || T <= 0 || H <= 0 || Tp % PT != 0 || Tp < T) return -3;
  if (!strides_ok(do_sb, do_st, do_sh) || !strides_ok(k_sb, k_st, k_sh)) return -3;
  const int N = (T + CH - 1) / CH;
  const uint64_t rows = static_cast<uint64_t>(B) * H * Tp;
  CUtensorMap tdo, tk, tw, tqg, tp;
  int r;
  if ((r = make_bthd_map(&tdo, d_out, B, T, H, do_sb, do_st, do_sh, CH))) return 1000 + r;
  if (rep <= 0 || H % rep != 0) return -3;
  if ((r = make_bthd_map(&tk, k, B, T, H / rep, k_sb, k_st, k_sh, CH))) return 2000 + r;
  if ((r = dewb::make_tmap_2d(&tw, W, rows, HD, HD, CH, 64, 2, true))) return 3000 + r;
  if ((r = dewb::make_tmap_2d(&tqg, Qg, rows, HD, HD, CH, 64, 2, true))) return 4000 + r;
  if ((r = dewb::make_tmap_2d(&tp, P, rows, CH, CH, CH, 64, 2, true))) return 5000 + r;
  // What the local kernels read and nothing else, or any other selection, by the threads that hold it.
  const bool send = dstates == nullptr && dstates_bf16 != nullptr && dvn_out != nullptr;
  CUtensorMap ts = tw, tv = tw;                                            // (not read where nothing is sent)
  if (send) {
    if ((r = dewb::make_tmap_2d(&ts, dstates_bf16, static_cast<uint64_t>(B) * H * N * HD, HD, HD, HD, 64, 2, true))) return 6000 + r;
    if ((r = dewb::make_tmap_2d(&tv, dvn_out, rows, HD, HD, CH, 64, 2, true))) return 7000 + r;
  }
  auto fn = send ? gdn_scan_bwd_kernel<true> : gdn_scan_bwd_kernel<false>;
  const int smem = send ? Bwd<true>::SMEM : Bwd<false>::SMEM;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  fn<<<B * H, Bwd<true>::THREADS, smem, reinterpret_cast<cudaStream_t>(stream_ptr)>>>(tdo, tk, tw, tqg, tp, ts, tv, gc, d_final, dstates, reinterpret_cast<__nv_bfloat16*>(dstates_bf16),
                                                                                      reinterpret_cast<__nv_bfloat16*>(dvn_out), d_initial, T, H, rep, Tp, N, err);
  return static_cast<int>(cudaGetLastError());
}
