// Block-scaled fp8 GEMM for sm_100a (MXFP8: e4m3 values, one power-of-two ue8m0 scale per 32 consecutive elements of the
// reduction dimension), dense or grouped by rows (mixture-of-experts):
//
//     D[M,N] (bf16) = sum_k (A_q[m,k] * 2^(sa[m, k / 32] - 127)) * (B_q[n,k] * 2^(sb[n, k / 32] - 127))
//
// computed by tcgen05.mma kind::mxf8f6f4.block_scale: the tensor core applies both operands' scales per 32-element block
// while it accumulates in fp32, so nothing is rescaled in the epilogue and a block with small values keeps its precision.
//
// One persistent CTA per SM, 320 threads:
//   warp 0      TMA producer : A [128 x 128 B] and B [192 x 128 B] tiles into a 5-stage ring (cp.async.bulk.tensor, no multicast)
//   warp 1      MMA issuer   : four K = 32 products per stage into one of two TMEM accumulators; each product names the scale
//                              factors of its 32-element block through the descriptor's scale-factor ids
//   warps 2..5  epilogue     : tcgen05.ld the finished accumulator, store bf16; overlaps the next tile's products
//   warps 6..9  scale stagers: per stage, load the packed scales of the tile's 128 A rows and 192 B rows (one 32-bit word =
//                              the four blocks of the stage for one row) and write them to tensor memory (tcgen05.st) in the
//                              layout the tensor core reads them from: lane = row % 32, column = row / 32, byte = block,
//                              the same words in all four lane quarters
//
// Tensor memory: 2 accumulators x 192 columns, then 5 scale slots x 16 columns (4 for A, 6 for B) = 464 of 512 columns.
//
// Scale storage (what `dewb_quantize_mx` writes): sf[kb][row] is one 32-bit word holding the four ue8m0 bytes of row `row`
// for reduction blocks 4 kb .. 4 kb + 3 (byte j = block 4 kb + j), rows padded so that a tile's loads stay in range.
//
// Replaces the reference's MX grouped GEMM (src/dew/nn/kernels/grouped_matmul.py:1746 `MosaicMxGmm`; formats.py:186 `MxFp8`).
#include "../common/ptx.cuh"
#include "../common/tmap.h"
#include <cuda_fp8.h>

namespace dewb {
namespace gemm_mx {

constexpr int BM = 128;
constexpr int BN = 192;
constexpr int BK = 128;                 // fp8 elements = bytes per row of a stage: one 128-byte swizzle row, four K = 32 products
constexpr int STAGES = 5;
constexpr int A_BYTES = BM * BK;        // 16 KiB
constexpr int B_BYTES = BN * BK;        // 24 KiB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int ACC_COLS = BN;
constexpr int SF_BASE = 2 * ACC_COLS;   // 384
constexpr int SF_SLOT = 16;             // columns per stage: A at +0 (4 columns), B at +4 (6 columns)
constexpr int TMEM_COLS = 512;
constexpr int AHEAD = 4;                // stages whose scales a stager has on their way
constexpr int THREADS = 320;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;

struct Shared {
  uint64_t full[STAGES];        // TMA bytes of the stage have landed
  uint64_t sf_full[STAGES];     // the stage's scale factors are in tensor memory (4 arrivals: one per stager warp)
  uint64_t empty[STAGES];       // the products that read the stage (operands and scales) have completed
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

struct Args {
  const int* tile_group;        // grouped rows: group of each 128-row tile of A (< 0: empty), or null for a dense product
  int b_rows_per_group;         // rows of B per group (N)
  const uint32_t* sfa;          // [K / 128][sfa_rows] packed scales of A
  const uint32_t* sfb;          // [K / 128][sfb_rows] packed scales of the stacked B
  long long sfa_rows, sfb_rows;
};

__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int& m_blk, int& n_blk) {
  constexpr int GROUP_M = 8;
  const int per_group = GROUP_M * tiles_n;
  const int group = t / per_group;
  const int first_m = group * GROUP_M;
  const int gsize = min(tiles_m - first_m, GROUP_M);
  const int r = t - group * per_group;
  m_blk = first_m + r % gsize;
  n_blk = r / gsize;
}

// Instruction descriptor of kind::mxf8f6f4.block_scale: e4m3 x e4m3, both K-major, ue8m0 scales, dense, K = 32.
//   [4,6) B scale-factor id, [7,10) A format (0 = e4m3), [10,13) B format, [15] A major, [16] B major, [17,23) N >> 3,
//   [23] scale format (1 = ue8m0), [24,29) M >> 4, [29,31) A scale-factor id.  The ids pick the byte of the 32-bit scale word.
__host__ __device__ constexpr uint32_t make_idesc_mx(int M, int N, int sf_id) {
  return (static_cast<uint32_t>(sf_id) << 4) | (static_cast<uint32_t>(N >> 3) << 17) | (1u << 23) |
         (static_cast<uint32_t>(M >> 4) << 24) | (static_cast<uint32_t>(sf_id) << 29);
}

__device__ __forceinline__ void umma_mxf8_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n\t"
      "}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
      : "memory");
}

__device__ __forceinline__ void tmem_st_32x32b_x4(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x2(uint32_t taddr, uint32_t a, uint32_t b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_mx_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
               __nv_bfloat16* __restrict__ D, int M, int N, int K, long long ldd, const Args ga, int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  {
    __shared__ int poisoned;
    if (threadIdx.x == 0) poisoned = *reinterpret_cast<volatile int*>(err);
    __syncthreads();
    if (poisoned != 0) return;        // an earlier launch reported a timed-out wait
  }
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Shared* sh = reinterpret_cast<Shared*>(smem + STAGES * STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int k_iters = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->sf_full[s], 4); mbar_init(&sh->empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&sh->tmem_full[a], 1); mbar_init(&sh->tmem_empty[a], 4); }
    sh->abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) { tmem_alloc(&sh->tmem_base, TMEM_COLS); tmem_relinquish(); }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tma_a); tma_prefetch_desc(&tma_b); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  volatile int* abort_flag = &sh->abort_flag;

  auto tile_of = [&](int t, int& m0, int& n0, int& b_row0) -> bool {       // false: the tile holds no rows
    int m_blk, n_blk;
    tile_coords(t, tiles_m, tiles_n, m_blk, n_blk);
    m0 = m_blk * BM; n0 = n_blk * BN; b_row0 = 0;
    if (ga.tile_group != nullptr) {
      const int g = ga.tile_group[m_blk];
      if (g < 0) return false;
      b_row0 = g * ga.b_rows_per_group;
    }
    return true;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      long long issued = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        int m0, n0, b_row0;
        if (!tile_of(t, m0, n0, b_row0)) continue;
        for (int k = 0; k < k_iters; ++k) {
          if (!mbar_wait(&sh->empty[stage], phase ^ 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); ok = false; break; }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          mbar_expect_tx(&sh->full[stage], STAGE_BYTES);
          tma_load_2d(sa, &tma_a, &sh->full[stage], k * BK, m0);
          tma_load_2d(sa + A_BYTES, &tma_b, &sh->full[stage], k * BK, b_row0 + n0);
          ++issued;
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        const long long pending = issued < STAGES ? issued : STAGES;
        for (long long i = 0; i < pending; ++i) {
          int s = static_cast<int>((issued - 1 - i) % STAGES);
          uint32_t ph = static_cast<uint32_t>(((issued - 1 - i) / STAGES) & 1);
          mbar_wait(&sh->full[s], ph, nullptr, 20000000ull);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp runs this loop and waits together; one elected lane issues (see mbar_wait_warp).
    int stage = 0; uint32_t phase = 0;
    int acc = 0; uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      int m0, n0, b_row0;
      if (!tile_of(t, m0, n0, b_row0)) continue;
      if (!mbar_wait_warp(&sh->tmem_empty[acc], acc_phase ^ 1, abort_flag)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_TMEM_EMPTY); break; }
      const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
      for (int k = 0; k < k_iters; ++k) {
        // every lane waits for the stage's operands and for its scales: the lane that issues has to have seen both itself, since a vote orders no memory between lanes
        if (!mbar_wait_warp(&sh->full[stage], phase, abort_flag) || !mbar_wait_warp(&sh->sf_full[stage], phase, abort_flag)) {
          if (lane == 0) atomicCAS(err, 0, ERR_WAIT_FULL);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
        const uint32_t sb = sa + A_BYTES;
        const uint32_t sfa = tmem_base + SF_BASE + stage * SF_SLOT, sfb = sfa + 4;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {          // 32 fp8 elements = 32 bytes per product
            const uint64_t da = make_sdesc_sw128(sa + kk * 32, 16, 1024);
            const uint64_t db = make_sdesc_sw128(sb + kk * 32, 16, 1024);
            umma_mxf8_ss(d_tmem, da, db, make_idesc_mx(BM, BN, kk), sfa, sfb, (k > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(&sh->empty[stage]);
          if (k == k_iters - 1) umma_commit(&sh->tmem_full[acc]);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;
    int acc = 0; uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      int m0, n0, b_row0;
      if (!tile_of(t, m0, n0, b_row0)) continue;
      const int row = m0 + q * 32 + lane;
      if (!mbar_wait(&sh->tmem_full[acc], acc_phase, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_TMEM_FULL); ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * ACC_COLS + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + c * 32, r);
        tmem_ld_wait();
        const int col = n0 + c * 32;
        if (row < M && col < N) {
          __nv_bfloat16* out = D + static_cast<long long>(row) * ldd + col;
          if (col + 32 <= N && ((reinterpret_cast<uintptr_t>(out) & 15) == 0)) {
            store_row_32<false>(out, r, 1.f);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) if (col + i < N) out[i] = __float2bfloat16(__uint_as_float(r[i]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->tmem_empty[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  } else {
    // ------------------------------------------------------------------ scale stagers (warps 6..9): warp w fills lane quarter w & 3
    const int q = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    // The words of the next AHEAD stages are on their way while one is staged: a stage's products take 400 cycles, and loads that were waited for one stage after another
    // took longer than that (the four products of a 64-expert layer's step, 8192 tokens, 2048 x 1408, top 6: 1375 us, with the issue out of one lane of a divergent warp; 1000 now).
    int t = blockIdx.x, k = 0;                       // the next stage to load
    const uint32_t *pa = nullptr, *pb = nullptr;
    auto begin_tile = [&]() -> bool {
      for (; t < num_tiles; t += gridDim.x) {
        int m0, n0, b_row0;
        if (!tile_of(t, m0, n0, b_row0)) continue;
        pa = ga.sfa + m0 + lane;
        pb = ga.sfb + b_row0 + n0 + lane;
        k = 0;
        return true;
      }
      return false;
    };
    bool more = begin_tile() && k_iters > 0;
    uint32_t words[AHEAD][10];
    bool loaded[AHEAD];
    auto load = [&](uint32_t (&w)[10]) -> bool {
      if (!more) return false;
      const uint32_t *a = pa + static_cast<long long>(k) * ga.sfa_rows, *b = pb + static_cast<long long>(k) * ga.sfb_rows;
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = __ldg(a + i * 32);
#pragma unroll
      for (int i = 0; i < 6; ++i) w[4 + i] = __ldg(b + i * 32);
      if (++k == k_iters) { t += gridDim.x; more = begin_tile(); }
      return true;
    };
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) loaded[u] = load(words[u]);
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    while (ok && loaded[0]) {
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        if (!ok || !loaded[u]) { ok = false; continue; }
        // the slot is free once the products of its previous use have completed (the same event that frees the operands)
        const bool got = mbar_wait(&sh->empty[stage], phase ^ 1, abort_flag);
        if (!__all_sync(0xffffffffu, got)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); ok = false; continue; }
        tc_fence_after();
        const uint32_t base = tmem_base + lane_addr + SF_BASE + stage * SF_SLOT;
        tmem_st_32x32b_x4(base, words[u][0], words[u][1], words[u][2], words[u][3]);
        tmem_st_32x32b_x4(base + 4, words[u][4], words[u][5], words[u][6], words[u][7]);
        tmem_st_32x32b_x2(base + 8, words[u][8], words[u][9]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->sf_full[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
        loaded[u] = load(words[u]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Quantiser: x [rows, K] bf16 -> q [rows, K] e4m3 and packed scales sf[K / 128][sf_rows] (one word per row per 128
// elements, byte j = block 4 kb + j).  The scale of a block is the smallest power of two that brings its largest magnitude
// within e4m3's range (448): e = ceil(log2(amax / 448)), stored as e + 127 (ue8m0); an all-zero block stores 2^-127.
// A warp takes whole rows, QU pieces of 8 elements a lane in flight; the four lanes of a 32-element block share the maximum through shuffles.  Bound by memory
// (two bytes read, one written per element); one thread per 8 elements of the whole array, found by a 64-bit division, took 126 us a call on average over the six
// arrays of a 64-expert layer's step (8192 tokens, 2048 x 1408); this form takes 78.
constexpr int QU = 4;
// smallest integer e with amax <= 448 * 2^e, from the bits (exact): amax = f * 2^k with f in [1, 2) and 448 = 1.75 * 2^8
__device__ __forceinline__ int block_exponent(float amax) {
  if (!(amax > 0.f)) return -127;
  const uint32_t bits = __float_as_uint(amax);
  const int k = static_cast<int>((bits >> 23) & 0xff) - 127;
  return max(-127, min(127, k - 8 + ((bits & 0x7fffffu) > 0x600000u ? 1 : 0)));
}

__global__ void __launch_bounds__(256)
quantize_mx_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, uint8_t* __restrict__ sf, long long rows, int K, long long ldx, long long sf_rows) {
  const int lane = threadIdx.x & 31, pieces = K >> 3;
  for (long long row = blockIdx.x * 8ll + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8ll) {
    const uint4* src = reinterpret_cast<const uint4*>(x + row * ldx);
    for (int first = 0; first < pieces; first += 32 * QU) {
      uint4 raw[QU];
#pragma unroll
      for (int u = 0; u < QU; ++u) {
        const int at = first + u * 32 + lane;
        raw[u] = at < pieces ? src[at] : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < QU; ++u) {
        const int at = first + u * 32 + lane;
        const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
        float v[8], amax = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[2 * i] = bf16_lo(w[i]); v[2 * i + 1] = bf16_hi(w[i]); }
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
        // K is a multiple of 32, so the four lanes of a block are all inside the row or all behind it
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const int e = block_exponent(amax);
        const float inv = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);      // 2^-e, exact (e in [-127, 127] -> exponent field 0..254)
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          lo |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(v[i] * inv, __NV_SATFINITE, __NV_E4M3)) << (8 * i);
          hi |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(v[4 + i] * inv, __NV_SATFINITE, __NV_E4M3)) << (8 * i);
        }
        if (at < pieces) {
          *reinterpret_cast<uint2*>(q + row * K + at * 8) = make_uint2(lo, hi);
          if ((lane & 3) == 0) {
            const int block = at >> 2;                    // 32-element block index along K
            sf[(static_cast<long long>(block >> 2) * sf_rows + row) * 4 + (block & 3)] = static_cast<uint8_t>(e + 127);
          }
        }
      }
    }
  }
}

// The same values for the transpose: x [groups, rows, cols] bf16 (contiguous) -> q [groups * cols, rows] with blocks of 32 along the rows.  Bound by memory: two
// bytes read and one written per value.  A CTA takes 128 rows (one scale word) by 64 columns through shared memory; a thread then holds one column's 32 rows and
// writes them as one 32-byte sector.  Copying the transpose first and quantising the copy
// took 2.2 + 0.4 ms for the two weights of 64 experts of 2048 x 1408; this takes 0.37 (4.4 TB/s).
constexpr int QT_ROWS = 128, QT_COLS = 64;
__global__ void __launch_bounds__(256)
quantize_mx_t_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, uint32_t* __restrict__ sf, int rows, int cols, long long sf_rows) {
  __shared__ __align__(16) __nv_bfloat16 tile[QT_ROWS][QT_COLS];
  __shared__ __align__(4) uint8_t exps[QT_COLS][4];
  const int col0 = blockIdx.x * QT_COLS, row0 = blockIdx.y * QT_ROWS;
  const __nv_bfloat16* src = x + (static_cast<long long>(blockIdx.z) * rows + row0) * cols + col0;
#pragma unroll
  for (int i = 0; i < QT_ROWS * QT_COLS / 8 / 256; ++i) {
    const int at = i * 256 + threadIdx.x, r = at >> 3, c = at & 7;
    *reinterpret_cast<uint4*>(&tile[r][c * 8]) = *reinterpret_cast<const uint4*>(src + static_cast<long long>(r) * cols + c * 8);
  }
  __syncthreads();
  const int c = threadIdx.x & 63, block = threadIdx.x >> 6;
  float v[32], amax = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) { v[i] = __bfloat162float(tile[block * 32 + i][c]); amax = fmaxf(amax, fabsf(v[i])); }
  const int e = block_exponent(amax);
  const float inv = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    w[i] = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) w[i] |= static_cast<uint32_t>(__nv_cvt_float_to_fp8(v[i * 4 + j] * inv, __NV_SATFINITE, __NV_E4M3)) << (8 * j);
  }
  const long long out = static_cast<long long>(blockIdx.z) * cols + col0 + c;
  uint4* to = reinterpret_cast<uint4*>(q + out * rows + row0 + block * 32);
  to[0] = make_uint4(w[0], w[1], w[2], w[3]);
  to[1] = make_uint4(w[4], w[5], w[6], w[7]);
  exps[c][block] = static_cast<uint8_t>(e + 127);
  __syncthreads();
  if (threadIdx.x < QT_COLS) sf[static_cast<long long>(blockIdx.y) * sf_rows + out] = *reinterpret_cast<const uint32_t*>(exps[c]);
}

static int sm_count_mx() {
  static int n[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  if (n[dev] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    n[dev] = v;
  }
  return n[dev];
}

}  // namespace gemm_mx
}  // namespace dewb

// x [rows, K] bf16 (row stride ldx, K a multiple of 32, rows 16-byte aligned) -> q [rows, K] e4m3 bytes (contiguous) and packed
// ue8m0 scales sf [ceil(K / 128)][sf_rows] words (sf_rows >= rows; bytes of blocks past K and rows past `rows` are left as they are:
// allocate the array zeroed).
extern "C" int dewb_quantize_mx(const void* x, void* q, void* sf, long long rows, int K, long long ldx, long long sf_rows,
                                void* stream) {
  using namespace dewb::gemm_mx;
  if (K % 32 != 0 || (ldx % 8) != 0 || sf_rows < rows) return -3;
  if (rows <= 0) return 0;
  const long long blocks = (rows + 7) / 8;
  quantize_mx_kernel<<<static_cast<unsigned>(blocks < 148 * 64 ? blocks : 148 * 64), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<uint8_t*>(q), reinterpret_cast<uint8_t*>(sf), rows, K, ldx, sf_rows);
  return static_cast<int>(cudaGetLastError());
}

// x [groups, rows, cols] bf16 (contiguous, 16-byte aligned; rows a multiple of 128, cols of 64) -> its transpose quantised as above: q [groups * cols, rows] e4m3
// bytes, sf [rows / 128][sf_rows] words.
extern "C" int dewb_quantize_mx_t(const void* x, void* q, void* sf, int groups, int rows, int cols, long long sf_rows, void* stream) {
  using namespace dewb::gemm_mx;
  if (groups <= 0 || rows <= 0 || cols <= 0) return 0;
  if (rows % QT_ROWS || cols % QT_COLS || groups > 65535 || rows / QT_ROWS > 65535 || sf_rows < static_cast<long long>(groups) * cols ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(q)) & 15))
    return -3;
  quantize_mx_t_kernel<<<dim3(cols / QT_COLS, rows / QT_ROWS, groups), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<uint8_t*>(q), reinterpret_cast<uint32_t*>(sf), rows, cols, sf_rows);
  return static_cast<int>(cudaGetLastError());
}

// D[M,N] (bf16, row stride ldd) = block-scaled A_q [M,K] x B_q [groups * N, K]^T (e4m3 bytes, K contiguous, row strides lda / ldb
// multiples of 16 bytes, K a multiple of 128).  sfa [K / 128][sfa_rows], sfb [K / 128][sfb_rows]: packed scales as written by
// dewb_quantize_mx, with sfa_rows >= M rounded up to 128 and sfb_rows >= groups * N + 192 (a tile's loads stay in range).
// tile_group: null for a dense product (groups = 1), else the group of each 128-row tile of A (< 0: no rows).
extern "C" int dewb_gemm_mxfp8(const void* A, const void* B, void* D, const void* sfa, const void* sfb, const int* tile_group,
                               int M, int N, int K, int groups, long long lda, long long ldb, long long ldd, long long sfa_rows,
                               long long sfb_rows, int* err, void* stream_ptr) {
  using namespace dewb;
  using namespace dewb::gemm_mx;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((K % BK) || (lda % 16) || (ldb % 16) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -3;
  if (sfa_rows < (M + BM - 1) / BM * BM || sfb_rows < static_cast<long long>(groups) * N + BN) return -3;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  CUtensorMap ta, tb;
  int r = make_tmap_2d(&ta, A, M, K, lda, BM, BK, 1, true);
  if (r) return 1000 + r;
  r = make_tmap_2d(&tb, B, static_cast<uint64_t>(groups) * N, K, ldb, BN, BK, 1, true);
  if (r) return 2000 + r;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_mx_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  int ctas = sm_count_mx();
  if (tiles < ctas) ctas = tiles;
  Args ga{tile_group, N, reinterpret_cast<const uint32_t*>(sfa), reinterpret_cast<const uint32_t*>(sfb), sfa_rows, sfb_rows};
  gemm_mx_kernel<<<ctas, THREADS, SMEM_BYTES, stream>>>(ta, tb, reinterpret_cast<__nv_bfloat16*>(D), M, N, K, ldd, ga, err);
  return static_cast<int>(cudaGetLastError());
}
