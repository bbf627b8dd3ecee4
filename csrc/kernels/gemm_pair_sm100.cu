// Dense bf16 GEMM for sm_100a on CTA pairs: D[M,N] = A[M,K] * B[N,K]^T, fp32 accumulation in tensor memory.
//
// Two CTAs on neighbouring SMs (a thread-block cluster of 2) compute one 256 x 256 output tile with tcgen05.mma
// cta_group::2. Each CTA stages 128 rows of A and 128 rows of B per reduction step (32 KiB instead of the 48 KiB a
// lone CTA needs for a 128 x 256 tile), so the shared-memory fill rate per FLOP drops by a third - the limiter the
// single-CTA kernel's counters showed (L2 -> SM operand delivery). Each CTA keeps its 128 x 256 half of the
// accumulator in its own tensor memory and runs its own epilogue.
//
//   warp 0      TMA producer (both CTAs): own halves of A and B into a 6-stage ring; the byte counts of both CTAs are
//               credited to the leader CTA's "full" barrier (no multicast: every load lands in the issuing CTA only)
//   warp 1      MMA issuer (leader CTA only): tcgen05.mma.cta_group::2 256x256x16; tcgen05.commit to the "empty"
//               barrier of BOTH CTAs frees a stage; commit to both CTAs' "accumulator full" barriers ends a tile
//   warps 2..9  epilogue (both CTAs): tcgen05.ld the CTA's own accumulator half, convert, store; the leader's MMA
//               warp learns from both CTAs' epilogues (remote mbarrier arrive) that an accumulator is free again.  Two warps share a quarter of the rows and
//               take half of the columns each: at short reductions a tile's products take less than one warp's way through 256 columns (K = 768: 6100 cycles)
//
// Operand layouts as in the single-CTA kernel (K-major or MN-major per operand), so forward, input gradient and weight
// gradient of a linear layer read their operands in place.
//
// Replaces the reference's paired ("PAIRED" topology, 2-CTA UMMA 256x256) GEMM bundle
// (src/dew/nn/kernels/templates/mosaic_sm100.py:1-220).
#include "../common/ptx.cuh"
#include "../common/tmap.h"
#include "../common/reduction_ranges.cuh"
#include <cstdlib>

namespace dewb {
namespace gemm_pair {

constexpr int BM = 128;          // accumulator rows per CTA (pair tile: 256)
constexpr int PAIR_M = 256;
constexpr int BN = 256;          // pair tile columns
constexpr int HALF_N = BN / 2;   // rows of B staged by each CTA
constexpr int BK = 64;           // 64 bf16 = 128 bytes = one swizzle row
constexpr int STAGES = 6;
constexpr int A_BYTES = BM * BK * 2;        // 16 KiB
constexpr int B_BYTES = HALF_N * BK * 2;    // 16 KiB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int ACC_COLS = BN;
constexpr int TMEM_COLS = 2 * ACC_COLS;     // both accumulators
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;

enum Epilogue : int { EPI_BF16 = 0, EPI_F32 = 1, EPI_F32_ACC = 2, EPI_BF16_ACC = 3 };

struct Shared {
  uint64_t full[STAGES];       // used in the leader: both CTAs' loads of a stage have landed
  uint64_t empty[STAGES];      // in each CTA: the pair MMAs that read the stage have completed
  uint64_t tmem_full[2];       // in each CTA: the accumulator is complete
  uint64_t tmem_empty[2];      // used in the leader: both CTAs' epilogues have drained the accumulator (EPI_WARPS warps each)
  uint32_t tmem_base;
  int abort_flag;
  int poisoned;
};

// `group_m` row blocks (of 256 rows) share their B tiles in L2 before the walk moves along N: the A rows of a group stay
// resident while B streams past once per group.
__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int group_m, int& m_blk, int& n_blk) {
  const int per_group = group_m * tiles_n;
  const int group = t / per_group;
  const int first_m = group * group_m;
  const int gsize = min(tiles_m - first_m, group_m);
  const int r = t - group * per_group;
  m_blk = first_m + r % gsize;
  n_blk = r / gsize;
}

// Several products side by side (GROUPED: Ranges).  A pair fetches two thirds of the operand bytes that two lone CTAs do, which shows where reductions are long (64 groups of
// 768 rows into 2816 x 2048: lone CTAs 498 us, pairs 430; 8 of 4096 into 512 x 1024 33.8 and 30.3; the twelve split weight gradients of a diffusion transformer's step,
// 768 x 768 to 3072 over 16384, 684 and 600).  Short ones over few tiles, and outputs of up to 128 rows, are left to lone CTAs (gemm_sm100.cu): 16 of 128 into 512 x 256 10.0
// and 10.9.  A group without rows is cleared in wide stores (one among 16 of 640 x 1408: 77 us in single values, some 30 now).
struct Tile {
  int m_blk, n_blk, k0, k_iters;
  long long d_off;
};

template <bool GROUPED>
__device__ __forceinline__ Tile tile_of(int t, int tiles_m, int tiles_n, int group_m, int K, const Ranges& gr) {
  Tile ti;
  ti.k0 = 0; ti.k_iters = (K + BK - 1) / BK; ti.d_off = 0;
  if constexpr (GROUPED) {
    const int per = tiles_m * tiles_n, g = t / per;
    t -= g * per;
    const Range of = range_of(gr, g, K, BK);
    ti.k0 = of.k0;
    ti.k_iters = of.k_iters;
    ti.d_off = of.d_off;
  }
  tile_coords(t, tiles_m, tiles_n, group_m, ti.m_blk, ti.n_blk);
  return ti;
}

template <int EPI>
__device__ __forceinline__ void store_chunk(const uint32_t (&r_in)[32], void* Dptr, int row, int col, int N, long long ldd,
                                            float alpha_in, const __nv_bfloat16* __restrict__ bias) {
  const bool full = (col + 32 <= N);
  // scale, then the bias (one bf16 value per output column); the stores below see the finished values
  uint32_t r[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) r[i] = bias != nullptr ? r_in[i] : __float_as_uint(alpha_in * __uint_as_float(r_in[i]));
  if (bias != nullptr) scale_and_bias(r, alpha_in, bias + col, N - col);
  constexpr float alpha = 1.f;
  if (EPI == EPI_BF16 || EPI == EPI_BF16_ACC) {
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(Dptr) + static_cast<long long>(row) * ldd + col;
    if (full && ((reinterpret_cast<uintptr_t>(out) & 15) == 0)) {
      store_row_32<EPI == EPI_BF16_ACC>(out, r, alpha);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (col + i < N) {
          float v = alpha * __uint_as_float(r[i]);
          if (EPI == EPI_BF16_ACC) v += __bfloat162float(out[i]);
          out[i] = __float2bfloat16(v);
        }
      }
    }
  } else {
    float* out = reinterpret_cast<float*>(Dptr) + static_cast<long long>(row) * ldd + col;
    if (full && ((reinterpret_cast<uintptr_t>(out) & 15) == 0)) {
      store_row_32<EPI == EPI_F32_ACC>(out, r, alpha);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (col + i < N) {
          float v = alpha * __uint_as_float(r[i]);
          if (EPI == EPI_F32_ACC) v += out[i];
          out[i] = v;
        }
      }
    }
  }
}

template <bool A_MN, bool B_MN, int EPI, bool GROUPED>
__global__ void __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 void* __restrict__ Dptr, int M, int N, int K, long long ldd, float alpha, int group_m,
                 const __nv_bfloat16* __restrict__ bias, const Ranges groups,
                 int* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment: required by the 128-byte swizzle atoms the descriptors assume. The dynamic shared memory
  // starts at the same offset in both CTAs, so the aligned layout is identical in both (the pair MMA addresses the
  // two CTAs' operands by one shared-memory offset).
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Shared* sh = reinterpret_cast<Shared*>(smem + STAGES * STAGE_BYTES);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();          // 0 = leader
  const uint32_t leader = 0;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int tiles_m = (M + PAIR_M - 1) / PAIR_M;
  const int tiles_n = (N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n * (GROUPED ? groups.count : 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&sh->tmem_full[a], 1); mbar_init(&sh->tmem_empty[a], 2 * EPI_WARPS); }
    sh->abort_flag = 0;
    // an earlier launch reported a timed-out wait: do no work (decided for the pair as a whole, below)
    sh->poisoned = *reinterpret_cast<volatile int*>(err);
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp == 1) {
    tmem_alloc_pair(&sh->tmem_base, TMEM_COLS);
    tmem_relinquish_pair();
  }
  if (warp == 0 && lane == 0) { tma_prefetch_desc(&tma_a); tma_prefetch_desc(&tma_b); }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();            // both CTAs' barriers exist before either CTA's copies or commits can reach them
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  volatile int* abort_flag = &sh->abort_flag;
  const bool poisoned = (sh->poisoned | ld_remote_s32(map_to_cta(smem_u32(&sh->poisoned), rank ^ 1))) != 0;

  if (poisoned) {
    // fall through to the teardown: the pair leaves together
  } else if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      long long issued = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        const Tile ti = tile_of<GROUPED>(t, tiles_m, tiles_n, group_m, K, groups);
        const int m0 = ti.m_blk * PAIR_M + static_cast<int>(rank) * BM;
        const int n0 = ti.n_blk * BN + static_cast<int>(rank) * HALF_N;
        for (int k = 0; k < ti.k_iters; ++k) {
          if (!mbar_wait(&sh->empty[stage], phase ^ 1, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_EMPTY); ok = false; break; }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          if (rank == leader) mbar_expect_tx(&sh->full[stage], 2 * STAGE_BYTES);     // both CTAs' bytes
          const uint32_t full_bar = map_to_cta(smem_u32(&sh->full[stage]), leader);
          const int k0 = ti.k0 + k * BK;
          if (!A_MN) {
            tma_load_2d_pair(sa, &tma_a, full_bar, k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * 8192, &tma_a, full_bar, m0 + j * 64, k0);
          }
          if (!B_MN) {
            tma_load_2d_pair(sb, &tma_b, full_bar, k0, n0);
          } else {
#pragma unroll
            for (int j = 0; j < HALF_N / 64; ++j) tma_load_2d_pair(sb + j * 8192, &tma_b, full_bar, n0 + j * 64, k0);
          }
          ++issued;
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // Give the stages still in use a bounded chance to drain before shared memory is released: a stage is
        // drained when its "empty" barrier completes (the MMAs that read it are done), which implies its copies landed.
        const long long pending = issued < STAGES ? issued : STAGES;
        for (long long i = 0; i < pending; ++i) {
          int s = static_cast<int>((issued - 1 - i) % STAGES);
          uint32_t ph = static_cast<uint32_t>(((issued - 1 - i) / STAGES) & 1);
          mbar_wait(&sh->empty[s], ph, nullptr, 20000000ull);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    // The whole warp runs this loop and waits together; one elected lane issues (see mbar_wait_warp).  8192 x 5632 x 2048 and 8192 x 2048 x 2816 took
    // 199 us together from a single lane's loop and take 185.
    if (rank == leader) {
      constexpr uint32_t idesc = make_idesc(PAIR_M, BN, 1, 1, A_MN ? 1 : 0, B_MN ? 1 : 0);
      const uint32_t peer = rank ^ 1;
      int stage = 0; uint32_t phase = 0;
      int acc = 0; uint32_t acc_phase = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        const int k_iters = tile_of<GROUPED>(t, tiles_m, tiles_n, group_m, K, groups).k_iters;
        if (k_iters <= 0) continue;
        if (!mbar_wait_warp(&sh->tmem_empty[acc], acc_phase ^ 1, abort_flag)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_TMEM_EMPTY); break; }
        const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
        for (int k = 0; k < k_iters; ++k) {
          if (!mbar_wait_warp(&sh->full[stage], phase, abort_flag)) { if (lane == 0) atomicCAS(err, 0, ERR_WAIT_FULL); ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) {
              const uint64_t da = A_MN ? make_sdesc_sw128(sa + kk * 2048, 8192, 1024) : make_sdesc_sw128(sa + kk * 32, 16, 1024);
              const uint64_t db = B_MN ? make_sdesc_sw128(sb + kk * 2048, 8192, 1024) : make_sdesc_sw128(sb + kk * 32, 16, 1024);
              umma_bf16_ss_pair(d_tmem, da, db, idesc, (k > 0 || kk > 0) ? 1u : 0u);
            }
            // frees the stage in both CTAs once these MMAs have read it
            umma_commit_pair(smem_u32(&sh->empty[stage]));
            umma_commit_pair(map_to_cta(smem_u32(&sh->empty[stage]), peer));
            if (k == k_iters - 1) {
              umma_commit_pair(smem_u32(&sh->tmem_full[acc]));                         // accumulator complete, both halves
              umma_commit_pair(map_to_cta(smem_u32(&sh->tmem_full[acc]), peer));
            }
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9, both CTAs)
    const int q = warp & 3;                 // TMEM lane quarter this warp may read
    const int first = (warp - 2) / 4 * (BN / 64);      // its first chunk of 32 columns
    int acc = 0; uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = pair; t < num_tiles && ok; t += num_pairs) {
      const Tile ti = tile_of<GROUPED>(t, tiles_m, tiles_n, group_m, K, groups);
      const int row = ti.m_blk * PAIR_M + static_cast<int>(rank) * BM + q * 32 + lane;
      const int n0 = ti.n_blk * BN;
      constexpr bool F32 = EPI == EPI_F32 || EPI == EPI_F32_ACC;
      void* D = F32 ? static_cast<void*>(static_cast<float*>(Dptr) + ti.d_off) : static_cast<void*>(static_cast<__nv_bfloat16*>(Dptr) + ti.d_off);
      if (GROUPED && ti.k_iters <= 0) {
        // nothing to reduce over: the product is zero (nothing to add when accumulating)
        if ((EPI == EPI_BF16 || EPI == EPI_F32) && row < M) {
          const uint32_t zero[32] = {};
          for (int c = n0 + first * 32; c < min(N, n0 + first * 32 + BN / 2); c += 32) store_chunk<EPI>(zero, D, row, c, N, ldd, 1.f, nullptr);
        }
        continue;
      }
      if (!mbar_wait(&sh->tmem_full[acc], acc_phase, abort_flag)) { atomicCAS(err, 0, ERR_WAIT_TMEM_FULL); ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * ACC_COLS + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int c = first; c < first + BN / 64; c += 2) {
        uint32_t r0[32], r1[32];
        tmem_ld_32x32b_x32(taddr + c * 32, r0);
        tmem_ld_32x32b_x32(taddr + c * 32 + 32, r1);
        tmem_ld_wait();
        const int col = n0 + c * 32;
        if (row < M && col < N) store_chunk<EPI>(r0, D, row, col, N, ldd, alpha, bias);
        if (row < M && col + 32 < N) store_chunk<EPI>(r1, D, row, col + 32, N, ldd, alpha, bias);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(&sh->tmem_empty[acc]), leader));
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  // ------------------------------------------------------------------ teardown
  // Neither CTA may exit, nor tensor memory be freed, while the other's MMAs, commits or remote arrives can still
  // reach it: the pair meets at a cluster barrier first.
  tc_fence_before();
  __syncthreads();
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

template <bool A_MN, bool B_MN, int EPI, bool GROUPED = false>
static int launch_one(const CUtensorMap& ta, const CUtensorMap& tb, void* D, int M, int N, int K, long long ldd,
                      float alpha, int* err, int max_pairs, cudaStream_t stream, const __nv_bfloat16* bias = nullptr, const Ranges& groups = {nullptr, 0, 1, 0}) {
  auto kern = gemm_pair_kernel<A_MN, B_MN, EPI, GROUPED>;
  static int resident[64] = {};          // co-resident clusters of this instantiation per device (0 = not asked yet)
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return -5;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (resident[dev] == 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    cfg.gridDim = dim3(static_cast<unsigned>(sms), 1, 1);
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
    if (e != cudaSuccess || clusters <= 0) { cudaGetLastError(); return -6; }   // pairs cannot be placed: the caller takes lone CTAs
    resident[dev] = clusters;
  }
  int pairs = resident[dev];
  if (max_pairs > 0 && max_pairs < pairs) pairs = max_pairs;
  const int tiles = ((M + PAIR_M - 1) / PAIR_M) * ((N + BN - 1) / BN) * groups.count;
  if (tiles < pairs) pairs = tiles;
  cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs), 1, 1);
  // Measured on the layer shapes (gate|up forward, 8192 / 16384 x 28672 x 4096): 16 row blocks per group are 5 % faster than 4
  // (B streams from DRAM once per group); with a deep reduction (K >= 14336) 8 is as good and keeps the A rows of a group in L2.
  static int forced_group_m = -1;
  if (forced_group_m < 0) {
    const char* env = getenv("DEWB_PAIR_GROUP_M");
    forced_group_m = env != nullptr ? atoi(env) : 0;
  }
  int group_m = forced_group_m;
  if (group_m <= 0) {
    group_m = K <= 8192 ? 16 : 8;
  }
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ta, tb, D, M, N, K, ldd, alpha, group_m, bias, groups, err);
  return static_cast<int>(e);
}

static int operand_maps(CUtensorMap* ta, CUtensorMap* tb, const void* A, const void* B, int M, int N, int K, long long lda, long long ldb, int a_mn, int b_mn) {
  int r;
  if (!a_mn) r = make_tmap_2d(ta, A, M, K, lda, BM, BK, 2, true);
  else       r = make_tmap_2d(ta, A, K, M, lda, BK, 64, 2, true);
  if (r) return 1000 + r;
  if (!b_mn) r = make_tmap_2d(tb, B, N, K, ldb, HALF_N, BK, 2, true);
  else       r = make_tmap_2d(tb, B, K, N, ldb, BK, 64, 2, true);
  return r ? 2000 + r : 0;
}

template <bool A_MN, bool B_MN>
static int launch_epi(int epi, const CUtensorMap& ta, const CUtensorMap& tb, void* D, int M, int N, int K,
                      long long ldd, float alpha, int* err, int max_pairs, cudaStream_t stream, const __nv_bfloat16* bias = nullptr) {
  switch (epi) {
    case EPI_BF16: return launch_one<A_MN, B_MN, EPI_BF16>(ta, tb, D, M, N, K, ldd, alpha, err, max_pairs, stream, bias);
    case EPI_F32: return launch_one<A_MN, B_MN, EPI_F32>(ta, tb, D, M, N, K, ldd, alpha, err, max_pairs, stream, bias);
    case EPI_F32_ACC: return launch_one<A_MN, B_MN, EPI_F32_ACC>(ta, tb, D, M, N, K, ldd, alpha, err, max_pairs, stream, bias);
    case EPI_BF16_ACC: return launch_one<A_MN, B_MN, EPI_BF16_ACC>(ta, tb, D, M, N, K, ldd, alpha, err, max_pairs, stream, bias);
  }
  return -2;
}

// part [splits, M, N] fp32 -> D [M, N] (row stride ldd): the sum over the splits as bf16 (epi 0) or fp32 (1), or added to what is there in fp32 (2) or bf16 (3)
__global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ part, void* __restrict__ D, int M, int N, long long ldd, int splits, float alpha, int epi, const int* __restrict__ err) {
  if (*reinterpret_cast<const volatile int*>(err) != 0) return;
  const long long total = static_cast<long long>(M) * N, at = (blockIdx.x * 256ll + threadIdx.x) * 4;
  if (at >= total) return;
  float4 s = *reinterpret_cast<const float4*>(part + at);
  for (int k = 1; k < splits; ++k) {
    const float4 v = *reinterpret_cast<const float4*>(part + k * total + at);
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  s.x *= alpha; s.y *= alpha; s.z *= alpha; s.w *= alpha;
  const long long to = at / N * ldd + at % N;
  if (epi == EPI_F32 || epi == EPI_F32_ACC) {
    float4* d = reinterpret_cast<float4*>(reinterpret_cast<float*>(D) + to);
    if (epi == EPI_F32_ACC) { const float4 o = *d; s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w; }
    *d = s;
  } else {
    uint2* d = reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(D) + to);
    if (epi == EPI_BF16_ACC) { const uint2 o = *d; s.x += bf16_lo(o.x); s.y += bf16_hi(o.x); s.z += bf16_lo(o.y); s.w += bf16_hi(o.y); }
    *d = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
  }
}

int split_sum(const float* part, void* D, int M, int N, long long ldd, int splits, float alpha, int epi, const int* err, cudaStream_t stream) {
  const long long total = static_cast<long long>(M) * N;
  split_sum_kernel<<<static_cast<unsigned>((total / 4 + 255) / 256), 256, 0, stream>>>(part, D, M, N, ldd, splits, alpha, epi, err);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace gemm_pair
}  // namespace dewb

// host-side: the bias row of the call in flight on this thread (set by the `_bias` entry point around the common launcher)
static thread_local const __nv_bfloat16* g_pair_bias = nullptr;

// Same contract as dewb_gemm_bf16 (D[M,N] = alpha * op(A) * op(B)^T, operand layouts a_mn / b_mn, epilogues 0..3),
// computed by CTA pairs. `max_ctas` > 0 caps the grid (pairs = max_ctas / 2). Returns -6 if the device cannot place
// clusters of two CTAs of this kernel.
extern "C" int dewb_gemm_pair_bf16(const void* A, const void* B, void* D, int M, int N, int K, long long lda,
                                   long long ldb, long long ldd, int a_mn, int b_mn, int epi, float alpha, int* err,
                                   int max_ctas, void* stream_ptr) {
  using namespace dewb;
  using namespace dewb::gemm_pair;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -3;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  CUtensorMap ta, tb;
  const int r = operand_maps(&ta, &tb, A, B, M, N, K, lda, ldb, a_mn, b_mn);
  if (r) return r;
  const int max_pairs = max_ctas > 0 ? (max_ctas / 2 > 0 ? max_ctas / 2 : 1) : 0;
  const __nv_bfloat16* bias = g_pair_bias;
  if (!a_mn && !b_mn) return launch_epi<false, false>(epi, ta, tb, D, M, N, K, ldd, alpha, err, max_pairs, stream, bias);
  if (!a_mn && b_mn) return launch_epi<false, true>(epi, ta, tb, D, M, N, K, ldd, alpha, err, max_pairs, stream, bias);
  if (a_mn && !b_mn) return launch_epi<true, false>(epi, ta, tb, D, M, N, K, ldd, alpha, err, max_pairs, stream, bias);
  return launch_epi<true, true>(epi, ta, tb, D, M, N, K, ldd, alpha, err, max_pairs, stream, bias);
}

// The same product with a bias row (bf16 [N]) added in the epilogue: D = alpha * op(A) op(B)^T + bias.
extern "C" int dewb_gemm_pair_bf16_bias(const void* A, const void* B, void* D, const void* bias, int M, int N, int K, long long lda,
                                        long long ldb, long long ldd, int a_mn, int b_mn, int epi, float alpha, int* err,
                                        int max_ctas, void* stream_ptr) {
  g_pair_bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  const int rc = dewb_gemm_pair_bf16(A, B, D, M, N, K, lda, ldb, ldd, a_mn, b_mn, epi, alpha, err, max_ctas, stream_ptr);
  g_pair_bias = nullptr;
  return rc;
}

// The same product with its reduction in `splits` parts of `per` (a multiple of 64; splits * per >= K, every part with something in it): scratch holds
// splits * M * N floats.  N and ldd multiples of 4, D and scratch 16-byte aligned.
extern "C" int dewb_gemm_bf16_split(const void* A, const void* B, void* D, float* scratch, int M, int N, int K, int splits, int per, long long lda, long long ldb,
                                    long long ldd, int a_mn, int b_mn, int epi, float alpha, int* err, void* stream_ptr) {
  using namespace dewb;
  using namespace dewb::gemm_pair;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (N % 4) || (ldd % 4) ||
      (reinterpret_cast<uintptr_t>(D) & 15) || (reinterpret_cast<uintptr_t>(scratch) & 15) || splits < 1 || per % BK || per <= 0 ||
      static_cast<long long>(splits) * per < K || static_cast<long long>(splits - 1) * per >= K || epi < 0 || epi > 3)
    return -3;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  CUtensorMap ta, tb;
  int r = operand_maps(&ta, &tb, A, B, M, N, K, lda, ldb, a_mn, b_mn);
  if (r) return r;
  const Ranges gr{nullptr, per, splits, static_cast<long long>(M) * N};
  if (!a_mn && !b_mn) r = launch_one<false, false, EPI_F32, true>(ta, tb, scratch, M, N, K, N, 1.f, err, 0, stream, nullptr, gr);
  else if (!a_mn) r = launch_one<false, true, EPI_F32, true>(ta, tb, scratch, M, N, K, N, 1.f, err, 0, stream, nullptr, gr);
  else if (!b_mn) r = launch_one<true, false, EPI_F32, true>(ta, tb, scratch, M, N, K, N, 1.f, err, 0, stream, nullptr, gr);
  else r = launch_one<true, true, EPI_F32, true>(ta, tb, scratch, M, N, K, N, 1.f, err, 0, stream, nullptr, gr);
  return r ? r : split_sum(scratch, D, M, N, ldd, splits, alpha, epi, err, stream);
}

// Grouped reduction (mixture-of-experts weight gradient): for every group g,
//   D_g[M, N] (+)= A[rows of g, M]^T * B[rows of g, N]   with A stored [R, M] and B stored [R, N] (R = all rows),
//   rows of g = [group_offsets[g], group_offsets[g + 1]) (multiples of 64; padding rows are zero)
//   D stacks the groups: D_g = D + g * d_group_stride, row stride ldd.
extern "C" int dewb_tgmm_bf16(const void* A, const void* B, void* D, const int* group_offsets, int R, int M, int N,
                              int groups, long long lda, long long ldb, long long ldd, long long d_group_stride, int epi,
                              float alpha, int* err, void* stream_ptr) {
  using namespace dewb;
  using namespace dewb::gemm_pair;
  if (R <= 0 || M <= 0 || N <= 0 || groups <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -3;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  CUtensorMap ta, tb;
  const int r = operand_maps(&ta, &tb, A, B, M, N, R, lda, ldb, 1, 1);
  if (r) return r;
  const Ranges gr{group_offsets, 0, groups, d_group_stride};
  switch (epi) {
    case EPI_BF16: return launch_one<true, true, EPI_BF16, true>(ta, tb, D, M, N, R, ldd, alpha, err, 0, stream, nullptr, gr);
    case EPI_F32: return launch_one<true, true, EPI_F32, true>(ta, tb, D, M, N, R, ldd, alpha, err, 0, stream, nullptr, gr);
    case EPI_F32_ACC: return launch_one<true, true, EPI_F32_ACC, true>(ta, tb, D, M, N, R, ldd, alpha, err, 0, stream, nullptr, gr);
    case EPI_BF16_ACC: return launch_one<true, true, EPI_BF16_ACC, true>(ta, tb, D, M, N, R, ldd, alpha, err, 0, stream, nullptr, gr);
  }
  return -2;
}
