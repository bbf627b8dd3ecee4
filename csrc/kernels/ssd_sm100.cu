// Mamba-2 state space scan, forward and backward (head dimension P = 64, state dimension N = 128, chunks of 64 tokens).
//
// With g_i the running sum of dt A inside a chunk, S the state in front of it and h the head (several heads share one group's B and C):
//     y_i = e^{g_i} S C_i + sum_{j <= i} (C_i . B_j) e^{g_i - g_j} dt_j x_j + D x_i         S <- e^{g_L} S + sum_j e^{g_L - g_j} dt_j x_j B_j^T
// The work splits at the state:
//   ssd_states  one CTA per (batch, head, slice of the state's columns) walks the chunks and leaves the state in front of each of them in memory; run in reverse
//               with (dy, C, e^{g_i}) in the places of (x, B, dt e^{g_L - g}) it leaves the gradient of the state behind each chunk.  Nothing else is sequential.
//   ssd_output  y of one chunk and group, head after head: C B^T stays in registers for all of them.
//   ssd_local   the gradients of one chunk and group, head after head, from the two states.  dC, dB and the score gradients are summed over the heads in
//               registers, so that the product with B (C) is one per group and not one per head:
//                 E = dy x^T          M = (C B^T) o e^{g_i - g_j}        W = sum_h E o e^{g_i - g_j} dt_j
//                 dC = sum_h e^{g_i} (dy S) + W B          dB = sum_h dt_j e^{g_L - g_j} (x dS) + W^T C          dx = dt_j (M^T dy + e^{g_L - g_j} B dS^T) + D dy
//               and the gradients of the decays from row and column sums of M o E and from the dots of (dy S) with C and (x dS) with B.
//   ssd_reduce  sums what several CTAs made of one group's dB and dC, and dA and dD over the chunks, in a fixed order.
// x, B, C and dy enter every product as the bf16 numbers they are.  The forward rounds the state, the weights of a chunk's own tokens and the decayed x to bf16,
// once each.  The backward keeps all of them in fp32: such an operand goes through the tensor cores as three bf16 terms (24 bits of mantissa), smallest first.
//
// The products are narrow (64 rows, 64 to 128 columns, a reduction of 64 to 128) and their fp32 operands change with every head, so they run on mma.sync out of
// registers, where an operand is scaled and split without passing through memory; 146 GFLOP of them stand in the backward of 2 x 4096 x 64 heads.
//
// Replaces the reference's ported SSD kernels ChunkState / StatePassing / ChunkScan (src/dew/nn/kernels/mamba_ssd.py:421-660).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include "../common/mma_bf16.cuh"

namespace dewb {
namespace ssd {

using namespace mma16;

constexpr int N = 128, P = 64, L = 64;
constexpr uint32_t FULL = 0xffffffffu;
constexpr int SMS = 148;

// What the kernels read of the call's tensors: element strides between tokens and batch rows; heads (groups) of a token lie P (N) elements apart.
struct Call {
  const __nv_bfloat16 *x, *Bm, *Cm, *dy;
  const float *dt, *A, *D;
  long long xb, xt, bb, bt, cb, ct;      // dy is contiguous
  int B, T, H, G, chunks;
};

__device__ __forceinline__ void cp16(void* dst, const void* src, bool real) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(real ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// A tile of 64 rows of CH 16-byte pieces, piece c of row r at (c ^ swizzle(r)): eight rows of one column of pieces lie in eight different bank groups.
template <int CH>
__device__ __forceinline__ int piece(int r, int c) { return (r * CH + (CH >= 8 ? c ^ (r & 7) : c ^ ((r >> 1) & 3))) * 16; }

// rows [0, real) from memory, zeros behind them
template <int CH, int THREADS>
__device__ __forceinline__ void load_tile(uint8_t* dst, const __nv_bfloat16* src, long long stride, int real) {
#pragma unroll
  for (int i = 0; i < L * CH / THREADS; ++i) {
    const int at = i * THREADS + static_cast<int>(threadIdx.x), r = at / CH, c = at % CH;
    cp16(dst + piece<CH>(r, c), src + (r < real ? r * stride : 0) + c * 8, r < real);
  }
}

// Fragments.  A operand (16 rows x 16) of a row-major tile; of its transpose (16 columns x 16 rows).
template <int CH>
__device__ __forceinline__ void frag_a(uint32_t (&a)[4], const uint8_t* t, int row, int ks) {
  const int lane = threadIdx.x & 31, m = lane >> 3;
  ldsm4(a, smem_addr(t + piece<CH>(row + (m & 1) * 8 + (lane & 7), ks * 2 + (m >> 1))));
}
template <int CH>
__device__ __forceinline__ void frag_a_t(uint32_t (&a)[4], const uint8_t* t, int ks, int col) {      // col: in pieces of 8
  const int lane = threadIdx.x & 31, m = lane >> 3;
  ldsm4_t(a, smem_addr(t + piece<CH>(ks * 16 + (m >> 1) * 8 + (lane & 7), col + (m & 1))));
}
// B operands of two neighbouring column tiles: reduction along the tile's rows (columns: pieces col, col + 1), or along its columns (columns of the product: rows row ..)
template <int CH>
__device__ __forceinline__ void frag_b_t(uint32_t (&b)[4], const uint8_t* t, int ks, int col) {
  const int lane = threadIdx.x & 31, m = lane >> 3;
  ldsm4_t(b, smem_addr(t + piece<CH>(ks * 16 + (m & 1) * 8 + (lane & 7), col + (m >> 1))));
}
template <int CH>
__device__ __forceinline__ void frag_b(uint32_t (&b)[4], const uint8_t* t, int row, int ks) {
  const int lane = threadIdx.x & 31, m = lane >> 3;
  ldsm4(b, smem_addr(t + piece<CH>(row + (m >> 1) * 8 + (lane & 7), ks * 2 + (m & 1))));
}

// Two fp32 values as three bf16 pairs, the largest first: 24 bits of mantissa together.
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack2(a, b);
  const float ra = a - lo_f(hi), rb = b - hi_f(hi);
  mid = pack2(ra, rb);
  lo = pack2(ra - lo_f(mid), rb - hi_f(mid));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

// One warp: the running sums of dt A over a chunk, lane l the tokens 2l and 2l + 1.
__device__ __forceinline__ void running(float dt0, float dt1, float A, float& g0, float& g1) {
  const int lane = threadIdx.x & 31;
  const float v0 = dt0 * A, v1 = dt1 * A;
  float incl = v0 + v1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float up = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += up;
  }
  float before = __shfl_up_sync(FULL, incl, 1);
  if (lane == 0) before = 0.f;
  g0 = before + v0;
  g1 = before + (v0 + v1);
}

// ---------------------------------------------------------------------------------------------------------------
// The walk over the chunks, forward (blockIdx.z 0) and in reverse (1) side by side.  Four warps, 16 rows of the state each (S is kept [P, N]); NT column tiles of 8 a
// CTA.  The columns are independent of each other, and one CTA's step is a chain (scale, split, products, decay), so a call with few (batch, head) pairs is cut
// along them.  A fifth warp fetches the tiles two chunks ahead, a sixth makes the weights one ahead, so that a step has one barrier and nothing of either in its chain.
// (With both in the computing warps and a launch for each direction, 2 x 4096 tokens of 64 heads took 306 us both ways instead of 241, and 124 us for the forward pass instead of 88.)
constexpr int WALK_STAGES = 3, WALK_THREADS = 192;
template <int NT, int TERMS, typename Out>
__global__ void __launch_bounds__(WALK_THREADS, 2)
ssd_states(Call k, const float* __restrict__ initial, Out* __restrict__ states, float* __restrict__ last, const float* __restrict__ rev_initial, Out* __restrict__ rev_states,
           float* __restrict__ rev_last) {
  constexpr int CV = NT;                               // 16-byte pieces of a row of B (C)
  constexpr int U_BYTES = L * P * 2, V_BYTES = L * CV * 16;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(16) float weight[2][L], total[2];
  const bool rev = blockIdx.z != 0;
  if (rev) { initial = rev_initial; states = rev_states; last = rev_last; }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
  const int b = blockIdx.x / k.H, h = blockIdx.x % k.H, grp = h / (k.H / k.G), col0 = blockIdx.y * NT * 8;
  auto chunk = [&](int it) { return rev ? k.chunks - 1 - it : it; };
  if (warp == 4) {
    const __nv_bfloat16* u = rev ? k.dy + static_cast<long long>(b) * k.T * k.H * P + h * P : k.x + b * k.xb + h * P;
    const __nv_bfloat16* v = (rev ? k.Cm + b * k.cb : k.Bm + b * k.bb) + grp * N + col0;
    const long long us = rev ? static_cast<long long>(k.H) * P : k.xt, vs = rev ? k.ct : k.bt;
    auto fetch = [&](int it) {
      if (it < k.chunks) {
        const int t0 = chunk(it) * L, real = min(L, k.T - t0);
        uint8_t* st = smem + (it % WALK_STAGES) * (U_BYTES + V_BYTES);
#pragma unroll 4
        for (int i = 0; i < L * 8 / 32; ++i) {
          const int row = i * 4 + (lane >> 3), c = lane & 7;
          cp16(st + piece<8>(row, c), u + (t0 + (row < real ? row : 0)) * us + c * 8, row < real);
        }
#pragma unroll 4
        for (int i = 0; i < L * CV / 32; ++i) {
          const int row = (i * 32 + lane) / CV, c = (i * 32 + lane) % CV;
          cp16(st + U_BYTES + piece<CV>(row, c), v + (t0 + (row < real ? row : 0)) * vs + c * 8, row < real);
        }
      }
      cp_commit();                                     // (a group for every chunk, empty behind the last)
    };
    fetch(0);
    fetch(1);
    for (int it = 0; it < k.chunks; ++it) {
      cp_wait<1>();
      __syncthreads();                                 // chunk `it` is there, and chunk it - 1's stage is free
      fetch(it + 2);
    }
    return;
  }
  if (warp == 5) {
    const float A = k.A[h];
    const float* dt = k.dt + static_cast<long long>(b) * k.T * k.H + h;
    float next0, next1;
    auto fetch = [&](int it) {
      const int t = it < k.chunks ? chunk(it) * L + 2 * lane : k.T;
      next0 = t < k.T ? dt[static_cast<long long>(t) * k.H] : 0.f;
      next1 = t + 1 < k.T ? dt[static_cast<long long>(t + 1) * k.H] : 0.f;
    };
    auto weigh = [&](int it) {                         // e^{g_i}, or dt_j e^{g_L - g_j}
      const float dt0 = next0, dt1 = next1;
      fetch(it + 1);
      float g0, g1;
      running(dt0, dt1, A, g0, g1);
      const float gl = __shfl_sync(FULL, g1, 31);
      weight[it & 1][2 * lane] = rev ? expf(g0) : dt0 * expf(gl - g0);
      weight[it & 1][2 * lane + 1] = rev ? expf(g1) : dt1 * expf(gl - g1);
      if (lane == 0) total[it & 1] = expf(gl);
    };
    fetch(0);
    weigh(0);
    for (int it = 0; it < k.chunks; ++it) {
      __syncthreads();
      if (it + 1 < k.chunks) weigh(it + 1);            // (the other half: chunk it reads its own)
    }
    return;
  }
  const long long cell = static_cast<long long>(P) * N, at = (warp * 16 + r) * N + col0 + 2 * q;      // this thread's first value of a state
  float S[NT][4];
  const float* from = initial == nullptr ? nullptr : initial + blockIdx.x * cell + at;
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const float2 a = from == nullptr ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2*>(from + n * 8);
    const float2 c = from == nullptr ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2*>(from + n * 8 + 8 * N);
    S[n][0] = a.x; S[n][1] = a.y; S[n][2] = c.x; S[n][3] = c.y;
  }
  for (int it = 0; it < k.chunks; ++it) {
    __syncthreads();
    Out* to = states + (static_cast<long long>(blockIdx.x) * k.chunks + chunk(it)) * cell + at;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      if constexpr (sizeof(Out) == 4) {
        *reinterpret_cast<float2*>(to + n * 8) = make_float2(S[n][0], S[n][1]);
        *reinterpret_cast<float2*>(to + n * 8 + 8 * N) = make_float2(S[n][2], S[n][3]);
      } else {
        *reinterpret_cast<uint32_t*>(to + n * 8) = pack2(S[n][0], S[n][1]);
        *reinterpret_cast<uint32_t*>(to + n * 8 + 8 * N) = pack2(S[n][2], S[n][3]);
      }
    }
    const uint8_t* st = smem + (it % WALK_STAGES) * (U_BYTES + V_BYTES);
    uint32_t a[TERMS][4][4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t w[4];
      frag_a_t<8>(w, st, ks, warp * 2);
      const float2 s0 = *reinterpret_cast<const float2*>(&weight[it & 1][ks * 16 + 2 * q]), s1 = *reinterpret_cast<const float2*>(&weight[it & 1][ks * 16 + 8 + 2 * q]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 s = i < 2 ? s0 : s1;
        if constexpr (TERMS == 3) split3(lo_f(w[i]) * s.x, hi_f(w[i]) * s.y, a[0][ks][i], a[1][ks][i], a[2][ks][i]);
        else a[0][ks][i] = pack2(lo_f(w[i]) * s.x, hi_f(w[i]) * s.y);
      }
    }
    const float decay = total[it & 1];
#pragma unroll
    for (int n = 0; n < NT; n += 2) {
      uint32_t vb[4][4];
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) frag_b_t<CV>(vb[ks], st + U_BYTES, ks, n);
      // a chunk's share is summed by itself and joins the state in one rounded step
      float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int t = TERMS - 1; t >= 0; --t)
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) { mma(c0, a[t][ks], vb[ks][0], vb[ks][1]); mma(c1, a[t][ks], vb[ks][2], vb[ks][3]); }
#pragma unroll
      for (int i = 0; i < 4; ++i) { S[n][i] = fmaf(S[n][i], decay, c0[i]); S[n + 1][i] = fmaf(S[n + 1][i], decay, c1[i]); }
    }
  }
  if (last != nullptr) {
    float* to = last + blockIdx.x * cell + at;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      *reinterpret_cast<float2*>(to + n * 8) = make_float2(S[n][0], S[n][1]);
      *reinterpret_cast<float2*>(to + n * 8 + 8 * N) = make_float2(S[n][2], S[n][3]);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// y of one chunk, one group, `per` of its heads: four warps, 16 tokens each.
constexpr int OUT_STAGE = L * P * 2 + P * N * 2;
constexpr int OUT_SMEM = 2 * L * N * 2 + 2 * OUT_STAGE + L * P * 2;

__global__ void __launch_bounds__(128)
ssd_output(Call k, const __nv_bfloat16* __restrict__ states, __nv_bfloat16* __restrict__ y, int per) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(16) float sg[2][L], sdt[2][L];
  uint8_t *tC = smem, *tB = tC + L * N * 2, *stages = tB + L * N * 2, *tY = stages + 2 * OUT_STAGE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
  const int b = blockIdx.x / k.chunks, n = blockIdx.x % k.chunks, grp = blockIdx.y, h0 = grp * (k.H / k.G) + blockIdx.z * per;
  const int t0 = n * L, real = min(L, k.T - t0), row = warp * 16;
  auto fetch = [&](int i) {
    uint8_t* st = stages + (i & 1) * OUT_STAGE;
    load_tile<8, 128>(st, k.x + b * k.xb + t0 * k.xt + (h0 + i) * P, k.xt, real);
    load_tile<16, 128>(st + L * P * 2, states + ((static_cast<long long>(b) * k.H + h0 + i) * k.chunks + n) * P * N, N, P);
    cp_commit();
  };
  auto decays = [&](int i) {                           // warp 0
    const int t = t0 + 2 * lane;
    const float* dt = k.dt + static_cast<long long>(b) * k.T * k.H + h0 + i;
    const float a = t < k.T ? dt[static_cast<long long>(t) * k.H] : 0.f, c = t + 1 < k.T ? dt[static_cast<long long>(t + 1) * k.H] : 0.f;
    float g0, g1;
    running(a, c, k.A[h0 + i], g0, g1);
    *reinterpret_cast<float2*>(&sg[i & 1][2 * lane]) = make_float2(g0, g1);
    *reinterpret_cast<float2*>(&sdt[i & 1][2 * lane]) = make_float2(a, c);
  };
  load_tile<16, 128>(tC, k.Cm + b * k.cb + t0 * k.ct + grp * N, k.ct, real);
  load_tile<16, 128>(tB, k.Bm + b * k.bb + t0 * k.bt + grp * N, k.bt, real);
  cp_commit();
  fetch(0);
  if (warp == 0) decays(0);
  cp_wait<1>();
  __syncthreads();
  float G[8][4];                                       // C B^T of this warp's tokens; column tiles behind them stay unused
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) G[j][i] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    uint32_t a[4];
    frag_a<16>(a, tC, row, ks);
#pragma unroll
    for (int j = 0; j < 8; j += 2)
      if (j <= 2 * warp) {
        uint32_t bb[4];
        frag_b<16>(bb, tB, j * 8, ks);
        mma(G[j], a, bb[0], bb[1]);
        mma(G[j + 1], a, bb[2], bb[3]);
      }
  }
  for (int i = 0; i < per; ++i) {
    if (i + 1 < per) { fetch(i + 1); if (warp == 0) decays(i + 1); cp_wait<1>(); }
    else cp_wait<0>();
    __syncthreads();
    const uint8_t *tx = stages + (i & 1) * OUT_STAGE, *tS = tx + L * P * 2;
    const float *g = sg[i & 1], *dt = sdt[i & 1];
    const float gi0 = g[row + r], gi1 = g[row + r + 8];
    float acc[8][4];
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[p][c] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t a[4];
      frag_a<16>(a, tC, row, ks);
#pragma unroll
      for (int p = 0; p < 8; p += 2) {
        uint32_t bb[4];
        frag_b<16>(bb, tS, p * 8, ks);
        mma(acc[p], a, bb[0], bb[1]);
        mma(acc[p + 1], a, bb[2], bb[3]);
      }
    }
    const float e0 = expf(gi0), e1 = expf(gi1);
#pragma unroll
    for (int p = 0; p < 8; ++p) { acc[p][0] *= e0; acc[p][1] *= e0; acc[p][2] *= e1; acc[p][3] *= e1; }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      if (ks <= warp) {
        uint32_t a[4];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int j = ks * 16 + t * 8 + 2 * q;
          const float2 gj = *reinterpret_cast<const float2*>(g + j), d = *reinterpret_cast<const float2*>(dt + j);
          const float* w = G[ks * 2 + t];
          const int i0 = row + r, i1 = i0 + 8;
          a[2 * t] = pack2(j <= i0 ? w[0] * expf(gi0 - gj.x) * d.x : 0.f, j + 1 <= i0 ? w[1] * expf(gi0 - gj.y) * d.y : 0.f);
          a[2 * t + 1] = pack2(j <= i1 ? w[2] * expf(gi1 - gj.x) * d.x : 0.f, j + 1 <= i1 ? w[3] * expf(gi1 - gj.y) * d.y : 0.f);
        }
#pragma unroll
        for (int p = 0; p < 8; p += 2) {
          uint32_t bb[4];
          frag_b_t<8>(bb, tx, ks, p);
          mma(acc[p], a, bb[0], bb[1]);
          mma(acc[p + 1], a, bb[2], bb[3]);
        }
      }
    const float D = k.D == nullptr ? 0.f : k.D[h0 + i];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const uint32_t x0 = *reinterpret_cast<const uint32_t*>(tx + piece<8>(row + r, p) + q * 4), x1 = *reinterpret_cast<const uint32_t*>(tx + piece<8>(row + r + 8, p) + q * 4);
      *reinterpret_cast<uint32_t*>(tY + piece<8>(row + r, p) + q * 4) = pack2(fmaf(D, lo_f(x0), acc[p][0]), fmaf(D, hi_f(x0), acc[p][1]));
      *reinterpret_cast<uint32_t*>(tY + piece<8>(row + r + 8, p) + q * 4) = pack2(fmaf(D, lo_f(x1), acc[p][2]), fmaf(D, hi_f(x1), acc[p][3]));
    }
    __syncwarp();                                      // (a warp stores the rows it made)
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int at = row + s * 4 + (lane >> 3), c = lane & 7;
      if (at < real)
        *reinterpret_cast<uint4*>(y + ((static_cast<long long>(b) * k.T + t0 + at) * k.H + h0 + i) * P + c * 8) = *reinterpret_cast<const uint4*>(tY + piece<8>(at, c));
    }
    __syncthreads();                                   // the stage is free for the head after the next
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Gradients of one chunk, one group, `per` of its heads: sixteen warps, four a scheduler (with eight of twice the work each, the tensor pipe was busy for 30 % of the
// time and the rest went to waits: 610 us for 2 x 4096 tokens of 64 heads instead of 585).  The products over the state's columns give each warp 8 of the 128 columns and all
// 64 tokens, so that every fp32 value of a state is split into its bf16 terms by the one warp that needs it; E and M are made by 16 x 16 pieces.
constexpr int LOCAL_WARPS = 16, LOCAL_THREADS = 32 * LOCAL_WARPS;
constexpr int SLD = N + 4;                             // row of an fp32 state in shared memory: the fragment reads of both orders spread over the banks
constexpr int LOCAL_STAGE = 2 * L * P * 2 + 2 * P * SLD * 4;
constexpr int M_BYTES = 10 * 3 * 512;                  // the ten 16 x 16 blocks of M^T with i >= j, three terms each, as A fragments
struct LocalSums {
  float rows[4][L];                                    // sum over j < i of M o E dt_j, by the tile of j
  float cols[4][L], diag[L], edge[L];                  // sum over i > j of M o E, by the tile of i; its diagonal; the diagonal of E
  float dy_state[LOCAL_WARPS][L], x_state[LOCAL_WARPS][L];      // (dy S) . C and (x dS) . B, by the warps' columns
  float both[LOCAL_WARPS];                             // <S, dS>
  float g[2][L], dt[2][L], head[2][L], tail[2][L];     // of this head and the next: g, dt, e^g, e^{g_L - g}
};
constexpr int LOCAL_SMEM = 2 * L * N * 2 + 2 * LOCAL_STAGE + M_BYTES + static_cast<int>(sizeof(LocalSums));
static_assert(LOCAL_SMEM <= 232448, "ssd_local exceeds the shared memory of an SM");

struct Grads {
  __nv_bfloat16 *dx, *dB, *dC;
  float *ddt, *partB, *partC, *partA, *partD;          // partB / partC: [splits][B, T, G, N] when a group's heads are split, else null; partA / partD: [B * chunks, H]
};

// which of the ten blocks of the lower triangle (j tile, i tile >= j tile)
__device__ __forceinline__ int block_of(int jt, int it) { return jt * 4 - jt * (jt - 1) / 2 + it - jt; }

__global__ void __launch_bounds__(LOCAL_THREADS, 1)
ssd_local(Call k, const float* __restrict__ states, const float* __restrict__ dstates, Grads out, int per) {
  extern __shared__ __align__(128) uint8_t smem[];
  uint8_t *tB = smem, *tC = tB + L * N * 2, *stages = tC + L * N * 2, *tM = stages + 2 * LOCAL_STAGE;
  LocalSums& sum = *reinterpret_cast<LocalSums*>(tM + M_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
  const int b = blockIdx.x / k.chunks, n = blockIdx.x % k.chunks, grp = blockIdx.y, h0 = grp * (k.H / k.G) + blockIdx.z * per;
  const int t0 = n * L, real = min(L, k.T - t0);
  const int jt = warp >> 2, it = warp & 3;             // this warp's piece of E^T: tokens j of tile jt, tokens i of tile it
  const bool lower = it >= jt;                         // whether some i >= j is in it
  const int pt = warp & 7, side = warp >> 3;           // its piece of dx: columns 8 pt .. of the head, tokens of the tiles 0 and 3 or 1 and 2
  auto fetch = [&](int i) {
    uint8_t* st = stages + (i & 1) * LOCAL_STAGE;
    const int h = h0 + i;
    load_tile<8, LOCAL_THREADS>(st, k.x + b * k.xb + t0 * k.xt + h * P, k.xt, real);
    load_tile<8, LOCAL_THREADS>(st + L * P * 2, k.dy + ((static_cast<long long>(b) * k.T + t0) * k.H + h) * P, static_cast<long long>(k.H) * P, real);
    const long long cell = ((static_cast<long long>(b) * k.H + h) * k.chunks + n) * P * N;
    float* fs = reinterpret_cast<float*>(st + 2 * L * P * 2);
#pragma unroll
    for (int s = 0; s < P * N / 4 / LOCAL_THREADS; ++s) {
      const int at = s * LOCAL_THREADS + static_cast<int>(threadIdx.x), row = at >> 5, c = at & 31;
      cp16(fs + row * SLD + c * 4, states + cell + row * N + c * 4, true);
      cp16(fs + (P + row) * SLD + c * 4, dstates + cell + row * N + c * 4, true);
    }
    cp_commit();
  };
  auto decays = [&](int i) {                           // the last warp
    const int t = t0 + 2 * lane;
    const float* dt = k.dt + static_cast<long long>(b) * k.T * k.H + h0 + i;
    const float a = t < k.T ? dt[static_cast<long long>(t) * k.H] : 0.f, c = t + 1 < k.T ? dt[static_cast<long long>(t + 1) * k.H] : 0.f;
    float g0, g1;
    running(a, c, k.A[h0 + i], g0, g1);
    const float gl = __shfl_sync(FULL, g1, 31);
    *reinterpret_cast<float2*>(&sum.g[i & 1][2 * lane]) = make_float2(g0, g1);
    *reinterpret_cast<float2*>(&sum.dt[i & 1][2 * lane]) = make_float2(a, c);
    *reinterpret_cast<float2*>(&sum.head[i & 1][2 * lane]) = make_float2(expf(g0), expf(g1));
    *reinterpret_cast<float2*>(&sum.tail[i & 1][2 * lane]) = make_float2(expf(gl - g0), expf(gl - g1));
  };
  load_tile<16, LOCAL_THREADS>(tC, k.Cm + b * k.cb + t0 * k.ct + grp * N, k.ct, real);
  load_tile<16, LOCAL_THREADS>(tB, k.Bm + b * k.bb + t0 * k.bt + grp * N, k.bt, real);
  cp_commit();
  fetch(0);
  if (warp == LOCAL_WARPS - 1) decays(0);
  if (threadIdx.x < 8 * L) (threadIdx.x < 4 * L ? &sum.rows[0][0] : &sum.cols[0][0] - 4 * L)[threadIdx.x] = 0.f;      // pieces above the diagonal write none
  cp_wait<1>();
  __syncthreads();

  float G[2][4], W[2][4], dC[4][4], dB[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    G[0][c] = G[1][c] = W[0][c] = W[1][c] = 0.f;
#pragma unroll
    for (int t = 0; t < 4; ++t) dC[t][c] = dB[t][c] = 0.f;
  }
  if (lower) {
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t a[4], c[4];
      frag_a<16>(a, tB, jt * 16, ks);
      frag_b<16>(c, tC, it * 16, ks);
      mma(G[0], a, c[0], c[1]);
      mma(G[1], a, c[2], c[3]);
    }
  }

  for (int i = 0; i < per; ++i) {
    cp_wait<0>();
    __syncthreads();                                   // this head has arrived, and nobody reads the one before it any more
    if (i + 1 < per) { fetch(i + 1); if (warp == LOCAL_WARPS - 1) decays(i + 1); }
    const int h = h0 + i;
    const uint8_t *tx = stages + (i & 1) * LOCAL_STAGE, *ty = tx + L * P * 2;
    const float *S = reinterpret_cast<const float*>(ty + L * P * 2), *dS = S + P * SLD;
    const float *g = sum.g[i & 1], *dt = sum.dt[i & 1], *head = sum.head[i & 1], *tail = sum.tail[i & 1];

    if (lower) {
      // ---- E^T = x dy^T of this piece, then M^T, W^T and the sums of M o E
      float E[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint32_t a[4], c[4];
        frag_a<8>(a, tx, jt * 16, ks);
        frag_b<8>(c, ty, it * 16, ks);
        mma(E[0], a, c[0], c[1]);
        mma(E[1], a, c[2], c[3]);
      }
      const int j0 = jt * 16 + r, j1 = j0 + 8;
      const float gj0 = g[j0], gj1 = g[j1], d0 = dt[j0], d1 = dt[j1];
      float col0 = 0.f, col1 = 0.f;
      uint8_t* to = tM + block_of(jt, it) * 1536 + lane * 16;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int i0 = it * 16 + t * 8 + 2 * q;
        const float2 gi = *reinterpret_cast<const float2*>(g + i0);
        float m[4], row0 = 0.f, row1 = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int ii = i0 + (c & 1), jj = c < 2 ? j0 : j1;
          const float dec = ii >= jj ? expf((c & 1 ? gi.y : gi.x) - (c < 2 ? gj0 : gj1)) : 0.f, d = c < 2 ? d0 : d1;
          m[c] = ii >= jj ? G[t][c] * dec : 0.f;
          const float me = ii >= jj ? m[c] * E[t][c] : 0.f;
          W[t][c] += ii >= jj ? E[t][c] * dec * d : 0.f;
          if (ii == jj) { sum.diag[jj] = me; sum.edge[jj] = E[t][c]; }
          else {
            if (c < 2) col0 += me; else col1 += me;
            if (c & 1) row1 += me * d; else row0 += me * d;
          }
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) { row0 += __shfl_xor_sync(FULL, row0, o); row1 += __shfl_xor_sync(FULL, row1, o); }
        if (r == 0) *reinterpret_cast<float2*>(&sum.rows[jt][i0]) = make_float2(row0, row1);
        // the pair of column tiles is one A fragment of M^T
        uint32_t hi[2], mid[2], lo[2];
        split3(m[0], m[1], hi[0], mid[0], lo[0]);
        split3(m[2], m[3], hi[1], mid[1], lo[1]);
        *reinterpret_cast<uint2*>(to + t * 8) = make_uint2(hi[0], hi[1]);
        *reinterpret_cast<uint2*>(to + 512 + t * 8) = make_uint2(mid[0], mid[1]);
        *reinterpret_cast<uint2*>(to + 1024 + t * 8) = make_uint2(lo[0], lo[1]);
      }
      col0 += __shfl_xor_sync(FULL, col0, 1); col0 += __shfl_xor_sync(FULL, col0, 2);
      col1 += __shfl_xor_sync(FULL, col1, 1); col1 += __shfl_xor_sync(FULL, col1, 2);
      if (q == 0) { sum.cols[it][j0] = col0; sum.cols[it][j1] = col1; }
    }

    // ---- (dy S) and (x dS): this warp's 8 columns of all tokens
    float both = 0.f;
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const float* F = (which ? dS : S) + 2 * q * SLD + warp * 8 + r;
      uint32_t f[3][4][2];
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const float* at = F + ks * 16 * SLD;
        const float v0 = at[0], v1 = at[SLD], v2 = at[8 * SLD], v3 = at[9 * SLD];
        if (which) {
          const float* o = at - P * SLD;
          both += v0 * o[0] + v1 * o[SLD] + v2 * o[8 * SLD] + v3 * o[9 * SLD];
        }
        split3(v0, v1, f[0][ks][0], f[1][ks][0], f[2][ks][0]);
        split3(v2, v3, f[0][ks][1], f[1][ks][1], f[2][ks][1]);
      }
      const uint8_t *tu = which ? tx : ty, *tw = which ? tB : tC;
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        // two sums side by side, so that a product need not wait for the one before it
        float u[4] = {0.f, 0.f, 0.f, 0.f}, u2[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t a[4][4];
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) frag_a<8>(a[ks], tu, mt * 16, ks);
#pragma unroll
        for (int term = 2; term >= 0; --term)
#pragma unroll
          for (int ks = 0; ks < 4; ks += 2) {
            mma(u, a[ks], f[term][ks][0], f[term][ks][1]);
            mma(u2, a[ks + 1], f[term][ks + 1][0], f[term][ks + 1][1]);
          }
#pragma unroll
        for (int c = 0; c < 4; ++c) u[c] += u2[c];
        const int i0 = mt * 16 + r, i1 = i0 + 8;
        const float s0 = which ? dt[i0] * tail[i0] : head[i0], s1 = which ? dt[i1] * tail[i1] : head[i1];
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(tw + piece<16>(i0, warp) + q * 4), w1 = *reinterpret_cast<const uint32_t*>(tw + piece<16>(i1, warp) + q * 4);
        float dot0 = u[0] * lo_f(w0) + u[1] * hi_f(w0), dot1 = u[2] * lo_f(w1) + u[3] * hi_f(w1);
        float(&to)[4] = which ? dB[mt] : dC[mt];
        to[0] = fmaf(s0, u[0], to[0]); to[1] = fmaf(s0, u[1], to[1]);
        to[2] = fmaf(s1, u[2], to[2]); to[3] = fmaf(s1, u[3], to[3]);
        dot0 += __shfl_xor_sync(FULL, dot0, 1); dot0 += __shfl_xor_sync(FULL, dot0, 2);
        dot1 += __shfl_xor_sync(FULL, dot1, 1); dot1 += __shfl_xor_sync(FULL, dot1, 2);
        if (q == 0) {
          float* at = which ? sum.x_state[warp] : sum.dy_state[warp];
          at[i0] = dot0; at[i1] = dot1;
        }
      }
    }
    both = warp_sum(both);
    if (lane == 0) sum.both[warp] = both;

    // ---- dx of this warp's piece.  First through the state: B dS^T
    float X[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const float* at = dS + (pt * 8 + r) * SLD + ks * 16 + 2 * q;
      const float2 v0 = *reinterpret_cast<const float2*>(at), v1 = *reinterpret_cast<const float2*>(at + 8);
      uint32_t f[3][2];
      split3(v0.x, v0.y, f[0][0], f[1][0], f[2][0]);
      split3(v1.x, v1.y, f[0][1], f[1][1], f[2][1]);
      uint32_t a[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m) frag_a<16>(a[m], tB, (m ? 3 - side : side) * 16, ks);
#pragma unroll
      for (int term = 2; term >= 0; --term)
#pragma unroll
        for (int m = 0; m < 2; ++m) mma(X[m], a[m], f[term][0], f[term][1]);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int j = (m ? 3 - side : side) * 16 + r;
      X[m][0] *= tail[j]; X[m][1] *= tail[j]; X[m][2] *= tail[j + 8]; X[m][3] *= tail[j + 8];
    }
    __syncthreads();
    // then through the chunk's own tokens: M^T dy
    uint32_t yb[2][4];
#pragma unroll
    for (int s = 0; s < 2; ++s) ldsm4_t(yb[s], smem_addr(ty + piece<8>(s * 32 + lane, pt)));
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int mt = m ? 3 - side : side;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        if (ks < mt) continue;
        const uint8_t* at = tM + block_of(mt, ks) * 1536 + lane * 16;
#pragma unroll
        for (int term = 2; term >= 0; --term) {
          // (stored by column tile: rows r and r + 8 of the first, then of the second, which is the fragment's order)
          const uint4 w = *reinterpret_cast<const uint4*>(at + term * 512);
          const uint32_t a[4] = {w.x, w.y, w.z, w.w};
          mma(X[m], a, yb[ks >> 1][(ks & 1) * 2], yb[ks >> 1][(ks & 1) * 2 + 1]);
        }
      }
    }
    const float D = k.D == nullptr ? 0.f : k.D[h];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int j = (m ? 3 - side : side) * 16 + r + half * 8;
        const uint32_t w = *reinterpret_cast<const uint32_t*>(ty + piece<8>(j, pt) + q * 4);
        const float d = dt[j];
        if (j < real)
          *reinterpret_cast<uint32_t*>(out.dx + ((static_cast<long long>(b) * k.T + t0 + j) * k.H + h) * P + pt * 8 + 2 * q) =
              pack2(fmaf(D, lo_f(w), d * X[m][half * 2]), fmaf(D, hi_f(w), d * X[m][half * 2 + 1]));
      }
    if (warp == 0) {
      // ---- the decays: dg_i from what the token receives less what it gives, its sums to the chunk's end are the gradients of dt A
      float dg[2], direct[2], given = 0.f, d[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        float take = 0.f, give = 0.f;
#pragma unroll
        for (int w = 0; w < LOCAL_WARPS; ++w) { take += sum.dy_state[w][t]; give += sum.x_state[w][t]; }
        d[e] = dt[t];
        give *= tail[t];
        given += d[e] * give;
        const float own = ((sum.cols[0][t] + sum.cols[1][t]) + (sum.cols[2][t] + sum.cols[3][t])) + give;
        dg[e] = ((sum.rows[0][t] + sum.rows[1][t]) + (sum.rows[2][t] + sum.rows[3][t])) + head[t] * take - d[e] * own;
        direct[e] = own + sum.diag[t];
      }
      given = warp_sum(given);
      float held = 0.f;
#pragma unroll
      for (int w = 0; w < LOCAL_WARPS; ++w) held += sum.both[w];
      if (lane == 31) dg[1] += head[L - 1] * held + given;
      float suffix = dg[0] + dg[1];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float down = __shfl_down_sync(FULL, suffix, o);
        if (lane + o < 32) suffix += down;
      }
      float after = __shfl_down_sync(FULL, suffix, 1);
      if (lane == 31) after = 0.f;
      const float da1 = after + dg[1], da0 = after + (dg[0] + dg[1]), A = k.A[h];
      const int t = 2 * lane;
      float* to = out.ddt + (static_cast<long long>(b) * k.T + t0) * k.H + h;
      if (t < real) to[static_cast<long long>(t) * k.H] = fmaf(A, da0, direct[0]);
      if (t + 1 < real) to[static_cast<long long>(t + 1) * k.H] = fmaf(A, da1, direct[1]);
      const float sA = warp_sum(d[0] * da0 + d[1] * da1), sD = warp_sum(sum.edge[t] + sum.edge[t + 1]);
      if (lane == 0) {
        const long long at = static_cast<long long>(blockIdx.x) * k.H + h;
        out.partA[at] = sA;
        out.partD[at] = sD;
      }
    }
  }

  // ---- W B and W^T C, once for all heads: W^T [j][i] in fp32 through the stages' memory
  __syncthreads();
  float* tW = reinterpret_cast<float*>(stages);
  constexpr int WLD = L + 4;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    float* at = tW + (jt * 16 + r) * WLD + it * 16 + t * 8 + 2 * q;
    *reinterpret_cast<float2*>(at) = make_float2(W[t][0], W[t][1]);
    *reinterpret_cast<float2*>(at + 8 * WLD) = make_float2(W[t][2], W[t][3]);
  }
  __syncthreads();
  uint32_t fB[2][4], fC[2][4];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    ldsm4_t(fB[s], smem_addr(tB + piece<16>(s * 32 + lane, warp)));
    ldsm4_t(fC[s], smem_addr(tC + piece<16>(s * 32 + lane, warp)));
  }
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      if (ks <= mt) {                                  // dC_i += sum_j W_ij B_j
        const float* at = tW + (ks * 16 + 2 * q) * WLD + mt * 16 + r;
        uint32_t a[3][4];
        split3(at[0], at[WLD], a[0][0], a[1][0], a[2][0]);
        split3(at[8], at[WLD + 8], a[0][1], a[1][1], a[2][1]);
        split3(at[8 * WLD], at[9 * WLD], a[0][2], a[1][2], a[2][2]);
        split3(at[8 * WLD + 8], at[9 * WLD + 8], a[0][3], a[1][3], a[2][3]);
#pragma unroll
        for (int term = 2; term >= 0; --term) mma(dC[mt], a[term], fB[ks >> 1][(ks & 1) * 2], fB[ks >> 1][(ks & 1) * 2 + 1]);
      }
      if (ks >= mt) {                                  // dB_j += sum_i W_ij C_i
        const float* at = tW + (mt * 16 + r) * WLD + ks * 16 + 2 * q;
        uint32_t a[3][4];
        split3(at[0], at[1], a[0][0], a[1][0], a[2][0]);
        split3(at[8 * WLD], at[8 * WLD + 1], a[0][1], a[1][1], a[2][1]);
        split3(at[8], at[9], a[0][2], a[1][2], a[2][2]);
        split3(at[8 * WLD + 8], at[8 * WLD + 9], a[0][3], a[1][3], a[2][3]);
#pragma unroll
        for (int term = 2; term >= 0; --term) mma(dB[mt], a[term], fC[ks >> 1][(ks & 1) * 2], fC[ks >> 1][(ks & 1) * 2 + 1]);
      }
    }
#pragma unroll
  for (int mt = 0; mt < 4; ++mt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int t = mt * 16 + r + half * 8;
      if (t >= real) continue;
      const long long at = ((static_cast<long long>(b) * k.T + t0 + t) * k.G + grp) * N + warp * 8 + 2 * q;
      const float b0 = dB[mt][half * 2], b1 = dB[mt][half * 2 + 1], c0 = dC[mt][half * 2], c1 = dC[mt][half * 2 + 1];
      if (out.partB == nullptr) {
        *reinterpret_cast<uint32_t*>(out.dB + at) = pack2(b0, b1);
        *reinterpret_cast<uint32_t*>(out.dC + at) = pack2(c0, c1);
      } else {
        const long long part = blockIdx.z * (static_cast<long long>(k.B) * k.T * k.G * N);
        *reinterpret_cast<float2*>(out.partB + part + at) = make_float2(b0, b1);
        *reinterpret_cast<float2*>(out.partC + part + at) = make_float2(c0, c1);
      }
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Blocks [0, H): dA and dD of a head over all chunks; the others: four values of dB and of dC a thread over the splits.
__global__ void __launch_bounds__(256)
ssd_reduce(Grads g, float* __restrict__ dA, float* __restrict__ dD, int H, int parts, long long total, int splits) {
  if (blockIdx.x < H) {
    __shared__ float sA[8], sD[8];
    float a = 0.f, d = 0.f;
    for (int i = threadIdx.x; i < parts; i += 256) { a += g.partA[static_cast<long long>(i) * H + blockIdx.x]; d += g.partD[static_cast<long long>(i) * H + blockIdx.x]; }
    a = warp_sum(a); d = warp_sum(d);
    if ((threadIdx.x & 31) == 0) { sA[threadIdx.x >> 5] = a; sD[threadIdx.x >> 5] = d; }
    __syncthreads();
    if (threadIdx.x == 0) {
      a = d = 0.f;
      for (int w = 0; w < 8; ++w) { a += sA[w]; d += sD[w]; }
      dA[blockIdx.x] = a;
      if (dD != nullptr) dD[blockIdx.x] = d;
    }
    return;
  }
  const long long at = ((blockIdx.x - H) * 256ll + threadIdx.x) * 4;
  if (at >= total) return;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const float* from = (which ? g.partC : g.partB) + at;
    float4 s = *reinterpret_cast<const float4*>(from);
    for (int i = 1; i < splits; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(from + i * total);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *reinterpret_cast<uint2*>((which ? g.dC : g.dB) + at) = make_uint2(pack2(s.x, s.y), pack2(s.z, s.w));
  }
}

template <typename Out>
struct Walk { const float* initial; Out* states; float* last; };

template <int NT, int TERMS, typename Out>
static int run_states(const Call& k, const Walk<Out>& forward, const Walk<Out>* reverse, cudaStream_t stream) {
  auto fn = ssd_states<NT, TERMS, Out>;
  constexpr int bytes = WALK_STAGES * (L * P * 2 + L * NT * 16);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  const Walk<Out> none{nullptr, nullptr, nullptr}, &back = reverse == nullptr ? none : *reverse;
  fn<<<dim3(k.B * k.H, 16 / NT, reverse == nullptr ? 1 : 2), WALK_THREADS, bytes, stream>>>(k, forward.initial, forward.states, forward.last, back.initial, back.states, back.last);
  return static_cast<int>(cudaGetLastError());
}

// A quarter of the columns a CTA while that leaves every SM no more than two of them, else half (two more resident CTAs hide what a step's chain waits for, and a
// step of half the columns scales and splits half as often as two of a quarter).  In fp32, all of them where that alone makes one wave of two CTAs an SM: halves would
// make two waves, each of which scales and splits what the other does.  Both walks of 2 x 4096 tokens and 64 heads (256 CTAs): 278 us by quarters, 243 by halves, 226
// whole; of 4 x 2048 and 32 heads 141, 126, 117; but one walk of 128 CTAs, less than a CTA an SM, 121, 88, 103.  Where few SMs have two the others wait for them:
// 4096 tokens of 80 heads (160 CTAs) 218 us by halves and 223 whole, 2048 of 96 (192) 123 and 115; hence the line at five quarters of the SMs.
template <int TERMS, typename Out>
static int walk(const Call& k, const Walk<Out>& forward, const Walk<Out>* reverse, cudaStream_t stream) {
  const int rows = k.B * k.H * (reverse == nullptr ? 1 : 2);
  if (rows * 4 <= 2 * SMS) return run_states<4, TERMS, Out>(k, forward, reverse, stream);
  if constexpr (TERMS == 3)
    if (rows * 4 > 5 * SMS && rows <= 2 * SMS) return run_states<16, TERMS, Out>(k, forward, reverse, stream);
  return run_states<8, TERMS, Out>(k, forward, reverse, stream);
}

static int check(const Call& k) {
  if (k.B <= 0 || k.T <= 0 || k.H <= 0 || k.G <= 0 || k.H % k.G != 0 || k.G > 65535) return -3;
  // (batch rows by chunks, and by heads, lie along the grid's first dimension)
  if (static_cast<long long>(k.B) * k.chunks > 0x7fffffff || static_cast<long long>(k.B) * k.H > 0x7fffffff) return -3;
  if ((k.xb | k.xt | k.bb | k.bt | k.cb | k.ct) % 8) return -3;
  if ((reinterpret_cast<uintptr_t>(k.x) | reinterpret_cast<uintptr_t>(k.Bm) | reinterpret_cast<uintptr_t>(k.Cm) | reinterpret_cast<uintptr_t>(k.dy)) & 15) return -3;
  return 0;
}

}  // namespace ssd
}  // namespace dewb

// In how many parts the backward cuts the heads of a group (the leading size of its partial sums of dB and dC): the power of two that divides them with the
// shortest last wave, a CTA's start and end counted as a head and a half.
extern "C" int dewb_ssd_splits(int B, int T, int H, int G) {
  const int per_group = H / G;
  const long long base = static_cast<long long>(B) * ((T + dewb::ssd::L - 1) / dewb::ssd::L) * G;
  int best = 1;
  double least = 1e30;
  for (int s = 1; s <= per_group && per_group % s == 0; s *= 2) {
    const double cost = static_cast<double>((base * s + dewb::ssd::SMS - 1) / dewb::ssd::SMS) * (per_group / s + 1.5);
    if (cost < least * 0.97) { least = cost; best = s; }
  }
  return best;
}

// x bf16 [B, T, H, 64], Bm / Cm bf16 [B, T, G, 128] with the given strides (batch row, token; in elements, multiples of 8; 16-byte aligned), dt fp32
// [B, T, H], A [H], D [H] (may be null), initial fp32 [B, H, 64, 128] (may be null) -> y bf16 [B, T, H, 64], last fp32 [B, H, 64, 128]; states: scratch of
// B * H * ceil(T / 64) * 64 * 128 bf16.  What is not strided is contiguous.
extern "C" int dewb_ssd_fwd(const void* x, const float* dt, const float* A, const void* Bm, const void* Cm, const float* D, const float* initial, void* states,
                            void* y, float* last, int B, int T, int H, int G, const long long* strides, void* stream_ptr) {
  using namespace dewb::ssd;
  typedef const __nv_bfloat16* in;
  const Call k{static_cast<in>(x), static_cast<in>(Bm), static_cast<in>(Cm), nullptr, dt, A, D, strides[0], strides[1], strides[2], strides[3], strides[4], strides[5],
               B, T, H, G, (T + L - 1) / L};
  int e = check(k);
  if (e) return e;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  const Walk<__nv_bfloat16> forward{initial, static_cast<__nv_bfloat16*>(states), last};
  if ((e = walk<1, __nv_bfloat16>(k, forward, nullptr, stream))) return e;
  int splits = 1;                                      // two CTAs an SM
  while ((H / G) % (splits * 2) == 0 && static_cast<long long>(B) * k.chunks * G * splits < 2 * SMS) splits *= 2;
  cudaError_t c = cudaFuncSetAttribute(ssd_output, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_SMEM);
  if (c != cudaSuccess) return static_cast<int>(c);
  ssd_output<<<dim3(B * k.chunks, G, splits), 128, OUT_SMEM, stream>>>(k, static_cast<in>(states), static_cast<__nv_bfloat16*>(y), H / G / splits);
  return static_cast<int>(cudaGetLastError());
}

// The gradients of dewb_ssd_fwd's inputs for dy (bf16 [B, T, H, 64], contiguous) and dlast (fp32, gradient of `last`, may be null).  Scratch: states and dstates
// (fp32, B * H * ceil(T / 64) * 64 * 128 each), partA / partD (B * ceil(T / 64) * H), and with splits = dewb_ssd_splits(...) > 1 partB / partC
// (splits * B * T * G * 128).  dinitial and dD may be null.
extern "C" int dewb_ssd_bwd(const void* x, const float* dt, const float* A, const void* Bm, const void* Cm, const float* D, const float* initial, const void* dy,
                            const float* dlast, float* states, float* dstates, float* partA, float* partD, float* partB, float* partC, void* dx, float* ddt, float* dA,
                            void* dB, void* dC, float* dD, float* dinitial, int B, int T, int H, int G, const long long* strides, void* stream_ptr) {
  using namespace dewb::ssd;
  typedef const __nv_bfloat16* in;
  typedef __nv_bfloat16* to;
  const Call k{static_cast<in>(x), static_cast<in>(Bm), static_cast<in>(Cm), static_cast<in>(dy), dt, A, D, strides[0], strides[1], strides[2], strides[3], strides[4],
               strides[5], B, T, H, G, (T + L - 1) / L};
  int e = check(k);
  if (e) return e;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_ptr);
  const Walk<float> forward{initial, states, nullptr}, reverse{dlast, dstates, dinitial};
  if ((e = walk<3, float>(k, forward, &reverse, stream))) return e;
  const int splits = dewb_ssd_splits(B, T, H, G);
  if (splits > 1 && (partB == nullptr || partC == nullptr)) return -3;
  const Grads g{static_cast<to>(dx), static_cast<to>(dB), static_cast<to>(dC), ddt, splits > 1 ? partB : nullptr, splits > 1 ? partC : nullptr, partA, partD};
  cudaError_t c = cudaFuncSetAttribute(ssd_local, cudaFuncAttributeMaxDynamicSharedMemorySize, LOCAL_SMEM);
  if (c != cudaSuccess) return static_cast<int>(c);
  ssd_local<<<dim3(B * k.chunks, G, splits), LOCAL_THREADS, LOCAL_SMEM, stream>>>(k, states, dstates, g, H / G / splits);
  if ((c = cudaGetLastError()) != cudaSuccess) return static_cast<int>(c);
  const long long total = splits > 1 ? static_cast<long long>(B) * T * G * N : 0;
  ssd_reduce<<<static_cast<unsigned>(H + (total / 4 + 255) / 256), 256, 0, stream>>>(g, dA, dD, H, B * k.chunks, total, splits);
  return static_cast<int>(cudaGetLastError());
}
