// Products with one to four rows: y [M, N] = x [M, K] w [N, K]^T (+ bias), bf16 with fp32 sums - a generation step of a few requests, the conditioning of a few images.
//
// Bound by the read of w.  A warp makes COLS columns of all rows: its lanes walk K in 16-byte pieces, COLS x DEPTH of them in flight, and the pieces of x come from
// the first-level cache, where all the warps of an SM share them.  No tensor core: at four rows the products of a weight piece take less than its arrival, and a
// tensor-core tile would compute 124 rows of nothing.  COLS is the largest of 4, 2, 1 that still gives every SM sixteen warps: more columns share the pieces of x, but
// for matrices this small a warp's time is the latency of its chain of loads.  One row by 12288 x 512, COLS 1, 2, 4: 4.9, 5.0, 3.9 us; by 8192 x 256: 3.1, 2.7, 2.6; by
// 3072 x 2048: 5.6, 6.3, 7.0.  Three and four rows are taken up to 4096 columns, where it is 1.
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dewb {
namespace rowsmm {

constexpr int WARPS = 4, DEPTH = 4;

__device__ __forceinline__ float lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

template <int M, int COLS>
__global__ void __launch_bounds__(WARPS * 32)
rows_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ y, int N, int K,
            long long ldx, long long ldw, long long ldy) {
  const int lane = threadIdx.x & 31, col = (blockIdx.x * WARPS + (threadIdx.x >> 5)) * COLS;
  if (col >= N) return;
  float acc[M][COLS];
#pragma unroll
  for (int m = 0; m < M; ++m)
#pragma unroll
    for (int c = 0; c < COLS; ++c) acc[m][c] = 0.f;
  const uint4* wp[COLS];
#pragma unroll
  for (int c = 0; c < COLS; ++c) wp[c] = reinterpret_cast<const uint4*>(w + min(col + c, N - 1) * ldw);
  const int pieces = K / 8;
  auto add = [&](int at, const uint4 (&v)[COLS]) {
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const uint4 a = reinterpret_cast<const uint4*>(x + m * ldx)[at];
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        const uint32_t vw[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[m][c] = fmaf(hi(aw[i]), hi(vw[i]), fmaf(lo(aw[i]), lo(vw[i]), acc[m][c]));
      }
    }
  };
  int at = lane;
  for (; at + 32 * (DEPTH - 1) < pieces; at += 32 * DEPTH) {
    uint4 v[DEPTH][COLS];
#pragma unroll
    for (int u = 0; u < DEPTH; ++u)
#pragma unroll
      for (int c = 0; c < COLS; ++c) v[u][c] = __ldcs(wp[c] + at + u * 32);
#pragma unroll
    for (int u = 0; u < DEPTH; ++u) add(at + u * 32, v[u]);
  }
  for (; at < pieces; at += 32) {
    uint4 v[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) v[c] = __ldcs(wp[c] + at);
    add(at, v);
  }
#pragma unroll
  for (int m = 0; m < M; ++m)
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[m][c] += __shfl_xor_sync(0xffffffffu, acc[m][c], o);
      if (lane == m * COLS + c && col + c < N) y[m * ldy + col + c] = __float2bfloat16(acc[m][c] + (bias == nullptr ? 0.f : __bfloat162float(bias[col + c])));
    }
}

template <int M>
static int go(const void* x, const void* w, const void* bias, void* y, int N, int K, long long ldx, long long ldw, long long ldy, cudaStream_t stream) {
  typedef const __nv_bfloat16* in;
  int cols = 1;
  auto fn = rows_kernel<M, 1>;
  if constexpr (M <= 2) {
    cols = N >= 148 * WARPS * 4 * 4 ? 4 : N >= 148 * WARPS * 4 * 2 ? 2 : 1;
    fn = cols == 4 ? rows_kernel<M, 4> : cols == 2 ? rows_kernel<M, 2> : rows_kernel<M, 1>;
  }
  const unsigned blocks = static_cast<unsigned>((N + cols * WARPS - 1) / (cols * WARPS));
  fn<<<blocks, WARPS * 32, 0, stream>>>(static_cast<in>(x), static_cast<in>(w), static_cast<in>(bias), static_cast<__nv_bfloat16*>(y), N, K, ldx, ldw, ldy);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace rowsmm
}  // namespace dewb

// x [M, K], w [N, K], y [M, N] bf16 with the given row strides (elements; K, ldx, ldw multiples of 8, x and w 16-byte aligned), bias [N] bf16 or null; 1 <= M <= 4.
extern "C" int dewb_gemm_rows_bf16(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, long long ldx, long long ldw, long long ldy, void* stream_ptr) {
  using namespace dewb::rowsmm;
  if (M < 1 || M > 4 || K % 8 || ldx % 8 || ldw % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15)) return -3;
  if (N <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream_ptr);
  switch (M) {
    case 1: return go<1>(x, w, bias, y, N, K, ldx, ldw, ldy, s);
    case 2: return go<2>(x, w, bias, y, N, K, ldx, ldw, ldy, s);
    case 3: return go<3>(x, w, bias, y, N, K, ldx, ldw, ldy, s);
    default: return go<4>(x, w, bias, y, N, K, ldx, ldw, ldy, s);
  }
}
