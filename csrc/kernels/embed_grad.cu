// Gradient of an embedding table: dw[v] = sum of dy[t] over the tokens t with ids[t] = v, in the order of the tokens, fp32 sums rounded to bf16 once.
//
// The table's gradient is written once (cleared, then the rows that occur) and dy read once, which is what bounds it; the sums need the places of equal ids side by
// side.  A token's place in that order is the number of tokens in front of it, by id and then by place: up to 16384 tokens these are counted outright, every token
// against every other (a compare and an add a pair, spread over all SMs, the counts of the slices joined by integer atomics), where the library's sort of any length is
// a chain of eight launches and a bitonic network in one block's shared memory took 93 us for 8192 tokens (25 counted).  A block per place and 1024 columns then
// sums the run that begins there, if one does.  8192 tokens of 2048 features, 32768 ids: 450 us for the library's backward, 73 for this.
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dewb {
namespace embed {

constexpr int MOST = 16384;                            // tokens: the work grows with their square
constexpr int RANK_THREADS = 256, SLICE = 1024;
constexpr int SUM_THREADS = 128, UNROLL = 4;

// rank[i] += the tokens of slice blockIdx.y in front of token i.
__global__ void __launch_bounds__(RANK_THREADS)
rank_kernel(const long long* __restrict__ ids, int* __restrict__ rank, int T) {
  __shared__ __align__(16) int other[SLICE];
  const int first = blockIdx.y * SLICE, n = min(SLICE, T - first), i = blockIdx.x * RANK_THREADS + threadIdx.x;
  for (int j = threadIdx.x; j < SLICE; j += RANK_THREADS) other[j] = j < n ? static_cast<int>(ids[first + j]) : 0x7fffffff;      // (past the end: in front of nobody)
  __syncthreads();
  if (i >= T) return;
  const int mine = static_cast<int>(ids[i]);
  int count = 0;
  if (first + SLICE <= i) {                              // equal ids of an earlier slice come first
#pragma unroll 8
    for (int j = 0; j < SLICE; j += 4) {
      const int4 o = *reinterpret_cast<const int4*>(other + j);
      count += (o.x <= mine) + (o.y <= mine) + (o.z <= mine) + (o.w <= mine);
    }
  } else {
#pragma unroll 8
    for (int j = 0; j < SLICE; j += 4) {
      const int4 o = *reinterpret_cast<const int4*>(other + j);
      count += (o.x < mine) + (o.y < mine) + (o.z < mine) + (o.w < mine);
    }
    for (int j = 0; first + j < i && j < n; ++j) count += other[j] == mine;      // its own slice
  }
  if (count) atomicAdd(rank + i, count);
}

__global__ void __launch_bounds__(RANK_THREADS)
order_kernel(const long long* __restrict__ ids, const int* __restrict__ rank, int* __restrict__ sorted, int* __restrict__ place, int T) {
  const int i = blockIdx.x * RANK_THREADS + threadIdx.x;
  if (i >= T) return;
  sorted[rank[i]] = static_cast<int>(ids[i]);
  place[rank[i]] = i;
}

__global__ void __launch_bounds__(SUM_THREADS)
sum_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ sorted, const int* __restrict__ place, __nv_bfloat16* __restrict__ dw, int T, int d, int V) {
  const int first = blockIdx.x, id = sorted[first];
  if (static_cast<unsigned>(id) >= static_cast<unsigned>(V)) return;      // (the forward's lookup reports those)
  if (first > 0 && sorted[first - 1] == id) return;
  const int c = blockIdx.y * SUM_THREADS + threadIdx.x;
  if (c * 8 >= d) return;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  for (int at = first; at < T && sorted[at] == id; at += UNROLL) {
    uint4 v[UNROLL];
    bool mine[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      mine[u] = at + u < T && sorted[at + u] == id;
      v[u] = mine[u] ? __ldcs(reinterpret_cast<const uint4*>(dy + static_cast<long long>(place[at + u]) * d) + c) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      if (!mine[u]) break;
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) { acc[2 * i] += __uint_as_float(w[i] << 16); acc[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u); }
    }
  }
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
    o[i] = *reinterpret_cast<const uint32_t*>(&p);
  }
  reinterpret_cast<uint4*>(dw + static_cast<long long>(id) * d)[c] = make_uint4(o[0], o[1], o[2], o[3]);
}

}  // namespace embed
}  // namespace dewb

// Tokens it takes.
extern "C" int dewb_embed_grad_most() { return dewb::embed::MOST; }

// dy [T, d] bf16, ids [T] int64 in [0, V), both contiguous -> dw [V, d] bf16; scratch: 3 T int32.  d a multiple of 8, dy and dw on 16-byte boundaries, V below 2^31.
extern "C" int dewb_embed_grad(const void* dy, const long long* ids, void* dw, int* scratch, int T, int d, long long V, void* stream_ptr) {
  using namespace dewb::embed;
  if (T < 0 || T > MOST || d < 8 || d % 8 || V <= 0 || V > 0x7fffffff || d / 8 > 65535 * SUM_THREADS || ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dw)) & 15)) return -3;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  cudaError_t e = cudaMemsetAsync(dw, 0, static_cast<size_t>(V) * d * 2, stream);
  if (e != cudaSuccess || T == 0) return static_cast<int>(e);
  if ((e = cudaMemsetAsync(scratch, 0, static_cast<size_t>(T) * 4, stream)) != cudaSuccess) return static_cast<int>(e);
  const unsigned blocks = (T + RANK_THREADS - 1) / RANK_THREADS;
  int *sorted = scratch + T, *place = scratch + 2 * T;
  rank_kernel<<<dim3(blocks, (T + SLICE - 1) / SLICE), RANK_THREADS, 0, stream>>>(ids, scratch, T);
  order_kernel<<<blocks, RANK_THREADS, 0, stream>>>(ids, scratch, sorted, place, T);
  sum_kernel<<<dim3(T, (d / 8 + SUM_THREADS - 1) / SUM_THREADS), SUM_THREADS, 0, stream>>>(static_cast<const __nv_bfloat16*>(dy), sorted, place, static_cast<__nv_bfloat16*>(dw), T, d,
                                                                                           static_cast<int>(V));
  return static_cast<int>(cudaGetLastError());
}
