// Gradient of an embedding table: dw[v] = sum of dy[t] over the tokens t with ids[t] = v, fp32 sums in an order of the tokens' own, rounded to bf16 once.
//
// The table's gradient is written once (cleared, then the rows that occur) and dy read once, which is what bounds it; the sums need the places of equal ids side by
// side.  A token's place in that order is the number of tokens in front of it, by id and then by place: up to 16384 tokens these are counted outright, every token
// against every other (a compare and an add a pair, spread over all SMs, the counts of the slices joined by integer atomics), where the library's sort of any length is
// a chain of eight launches and a bitonic network in one block's shared memory took 93 us for 8192 tokens (13 counted).  A block per place and 1024 columns then
// sums the run that begins there, if one of up to 64 does.  Longer runs (the padding of packed batches, the ids of a byte vocabulary) have blocks of their own, 64 rows
// side by side for 16 columns each: a block that took all rows of a run, four a turn, waited 1.3 us for every turn.  8192 tokens of 2048 features: ids of 32768 that
// differ, 450 us for the library's backward, 69 for this; half of them one id, 373 and 72 (1371 by one block a run).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dewb {
namespace embed {

constexpr int MOST = 16384;                            // tokens: the work grows with their square
constexpr int RANK_THREADS = 256, SLICE = 1024;
constexpr int SUM_THREADS = 128, UNROLL = 4;
constexpr int LONG = 64;                               // places of a run that sum_run takes
constexpr int LONG_COLS = 16, LONG_ROWS = SUM_THREADS / (LONG_COLS / 8), LONG_BLOCKS = 4 * 148;

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
  // equal ids count where their place is in front: up to `near` all do, in the piece of four there some, behind it none
  const int own = min(max(i - first, 0), SLICE), near = own & ~3;
#pragma unroll 8
  for (int j = 0; j < near; j += 4) {
    const int4 o = *reinterpret_cast<const int4*>(other + j);
    count += (o.x <= mine) + (o.y <= mine) + (o.z <= mine) + (o.w <= mine);
  }
#pragma unroll 8
  for (int j = near; j < SLICE; j += 4) {
    const int4 o = *reinterpret_cast<const int4*>(other + j);
    count += (o.x < mine) + (o.y < mine) + (o.z < mine) + (o.w < mine);
  }
  for (int j = near; j < own; ++j) count += other[j] == mine;
  if (count) atomicAdd(rank + i, count);
}

__global__ void __launch_bounds__(RANK_THREADS)
order_kernel(const long long* __restrict__ ids, const int* __restrict__ rank, int* __restrict__ sorted, int* __restrict__ place, int T) {
  const int i = blockIdx.x * RANK_THREADS + threadIdx.x;
  if (i >= T) return;
  sorted[rank[i]] = static_cast<int>(ids[i]);
  place[rank[i]] = i;
}

// The run that begins at place `first`, if one of up to LONG does: eight columns from 8 c on.
__device__ __forceinline__ void sum_run(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ sorted, const int* __restrict__ place, __nv_bfloat16* __restrict__ dw, int T, int d,
                                        int V, int first, int c) {
  // (what decides, and where the first rows are, is asked for at once: a place is one of a thousand waits on its SM)
  const int id = sorted[first], before = first > 0 ? sorted[first - 1] : -1, far = first + LONG < T ? sorted[first + LONG] : -1;
  int row[UNROLL], same[UNROLL];
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    const int p = min(first + u, T - 1);
    row[u] = place[p];
    same[u] = sorted[p];
  }
  if (static_cast<unsigned>(id) >= static_cast<unsigned>(V)) return;      // (the forward's lookup reports those)
  if (before == id || far == id || c * 8 >= d) return;                    // (a run of more than LONG: sum_long_runs)
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  for (int at = first;;) {
    uint4 v[UNROLL];
    bool mine[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      mine[u] = at + u < T && same[u] == id;
      v[u] = mine[u] ? __ldcs(reinterpret_cast<const uint4*>(dy + static_cast<long long>(row[u]) * d) + c) : make_uint4(0u, 0u, 0u, 0u);
    }
    at += UNROLL;
    const bool more = mine[UNROLL - 1] && at < T;
    if (more) {
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int p = min(at + u, T - 1);
        row[u] = place[p];
        same[u] = sorted[p];
      }
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      if (!mine[u]) break;
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) { acc[2 * i] += __uint_as_float(w[i] << 16); acc[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u); }
    }
    if (!more) break;
  }
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
    o[i] = *reinterpret_cast<const uint32_t*>(&p);
  }
  reinterpret_cast<uint4*>(dw + static_cast<long long>(id) * d)[c] = make_uint4(o[0], o[1], o[2], o[3]);
}

// Runs of more than LONG places.  Each has a place that is a multiple of LONG, and the first such place is followed by one more of the run: each of the LONG_BLOCKS
// blocks finds all of them by these, in order, and takes its share of (run, LONG_COLS columns).  A row group sums every LONG_ROWS-th row, then the groups are added in order.
__device__ __forceinline__ void sum_long_runs(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ sorted, const int* __restrict__ place, __nv_bfloat16* __restrict__ dw, int T,
                                              int d, int V) {
  constexpr int SLOTS = MOST / LONG, TURNS = SLOTS / SUM_THREADS;
  static_assert(SLOTS % SUM_THREADS == 0, "a thread finds runs at SLOTS / SUM_THREADS slots");
  __shared__ int slot_id[SLOTS], run_from[SLOTS], run_to[SLOTS], found[SLOTS / 32];
  __shared__ float part[LONG_ROWS][LONG_COLS];
  const int tid = threadIdx.x, lane = tid & 31, slots = (T + LONG - 1) / LONG;
#pragma unroll
  for (int k = 0; k < TURNS; ++k) { const int s = k * SUM_THREADS + tid; if (s < slots) slot_id[s] = sorted[s * LONG]; }
  __syncthreads();
  int from[TURNS], to[TURNS];
  unsigned votes[TURNS];
#pragma unroll
  for (int k = 0; k < TURNS; ++k) {
    const int s = k * SUM_THREADS + tid;
    bool mine = false;
    from[k] = to[k] = 0;
    if (s < slots) {
      const int id = slot_id[s], p = s * LONG;
      if (static_cast<unsigned>(id) < static_cast<unsigned>(V) && (s == 0 || slot_id[s - 1] != id) && p + 1 < T && sorted[p + 1] == id) {
        int lo = s == 0 ? -1 : p - LONG, hi = p;                             // sorted[lo] != id (or in front of all), sorted[hi] == id
        while (hi - lo > 1) { const int m = (lo + hi) / 2; if (sorted[m] == id) hi = m; else lo = m; }
        from[k] = hi;
        mine = hi + LONG < T && sorted[hi + LONG] == id;
        if (mine) {
          int last = s, past = slots;                                        // slot_id[last] == id, slot_id[past] != id (or behind all)
          while (past - last > 1) { const int m = (last + past) / 2; if (slot_id[m] == id) last = m; else past = m; }
          lo = last * LONG;
          hi = min(lo + LONG, T);                                            // sorted[lo] == id, sorted[hi] != id (or behind all)
          while (hi - lo > 1) { const int m = (lo + hi) / 2; if (sorted[m] == id) lo = m; else hi = m; }
          to[k] = hi;
        }
      }
    }
    votes[k] = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) found[s / 32] = __popc(votes[k]);
  }
  __syncthreads();
  int runs = 0, before[TURNS] = {};
  for (int w = 0; w < SLOTS / 32; ++w) {
#pragma unroll
    for (int k = 0; k < TURNS; ++k) if (w < (k * SUM_THREADS + tid) / 32) before[k] += found[w];
    runs += found[w];
  }
#pragma unroll
  for (int k = 0; k < TURNS; ++k)
    if (votes[k] >> lane & 1) {
      const int at = before[k] + __popc(votes[k] & ((1u << lane) - 1));
      run_from[at] = from[k];
      run_to[at] = to[k];
    }
  __syncthreads();
  const int chunks = (d + LONG_COLS - 1) / LONG_COLS, sub = tid % (LONG_COLS / 8), group = tid / (LONG_COLS / 8);
  for (int item = blockIdx.x; item < runs * chunks; item += LONG_BLOCKS) {
    const int run = item / chunks, c0 = item % chunks * LONG_COLS, c = c0 + sub * 8, end = run_to[run];
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    if (c < d) {
      for (int at = run_from[run] + group; at < end; at += LONG_ROWS * UNROLL) {
        uint4 v[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          const int p = at + u * LONG_ROWS;
          v[u] = p < end ? *reinterpret_cast<const uint4*>(dy + static_cast<long long>(place[p]) * d + c) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) { acc[2 * i] += __uint_as_float(w[i] << 16); acc[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u); }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) part[group][sub * 8 + i] = acc[i];
    __syncthreads();
    // eight threads a column: eight groups each, then theirs
    const int column = tid % LONG_COLS, eighth = tid / LONG_COLS;
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < LONG_ROWS / 8; ++i) sum += part[eighth * (LONG_ROWS / 8) + i][column];
    __syncthreads();
    part[eighth][column] = sum;
    __syncthreads();
    if (tid < LONG_COLS && c0 + tid < d) {
      float all = part[0][tid];
#pragma unroll
      for (int i = 1; i < 8; ++i) all += part[i][tid];
      dw[static_cast<long long>(sorted[run_from[run]]) * d + c0 + tid] = __float2bfloat16(all);
    }
    __syncthreads();
  }
}

// The first `long_blocks` blocks (LONG_BLOCKS or none) take the long runs, the others a place and 8 SUM_THREADS columns each: one launch, since most batches have no long runs
// and the look for them is 4 us that others can work in.
__global__ void __launch_bounds__(SUM_THREADS, 10)
sum_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ sorted, const int* __restrict__ place, __nv_bfloat16* __restrict__ dw, int T, int d, int V, int long_blocks) {
  const int block = static_cast<int>(blockIdx.x) - long_blocks;
  if (block < 0) {
    sum_long_runs(dy, sorted, place, dw, T, d, V);
  } else {
    sum_run(dy, sorted, place, dw, T, d, V, block % T, block / T * SUM_THREADS + threadIdx.x);
  }
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
  const int long_blocks = T > LONG ? LONG_BLOCKS : 0, across = (d / 8 + SUM_THREADS - 1) / SUM_THREADS;
  sum_kernel<<<static_cast<unsigned>(long_blocks + static_cast<long long>(T) * across), SUM_THREADS, 0, stream>>>(static_cast<const __nv_bfloat16*>(dy), sorted, place,
                                                                                                               static_cast<__nv_bfloat16*>(dw), T, d, static_cast<int>(V), long_blocks);
  return static_cast<int>(cudaGetLastError());
}
