// Modulated layer norms of diffusion transformers and the gated residuals between them (bf16 tokens [B, n, d], one shift, scale and gate of width d per image):
//     h = x + gate o branch            y = (h - mean(h)) rstd(h) o (1 + scale) + shift
// in one pass each way, either half alone as well; and the fixed sine-cosine table of a patch grid.
//
// All bound by memory: forward reads x and branch and writes h and y (25 MB apiece at 64 x 256 x 768), backward reads h, branch and the gradients of both outputs and
// writes those of x and branch.  A warp holds a row in registers (d / 256 pieces of eight columns a lane); the sums over an image's tokens that make the gradients of
// shift, scale and gate stay in shared memory, one set per warp, since a lane adds to the same columns for every row: 144 cycles of shared memory a row against some
// 400 of its traffic.  A block takes a slab of one image's tokens and leaves one partial sum per column, which a last small kernel adds in order.
// As separate PyTorch operations, which round to bf16 between any two, norm, modulation, gate and residual took about 4 ms of a four-layer
// training step at that size; these take 0.17 forward and 0.48 backward.
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace dewb {
namespace ada {

typedef __nv_bfloat16 bf16;
constexpr uint32_t FULL = 0xffffffffu;
constexpr int MAX_D = 2048;

__device__ __forceinline__ float lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void unpack(const uint4& v, float (&f)[8]) {
  f[0] = lo(v.x); f[1] = hi(v.x); f[2] = lo(v.y); f[3] = hi(v.y); f[4] = lo(v.z); f[5] = hi(v.z); f[6] = lo(v.w); f[7] = hi(v.w);
}
__device__ __forceinline__ uint4 packed(const float (&f)[8]) { return make_uint4(pack(f[0], f[1]), pack(f[2], f[3]), pack(f[4], f[5]), pack(f[6], f[7])); }
__device__ __forceinline__ uint4 piece(const bf16* row, int at) { return reinterpret_cast<const uint4*>(row)[at]; }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}

// rows of the modulation (shift, scale, gate): one per image, `mod_stride` elements apart
struct Mod {
  const bf16 *shift, *scale, *gate;
  long long stride;
};

template <int NV, bool BRANCH, bool NORM>
__global__ void __launch_bounds__(256)
ada_fwd(const bf16* __restrict__ x, const bf16* __restrict__ branch, Mod mod, bf16* __restrict__ h_out, bf16* __restrict__ y, float2* __restrict__ stats, long long rows, int n,
        int d, float eps) {
  const int lane = threadIdx.x & 31, pieces = d / 8;
  const long long row = blockIdx.x * 8ll + (threadIdx.x >> 5);
  if (row >= rows) return;
  const long long image = row / n;
  float h[NV][8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int at = i * 32 + lane;
    if (at < pieces) {
      unpack(piece(x + row * d, at), h[i]);
      if (BRANCH) {
        float b[8], g[8];
        unpack(piece(branch + row * d, at), b);
        unpack(piece(mod.gate + image * mod.stride, at), g);
#pragma unroll
        for (int c = 0; c < 8; ++c) h[i][c] = fmaf(g[c], b[c], h[i][c]);
        const uint4 r = packed(h[i]);
        reinterpret_cast<uint4*>(h_out + row * d)[at] = r;
        unpack(r, h[i]);                               // what is normalised is what the stream carries on
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) sum += h[i][c];
    } else {
#pragma unroll
      for (int c = 0; c < 8; ++c) h[i][c] = 0.f;
    }
  }
  if constexpr (NORM) {
    const float mean = warp_sum(sum) / d;
    float var = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (i * 32 + lane < pieces) {
#pragma unroll
        for (int c = 0; c < 8; ++c) var += (h[i][c] - mean) * (h[i][c] - mean);
      }
    const float rstd = rsqrtf(warp_sum(var) / d + eps);
    if (lane == 0) stats[row] = make_float2(mean, rstd);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int at = i * 32 + lane;
      if (at >= pieces) continue;
      float s[8], t[8];
      unpack(piece(mod.scale + image * mod.stride, at), s);
      unpack(piece(mod.shift + image * mod.stride, at), t);
#pragma unroll
      for (int c = 0; c < 8; ++c) t[c] = fmaf((h[i][c] - mean) * rstd, 1.f + s[c], t[c]);
      reinterpret_cast<uint4*>(y + row * d)[at] = packed(t);
    }
  }
}

// dy: gradient of y (NORM); dh_in: gradient of h from elsewhere (may be null with NORM).  part [B, slabs, 3, d]: sums of shift's, scale's and gate's gradients.
template <int NV, bool BRANCH, bool NORM>
__global__ void __launch_bounds__(256)
ada_bwd(const bf16* __restrict__ dy, const bf16* __restrict__ dh_in, const bf16* __restrict__ h_in, const bf16* __restrict__ branch, Mod mod,
        const float2* __restrict__ stats, bf16* __restrict__ dx, bf16* __restrict__ dbranch, float* __restrict__ part, int n, int d, int slab) {
  extern __shared__ float sums[];                      // [warps][2 (NORM) + 1 (BRANCH)][d]
  constexpr int SETS = (NORM ? 2 : 0) + (BRANCH ? 1 : 0), GATE = NORM ? 2 : 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, pieces = d / 8;
  const long long image = blockIdx.y;
  for (int i = threadIdx.x; i < warps * SETS * d; i += blockDim.x) sums[i] = 0.f;
  __syncthreads();
  float* mine = sums + warp * SETS * d;
  const int end = min(n, (static_cast<int>(blockIdx.x) + 1) * slab);
  for (int t = blockIdx.x * slab + warp; t < end; t += warps) {
    const long long row = image * n + t;
    float g[NV][8];                                    // the gradient of h
    if constexpr (NORM) {
      const float2 st = stats[row];
      float xh[NV][8], a = 0.f, b = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int at = i * 32 + lane;
        if (at < pieces) {
          float v[8], s[8];
          unpack(piece(h_in + row * d, at), xh[i]);
          unpack(piece(dy + row * d, at), v);
          unpack(piece(mod.scale + image * mod.stride, at), s);
          float4* shift = reinterpret_cast<float4*>(mine + at * 8);
          float4* scale = reinterpret_cast<float4*>(mine + d + at * 8);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float4 u = shift[q], w = scale[q];
            float* up = &u.x;
            float* wp = &w.x;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const int e = q * 4 + c;
              xh[i][e] = (xh[i][e] - st.x) * st.y;
              up[c] += v[e];
              wp[c] = fmaf(v[e], xh[i][e], wp[c]);
              g[i][e] = v[e] * (1.f + s[e]);
              a += g[i][e];
              b = fmaf(g[i][e], xh[i][e], b);
            }
            shift[q] = u;
            scale[q] = w;
          }
        }
      }
      a = warp_sum(a) / d;
      b = warp_sum(b) / d;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int at = i * 32 + lane;
        if (at >= pieces) continue;
        float v[8];
        if (dh_in != nullptr) unpack(piece(dh_in + row * d, at), v);
#pragma unroll
        for (int c = 0; c < 8; ++c) g[i][c] = st.y * (g[i][c] - a - xh[i][c] * b) + (dh_in != nullptr ? v[c] : 0.f);
      }
    } else {
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (i * 32 + lane < pieces) unpack(piece(dh_in + row * d, i * 32 + lane), g[i]);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int at = i * 32 + lane;
      if (at >= pieces) continue;
      if (NORM) reinterpret_cast<uint4*>(dx + row * d)[at] = packed(g[i]);
      if (BRANCH) {
        float b[8], w[8];
        unpack(piece(branch + row * d, at), b);
        unpack(piece(mod.gate + image * mod.stride, at), w);
        float4* gate = reinterpret_cast<float4*>(mine + GATE * d + at * 8);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float4 u = gate[q];
          u.x = fmaf(g[i][q * 4], b[q * 4], u.x); u.y = fmaf(g[i][q * 4 + 1], b[q * 4 + 1], u.y);
          u.z = fmaf(g[i][q * 4 + 2], b[q * 4 + 2], u.z); u.w = fmaf(g[i][q * 4 + 3], b[q * 4 + 3], u.w);
          gate[q] = u;
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) w[c] *= g[i][c];
        reinterpret_cast<uint4*>(dbranch + row * d)[at] = packed(w);
      }
    }
  }
  __syncthreads();
  float* to = part + (image * gridDim.x + blockIdx.x) * SETS * d;
  for (int i = threadIdx.x; i < SETS * d; i += blockDim.x) {
    float s = 0.f;
    for (int w = 0; w < warps; ++w) s += sums[w * SETS * d + i];
    to[i] = s;
  }
}

// part [B, slabs, sets, d] -> out [B, sets, d] bf16
__global__ void __launch_bounds__(256)
ada_sums(const float* __restrict__ part, bf16* __restrict__ out, int B, int slabs, int per) {        // per = sets * d
  const long long i = blockIdx.x * 256ll + threadIdx.x;
  if (i >= static_cast<long long>(B) * per) return;
  const long long image = i / per, at = i % per;
  float s = 0.f;
  for (int k = 0; k < slabs; ++k) s += part[(image * slabs + k) * per + at];
  out[i] = __float2bfloat16(s);
}

__global__ void __launch_bounds__(256)
sincos_grid(bf16* __restrict__ out, int h, int w, int d) {
  const int i = blockIdx.x * 256 + threadIdx.x, half = d / 2, quarter = half / 2;
  if (i >= h * w * d) return;
  const int c = i % d, cell = i / d, pos = c < half ? cell / w : cell % w, k = c % half;
  const float omega = 1.f / powf(10000.f, static_cast<float>(k < quarter ? k : k - quarter) / static_cast<float>(quarter)), angle = static_cast<float>(pos) * omega;
  out[i] = __float2bfloat16(k < quarter ? sinf(angle) : cosf(angle));
}

// out [B, d]: cosines, then sines, of t scale max_period^(-k / half); an odd last column is 0.  One launch of two microseconds for what took eleven of elementwise
// operations: a sampler's denoising call on a few images is bound by the launches' issue (four images, four layers: 1794 us, with this and one silu of the conditioning
// for all blocks 1522).
template <typename Out>
__global__ void __launch_bounds__(256)
time_features(const float* __restrict__ t, Out* __restrict__ out, int B, int d, float minus_log_period, float scale) {
  const int i = blockIdx.x * 256 + threadIdx.x, half = d / 2;
  if (i >= B * d) return;
  const int row = i / d, c = i % d, k = c < half ? c : c - half;
  // (rounded where the operations one by one round)
  const float freq = expf(__fdiv_rn(__fmul_rn(minus_log_period, static_cast<float>(k)), static_cast<float>(half))), angle = __fmul_rn(__fmul_rn(t[row], scale), freq);
  const float v = c >= 2 * half ? 0.f : c < half ? cosf(angle) : sinf(angle);
  if constexpr (sizeof(Out) == 2) out[i] = __float2bfloat16(v); else out[i] = v;
}

template <int NV>
static int fwd(const bf16* x, const bf16* branch, const Mod& mod, bf16* h, bf16* y, float2* stats, long long rows, int n, int d, float eps, cudaStream_t s) {
  const unsigned blocks = static_cast<unsigned>((rows + 7) / 8);
  const bool norm = y != nullptr;
  if (branch != nullptr && norm) ada_fwd<NV, true, true><<<blocks, 256, 0, s>>>(x, branch, mod, h, y, stats, rows, n, d, eps);
  else if (norm) ada_fwd<NV, false, true><<<blocks, 256, 0, s>>>(x, branch, mod, h, y, stats, rows, n, d, eps);
  else ada_fwd<NV, true, false><<<blocks, 256, 0, s>>>(x, branch, mod, h, y, stats, rows, n, d, eps);
  return static_cast<int>(cudaGetLastError());
}

template <int NV, bool BRANCH, bool NORM>
static int bwd(const bf16* dy, const bf16* dh, const bf16* h, const bf16* branch, const Mod& mod, const float2* stats, bf16* dx, bf16* dbranch, float* part, bf16* dmod, int B, int n,
               int d, int slab, cudaStream_t s) {
  constexpr int sets = (NORM ? 2 : 0) + (BRANCH ? 1 : 0);
  const int warps = d <= 1024 ? 8 : 4, bytes = warps * sets * d * 4, slabs = (n + slab - 1) / slab;
  auto fn = ada_bwd<NV, BRANCH, NORM>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return static_cast<int>(e);
  fn<<<dim3(slabs, B), warps * 32, bytes, s>>>(dy, dh, h, branch, mod, stats, dx, dbranch, part, n, d, slab);
  if ((e = cudaGetLastError()) != cudaSuccess) return static_cast<int>(e);
  const long long total = static_cast<long long>(B) * sets * d;
  ada_sums<<<static_cast<unsigned>((total + 255) / 256), 256, 0, s>>>(part, dmod, B, slabs, sets * d);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ada
}  // namespace dewb

#define ADA_WIDTHS(GO) (d <= 256 ? GO(1) : d <= 512 ? GO(2) : d <= 768 ? GO(3) : d <= 1024 ? GO(4) : d <= 1536 ? GO(6) : GO(8))

// x, branch, h, y [rows, d] bf16 contiguous, rows = B * n; shift, scale, gate: the first of B rows `mod_stride` elements apart; everything 16-byte aligned, d and
// mod_stride multiples of 8, d <= 2048.  branch null: no gated residual (h is x and not written); y null: no norm.  stats [rows] (mean, 1 / deviation).
extern "C" int dewb_ada_fwd(const void* x, const void* branch, const void* shift, const void* scale, const void* gate, long long mod_stride, void* h, void* y, void* stats,
                            long long rows, int n, int d, float eps, void* stream) {
  using namespace dewb::ada;
  if (d % 8 || d <= 0 || d > MAX_D || mod_stride % 8 || n <= 0 || (branch == nullptr && y == nullptr)) return -3;
  if (rows <= 0) return 0;
  const Mod mod{static_cast<const bf16*>(shift), static_cast<const bf16*>(scale), static_cast<const bf16*>(gate), mod_stride};
#define ADA_GO(NV) fwd<NV>(static_cast<const bf16*>(x), static_cast<const bf16*>(branch), mod, static_cast<bf16*>(h), static_cast<bf16*>(y), static_cast<float2*>(stats), rows, n, d, eps, \
                           reinterpret_cast<cudaStream_t>(stream))
  return ADA_WIDTHS(ADA_GO);
#undef ADA_GO
}

// Tokens of an image that one block of the backward takes (the slabs of `part`): about two blocks an SM, at least a row for every warp.
extern "C" int dewb_ada_slab(int B, int n) {
  int slab = n;
  while (slab > 8 && static_cast<long long>(B) * ((n + slab - 1) / slab) < 2 * 148) slab = slab > 15 ? (slab + 1) / 2 : 8;      // (never below 8: 9 tokens are one block of eight rows and one of one, not five and four)
  return slab;
}

// Gradients of dewb_ada_fwd: dy of y (null: no norm), dh of h (null only with a norm); h as the forward normalised it (x where there was no branch).  dx is written
// with a norm alone (without one it is dh), dbranch with a branch.  part: fp32 scratch [B, slabs, sets, d], dmod [B, sets, d] bf16 with the sets shift, scale (with a
// norm) and gate (with a branch).
extern "C" int dewb_ada_bwd(const void* dy, const void* dh, const void* h, const void* branch, const void* scale, const void* gate, long long mod_stride, const void* stats,
                            void* dx, void* dbranch, float* part, void* dmod, int B, int n, int d, int slab, void* stream) {
  using namespace dewb::ada;
  if (d % 8 || d <= 0 || d > MAX_D || mod_stride % 8 || n <= 0 || slab <= 0 || B > 65535 || (branch == nullptr && dy == nullptr) || (dy == nullptr && dh == nullptr)) return -3;
  if (B <= 0) return 0;
  const Mod mod{nullptr, static_cast<const bf16*>(scale), static_cast<const bf16*>(gate), mod_stride};
#define ADA_ARGS static_cast<const bf16*>(dy), static_cast<const bf16*>(dh), static_cast<const bf16*>(h), static_cast<const bf16*>(branch), mod, static_cast<const float2*>(stats), \
                 static_cast<bf16*>(dx), static_cast<bf16*>(dbranch), part, static_cast<bf16*>(dmod), B, n, d, slab, reinterpret_cast<cudaStream_t>(stream)
#define ADA_BOTH(NV) bwd<NV, true, true>(ADA_ARGS)
#define ADA_NORM(NV) bwd<NV, false, true>(ADA_ARGS)
#define ADA_GATE(NV) bwd<NV, true, false>(ADA_ARGS)
  if (branch != nullptr && dy != nullptr) return ADA_WIDTHS(ADA_BOTH);
  if (dy != nullptr) return ADA_WIDTHS(ADA_NORM);
  return ADA_WIDTHS(ADA_GATE);
}

// t [B] fp32 -> out [B, d], bf16 or fp32: see time_features.  d of 2 and more.
extern "C" int dewb_time_features(const float* t, void* out, int out_bf16, int B, int d, float minus_log_period, float scale, void* stream) {
  using namespace dewb::ada;
  if (B < 0 || d < 2 || static_cast<long long>(B) * d > 0x7fffffffll - 256) return -3;
  if (B == 0) return 0;
  const unsigned blocks = (static_cast<unsigned>(B) * d + 255) / 256;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (out_bf16) time_features<<<blocks, 256, 0, s>>>(t, static_cast<bf16*>(out), B, d, minus_log_period, scale);
  else time_features<<<blocks, 256, 0, s>>>(t, static_cast<float*>(out), B, d, minus_log_period, scale);
  return static_cast<int>(cudaGetLastError());
}

// out [h * w, d] bf16: sines then cosines of the row in the first half of the columns, of the column in the second; d a multiple of 4.
extern "C" int dewb_sincos_grid(void* out, int h, int w, int d, void* stream) {
  using namespace dewb::ada;
  if (d % 4 || d <= 0 || h <= 0 || w <= 0 || static_cast<long long>(h) * w * d > 0x7fffffffll - 256) return -3;
  sincos_grid<<<(h * w * d + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(static_cast<bf16*>(out), h, w, d);
  return static_cast<int>(cudaGetLastError());
}
