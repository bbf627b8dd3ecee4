// A decoder's layers for one token a row, issued in one call: norm, packed projection, rotation and append, paged attention, output projection, norm, gate and up,
// activation, down - nine launches a layer of the kernels that the layers' own operations launch one by one, with the same operands in the same order.
//
// What bounds a step of one to four rows of a small decoder is the host: a launch through the interpreter and a module takes 23 us, the kernels 2 to 13 (eight layers of
// width 1024, one row: 1719 us a step, 332 us of them on the GPU).  From here a launch takes some 2 us and the step 460, two thirds of it the GPU's.
#include <cuda_runtime.h>
#include <cstdint>

extern "C" {
int dewb_rmsnorm_fwd(const void* x, const void* other, const void* w, void* y, void* h_out, float* rstd, long long rows, int d, float eps, int mode, void* stream);
int dewb_gemm_rows_bf16(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, long long ldx, long long ldw, long long ldy, void* stream);
int dewb_rope_append(void* qkv, const float* cosb, const float* sinb, const int* positions, int rows, int Hq, int Hkv, int D, int table_rows, void* kpool, void* vpool,
                     const int* page_table, int page_size, int max_pages, void* stream);
int dewb_paged_decode_persist(const void* q, const void* kpool, const void* vpool, long long pool_tokens, const int* page_table, const int* lengths, float* part_m, float* part_l,
                              float* part_acc, unsigned int* arrivals, const float* sinks, void* out, int rows, int Hq, int Hkv, int page_size, int max_pages, int max_parts,
                              int min_tiles, float scale, int window, int keep, int chunk, float softcap, const float* gain, const float* sig, long long q_row_stride, int ctas,
                              int* err, void* stream);
int dewb_swiglu_fwd(const void* gate, const void* up, void* out, long long rows, int F, long long in_stride, void* stream);

// Weights [out, in] contiguous bf16, norms [width] bf16, the layer's pages of keys and values; sinks [heads] fp32 or null; window 0: none.
struct dewb_decode_layer {
  const void *in_norm, *qkv, *out, *post_norm, *gate_up, *down;
  void *keys, *values;
  const float* sinks;
  float in_eps, post_eps;
  int window, max_parts, ff;
};

// Of the call: the embedded rows [rows, width], two streams and a branch of that size for the results, and scratch: normed [rows, width], packed
// [rows, (heads + 2 kv_heads) dim], attended [rows, heads dim], gates [rows, 2 ff], active [rows, ff] (ff: the largest of the layers'), rstd [rows].
struct dewb_decode_call {
  const void* embedded;
  void *stream0, *stream1, *branch, *normed, *packed, *attended, *gates, *active;
  float* rstd;
  const float *cosb, *sinb;
  const int *positions, *lengths, *page_table;
  float *part_m, *part_l, *part_acc;
  unsigned int* arrivals;
  int* err;
  long long pool_tokens;
  float scale;
  int rows, width, heads, kv_heads, dim, table_rows, page_size, max_pages, min_tiles, ctas;
};

// -> stream0: the stream behind the last layer's second norm; branch: its down projection, not yet added.
int dewb_decode_step(const dewb_decode_layer* layers, int n, const dewb_decode_call* call, void* stream) {
  const dewb_decode_call& c = *call;
  if (n < 1 || c.rows < 1 || c.rows > 4) return -3;
  const int packed = (c.heads + 2 * c.kv_heads) * c.dim, attended = c.heads * c.dim;
  const void* h = c.embedded;
  void* next[2] = {c.stream0, c.stream1};
  int r, turn = 0;
  for (int i = 0; i < n; ++i) {
    const dewb_decode_layer& l = layers[i];
    if (i == 0) {
      if ((r = dewb_rmsnorm_fwd(h, nullptr, l.in_norm, c.normed, nullptr, c.rstd, c.rows, c.width, l.in_eps, 0, stream))) return r;
    } else {
      if ((r = dewb_rmsnorm_fwd(h, c.branch, l.in_norm, c.normed, next[turn], c.rstd, c.rows, c.width, l.in_eps, 1, stream))) return r;
      h = next[turn];
      turn ^= 1;
    }
    if ((r = dewb_gemm_rows_bf16(c.normed, l.qkv, nullptr, c.packed, c.rows, packed, c.width, c.width, c.width, packed, stream))) return r;
    if ((r = dewb_rope_append(c.packed, c.cosb, c.sinb, c.positions, c.rows, c.heads, c.kv_heads, c.dim, c.table_rows, l.keys, l.values, c.page_table, c.page_size, c.max_pages, stream)))
      return r;
    if ((r = dewb_paged_decode_persist(c.packed, l.keys, l.values, c.pool_tokens, c.page_table, c.lengths, c.part_m, c.part_l, c.part_acc, c.arrivals, l.sinks, c.attended, c.rows,
                                       c.heads, c.kv_heads, c.page_size, c.max_pages, l.max_parts, c.min_tiles, c.scale, l.window, 0, 0, 0.f, nullptr, nullptr, packed, c.ctas, c.err,
                                       stream)))
      return r;
    if ((r = dewb_gemm_rows_bf16(c.attended, l.out, nullptr, c.branch, c.rows, c.width, attended, attended, attended, c.width, stream))) return r;
    if ((r = dewb_rmsnorm_fwd(h, c.branch, l.post_norm, c.normed, next[turn], c.rstd, c.rows, c.width, l.post_eps, 1, stream))) return r;
    h = next[turn];
    turn ^= 1;
    if ((r = dewb_gemm_rows_bf16(c.normed, l.gate_up, nullptr, c.gates, c.rows, 2 * l.ff, c.width, c.width, c.width, 2 * l.ff, stream))) return r;
    if ((r = dewb_swiglu_fwd(c.gates, static_cast<const char*>(c.gates) + 2ll * l.ff, c.active, c.rows, l.ff, 2 * l.ff, stream))) return r;
    if ((r = dewb_gemm_rows_bf16(c.active, l.down, nullptr, c.branch, c.rows, c.width, l.ff, l.ff, l.ff, c.width, stream))) return r;
  }
  return 0;
}
}
