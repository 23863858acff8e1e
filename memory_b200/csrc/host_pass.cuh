// Host-side helpers of the files that issue a whole pass per call (layer.cu, cross_attn.cu): carving one buffer into
// typed pieces, ordering two streams, and the projections in the shapes those passes need.
#pragma once
#include <algorithm>

#include "moc_common.cuh"

namespace moc {

#define MOC_TRY(expr)                    \
  do {                                   \
    const int _rc = (expr);              \
    if (_rc != MOC_OK) return _rc;       \
  } while (0)

struct Carver {
  char* base;
  int64_t off;
  template <typename T> T* take(int64_t n) {
    T* r = reinterpret_cast<T*>(base + off);
    off += (n * static_cast<int64_t>(sizeof(T)) + 255) & ~int64_t(255);
    return r;
  }
  void* take_as(int dtype, int64_t n) {
    return dtype == MOC_F32 ? static_cast<void*>(take<float>(n)) : static_cast<void*>(take<__nv_bfloat16>(n));
  }
};

// Records an event on `from`.  A wait refers to the record before it, so a thread can use the same few events for every
// pass it issues; they belong to the device they were made on.
int fork_event(cudaStream_t from, cudaEvent_t* out);
// `after` continues behind what `before` holds now.
int order(cudaStream_t before, cudaStream_t after);

// A pass that forked `side` off `main` joins it again on every way out.  On an error too: the caller then gives the pass's
// buffers back, and their next use is ordered behind `main` alone.
struct Join {
  cudaStream_t side, main;
  bool open;
  Join(cudaStream_t side_, cudaStream_t main_) : side(side_), main(main_), open(side_ != main_) {}
  Join(const Join&) = delete;
  ~Join() { done(); }
  int done() {
    const bool was = open;
    open = false;
    return was ? order(side, main) : MOC_OK;
  }
};

// A projection of up to two rows (bf16, 16-byte rows, k <= 1,024) that a launch of the router can take along; n = 0: none
struct RowsProduct {
  const __nv_bfloat16 *a = nullptr, *w = nullptr;
  __nv_bfloat16* c = nullptr;
  long long lda = 0, ldb = 0, ldc = 0;
  int m = 0, n = 0, k = 0;
};
// What a router call did: whether the projection given along ran, and the kernels of pooling, logits and selection
struct RouteRun {
  bool q_done = false;
  int launches = 0;
};
// moc_router_fwd_parts / moc_route_fwd with one (q may be NULL), reporting to *run (may be NULL)
int router_fwd_parts_impl(const moc_router_shape* s, const void* h, const float* w, const float* bias, float* pooled, float* logits,
                          float* probs, int64_t* idx, float* weights, int32_t* comb_idx, float* comb_w, float* row_stats,
                          float* chapter_stats, float* losses, void* workspace, size_t workspace_bytes, int32_t parts,
                          const RowsProduct* q, RouteRun* run, int32_t* status, void* stream);
int route_fwd_impl(const moc_route_desc* s, const RowsProduct* q, RouteRun* run);

// What the bf16 projection kernel can do beside moc_gemm_desc:
// terms > 1: C = sum over t of op(A_t) op(B_t), all in one accumulator, the last term first; A_t / B_t start
//   t * a_term_rows / b_term_rows stored rows behind A / B (0: the same operand in every term).
// limit (device): only the first *limit * limit_block of the M rows (limit_k: of the K range, limit_block a multiple of 64)
//   exist; what lies behind is not read into a stored result nor, for M, defined in C.
// c_row_blocks (device): block i of c_block_rows (a multiple of 32) rows of C is stored as block c_row_blocks[i] of a matrix
//   of c_stored_rows rows.
struct GemmExtra {
  int terms = 1, a_term_rows = 0, b_term_rows = 0;
  int limit_block = 0, limit_k = 0, c_block_rows = 0;
  int64_t c_stored_rows = 0;
  const int32_t *limit = nullptr, *c_row_blocks = nullptr;
};
int launch_gemm_tc(const moc_gemm_desc* g, const void* a, const void* b, void* c, const float* row_scale,
                   const int32_t* a_row_blocks, int32_t* status, cudaStream_t stream,
                   const int32_t* b_row_blocks, int32_t b_block_rows, int64_t b_stored_rows, const GemmExtra* extra);

// C [m, n] = op(A) op(B), dense operands
struct Gemm : moc_gemm_desc {
  GemmExtra extra;
  Gemm(int dt, int64_t m_, int64_t n_, int64_t k_, bool a_k, bool b_k, int c_dt) {
    dtype = dt; c_dtype = c_dt;
    m = static_cast<int>(m_); n = static_cast<int>(n_); k = static_cast<int>(k_);
    a_kmajor = a_k; b_kmajor = b_k;
    lda = a_k ? k : m; ldb = b_k ? k : n; ldc = n;
    accumulate = 0; split_k = 1; scale_block_rows = 1; a_block_rows = 0;
    a_stored_rows = a_k ? m : k;
    residual = nullptr; ldr = 0;
  }
};
// with its extras (bf16 operands)
inline int gemm_extra(const Gemm& g, const void* a, const void* b, void* c, int32_t* status, cudaStream_t stream) {
  return launch_gemm_tc(&g, a, b, c, nullptr, nullptr, status, stream, nullptr, 0, 0, &g.extra);
}
// K-splits of a weight gradient [out_rows, out_cols] over `rows`: enough (tile, split) items to fill the SMs once
inline int splits(int64_t rows, int64_t out_rows, int64_t out_cols) {
  const int64_t tiles = ((out_rows + 127) / 128) * ((out_cols + 255) / 256);
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(148 / std::max<int64_t>(tiles, 1), rows / 512)));
}
// dW [m, n] fp32 = A^T B over `rows`
int weight_grad(int dtype, int64_t m, int64_t n, int64_t rows, const void* a, const void* b, float* out, int* status,
                void* stream);
// dst (dtype) = src (src_dtype); the source itself where the types agree
inline int as_dtype(const void* src, int src_dtype, void* dst, int dtype, int64_t n, void* stream, const void** out) {
  *out = src;
  if (src_dtype == dtype) return MOC_OK;
  *out = dst;
  return dtype == MOC_BF16 ? moc_cast_f32_to_bf16(static_cast<const float*>(src), dst, n, stream)
                           : moc_cast_bf16_to_f32(src, static_cast<float*>(dst), n, stream);
}

// moc_gather_rows_bwd / _prescaled; with `dense` the fp32 rows go to their places in a bank-shaped, cleared bank_grad
int gather_rows_bwd_impl(const void* d_mem, int32_t d_mem_dtype, const void* bank, int32_t bank_dtype, int64_t bank_rows, int32_t dim, int32_t T, const int32_t* comb_idx, const float* comb_w, int32_t batch, int32_t k_sel, int32_t norm_type, float eps, const float* row_stats, const int32_t* uniq, const int32_t* seg_offsets, const int32_t* seg_pairs, const int32_t* num_unique, float* d_comb_w, float* bank_grad, void* bank_grad_bf16, int32_t* status, void* stream_, int dense);
int gather_rows_bwd_prescaled_impl(const void* g, int32_t g_dtype, const void* bank, int32_t bank_dtype, int64_t bank_rows, int32_t dim, int32_t T, const int32_t* comb_idx, const float* comb_w, int32_t n_pairs, const float* inv_rms, const int32_t* uniq, const int32_t* seg_offsets, const int32_t* seg_pairs, const int32_t* num_unique, float* d_comb_w, float* bank_grad, void* bank_grad_bf16, int32_t* status, void* stream_, int dense);
// the bank-shaped gradient: cleared, then its touched rows written in place (no compact copy to scatter afterwards)
inline int clear_dense(float* dense, int64_t elems, cudaStream_t st) {
  MOC_CUDA_OK(cudaMemsetAsync(dense, 0, static_cast<size_t>(elems) * 4, st));
  return MOC_OK;
}

}  // namespace moc
