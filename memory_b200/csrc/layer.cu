// One memory layer per call: the host code that issues the kernels of a whole forward or backward pass on two streams.
//
// Issued one operator at a time from Python, a training step of this layer is 38 launches at 25 to 45 us of host time
// each (tensor allocation, argument conversion, stream look-ups): 1.15 ms for a step whose kernels take 0.36 ms on one
// 320-token sequence, 0.43 ms for a forward whose kernels take 0.18 ms.  Here a pass is one call with one arena.
#include "host_pass.cuh"

namespace moc {
namespace {

// d_comb_w[b, i] = sum over KV heads of kv_dot[b, i, :] / max(comb_w, 1e-30) (+ g): the chapter-weight gradient from the
// per-chapter sums that the dK/dV kernel leaves
__global__ void comb_w_grad_kernel(const float* __restrict__ kv_dot, const float* __restrict__ comb_w,
                                   const float* __restrict__ g, float* __restrict__ out, int n, int HK) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
  for (int h = 0; h < HK; ++h) s += kv_dot[static_cast<long long>(i) * HK + h];
  s /= fmaxf(comb_w[i], 1e-30f);
  out[i] = g != nullptr ? s + g[i] : s;
}
__global__ void add_kernel(float* __restrict__ a, const float* __restrict__ b, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] += b[i];
}

struct Dims {
  int64_t rows, n_sel, sel_rows, pairs, d, dkv, rd;   // rd: width of the router's states
  int k_sel;
};
Dims dims_of(const moc_layer_desc* s) {
  Dims x;
  x.k_sel = std::max(0, std::min(s->top_k, s->num_chapters - s->num_shared));
  x.d = s->hidden_dim;
  x.rd = s->router_dim ? s->router_dim : s->hidden_dim;
  x.dkv = static_cast<int64_t>(s->num_kv_heads) * (s->hidden_dim / s->num_heads);
  x.rows = static_cast<int64_t>(s->batch) * s->seq;
  x.pairs = static_cast<int64_t>(s->batch) * (s->num_shared + x.k_sel);
  x.n_sel = static_cast<int64_t>(s->num_shared + x.k_sel) * s->tokens_per_chapter;
  x.sel_rows = s->batch * x.n_sel;
  return x;
}
moc_router_shape router_shape(const moc_layer_desc* s) {
  return {s->batch, s->router_seq, s->router_dim ? s->router_dim : s->hidden_dim, s->num_chapters, s->top_k, s->num_shared, s->routed_scale, s->router_dtype};
}

// what the forward pass leaves for the backward pass
struct Saved {
  float *pooled, *logits, *probs, *row_stats, *chapter_stats;
  char* router_ws;
  int *seg_off, *seg_pairs, *pair_to_uniq;
  __nv_bfloat16 *w_all, *wq, *wkv, *wo, *wq_t, *wkv_t, *wo_t;
  float* x2;              // the attention input in fp32, where it is needed and the input is not fp32 itself
  __nv_bfloat16* h2;      // the projection operand, where it is not the input itself
  float* stats_n;
  __nv_bfloat16 *q, *kv, *o, *m2;
  float *lse, *row_scale, *stats_m;
};
int64_t carve(const moc_layer_desc* s, const Dims& x, void* arena, Saved* a) {
  Carver c{static_cast<char*>(arena), 0};
  const moc_router_shape rs = router_shape(s);
  const int64_t B = s->batch, C = s->num_chapters;
  a->pooled = c.take<float>(B * x.rd); a->logits = c.take<float>(B * C); a->probs = c.take<float>(B * C);
  a->row_stats = c.take<float>(B * 4); a->chapter_stats = c.take<float>(2 * C);
  a->router_ws = c.take<char>(static_cast<int64_t>(moc_router_workspace_bytes(&rs)));
  a->seg_off = c.take<int>(x.pairs + 1); a->seg_pairs = c.take<int>(x.pairs); a->pair_to_uniq = c.take<int>(x.pairs);
  a->w_all = c.take<__nv_bfloat16>((2 * x.d + 2 * x.dkv) * x.d);
  a->wq = a->w_all; a->wkv = a->w_all + x.d * x.d; a->wo = a->wkv + 2 * x.dkv * x.d;
  a->wq_t = a->wkv_t = a->wo_t = nullptr;
  if (s->for_backward) {
    a->wq_t = c.take<__nv_bfloat16>(x.d * x.d); a->wkv_t = c.take<__nv_bfloat16>(2 * x.dkv * x.d);
    a->wo_t = c.take<__nv_bfloat16>(x.d * x.d);
  }
  const bool f32 = s->attn_dtype == MOC_F32, norm = s->pre_norm != MOC_NORM_NONE;
  a->x2 = (norm || s->add_residual) && !f32 ? c.take<float>(x.rows * x.d) : nullptr;
  a->h2 = norm || f32 ? c.take<__nv_bfloat16>(x.rows * x.d) : nullptr;
  a->stats_n = norm ? c.take<float>(2 * x.rows) : nullptr;
  a->q = c.take<__nv_bfloat16>(x.rows * x.d); a->kv = c.take<__nv_bfloat16>(x.sel_rows * 2 * x.dkv);
  a->o = c.take<__nv_bfloat16>(x.rows * x.d); a->lse = c.take<float>(x.rows * s->num_heads);
  a->row_scale = s->fused ? c.take<float>(x.sel_rows) : nullptr;
  a->m2 = s->fused ? nullptr : c.take<__nv_bfloat16>(x.sel_rows * x.d);
  a->stats_m = !s->fused && s->row_norm != MOC_NORM_NONE ? c.take<float>(2 * x.sel_rows) : nullptr;
  return c.off;
}

int check(const moc_layer_desc* s) {
  MOC_REQUIRE(s != nullptr, "layer descriptor is NULL");
  MOC_REQUIRE(s->batch > 0 && s->seq > 0 && s->hidden_dim > 0 && s->num_heads > 0 && s->num_kv_heads > 0 &&
                  s->tokens_per_chapter > 0 && s->num_chapters > 0 && s->bank_rows >= s->tokens_per_chapter, "empty layer problem");
  MOC_REQUIRE(s->hidden_dim % s->num_heads == 0, "hidden_dim must be divisible by num_heads");
  MOC_REQUIRE(s->router_dim >= 0, "bad router_dim");
  MOC_REQUIRE(s->attn_dtype == MOC_F32 || s->attn_dtype == MOC_BF16, "bad attn_dtype");
  MOC_REQUIRE(!s->fused || (s->bank_shadow && (s->row_norm == MOC_NORM_NONE ||
                                               (s->row_norm == MOC_NORM_RMS && s->bank_inv_rms))),
              "the fused gather needs the bf16 bank and, with RMS rows, their 1/rms");
  MOC_REQUIRE(s->pre_norm == MOC_NORM_NONE || s->norm_w, "pre_norm needs norm_w");
  MOC_REQUIRE(s->num_shared + std::min(s->top_k, s->num_chapters - s->num_shared) > 0, "no chapter is selected");
  return MOC_OK;
}

}  // namespace

struct EventRing {
  static constexpr int kMax = 16;
  cudaEvent_t ev[kMax];
  bool made = false;
  int next = 0;
  ~EventRing() {                 // a thread that ends gives its events back
    if (made)
      for (cudaEvent_t e : ev) cudaEventDestroy(e);
  }
};
int fork_event(cudaStream_t from, cudaEvent_t* out) {
  thread_local EventRing ring[16];
  int dev = 0;
  MOC_CUDA_OK(cudaGetDevice(&dev));
  MOC_REQUIRE(dev >= 0 && dev < 16, "device index out of range");
  EventRing& r = ring[dev];
  if (!r.made) {
    for (int i = 0; i < EventRing::kMax; ++i) MOC_CUDA_OK(cudaEventCreateWithFlags(&r.ev[i], cudaEventDisableTiming));
    r.made = true;
  }
  *out = r.ev[r.next];
  r.next = (r.next + 1) % EventRing::kMax;
  MOC_CUDA_OK(cudaEventRecord(*out, from));
  return MOC_OK;
}
int order(cudaStream_t before, cudaStream_t after) {
  cudaEvent_t e;
  MOC_TRY(fork_event(before, &e));
  MOC_CUDA_OK(cudaStreamWaitEvent(after, e, 0));
  return MOC_OK;
}
int weight_grad(int dtype, int64_t m, int64_t n, int64_t rows, const void* a, const void* b, float* out, int* status,
                void* stream) {
  Gemm g(dtype, m, n, rows, false, false, MOC_F32);
  if (dtype == MOC_BF16) g.split_k = splits(rows, m, n);
  if (g.split_k > 1)
    MOC_CUDA_OK(cudaMemsetAsync(out, 0, static_cast<size_t>(m * n) * 4, static_cast<cudaStream_t>(stream)));
  return moc_gemm(&g, a, b, out, nullptr, nullptr, status, stream);
}

}  // namespace moc

using namespace moc;

extern "C" int64_t moc_layer_arena_bytes(const moc_layer_desc* s) {
  if (check(s) != MOC_OK) return -1;
  Saved a;
  return carve(s, dims_of(s), nullptr, &a);
}

extern "C" int moc_layer_fwd(const moc_layer_desc* s) {
  MOC_TRY(check(s));
  MOC_REQUIRE(s->h_router && s->h_attn && s->bank && s->router_w && s->wq && s->wk && s->wv && s->wo && s->out &&
                  s->comb_idx && s->comb_w && s->arena && s->status, "NULL layer buffer");
  const Dims x = dims_of(s);
  Saved a;
  carve(s, x, s->arena, &a);
  const int B = s->batch, L = s->seq, d = s->hidden_dim;
  cudaStream_t main = static_cast<cudaStream_t>(s->stream), side = static_cast<cudaStream_t>(s->side_stream);
  const moc_router_shape rs = router_shape(s);
  const size_t ws_bytes = moc_router_workspace_bytes(&rs);

  // side stream: routing; then what nothing before the join reads (loss terms, touched-chapter lists)
  MOC_TRY(order(main, side));
  Join join(side, main);
  auto router = [&](int parts) {
    return moc_router_fwd_parts(&rs, s->h_router, s->router_w, s->router_b, a.pooled, a.logits, a.probs, s->idx, s->weights,
                                s->comb_idx, s->comb_w, a.row_stats, a.chapter_stats, s->losses, a.router_ws, ws_bytes,
                                parts, s->status, side);
  };
  MOC_TRY(router(1));
  cudaEvent_t routed;
  MOC_TRY(fork_event(side, &routed));
  if (s->with_losses) MOC_TRY(router(2));
  if (s->for_backward)
    MOC_TRY(moc_chapter_segments(s->comb_idx, static_cast<int>(x.pairs),
                                 static_cast<int>(s->bank_rows / s->tokens_per_chapter), s->uniq, a.seg_off, a.seg_pairs,
                                 a.pair_to_uniq, s->num_unique, s->status, side));

  // main stream meanwhile: bf16 weights (and transposes for the backward pass), normalisation, query projection
  {
    const void* src[4] = {s->wq, s->wk, s->wv, s->wo};
    void* dst[4] = {a.wq, a.wkv, a.wkv + x.dkv * d, a.wo};
    void* dst_t[4] = {a.wq_t, a.wkv_t, a.wkv_t ? a.wkv_t + x.dkv : nullptr, a.wo_t};
    const int dkv = static_cast<int>(x.dkv);
    const int32_t rows[4] = {d, dkv, dkv, d}, cols[4] = {d, d, d, d}, ldt[4] = {0, 2 * dkv, 2 * dkv, 0};
    MOC_TRY(moc_pack_weights(4, src, s->weight_dtype, dst, dst_t, rows, cols, ldt, main));
  }
  const float* x2 = s->attn_dtype == MOC_F32 ? static_cast<const float*>(s->h_attn) : a.x2;
  if (a.x2) MOC_TRY(moc_cast_bf16_to_f32(s->h_attn, a.x2, x.rows * d, main));
  const void* h2 = a.h2 ? a.h2 : s->h_attn;
  if (s->pre_norm != MOC_NORM_NONE)
    MOC_TRY(moc_norm_fwd(x2, s->norm_w, s->norm_b, s->pre_norm, s->pre_eps, x.rows, d, nullptr, a.h2, a.stats_n, main));
  else if (a.h2)
    MOC_TRY(moc_cast_f32_to_bf16(static_cast<const float*>(s->h_attn), a.h2, x.rows * d, main));
  {
    const Gemm g(MOC_BF16, x.rows, d, d, true, true, MOC_BF16);
    MOC_TRY(moc_gemm(&g, h2, a.wq, a.q, nullptr, nullptr, s->status, main));
  }

  MOC_CUDA_OK(cudaStreamWaitEvent(main, routed, 0));
  Gemm g(MOC_BF16, x.sel_rows, 2 * x.dkv, d, true, true, MOC_BF16);
  if (s->fused) {
    // gather, normalisation, weight multiply and the K/V projection in one kernel: chapters are read from the bf16 copy
    // of the bank through the TMA gather list, u~ (and 1/rms) is the epilogue's row scale
    MOC_TRY(moc_chapter_row_scale(s->comb_idx, s->comb_w, s->row_norm == MOC_NORM_RMS ? s->bank_inv_rms : nullptr,
                                  s->bank_rows, static_cast<int>(x.pairs), s->tokens_per_chapter, a.row_scale, s->status, main));
    g.a_block_rows = s->tokens_per_chapter;
    g.a_stored_rows = s->bank_rows;
    MOC_TRY(moc_gemm(&g, s->bank_shadow, a.wkv, a.kv, a.row_scale, s->comb_idx, s->status, main));
  } else {
    MOC_TRY(moc_gather_rows_fwd(s->bank, s->bank_dtype, s->bank_rows, d, s->tokens_per_chapter, s->comb_idx, s->comb_w, B, s->num_shared + x.k_sel, s->row_norm,
                                s->row_eps, a.m2, MOC_BF16, a.stats_m, s->status, main));
    MOC_TRY(moc_gemm(&g, a.m2, a.wkv, a.kv, nullptr, nullptr, s->status, main));
  }
  const int hd = d / s->num_heads;
  const moc_attn_shape as = {B, L, static_cast<int32_t>(x.n_sel), s->num_heads, s->num_kv_heads, hd,
                             1.0f / sqrtf(static_cast<float>(hd)), MOC_BF16};
  MOC_TRY(moc_attn_fwd(&as, a.q, a.kv, a.o, a.lse, s->status, main));
  Gemm go(MOC_BF16, x.rows, d, d, true, true, s->attn_dtype);
  if (s->add_residual) { go.residual = x2; go.ldr = d; }
  MOC_TRY(moc_gemm(&go, a.o, a.wo, s->out, nullptr, nullptr, s->status, main));
  return join.done();
}

namespace moc {
namespace {

struct Scratch {
  __nv_bfloat16 *g2, *d_o, *d_q, *d_kv, *d_mem, *m_raw;
  float *g32, *dh32, *dx32;         // fp32 forms of the output gradient / the attention input's gradient
  float *attn, *kv_dot, *d_comb_w, *d_logits, *d_pooled, *dummy_b;
  char *router_ws, *norm_ws;
};
int64_t carve_bwd(const moc_layer_desc* s, const moc_layer_bwd_desc* b, const Dims& x, void* scratch, Scratch* t) {
  Carver c{static_cast<char*>(scratch), 0};
  const bool f32 = s->attn_dtype == MOC_F32, norm = s->pre_norm != MOC_NORM_NONE;
  const moc_router_shape rs = router_shape(s);
  t->g2 = f32 ? c.take<__nv_bfloat16>(x.rows * x.d) : nullptr;
  t->g32 = s->add_residual && !f32 ? c.take<float>(x.rows * x.d) : nullptr;
  t->dh32 = norm ? c.take<float>(x.rows * x.d) : nullptr;
  t->dx32 = norm && !f32 ? c.take<float>(x.rows * x.d) : nullptr;
  t->norm_ws = norm ? c.take<char>(static_cast<int64_t>(moc_norm_bwd_workspace_bytes(x.rows, s->hidden_dim))) : nullptr;
  t->d_o = c.take<__nv_bfloat16>(x.rows * x.d); t->d_q = c.take<__nv_bfloat16>(x.rows * x.d);
  t->d_kv = c.take<__nv_bfloat16>(x.sel_rows * 2 * x.dkv); t->d_mem = c.take<__nv_bfloat16>(x.sel_rows * x.d);
  t->m_raw = s->fused && !b->wkv_grad_in_place ? c.take<__nv_bfloat16>(x.sel_rows * x.d) : nullptr;
  t->attn = c.take<float>(6 * x.rows * s->num_heads);
  t->kv_dot = s->fused && s->tokens_per_chapter == 64 ? c.take<float>(x.pairs * s->num_kv_heads) : nullptr;
  t->d_comb_w = c.take<float>(x.pairs);
  t->d_logits = c.take<float>(static_cast<int64_t>(s->batch) * s->num_chapters);
  t->d_pooled = c.take<float>(static_cast<int64_t>(s->batch) * x.rd);
  t->dummy_b = c.take<float>(s->num_chapters);
  t->router_ws = c.take<char>(static_cast<int64_t>(moc_router_workspace_bytes(&rs)));
  return c.off;
}

}  // namespace
}  // namespace moc

extern "C" int64_t moc_layer_bwd_scratch_bytes(const moc_layer_desc* s, const moc_layer_bwd_desc* b) {
  if (check(s) != MOC_OK || b == nullptr) return -1;
  Scratch t;
  return carve_bwd(s, b, dims_of(s), nullptr, &t);
}

extern "C" int moc_layer_bwd(const moc_layer_desc* s, const moc_layer_bwd_desc* b) {
  MOC_TRY(check(s));
  MOC_REQUIRE(s->for_backward && b && b->g && b->d_h_attn && b->d_wq && b->d_wkv && b->d_wo && b->scratch && s->arena &&
                  s->uniq && s->num_unique && s->status, "NULL layer gradient buffer");
  MOC_REQUIRE(!b->want_router_w || b->d_router_w, "NULL router gradient buffer");
  MOC_REQUIRE(!b->want_dh_router || b->d_h_router || s->router_dim == 0 || s->router_dim == s->hidden_dim,
              "router states of another width have a gradient of their own");
  const Dims x = dims_of(s);
  Saved a;
  Scratch t;
  carve(s, x, s->arena, &a);
  carve_bwd(s, b, x, b->scratch, &t);
  const int B = s->batch, L = s->seq, d = s->hidden_dim, hd = d / s->num_heads;
  const int64_t n_el = x.rows * d, bank_rows_n = s->bank_rows;
  cudaStream_t main = static_cast<cudaStream_t>(s->stream), side = static_cast<cudaStream_t>(s->side_stream);
  const bool f32 = s->attn_dtype == MOC_F32, norm = s->pre_norm != MOC_NORM_NONE;
  const void* h2 = a.h2 ? a.h2 : s->h_attn;
  int* st = s->status;

  const void* g2 = b->g;
  if (f32) {
    MOC_TRY(moc_cast_f32_to_bf16(static_cast<const float*>(b->g), t.g2, n_el, main));
    g2 = t.g2;
  }
  MOC_TRY(order(main, side));
  Join join(side, main);
  MOC_TRY(weight_grad(MOC_BF16, d, d, x.rows, g2, a.o, b->d_wo, st, side));
  {
    const Gemm g(MOC_BF16, x.rows, d, d, true, true, MOC_BF16);
    MOC_TRY(moc_gemm(&g, g2, a.wo_t, t.d_o, nullptr, nullptr, st, main));
  }
  // With 64-row chapters the chapter-weight gradient is taken in the dK/dV epilogue, where K and V are still in shared
  // memory (kv_dot).  The dQ kernel runs on the side stream beside the dK/dV kernel: each fills the tail of the other's
  // last round of CTAs.
  const moc_attn_shape as = {B, L, static_cast<int32_t>(x.n_sel), s->num_heads, s->num_kv_heads, hd,
                             1.0f / sqrtf(static_cast<float>(hd)), MOC_BF16};
  auto attn = [&](int parts, cudaStream_t stream) {
    return moc_attn_bwd_scaled_parts(&as, a.q, a.kv, a.o, a.lse, t.d_o, t.d_q, t.d_kv, t.attn, a.row_scale, t.kv_dot, parts,
                                     st, stream);
  };
  const bool split = s->fused && b->dq_on_side_stream;
  MOC_TRY(attn(1, main));
  if (split) {
    MOC_TRY(order(main, side));
    MOC_TRY(attn(2, side));
    MOC_TRY(attn(4, main));
  } else {
    MOC_TRY(attn(2, main));
    MOC_TRY(attn(4, main));
    MOC_TRY(order(main, side));
  }

  // side stream: what only the dQ path feeds
  MOC_TRY(weight_grad(MOC_BF16, d, d, x.rows, t.d_q, h2, b->d_wq, st, side));
  {
    Gemm g(MOC_BF16, x.rows, d, d, true, true, norm ? MOC_F32 : s->attn_dtype);
    const float* g32 = f32 ? static_cast<const float*>(b->g) : t.g32;
    if (s->add_residual && t.g32) MOC_TRY(moc_cast_bf16_to_f32(b->g, t.g32, n_el, side));
    if (norm) {
      MOC_TRY(moc_gemm(&g, t.d_q, a.wq_t, t.dh32, nullptr, nullptr, st, side));
      float* dx = f32 ? static_cast<float*>(b->d_h_attn) : t.dx32;
      MOC_TRY(moc_norm_bwd(t.dh32, f32 ? static_cast<const float*>(s->h_attn) : a.x2, s->norm_w, a.stats_n,
                           s->add_residual ? g32 : nullptr, s->pre_norm, x.rows, d, dx, b->d_norm_w, b->d_norm_b, t.norm_ws,
                           side));
      if (!f32) MOC_TRY(moc_cast_f32_to_bf16(dx, b->d_h_attn, n_el, side));
    } else {
      if (s->add_residual) { g.residual = g32; g.ldr = d; }
      MOC_TRY(moc_gemm(&g, t.d_q, a.wq_t, b->d_h_attn, nullptr, nullptr, st, side));
    }
  }
  cudaEvent_t dh_done;
  MOC_TRY(fork_event(side, &dh_done));
  if (split) MOC_TRY(order(main, side));          // dK/dV is on the main stream
  if (!s->fused) {
    MOC_TRY(weight_grad(MOC_BF16, 2 * x.dkv, d, x.sel_rows, t.d_kv, a.m2, b->d_wkv, st, side));
  } else if (b->wkv_grad_in_place) {
    // dKV' already carries the row scale, so the raw bank rows can be read in place through a gather list on B
    Gemm g(MOC_BF16, 2 * x.dkv, d, x.sel_rows, false, false, MOC_F32);
    g.split_k = splits(x.sel_rows, 2 * x.dkv, d);
    if (g.split_k > 1) MOC_CUDA_OK(cudaMemsetAsync(b->d_wkv, 0, static_cast<size_t>(2 * x.dkv * d) * 4, side));
    MOC_TRY(moc_gemm_gather_b(&g, t.d_kv, s->bank_shadow, b->d_wkv, nullptr, s->comb_idx, s->tokens_per_chapter, bank_rows_n,
                              st, side));
  } else {
    // ... but with the contraction running over chapters every K step of that product lands in another chapter of the
    // 403 MB copy, which measured twice as slow; the raw selected rows are copied out once, off the critical path
    MOC_TRY(moc_gather_rows_fwd(s->bank_shadow, MOC_BF16, bank_rows_n, d, s->tokens_per_chapter, s->comb_idx, nullptr, B,
                                s->num_shared + x.k_sel, MOC_NORM_NONE, s->row_eps, t.m_raw, MOC_BF16, nullptr, st, side));
    MOC_TRY(weight_grad(MOC_BF16, 2 * x.dkv, d, x.sel_rows, t.d_kv, t.m_raw, b->d_wkv, st, side));
  }

  {
    const Gemm g(MOC_BF16, x.sel_rows, d, 2 * x.dkv, true, true, MOC_BF16);
    MOC_TRY(moc_gemm(&g, t.d_kv, a.wkv_t, t.d_mem, nullptr, nullptr, st, main));
  }
  const bool want_bank = b->bank_rows || b->bank_rows_bf16 || b->bank_dense;
  const int dense = b->bank_dense != nullptr;
  float* rows_out = dense ? b->bank_dense : b->bank_rows;
  auto bank_grad = [&](float* d_cw, cudaStream_t stream) -> int {
    if (dense) MOC_TRY(clear_dense(b->bank_dense, bank_rows_n * d, stream));
    if (s->fused) {
      if (!d_cw && !want_bank) return MOC_OK;
      return gather_rows_bwd_prescaled_impl(t.d_mem, MOC_BF16, s->bank_shadow, MOC_BF16, bank_rows_n, d,
                                            s->tokens_per_chapter, s->comb_idx, s->comb_w, static_cast<int>(x.pairs),
                                            s->row_norm == MOC_NORM_RMS ? s->bank_inv_rms : nullptr, s->uniq, a.seg_off,
                                            a.seg_pairs, s->num_unique, d_cw, rows_out, b->bank_rows_bf16, st, stream, dense);
    }
    return gather_rows_bwd_impl(t.d_mem, MOC_BF16, s->bank, s->bank_dtype, bank_rows_n, d, s->tokens_per_chapter, s->comb_idx,
                                s->comb_w, B, s->num_shared + x.k_sel, s->row_norm, s->row_eps, a.stats_m, s->uniq,
                                a.seg_off, a.seg_pairs, s->num_unique, d_cw, rows_out, b->bank_rows_bf16, st, stream, dense);
  };
  const int n_pairs = static_cast<int>(x.pairs), pair_blocks = ceil_div(n_pairs, 256);
  if (t.kv_dot) {
    comb_w_grad_kernel<<<pair_blocks, 256, 0, main>>>(t.kv_dot, s->comb_w, b->g_comb_w, t.d_comb_w, n_pairs,
                                                      s->num_kv_heads);
    if (want_bank) {                     // nothing downstream reads the bank gradient: off the path to the router
      MOC_TRY(order(main, side));
      MOC_TRY(bank_grad(nullptr, side));
    }
  } else {
    MOC_TRY(bank_grad(t.d_comb_w, main));
    if (b->g_comb_w) add_kernel<<<pair_blocks, 256, 0, main>>>(t.d_comb_w, b->g_comb_w, n_pairs);
  }
  MOC_CUDA_OK(cudaGetLastError());

  // router: logit gradient on the main stream, its weight gradient (nothing downstream reads it) on the side stream
  const moc_router_shape rs = router_shape(s);
  const size_t ws_bytes = moc_router_workspace_bytes(&rs);
  void* d_h = b->d_h_router ? b->d_h_router : b->d_h_attn;
  auto router = [&](int parts, cudaStream_t stream) {
    return moc_router_bwd_parts(&rs, s->router_w, a.pooled, a.probs, s->idx, s->weights, s->comb_w, a.row_stats,
                                a.chapter_stats, b->g_weights, t.d_comb_w, b->g_losses, t.d_logits,
                                b->d_router_w ? b->d_router_w : t.d_logits, b->d_router_b ? b->d_router_b : t.dummy_b,
                                t.d_pooled, (parts & 4) ? d_h : nullptr, b->d_h_router ? 0 : 1, t.router_ws, ws_bytes, parts,
                                st, stream);
  };
  if (b->want_dh_router || b->want_router_w) MOC_TRY(router(1, main));
  if (b->want_router_w) {
    MOC_TRY(order(main, side));
    MOC_TRY(router(2, side));
  }
  if (b->want_dh_router) {
    if (!b->d_h_router) MOC_CUDA_OK(cudaStreamWaitEvent(main, dh_done, 0));
    MOC_TRY(router(4, main));
  }
  return join.done();
}
