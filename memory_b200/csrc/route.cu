// The sequence-level router in one call per pass (scratch and saved state are pieces of one buffer each), and the chapter
// gather's backward pass from the chapter lists.
#include "host_pass.cuh"

namespace moc {
namespace {

struct Saved {
  float *pooled, *logits, *probs, *row_stats, *chapter_stats;
  char* ws;
};
int64_t carve(const moc_router_shape* r, void* arena, Saved* a) {
  Carver c{static_cast<char*>(arena), 0};
  const int64_t B = r->batch, C = r->num_chapters;
  a->pooled = c.take<float>(B * r->hidden_dim); a->logits = c.take<float>(B * C); a->probs = c.take<float>(B * C);
  a->row_stats = c.take<float>(4 * B); a->chapter_stats = c.take<float>(2 * C);
  // (the position-weighted pooling keeps its partial sums here too)
  a->ws = c.take<char>(static_cast<int64_t>(moc_router_workspace_bytes(r)));
  return c.off;
}
struct Scratch {
  float *d_logits, *d_pooled, *dummy_b;
  char* ws;
};
int64_t carve_bwd(const moc_router_shape* r, void* scratch, Scratch* t) {
  Carver c{static_cast<char*>(scratch), 0};
  const int64_t B = r->batch, C = r->num_chapters;
  t->d_logits = c.take<float>(B * C); t->d_pooled = c.take<float>(B * r->hidden_dim); t->dummy_b = c.take<float>(C);
  t->ws = c.take<char>(static_cast<int64_t>(moc_router_workspace_bytes(r)));
  return c.off;
}

}  // namespace
}  // namespace moc

using namespace moc;

extern "C" int64_t moc_route_arena_bytes(const moc_route_desc* s) {
  Saved a;
  return s ? carve(&s->shape, nullptr, &a) : -1;
}
extern "C" int64_t moc_route_bwd_scratch_bytes(const moc_route_desc* s) {
  Scratch t;
  return s ? carve_bwd(&s->shape, nullptr, &t) : -1;
}

int moc::route_fwd_impl(const moc_route_desc* s, const RowsProduct* q, RouteRun* run) {
  MOC_REQUIRE(s && s->h && s->w && s->comb_idx && s->comb_w && s->arena && s->status, "NULL router buffer");
  const moc_router_shape* r = &s->shape;
  Saved a;
  carve(r, s->arena, &a);
  const size_t ws_bytes = moc_router_workspace_bytes(r);
  int parts = s->losses ? 3 : 1;
  if (s->pos_weight) {
    MOC_TRY(moc_pool_weighted_fwd(s->h, r->h_dtype, s->pos_weight, a.pooled, r->batch, r->seq, r->hidden_dim, a.ws, ws_bytes,
                                  s->stream));
    parts |= 8;
  }
  return router_fwd_parts_impl(r, s->h, s->w, s->bias, a.pooled, a.logits, a.probs, s->idx, s->weights, s->comb_idx,
                               s->comb_w, a.row_stats, a.chapter_stats, s->losses, a.ws, ws_bytes, parts, q, run, s->status,
                               s->stream);
}
extern "C" int moc_route_fwd(const moc_route_desc* s) { return route_fwd_impl(s, nullptr, nullptr); }

extern "C" int moc_route_bwd(const moc_route_desc* s, const float* g_weights, const float* g_comb_w, const float* g_losses,
                             void* d_h, float* d_w, float* d_bias, void* scratch) {
  MOC_REQUIRE(s && s->w && s->comb_w && s->arena && scratch && s->status, "NULL router buffer");
  const moc_router_shape* r = &s->shape;
  Saved a;
  Scratch t;
  carve(r, s->arena, &a);
  carve_bwd(r, scratch, &t);
  const bool rolling = s->pos_weight != nullptr;
  const int parts = 1 | (d_w ? 2 : 0) | (d_h ? 4 : 0);
  MOC_TRY(moc_router_bwd_parts(r, s->w, a.pooled, a.probs, s->idx, s->weights, s->comb_w, a.row_stats, a.chapter_stats,
                               g_weights, g_comb_w, g_losses, t.d_logits, d_w ? d_w : t.d_logits,
                               d_bias ? d_bias : t.dummy_b, t.d_pooled, rolling ? nullptr : d_h, 0, t.ws,
                               moc_router_workspace_bytes(r), parts, s->status, s->stream));
  if (rolling && d_h)
    MOC_TRY(moc_pool_weighted_bwd(t.d_pooled, s->pos_weight, d_h, r->h_dtype, r->batch, r->seq, r->hidden_dim, 0, s->stream));
  return MOC_OK;
}

extern "C" int moc_gather_rows_bwd_lists(const void* d_mem, int32_t d_mem_dtype, const void* bank, int32_t bank_dtype,
                                         int64_t bank_rows, int32_t dim, int32_t T, const int32_t* comb_idx,
                                         const float* comb_w, int32_t batch, int32_t k_sel, int32_t norm_type, float eps,
                                         const float* row_stats, int32_t* segments, float* d_comb_w, float* bank_grad,
                                         void* bank_grad_bf16, float* bank_dense, int32_t* status, void* stream) {
  MOC_REQUIRE(segments && T > 0 && !(bank_grad && bank_dense), "bad gather gradient arguments");
  const int n = batch * k_sel;
  int32_t *uniq = segments, *num = uniq + n, *off = num + 1, *pairs = off + n + 1, *to_uniq = pairs + n;
  MOC_TRY(moc_chapter_segments(comb_idx, n, static_cast<int32_t>(bank_rows / T), uniq, off, pairs, to_uniq, num, status, stream));
  if (bank_dense) MOC_TRY(clear_dense(bank_dense, bank_rows * dim, static_cast<cudaStream_t>(stream)));
  return gather_rows_bwd_impl(d_mem, d_mem_dtype, bank, bank_dtype, bank_rows, dim, T, comb_idx, comb_w, batch, k_sel,
                              norm_type, eps, row_stats, uniq, off, pairs, num, d_comb_w, bank_dense ? bank_dense : bank_grad,
                              bank_grad_bf16, status, stream, bank_dense != nullptr);
}
