// Cross attention over given memory rows, projections included: one call per pass, every kernel of it issued from here
// (the operator-by-operator form spent 25 to 45 us of host time on each of the 10 forward and 13 backward kernels).
// The weight-gradient products, which nothing downstream reads, run on the side stream.
#include "host_pass.cuh"

namespace moc {
namespace {

// dst [B, n] = src [n] for every batch item, 16 bytes per thread
__global__ void repeat_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, long long n, long long total) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i < total) dst[i] = src[i % n];
}
// dst [n] = sum over the batch of src [B, n], fp32 sums in batch order
template <typename T>
__global__ void batch_sum_kernel(const T* __restrict__ src, T* __restrict__ dst, long long n, int B) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  float acc = 0.f;
  for (int b = 0; b < B; ++b) acc += static_cast<float>(src[b * n + i]);
  dst[i] = static_cast<T>(acc);
}

struct Dims {
  int64_t rows, d, md, hd, od, dkv, mem_rows, kv_rows;   // hd: width of Q and O; kv_rows: rows of K / V the attention sees
  bool bf16, norm;
};
Dims dims_of(const moc_xattn_desc* s) {
  Dims x;
  x.rows = static_cast<int64_t>(s->batch) * s->seq;
  x.d = s->hidden_dim; x.md = s->mem_dim;
  x.hd = s->attn_dim ? s->attn_dim : s->hidden_dim; x.od = s->out_dim ? s->out_dim : s->hidden_dim;
  x.dkv = s->num_kv_heads * (x.hd / s->num_heads);
  x.kv_rows = static_cast<int64_t>(s->batch) * s->n_sel;
  x.mem_rows = s->mem_shared ? s->n_sel : x.kv_rows;
  x.bf16 = s->compute_dtype == MOC_BF16;
  x.norm = s->pre_norm != MOC_NORM_NONE;
  return x;
}
struct Saved {
  void *wq, *wkv, *wo;                       // weights in the compute dtype, where they are not the inputs themselves
  __nv_bfloat16 *wq_t, *wkv_t, *wo_t;
  float *x2, *stats, *lse;
  void *h2, *m2, *q, *kv, *kv1, *o;          // h2 / m2: where not the inputs themselves; kv1: before the repeat
};
int64_t carve(const moc_xattn_desc* s, const Dims& x, void* arena, Saved* a) {
  Carver c{static_cast<char*>(arena), 0};
  const int cd = s->compute_dtype;
  const bool pack = x.bf16 || s->weight_dtype != cd;
  a->wq = pack ? c.take_as(cd, x.hd * x.d) : nullptr;
  a->wkv = c.take_as(cd, 2 * x.dkv * x.md);
  a->wo = pack ? c.take_as(cd, x.od * x.hd) : nullptr;
  a->wq_t = a->wkv_t = a->wo_t = nullptr;
  if (x.bf16 && s->for_backward) {
    a->wq_t = c.take<__nv_bfloat16>(x.hd * x.d); a->wkv_t = c.take<__nv_bfloat16>(2 * x.dkv * x.md);
    a->wo_t = c.take<__nv_bfloat16>(x.od * x.hd);
  }
  a->x2 = (x.norm || s->add_residual) && s->h_dtype != MOC_F32 ? c.take<float>(x.rows * x.d) : nullptr;
  a->stats = x.norm ? c.take<float>(2 * x.rows) : nullptr;
  a->h2 = x.norm || s->h_dtype != cd ? c.take_as(cd, x.rows * x.d) : nullptr;
  a->m2 = s->mem_dtype != cd ? c.take_as(cd, x.mem_rows * x.md) : nullptr;
  a->q = c.take_as(cd, x.rows * x.hd);
  a->kv = c.take_as(cd, x.kv_rows * 2 * x.dkv);
  a->kv1 = s->mem_shared ? c.take_as(cd, x.mem_rows * 2 * x.dkv) : nullptr;
  a->o = c.take_as(cd, x.rows * x.hd);
  a->lse = c.take<float>(x.rows * s->num_heads);
  return c.off;
}
struct Scratch {
  void *g2, *d_o, *d_q, *d_kv, *d_kv1;
  float *g32, *dh32, *attn;
  void* dx;
  char* norm_ws;
};
int64_t carve_bwd(const moc_xattn_desc* s, const moc_xattn_bwd_desc* b, const Dims& x, void* scratch, Scratch* t) {
  Carver c{static_cast<char*>(scratch), 0};
  const int cd = s->compute_dtype;
  t->g2 = b->g_dtype != cd ? c.take_as(cd, x.rows * x.od) : nullptr;
  t->g32 = s->add_residual && b->g_dtype != MOC_F32 ? c.take<float>(x.rows * x.od) : nullptr;
  t->dh32 = x.norm ? c.take<float>(x.rows * x.d) : nullptr;
  t->dx = x.norm && b->d_h_dtype != MOC_F32 ? c.take<float>(x.rows * x.d) : nullptr;
  t->norm_ws = x.norm ? c.take<char>(static_cast<int64_t>(moc_norm_bwd_workspace_bytes(x.rows, s->hidden_dim))) : nullptr;
  t->d_o = c.take_as(cd, x.rows * x.hd); t->d_q = c.take_as(cd, x.rows * x.hd);
  t->d_kv = c.take_as(cd, x.kv_rows * 2 * x.dkv);
  t->d_kv1 = s->mem_shared ? c.take_as(cd, x.mem_rows * 2 * x.dkv) : nullptr;
  t->attn = c.take<float>(6 * x.rows * s->num_heads);
  return c.off;
}
int check(const moc_xattn_desc* s) {
  MOC_REQUIRE(s != nullptr, "cross-attention descriptor is NULL");
  MOC_REQUIRE(s->batch > 0 && s->seq > 0 && s->n_sel > 0 && s->hidden_dim > 0 && s->mem_dim > 0 && s->num_heads > 0 &&
                  s->num_kv_heads > 0 && s->hidden_dim >= s->num_heads && s->attn_dim >= 0 && s->out_dim >= 0 &&
                  (s->attn_dim ? s->attn_dim : s->hidden_dim) % s->num_heads == 0, "bad cross-attention shape");
  MOC_REQUIRE(!s->add_residual || s->out_dim == 0 || s->out_dim == s->hidden_dim, "the residual is as wide as the result");
  for (int dt : {s->h_dtype, s->mem_dtype, s->weight_dtype, s->compute_dtype, s->out_dtype})
    MOC_REQUIRE(dt == MOC_F32 || dt == MOC_BF16, "unknown dtype");
  MOC_REQUIRE(s->out_dtype == MOC_F32 || s->out_dtype == s->compute_dtype, "out must be fp32 or the compute dtype");
  MOC_REQUIRE(!(s->pre_norm != MOC_NORM_NONE) || s->norm_w, "pre_norm needs norm_w");
  return MOC_OK;
}
moc_attn_shape attn_shape(const moc_xattn_desc* s) {
  // (the softmax scale is that of the hidden width also where wq projects to another)
  const int hd = (s->attn_dim ? s->attn_dim : s->hidden_dim) / s->num_heads;
  return {s->batch, s->seq, s->n_sel, s->num_heads, s->num_kv_heads, hd,
          1.0f / sqrtf(static_cast<float>(s->hidden_dim / s->num_heads)), s->compute_dtype};
}

}  // namespace
}  // namespace moc

using namespace moc;

extern "C" int64_t moc_xattn_arena_bytes(const moc_xattn_desc* s) {
  if (check(s) != MOC_OK) return -1;
  Saved a;
  return carve(s, dims_of(s), nullptr, &a);
}
extern "C" int64_t moc_xattn_bwd_scratch_bytes(const moc_xattn_desc* s, const moc_xattn_bwd_desc* b) {
  if (check(s) != MOC_OK || b == nullptr) return -1;
  Scratch t;
  return carve_bwd(s, b, dims_of(s), nullptr, &t);
}

extern "C" int moc_xattn_fwd(const moc_xattn_desc* s) {
  MOC_TRY(check(s));
  MOC_REQUIRE(s->h && s->memory && s->wq && s->wk && s->wv && s->wo && s->out && s->arena && s->status, "NULL buffer");
  const Dims x = dims_of(s);
  Saved a;
  carve(s, x, s->arena, &a);
  const int cd = s->compute_dtype, d = s->hidden_dim, md = s->mem_dim, dkv = static_cast<int>(x.dkv);
  const int hd = static_cast<int>(x.hd), od = static_cast<int>(x.od);
  cudaStream_t st = static_cast<cudaStream_t>(s->stream);
  const int esize = x.bf16 ? 2 : 4;
  char* wv_dst = static_cast<char*>(a.wkv) + x.dkv * md * esize;
  const void *wq = s->wq, *wo = s->wo;
  if (x.bf16) {
    // one launch: bf16 working copies (Wk and Wv stacked) and, for the backward pass, their transposes
    const void* src[4] = {s->wq, s->wk, s->wv, s->wo};
    void* dst[4] = {a.wq, a.wkv, wv_dst, a.wo};
    void* dst_t[4] = {a.wq_t, a.wkv_t, a.wkv_t ? a.wkv_t + x.dkv : nullptr, a.wo_t};
    const int32_t rows[4] = {hd, dkv, dkv, od}, cols[4] = {d, md, md, hd}, ldt[4] = {0, 2 * dkv, 2 * dkv, 0};
    MOC_TRY(moc_pack_weights(4, src, s->weight_dtype, dst, dst_t, rows, cols, ldt, st));
    wq = a.wq; wo = a.wo;
  } else if (s->weight_dtype == MOC_F32) {
    MOC_CUDA_OK(cudaMemcpyAsync(a.wkv, s->wk, static_cast<size_t>(x.dkv * md) * 4, cudaMemcpyDeviceToDevice, st));
    MOC_CUDA_OK(cudaMemcpyAsync(wv_dst, s->wv, static_cast<size_t>(x.dkv * md) * 4, cudaMemcpyDeviceToDevice, st));
  } else {
    MOC_TRY(moc_cast_bf16_to_f32(s->wq, static_cast<float*>(a.wq), x.hd * d, st));
    MOC_TRY(moc_cast_bf16_to_f32(s->wk, static_cast<float*>(a.wkv), x.dkv * md, st));
    MOC_TRY(moc_cast_bf16_to_f32(s->wv, reinterpret_cast<float*>(wv_dst), x.dkv * md, st));
    MOC_TRY(moc_cast_bf16_to_f32(s->wo, static_cast<float*>(a.wo), x.od * x.hd, st));
    wq = a.wq; wo = a.wo;
  }
  const float* x2 = s->h_dtype == MOC_F32 ? static_cast<const float*>(s->h) : a.x2;
  if (a.x2) MOC_TRY(moc_cast_bf16_to_f32(s->h, a.x2, x.rows * d, st));
  const void *h2, *m2;
  if (x.norm) {
    MOC_TRY(moc_norm_fwd(x2, s->norm_w, s->norm_b, s->pre_norm, s->pre_eps, x.rows, d,
                         x.bf16 ? nullptr : static_cast<float*>(a.h2), x.bf16 ? a.h2 : nullptr, a.stats, st));
    h2 = a.h2;
  } else {
    MOC_TRY(as_dtype(s->h, s->h_dtype, a.h2, cd, x.rows * d, st, &h2));
  }
  MOC_TRY(as_dtype(s->memory, s->mem_dtype, a.m2, cd, x.mem_rows * md, st, &m2));
  const Gemm gq(cd, x.rows, hd, d, true, true, cd), gkv(cd, x.mem_rows, 2 * x.dkv, md, true, true, cd);
  MOC_TRY(moc_gemm(&gq, h2, wq, a.q, nullptr, nullptr, s->status, st));
  MOC_TRY(moc_gemm(&gkv, m2, a.wkv, a.kv1 ? a.kv1 : a.kv, nullptr, nullptr, s->status, st));
  if (a.kv1) {
    const long long n = x.mem_rows * 2 * x.dkv * esize / 16, total = n * s->batch;
    repeat_kernel<<<static_cast<int>((total + 255) / 256), 256, 0, st>>>(static_cast<const uint4*>(a.kv1),
                                                                         static_cast<uint4*>(a.kv), n, total);
  }
  const moc_attn_shape as = attn_shape(s);
  MOC_TRY(moc_attn_fwd(&as, a.q, a.kv, a.o, a.lse, s->status, st));
  Gemm go(cd, x.rows, od, hd, true, true, s->out_dtype);
  if (s->add_residual) { go.residual = x2; go.ldr = d; }
  return moc_gemm(&go, a.o, wo, s->out, nullptr, nullptr, s->status, st);
}

extern "C" int moc_xattn_bwd(const moc_xattn_desc* s, const moc_xattn_bwd_desc* b) {
  MOC_TRY(check(s));
  MOC_REQUIRE(s->for_backward && b && b->g && b->d_wq && b->d_wkv && b->d_wo && b->scratch && s->arena && s->status,
              "NULL buffer");
  const Dims x = dims_of(s);
  Saved a;
  Scratch t;
  carve(s, x, s->arena, &a);
  carve_bwd(s, b, x, b->scratch, &t);
  const int cd = s->compute_dtype, d = s->hidden_dim, md = s->mem_dim;
  const int64_t hd = x.hd, od = x.od;
  int* status = s->status;
  cudaStream_t main = static_cast<cudaStream_t>(s->stream), side = static_cast<cudaStream_t>(s->side_stream);
  const void* h2 = a.h2 ? a.h2 : s->h;
  const void* m2 = a.m2 ? a.m2 : s->memory;
  // dX = dY W: the tensor-core kernel is fastest with both operands K-major and takes the transposed copy of the
  // weight; the fp32 kernel takes the strided operand directly
  auto grad_in = [&](int64_t m, int64_t n, int64_t k, const void* dy, const void* w, const void* w_t, void* out, int dt,
                     const float* res, cudaStream_t st) {
    Gemm g(cd, m, n, k, true, x.bf16, dt);
    if (res) { g.residual = res; g.ldr = n; }
    return moc_gemm(&g, dy, x.bf16 ? w_t : w, out, nullptr, nullptr, status, st);
  };
  const void *wq = a.wq ? a.wq : s->wq, *wo = a.wo ? a.wo : s->wo;
  const void* g2;
  MOC_TRY(as_dtype(b->g, b->g_dtype, t.g2, cd, x.rows * od, main, &g2));
  MOC_TRY(order(main, side));
  Join join(side, main);
  MOC_TRY(weight_grad(cd, od, hd, x.rows, g2, a.o, b->d_wo, status, side));
  MOC_TRY(grad_in(x.rows, hd, od, g2, wo, a.wo_t, t.d_o, cd, nullptr, main));
  const moc_attn_shape as = attn_shape(s);
  if (x.bf16) {
    // the dQ kernel on the side stream, where its consumers follow it, beside the dK/dV kernel
    auto attn = [&](int parts, cudaStream_t st) {
      return moc_attn_bwd_parts(&as, a.q, a.kv, a.o, a.lse, t.d_o, t.d_q, t.d_kv, t.attn, parts, status, st);
    };
    MOC_TRY(attn(1, main));
    MOC_TRY(order(main, side));
    MOC_TRY(attn(2, side));
    MOC_TRY(attn(4, main));
  } else {
    MOC_TRY(moc_attn_bwd(&as, a.q, a.kv, a.o, a.lse, t.d_o, t.d_q, t.d_kv, t.attn, status, main));
    MOC_TRY(order(main, side));
  }
  MOC_TRY(weight_grad(cd, hd, d, x.rows, t.d_q, h2, b->d_wq, status, side));
  if (b->d_h || b->d_norm_w) {
    const float* g32 = nullptr;
    if (s->add_residual) {
      g32 = b->g_dtype == MOC_F32 ? static_cast<const float*>(b->g) : t.g32;
      if (t.g32) MOC_TRY(moc_cast_bf16_to_f32(b->g, t.g32, x.rows * d, side));
    }
    if (x.norm) {
      MOC_TRY(grad_in(x.rows, d, hd, t.d_q, wq, a.wq_t, t.dh32, MOC_F32, nullptr, side));
      float* dx = t.dx ? static_cast<float*>(t.dx) : static_cast<float*>(b->d_h);
      MOC_TRY(moc_norm_bwd(t.dh32, s->h_dtype == MOC_F32 ? static_cast<const float*>(s->h) : a.x2, s->norm_w, a.stats, g32,
                           s->pre_norm, x.rows, d, dx, b->d_norm_w, b->d_norm_b, t.norm_ws, side));
      if (t.dx) MOC_TRY(moc_cast_f32_to_bf16(dx, b->d_h, x.rows * d, side));
    } else {
      MOC_TRY(grad_in(x.rows, d, hd, t.d_q, wq, a.wq_t, b->d_h, b->d_h_dtype, g32, side));
    }
  }
  const void* d_kv = t.d_kv;
  if (t.d_kv1) {
    const long long n = x.mem_rows * 2 * x.dkv;
    const int blocks = static_cast<int>((n + 255) / 256);
    if (x.bf16)
      batch_sum_kernel<<<blocks, 256, 0, main>>>(static_cast<const __nv_bfloat16*>(t.d_kv),
                                                 static_cast<__nv_bfloat16*>(t.d_kv1), n, s->batch);
    else
      batch_sum_kernel<<<blocks, 256, 0, main>>>(static_cast<const float*>(t.d_kv), static_cast<float*>(t.d_kv1), n,
                                                 s->batch);
    d_kv = t.d_kv1;
  }
  MOC_TRY(order(main, side));
  MOC_TRY(weight_grad(cd, 2 * x.dkv, md, x.mem_rows, d_kv, m2, b->d_wkv, status, side));
  if (b->d_memory)
    MOC_TRY(grad_in(x.mem_rows, md, 2 * x.dkv, d_kv, a.wkv, a.wkv_t, b->d_memory, b->d_mem_dtype, nullptr, main));
  return join.done();
}
