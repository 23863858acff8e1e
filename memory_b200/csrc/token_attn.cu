// Token-routed memory attention (memory_attention.py:480-716, 452-456 with per-token chapter weights) in one call per pass:
//
//   out = Wo [ attn(q, shared rows)  +  rho * sum_s w[t, s] softmax(q K_c(t,s)^T) V_c(t,s) ],   bf16, head_dim 64, 64-row chapters.
//
// The routed bank is projected once for all tokens, and only where somebody looks: with few (token, slot) pairs the chapters
// that were selected are listed on the device, their rows converted into a compact copy, and every product over bank rows
// stops at the listed count (the host sizes buffers and grids for the most there could be).  250 tokens x 16 chapters of
// 4,096: the conversion and the K/V projection of the whole bank were 725 of 975 us.
#include "host_pass.cuh"

namespace moc {
namespace {

constexpr int kT = 64;       // rows of a chapter
constexpr int kD = 64;       // head dim

__global__ void mark_kernel(const int* __restrict__ idx, long long n, int M, int* __restrict__ flag, int* __restrict__ status) {
  const long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (p >= n) return;
  const int c = idx[p];
  if (c < 0 || c >= M) { atomicMax(status, MOC_DEV_BAD_INDEX); return; }
  flag[c] = 1;
}
// flag -> place of the chapter in the list (ascending ids); one CTA
__global__ void __launch_bounds__(1024)
list_kernel(int* __restrict__ flag, int M, int* __restrict__ uniq, int* __restrict__ count) {
  __shared__ int warp_tot[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (M + 1023) / 1024, lo = min(M, static_cast<int>(threadIdx.x) * per), hi = min(M, lo + per);
  int n = 0;
  for (int c = lo; c < hi; ++c) n += flag[c];
  int incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  int at = incl - n;
  for (int w = 0; w < warp; ++w) at += warp_tot[w];
  if (threadIdx.x == 1023) *count = at + n;
  for (int c = lo; c < hi; ++c) {
    const int f = flag[c];
    flag[c] = f ? at : -1;
    if (f) uniq[at++] = c;
  }
}
__global__ void remap_kernel(const int* __restrict__ idx, long long n, int M, const int* __restrict__ place, int* __restrict__ out) {
  const long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (p >= n) return;
  const int c = idx[p];
  out[p] = (c < 0 || c >= M) ? -1 : place[c];
}
// rows of the listed chapters, bf16, behind each other; 16 rows a CTA.  Bound by HBM.
template <typename T>
__global__ void __launch_bounds__(256)
take_rows_kernel(const T* __restrict__ bank, int d, const int* __restrict__ uniq, const int* __restrict__ count,
                 __nv_bfloat16* __restrict__ out) {
  if (static_cast<int>(blockIdx.x) >= *count) return;
  const long long n = static_cast<long long>(16) * d;
  const T* src = bank + (static_cast<long long>(uniq[blockIdx.x]) * kT + blockIdx.y * 16) * d;
  uint4* dst = reinterpret_cast<uint4*>(out + (static_cast<long long>(blockIdx.x) * kT + blockIdx.y * 16) * d);
#pragma unroll 4
  for (int i = threadIdx.x; i < n / 8; i += 256) {
    if constexpr (sizeof(T) == 2) {
      dst[i] = reinterpret_cast<const uint4*>(src)[i];
    } else {
      const float4 a = reinterpret_cast<const float4*>(src)[2 * i], b = reinterpret_cast<const float4*>(src)[2 * i + 1];
      dst[i] = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
    }
  }
}
// d_w[t, s] = sum over heads of d_w_heads[t, h, s]
__global__ void head_sum_kernel(const float* __restrict__ src, float* __restrict__ dst, long long rows, int H, int S) {
  const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (i >= rows * S) return;
  const float* p = src + (i / S) * H * S + i % S;
  float t = 0.f;
  for (int h = 0; h < H; ++h) t += p[h * S];
  dst[i] = t;
}

struct Dims {
  int64_t rows, rows_pad, pairs, d, hd, dkv, M, U, s_rows;
  bool listed, shared;
};
Dims dims_of(const moc_token_attn_desc* s) {
  Dims x;
  x.rows = s->rows; x.d = s->hidden_dim;
  // a bf16 attention backward takes queries in multiples of 64: zero rows fill up
  x.rows_pad = s->for_backward ? (x.rows + 63) / 64 * 64 : x.rows;
  x.pairs = x.rows * s->n_select;
  x.hd = static_cast<int64_t>(s->num_heads) * kD; x.dkv = static_cast<int64_t>(s->num_kv_heads) * kD;
  x.M = s->routed_rows / kT;
  x.s_rows = s->shared_rows; x.shared = s->shared_rows > 0;
  // Twice as many pairs as chapters leave 13 % of the chapters unselected (uniform picks): the copy no longer pays
  x.listed = x.pairs < 2 * x.M;
  x.U = x.listed ? std::min(x.M, x.pairs) : x.M;
  return x;
}
moc_sparse_attn_shape mix_shape(const moc_token_attn_desc* s, const Dims& x) {
  return {1, s->rows, static_cast<int32_t>(x.U * kT), s->num_heads, s->num_kv_heads, kD, s->n_select, kT, 0.125f, MOC_BF16};
}
moc_attn_shape shared_shape(const moc_token_attn_desc* s, const Dims& x) {
  return {1, static_cast<int32_t>(x.rows_pad), s->shared_rows, s->num_heads, s->num_kv_heads, kD, 0.125f, MOC_BF16};
}

using bf16 = __nv_bfloat16;
struct Saved {
  bf16 *h2, *wq, *wkv, *wo, *wq_t, *wkv_t, *wo_t, *q, *sm2, *kv_sh, *o_sh, *rm2, *kv, *comb;
  float *lse_sh, *lse_slots;
  int *place, *uniq, *count, *bidx;
  void* index;
};
int64_t carve(const moc_token_attn_desc* s, const Dims& x, void* arena, Saved* a) {
  Carver c{static_cast<char*>(arena), 0};
  const bool bwd = s->for_backward;
  a->h2 = s->h_dtype == MOC_F32 ? c.take<bf16>(x.rows * x.d) : nullptr;
  a->wq = c.take<bf16>(x.hd * x.d); a->wkv = c.take<bf16>(2 * x.dkv * x.d); a->wo = c.take<bf16>(x.d * x.hd);
  a->wq_t = bwd ? c.take<bf16>(x.hd * x.d) : nullptr;
  a->wkv_t = bwd ? c.take<bf16>(2 * x.dkv * x.d) : nullptr;
  a->wo_t = bwd ? c.take<bf16>(x.d * x.hd) : nullptr;
  a->q = c.take<bf16>(x.rows_pad * x.hd);
  a->sm2 = x.shared && s->shared_dtype == MOC_F32 ? c.take<bf16>(x.s_rows * x.d) : nullptr;
  a->kv_sh = x.shared ? c.take<bf16>(x.s_rows * 2 * x.dkv) : nullptr;
  a->o_sh = x.shared ? c.take<bf16>(x.rows_pad * x.hd) : nullptr;
  a->lse_sh = x.shared ? c.take<float>(x.rows_pad * s->num_heads) : nullptr;
  a->rm2 = x.listed || s->routed_dtype == MOC_F32 ? c.take<bf16>(x.U * kT * x.d) : nullptr;
  a->kv = c.take<bf16>(x.U * kT * 2 * x.dkv);
  a->comb = c.take<bf16>(x.rows * x.hd);
  a->lse_slots = c.take<float>(x.pairs * s->num_heads);
  a->place = x.listed ? c.take<int>(x.M) : nullptr;
  a->uniq = x.listed ? c.take<int>(x.U) : nullptr;
  a->count = x.listed ? c.take<int>(1) : nullptr;
  a->bidx = x.listed ? c.take<int>(x.pairs) : nullptr;
  const moc_sparse_attn_shape ms = mix_shape(s, x);
  a->index = c.take<char>(static_cast<int64_t>(moc_token_mix_workspace_bytes(&ms, 1)));
  return c.off;
}
struct Scratch {
  bf16 *g2, *d_o, *d_q, *d_q_sh, *d_kv_sh, *d_kv, *partial;
  float *attn, *d_w_heads;
};
int64_t carve_bwd(const moc_token_attn_desc* s, const moc_token_attn_bwd_desc* b, const Dims& x, void* scratch, Scratch* t) {
  Carver c{static_cast<char*>(scratch), 0};
  t->g2 = b->g_dtype == MOC_F32 ? c.take<bf16>(x.rows * x.d) : nullptr;
  t->d_o = c.take<bf16>(x.rows_pad * x.hd); t->d_q = c.take<bf16>(x.rows * x.hd);
  t->d_q_sh = x.shared ? c.take<bf16>(x.rows_pad * x.hd) : nullptr;
  t->d_kv_sh = x.shared ? c.take<bf16>(x.s_rows * 2 * x.dkv) : nullptr;
  t->attn = x.shared ? c.take<float>(6 * x.rows_pad * s->num_heads) : nullptr;
  t->d_kv = c.take<bf16>(x.U * kT * 2 * x.dkv);
  t->partial = c.take<bf16>(x.pairs * x.hd);
  t->d_w_heads = c.take<float>(x.pairs * s->num_heads);
  return c.off;
}

int check(const moc_token_attn_desc* s) {
  MOC_REQUIRE(s != nullptr, "token-attention descriptor is NULL");
  MOC_REQUIRE(s->rows > 0 && s->n_select > 0 && s->hidden_dim > 0 && s->num_heads > 0 && s->num_kv_heads > 0 &&
              s->num_heads % s->num_kv_heads == 0, "empty token-attention problem");
  MOC_REQUIRE(s->hidden_dim == s->num_heads * kD, "token attention needs head_dim 64");
  MOC_REQUIRE(s->routed_rows >= kT && s->routed_rows % kT == 0 && s->shared_rows >= 0, "whole 64-row chapters only");
  MOC_REQUIRE(static_cast<int64_t>(s->rows) * s->n_select < (int64_t{1} << 31), "too many (token, slot) pairs");
  return MOC_OK;
}
inline int blocks_of(int64_t n) { return static_cast<int>((n + 255) / 256); }

}  // namespace
}  // namespace moc

using namespace moc;

extern "C" int64_t moc_token_attn_arena_bytes(const moc_token_attn_desc* s) {
  if (check(s) != MOC_OK) return -1;
  Saved a;
  return carve(s, dims_of(s), nullptr, &a);
}
extern "C" int64_t moc_token_attn_fwd_scratch_bytes(const moc_token_attn_desc* s) {
  if (check(s) != MOC_OK) return -1;
  const Dims x = dims_of(s);
  return x.pairs * x.hd * 2;
}
extern "C" int64_t moc_token_attn_bwd_scratch_bytes(const moc_token_attn_desc* s, const moc_token_attn_bwd_desc* b) {
  if (check(s) != MOC_OK || b == nullptr) return -1;
  Scratch t;
  return carve_bwd(s, b, dims_of(s), nullptr, &t);
}

extern "C" int moc_token_attn_fwd(const moc_token_attn_desc* s, void* scratch) {
  MOC_TRY(check(s));
  MOC_REQUIRE(s->h && s->routed && (s->shared || s->shared_rows == 0) && s->idx && s->weights && s->wq && s->wk && s->wv &&
              s->wo && s->out && s->arena && scratch && s->status, "NULL token-attention buffer");
  const Dims x = dims_of(s);
  Saved a;
  carve(s, x, s->arena, &a);
  cudaStream_t st = static_cast<cudaStream_t>(s->stream);
  const int d = s->hidden_dim, hd = static_cast<int>(x.hd), dkv = static_cast<int>(x.dkv);
  const void* src[4] = {s->wq, s->wk, s->wv, s->wo};
  void* dst[4] = {a.wq, a.wkv, a.wkv + x.dkv * d, a.wo};
  void* dst_t[4] = {a.wq_t, a.wkv_t, a.wkv_t ? a.wkv_t + x.dkv : nullptr, a.wo_t};
  const int32_t prows[4] = {hd, dkv, dkv, d}, pcols[4] = {d, d, d, hd}, ldt[4] = {0, 2 * dkv, 2 * dkv, 0};
  MOC_TRY(moc_pack_weights(4, src, s->weight_dtype, dst, dst_t, prows, pcols, ldt, st));
  const void *h2, *sm2, *rm2;
  MOC_TRY(as_dtype(s->h, s->h_dtype, a.h2, MOC_BF16, x.rows * d, st, &h2));
  const Gemm gq(MOC_BF16, x.rows, x.hd, d, true, true, MOC_BF16);
  MOC_TRY(moc_gemm(&gq, h2, a.wq, a.q, nullptr, nullptr, s->status, st));
  if (x.shared) {
    if (x.rows_pad > x.rows)
      MOC_CUDA_OK(cudaMemsetAsync(a.q + x.rows * x.hd, 0, static_cast<size_t>((x.rows_pad - x.rows) * x.hd) * 2, st));
    MOC_TRY(as_dtype(s->shared, s->shared_dtype, a.sm2, MOC_BF16, x.s_rows * d, st, &sm2));
    const Gemm g(MOC_BF16, x.s_rows, 2 * x.dkv, d, true, true, MOC_BF16);
    MOC_TRY(moc_gemm(&g, sm2, a.wkv, a.kv_sh, nullptr, nullptr, s->status, st));
    const moc_attn_shape as = shared_shape(s, x);
    MOC_TRY(moc_attn_fwd(&as, a.q, a.kv_sh, a.o_sh, a.lse_sh, s->status, st));
  }
  const int32_t* bidx = s->idx;
  Gemm gkv(MOC_BF16, x.U * kT, 2 * x.dkv, d, true, true, MOC_BF16);
  if (x.listed) {
    MOC_CUDA_OK(cudaMemsetAsync(a.place, 0, static_cast<size_t>(x.M) * 4, st));
    mark_kernel<<<blocks_of(x.pairs), 256, 0, st>>>(s->idx, x.pairs, static_cast<int>(x.M), a.place, s->status);
    list_kernel<<<1, 1024, 0, st>>>(a.place, static_cast<int>(x.M), a.uniq, a.count);
    remap_kernel<<<blocks_of(x.pairs), 256, 0, st>>>(s->idx, x.pairs, static_cast<int>(x.M), a.place, a.bidx);
    const dim3 grid(static_cast<unsigned>(x.U), kT / 16);
    if (s->routed_dtype == MOC_F32)
      take_rows_kernel<float><<<grid, 256, 0, st>>>(static_cast<const float*>(s->routed), d, a.uniq, a.count, a.rm2);
    else
      take_rows_kernel<bf16><<<grid, 256, 0, st>>>(static_cast<const bf16*>(s->routed), d, a.uniq, a.count, a.rm2);
    MOC_CUDA_OK(cudaGetLastError());
    bidx = a.bidx;
    rm2 = a.rm2;
    gkv.extra.limit = a.count; gkv.extra.limit_block = kT;
  } else {
    MOC_TRY(as_dtype(s->routed, s->routed_dtype, a.rm2, MOC_BF16, x.M * kT * d, st, &rm2));
  }
  MOC_TRY(gemm_extra(gkv, rm2, a.wkv, a.kv, s->status, st));
  const moc_sparse_attn_shape ms = mix_shape(s, x);
  MOC_TRY(moc_token_mix_index(&ms, 1, bidx, a.index, s->status, st));
  MOC_TRY(moc_token_mix_fwd(&ms, 1, a.q, a.kv, a.kv + x.dkv, 2 * x.dkv, bidx, s->weights, a.o_sh, s->routed_scale, a.index,
                            scratch, a.comb, a.lse_slots, s->status, st));
  const Gemm go(MOC_BF16, x.rows, d, x.hd, true, true, s->out_dtype);
  return moc_gemm(&go, a.comb, a.wo, s->out, nullptr, nullptr, s->status, st);
}

extern "C" int moc_token_attn_bwd(const moc_token_attn_desc* s, const moc_token_attn_bwd_desc* b) {
  MOC_TRY(check(s));
  MOC_REQUIRE(s->for_backward && b && b->g && b->d_h && b->d_wq && b->d_wkv && b->d_wo && b->d_weights && b->scratch &&
              s->arena && s->status, "NULL token-attention gradient buffer");
  const Dims x = dims_of(s);
  Saved a;
  Scratch t;
  carve(s, x, s->arena, &a);
  carve_bwd(s, b, x, b->scratch, &t);
  cudaStream_t st = static_cast<cudaStream_t>(s->stream);
  const int d = s->hidden_dim;
  const void *h2 = a.h2 ? a.h2 : s->h, *sm2 = a.sm2 ? a.sm2 : s->shared, *rm2 = a.rm2 ? a.rm2 : s->routed;
  const int32_t* bidx = x.listed ? a.bidx : s->idx;
  const void* g2;
  MOC_TRY(as_dtype(b->g, b->g_dtype, t.g2, MOC_BF16, x.rows * d, st, &g2));
  const Gemm go(MOC_BF16, x.rows, x.hd, d, true, true, MOC_BF16);
  MOC_TRY(moc_gemm(&go, g2, a.wo_t, t.d_o, nullptr, nullptr, s->status, st));
  MOC_TRY(weight_grad(MOC_BF16, d, x.hd, x.rows, g2, a.comb, b->d_wo, s->status, st));
  // dWkv: every product below adds to it
  MOC_CUDA_OK(cudaMemsetAsync(b->d_wkv, 0, static_cast<size_t>(2 * x.dkv * d) * 4, st));
  auto wkv_grad = [&](int64_t rows, const void* d_kv, const void* mem, const int32_t* limit) {
    Gemm g(MOC_BF16, 2 * x.dkv, d, rows, false, false, MOC_F32);
    g.accumulate = 1;
    g.split_k = splits(rows, 2 * x.dkv, d);
    g.extra.limit = limit; g.extra.limit_block = kT; g.extra.limit_k = 1;
    return gemm_extra(g, d_kv, mem, b->d_wkv, s->status, st);
  };
  if (x.shared) {
    if (x.rows_pad > x.rows)
      MOC_CUDA_OK(cudaMemsetAsync(t.d_o + x.rows * x.hd, 0, static_cast<size_t>((x.rows_pad - x.rows) * x.hd) * 2, st));
    const moc_attn_shape as = shared_shape(s, x);
    MOC_TRY(moc_attn_bwd(&as, a.q, a.kv_sh, a.o_sh, a.lse_sh, t.d_o, t.d_q_sh, t.d_kv_sh, t.attn, s->status, st));
    MOC_TRY(wkv_grad(x.s_rows, t.d_kv_sh, sm2, nullptr));
    if (b->d_shared) {
      const Gemm g(MOC_BF16, x.s_rows, d, 2 * x.dkv, true, true, s->shared_dtype);
      MOC_TRY(moc_gemm(&g, t.d_kv_sh, a.wkv_t, b->d_shared, nullptr, nullptr, s->status, st));
    }
  }
  const moc_sparse_attn_shape ms = mix_shape(s, x);
  MOC_CUDA_OK(cudaMemsetAsync(t.d_w_heads, 0, static_cast<size_t>(x.pairs * s->num_heads) * 4, st));
  MOC_TRY(moc_token_mix_bwd(&ms, 1, a.q, a.kv, a.kv + x.dkv, 2 * x.dkv, bidx, s->weights, s->routed_scale, a.lse_slots, t.d_o,
                            a.index, t.partial, t.d_q_sh, t.d_q, t.d_kv, t.d_kv + x.dkv, 2 * x.dkv, t.d_w_heads, s->status, st));
  head_sum_kernel<<<blocks_of(x.pairs), 256, 0, st>>>(t.d_w_heads, b->d_weights, x.rows, s->num_heads, s->n_select);
  MOC_CUDA_OK(cudaGetLastError());
  if (b->d_routed) {
    // dense over the bank, in its dtype; listed chapters go to their places among zeros
    Gemm g(MOC_BF16, x.U * kT, d, 2 * x.dkv, true, true, s->routed_dtype);
    if (x.listed) {
      MOC_CUDA_OK(cudaMemsetAsync(b->d_routed, 0, static_cast<size_t>(x.M * kT * d) * (s->routed_dtype == MOC_F32 ? 4 : 2), st));
      g.extra.limit = a.count; g.extra.limit_block = kT;
      g.extra.c_row_blocks = a.uniq; g.extra.c_block_rows = kT; g.extra.c_stored_rows = x.M * kT;
    }
    MOC_TRY(gemm_extra(g, t.d_kv, a.wkv_t, b->d_routed, s->status, st));
  }
  MOC_TRY(wkv_grad(x.U * kT, t.d_kv, rm2, x.listed ? a.count : nullptr));
  const Gemm gh(MOC_BF16, x.rows, d, x.hd, true, true, s->h_dtype);
  MOC_TRY(moc_gemm(&gh, t.d_q, a.wq_t, b->d_h, nullptr, nullptr, s->status, st));
  return weight_grad(MOC_BF16, x.hd, d, x.rows, t.d_q, h2, b->d_wq, s->status, st);
}
