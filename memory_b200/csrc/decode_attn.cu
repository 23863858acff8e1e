// Decode-time memory attention over a cache of projected bank rows.
//
// The reference re-gathers (S+k)*T bank rows per sequence at every generated token and re-projects them with Wk / Wv
// (inference/generate.py:194-210 -> model.py:624-692 -> memory_attention.py:241-243).  The bank and the projections
// are constant while decoding, and the chapter weight multiplies a gathered row before the (linear) projection, so
//   K = (u_c * norm(m)) Wk^T = u_c * (norm(m) Wk^T)
// and a per-layer cache  KV_bank = norm(M) [Wk; Wv]^T  (bf16, [C*T, 2*HK*64]) turns the step into a gather of
// cached rows scaled by the chapter weight, followed by one joint softmax over all selected keys:
//   s_r = scale * u_c * <q, K_bank[r]>,   out = sum_r softmax(s)_r * u_c * V_bank[r].
// The kernel is bound by HBM (a full batch) or by latency (a few sequences).  A cluster of CTAs takes the selected rows of
// one (sequence, query token, group of G query heads on one KV head) in turns of 32 rows per warp; parts merge through
// shared memory, then distributed shared memory.  One sequence, 12 heads, 4,160 rows: 34 us with a CTA per head -> 7.4 with
// a cluster of eight; 64 sequences: 162 us -> 120.
#include "host_pass.cuh"

namespace moc {
namespace {

constexpr int kDD = 64;
constexpr int kDecThreads = 256;
constexpr int kDecWarps = kDecThreads / 32;
constexpr float kDecLog2e = 1.4426950408889634f;

__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

// Lane layout: eight lanes share a row (16 bytes of its 128-byte K slice and of its V slice each), so one warp load
// instruction touches four whole 128-byte lines instead of 32 scattered 16-byte pieces; a warp takes 32 rows at a time, all
// requested before any arithmetic.  The eight products of a lane are reduced together over the eight lanes of a row group
// (7 shuffles), after which lane `part` holds the score of the group's step `part`: one exponential per row and head.
constexpr int kDecUnroll = 8;
constexpr int kDecRows = 4 * kDecUnroll;

template <int G>
__global__ void __launch_bounds__(kDecThreads, G == 1 ? 2 : 1)
decode_attn_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ kv_bank,
                   long long bank_rows, const int* __restrict__ comb_idx, const float* __restrict__ comb_w,
                   __nv_bfloat16* __restrict__ out, float* __restrict__ lse, int n_q, int H, int HK, int n_ch, int T,
                   float scale, int split, int* __restrict__ status) {
  __shared__ __align__(16) float red[G][kDecWarps][kDD + 4];
  __shared__ __align__(16) float cta_part[G][kDD + 4];        // accumulator, maximum, sum of this CTA
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rg = lane >> 3, part = lane & 7;          // row group 0..3, 8-element slice of the head dimension
  const int rank = static_cast<int>(blockIdx.x) % split, h0 = static_cast<int>(blockIdx.x) / split * G;
  const int iq = blockIdx.y, b = blockIdx.z;
  const int kh = h0 / (H / HK);
  const long long row_elems = 2ll * HK * kDD;
  const long long q_row = (static_cast<long long>(b) * n_q + iq) * H;

  float qf[G][8], acc[G][8], m[G], l[G];              // running maximum (log2 domain), this lane's share of the sum
  const float c2 = scale * kDecLog2e;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    unpack8(*reinterpret_cast<const uint4*>(q + (q_row + h0 + g) * kDD + part * 8), qf[g]);
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[g][i] = 0.f;
  }

  const int runs = (T + kDecRows - 1) / kDecRows;
  for (int unit = rank * kDecWarps + warp; unit < n_ch * runs; unit += split * kDecWarps) {
    const int c = unit / runs, r0 = (unit - c * runs) * kDecRows;
    const int ch = comb_idx[b * n_ch + c];
    if (ch < 0 || (static_cast<long long>(ch) + 1) * T > bank_rows) {
      if (lane == 0) atomicMax(status, MOC_DEV_BAD_INDEX);
      continue;
    }
    const float u = comb_w[b * n_ch + c];
    const __nv_bfloat16* base = kv_bank + static_cast<long long>(ch) * T * row_elems + kh * kDD + part * 8;
    uint4 kr[kDecUnroll], vr[kDecUnroll];
#pragma unroll
    for (int sidx = 0; sidx < kDecUnroll; ++sidx) {
      const int r = r0 + sidx * 4 + rg;
      const __nv_bfloat16* rp = base + static_cast<long long>(r < T ? r : 0) * row_elems;
      kr[sidx] = *reinterpret_cast<const uint4*>(rp);
      vr[sidx] = *reinterpret_cast<const uint4*>(rp + HK * kDD);
    }
    float dot[G][kDecUnroll];
#pragma unroll
    for (int sidx = 0; sidx < kDecUnroll; ++sidx) {
      float f[8];
      unpack8(kr[sidx], f);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float t = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) t = fmaf(qf[g][j], f[j], t);
        dot[g][sidx] = t;
      }
    }
    const bool in = r0 + part * 4 + rg < T;           // the row whose score this lane ends up with
    float pu[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
#pragma unroll
      for (int n = kDecUnroll / 2; n > 0; n >>= 1) {
        const bool up = lane & n;
#pragma unroll
        for (int i = 0; i < n; ++i) {
          const float send = up ? dot[g][i] : dot[g][i + n];
          const float keep = up ? dot[g][i + n] : dot[g][i];
          dot[g][i] = keep + __shfl_xor_sync(0xffffffffu, send, n);
        }
      }
      const float sc = in ? dot[g][0] * u * c2 : -INFINITY;
      float mx = fmaxf(sc, __shfl_xor_sync(0xffffffffu, sc, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
      const float m_new = fmaxf(m[g], mx);
      const float ref = m_new == -INFINITY ? 0.f : m_new;      // (a row group past the end of a short chapter)
      const float corr = exp2f(m[g] - ref);                    // 0 on the first rows (m = -inf)
      const float pr = exp2f(sc - ref);
      l[g] = l[g] * corr + pr;
      pu[g] = pr * u;
      m[g] = m_new;
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[g][j] *= corr;
    }
#pragma unroll
    for (int sidx = 0; sidx < kDecUnroll; ++sidx) {
      float f[8];
      unpack8(vr[sidx], f);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float p = __shfl_sync(0xffffffffu, pu[g], (lane & 24) | sidx);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[g][j] = fmaf(p, f[j], acc[g][j]);
      }
    }
  }

  // row groups -> warp (lanes with the same `part` hold the same 8 output elements)
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float mw = m[g];
    mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, 8));
    mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, 16));
    const float f_lane = (m[g] == -INFINITY) ? 0.f : exp2f(m[g] - mw);
    const float lw = warp_sum(l[g] * f_lane);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float a = acc[g][j] * f_lane;
      a += __shfl_xor_sync(0xffffffffu, a, 8);
      a += __shfl_xor_sync(0xffffffffu, a, 16);
      if (rg == 0) red[g][warp][part * 8 + j] = a;
    }
    if (lane == 0) {
      red[g][warp][kDD] = mw;
      red[g][warp][kDD + 1] = lw;
    }
  }
  __syncthreads();
  // warps -> CTA: thread i finishes output element i % 64 of head i / 64
  for (int i = threadIdx.x; i < G * kDD; i += kDecThreads) {
    const int g = i / kDD, e = i % kDD;
    float mt = -INFINITY;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) mt = fmaxf(mt, red[g][w][kDD]);
    float lt = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      const float f = (red[g][w][kDD] == -INFINITY) ? 0.f : exp2f(red[g][w][kDD] - mt);
      lt += red[g][w][kDD + 1] * f;
      a += red[g][w][e] * f;
    }
    cta_part[g][e] = a;
    if (e == 0) { cta_part[g][kDD] = mt; cta_part[g][kDD + 1] = lt; }
  }
  // CTAs -> output: the cluster's first CTA reads the others' parts (one of its own needs no barrier beyond the CTA's)
  if (split > 1) cluster_sync(); else __syncthreads();
  if (rank == 0) {
    for (int i = threadIdx.x; i < G * kDD; i += kDecThreads) {
      const int g = i / kDD, e = i % kDD;
      const uint32_t stat = static_cast<uint32_t>(__cvta_generic_to_shared(&cta_part[g][kDD]));
      const uint32_t elem = static_cast<uint32_t>(__cvta_generic_to_shared(&cta_part[g][e & ~1]));
      float mt = -INFINITY, lt = 0.f, a = 0.f;
      for (int r = 0; r < split; ++r) {
        const float2 st = split > 1 ? cluster_ld2(cluster_map(stat, r)) : make_float2(cta_part[g][kDD], cta_part[g][kDD + 1]);
        const float2 ab = split > 1 ? cluster_ld2(cluster_map(elem, r))
                                    : make_float2(cta_part[g][e & ~1], cta_part[g][e | 1]);
        const float m_new = fmaxf(mt, st.x);
        const float f0 = mt == -INFINITY ? 0.f : exp2f(mt - m_new), f1 = st.x == -INFINITY ? 0.f : exp2f(st.x - m_new);
        lt = lt * f0 + st.y * f1;
        a = a * f0 + ((e & 1) ? ab.y : ab.x) * f1;
        mt = m_new;
      }
      out[(q_row + h0 + g) * kDD + e] = __float2bfloat16(lt > 0.f ? a / lt : 0.f);
      if (e == 0 && lse != nullptr) lse[q_row + h0 + g] = lt > 0.f ? (mt + log2f(lt)) / kDecLog2e : -INFINITY;
    }
  }
  if (split > 1) cluster_sync();       // nobody leaves while its part is read
}

// dst[b] = the last dst_rows of (cache[b] followed by h[b]); rows of 16-byte pieces
__global__ void __launch_bounds__(256)
roll_window_kernel(const uint4* __restrict__ cache, long long cache_stride, int cache_rows, const uint4* __restrict__ h,
                   long long h_stride, int h_rows, uint4* __restrict__ dst, int dst_rows, int pieces) {
  const int b = blockIdx.y, skip = cache_rows + h_rows - dst_rows;
  const int total = dst_rows * pieces;
  uint4* out = dst + static_cast<long long>(b) * total;
  const uint4* c = cache + b * cache_stride + static_cast<long long>(skip) * pieces;
  const uint4* n = h + b * h_stride + static_cast<long long>(skip - cache_rows) * pieces;
  const int from_cache = (cache_rows - skip) * pieces;       // (negative where h alone fills the window)
  for (int i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) out[i] = i < from_cache ? c[i] : n[i];
}

struct StepArena {
  moc_route_desc route;
  __nv_bfloat16 *x, *q, *o;
  char* route_arena;
};
int64_t width_of(const moc_decode_step_desc* s) { return s->hidden_dim ? s->hidden_dim : s->router.hidden_dim; }
int64_t carve(const moc_decode_step_desc* s, StepArena* a) {
  a->route = moc_route_desc{};
  a->route.shape = s->router;
  Carver c{static_cast<char*>(s->arena), 0};
  const int64_t rows = static_cast<int64_t>(s->attn.batch) * s->attn.n_q, width = static_cast<int64_t>(s->attn.num_heads) * kDD;
  a->x = c.take<__nv_bfloat16>(rows * width_of(s));
  a->q = c.take<__nv_bfloat16>(rows * width);
  a->o = c.take<__nv_bfloat16>(rows * width);
  a->route_arena = c.take<char>(moc_route_arena_bytes(&a->route));
  return c.off;
}

}  // namespace
}  // namespace moc

using namespace moc;

extern "C" int moc_decode_attn(const moc_decode_shape* s, const void* q, const void* kv_bank, int64_t bank_rows,
                               const int32_t* comb_idx, const float* comb_w, void* out, float* lse,
                               int32_t* status, void* stream_) {
  MOC_REQUIRE(s && q && kv_bank && comb_idx && comb_w && out && status, "NULL decode-attention argument");
  MOC_REQUIRE(s->head_dim == kDD, "decode attention needs head_dim 64");
  MOC_REQUIRE(s->batch > 0 && s->n_q > 0 && s->n_chapters > 0 && s->tokens_per_chapter > 0 && bank_rows > 0,
              "empty decode-attention problem");
  MOC_REQUIRE(s->num_heads > 0 && s->num_kv_heads > 0 && s->num_heads % s->num_kv_heads == 0,
              "num_heads must be a positive multiple of num_kv_heads");
  MOC_REQUIRE(s->n_q <= 65535 && s->batch <= 65535, "too many query tokens or sequences for one launch");
  MOC_REQUIRE((reinterpret_cast<uintptr_t>(q) & 15) == 0 && (reinterpret_cast<uintptr_t>(kv_bank) & 15) == 0,
              "q and the K/V cache must be 16-byte aligned");
  // query heads that share a KV head go together: their rows are fetched once
  const int per_kv = s->num_heads / s->num_kv_heads;
  const int group = per_kv % 4 == 0 ? 4 : per_kv % 3 == 0 ? 3 : per_kv % 2 == 0 ? 2 : 1;
  auto kern = group == 4 ? decode_attn_kernel<4> : group == 3 ? decode_attn_kernel<3>
              : group == 2 ? decode_attn_kernel<2> : decode_attn_kernel<1>;
  // A cluster per group while all of them are resident at once and every warp has rows to take.  How many are depends on
  // the registers (an SM holds two CTAs of one head, one of a group) and on what is left of each GPC beside whole clusters:
  // 33 clusters of eight single-head CTAs, 15 of grouped ones.  With 296 slots counted for either, 12 heads on 4 KV heads
  // and 65 chapters took 14.8 us for 4 sequences, 22.0 for 8, 19.9 for 12, now 10.3, 10.8, 16.1; 12 heads of their own
  // 13.6 us for 3 sequences and 18.0 for 6, now 10.8 and 14.2.
  const long long groups = static_cast<long long>(s->num_heads / group) * s->n_q * s->batch;
  const int units = s->n_chapters * ceil_div(s->tokens_per_chapter, kDecRows);
  int split = 8;
  while (split > 1 && (split / 2 * kDecWarps >= units || groups > resident_clusters(kern, kDecThreads, 0, split))) split /= 2;
  dim3 grid(s->num_heads / group * split, s->n_q, s->batch);
  MOC_CUDA_OK(launch_clustered(kern, grid, kDecThreads, 0, split, static_cast<cudaStream_t>(stream_),
                               static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(kv_bank),
                               static_cast<long long>(bank_rows), comb_idx, comb_w, static_cast<__nv_bfloat16*>(out), lse,
                               s->n_q, s->num_heads, s->num_kv_heads, s->n_chapters, s->tokens_per_chapter, s->scale, split,
                               status));
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" int moc_roll_window(const void* cache, int64_t cache_stride, int32_t cache_rows, const void* h, int64_t h_stride,
                               int32_t h_rows, void* dst, int32_t dst_rows, int32_t batch, int32_t row_bytes, void* stream) {
  MOC_REQUIRE(cache && h && dst, "NULL routing window buffer");
  MOC_REQUIRE(batch > 0 && batch <= 65535 && cache_rows >= 0 && h_rows > 0 && dst_rows > 0 && dst_rows <= cache_rows + h_rows,
              "bad routing window");
  MOC_REQUIRE(row_bytes > 0 && row_bytes % 16 == 0 && cache_stride % 16 == 0 && h_stride % 16 == 0 &&
              ((reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0,
              "routing window rows must be 16-byte pieces");
  MOC_REQUIRE(static_cast<int64_t>(dst_rows) * row_bytes < (int64_t{1} << 31), "routing window too large");
  const int pieces = row_bytes / 16;
  // eight pieces per thread keep enough loads in flight; a single sequence is spread over more CTAs
  const int per_block = batch >= 32 ? 2048 : 256;
  dim3 grid(ceil_div(dst_rows * pieces, per_block), batch);
  roll_window_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(cache), cache_stride / 16, cache_rows, static_cast<const uint4*>(h), h_stride / 16, h_rows,
      static_cast<uint4*>(dst), dst_rows, pieces);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" int64_t moc_decode_step_arena_bytes(const moc_decode_step_desc* s) {
  StepArena a;
  return s ? carve(s, &a) : -1;
}

extern "C" int moc_decode_step(moc_decode_step_desc* s) {
  MOC_REQUIRE(s && s->routing_states && s->hidden && s->router_w && s->wq && s->wo && s->kv_bank && s->out && s->arena &&
              s->status, "NULL decode-step buffer");
  MOC_REQUIRE(s->attn.head_dim == kDD, "decode attention needs head_dim 64");
  MOC_REQUIRE(s->router.batch == s->attn.batch && s->out_dim > 0 && s->hidden_dim >= 0, "bad decode-step shape");
  StepArena a;
  carve(s, &a);
  moc_route_desc* r = &a.route;
  r->h = s->routing_states; r->w = s->router_w; r->bias = s->router_b;
  r->idx = s->idx; r->weights = s->weights; r->comb_idx = s->comb_idx; r->comb_w = s->comb_w;
  r->arena = a.route_arena; r->status = s->status; r->stream = s->stream;
  const int64_t rows = static_cast<int64_t>(s->attn.batch) * s->attn.n_q, d = width_of(s);
  const int64_t width = static_cast<int64_t>(s->attn.num_heads) * kDD;
  // The query projection needs nothing of the router: for a row or two in the router's launch, beside it from a dozen rows on, where
  // it takes longer than the events.
  cudaStream_t main = static_cast<cudaStream_t>(s->stream);
  cudaStream_t side = rows > 8 && s->side_stream ? static_cast<cudaStream_t>(s->side_stream) : main;
  if (side != main) MOC_TRY(order(main, side));
  Join join(side, main);
  const void* x;
  MOC_TRY(as_dtype(s->hidden, s->hidden_dtype, a.x, MOC_BF16, rows * d, side, &x));
  const bool few = rows <= 2 && d % 8 == 0 && d <= 1024 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(s->wq)) & 15) == 0;
  const RowsProduct q{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(s->wq), a.q, d, d, width,
                      static_cast<int>(rows), static_cast<int>(width), static_cast<int>(d)};
  RouteRun run;
  if (few) MOC_TRY(route_fwd_impl(r, &q, &run));
  if (!run.q_done) {
    Gemm gq(MOC_BF16, rows, width, d, true, true, MOC_BF16);
    MOC_TRY(moc_gemm(&gq, x, s->wq, a.q, nullptr, nullptr, s->status, side));
  }
  if (!few) MOC_TRY(route_fwd_impl(r, nullptr, &run));
  MOC_TRY(join.done());
  MOC_TRY(moc_decode_attn(&s->attn, a.q, s->kv_bank, s->bank_rows, s->comb_idx, s->comb_w, a.o, nullptr, s->status, s->stream));
  Gemm go(MOC_BF16, rows, s->out_dim, width, true, true, s->hidden_dtype);
  MOC_TRY(moc_gemm(&go, a.o, s->wo, s->out, nullptr, nullptr, s->status, s->stream));
  // (the cast of fp32 states; the queries where the router did not take them along; attention and output projection)
  s->launches = run.launches + (x != s->hidden ? 1 : 0) + (run.q_done ? 0 : 1) + 2;
  return MOC_OK;
}
