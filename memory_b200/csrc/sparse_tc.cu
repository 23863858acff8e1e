// Per-token chapter-sparse attention with one softmax over a token's selected chapters, on the tensor cores (bf16,
// head_dim 64, chapters of a multiple of 64 rows), for sm_100a.
//
//   out[t, hq] = softmax over all keys of the blocks listed for (t, hq / G) of (q . k * scale) times V
//
// Every (token, KV head) has its own list, so the work is turned round: an inverted index groups the (token, slot)
// pairs by key unit (64 or 128 keys), a CTA holds the unit's K / V tile and multiplies it with 128 gathered rows, a row
// being one query head of the group of one pair (sparse_tc_index.cuh).  Forward: each row's softmax over the unit
// gives a normalised fp32 partial output and its log-sum-exp; a second kernel merges a token's partials.  Backward:
// with the row's total log-sum-exp and delta = <o, do> known, units are independent: P = exp(s - lse),
// dS = P (dP - delta); dQ leaves as fp32 partials summed in slot order, dK / dV accumulate in tensor memory over all
// rows of the unit through one 128 x 128 product [P | dS]^T [dO | Q] whose diagonal blocks are dV and dK.
// Nothing is added with atomics.
//
// What the CUDA-core kernels of sparse_attn.cu did with these shapes (a warp per (token, head), K / V rows read once
// per token, dK / dV by fp32 atomics): 59.7 ms forward, 129 ms backward at 8,192 tokens x 16 heads on one KV head,
// 8 of 512 chapters of 128 rows.
#define MOC_KERNEL_TAG 6
#include <algorithm>

#include "sparse_tc_index.cuh"

namespace moc {
namespace sparse_tc {

constexpr int kRows = 128;                 // rows per tile
constexpr int kD = 64;
constexpr int kTileBytes = kRows * kD * 2; // 16 KiB
constexpr int kFwdThreads = 192;           // 4 row-owning warps, 1 that issues the products, 1 that loads
constexpr int kBwdThreads = 224;           // ... 2 that load
constexpr int kMma = 4, kLoad = 5;         // their places
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 32 bytes per thread: one full sector
__device__ __forceinline__ void st_v8(float* dst, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}
// D (+)= A B over KSTEPS steps of 16, issued by one elected lane of the converged warp
template <int KSTEPS, int ASTEP, int BSTEP>
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
#pragma unroll
  for (int kk = 0; kk < KSTEPS; ++kk) umma_ss_w(d, a + kk * ASTEP, b + kk * BSTEP, idesc, kk > 0 ? 1u : acc);
}

// Row r of a tile: pair `first + r / G` of the entries, query head r % G of the group.  Rows past the end repeat the
// tile's first pair (their results are not used).
struct RowRef { long long tok; int hq; };
__device__ __forceinline__ RowRef row_ref(const Shape& x, const int* entries, int first, int cnt, int r) {
  int i = r / x.G, g = r - i * x.G;
  if (i >= cnt) { i = 0; g = 0; }
  const int p = entries[first + i];
  const int bth = p / (x.S * x.U);
  const int tok = bth / x.H;
  return {tok, (bth - tok * x.H) * x.G + g};
}
// The 128 rows of a tile from a [tokens * HQ, 64] tensor.  The query heads of a pair lie behind each other: a box for each pair where
// they are whole swizzle groups that fill the tile; else every lane fetches four rows.
// A warp's gathers of four rows follow each other 41 ns apart (128 rows: 1.3 us a warp, whatever the SM's other warps issue), a box
// of 128 rows takes 0.2 us.  So groups of 16 heads go as 8 boxes instead of 32 gathers, and the loads have warps of their own: in
// the warp that issues the products they stood in front of the next tile's.  8,192 tokens x 16 heads on one KV head, 8 of 512
// chapters of 128 rows: forward 160 -> 116 us, backward 383 -> 252.
__host__ __device__ inline bool boxes(const Shape& x) { return x.G % 8 == 0 && kRows % x.G == 0; }
__device__ __forceinline__ void load_rows(const Shape& x, const int* entries, int first, int cnt, uint8_t* dst, const CUtensorMap* map,
                                          uint64_t* bar, int lane) {
  if (lane == 0) mbar_arrive_expect_tx(bar, kTileBytes);
  __syncwarp();
  if (boxes(x)) {
    if (lane < x.ppt) {
      const RowRef rr = row_ref(x, entries, first, cnt, lane * x.G);
      tma_load_2d(dst + lane * x.G * 128, map, bar, 0, static_cast<int>(rr.tok) * x.HQ + rr.hq);
    }
  } else {
    int row[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const RowRef rr = row_ref(x, entries, first, cnt, lane * 4 + i);
      row[i] = static_cast<int>(rr.tok) * x.HQ + rr.hq;
    }
    tma_gather4(dst + lane * 512, map, bar, 0, row[0], row[1], row[2], row[3]);
  }
  __syncwarp();
}

// ---- forward -------------------------------------------------------------------------------------------------
struct FwdParams {
  Shape x;
  Index ib;
  float* partial;      // [n_pairs * G, 64] normalised per-unit outputs, in entry order
  float* lse_rows;     // [n_pairs * G]
  int* status;
};
template <int KU> struct FwdCfg {
  static constexpr int kKv = KU * kD * 2;
  static constexpr int kStage = kTileBytes + 2 * kKv;
  static constexpr int kSmem = 2 * kStage + 1024;
  static constexpr int kCols = KU == 64 ? 128 : 256;       // S (P over its first half), then O
  static constexpr int kCtas = KU == 64 ? 3 : 2;
};

// Loads of tile i + 1 go out as soon as tile i - 1 has left the tensor pipe, so a tile's rows and K / V copies run under its
// predecessor's softmax; the second and third CTA of the SM fill the rest of the chain S -> softmax -> PV -> read-out.
template <int KU>
__global__ void __launch_bounds__(kFwdThreads, FwdCfg<KU>::kCtas)
sparse_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                     const __grid_constant__ CUtensorMap tmap_v, FwdParams p) {
  using C = FwdCfg<KU>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[2], empty[2], s_bar, p_bar, o_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const Shape& x = p.x;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < 2; ++i) { mbar_init(&full[i], 2); mbar_init(&empty[i], 1); }
    mbar_init(&s_bar, 1); mbar_init(&p_bar, 4); mbar_init(&o_bar, 1);
    fence_mbar_init();
    prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v);
  }
  if (warp == kMma) { tmem_alloc(&tmem_slot, C::kCols); tmem_relinquish(); tc_fence_before(); }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const int n_tiles = p.ib.totals[0];
  bool ok = true;
  uint32_t it = 0;

  if (warp == kLoad) {
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++it) {
      uint8_t* st = base + (it & 1) * C::kStage;
      const int bkt = p.ib.tile_bucket[tile], first = p.ib.tile_first[tile], cnt = p.ib.tile_cnt[tile];
      const int bh = bkt / x.M, u = bkt - bh * x.M, b = bh / x.H, h = bh - b * x.H;
      if (it >= 2) ok = mbar_wait_w(&empty[it & 1], ((it >> 1) & 1) ^ 1, &abort_flag, p.status);
      if (!ok) break;
      if (lane == 0) {
        mbar_arrive_expect_tx(&full[it & 1], 2 * C::kKv);
        tma_load_2d(st + kTileBytes, &tmap_k, &full[it & 1], h * kD, b * x.TK + u * KU);
        tma_load_2d(st + kTileBytes + C::kKv, &tmap_v, &full[it & 1], h * kD, b * x.TK + u * KU);
      }
      load_rows(x, p.ib.entries, first, cnt, st, &tmap_q, &full[it & 1], lane);
    }
  } else if (warp == kMma) {
    const uint32_t idesc_s = umma_idesc_bf16(kRows, KU, 0, 0);
    const uint32_t idesc_o = umma_idesc_bf16(kRows, kD, 0, 1);
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++it) {
      ok = mbar_wait_w(&full[it & 1], (it >> 1) & 1, &abort_flag, p.status);
      if (ok && it > 0) ok = mbar_wait_w(&o_bar, (it - 1) & 1, &abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      const uint32_t st = smem_u32(base) + (it & 1) * C::kStage;
      mma_ss<4, 2, 2>(tmem, umma_desc_sw128(st, 16, 1024), umma_desc_sw128(st + kTileBytes, 16, 1024), idesc_s, 0u);
      tc_commit_w(&s_bar);
      ok = mbar_wait_w(&p_bar, it & 1, &abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      const uint64_t vd = umma_desc_sw128(st + kTileBytes + C::kKv, 8192, 1024);
#pragma unroll
      for (int kk = 0; kk < KU / 16; ++kk) umma_ts_w(tmem + KU, tmem + kk * 8, vd + kk * 128, idesc_o, kk > 0 ? 1u : 0u);
      tc_commit_w(&o_bar);
      tc_commit_w(&empty[it & 1]);
    }
  } else {
    const int r = threadIdx.x;
    const uint32_t t_row = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++it) {
      const long long row0 = static_cast<long long>(p.ib.tile_first[tile]) * x.G;
      const bool valid = r < p.ib.tile_cnt[tile] * x.G;
      ok = mbar_wait_w(&s_bar, it & 1, &abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      uint32_t s[KU];
#pragma unroll
      for (int c = 0; c < KU / 32; ++c) tmem_ld32(t_row + c * 32, *reinterpret_cast<uint32_t(*)[32]>(s + c * 32));
      tmem_wait_ld();
      float m = __uint_as_float(s[0]);
#pragma unroll
      for (int c = 1; c < KU; ++c) m = fmaxf(m, __uint_as_float(s[c]));
      const float mm = m * x.scale_log2;
      float l0 = 0.f, l1 = 0.f;
#pragma unroll
      for (int c = 0; c < KU; c += 2) {
        const float e0 = ex2(fmaf(__uint_as_float(s[c]), x.scale_log2, -mm));
        const float e1 = ex2(fmaf(__uint_as_float(s[c + 1]), x.scale_log2, -mm));
        l0 += e0; l1 += e1;
        s[c / 2] = pack_bf16x2(e0, e1);
      }
#pragma unroll
      for (int c = 0; c < KU / 64; ++c) tmem_st32(t_row + c * 32, *reinterpret_cast<uint32_t(*)[32]>(s + c * 32));
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(&p_bar);
      const float l = l0 + l1, inv = 1.f / l;
      ok = mbar_wait_w(&o_bar, it & 1, &abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      float* dst = p.partial + (row0 + r) * kD;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t o[32];
        tmem_ld32(t_row + KU + half * 32, o);
        tmem_wait_ld();
        if (valid) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(o[8 * j + e]) * inv;
            st_v8(dst + half * 32 + j * 8, v);
          }
        }
      }
      if (valid) p.lse_rows[row0 + r] = fmaf(m, x.scale, logf(l));
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag) { for (int i = 0; i < 200; ++i) __nanosleep(1000); }
  if (warp == kMma) { tc_fence_after(); tmem_dealloc(tmem, C::kCols); }
}

// out[t, hq] = sum_s exp(lse_s - lse) partial_s, lse = log sum_s exp(lse_s); 16 lanes per (token, head), four columns
// each.  A token none of whose listed blocks exists gets zeros and lse = -inf.
__global__ void merge_kernel(Shape x, const int* __restrict__ pos, const float* __restrict__ partial,
                             const float* __restrict__ lse_rows, __nv_bfloat16* __restrict__ out,
                             float* __restrict__ lse) {
  const long long w = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 4;
  const int lane = threadIdx.x & 15;
  if (w >= static_cast<long long>(x.B) * x.TQ * x.HQ) return;
  const long long bt = w / x.HQ;
  const int hq = static_cast<int>(w - bt * x.HQ), h = hq / x.G, g = hq - h * x.G;
  const int n = x.S * x.U;
  const int* ps = pos + (bt * x.H + h) * n;
  float m = -INFINITY, den = 0.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = 0; s0 < n; s0 += 4) {
    float ls[4];
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = s0 + i < n ? ps[s0 + i] : -1;
      const long long row = static_cast<long long>(e < 0 ? 0 : e) * x.G + g;
      ls[i] = e < 0 ? -INFINITY : lse_rows[row] * kLog2e;
      v[i] = e < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : reinterpret_cast<const float4*>(partial + row * kD)[lane];
    }
    const float mn = max_nan(max_nan(max_nan(ls[0], ls[1]), max_nan(ls[2], ls[3])), m);
    if (mn == -INFINITY) continue;             // no listed block exists so far (a NaN sum is no reason to skip)
    const float a = ex2(m - mn);
    den *= a; acc.x *= a; acc.y *= a; acc.z *= a; acc.w *= a;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float f = ex2(ls[i] - mn);
      den += f;
      acc.x = fmaf(f, v[i].x, acc.x); acc.y = fmaf(f, v[i].y, acc.y);
      acc.z = fmaf(f, v[i].z, acc.z); acc.w = fmaf(f, v[i].w, acc.w);
    }
    m = mn;
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
  reinterpret_cast<uint2*>(out + w * kD)[lane] =
      make_uint2(pack_bf16x2(acc.x * inv, acc.y * inv), pack_bf16x2(acc.z * inv, acc.w * inv));
  if (lane == 0) lse[w] = m * 0.6931471805599453f + logf(den);
}

// ---- backward ------------------------------------------------------------------------------------------------
struct BwdParams {
  Shape x;
  Index ib;
  const float* lse;          // [B * TQ, HQ]
  const float* delta;        // [B * TQ, HQ]
  float* dq_partial;         // [KU / 64][n_pairs * G, 64], in entry order
  __nv_bfloat16 *d_k, *d_v;  // [B, TK, H, 64]
  float *acc_k, *acc_v;      // the same in fp32, added to in their place: a slice of a batch item's tokens; else NULL
  float* part;               // [parts][KU / 64][128, 64]: dV rows, then dK rows, of buckets cut into several items
  int* status;
};
constexpr int kKvBytes = 64 * kD * 2;                         // K or V of 64 keys
constexpr int kBwdTiles = 4 * kTileBytes + 2 * kTileBytes + 2 * kKvBytes;   // 2 x (dO, Q), P, dS, K, V: 112 KiB
constexpr int kBwdSmem = kBwdTiles + 256;                     // + barriers; two CTAs fill an SM's 228 KiB
constexpr uint32_t kColS = 0, kColDP = 64, kColD = 128;       // dQ takes S's columns

// The row tiles a CTA works through: items blockIdx.x, + gridDim.x, ... (an item is up to `chunk` row tiles of one
// bucket against 64 of its keys).  Control warp and row warps walk the same sequence.
struct TileIter {
  int w, bkt, half, part, t, nt, first, end;
  __device__ __forceinline__ void open(const BwdParams& p) {
    const int halves = p.x.KU / 64, base = w / halves;
    half = w - base * halves;
    bkt = p.ib.item_bucket[base];
    part = p.ib.item_part[base];
    const int t0 = p.ib.item_tile[base];
    end = p.ib.pair_off[bkt + 1];
    first = p.ib.pair_off[bkt] + t0 * p.x.ppt;
    nt = p.ib.item_nt[base];
    t = 0;
  }
  __device__ __forceinline__ int tile_first(const BwdParams& p) const { return first + t * p.x.ppt; }
  __device__ __forceinline__ int tile_cnt(const BwdParams& p) const { return min(p.x.ppt, end - tile_first(p)); }
  // b * TK + first key of the item's 64, and the KV head
  __device__ __forceinline__ int key_row(const BwdParams& p, int* h) const {
    const int bh = bkt / p.x.M, b = bh / p.x.H;
    *h = bh - b * p.x.H;
    return b * p.x.TK + (bkt - bh * p.x.M) * p.x.KU + half * 64;
  }
};

__global__ void __launch_bounds__(kBwdThreads, 2)
sparse_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_do,
                     const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                     BwdParams p) {
  extern __shared__ __align__(1024) uint8_t bwd_smem[];
  uint8_t* ps_s = bwd_smem + 4 * kTileBytes;      // [P | dS]: the two 64-row blocks of the MN-major A operand of D
  uint8_t* ds_s = ps_s + kTileBytes;
  uint8_t* k_s = ds_s + kTileBytes;
  uint8_t* v_s = k_s + kKvBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(bwd_smem + kBwdTiles);
  uint64_t *full = bars, *kv_bar = bars + 2, *sdp = bars + 3, *ds_ready = bars + 4, *done = bars + 5, *s_free = bars + 6,
           *d_read = bars + 7, *empty = bars + 8, *kv_empty = bars + 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  int* abort_flag = reinterpret_cast<int*>(bars + 12);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Shape& x = p.x;
  if ((smem_u32(bwd_smem) & 1023u) != 0) {        // the swizzled tiles need it; uniform over the grid
    if (threadIdx.x == 0) atomicMax(p.status, MOC_DEV_TIMEOUT | (MOC_KERNEL_TAG << 8) | (__LINE__ << 12));
    return;
  }
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) { mbar_init(&full[i], 2); mbar_init(&empty[i], 1); }
    mbar_init(kv_bar, 1); mbar_init(kv_empty, 1); mbar_init(sdp, 1);
    mbar_init(ds_ready, 4); mbar_init(done, 1); mbar_init(s_free, 4); mbar_init(d_read, 4);
    fence_mbar_init();
    prefetch_tmap(&tmap_q); prefetch_tmap(&tmap_do); prefetch_tmap(&tmap_k); prefetch_tmap(&tmap_v);
  }
  if (warp == kMma) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); tc_fence_before(); }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int n_work = p.ib.totals[1] * (x.KU / 64);
  bool ok = true;
  uint32_t it = 0, n = 0;                          // row tiles and non-empty items this CTA has run

  auto advance = [&](TileIter& i) {                 // next row tile, past empty items
    if (i.t + 1 < i.nt) { ++i.t; return; }
    do {
      i.w += gridDim.x;
      if (i.w >= n_work) return;
      i.open(p);
    } while (i.nt == 0);
  };
  auto start = [&]() {
    TileIter i;
    i.w = blockIdx.x; i.t = 0; i.nt = 0;
    if (i.w < n_work) { i.open(p); if (i.nt == 0) advance(i); }
    return i;
  };
  if (warp >= kLoad) {                              // the first loads dO and K / V, the second Q
    for (TileIter cur = start(); cur.w < n_work; advance(cur), ++it) {
      if (it >= 2) ok = mbar_wait_w(&empty[it & 1], ((it >> 1) & 1) ^ 1, abort_flag, p.status);
      if (!ok) break;
      uint8_t* st = bwd_smem + (it & 1) * 2 * kTileBytes;
      if (warp == kLoad) load_rows(x, p.ib.entries, cur.tile_first(p), cur.tile_cnt(p), st, &tmap_do, &full[it & 1], lane);
      else load_rows(x, p.ib.entries, cur.tile_first(p), cur.tile_cnt(p), st + kTileBytes, &tmap_q, &full[it & 1], lane);
      if (warp == kLoad && cur.t == 0) {            // behind the rows: it may wait for the last item's products
        if (n > 0) ok = mbar_wait_w(kv_empty, (n - 1) & 1, abort_flag, p.status);
        if (!ok) break;
        if (lane == 0) {
          int h;
          const int row = cur.key_row(p, &h);
          mbar_arrive_expect_tx(kv_bar, 2 * kKvBytes);
          tma_load_2d(k_s, &tmap_k, kv_bar, h * kD, row);
          tma_load_2d(v_s, &tmap_v, kv_bar, h * kD, row);
        }
        __syncwarp();
        ++n;
      }
    }
  } else if (warp == kMma) {
    const uint32_t idesc_kk = umma_idesc_bf16(kRows, 64, 0, 0);      // S, dP: both operands K-major
    const uint32_t idesc_dq = umma_idesc_bf16(kRows, kD, 0, 1);      // dQ = dS K: K tile as MN-major B
    const uint32_t idesc_d = umma_idesc_bf16(128, 128, 1, 1);        // D = [P | dS]^T [dO | Q]
    const uint64_t k_desc = umma_desc_sw128(smem_u32(k_s), 16, 1024), v_desc = umma_desc_sw128(smem_u32(v_s), 16, 1024);
    const uint64_t kmn_desc = umma_desc_sw128(smem_u32(k_s), 8192, 1024);
    const uint64_t ds_desc = umma_desc_sw128(smem_u32(ds_s), 16, 1024);
    const uint64_t a_d = umma_desc_sw128(smem_u32(ps_s), kTileBytes, 1024);
    for (TileIter cur = start(); cur.w < n_work; advance(cur)) {
      if (cur.t == 0) ok = mbar_wait_w(kv_bar, n & 1, abort_flag, p.status);
      ok = ok && mbar_wait_w(&full[it & 1], (it >> 1) & 1, abort_flag, p.status);
      if (ok && it > 0) ok = mbar_wait_w(s_free, (it - 1) & 1, abort_flag, p.status);   // dQ of the last tile is read
      if (!ok) break;
      tc_fence_after();
      const uint32_t st = smem_u32(bwd_smem) + (it & 1) * 2 * kTileBytes;
      mma_ss<4, 2, 2>(tmem + kColS, umma_desc_sw128(st + kTileBytes, 16, 1024), k_desc, idesc_kk, 0u);
      mma_ss<4, 2, 2>(tmem + kColDP, umma_desc_sw128(st, 16, 1024), v_desc, idesc_kk, 0u);
      tc_commit_w(sdp);
      ok = mbar_wait_w(ds_ready, it & 1, abort_flag, p.status);
      if (ok && cur.t == 0 && n > 0) ok = mbar_wait_w(d_read, (n - 1) & 1, abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      mma_ss<4, 2, 128>(tmem + kColS, ds_desc, kmn_desc, idesc_dq, 0u);
      mma_ss<8, 128, 128>(tmem + kColD, a_d, umma_desc_sw128(st, kTileBytes, 1024), idesc_d, cur.t > 0 ? 1u : 0u);
      tc_commit_w(done);
      tc_commit_w(&empty[it & 1]);
      if (cur.t + 1 == cur.nt) { tc_commit_w(kv_empty); ++n; }
      ++it;
    }
  } else {
    const int r = threadIdx.x;
    const uint32_t t_row = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    // where a key row of an item's dK (threads 64..127) or dV starts
    auto out_at = [&](const TileIter& i) {
      int h;
      const long long row = i.key_row(p, &h);
      return ((row + (r & 63)) * x.H + h) * kD;
    };
    auto advance_rows = [&](TileIter& i) {               // as above; the dK / dV rows of empty items are zero-filled
      if (i.t + 1 < i.nt) { ++i.t; return; }
      while (true) {
        i.w += gridDim.x;
        if (i.w >= n_work) return;
        i.open(p);
        if (i.nt > 0) return;
        if (p.acc_k != nullptr) continue;
        uint4* dst = reinterpret_cast<uint4*>((r >= 64 ? p.d_k : p.d_v) + out_at(i));
#pragma unroll
        for (int e = 0; e < 8; ++e) dst[e] = make_uint4(0u, 0u, 0u, 0u);
      }
    };
    struct Meta { float nl2, delta; bool valid; };
    auto fetch = [&](const TileIter& i) {           // requested a tile ahead: two dependent global loads
      const int first = i.tile_first(p), cnt = i.tile_cnt(p);
      const RowRef rr = row_ref(x, p.ib.entries, first, cnt, r);
      const long long at = rr.tok * x.HQ + rr.hq;
      return Meta{-p.lse[at] * kLog2e, p.delta[at], r < cnt * x.G};
    };
    TileIter cur;
    cur.w = static_cast<int>(blockIdx.x) - static_cast<int>(gridDim.x); cur.t = 0; cur.nt = 0;
    advance_rows(cur);
    Meta next_m = {0.f, 0.f, false};
    if (cur.w < n_work) next_m = fetch(cur);
    while (cur.w < n_work && ok) {
      const Meta m = next_m;
      ok = mbar_wait_w(sdp, it & 1, abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t s[32], d[32];
        tmem_ld32(t_row + kColS + half * 32, s);
        tmem_ld32(t_row + kColDP + half * 32, d);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t a[4], g[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = j * 8 + 2 * e;
            const float p0 = ex2(fmaf(__uint_as_float(s[c]), x.scale_log2, m.nl2));
            const float p1 = ex2(fmaf(__uint_as_float(s[c + 1]), x.scale_log2, m.nl2));
            a[e] = m.valid ? pack_bf16x2(p0, p1) : 0u;
            g[e] = m.valid ? pack_bf16x2(p0 * (__uint_as_float(d[c]) - m.delta), p1 * (__uint_as_float(d[c + 1]) - m.delta))
                           : 0u;
          }
          const int chunk = ((half * 4 + j) ^ (r & 7)) << 4;
          *reinterpret_cast<uint4*>(ps_s + r * 128 + chunk) = make_uint4(a[0], a[1], a[2], a[3]);
          *reinterpret_cast<uint4*>(ds_s + r * 128 + chunk) = make_uint4(g[0], g[1], g[2], g[3]);
        }
      }
      tc_fence_before();
      fence_proxy_async();
      mbar_arrive_warp(ds_ready);
      const bool last = cur.t + 1 == cur.nt;
      TileIter nxt = cur;
      advance_rows(nxt);
      if (nxt.w < n_work) next_m = fetch(nxt);
      ok = mbar_wait_w(done, it & 1, abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t o0[32], o1[32];
        tmem_ld32(t_row + kColS, o0);
        tmem_ld32(t_row + kColS + 32, o1);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive_warp(s_free);
        if (m.valid) {
          float* dst = p.dq_partial +
                       (static_cast<long long>(cur.half) * x.n_pairs * x.G + static_cast<long long>(cur.tile_first(p)) * x.G + r) * kD;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(j < 4 ? o0[8 * j + e] : o1[8 * (j - 4) + e]) * x.scale;
            st_v8(dst + j * 8, v);
          }
        }
      }
      if (last) {
        const float f = r >= 64 ? x.scale : 1.f;
        uint32_t o0[32], o1[32];
        tmem_ld32(t_row + kColD + (r >= 64 ? 64 : 0), o0);
        tmem_ld32(t_row + kColD + (r >= 64 ? 64 : 0) + 32, o1);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive_warp(d_read);
        if (cur.part < 0 && p.acc_k != nullptr) {      // (these rows are this item's alone)
          float* dst = (r >= 64 ? p.acc_k : p.acc_v) + out_at(cur);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 a0 = reinterpret_cast<const float4*>(dst + j * 8)[0], a1 = reinterpret_cast<const float4*>(dst + j * 8)[1];
            const uint32_t* o = j < 4 ? o0 + 8 * j : o1 + 8 * (j - 4);
            const float v[8] = {fmaf(__uint_as_float(o[0]), f, a0.x), fmaf(__uint_as_float(o[1]), f, a0.y),
                                fmaf(__uint_as_float(o[2]), f, a0.z), fmaf(__uint_as_float(o[3]), f, a0.w),
                                fmaf(__uint_as_float(o[4]), f, a1.x), fmaf(__uint_as_float(o[5]), f, a1.y),
                                fmaf(__uint_as_float(o[6]), f, a1.z), fmaf(__uint_as_float(o[7]), f, a1.w)};
            st_v8(dst + j * 8, v);
          }
        } else if (cur.part < 0) {
          uint4* dst = reinterpret_cast<uint4*>((r >= 64 ? p.d_k : p.d_v) + out_at(cur));
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t* o = j < 4 ? o0 + 8 * j : o1 + 8 * (j - 4);
            dst[j] = make_uint4(pack_bf16x2(__uint_as_float(o[0]) * f, __uint_as_float(o[1]) * f),
                                pack_bf16x2(__uint_as_float(o[2]) * f, __uint_as_float(o[3]) * f),
                                pack_bf16x2(__uint_as_float(o[4]) * f, __uint_as_float(o[5]) * f),
                                pack_bf16x2(__uint_as_float(o[6]) * f, __uint_as_float(o[7]) * f));
          }
        } else {
          float* dst = p.part + ((static_cast<long long>(cur.part) * (x.KU / 64) + cur.half) * 128 + r) * kD;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(j < 4 ? o0[8 * j + e] : o1[8 * (j - 4) + e]) * f;
            st_v8(dst + j * 8, v);
          }
        }
      }
      ++it;
      cur = nxt;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) { for (int i = 0; i < 200; ++i) __nanosleep(1000); }
  if (warp == kMma) { tc_fence_after(); tmem_dealloc(tmem, 256); }
}

// dK / dV of the buckets that were cut into several items: their fp32 partials in item order.  One CTA per bucket.
__global__ void part_sum_kernel(Shape x, Index ib, const float* __restrict__ part, __nv_bfloat16* __restrict__ d_k,
                                __nv_bfloat16* __restrict__ d_v, float* __restrict__ acc_k, float* __restrict__ acc_v) {
  const int bkt = blockIdx.x;
  const int p0 = ib.part_off[bkt], n = ib.part_off[bkt + 1] - p0;
  if (n == 0) return;
  const int halves = x.KU / 64, bh = bkt / x.M, b = bh / x.H, h = bh - b * x.H;
  const long long row0 = static_cast<long long>(b) * x.TK + static_cast<long long>(bkt - bh * x.M) * x.KU;
  for (int i = threadIdx.x; i < halves * 128 * 16; i += blockDim.x) {
    const int c4 = i & 15, r = (i >> 4) & 127, half = i >> 11;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < n; ++k) {
      const float4 v = reinterpret_cast<const float4*>(part + ((static_cast<long long>(p0 + k) * halves + half) * 128 + r) * kD)[c4];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    const long long at = ((row0 + half * 64 + (r & 63)) * x.H + h) * kD;
    if (acc_k != nullptr) {
      float4* dst = reinterpret_cast<float4*>((r >= 64 ? acc_k : acc_v) + at) + c4;
      *dst = make_float4(dst->x + acc.x, dst->y + acc.y, dst->z + acc.z, dst->w + acc.w);
    } else {
      reinterpret_cast<uint2*>((r >= 64 ? d_k : d_v) + at)[c4] = make_uint2(pack_bf16x2(acc.x, acc.y), pack_bf16x2(acc.z, acc.w));
    }
  }
}

// dq[t, hq] = sum of the partials of its pairs, in slot order
__global__ void dq_sum_kernel(Shape x, const int* __restrict__ pos, const float* __restrict__ partial,
                              __nv_bfloat16* __restrict__ d_q) {
  const long long w = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 4;
  const int lane = threadIdx.x & 15;
  if (w >= static_cast<long long>(x.B) * x.TQ * x.HQ) return;
  const long long bt = w / x.HQ;
  const int hq = static_cast<int>(w - bt * x.HQ), h = hq / x.G, g = hq - h * x.G;
  const int n = x.S * x.U, halves = x.KU / 64;
  const int* ps = pos + (bt * x.H + h) * n;
  const long long stride = x.n_pairs * x.G;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  // eight rows requested together: their places, then their values, then the sum in slot order (537 MB of partials: 109 -> 79 us,
  // 6.8 TB/s; the compiler had kept each load behind the test of the one before)
  const int total = n * halves, sh = halves - 1;             // (halves is 1 or 2)
  for (int i0 = 0; i0 < total; i0 += 8) {
    int e[8];
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = i0 + i < total ? ps[(i0 + i) >> sh] : -1;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float* src = partial + (((i0 + i) & sh) * stride + static_cast<long long>(e[i]) * x.G + g) * kD;
      v[i] = e[i] < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcs(reinterpret_cast<const float4*>(src) + lane);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) { acc.x += v[i].x; acc.y += v[i].y; acc.z += v[i].z; acc.w += v[i].w; }
  }
  reinterpret_cast<uint2*>(d_q + w * kD)[lane] = make_uint2(pack_bf16x2(acc.x, acc.y), pack_bf16x2(acc.z, acc.w));
}

// ---- host ----------------------------------------------------------------------------------------------------
static int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
  }
  return n;
}

static int make_shape(const moc_sparse_attn_shape* s, Shape* x) {
  MOC_REQUIRE(s != nullptr, "shape is NULL");
  MOC_REQUIRE(s->dtype == MOC_BF16 && s->head_dim == kD && s->block_size > 0 && s->block_size % 64 == 0,
              "the tensor-core sparse attention takes bf16, head_dim 64 and chapters of a multiple of 64 rows");
  MOC_REQUIRE(s->batch > 0 && s->tq > 0 && s->tk > 0 && s->n_select > 0, "empty problem");
  MOC_REQUIRE(s->h > 0 && s->hq % s->h == 0 && s->hq / s->h <= kRows, "HQ must be a multiple of H, at most 128 times it");
  MOC_REQUIRE(s->tk % s->block_size == 0, "TK must be divisible by block_size (chapter size) for clean chapter blocks.");
  x->B = s->batch; x->TQ = s->tq; x->TK = s->tk; x->HQ = s->hq; x->H = s->h; x->G = s->hq / s->h; x->S = s->n_select;
  x->KU = s->block_size % 128 == 0 ? 128 : 64;      // 128-key units halve the partial outputs per key
  x->U = s->block_size / x->KU; x->M = s->tk / x->KU;
  x->ppt = kRows / x->G;
  x->n_pairs = static_cast<long long>(s->batch) * s->tq * s->h * s->n_select * x->U;
  x->n_buckets = static_cast<long long>(s->batch) * s->h * x->M;
  // backward items: about three per resident CTA when the buckets are too few or too uneven to fill the chip
  x->chunk = 1;
  x->chunk = static_cast<int>(std::max<long long>(1, max_tiles(*x) * (x->KU / 64) / (sm_count() * 2 * 3)));
  x->scale = s->scale; x->scale_log2 = s->scale * kLog2e;
  return MOC_OK;
}

// Fixed-size pieces of a problem.  Its scratch grows with the listed (token, slot) pairs: 512 bytes a pair and query head
// with 128-key units, 0.54 GB for 8,192 tokens x 8 blocks x 16 heads on one KV head.  What needs more than kScratchLimit
// runs in slices that share one scratch: whole batch items where one fits, else runs of one item's tokens, whose dK / dV
// add up in fp32.  The limit keeps problems of the size measured whole, and a slice fills the chip many times over.
constexpr int64_t kScratchLimit = int64_t{1} << 30;
struct Sizes { int64_t index, fwd, bwd; };
static bool sizes_of(const Shape& x, Sizes* z) {          // false: beyond 32-bit row and pair ids
  Index ib;
  z->index = static_cast<int64_t>(carve(x, nullptr, &ib));
  const int64_t rows = x.n_pairs * x.G, toks = static_cast<int64_t>(x.B) * x.TQ * x.HQ;
  z->fwd = rows * (kD + 1) * 4 + 64;
  z->bwd = rows * (x.KU / 64) * kD * 4 + max_parts(x) * (x.KU / 64) * 128 * kD * 4 + toks * 4 + 64;
  return x.n_pairs < (1ll << 30) && x.n_buckets < (1ll << 28) && toks < (1ll << 31) &&
         static_cast<long long>(x.B) * x.TK < (1ll << 31);
}
struct Slices { int items, tokens; };                     // batch items and tokens of a slice (the last may have fewer)
static int slice(const moc_sparse_attn_shape* s, Slices* p, Sizes* z) {
  MOC_REQUIRE(s != nullptr, "shape is NULL");
  p->items = s->batch; p->tokens = s->tq;
  bool ids = false;
  auto size = [&](int items, int tokens, Sizes* out) -> int {
    moc_sparse_attn_shape part = *s;
    part.batch = items; part.tq = tokens;
    Shape x;
    const int rc = make_shape(&part, &x);
    if (rc == MOC_OK) ids = sizes_of(x, out);
    return rc;
  };
  for (;;) {
    const int rc = size(p->items, p->tokens, z);
    if (rc != MOC_OK) return rc;
    const int64_t bytes = std::max(z->fwd, z->bwd);
    if ((ids && bytes <= kScratchLimit) || (p->items == 1 && p->tokens == 1)) break;
    int& n = p->items > 1 ? p->items : p->tokens;         // equal shares of as many pieces as the bytes ask for
    const int64_t total = p->items > 1 ? s->batch : s->tq, now = (total + n - 1) / n;
    const int64_t pieces = std::max(now + 1, now * ((bytes + kScratchLimit - 1) / kScratchLimit));
    n = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(n - 1, (total + pieces - 1) / pieces)));
  }
  MOC_REQUIRE(ids, "problem too large for 32-bit row ids");
  // the tail can need more than a full slice: its buckets may be cut finer
  const int tail_items = s->batch % p->items, tail_tokens = s->tq % p->tokens;
  if (tail_items || tail_tokens) {
    Sizes t;
    const int rc = size(tail_items ? tail_items : p->items, tail_tokens ? tail_tokens : p->tokens, &t);
    if (rc != MOC_OK) return rc;
    z->index = std::max(z->index, t.index); z->fwd = std::max(z->fwd, t.fwd); z->bwd = std::max(z->bwd, t.bwd);
  }
  if (p->tokens < s->tq) z->bwd += 2 * static_cast<int64_t>(s->tk) * s->h * kD * 4;       // fp32 dK / dV of one item
  return MOC_OK;
}
// what a slice starts with: its shape, its first (batch item, token) and (batch item, key row)
template <typename Fn> static int for_slices(const moc_sparse_attn_shape* s, const Slices& p, Fn fn) {
  for (int b0 = 0; b0 < s->batch; b0 += p.items) {
    for (int t0 = 0; t0 < s->tq; t0 += p.tokens) {
      moc_sparse_attn_shape part = *s;
      part.batch = std::min(p.items, s->batch - b0); part.tq = std::min(p.tokens, s->tq - t0);
      Shape x;
      int rc = make_shape(&part, &x);
      if (rc != MOC_OK) return rc;
      rc = fn(x, static_cast<int64_t>(b0) * s->tq + t0, static_cast<int64_t>(b0) * s->tk, t0 == 0, t0 + part.tq == s->tq);
      if (rc != MOC_OK) return rc;
    }
  }
  return MOC_OK;
}
static int kv_maps(const Shape& x, const void* k, const void* v, int rows, CUtensorMap* mk, CUtensorMap* mv) {
  const uint64_t n = static_cast<uint64_t>(x.B) * x.TK, cols = static_cast<uint64_t>(x.H) * kD;
  const int rc = make_tmap_bf16_2d(mk, k, n, cols, cols, rows, kD);
  return rc != MOC_OK ? rc : make_tmap_bf16_2d(mv, v, n, cols, cols, rows, kD);
}
static int row_map(const Shape& x, const void* q, CUtensorMap* m) {
  return make_tmap_bf16_2d(m, q, static_cast<uint64_t>(x.B) * x.TQ * x.HQ, kD, kD, boxes(x) ? x.G : 1, kD);
}

template <int KU>
static int launch_fwd(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const FwdParams& p,
                      cudaStream_t st) {
  using C = FwdCfg<KU>;
  MOC_CUDA_OK(cudaFuncSetAttribute(sparse_fwd_tc_kernel<KU>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
  const long long grid = std::min<long long>(max_tiles(p.x), static_cast<long long>(sm_count()) * C::kCtas);
  sparse_fwd_tc_kernel<KU><<<static_cast<int>(grid), kFwdThreads, C::kSmem, st>>>(mq, mk, mv, p);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

}  // namespace sparse_tc
}  // namespace moc

using namespace moc;
using namespace moc::sparse_tc;

extern "C" int moc_sparse_attn_tc_sizes(const moc_sparse_attn_shape* s, int64_t* index_bytes, int64_t* fwd_bytes,
                                        int64_t* bwd_bytes) {
  Slices p;
  Sizes z;
  const int rc = slice(s, &p, &z);
  if (rc != MOC_OK) return rc;
  MOC_REQUIRE(index_bytes && fwd_bytes && bwd_bytes, "NULL argument");
  *index_bytes = z.index; *fwd_bytes = z.fwd; *bwd_bytes = z.bwd;
  return MOC_OK;
}

extern "C" int moc_sparse_attn_tc_fwd(const moc_sparse_attn_shape* s, const void* q_, const void* k_, const void* v_,
                                      const int32_t* block_indices, void* index, void* scratch, void* o_, float* lse,
                                      int32_t* status, void* stream) {
  Slices sl;
  Sizes z;
  const int rc = slice(s, &sl, &z);
  if (rc != MOC_OK) return rc;
  MOC_REQUIRE(q_ && k_ && v_ && block_indices && index && scratch && o_ && lse && status, "NULL buffer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  using bf16 = __nv_bfloat16;
  return for_slices(s, sl, [&](const Shape& x, int64_t tok, int64_t key, bool, bool) -> int {
    const bf16 *q = static_cast<const bf16*>(q_) + tok * x.HQ * kD, *k = static_cast<const bf16*>(k_) + key * x.H * kD,
               *v = static_cast<const bf16*>(v_) + key * x.H * kD;
    FwdParams p;
    p.x = x;
    int rc;
    CUtensorMap mq, mk, mv;
    if ((rc = row_map(x, q, &mq)) != MOC_OK || (rc = kv_maps(x, k, v, x.KU, &mk, &mv)) != MOC_OK) return rc;
    carve(x, static_cast<int*>(index), &p.ib);
    if ((rc = build_index(block_indices + tok * x.H * x.S, x, p.ib, status, st)) != MOC_OK) return rc;
    p.partial = static_cast<float*>(scratch);
    p.lse_rows = p.partial + x.n_pairs * x.G * kD;
    p.status = status;
    rc = x.KU == 128 ? launch_fwd<128>(mq, mk, mv, p, st) : launch_fwd<64>(mq, mk, mv, p, st);
    if (rc != MOC_OK) return rc;
    const long long threads = static_cast<long long>(x.B) * x.TQ * x.HQ * 16;
    merge_kernel<<<static_cast<int>((threads + 255) / 256), 256, 0, st>>>(
        x, p.ib.pos, p.partial, p.lse_rows, static_cast<bf16*>(o_) + tok * x.HQ * kD, lse + tok * x.HQ);
    MOC_CUDA_OK(cudaGetLastError());
    return MOC_OK;
  });
}

extern "C" int moc_sparse_attn_tc_bwd(const moc_sparse_attn_shape* s, const void* q_, const void* k_, const void* v_,
                                      const int32_t* block_indices, void* index, int32_t have_index, void* scratch,
                                      const void* o_, const float* lse, const void* d_o_, void* d_q, void* d_k, void* d_v,
                                      int32_t* status, void* stream) {
  Slices sl;
  Sizes z;
  const int rc = slice(s, &sl, &z);
  if (rc != MOC_OK) return rc;
  MOC_REQUIRE(q_ && k_ && v_ && block_indices && index && scratch && o_ && lse && d_o_ && d_q && d_k && d_v && status,
              "NULL buffer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  using bf16 = __nv_bfloat16;
  const bool whole = sl.items == s->batch && sl.tokens == s->tq, add = sl.tokens < s->tq;
  return for_slices(s, sl, [&](const Shape& x, int64_t tok, int64_t key, bool first, bool last) -> int {
    const int64_t row = tok * x.HQ, kv = key * x.H * kD, n_kv = static_cast<int64_t>(x.B) * x.TK * x.H * kD;
    const bf16 *q = static_cast<const bf16*>(q_) + row * kD, *k = static_cast<const bf16*>(k_) + kv,
               *v = static_cast<const bf16*>(v_) + kv, *o = static_cast<const bf16*>(o_) + row * kD,
               *d_o = static_cast<const bf16*>(d_o_) + row * kD;
    BwdParams p;
    p.x = x;
    int rc;
    CUtensorMap mq, mdo, mk, mv;
    if ((rc = row_map(x, q, &mq)) != MOC_OK || (rc = row_map(x, d_o, &mdo)) != MOC_OK ||
        (rc = kv_maps(x, k, v, 64, &mk, &mv)) != MOC_OK) return rc;
    carve(x, static_cast<int*>(index), &p.ib);
    if (!(have_index && whole) && (rc = build_index(block_indices + tok * x.H * x.S, x, p.ib, status, st)) != MOC_OK) return rc;
    const int halves = x.KU / 64;
    p.acc_k = p.acc_v = nullptr;
    p.dq_partial = static_cast<float*>(scratch);
    if (add) {                                  // a slice is part of one item, whose sums stand before the rest
      p.acc_k = p.dq_partial; p.acc_v = p.acc_k + n_kv;
      p.dq_partial = p.acc_v + n_kv;
      if (first) MOC_CUDA_OK(cudaMemsetAsync(p.acc_k, 0, static_cast<size_t>(2 * n_kv) * 4, st));
    }
    p.part = p.dq_partial + x.n_pairs * x.G * halves * kD;
    float* delta = p.part + max_parts(x) * halves * 128 * kD;
    p.d_k = static_cast<bf16*>(d_k) + kv; p.d_v = static_cast<bf16*>(d_v) + kv;
    p.lse = lse + row; p.delta = delta;
    p.status = status;
    rc = moc_row_dot(o, d_o, MOC_BF16, delta, static_cast<int64_t>(x.B) * x.TQ * x.HQ, kD, stream);
    if (rc != MOC_OK) return rc;
    MOC_CUDA_OK(cudaFuncSetAttribute(sparse_bwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem));
    const long long grid = std::min<long long>(max_items(x) * halves, static_cast<long long>(sm_count()) * 2);
    sparse_bwd_tc_kernel<<<static_cast<int>(grid), kBwdThreads, kBwdSmem, st>>>(mq, mdo, mk, mv, p);
    part_sum_kernel<<<static_cast<int>(x.n_buckets), 256, 0, st>>>(x, p.ib, p.part, p.d_k, p.d_v, p.acc_k, p.acc_v);
    const long long threads = static_cast<long long>(x.B) * x.TQ * x.HQ * 16;
    dq_sum_kernel<<<static_cast<int>((threads + 255) / 256), 256, 0, st>>>(x, p.ib.pos, p.dq_partial,
                                                                           static_cast<bf16*>(d_q) + row * kD);
    MOC_CUDA_OK(cudaGetLastError());
    if (add && last) {
      if ((rc = moc_cast_f32_to_bf16(p.acc_k, p.d_k, n_kv, stream)) != MOC_OK) return rc;
      return moc_cast_f32_to_bf16(p.acc_v, p.d_v, n_kv, stream);
    }
    return MOC_OK;
  });
}
