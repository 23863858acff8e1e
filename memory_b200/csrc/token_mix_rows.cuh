// The token mixture for chapters with few (token, slot) pairs: kernels on the matrix instructions of single warps, beside the
// tcgen05 kernels of token_mix_tc.cu, which include this file (the shapes, the inverted index and the sums over slots are theirs).
//
// A routed bank of thousands of chapters leaves a chapter a few dozen pairs: 32 at 8,192 tokens x 16 of 4,096, one or two for a
// prompt.  A 128-row tcgen05 tile is then three quarters padding, and its chain -- gather, product, tensor memory, softmax,
// product, read-out, with a barrier at every turn -- takes 3.6 us (forward) and 7 us (backward) whatever the rows are, with two to
// four of them at a time on an SM.  Here a step is 16 or 32 pairs, the scores stay in the registers that multiplied them, and a
// warp's chain is a few hundred instructions long.
#pragma once

namespace moc {
namespace {

// Fragments of 128-byte rows (64 bf16) in 128-byte-swizzled tiles, for ldmatrix: a lane's place in a tile.  Tiles start on 1 KiB,
// so 16 rows on is + 2048 and 16 columns on is ^ 32 (bits 5 and 6 of the address hold nothing but the swizzled column).
// 16 rows x 16 columns in the order of an A operand (rows 0-7, rows 8-15, then the next 8 columns) ...
__device__ __forceinline__ uint32_t frag_a(int lane) { return (lane & 15) * 128 + (((lane >> 4) ^ (lane & 7)) << 4); }
// ... and in the order of two B operands whose columns are rows of the tile (rows 0-7 with both column halves, then 8-15)
__device__ __forceinline__ uint32_t frag_b(int lane) {
  return ((lane & 7) + ((lane >> 4) << 3)) * 128 + ((((lane >> 3) & 1) ^ (lane & 7)) << 4);
}
struct PairDiv { FastDiv s, hi; };       // pair number -> (token row, list) -> token row
// token row and slot of a pair
__device__ __forceinline__ int token_of(const PairDiv& d, int pair) { return div_of(div_of(pair, d.s), d.hi); }
__device__ __forceinline__ int slot_of(const PairDiv& d, int pair) { return pair - div_of(pair, d.s) * d.s.d; }

// A CTA of the backward walks the (chapter bucket, head) items first, first + step, ...: whole chapters, whose dK and dV it sums.
// One head an item: buckets differ (at 32 pairs on average the largest have 300 to 500), and what evens them out is that
// each CTA has many.  8,192 tokens, in-use buckets: runs of 12 / 4 / 2 / 1 heads 1,008 / 721 / 658 / 605 us; a CTA for each
// item instead of 444 that walk them 793 (every item then starts cold).
struct RowItems {
  const int* bucket_off;
  int n;
  PairDiv div;
};
struct RowGroup {
  int item, head, first, n, kv_row;      // n = 0: no item is left
  // first item with pairs at or after `item`; `empty` is told of the ones without on the way.  heads: of all lists together
  template <class Empty>
  __device__ __forceinline__ void seek(const MixShape& x, int heads, const RowItems& items, int step, Empty empty) {
    const int per_list = heads / x.HI;
    for (n = 0; item < items.n; item += step) {
      const int bkt = item / per_list, c = bkt % x.M, bh = bkt / x.M, hi = bh % x.HI;
      head = hi * per_list + (item - bkt * per_list);
      kv_row = bh / x.HI * x.TK + c * kKeys;
      first = items.bucket_off[bkt];
      n = items.bucket_off[bkt + 1] - first;
      if (n > 0) break;
      empty(*this);
    }
  }
};

// ---- forward -------------------------------------------------------------------------------------------------
// A warp an item (a tile of up to 128 pairs of one chapter, and a head): its chapter's K / V tile (TMA), blocks of 16 query rows
// (four rows a TMA gather, the next block's under this one's products), S and P in registers, the outputs through the query block's
// place as whole lines.  Nothing is shared between warps, so none waits for another.  10 warps an SM (20 KiB each); bound by their
// instructions' latency (36 % of issue slots) at 32 pairs a chapter and by HBM at one.  Two warps on one tile (16 of them an SM) were
// no faster at 32 pairs and slower below: an odd block leaves one of them idle.
// Tiles and not whole chapters: a warp that walks a popular chapter alone is what the call waits for.  8,192 tokens x 16 of 4,096
// chapters, us with the sum over slots, whole chapters and tiles: uniform picks 272 and 273, a router's (up to 452 pairs a chapter) 340
// and 312, all picks in 32 chapters 957 and 211.
constexpr int kRowFwdWarps = 2;
constexpr int kRowFwdRows = 16;                                    // pairs of a step
constexpr int kRowFwdBytes = kRowFwdRows * kD * 2;                 // 2 KiB
constexpr int kRowFwdWarpBytes = 2 * kTileKV + 2 * kRowFwdBytes;   // K, V, two query blocks (the older one holds the outputs)
constexpr int kRowFwdSmem = kRowFwdWarps * kRowFwdWarpBytes + 1024;
constexpr int kRowFwdCtas = 5;                                     // an SM

__global__ void __launch_bounds__(kRowFwdWarps * 32, kRowFwdCtas)
token_mix_rows_fwd_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                          const __grid_constant__ CUtensorMap tmap_q, MixFwdParams p, PairDiv div) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t kv_bar[kRowFwdWarps], q_bar[kRowFwdWarps][2];
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023)) + warp * kRowFwdWarpBytes;
  const uint32_t k_s = smem_u32(base), v_s = k_s + kTileKV, q_s = v_s + kTileKV;
  const MixShape& x = p.x;
  const int G = x.HQ / x.HK, no_row = x.B * x.TQ;
  if (p.ask && tiles_full(p.totals)) return;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < kRowFwdWarps; ++i) { mbar_init(&kv_bar[i], 1); mbar_init(&q_bar[i][0], 1); mbar_init(&q_bar[i][1], 1); }
    fence_mbar_init();
  }
  __syncthreads();
  const int step = gridDim.x * kRowFwdWarps, per_list = x.HQ / x.HI, n_items = p.totals[kTiles] * per_list;
  auto open = [&](int item) {
    RowGroup g;
    g.item = item; g.n = 0;
    if (item < n_items) {
      const int tile = item / per_list, bkt = p.tile_bucket[tile], c = bkt % x.M, bh = bkt / x.M, hi = bh % x.HI;
      g.head = hi * per_list + (item - tile * per_list);
      g.kv_row = bh / x.HI * x.TK + c * kKeys;
      g.first = p.tile_first[tile];
      g.n = p.tile_cnt[tile];
    }
    return g;
  };
  RowGroup gi = open(blockIdx.x * kRowFwdWarps + warp);

  auto load_kv = [&](const RowGroup& g) {
    if (lane == 0) {
      mbar_arrive_expect_tx(&kv_bar[warp], 2 * kTileKV);
      tma_load_2d(base, &tmap_k, &kv_bar[warp], g.head / G * kD, g.kv_row);
      tma_load_2d(base + kTileKV, &tmap_v, &kv_bar[warp], g.head / G * kD, g.kv_row);
    }
    __syncwarp();
  };
  // lanes 0 .. 15 know a row of the block each: its pair
  auto load_id = [&](const RowGroup& g, int blk) { return lane < kRowFwdRows && blk + lane < g.n ? p.entries[g.first + blk + lane] : -1; };
  auto load_rows = [&](int hq, int id, uint32_t buf) {
    const int row = id < 0 ? no_row : token_of(div, id);       // (behind the last row: zeros)
    if (lane == 0) mbar_arrive_expect_tx(&q_bar[warp][buf], kRowFwdBytes);
    const int from = (lane & 3) * 4;
    const int r0 = __shfl_sync(0xffffffffu, row, from), r1 = __shfl_sync(0xffffffffu, row, from + 1);
    const int r2 = __shfl_sync(0xffffffffu, row, from + 2), r3 = __shfl_sync(0xffffffffu, row, from + 3);
    if (lane < 4) tma_gather4(base + 2 * kTileKV + buf * kRowFwdBytes + lane * 512, &tmap_q, &q_bar[warp][buf], hq * kD, r0, r1, r2, r3);
    __syncwarp();
  };

  const uint32_t la = frag_a(lane), lb = frag_b(lane);
  const uint64_t scale2 = f2_pack(x.scale_log2, x.scale_log2);
  uint32_t n_groups = 0, it = 0;
  bool ok = true;
  int id = -1;
  if (gi.n) {
    load_kv(gi);
    id = load_id(gi, 0);
    load_rows(gi.head, id, 0);
  }
  while (gi.n && ok) {
    const RowGroup ng = open(gi.item + step);
    ok = mbar_wait_w(&kv_bar[warp], n_groups & 1, &abort_flag, p.status);
    ++n_groups;
    const int hq = gi.head;
    int blk = 0;
    for (bool last = false; !last; ++it) {
      const uint32_t buf = it & 1;
      const int nblk = blk + kRowFwdRows;
      last = nblk >= gi.n;
      const bool more = !last || ng.n;                       // a next step: the group's next block, or the next group's first
      int next_id = -1;
      if (more) next_id = last ? load_id(ng, 0) : load_id(gi, nblk);
      // row (token, slot) of the partial outputs and of the weights; rows lane / 4 and lane / 4 + 8 are this lane's in the products
      const int pair = id < 0 ? 0 : id, tok = token_of(div, pair), slot = slot_of(div, pair);
      const long long at = static_cast<long long>(tok) * x.S + slot;
      const float w_own = id < 0 ? 0.f : p.w[at];
      ok = ok && mbar_wait_w(&q_bar[warp][buf], (it >> 1) & 1, &abort_flag, p.status);
      if (!ok) break;
      const uint32_t qb = q_s + buf * kRowFwdBytes;
      float sc[8][4];
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t a[4];
        ldsm4(a, (qb + la) ^ (kk << 5));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t b[4];
          ldsm4(b, ((k_s + lb) ^ (kk << 5)) + 2048 * j);
          if (kk == 0) { mma_16816_new(sc[2 * j], a, b[0], b[1]); mma_16816_new(sc[2 * j + 1], a, b[2], b[3]); }
          else { mma_16816(sc[2 * j], a, b[0], b[1]); mma_16816(sc[2 * j + 1], a, b[2], b[3]); }
        }
      }
      if (more) load_rows(last ? ng.head : hq, next_id, buf ^ 1);
      float l[2], m[2];
      uint32_t pk[8][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float mx = fmaxf(sc[0][2 * i], sc[0][2 * i + 1]);
#pragma unroll
        for (int j = 1; j < 8; ++j) mx = max3(mx, sc[j][2 * i], sc[j][2 * i + 1]);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        m[i] = mx;
        const float mm = -mx * x.scale_log2;
        const uint64_t mm2 = f2_pack(mm, mm);
        uint64_t sum2 = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float p0, p1;
          f2_unpack(f2_fma(f2_pack(sc[j][2 * i], sc[j][2 * i + 1]), scale2, mm2), p0, p1);
          p0 = ex2(p0); p1 = ex2(p1);
          sum2 = j ? f2_add(sum2, f2_pack(p0, p1)) : f2_pack(p0, p1);
          pk[j][i] = pack_bf16x2(p0, p1);
        }
        float s0, s1;
        f2_unpack(sum2, s0, s1);
        s0 += s1;
        s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
        l[i] = s0 + __shfl_xor_sync(0xffffffffu, s0, 2);
      }
      float o[8][4];
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const uint32_t a[4] = {pk[2 * kk][0], pk[2 * kk][1], pk[2 * kk + 1][0], pk[2 * kk + 1][1]};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t b[4];
          ldsm4_t(b, ((v_s + la) ^ (j << 5)) + 2048 * kk);
          if (kk == 0) { mma_16816_new(o[2 * j], a, b[0], b[1]); mma_16816_new(o[2 * j + 1], a, b[2], b[3]); }
          else { mma_16816(o[2 * j], a, b[0], b[1]); mma_16816(o[2 * j + 1], a, b[2], b[3]); }
        }
      }
      if (last) {
        __syncwarp();                                        // every lane has read the K / V tile
        if (ng.n) load_kv(ng);
      }
      const int g8 = lane >> 2;
      const float f0 = x.out_scale * __shfl_sync(0xffffffffu, w_own, g8) / l[0];
      const float f1 = x.out_scale * __shfl_sync(0xffffffffu, w_own, g8 + 8) / l[1];
#pragma unroll
      for (int j = 0; j < 8; j += 2)
        stsm4((qb + la) ^ (j << 4), pack_bf16x2(o[j][0] * f0, o[j][1] * f0), pack_bf16x2(o[j][2] * f1, o[j][3] * f1),
              pack_bf16x2(o[j + 1][0] * f0, o[j + 1][1] * f0), pack_bf16x2(o[j + 1][2] * f1, o[j + 1][3] * f1));
      // log-sum-exp of row `lane`: from the lanes that hold its sum
      const float lse0 = fmaf(m[0], x.scale, __logf(l[0])), lse1 = fmaf(m[1], x.scale, __logf(l[1]));
      const float t0 = __shfl_sync(0xffffffffu, lse0, (lane & 7) * 4), t1 = __shfl_sync(0xffffffffu, lse1, (lane & 7) * 4);
      if (id >= 0) p.lse_slots[(static_cast<long long>(tok) * x.HQ + hq) * x.S + slot] = lane < 8 ? t0 : t1;
      __syncwarp();
      const int own = id < 0 ? -1 : static_cast<int>(at);    // (fewer pairs than 2^31)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = (lane >> 3) + 4 * i, row = __shfl_sync(0xffffffffu, own, r);
        if (row >= 0) {
          uint4 v;
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(qb + tile_at(r, lane & 7)) : "memory");
          *reinterpret_cast<uint4*>(p.partial + (static_cast<long long>(row) * x.HQ + hq) * kD + (lane & 7) * 8) = v;
        }
      }
      fence_proxy_async();                                   // the block's buffer takes the rows of the step after next
      __syncwarp();
      id = next_id; blk = nblk;
    }
    gi = ng;
  }
  __syncthreads();
  if (abort_flag) { for (int i = 0; i < 200; ++i) __nanosleep(1000); }
}

// ---- backward ------------------------------------------------------------------------------------------------
// A CTA an item: four warps multiply, a fifth copies (K / V of the next item, rows and constants of the next step) and leaves
// beside each step's rows where its results go.  A step is 32 pairs: each warp forms S^T and dP^T of eight of them against all 64
// keys, so that a pair's delta stays inside a warp; Pw^T and dS^T go to shared memory (the one barrier of a step), and from there
// each warp takes 16 keys of dV and dK (accumulated in registers over the item) and a quarter of dQ.
// 8,192 tokens, 32 pairs a chapter, uniform, with the sum over slots: 1,115 -> 633 us; 250 tokens 732 -> 359, of which 246 are HBM.
// What is left is shared memory latency with 12 warps an SM (registers): splitting by keys instead (two barriers, less operand
// traffic) made nothing faster, eight warps of half the registers took a quarter more.
constexpr int kRowBwdThreads = 160;                                // 4 warps for the products, 1 for the copies
constexpr int kRowBwdRows = 32;                                    // pairs of a step
constexpr int kRowBwdBytes = kRowBwdRows * kD * 2;                 // 4 KiB
constexpr int kPairBytes = kKeys * kRowBwdRows * 2;                // [key][pair], 4 KiB
constexpr int kStageStride = 80, kStageBytes = 16 * kStageStride;   // a warp's: 16 rows of 32 outputs
constexpr int kRowBwdSmem = 4 * kTileKV + 4 * kRowBwdBytes + 4 * kPairBytes + 4 * kStageBytes + 1024;
constexpr int kRowBwdCtas = 3;                                     // an SM

// What the copying warp tells about a step
struct BwdStep {
  long long out_at[kRowBwdRows];          // row of the partial dQ of a pair's head; < 0: no pair
  long long dw_at[kRowBwdRows];           // its place in d_w_heads
  float w[kRowBwdRows], lse[kRowBwdRows];
  long long dkv_at;                    // of the group: where its dK / dV rows start
  int pairs, last, final;              // pairs in the step; the last of its group; the last of all
};

__global__ void __launch_bounds__(kRowBwdThreads, kRowBwdCtas)
token_mix_rows_bwd_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                          const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_do, MixBwdParams p,
                          RowItems items) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t kv_full[2], kv_empty[2], full[2], empty[2];
  __shared__ int abort_flag;
  __shared__ BwdStep steps[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* rows = base + 4 * kTileKV;                            // two (dO, Q) row blocks behind two (K, V) tile pairs
  const MixShape& x = p.x;
  if (p.ask && tiles_end_sooner(p.totals)) return;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 4);
      mbar_init(&full[i], 33); mbar_init(&empty[i], 4);
    }
    fence_mbar_init();
  }
  __syncthreads();
  RowGroup gi;
  gi.item = blockIdx.x;

  if (warp == 4) {
    const int G = x.HQ / x.HK, no_row = x.B * x.TQ;
    // dK / dV rows of buckets without pairs are zero-filled on the way, so the caller need not clear the buffers
    auto zero = [&](const RowGroup& g) {
      for (int r = lane; r < 128; r += 32) {
        __nv_bfloat16* dst = (r >= 64 ? p.d_k : p.d_v) + (static_cast<long long>(g.kv_row) + (r & 63)) * p.dkv_ld;
        for (int e = 0; e < kD / 8; ++e) reinterpret_cast<uint4*>(dst + g.head * kD)[e] = make_uint4(0u, 0u, 0u, 0u);
      }
    };
    auto load_kv = [&](const RowGroup& g, uint32_t n) {
      if (lane == 0) {
        uint8_t* dst = base + (n & 1) * 2 * kTileKV;
        mbar_arrive_expect_tx(&kv_full[n & 1], 2 * kTileKV);
        tma_load_2d(dst, &tmap_k, &kv_full[n & 1], g.head * kD, g.kv_row);
        tma_load_2d(dst + kTileKV, &tmap_v, &kv_full[n & 1], g.head * kD, g.kv_row);
      }
      __syncwarp();
    };
    auto load_id = [&](const RowGroup& g, int blk) { return blk + lane < g.n ? p.entries[g.first + blk + lane] : -1; };
    gi.seek(x, x.HK, items, gridDim.x, zero);
    uint32_t it = 0, n = 0;
    bool ok = true;
    int id = -1;
    RowGroup ng = gi;
    if (gi.n) {
      load_kv(gi, 0);
      id = load_id(gi, 0);
      ng.item += gridDim.x;
      ng.seek(x, x.HK, items, gridDim.x, zero);
    }
    for (; gi.n && ok; ++n) {
      RowGroup nn = ng;
      int hq = gi.head * G, blk = 0;
      for (bool last = false; !last; ++it) {
        int nblk = blk + kRowBwdRows, nhq = hq;
        if (nblk >= gi.n) { nblk = 0; ++nhq; }
        last = nhq == (gi.head + 1) * G;
        int next_id = -1;
        if (!last) next_id = load_id(gi, nblk);
        else if (ng.n) next_id = load_id(ng, 0);
        const uint32_t buf = it & 1;
        if (it >= 2) ok = mbar_wait_w(&empty[buf], ((it >> 1) & 1) ^ 1, &abort_flag, p.status);
        if (!ok) break;
        BwdStep& st = steps[buf];
        const bool valid = id >= 0;
        const int pair = valid ? id : 0, tok = token_of(items.div, pair), s = slot_of(items.div, pair);
        const long long tok_s = static_cast<long long>(tok) * x.S + s, dw_at = (static_cast<long long>(tok) * x.HQ + hq) * x.S + s;
        st.out_at[lane] = valid ? tok_s * x.HQ + hq : -1;
        st.dw_at[lane] = dw_at;
        const int pairs = min(kRowBwdRows, gi.n - blk), quads = pairs > 16 ? 8 : 4;     // whole 16-pair halves are filled
        if (lane == 0) {
          st.dkv_at = gi.kv_row * p.dkv_ld + gi.head * kD;
          st.pairs = pairs; st.last = last; st.final = last && !ng.n;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_expect_tx(&full[buf], quads * 2 * 512);
        cp_async4_or_zero(smem_u32(&st.w[lane]), p.w + tok_s, valid);
        cp_async4_or_zero(smem_u32(&st.lse[lane]), p.lse_slots + dw_at, valid);
        cp_async_arrive(&full[buf]);
        const int row = valid ? tok : no_row;
        const int r0 = __shfl_sync(0xffffffffu, row, (lane & 7) * 4), r1 = __shfl_sync(0xffffffffu, row, (lane & 7) * 4 + 1);
        const int r2 = __shfl_sync(0xffffffffu, row, (lane & 7) * 4 + 2), r3 = __shfl_sync(0xffffffffu, row, (lane & 7) * 4 + 3);
        if (lane < 16 && (lane & 7) < quads)
          tma_gather4(rows + buf * 2 * kRowBwdBytes + (lane >> 3) * kRowBwdBytes + (lane & 7) * 512, lane < 8 ? &tmap_do : &tmap_q,
                      &full[buf], hq * kD, r0, r1, r2, r3);
        __syncwarp();
        // Behind the rows of its first step: the wait for the last group's tiles would hold them up.
        if (blk == 0 && hq == gi.head * G && ng.n) {
          if (n > 0) ok = mbar_wait_w(&kv_empty[(n + 1) & 1], (((n + 1) >> 1) & 1) ^ 1, &abort_flag, p.status);
          if (!ok) break;
          load_kv(ng, n + 1);                                    // they arrive under this group's steps
          nn.item += gridDim.x;
          nn.seek(x, x.HK, items, gridDim.x, zero);
        }
        id = next_id; hq = nhq; blk = nblk;
      }
      gi = ng;
      ng = nn;
    }
    cp_async_wait<0>();
  } else {
    gi.seek(x, x.HK, items, gridDim.x, [](const RowGroup&) {});
    const uint32_t kv_s = smem_u32(base), rows_s = smem_u32(rows);
    const uint32_t pt_s = rows_s + 4 * kRowBwdBytes;             // two (Pw^T, dS^T): [key][pair], 64-byte rows, 16-byte pieces swizzled
    const uint32_t stage = pt_s + 4 * kPairBytes + warp * kStageBytes;
    const int g8 = lane >> 2, c2 = (lane & 3) * 2;
    const uint32_t la = frag_a(lane), lb = ((lane & 7) * 128) + (((lane >> 3) ^ (lane & 7)) << 4);   // lb: eight rows x 32 columns
    auto pt_at = [](int key, int piece) { return static_cast<uint32_t>(key * 64 + ((piece ^ ((key >> 1) & 3)) << 4)); };
    const uint32_t pt_to = pt_at(lane, warp);                                            // + 2048: keys 32 on
    const uint32_t pt_a = pt_at(16 * warp + (lane & 15), lane >> 4);                     // ^ 32: pairs 16 on
    const uint32_t ds_t = pt_at((lane & 7) + ((lane >> 4) << 3), ((lane >> 3) & 1) + 2 * (warp & 1));   // + 1024: keys 16 on
    const uint32_t st_to = stage + (lane & 15) * kStageStride + (lane >> 4) * 16, st_from = stage + g8 * kStageStride + (lane & 3) * 16;
    const uint64_t scale2 = f2_pack(x.scale_log2, x.scale_log2), out2 = f2_pack(x.out_scale, x.out_scale);
    auto take = [&](uint32_t from) {
      uint4 v;
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(from) : "memory");
      return v;
    };
    float dk[8][4], dv[8][4];                                    // 16 keys x 64 columns
    bool fresh = true, more = gi.n > 0;
    uint32_t n = 0;
    for (uint32_t it = 0; more; ++it) {
      const uint32_t buf = it & 1;
      bool ok = mbar_wait_w(&full[buf], (it >> 1) & 1, &abort_flag, p.status);
      if (fresh) {
        ok = ok && mbar_wait_w(&kv_full[n & 1], (n >> 1) & 1, &abort_flag, p.status);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) dk[j][i] = dv[j][i] = 0.f;
      }
      const BwdStep& st = steps[buf];
      const uint32_t k_s = kv_s + (n & 1) * 2 * kTileKV;         // (V behind it)
      const uint32_t do_s = rows_s + buf * 2 * kRowBwdBytes;     // (Q behind it)
      const uint32_t pt = pt_s + buf * 2 * kPairBytes;
      // 16-pair halves of the step that hold pairs.  None where a wait ran out: the step's record and rows may never have been
      // written, so nothing of them is read or stored on the way to the meeting below, where every warp is awaited.
      const int halves = !ok ? 0 : st.pairs > 16 ? 2 : 1;
      // S^T and dP^T: 64 keys x 8 pairs a warp; this lane's keys are 16 m + g8 and that + 8, its pairs c2 and the next.  A chain in the
      // instruction's accumulator is truncated at each step, so two chains of 32 columns are added in fp32: dW (fp32) is 2.7e-7 from
      // fp64 then, 3.1e-7 with chains of 64 columns, 2.75e-7 in the 128-row kernel.  (32 pairs a chapter: 621 -> 633 us.)
      if (warp < 2 * halves) {
        float sc[4][4], dp[4][4];
#pragma unroll
        for (int kk = 0; kk < 4; kk += 2) {
          uint32_t bq[4], bd[4];
          const uint32_t from = ((do_s + lb) ^ (kk << 5)) + 1024 * warp;
          ldsm4(bd, from);
          ldsm4(bq, from + kRowBwdBytes);
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            uint32_t ak[4], av[4];
            float ts[4], td[4];
            const uint32_t a0 = ((k_s + la) ^ (kk << 5)) + 2048 * m, a1 = ((k_s + la) ^ ((kk + 1) << 5)) + 2048 * m;
            ldsm4(ak, a0);
            ldsm4(av, a0 + kTileKV);
            mma_16816_new(ts, ak, bq[0], bq[1]); mma_16816_new(td, av, bd[0], bd[1]);
            ldsm4(ak, a1);
            ldsm4(av, a1 + kTileKV);
            mma_16816(ts, ak, bq[2], bq[3]); mma_16816(td, av, bd[2], bd[3]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              sc[m][i] = kk == 0 ? ts[i] : sc[m][i] + ts[i];
              dp[m][i] = kk == 0 ? td[i] : dp[m][i] + td[i];
            }
          }
        }
        // P^T; a pair's delta = <P, dP> over its 64 keys
        auto two = [](const float* v) { return *reinterpret_cast<const uint64_t*>(v); };
        const int at = 8 * warp + c2;
        const uint64_t n2 = f2_mul(two(&st.lse[at]), f2_pack(-kLog2e, -kLog2e)), wt = f2_mul(two(&st.w[at]), out2);
        uint64_t delta = 0;
#pragma unroll
        for (int m = 0; m < 4; ++m) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            float p0, p1;
            f2_unpack(f2_fma(f2_pack(sc[m][2 * i], sc[m][2 * i + 1]), scale2, n2), p0, p1);
            sc[m][2 * i] = ex2(p0); sc[m][2 * i + 1] = ex2(p1);
            delta = f2_fma(f2_pack(sc[m][2 * i], sc[m][2 * i + 1]), f2_pack(dp[m][2 * i], dp[m][2 * i + 1]), delta);
          }
        }
        float d0, d1;
        f2_unpack(delta, d0, d1);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          d0 += __shfl_xor_sync(0xffffffffu, d0, o);
          d1 += __shfl_xor_sync(0xffffffffu, d1, o);
        }
        if (lane < 4) {
          if (st.out_at[at] >= 0) p.d_w_heads[st.dw_at[at]] = x.out_scale * d0;
          if (st.out_at[at + 1] >= 0) p.d_w_heads[st.dw_at[at + 1]] = x.out_scale * d1;
        }
        const uint64_t minus = f2_pack(-d0, -d1);
        // Columns of the step without a pair are zero whatever their products gave: against an infinite key their zero rows give NaN,
        // which the sums over the chapter's pairs would spread to all of its keys.
        const uint32_t keep = (at < st.pairs ? 0xFFFFu : 0u) | (at + 1 < st.pairs ? 0xFFFF0000u : 0u);
#pragma unroll
        for (int m = 0; m < 4; m += 2) {
          uint32_t a[4], d[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int mm = m + (i >> 1), c = 2 * (i & 1);
            const uint64_t pw = f2_mul(wt, f2_pack(sc[mm][c], sc[mm][c + 1]));
            float v0, v1;
            f2_unpack(pw, v0, v1);
            a[i] = pack_bf16x2(v0, v1) & keep;
            f2_unpack(f2_mul(pw, f2_add(f2_pack(dp[mm][c], dp[mm][c + 1]), minus)), v0, v1);
            d[i] = pack_bf16x2(v0, v1) & keep;
          }
          stsm4(pt + pt_to + m * 1024, a[0], a[1], a[2], a[3]);
          stsm4(pt + kPairBytes + pt_to + m * 1024, d[0], d[1], d[2], d[3]);
        }
      }
      // Pw^T and dS^T are complete; the step before last, whose buffers these are, was done with two such barriers ago
      if (!warps_agree<1, 128>(halves > 0)) break;
      // dQ = dS K: 16 pairs x 32 columns a warp
      if ((warp & 1) < halves) {
        float dq[4][4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          uint32_t a[4];
          ldsm4_t(a, pt + kPairBytes + ds_t + 1024 * kk);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            uint32_t b[4];
            ldsm4_t(b, ((k_s + la) ^ ((warp >> 1) << 6) ^ (j << 5)) + 2048 * kk);
            if (kk == 0) { mma_16816_new(dq[2 * j], a, b[0], b[1]); mma_16816_new(dq[2 * j + 1], a, b[2], b[3]); }
            else { mma_16816(dq[2 * j], a, b[0], b[1]); mma_16816(dq[2 * j + 1], a, b[2], b[3]); }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; j += 2)
          stsm4(st_to + j * 16, pack_bf16x2(dq[j][0] * x.scale, dq[j][1] * x.scale), pack_bf16x2(dq[j][2] * x.scale, dq[j][3] * x.scale),
                pack_bf16x2(dq[j + 1][0] * x.scale, dq[j + 1][1] * x.scale), pack_bf16x2(dq[j + 1][2] * x.scale, dq[j + 1][3] * x.scale));
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const long long row = st.out_at[16 * (warp & 1) + g8 + 8 * i];
          if (row >= 0)
            *reinterpret_cast<uint4*>(p.dq_partial + row * kD + (warp >> 1) * 32 + (lane & 3) * 8) = take(st_from + 8 * i * kStageStride);
        }
      }
      // dV += Pw^T dO, dK += dS^T Q: 16 keys a warp
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h < halves) {
          uint32_t ap[4], as[4];
          ldsm4(ap, pt + (pt_a ^ (32 * h)));
          ldsm4(as, pt + kPairBytes + (pt_a ^ (32 * h)));
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t bd[4], bq[4];
            const uint32_t from = ((do_s + la) ^ (j << 5)) + 2048 * h;
            ldsm4_t(bd, from);
            ldsm4_t(bq, from + kRowBwdBytes);
            mma_16816(dv[2 * j], ap, bd[0], bd[1]);
            mma_16816(dv[2 * j + 1], ap, bd[2], bd[3]);
            mma_16816(dk[2 * j], as, bq[0], bq[1]);
            mma_16816(dk[2 * j + 1], as, bq[2], bq[3]);
          }
        }
      }
      const bool last = st.last;
      const long long dkv_at = st.dkv_at + 16 * warp * p.dkv_ld;
      more = !st.final;
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&empty[buf]);
        if (last) mbar_arrive(&kv_empty[n & 1]);
      }
      fresh = last;
      if (last) {                                                // this warp's 16 rows of dV, then of dK, 32 columns at a time
        ++n;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float f = t >= 2 ? x.scale : 1.f;
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            const float(&u)[4] = t >= 2 ? dk[4 * (t & 1) + j] : dv[4 * (t & 1) + j];
            const float(&v)[4] = t >= 2 ? dk[4 * (t & 1) + j + 1] : dv[4 * (t & 1) + j + 1];
            stsm4(st_to + j * 16, pack_bf16x2(u[0] * f, u[1] * f), pack_bf16x2(u[2] * f, u[3] * f), pack_bf16x2(v[0] * f, v[1] * f),
                  pack_bf16x2(v[2] * f, v[3] * f));
          }
          __syncwarp();
          __nv_bfloat16* dst = (t >= 2 ? p.d_k : p.d_v) + dkv_at + g8 * p.dkv_ld + (t & 1) * 32 + (lane & 3) * 8;
          *reinterpret_cast<uint4*>(dst) = take(st_from);
          *reinterpret_cast<uint4*>(dst + 8 * p.dkv_ld) = take(st_from + 8 * kStageStride);
          __syncwarp();
        }
      }
    }
  }
  __syncthreads();
  if (abort_flag) { for (int i = 0; i < 200; ++i) __nanosleep(1000); }
}

}  // namespace
}  // namespace moc
