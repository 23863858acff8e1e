// bf16 joint-softmax cross attention, forward, for sm_100a.
//
// One CTA = 128 queries of one (batch, head); it streams the (S+k) gathered chapters as tiles of
// 64 keys:   S_j = Q K_j^T  (tcgen05.mma, operands in 128-byte-swizzled shared memory filled by TMA,
// accumulator in tensor memory) -> online softmax by 128 threads that each own one query row
// (tcgen05.ld, exp2 on the scaled scores, P written back to tensor memory as packed bf16) ->
// O += P_j V_j (tcgen05.mma with A = P from tensor memory, B = the V tile as an MN-major operand).
// A CTA holds 256 TMEM columns -- three 64-column score buffers (P_j is written as packed bf16 over the first 32 columns
// of its own buffer) and the 64-column O accumulator -- about 97 KiB of shared memory and 192 threads, and two CTAs share
// an SM (__launch_bounds__(192, 2)).  Scores run three tiles ahead of PV.  The
// running maximum is only raised (and O rescaled) when it grows by more than 2^8, which keeps P
// within bf16 range while skipping almost every rescale.
//
// What bounds it: at 8 x 1024 queries, 12 heads, 4,160 keys a 128 x 64 tile takes an SM about 410 ns (770 cycles) of which
// the exponential unit is busy 450 and the tensor pipe 256; the rest is the chain wait -> tensor-memory load ->
// exponentials -> store -> wait with two row-owning warps per scheduler.  Four CTAs per SM with one score buffer each, and
// two query tiles per CTA sharing the K / V tiles, measured the same or worse (460 and 445 ns).  190 us before, 167 us now.
//
// With few query tiles (short or few sequences) the key range is cut into up to eight runs, one CTA of a cluster each,
// merged through distributed shared memory at the end: 320 queries of one sequence 52 -> 25 us.
#define MOC_KERNEL_TAG 2
#include "moc_common.cuh"

namespace moc {
namespace {

constexpr int kQ = 128;          // queries per CTA
constexpr int kKeys = 64;        // keys per tile
constexpr int kD = 64;           // head dim
constexpr int kStages = 5;       // K/V ring depth (K_j is read three tiles before V_j)
constexpr int kBufs = 3;         // score buffers
constexpr int kThreads = 192;    // 4 softmax warps + a warp for loads and scores + a warp for P V
constexpr int kQBytes = kQ * kD * 2;
constexpr int kTileBytes = kKeys * kD * 2;
constexpr int kSmemBytes = kQBytes + kStages * 2 * kTileBytes + 1024;
constexpr int kTmemCols = 256;
constexpr uint32_t kColS = 0;      // S buffers of 64 columns, tile j uses buffer j % 3
constexpr uint32_t kColP = 0;      // P_j as packed bf16 over the first 32 columns of its S buffer
constexpr uint32_t kColO = 192;    // O accumulator: 64 columns
// Of every eight columns, how many take the polynomial instead of the exponential unit (0, 1, 2, 3 pairs of four in the
// second half measured 428, 416, 428, 462 ns per 128 x 64 tile and SM).
constexpr int kPolyOf4 = 1;
constexpr float kRescaleThreshold = 8.0f;

struct FwdParams {
  __nv_bfloat16* o;
  float* lse;
  int L, n_sel, H, HK, split;
  float scale_log2;   // softmax scale * log2(e)
  int* status;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^x for two values on the FMA pipe: x = n + f with |f| <= 1/2 (Cody-Waite with the round-to-nearest addition of
// 1.5 * 2^23), a degree-5 polynomial fitted to 2^f for least relative error (2.3e-7 in fp32, that of the hardware
// instruction), n added to the exponent.  Arguments count as no less than -127, whose 2^n comes out as the smallest
// subnormal: 0 as bf16, and nothing beside the row's largest term, so a masked column (-inf) adds nothing.  NaN is not
// kept; the row maximum sees it.
__device__ __forceinline__ void ex2_poly2(uint64_t x, float& y0, float& y1) {
  float x0, x1;
  f2_unpack(x, x0, x1);
  x = f2_pack(fmaxf(x0, -127.f), fmaxf(x1, -127.f));
  const uint64_t magic = f2_pack(12582912.f, 12582912.f), nmagic = f2_pack(-12582912.f, -12582912.f);
  const uint64_t t = f2_add(x, magic);
  const uint64_t n = f2_add(t, nmagic);
  const uint64_t f = f2_fma(n, f2_pack(-1.f, -1.f), x);
  uint64_t p = f2_pack(0.001327647129073739f, 0.001327647129073739f);
  p = f2_fma(p, f, f2_pack(0.009675540961325169f, 0.009675540961325169f));
  p = f2_fma(p, f, f2_pack(0.05550713092088699f, 0.05550713092088699f));
  p = f2_fma(p, f, f2_pack(0.24022120237350464f, 0.24022120237350464f));
  p = f2_fma(p, f, f2_pack(0.6931469440460205f, 0.6931469440460205f));
  p = f2_fma(p, f, f2_pack(1.0000001192092896f, 1.0000001192092896f));
  float p0, p1, t0, t1;
  f2_unpack(p, p0, p1);
  f2_unpack(t, t0, t1);
  y0 = __int_as_float(__float_as_int(p0) + (__float_as_int(t0) << 23));
  y1 = __int_as_float(__float_as_int(p1) + (__float_as_int(t1) << 23));
}

__global__ void exp2_probe_kernel(const float* __restrict__ x, float* __restrict__ y, int pairs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pairs) return;
  ex2_poly2(f2_pack(x[2 * i], x[2 * i + 1]), y[2 * i], y[2 * i + 1]);
}

// MMA groups issued as one instruction block by one elected lane (~3 instructions per MMA): the MMA warp
// shares its scheduler partition with busy row-owning warps, so instructions per MMA set the issue rate.
// [d] = A * B^T over 4 K steps, both operands K-major in shared memory.
__device__ __forceinline__ void issue_ss_single(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
#define MOC_SS1_STEP(KK, PACC)                                                  \
  "add.s64 ta, %1, " #KK "*2;\n\t add.s64 tb, %2, " #KK "*2;\n\t"                \
  "@q tcgen05.mma.cta_group::1.kind::f16 [%0], ta, tb, %3, " PACC ";\n\t"
  asm volatile(
      "{\n\t.reg .pred q, pt, pf;\n\t.reg .b64 ta, tb;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.eq.b32 pt, 0, 0;\n\t"
      "setp.ne.b32 pf, 0, 0;\n\t"
      MOC_SS1_STEP(0, "pf") MOC_SS1_STEP(1, "pt") MOC_SS1_STEP(2, "pt") MOC_SS1_STEP(3, "pt")
      "}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc)
      : "memory");
#undef MOC_SS1_STEP
}
// [d] += A * B over 4 K steps: A packed bf16 in tensor memory (K step kk at column a + 8 kk), B MN-major.
__device__ __forceinline__ void issue_ts_single(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
#define MOC_TS1_STEP(KK, PACC)                                                  \
  "add.u32 ca, %1, " #KK "*8;\n\t add.s64 tb, %2, " #KK "*128;\n\t"               \
  "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [ca], tb, %3, " PACC ";\n\t"
  asm volatile(
      "{\n\t.reg .pred q, pa, pt;\n\t.reg .b64 tb;\n\t.reg .b32 ca;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 pa, %4, 0;\n\t"
      "setp.eq.b32 pt, 0, 0;\n\t"
      MOC_TS1_STEP(0, "pa") MOC_TS1_STEP(1, "pt") MOC_TS1_STEP(2, "pt") MOC_TS1_STEP(3, "pt")
      "}"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
#undef MOC_TS1_STEP
}

__global__ void __launch_bounds__(kThreads, 2)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv,
                   FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  // p_full is one barrier per score buffer: scores are issued ahead of P, so the row owners can finish tile j+1 (the next
  // buffer) while the MMA warp has not yet observed tile j's phase; with a single barrier two completed phases would look
  // like none to a parity wait and the warp would wait forever.
  __shared__ __align__(8) uint64_t q_bar, kv_full[kStages], s_full[kBufs], p_full[kBufs], pv_done[kBufs], o_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = base;
  uint8_t* kv_s = base + kQBytes;

  // a cluster of p.split CTAs shares one query tile; each takes a run of the key tiles
  const int rank = p.split > 1 ? static_cast<int>(cluster_rank()) : 0;
  const int q0 = blockIdx.x / p.split * kQ;
  const int h = blockIdx.y, b = blockIdx.z;
  const int kh = h / (p.H / p.HK);
  const int all_tiles = (p.n_sel + kKeys - 1) / kKeys;
  const int tile0 = rank * all_tiles / p.split, n_tiles = (rank + 1) * all_tiles / p.split - tile0;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(&q_bar, 1);
    for (int s = 0; s < kStages; ++s) mbar_init(&kv_full[s], 1);
    for (int i = 0; i < kBufs; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 128); mbar_init(&pv_done[i], 1); }
    mbar_init(&o_bar, 1);
    fence_mbar_init();
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_kv);
  }
  if (warp == 5) {
    tmem_alloc(&tmem_slot, kTmemCols);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  // Two control warps, warp-uniform, one elected lane issues.  Each passes one or two waits and four MMAs per tile; as one
  // warp, competing for issue slots with the softmax warps of its scheduler, their chain took longer than the softmax.
  if (warp == 4) {
    // ---------------- loads and scores ----------------
    const uint32_t idesc_s = umma_idesc_bf16(kQ, kKeys, 0, 0);
    const uint64_t q_desc = umma_desc_sw128(smem_u32(q_s), 16, 1024);
    const uint64_t k_desc0 = umma_desc_sw128(smem_u32(kv_s), 16, 1024);
    constexpr uint64_t kStageOff = (2 * kTileBytes) >> 4;
    auto load = [&](int j, int stage) {
      if (lane == 0) {
        uint8_t* k_s = kv_s + stage * 2 * kTileBytes;
        const int row = b * p.n_sel + (tile0 + j) * kKeys;
        mbar_arrive_expect_tx(&kv_full[stage], 2 * kTileBytes);
        tma_load_2d(k_s, &tmap_kv, &kv_full[stage], kh * kD, row);
        tma_load_2d(k_s + kTileBytes, &tmap_kv, &kv_full[stage], p.HK * kD + kh * kD, row);
      }
      __syncwarp();
    };
    if (lane == 0) {
      mbar_arrive_expect_tx(&q_bar, kQBytes);
      tma_load_2d(q_s, &tmap_q, &q_bar, h * kD, b * p.L + q0);
    }
    for (int j = 0; j < kStages && j < n_tiles; ++j) load(j, j);
    bool ok = mbar_wait_w(&q_bar, 0, &abort_flag, p.status);
    // Scores run three tiles ahead: S_j takes the buffer of P_{j-3} as soon as P_{j-3} V_{j-3} is complete, which also
    // frees that tile's stage.
    int buf = 0, s = 0, s3 = kStages - kBufs;       // j % 3, j % kStages, (j - 3) % kStages
    uint32_t bph = 1, sph = 0;                      // parities: PV that last used `buf`, fill of stage s
    for (int j = 0; j < n_tiles && ok; ++j) {
      if (j >= kBufs) {
        ok = mbar_wait_w(&pv_done[buf], bph, &abort_flag, p.status);
        if (!ok) break;
        if (j - kBufs + kStages < n_tiles) load(j - kBufs + kStages, s3);
      }
      ok = mbar_wait_w(&kv_full[s], sph, &abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      issue_ss_single(tmem + kColS + buf * 64, q_desc, k_desc0 + s * kStageOff, idesc_s);
      tc_commit_w(&s_full[buf]);
      if (++buf == kBufs) { buf = 0; bph ^= 1; }
      if (++s == kStages) { s = 0; sph ^= 1; }
      if (++s3 == kStages) s3 = 0;
    }
  } else if (warp == 5) {
    // ---------------- P V ----------------
    const uint32_t idesc_o = umma_idesc_bf16(kQ, kD, 0, 1);
    const uint64_t v_desc0 = umma_desc_sw128(smem_u32(kv_s) + kTileBytes, 8192, 1024);
    constexpr uint64_t kStageOff = (2 * kTileBytes) >> 4;
    bool ok = true;
    int buf = 0, s = 0;
    uint32_t bph = 0;
    for (int j = 0; j < n_tiles && ok; ++j) {
      ok = mbar_wait_w(&p_full[buf], bph, &abort_flag, p.status);    // (S_j was complete before, and K_j / V_j with it)
      if (!ok) break;
      tc_fence_after();
      issue_ts_single(tmem + kColO, tmem + kColP + buf * 64, v_desc0 + s * kStageOff, idesc_o, j > 0 ? 1u : 0u);
      tc_commit_w(&pv_done[buf]);
      if (++buf == kBufs) { buf = 0; bph ^= 1; }
      if (++s == kStages) s = 0;
    }
    tc_commit_w(&o_bar);
  } else {
    // ---------------- softmax: thread <-> query row ----------------
    const uint32_t lane_sel = static_cast<uint32_t>(warp * 32) << 16;
    const int row = warp * 32 + lane;
    float m_used = -INFINITY, l_sum = 0.f;
    bool ok = true;
    int buf = 0;
    uint32_t bph = 0;
    for (int j = 0; j < n_tiles; ++j) {
      ok = mbar_wait_w(&s_full[buf], bph, &abort_flag, p.status);
      if (!ok) break;
      tc_fence_after();
      const uint32_t s_addr = tmem + lane_sel + kColS + buf * 64;
      const int valid = p.n_sel - (tile0 + j) * kKeys;   // keys of this tile that exist
      uint32_t r0[32], r1[32];                 // the whole score row stays in registers
      tmem_ld32(s_addr, r0);
      tmem_ld32(s_addr + 32, r1);
      tmem_wait_ld();
      if (valid < kKeys) {                     // last, partial tile: columns past the end count as -inf
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          if (c >= valid) r0[c] = 0xFF800000u;
          if (32 + c >= valid) r1[c] = 0xFF800000u;
        }
      }
      uint32_t pk[32];
      float psum;
      // exp2 of the scaled scores against the running maximum; exp2 of -inf is 0, so masked columns add nothing.  Scaling
      // and the row sum take two columns per instruction.
      auto exps = [&]() {
        const uint64_t sc = f2_pack(p.scale_log2, p.scale_log2), nm = f2_pack(-m_used, -m_used);
        uint64_t sum0 = 0ull, sum1 = 0ull;
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          float e0, e1, g0, g1;
          const uint64_t xe = f2_fma(f2_pack(__uint_as_float(r0[c]), __uint_as_float(r0[c + 1])), sc, nm);
          const uint64_t xg = f2_fma(f2_pack(__uint_as_float(r1[c]), __uint_as_float(r1[c + 1])), sc, nm);
          f2_unpack(xe, e0, e1);
          e0 = ex2(e0); e1 = ex2(e1);
          if ((c & 7) / 2 < kPolyOf4) {
            ex2_poly2(xg, g0, g1);
          } else {
            f2_unpack(xg, g0, g1);
            g0 = ex2(g0); g1 = ex2(g1);
          }
          sum0 = f2_add(sum0, f2_pack(e0, e1));
          sum1 = f2_add(sum1, f2_pack(g0, g1));
          pk[c / 2] = pack_bf16x2(e0, e1);
          pk[16 + c / 2] = pack_bf16x2(g0, g1);
        }
        float x0, x1;
        f2_unpack(f2_add(sum0, sum1), x0, x1);
        psum = x0 + x1;
      };
      auto row_max = [&]() {
        float t[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 32; c += 4)
#pragma unroll
          for (int i = 0; i < 4; ++i) t[i] = max3_nan(t[i], __uint_as_float(r0[c + i]), __uint_as_float(r1[c + i]));
        return max_nan(max3_nan(t[0], t[1], t[2]), t[3]);
      };
      // The maximum is off the critical path: from the second tile on the exponentials are taken against the running
      // maximum at once, and only a tile that exceeds it by more than 2^8 (P would leave bf16's accurate range) is taken
      // again after the rescale.  A NaN score, seen here for all columns, takes that way too and makes the row NaN.
      if (j > 0) exps();
      const float m_new = max_nan(m_used, row_max() * p.scale_log2);
      const bool need = (j == 0) || !(m_new - m_used <= kRescaleThreshold);
      if (__any_sync(0xffffffffu, need)) {
        if (j > 0) {
          const int pb = buf == 0 ? kBufs - 1 : buf - 1;      // O is complete up to tile j-1
          ok = mbar_wait_w(&pv_done[pb], buf == 0 ? bph ^ 1 : bph, &abort_flag, p.status);
          if (!ok) break;
          tc_fence_after();
          const float alpha = need ? ex2(m_used - m_new) : 1.f;
          uint32_t r[32];
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            tmem_ld32(tmem + lane_sel + kColO + half * 32, r);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 32; ++c) r[c] = __float_as_uint(__uint_as_float(r[c]) * alpha);
            tmem_st32(tmem + lane_sel + kColO + half * 32, r);
          }
          l_sum *= alpha;
        }
        if (need) m_used = m_new;
        exps();
      }
      l_sum += psum;
      // every S value of this row is in registers: P goes over the first 32 columns of this tile's S buffer
      tmem_st32(tmem + lane_sel + kColP + buf * 64, pk);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&p_full[buf]);
      if (++buf == kBufs) { buf = 0; bph ^= 1; }
    }
    if (ok) {
      // A barrier of its own for the finished accumulator: when this warp has handed over its last tile, the products of
      // up to two tiles before may still be waiting for another warp's rows (scores run ahead of them).
      ok = mbar_wait_w(&o_bar, 0, &abort_flag, p.status);
    }
    if (ok) {
      tc_fence_after();
      const float inv = 1.f / l_sum;
      const int l = q0 + row;
      __nv_bfloat16* dst = p.o + (static_cast<long long>(b) * p.L + l) * (p.H * kD) + h * kD;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t r[32];
        tmem_ld32(tmem + lane_sel + kColO + half * 32, r);
        tmem_wait_ld();
        if (p.split > 1) {
          // unnormalised rows into the idle tile ring, 16-byte chunks rotated by the row against bank conflicts
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint32_t addr = smem_u32(kv_s) + row * 256 + (((half * 8 + c) ^ (row & 15)) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[4 * c]), "r"(r[4 * c + 1]),
                         "r"(r[4 * c + 2]), "r"(r[4 * c + 3]) : "memory");
          }
        } else if (l < p.L) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint4 v;
            v.x = pack_bf16x2(__uint_as_float(r[8 * c + 0]) * inv, __uint_as_float(r[8 * c + 1]) * inv);
            v.y = pack_bf16x2(__uint_as_float(r[8 * c + 2]) * inv, __uint_as_float(r[8 * c + 3]) * inv);
            v.z = pack_bf16x2(__uint_as_float(r[8 * c + 4]) * inv, __uint_as_float(r[8 * c + 5]) * inv);
            v.w = pack_bf16x2(__uint_as_float(r[8 * c + 6]) * inv, __uint_as_float(r[8 * c + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + half * 32 + c * 8) = v;
          }
        }
      }
      if (p.split > 1)
        reinterpret_cast<float2*>(q_s)[row] = make_float2(m_used, l_sum);
      else if (l < p.L)             // (an infinite maximum is NaN against itself, as its row is: 0 over a sum of next to 0)
        p.lse[(static_cast<long long>(b) * p.H + h) * p.L + l] = (m_used + log2f(l_sum) + (m_used - m_used)) * 0.6931471805599453f;
    }
    tc_fence_before();
  }

  __syncthreads();
  if (abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  if (p.split > 1) {
    // The CTAs of the cluster merge their parts of the key range: each takes a share of the query rows and reads every
    // CTA's (maximum, sum, row) through distributed shared memory; 16 lanes per row, four columns each.
    cluster_sync();
    if (!abort_flag) {
      const int row_lo = rank * kQ / p.split, row_hi = (rank + 1) * kQ / p.split;
      const int c = threadIdx.x & 15;
      for (int row = row_lo + static_cast<int>(threadIdx.x >> 4); row < row_hi && q0 + row < p.L; row += kThreads / 16) {
        float m = -INFINITY, l = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = 0; i < p.split; ++i) {
          const float2 ml = cluster_ld2(cluster_map(smem_u32(q_s) + row * 8, i));
          const float4 v = cluster_ld4(cluster_map(smem_u32(kv_s) + row * 256 + ((c ^ (row & 15)) << 4), i));
          const float mn = fmaxf(m, ml.x), a = ex2(m - mn), f = ex2(ml.x - mn);
          l = l * a + ml.y * f;
          acc.x = acc.x * a + v.x * f; acc.y = acc.y * a + v.y * f;
          acc.z = acc.z * a + v.z * f; acc.w = acc.w * a + v.w * f;
          m = mn;
        }
        const float inv = 1.f / l;
        __nv_bfloat16* dst = p.o + (static_cast<long long>(b) * p.L + q0 + row) * (p.H * kD) + h * kD;
        reinterpret_cast<uint2*>(dst)[c] =
            make_uint2(pack_bf16x2(acc.x * inv, acc.y * inv), pack_bf16x2(acc.z * inv, acc.w * inv));
        if (c == 0)
          p.lse[(static_cast<long long>(b) * p.H + h) * p.L + q0 + row] = (m + log2f(l)) * 0.6931471805599453f;
      }
    }
    cluster_sync();                            // no CTA leaves while another still reads its rows
  }
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace

int launch_attn_tc_fwd(const moc_attn_shape* s, const void* q, const void* kv, void* o, float* lse,
                       int32_t* status, cudaStream_t stream) {
  MOC_REQUIRE(s->head_dim == kD, "bf16 attention needs head_dim 64");
  MOC_REQUIRE(s->num_heads % s->num_kv_heads == 0, "num_heads must be a multiple of num_kv_heads");
  MOC_REQUIRE((reinterpret_cast<uintptr_t>(o) & 15) == 0, "output must be 16-byte aligned");
  CUtensorMap tq, tkv;
  int rc = make_tmap_bf16_2d(&tq, q, static_cast<uint64_t>(s->batch) * s->seq,
                             static_cast<uint64_t>(s->num_heads) * kD, static_cast<uint64_t>(s->num_heads) * kD,
                             kQ, kD);
  if (rc != MOC_OK) return rc;
  rc = make_tmap_bf16_2d(&tkv, kv, static_cast<uint64_t>(s->batch) * s->n_sel,
                         static_cast<uint64_t>(2 * s->num_kv_heads) * kD,
                         static_cast<uint64_t>(2 * s->num_kv_heads) * kD, kKeys, kD);
  if (rc != MOC_OK) return rc;
  MOC_CUDA_OK(cudaFuncSetAttribute(attn_fwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
  FwdParams p;
  p.o = static_cast<__nv_bfloat16*>(o);
  p.lse = lse;
  p.L = s->seq; p.n_sel = s->n_sel; p.H = s->num_heads; p.HK = s->num_kv_heads;
  p.scale_log2 = s->scale * 1.4426950408889634f;
  p.status = status;
  p.split = attn_key_split(ceil_div(s->seq, kQ) * s->num_heads * s->batch, ceil_div(s->n_sel, kKeys));
  dim3 grid(ceil_div(s->seq, kQ) * p.split, s->num_heads, s->batch);
  MOC_CUDA_OK(launch_clustered(attn_fwd_tc_kernel, grid, kThreads, kSmemBytes, p.split, stream, tq, tkv, p));
  return MOC_OK;
}

}  // namespace moc

extern "C" int moc_exp2_probe(const float* x, float* y, int32_t n, void* stream) {
  using namespace moc;
  MOC_REQUIRE(x && y && n > 0 && n % 2 == 0, "bad exponential probe");
  exp2_probe_kernel<<<ceil_div(n / 2, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, y, n / 2);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}
