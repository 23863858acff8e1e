// Chapter router: fp32 mean-pool, router GEMV, softmax, prefix mask, exact top-k with the total
// order (value descending, chapter id ascending), weight renormalisation, shared-chapter prefix,
// load-balance / auxiliary / z losses and entropy -- and the backward of all of it.
//
// All kernels here are bandwidth or latency bound (the router is ~5e7 FLOPs); reductions are
// done in a fixed order so results do not depend on scheduling.
#include <math.h>

#include <type_traits>

#include "rows_product.cuh"

namespace moc {
namespace {

constexpr int kPoolSplits = 32;       // sequence splits of the mean-pool
constexpr int kLossChunk = 256;       // chapters per CTA in the loss kernels
constexpr int kDpChunk = 16;          // chapters per CTA in the d_pooled kernel

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// x / d for many x and one d, r = 1 / d: the quotient of the rounded reciprocal, corrected by its remainder (Markstein).
// Equal to the division for x = 0 and x >= 2^-100.  The remainder is a multiple of about 2^-47 x: from 2^-102 down fp32
// cannot hold it, and the last bit is off in one of a hundred quotients.
__device__ __forceinline__ float quotient(float x, float d, float r) {
  const float q = x * r;
  return fmaf(fmaf(-q, d, x), r, q);
}
__global__ void quotient_probe_kernel(const float* __restrict__ x, const float* __restrict__ d, float* __restrict__ y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = quotient(x[i], d[i], 1.f / d[i]);
}

// ---- block reductions (fixed order) ----------------------------------------------------------
// (one barrier each: every reduction of a kernel has 32 floats of its own)
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  return warp_sum(lane < nw ? red[lane] : 0.f);
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  return warp_max(lane < nw ? red[lane] : -INFINITY);
}

// ---- forward ---------------------------------------------------------------------------------
// partial[b][split][c] = sum over the split's positions of h[b, t, c]
template <typename T>
__global__ void pool_partial_kernel(const T* __restrict__ h, float* __restrict__ partial, int L, int d) {
  const int b = blockIdx.x, sp = blockIdx.y;
  const int rows_per = (L + kPoolSplits - 1) / kPoolSplits;
  const int t0 = sp * rows_per;
  const int t1 = min(L, t0 + rows_per);
  const T* base = h + (static_cast<long long>(b) * L) * d;
  float* dst = partial + (static_cast<long long>(b) * kPoolSplits + sp) * d;
  if (sizeof(T) == 2 && (d & 7) == 0 && (reinterpret_cast<uintptr_t>(h) & 15) == 0) {
    // bf16 rows in 16-byte pieces: eight columns per thread, four independent row loads in flight
    for (int c8 = threadIdx.x; c8 < (d >> 3); c8 += blockDim.x) {
      float acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
      const uint4* col = reinterpret_cast<const uint4*>(base) + c8;
      const long long stride = d >> 3;
      int t = t0;
      for (; t + 4 <= t1; t += 4) {
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = col[(t + i) * stride];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[2 * j] += __uint_as_float(w[j] << 16);
            acc[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
          }
        }
      }
      for (; t < t1; ++t) {
        const uint4 v = col[t * stride];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[2 * j] += __uint_as_float(w[j] << 16);
          acc[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) dst[c8 * 8 + j] = acc[j];
    }
    return;
  }
  for (int c = threadIdx.x; c < d; c += blockDim.x) {
    float acc = 0.f;
    for (int t = t0; t < t1; ++t) acc += to_f32(base[static_cast<long long>(t) * d + c]);
    dst[c] = acc;
  }
}
// Sequences of up to 1,024 positions in one launch: a CTA owns eight 16-byte pieces of columns, 32 groups of eight lanes sum
// one split each and the partial sums are added in split order (the same sums as the two kernels).  Bound by the latency of
// its row loads; a window of 128 rows: 4.2 us in two launches -> 2.5.
constexpr int kPoolOneMaxRows = 32;     // positions per split up to which one CTA per column piece has loads enough in flight
template <typename T>
__global__ void __launch_bounds__(8 * kPoolSplits)
pool_mean_kernel(const T* __restrict__ h, float* __restrict__ pooled, int L, int d) {
  constexpr int kV = 16 / sizeof(T);
  __shared__ float part[kPoolSplits][8 * kV + 4];
  const int b = blockIdx.x, piece = threadIdx.x & 7, sp = threadIdx.x >> 3;
  const int c0 = (blockIdx.y * 8 + piece) * kV;
  const int rows_per = (L + kPoolSplits - 1) / kPoolSplits;
  const int t0 = sp * rows_per, t1 = min(L, t0 + rows_per);
  float acc[kV];
#pragma unroll
  for (int j = 0; j < kV; ++j) acc[j] = 0.f;
  if (c0 < d) {
    const T* src = h + static_cast<long long>(b) * L * d + c0;
#pragma unroll 8
    for (int t = t0; t < t1; ++t) {
      const uint4 v = *reinterpret_cast<const uint4*>(src + static_cast<long long>(t) * d);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if constexpr (sizeof(T) == 2) {
          acc[2 * j] += __uint_as_float(w[j] << 16);
          acc[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
        } else {
          acc[j] += __uint_as_float(w[j]);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kV; ++j) part[sp][piece * kV + j] = acc[j];
  __syncthreads();
  const int c = blockIdx.y * 8 * kV + threadIdx.x;
  if (threadIdx.x < 8 * kV && c < d) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < kPoolSplits; ++i) t += part[i][threadIdx.x];
    pooled[static_cast<long long>(b) * d + c] = t / static_cast<float>(L);
  }
}
__global__ void pool_finish_kernel(const float* __restrict__ partial, float* __restrict__ pooled, int L, int d,
                                   int total) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int b = i / d, c = i - b * d;
  float acc = 0.f;
  for (int sp = 0; sp < kPoolSplits; ++sp) acc += partial[(static_cast<long long>(b) * kPoolSplits + sp) * d + c];
  pooled[i] = acc / static_cast<float>(L);
}

// pooled[b, c] = sum_t pos_weight[t] * h[b, t, c]: the sequence-rolling pooling of the reference collapses to one
// coefficient per position (the average over t of the rolling-window means is linear in h).  Same split layout
// as the plain mean: partial sums per (batch row, sequence split), then a fixed-order sum over the splits.
template <typename T>
__global__ void pool_weighted_partial_kernel(const T* __restrict__ h, const float* __restrict__ pos_weight,
                                             float* __restrict__ partial, int L, int d) {
  const int b = blockIdx.x, sp = blockIdx.y;
  const int rows_per = (L + kPoolSplits - 1) / kPoolSplits;
  const int t0 = sp * rows_per;
  const int t1 = min(L, t0 + rows_per);
  const T* base = h + (static_cast<long long>(b) * L) * d;
  float* dst = partial + (static_cast<long long>(b) * kPoolSplits + sp) * d;
  for (int c = threadIdx.x; c < d; c += blockDim.x) {
    float acc = 0.f;
    for (int t = t0; t < t1; ++t) acc = fmaf(pos_weight[t], to_f32(base[static_cast<long long>(t) * d + c]), acc);
    dst[c] = acc;
  }
}
__global__ void pool_weighted_finish_kernel(const float* __restrict__ partial, float* __restrict__ pooled, int d,
                                            int total) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int b = i / d, c = i - b * d;
  float acc = 0.f;
  for (int sp = 0; sp < kPoolSplits; ++sp) acc += partial[(static_cast<long long>(b) * kPoolSplits + sp) * d + c];
  pooled[i] = acc;
}
// d_h[b, t, :] (+)= pos_weight[t] * d_pooled[b, :]
template <typename T>
__global__ void pool_weighted_bwd_kernel(const float* __restrict__ d_pooled, const float* __restrict__ pos_weight,
                                         T* __restrict__ d_h, int L, int d, long long total, int accumulate) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long row = i / d;
    const int c = static_cast<int>(i - row * d);
    const int b = static_cast<int>(row / L), t = static_cast<int>(row - static_cast<long long>(b) * L);
    float v = d_pooled[static_cast<long long>(b) * d + c] * pos_weight[t];
    if (accumulate) v += to_f32(d_h[i]);
    if constexpr (sizeof(T) == 4) d_h[i] = v; else d_h[i] = __float2bfloat16(v);
  }
}

// logits[b,c] = <pooled[b,:], w[c,:]> + bias[c].  A warp keeps CH weight rows in registers (NV float4 a lane each) and takes
// eight batch rows at a time from shared memory, the next eight on their way; the 8 CH sums of a lane are reduced together
// (each lane ends up with its own, 31 shuffles for 32 sums instead of 160).  Up to eight rows the kernel is bound by latency
// and takes one chapter per warp; beyond, by shared-memory reads, and four chapters share each of them.  4,097 chapters,
// d 768: 125 -> 19 us for 64 rows against a weight row read again for every eight, 6.5 -> 3.3 for one, 17 -> 9 for eight.
template <int NV, int CH>
__global__ void __launch_bounds__(256)
logits_rows_kernel(const float* __restrict__ pooled, const float* __restrict__ w, const float* __restrict__ bias,
                   float* __restrict__ logits, int B, int d, int C) {
  extern __shared__ float4 sp4[];            // [1 or 2][8][d / 4]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, d4 = d >> 2;
  const int c0 = (blockIdx.x * 8 + warp) * CH;
  const float4* p4 = reinterpret_cast<const float4*>(pooled);
  auto stage = [&](int b0, int buf) {
    const int n = min(8, B - b0) * d4;
    for (int i = threadIdx.x; i < n; i += 256)
      cp_async16(sp4 + buf * 8 * d4 + i, p4 + static_cast<long long>(b0) * d4 + i);
    cp_async_commit();
  };
  stage(0, 0);
  float4 wv[CH][NV];
#pragma unroll
  for (int ch = 0; ch < CH; ++ch) {
    const float4* w4 = reinterpret_cast<const float4*>(w + static_cast<long long>(min(c0 + ch, C - 1)) * d);
#pragma unroll
    for (int i = 0; i < NV; ++i) wv[ch][i] = (lane + 32 * i < d4) ? w4[lane + 32 * i] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int mine = CH == 4 ? lane >> 3 : 0, row = CH == 4 ? lane & 7 : lane >> 2;
  const float bc = (bias != nullptr && c0 + mine < C) ? bias[c0 + mine] : 0.f;
  for (int b0 = 0, buf = 0; b0 < B; b0 += 8, buf ^= 1) {
    if (b0 + 8 < B) { stage(b0 + 8, buf ^ 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
    __syncthreads();
    float a[CH * 8];
#pragma unroll
    for (int i = 0; i < CH * 8; ++i) a[i] = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (lane + 32 * i < d4) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (CH == 1 && b0 + j >= B) break;      // (four chapters: the branch costs more than the last rows)
          const float4 pv = sp4[(buf * 8 + j) * d4 + lane + 32 * i];
#pragma unroll
          for (int ch = 0; ch < CH; ++ch)
            a[ch * 8 + j] = fmaf(wv[ch][i].x, pv.x, fmaf(wv[ch][i].y, pv.y,
                            fmaf(wv[ch][i].z, pv.z, fmaf(wv[ch][i].w, pv.w, a[ch * 8 + j]))));
        }
      }
    }
    // sum i ends in the lanes whose upper bits are i
    int o = 16;
#pragma unroll
    for (int n = CH * 8; n > 1; n >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < n / 2; ++i) {
        const float send = up ? a[i] : a[i + n / 2];
        const float keep = up ? a[i + n / 2] : a[i];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
      o >>= 1;
    }
#pragma unroll
    for (int q = 16 / (CH * 4) / 2; q > 0; q >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], q);
    if (c0 + mine < C && b0 + row < B && (CH == 4 || (lane & 3) == 0))
      logits[static_cast<long long>(b0 + row) * C + c0 + mine] = a[0] + bc;
    __syncthreads();
  }
}
// any other width: one warp per chapter, 8 batch rows per pass
__global__ void logits_kernel(const float* __restrict__ pooled, const float* __restrict__ w,
                              const float* __restrict__ bias, float* __restrict__ logits, int B, int d, int C) {
  extern __shared__ float sp[];   // [8][d]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * (blockDim.x >> 5) + warp;
  for (int b0 = 0; b0 < B; b0 += 8) {
    const int nb = min(8, B - b0);
    __syncthreads();
    for (int i = threadIdx.x; i < nb * d; i += blockDim.x) sp[i] = pooled[static_cast<long long>(b0) * d + i];
    __syncthreads();
    if (c >= C) continue;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    const float* wr = w + static_cast<long long>(c) * d;
    if ((d & 3) == 0) {
      const float4* w4 = reinterpret_cast<const float4*>(wr);
      for (int k = lane; k < d / 4; k += 32) {
        const float4 wv = w4[k];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < nb) {
            const float4 pv = reinterpret_cast<const float4*>(sp + j * d)[k];
            acc[j] = fmaf(wv.x, pv.x, fmaf(wv.y, pv.y, fmaf(wv.z, pv.z, fmaf(wv.w, pv.w, acc[j]))));
          }
      }
    } else {
      for (int k = lane; k < d; k += 32) {
        const float wv = wr[k];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < nb) acc[j] = fmaf(wv, sp[j * d + k], acc[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j < nb) {
        const float s = warp_sum(acc[j]);
        if (lane == 0) logits[static_cast<long long>(b0 + j) * C + c] = s + (bias ? bias[c] : 0.f);
      }
    }
  }
}

// One CTA per batch row: softmax, prefix mask + renormalise, exact top-k, weights, shared prefix.  NV: values per thread
// (rows of up to TH NV chapters), 0 for longer rows.  Bound by its chain of block-wide steps for a few rows: at 4,097 chapters,
// k 64, 16 -> 10 us with TH 1,024 against four radix passes over shared memory.  Thousands of rows take CTAs of 256 threads, whose
// barriers are shorter and chains more, and are bound by the instructions they issue (91 a value and lane, 2.3 a cycle and SM):
// tests of the row's end at the loads and stores alone, addresses that are constants behind one pointer, a fourth CTA an SM that the
// registers then leave room for, lists finished by one warp, candidates ranked as 64-bit words.  8,192 rows of 4,097, k 16: 252 us
// with TH 1,024, 153 with 256, 112 with these (41 for the bytes); 1,000 rows, k 8: 21 -> 17.  128 threads of 33 values: 120 and 26.
constexpr int kBins = 512, kBinBits = 9, kCand = 512, kTailCand = 64;
// (sm: [C] masked probabilities, then [2 k_sel] selection scratch.  Plain pointers: a kernel may have written the logits itself.)
template <int NV, int TH>
__device__ __forceinline__ void select_row(const int b, const float* logits, long long ld, const float* bias, float* probs,
                                           long long* idx, float* weights, int* comb_idx, float* comb_w, float* row_stats,
                                           int C, int k_sel, int S, float rho, float* sm) {
  float* pt = sm;                          // p~
  uint32_t* sel_key = reinterpret_cast<uint32_t*>(sm + C);   // [k_sel]
  int* sel_idx = reinterpret_cast<int*>(sel_key + k_sel);    // [k_sel]
  __shared__ float red[5][32];
  __shared__ int hist[256];
  __shared__ uint32_t s_prefix;
  __shared__ int s_krem, s_count, s_ties;
  __shared__ int bins[NV > 0 ? kBins : 1], wsum[32];
  __shared__ uint32_t mm[64];
  __shared__ unsigned long long cand[NV > 0 ? kCand : 1];       // value, then the id's complement: larger is earlier

  const float* z = logits + b * ld;       // (bias: not yet in the logits, or nullptr)
  auto logit = [&](int c) { return bias != nullptr ? z[c] + bias[c] : z[c]; };
  float* p = probs + static_cast<long long>(b) * C;

  // NV > 0: the row's values stay in registers between the passes (c = threadIdx.x + i * blockDim.x), and the shared copy
  // is only made for the radix select.  Sums run in the same order either way.
  constexpr int kN = NV > 0 ? NV : 1;
  float v[kN];
  // Columns past the row hold -inf, whose exponential adds nothing: one comparison at the loads instead of one in every pass.
  const int left = C - static_cast<int>(threadIdx.x);
  float m = -INFINITY;
  if constexpr (NV > 0) {
    const float* zt = z + threadIdx.x;
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = i * TH < left ? zt[i * TH] : -INFINITY;       // (all loads first: they are independent)
    if (bias != nullptr) {
      const float* bt = bias + threadIdx.x;
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (i * TH < left) v[i] += bt[i * TH];
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) m = fmaxf(m, v[i]);
  } else {
    for (int c = threadIdx.x; c < C; c += blockDim.x) m = fmaxf(m, logit(c));
  }
  m = block_max(m, red[0]);
  // A thread with an exponential below 2^-83 (other than zero) divides.  Both quotients below stay within what `quotient` is
  // exact for otherwise: the exponentials, and those over a sum of at most 2^14.  (8,192 rows of 4,097 chapters: 157 us
  // without the test, 161 with it, 184 with a test of every value on its own.)
  uint32_t least = 0xFFFFFFFFu;
  auto divide = [&](float d) {             // v[i] = v[i] / d
    if constexpr (NV > 0) {
      if (least < (static_cast<uint32_t>(127 - 83) << 23) - 1u) {
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = v[i] / d;
      } else {
        const float r = 1.f / d;
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = quotient(v[i], d, r);
      }
    }
  };
  float s = 0.f;
  if constexpr (NV > 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      v[i] = expf(v[i] - m);
      s += v[i];
      least = min(least, __float_as_uint(v[i]) - 1u);       // (zero wraps around)
    }
  } else {
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      const float e = expf(logit(c) - m);
      pt[c] = e;
      s += e;
    }
  }
  const float denom = block_sum(s, red[1]);
  float ms = 0.f;
  if constexpr (NV > 0) {
    divide(denom);
    float* ptr = p + threadIdx.x;
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (i * TH < left) ptr[i * TH] = v[i];
    if (S > 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (static_cast<int>(threadIdx.x) + i * TH < S) v[i] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) ms += v[i];
  } else {
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      const float pv = pt[c] / denom;
      p[c] = pv;
      const float pm = (c < S) ? 0.f : pv;
      pt[c] = pm;
      ms += pm;
    }
  }
  // without shared chapters nothing waits for this sum: its second half runs at the end, past the barriers in between
  const bool late_mass = NV > 0 && S == 0 && k_sel > 0;
  float masked_mass = 0.f;
  if (late_mass) {
    ms = warp_sum(ms);
    if ((threadIdx.x & 31) == 0) red[2][threadIdx.x >> 5] = ms;
  } else {
    masked_mass = block_sum(ms, red[2]);
    const float dn0 = fmaxf(masked_mass, 1e-12f);
    if constexpr (NV > 0) {
      if (S > 0) divide(dn0);
    } else {
      if (S > 0)
        for (int c = threadIdx.x; c < C; c += blockDim.x) pt[c] = pt[c] / dn0;
    }
    __syncthreads();
  }

  float topk_mass = 0.f, comb_mass = static_cast<float>(S);
  // Lists of up to 32 entries are finished by the first warp alone, without barriers (the sums of the other warps are zero).
  int step = blockDim.x;
  auto tail_sum = [&](float x, float* r) { return step == 32 ? warp_sum(x) : block_sum(x, r); };
  if (k_sel > 0) {
    float* srt_w = sm;                         // sorted: weight and id, over p~ (no longer needed by then)
    int* srt_i = reinterpret_cast<int*>(sm + k_sel);
    bool selected = false;
    if constexpr (NV > 0) {
      // At least k values are as large as the k-th largest of the threads' own maxima, and few more: a histogram of the TH
      // maxima over their range (one atomic per thread; the probabilities of one row share their leading bits, so radix
      // passes over all of them pile up in a few bins) gives a bound, and what lies above it is ranked.
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      constexpr int kPer = kBins / TH > 2 ? kBins / TH : 2, kOwners = kBins / kPer, kWarps = TH / 32;
      uint32_t top = 0u;
#pragma unroll
      for (int i = 0; i < NV; ++i) top = max(top, __float_as_uint(v[i]));       // (zero past the row and for shared chapters)
      uint32_t lo = __reduce_min_sync(0xffffffffu, top), hi = __reduce_max_sync(0xffffffffu, top);
      for (int i = threadIdx.x; i < kBins; i += TH) bins[i] = 0;
      if (lane == 0) { mm[warp] = lo; mm[32 + warp] = hi; }
      if (threadIdx.x == 0) { s_count = 0; s_prefix = 0u; }
      __syncthreads();
      lo = __reduce_min_sync(0xffffffffu, lane < kWarps ? mm[lane] : 0xFFFFFFFFu);
      hi = __reduce_max_sync(0xffffffffu, lane < kWarps ? mm[32 + lane] : 0u);
      const int sh = max(0, 32 - __clz(hi - lo) - kBinBits);
      if (k_sel <= TH / 2) {
        atomicAdd(&bins[(top - lo) >> sh], 1);
        __syncthreads();
        // an owner has kPer bins, from the top down; the one whose bin reaches k publishes it
        if (threadIdx.x < kOwners) {
          const int first = kBins - 1 - kPer * static_cast<int>(threadIdx.x);
          int h[kPer], incl = 0;
#pragma unroll
          for (int i = 0; i < kPer; ++i) { h[i] = bins[first - i]; incl += h[i]; }
          const int mine = incl;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
          }
          if (lane == 31) wsum[warp] = incl;
          asm volatile("bar.sync 1, %0;" ::"n"(kOwners) : "memory");
          int above = incl - mine;
          for (int w = 0; w < warp; ++w) above += wsum[w];
#pragma unroll
          for (int i = 0; i < kPer; ++i) {
            if (above < k_sel && k_sel <= above + h[i]) s_prefix = first - i;
            above += h[i];
          }
        }
        __syncthreads();
        const uint32_t edge = lo + (s_prefix << sh);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int c = threadIdx.x + i * TH;
          if (__float_as_uint(v[i]) >= edge && c < C && c >= S) {
            const int pos = atomicAdd(&s_count, 1);
            if (pos < kCand) cand[pos] = static_cast<unsigned long long>(__float_as_uint(v[i])) << 32 | ~static_cast<uint32_t>(c);
          }
        }
        __syncthreads();
        const int n = s_count;
        if (n >= k_sel && n <= kCand) {
          if (n <= kTailCand && S + k_sel <= 32) {
            if (warp > 0) return;
            step = 32;
          }
          for (int t = threadIdx.x; t < n; t += step) {
            const unsigned long long mine = cand[t];
            int rank = 0;
#pragma unroll 4
            for (int j = 0; j < n; ++j) rank += cand[j] > mine;
            if (rank < k_sel) {
              srt_w[rank] = __uint_as_float(static_cast<uint32_t>(mine >> 32));
              srt_i[rank] = ~static_cast<uint32_t>(mine);
            }
          }
          selected = true;
        }
      }
      if (!selected) {
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (threadIdx.x + i * TH < C) pt[threadIdx.x + i * TH] = v[i];
      }
      if (step == 32) __syncwarp(); else __syncthreads();
    }
    if (!selected) {
    // radix select on the fp32 bit pattern (non-negative values order like unsigned integers)
    if (threadIdx.x == 0) { s_prefix = 0u; s_krem = k_sel; }
    uint32_t mask = 0u;
    for (int pass = 3; pass >= 0; --pass) {
      for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
      __syncthreads();
      const uint32_t prefix = s_prefix;
      for (int c = threadIdx.x; c < C; c += blockDim.x) {
        const uint32_t key = __float_as_uint(pt[c]);
        if ((key & mask) == prefix) atomicAdd(&hist[(key >> (8 * pass)) & 255u], 1);
      }
      __syncthreads();
      if (threadIdx.x < 32) {
        // warp 0 finds, from the top bin down, the bin in which the running count reaches s_krem
        const int lane = threadIdx.x;
        int h8[8], sl = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) { h8[i] = hist[lane * 8 + i]; sl += h8[i]; }
        int incl = sl;                       // inclusive suffix sum over lanes lane..31
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_down_sync(0xffffffffu, incl, o);
          if (lane + o < 32) incl += t;
        }
        const int above = incl - sl;         // elements in bins owned by higher lanes
        const int rem0 = s_krem;
        const bool mine = (above < rem0) && (rem0 <= incl);
        const unsigned who = __ballot_sync(0xffffffffu, mine);
        // all remaining elements sit in bin 0 of lane 0 when no lane qualifies (cannot happen while rem0 <= count)
        const int owner = who ? (31 - __clz(who)) : 0;
        if (lane == owner) {
          int rem = rem0 - above, i = 7;
          for (; i > 0; --i) {
            if (h8[i] >= rem) break;
            rem -= h8[i];
          }
          s_krem = rem;
          s_prefix = prefix | (static_cast<uint32_t>(lane * 8 + i) << (8 * pass));
          s_ties = h8[i];
        }
      }
      mask |= 0xFFu << (8 * pass);
      __syncthreads();
    }
    const uint32_t thr = s_prefix;     // bit pattern of the k-th largest value
    const int need_ties = s_krem;      // how many entries equal to it are selected
    const int have_ties = s_ties;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      const uint32_t key = __float_as_uint(pt[c]);
      if (key > thr || (key == thr && have_ties == need_ties)) {
        const int pos = atomicAdd(&s_count, 1);
        if (pos < k_sel) { sel_key[pos] = key; sel_idx[pos] = c; }
      }
    }
    __syncthreads();
    if (have_ties != need_ties && threadIdx.x == 0) {
      int pos = s_count, taken = 0;            // more ties than slots: lowest chapter ids win
      for (int c = 0; c < C && taken < need_ties; ++c) {
        if (__float_as_uint(pt[c]) == thr) {
          if (pos < k_sel) { sel_key[pos] = thr; sel_idx[pos] = c; }
          ++pos; ++taken;
        }
      }
    }
    __syncthreads();
    // rank sort of the k selected entries: value descending, chapter id ascending (shared memory)
    constexpr int kMine = 1024 / TH;           // k_sel <= 1024
    uint32_t kt_reg[kMine]; int it_reg[kMine]; int rk_reg[kMine];
#pragma unroll
    for (int q = 0; q < kMine; ++q) {
      const int t = threadIdx.x + q * TH;
      if (t < k_sel) {
        const uint32_t kt = sel_key[t];
        const int it = sel_idx[t];
        int rank = 0;
        for (int j = 0; j < k_sel; ++j) {
          const uint32_t kj = sel_key[j];
          rank += (kj > kt) || (kj == kt && sel_idx[j] < it);
        }
        kt_reg[q] = kt; it_reg[q] = it; rk_reg[q] = rank;
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kMine; ++q)
      if (threadIdx.x + q * TH < k_sel) { srt_w[rk_reg[q]] = __uint_as_float(kt_reg[q]); srt_i[rk_reg[q]] = it_reg[q]; }
    __syncthreads();
    }
    float part = 0.f;
    for (int j = threadIdx.x; j < k_sel; j += step) part += srt_w[j];
    topk_mass = tail_sum(part, red[3]);
    const float dn = fmaxf(topk_mass, 1e-12f);
    long long* out_idx = idx + static_cast<long long>(b) * k_sel;
    float* out_w = weights + static_cast<long long>(b) * k_sel;
    float cpart = 0.f;
    for (int j = threadIdx.x; j < k_sel; j += step) {
      const float wj = srt_w[j] / dn;
      srt_w[j] = wj;
      out_w[j] = wj;
      out_idx[j] = srt_i[j];
      cpart += wj * rho;
    }
    comb_mass = static_cast<float>(S) + tail_sum(cpart, red[4]);
    if (step == 32) __syncwarp();
  }
  if (late_mass) masked_mass = warp_sum(static_cast<int>(threadIdx.x) < TH / 32 ? red[2][threadIdx.x & 31] : 0.f);   // (read by thread 0)
  // shared prefix + renormalised combined weights (only meaningful when S > 0; with S == 0 the
  // combined lists are the routed lists unchanged)
  const int kc = S + k_sel;
  for (int j = threadIdx.x; j < kc; j += step) {
    int ci; float u;
    if (j < S) { ci = j; u = 1.f; }
    else { ci = reinterpret_cast<int*>(sm + k_sel)[j - S]; u = sm[j - S] * (S > 0 ? rho : 1.f); }
    if (comb_idx == nullptr) break;        // (uniform: a caller of token rows has no use for the joint list)
    comb_idx[static_cast<long long>(b) * kc + j] = ci;
    comb_w[static_cast<long long>(b) * kc + j] = (S > 0) ? u / fmaxf(comb_mass, 1e-12f) : u;
  }
  if (threadIdx.x == 0) {
    float* rs = row_stats + static_cast<long long>(b) * 4;
    rs[0] = m + logf(denom);
    rs[1] = masked_mass;
    rs[2] = topk_mass;
    rs[3] = comb_mass;
  }
}
template <int NV, int TH>
__global__ void __launch_bounds__(TH, TH == 256 ? (NV > 17 ? 2 : NV > 5 ? 4 : 6) : (NV > 5 ? 1 : 2))
select_kernel(const float* __restrict__ logits, long long ld, const float* __restrict__ bias, float* __restrict__ probs, long long* __restrict__ idx,
              float* __restrict__ weights, int* __restrict__ comb_idx, float* __restrict__ comb_w,
              float* __restrict__ row_stats, int C, int k_sel, int S, float rho) {
  extern __shared__ float sm[];
  select_row<NV, TH>(blockIdx.x, logits, ld, bias, probs, idx, weights, comb_idx, comb_w, row_stats, C, k_sel, S, rho, sm);
}

// A decoding step of one or two sequences, issued by the host: pooling, logits and selection in one launch, by one cluster of 16 CTAs
// that meets at its hardware barrier between them (the same sums in the same order as the kernels above).  Such a step waits for the
// host, which needs some 4 us for each launch; on the device 16 SMs take longer than all of them (23 us against 15 for one sequence,
// 27 against 15 for two, of a window of 128 and 4,097 chapters), so passes that are captured, whose launches cost nothing when they are
// replayed, and those with work enough to hide the launches keep the kernels above.  The remaining CTAs, clusters of their own,
// are a projection of as many rows that needs nothing of the routing: the step's queries, one warp a column.
// One sequence, host and device overlapped: 52 -> 44 us a step, 7 launches -> 4.
constexpr int kFrontCtas = 16, kFrontRows = 2, kFrontChapters = 9 * 1024;
constexpr int kFrontSmemMost = (kFrontChapters + 2 * 1024) * 4;    // the selection's (the pooling takes 33 KiB, the pooled states 8)
struct FrontParams {
  float *pooled, *logits, *probs;
  long long* idx;
  float* weights;
  int* comb_idx;
  float *comb_w, *row_stats;
  int B, L, d, C, k_sel, S;
  float rho;
  RowsProduct q;
};
// ND: float4 of a weight row per lane
template <typename T, int NV, int ND>
__global__ void __launch_bounds__(1024, 1)
route_front_kernel(const T* __restrict__ h, const float* __restrict__ w, const float* __restrict__ bias, FrontParams p) {
  extern __shared__ float4 front_smem[];
  float* sm = reinterpret_cast<float*>(front_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x >= kFrontCtas) {
    const int col = (static_cast<int>(blockIdx.x) - kFrontCtas) * 32 + warp;
    if (col < p.q.n) rows_product_column<kFrontRows>(p.q, col, lane);
    return;
  }
  const int rank = static_cast<int>(blockIdx.x);
  const int B = p.B, L = p.L, d = p.d, C = p.C;
  {
    // mean over the positions: warp = split of the sequence, lane = (sequence, 16-byte piece of columns)
    constexpr int kV = 16 / sizeof(T), kPart = 32 * kV + 4;
    const int pieces = d / kV, p0 = rank * pieces / kFrontCtas, np = (rank + 1) * pieces / kFrontCtas - p0, items = B * np;
    const int rows_per = (L + kPoolSplits - 1) / kPoolSplits, t0 = warp * rows_per, t1 = min(L, t0 + rows_per);
    for (int i0 = 0; i0 < items; i0 += 32) {
      float acc[kV];
#pragma unroll
      for (int j = 0; j < kV; ++j) acc[j] = 0.f;
      if (i0 + lane < items) {
        const int b = (i0 + lane) / np, piece = p0 + (i0 + lane) - b * np;
        const T* src = h + static_cast<long long>(b) * L * d + piece * kV;
#pragma unroll 4
        for (int t = t0; t < t1; ++t) {
          const uint4 v = *reinterpret_cast<const uint4*>(src + static_cast<long long>(t) * d);
          const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if constexpr (sizeof(T) == 2) {
              acc[2 * j] += __uint_as_float(x[j] << 16);
              acc[2 * j + 1] += __uint_as_float(x[j] & 0xFFFF0000u);
            } else {
              acc[j] += __uint_as_float(x[j]);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kV; ++j) sm[warp * kPart + lane * kV + j] = acc[j];
      __syncthreads();
      const int n = min(32, items - i0) * kV;
      if (static_cast<int>(threadIdx.x) < n) {
        const int item = i0 + static_cast<int>(threadIdx.x) / kV, b = item / np;
        float t = 0.f;
#pragma unroll 8
        for (int i = 0; i < kPoolSplits; ++i) t += sm[i * kPart + threadIdx.x];
        p.pooled[static_cast<long long>(b) * d + (p0 + item - b * np) * kV + threadIdx.x % kV] = t / static_cast<float>(L);
      }
      __syncthreads();
    }
  }
  cluster_sync();
  {
    const int d4 = d >> 2;
    float4* sp4 = front_smem;
    for (int i = threadIdx.x; i < B * d4; i += 1024) sp4[i] = __ldcg(reinterpret_cast<const float4*>(p.pooled) + i);
    __syncthreads();
    const int c_hi = static_cast<int>(static_cast<long long>(rank + 1) * C / kFrontCtas);
    for (int c = static_cast<int>(static_cast<long long>(rank) * C / kFrontCtas) + warp; c < c_hi; c += 32) {
      const float4* w4 = reinterpret_cast<const float4*>(w + static_cast<long long>(c) * d);
      float4 wv[ND];
#pragma unroll
      for (int i = 0; i < ND; ++i) wv[i] = lane + 32 * i < d4 ? w4[lane + 32 * i] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float bc = bias != nullptr ? bias[c] : 0.f;
      for (int b = 0; b < B; ++b) {
        float a = 0.f;
#pragma unroll
        for (int i = 0; i < ND; ++i) {
          if (lane + 32 * i < d4) {
            const float4 pv = sp4[b * d4 + lane + 32 * i];
            a = fmaf(wv[i].x, pv.x, fmaf(wv[i].y, pv.y, fmaf(wv[i].z, pv.z, fmaf(wv[i].w, pv.w, a))));
          }
        }
        a = warp_sum(a);
        if (lane == 0) p.logits[static_cast<long long>(b) * C + c] = a + bc;
      }
    }
  }
  cluster_sync();
  if (rank < B)
    select_row<NV, 1024>(rank, p.logits, C, nullptr, p.probs, p.idx, p.weights, p.comb_idx, p.comb_w, p.row_stats, C, p.k_sel, p.S,
                         p.rho, sm);
}

// Per chapter chunk: f, mean p^2, and partial sums of the three chapter-separable loss terms.
__global__ void loss_partial_kernel(const float* __restrict__ probs, const long long* __restrict__ idx,
                                    float* __restrict__ chapter_stats, float* __restrict__ partial,
                                    int B, int C, int k_sel) {
  __shared__ int cnt[kLossChunk];
  __shared__ float red[5][32];
  const int c0 = blockIdx.x * kLossChunk;
  for (int i = threadIdx.x; i < kLossChunk; i += blockDim.x) cnt[i] = 0;
  __syncthreads();
  const long long n_idx = static_cast<long long>(B) * k_sel;
  for (long long i = threadIdx.x; i < n_idx; i += blockDim.x) {
    const int c = static_cast<int>(idx[i]) - c0;
    if (c >= 0 && c < kLossChunk) atomicAdd(&cnt[c], 1);
  }
  __syncthreads();
  float lb = 0.f, aux = 0.f, ent = 0.f;
  const int c = c0 + threadIdx.x;
  if (threadIdx.x < kLossChunk && c < C) {
    float ps = 0.f, p2 = 0.f, e = 0.f;
    for (int b = 0; b < B; ++b) {
      const float pv = probs[static_cast<long long>(b) * C + c];
      ps += pv;
      p2 += pv * pv;
      e += pv * logf(fmaxf(pv, 1e-12f));
    }
    const float f = static_cast<float>(cnt[threadIdx.x]) / static_cast<float>(B);
    const float P = ps / static_cast<float>(B);
    const float q = p2 / static_cast<float>(B);
    chapter_stats[c] = f;
    chapter_stats[C + c] = q;
    lb = f * P;
    const float dv = q - 1.f / static_cast<float>(C);
    aux = dv * dv;
    ent = e;
  }
  lb = block_sum(lb, red[0]);
  aux = block_sum(aux, red[1]);
  ent = block_sum(ent, red[2]);
  if (threadIdx.x == 0) {
    partial[blockIdx.x * 3 + 0] = lb;
    partial[blockIdx.x * 3 + 1] = aux;
    partial[blockIdx.x * 3 + 2] = ent;
  }
}
// The same statistics for many routing rows (token-level routing: B = batch * seq): the rows are cut into `splits`
// ranges, every (chapter chunk, range) CTA leaves {sum p, sum p^2, sum p log p, count} per chapter, and a second kernel
// adds the ranges in order before the non-linear terms are formed.
__global__ void loss_rows_partial_kernel(const float* __restrict__ probs, const long long* __restrict__ idx,
                                         float* __restrict__ part, int B, int C, int k_sel, int rows_per_split) {
  __shared__ int cnt[kLossChunk];
  const int c0 = blockIdx.x * kLossChunk;
  const int r0 = blockIdx.y * rows_per_split, r1 = min(B, r0 + rows_per_split);
  cnt[threadIdx.x] = 0;
  __syncthreads();
  for (long long i = static_cast<long long>(r0) * k_sel + threadIdx.x; i < static_cast<long long>(r1) * k_sel;
       i += blockDim.x) {
    const int c = static_cast<int>(idx[i]) - c0;
    if (c >= 0 && c < kLossChunk) atomicAdd(&cnt[c], 1);
  }
  __syncthreads();
  const int c = c0 + threadIdx.x;
  if (c >= C) return;
  float ps = 0.f, p2 = 0.f, e = 0.f;
  for (int b = r0; b < r1; ++b) {
    const float pv = probs[static_cast<long long>(b) * C + c];
    ps += pv;
    p2 += pv * pv;
    e += pv * logf(fmaxf(pv, 1e-12f));
  }
  float4* dst = reinterpret_cast<float4*>(part) + static_cast<long long>(blockIdx.y) * C + c;
  *dst = make_float4(ps, p2, e, static_cast<float>(cnt[threadIdx.x]));
}
__global__ void loss_rows_finish_kernel(const float* __restrict__ part, float* __restrict__ chapter_stats,
                                        float* __restrict__ partial, int B, int C, int splits) {
  __shared__ float red[5][32];
  const int c = blockIdx.x * kLossChunk + threadIdx.x;
  float lb = 0.f, aux = 0.f, ent = 0.f;
  if (c < C) {
    float ps = 0.f, p2 = 0.f, e = 0.f, n = 0.f;
    for (int sp = 0; sp < splits; ++sp) {
      const float4 v = reinterpret_cast<const float4*>(part)[static_cast<long long>(sp) * C + c];
      ps += v.x; p2 += v.y; e += v.z; n += v.w;
    }
    const float f = n / static_cast<float>(B);
    const float P = ps / static_cast<float>(B);
    const float q = p2 / static_cast<float>(B);
    chapter_stats[c] = f;
    chapter_stats[C + c] = q;
    lb = f * P;
    const float dv = q - 1.f / static_cast<float>(C);
    aux = dv * dv;
    ent = e;
  }
  lb = block_sum(lb, red[0]);
  aux = block_sum(aux, red[1]);
  ent = block_sum(ent, red[2]);
  if (threadIdx.x == 0) {
    partial[blockIdx.x * 3 + 0] = lb;
    partial[blockIdx.x * 3 + 1] = aux;
    partial[blockIdx.x * 3 + 2] = ent;
  }
}
__global__ void loss_finish_kernel(const float* __restrict__ partial, const float* __restrict__ row_stats,
                                   float* __restrict__ losses, int nblk, int B, int C) {
  // one CTA, of one warp for a few rows; every thread sums a strided share in a fixed order, then a fixed-order tree.  8,192 rows:
  // 16 us with one warp, 6 with 1,024 threads; 500: 3.6 and 2.3
  __shared__ float red[4][32];
  float lb = 0.f, aux = 0.f, ent = 0.f, z = 0.f;
  for (int i = threadIdx.x; i < nblk; i += blockDim.x) { lb += partial[i * 3]; aux += partial[i * 3 + 1]; ent += partial[i * 3 + 2]; }
  for (int b = threadIdx.x; b < B; b += blockDim.x) { const float l = row_stats[static_cast<long long>(b) * 4]; z += l * l; }
  lb = block_sum(lb, red[0]); aux = block_sum(aux, red[1]); ent = block_sum(ent, red[2]); z = block_sum(z, red[3]);
  if (threadIdx.x == 0) {
    losses[0] = static_cast<float>(C) * lb;
    losses[1] = aux / static_cast<float>(C);
    losses[2] = z / static_cast<float>(B);
    losses[3] = -ent / static_cast<float>(B);
  }
}

// out[0] = c . losses, or with grad: out[0..3] = grad * c
__global__ void loss_total_kernel(const float* __restrict__ losses, const float* __restrict__ grad, float4 c,
                                  float* __restrict__ out) {
  const float cs[4] = {c.x, c.y, c.z, c.w};
  if (grad != nullptr) {
    if (threadIdx.x < 4) out[threadIdx.x] = grad[0] * cs[threadIdx.x];
  } else if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < 4; ++i)
      if (cs[i] != 0.f) t += cs[i] * losses[i];
    out[0] = t;
  }
}

// dst[r, c] = bias[c] + sum_t src[r, t * ld + c], smallest term (highest t) first
__global__ void sum_terms_kernel(const float* __restrict__ src, const float* __restrict__ bias,
                                 float* __restrict__ dst, long long rows, int cols, int ld, int terms) {
  const long long total = rows * cols;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / cols;
    const int c = static_cast<int>(i - r * cols);
    const float* p = src + r * static_cast<long long>(ld) * terms + c;
    float acc = 0.f;
    for (int t = terms - 1; t >= 0; --t) acc += p[static_cast<long long>(t) * ld];
    dst[i] = bias != nullptr ? acc + bias[c] : acc;
  }
}
// partial[chunk][c] = sum over the chunk's rows of the three terms of column c: 32 groups of eight 16-byte pieces
constexpr int kTermRows = 256;
__global__ void __launch_bounds__(256)
term_col_sum_kernel(const __nv_bfloat16* __restrict__ terms, float* __restrict__ partial, int rows, int ld) {
  __shared__ float red[32][65];
  const int piece = threadIdx.x & 7, g = threadIdx.x >> 3;
  const int c = blockIdx.x * 64 + piece * 8, r0 = blockIdx.y * kTermRows;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (c < ld) {
#pragma unroll 4
    for (int r = r0 + g; r < min(rows, r0 + kTermRows); r += 32) {
#pragma unroll
      for (int t = 2; t >= 0; --t) {
        const uint4 v = *reinterpret_cast<const uint4*>(terms + (static_cast<long long>(t) * rows + r) * ld + c);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[2 * j] += __uint_as_float(w[j] << 16);
          acc[2 * j + 1] += __uint_as_float(w[j] & 0xFFFF0000u);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) red[g][piece * 8 + j] = acc[j];
  __syncthreads();
  const int col = blockIdx.x * 64 + threadIdx.x;
  if (threadIdx.x < 64 && col < ld) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) t += red[i][threadIdx.x];
    partial[static_cast<long long>(blockIdx.y) * ld + col] = t;
  }
}
// out[c] = sum_r x[r, c]: one CTA per 32 columns, 8 row groups, fixed-order sums
__global__ void col_sum_kernel(const float* __restrict__ x, float* __restrict__ out, long long rows, int cols, int ld) {
  __shared__ float part[8][32];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), g = threadIdx.x >> 5;
  float acc = 0.f;
  if (c < cols)
    for (long long r = g; r < rows; r += 8) acc += x[r * ld + c];
  part[g][threadIdx.x & 31] = acc;
  __syncthreads();
  if (g == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += part[i][threadIdx.x];
    out[c] = t;
  }
}

// ---- backward --------------------------------------------------------------------------------
// One CTA per row: gradient of everything downstream of the logits.  TERMS: the gradient leaves as three bf16 terms ([3][B][ld],
// zeros behind column C), what the products that follow on the tensor cores read.
// NV > 0: the row's probabilities stay in registers (rows of up to TH NV chapters), all loads in flight together.  8,192 rows
// of 4,097: 227 us with TH 1,024, a pad copy of 93 us and a pass of 133 us into the terms -> 138 us in all.  Those issued 89
// instructions a value and lane: with the layout of the columns known to the compiler, no test of the row's end but at the loads,
// and the sums over the list left to one warp while the others load, 80 us (52 for the bytes); 1,000 rows, k 8: 23 -> 14.
template <int NV, int TH, bool TERMS>
__global__ void __launch_bounds__(TH, TH == 256 ? 4 : 1)
dlogits_kernel(const float* __restrict__ probs, const long long* __restrict__ idx,
               const float* __restrict__ weights, const float* __restrict__ comb_w,
               const float* __restrict__ row_stats, const float* __restrict__ chapter_stats,
               const float* __restrict__ d_weights, const float* __restrict__ d_comb_w,
               const float* __restrict__ d_losses, float* __restrict__ d_logits, __nv_bfloat16* __restrict__ terms, int ld,
               int B, int C, int k_sel, int S, float rho) {
  extern __shared__ float4 dp_smem[];
  float* dp = reinterpret_cast<float*>(dp_smem);        // [NV TH], or [C]
  __shared__ float red[5][32];
  __shared__ float s_dv[1024];    // k_sel <= 1024
  const int b = blockIdx.x;
  const float* p = probs + static_cast<long long>(b) * C;
  const float lse = row_stats[b * 4 + 0], s_mass = row_stats[b * 4 + 1];
  const float v_mass = row_stats[b * 4 + 2], u_mass = row_stats[b * 4 + 3];
  const float g_lb = d_losses ? d_losses[0] : 0.f, g_aux = d_losses ? d_losses[1] : 0.f;
  const float g_z = d_losses ? d_losses[2] : 0.f, g_ent = d_losses ? d_losses[3] : 0.f;
  const int kc = S + k_sel;

  // A thread's columns: pairs where terms go out in pairs, single ones otherwise.  Past the row the probabilities are zero.
  constexpr int kN = NV > 0 ? NV : 1;
  float pr[kN], g[kN];
  const int first = TERMS ? 2 * static_cast<int>(threadIdx.x) : static_cast<int>(threadIdx.x), left = C - first;
  auto off = [](int i) { return TERMS ? (i & 1) + (i >> 1) * 2 * TH : i * TH; };
  if constexpr (NV > 0) {
    const float* pt = p + first;
#pragma unroll
    for (int i = 0; i < kN; ++i) pr[i] = off(i) < left ? pt[off(i)] : 0.f;
  }
  // (a)+(b): gradients of the k selected (unnormalised) masked probabilities v_j
  __shared__ float s_w[1024];
  const bool one_warp = kc <= 32;        // the first warp takes these sums alone, the others go on
  float A = 0.f;
  long long my_idx = 0;
  if (!one_warp || threadIdx.x < 32) {
    const int step = one_warp ? 32 : static_cast<int>(blockDim.x);
    auto list_sum = [&](float x, float* r) { return one_warp ? warp_sum(x) : block_sum(x, r); };
    if (one_warp && static_cast<int>(threadIdx.x) < k_sel) my_idx = idx[static_cast<long long>(b) * k_sel + threadIdx.x];
    float dotu_p = 0.f;
    if (d_comb_w != nullptr && S > 0)
      for (int i = threadIdx.x; i < kc; i += step)
        dotu_p += d_comb_w[static_cast<long long>(b) * kc + i] * comb_w[static_cast<long long>(b) * kc + i];
    const float dotu = (d_comb_w != nullptr && S > 0) ? list_sum(dotu_p, red[0]) : 0.f;
    float dotw_p = 0.f;
    for (int j = threadIdx.x; j < k_sel; j += step) {
      float dw = d_weights ? d_weights[static_cast<long long>(b) * k_sel + j] : 0.f;
      if (d_comb_w != nullptr) {
        const float dcu = d_comb_w[static_cast<long long>(b) * kc + S + j];
        if (S > 0) dw += rho * ((u_mass >= 1e-12f) ? (dcu - dotu) / u_mass : dcu / 1e-12f);
        else dw += dcu;
      }
      const float wj = weights[static_cast<long long>(b) * k_sel + j];
      s_dv[j] = dw;
      s_w[j] = wj;
      dotw_p += dw * wj;
    }
    const float dotw = list_sum(dotw_p, red[1]);
    float a_p = 0.f;
    for (int j = threadIdx.x; j < k_sel; j += step) {
      const float dv = (v_mass >= 1e-12f) ? (s_dv[j] - dotw) / v_mass : s_dv[j] / 1e-12f;
      s_dv[j] = dv;
      a_p += dv * (s_w[j] * fmaxf(v_mass, 1e-12f));   // v_j
    }
    A = list_sum(a_p, red[2]);
  }
  if (one_warp && S > 0) {               // (only shared chapters make the sum a part of every column)
    if (threadIdx.x == 0) red[4][0] = A;
    __syncthreads();
    A = red[4][0];
  }
  const bool renorm = (S > 0);
  const float inv_s = renorm ? ((s_mass >= 1e-12f) ? 1.f / s_mass : 1e12f) : 1.f;
  const float dense = (renorm && s_mass >= 1e-12f) ? -A * inv_s : 0.f;
  const float invB = 1.f / static_cast<float>(B), invC = 1.f / static_cast<float>(C);
  auto dense_grad = [&](int c, float pv) {
    float g = (c >= S) ? dense : 0.f;
    // (a loss without a gradient costs nothing, and its statistics may not have been computed)
    if (g_lb != 0.f) g += g_lb * static_cast<float>(C) * chapter_stats[c] * invB;
    if (g_aux != 0.f) g += g_aux * (2.f * invC) * (chapter_stats[C + c] - invC) * (2.f * pv * invB);
    if (g_ent != 0.f) g += g_ent * (-invB) * (logf(fmaxf(pv, 1e-12f)) + (pv > 1e-12f ? 1.f : 0.f));
    return g;
  };
  if constexpr (NV > 0) {
    if (g_aux == 0.f && g_ent == 0.f) {          // the usual losses; all loads first, they are independent
      const float* ft = chapter_stats + first;
#pragma unroll
      for (int i = 0; i < kN; ++i) g[i] = 0.f;
      if (g_lb != 0.f) {
#pragma unroll
        for (int i = 0; i < kN; ++i) g[i] = off(i) < left ? ft[off(i)] : 0.f;
#pragma unroll
        for (int i = 0; i < kN; ++i) g[i] = g_lb * static_cast<float>(C) * g[i] * invB;
      }
      if (S > 0) {
#pragma unroll
        for (int i = 0; i < kN; ++i) g[i] += first + off(i) >= S && off(i) < left ? dense : 0.f;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kN; ++i) g[i] = off(i) < left ? dense_grad(first + off(i), pr[i]) : 0.f;
    }
    if constexpr (TERMS) {
#pragma unroll
      for (int i = 0; i < kN; i += 2) *reinterpret_cast<float2*>(dp + first + off(i)) = make_float2(g[i], g[i + 1]);
    } else {
#pragma unroll
      for (int i = 0; i < kN; ++i) dp[first + off(i)] = g[i];
    }
  } else {
    for (int c = threadIdx.x; c < C; c += blockDim.x) dp[c] = dense_grad(c, p[c]);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < k_sel; j += blockDim.x) {
    const int c = static_cast<int>(one_warp ? my_idx : idx[static_cast<long long>(b) * k_sel + j]);
    dp[c] += s_dv[j] * inv_s;    // chapter ids in one row are distinct
  }
  __syncthreads();
  float dot = 0.f;
  if constexpr (NV > 0) {
    if constexpr (TERMS) {
#pragma unroll
      for (int i = 0; i < kN; i += 2) {
        const float2 x = *reinterpret_cast<const float2*>(dp + first + off(i));
        g[i] = x.x; g[i + 1] = x.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kN; ++i) g[i] = dp[first + off(i)];
    }
#pragma unroll
    for (int i = 0; i < kN; ++i) dot += g[i] * pr[i];
  } else {
    for (int c = threadIdx.x; c < C; c += blockDim.x) dot += dp[c] * p[c];
  }
  dot = block_sum(dot, red[3]);
  const float zc = g_z * 2.f * lse * invB;
  if constexpr (TERMS) {
    const long long stride = static_cast<long long>(B) * ld;
    __nv_bfloat16* t0 = terms + static_cast<long long>(b) * ld + first;
    __nv_bfloat16 *t1 = t0 + stride, *t2 = t1 + stride;
    auto emit = [&](int o, float x, float y) {            // (o: columns behind the thread's first)
      const __nv_bfloat162 u = __floats2bfloat162_rn(x, y);
      x -= __low2float(u); y -= __high2float(u);
      const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
      x -= __low2float(v); y -= __high2float(v);
      *reinterpret_cast<__nv_bfloat162*>(t0 + o) = u;
      *reinterpret_cast<__nv_bfloat162*>(t1 + o) = v;
      *reinterpret_cast<__nv_bfloat162*>(t2 + o) = __floats2bfloat162_rn(x, y);
    };
    if constexpr (NV > 0) {
#pragma unroll
      for (int i = 0; i < kN; i += 2)
        if (off(i) < ld - first) emit(off(i), pr[i] * (g[i] - dot + zc), pr[i + 1] * (g[i + 1] - dot + zc));
    } else {
      auto grad = [&](int c) { return c < C ? p[c] * (dp[c] - dot + zc) : 0.f; };
      for (int c = first; c < ld; c += 2 * TH) emit(c - first, grad(c), grad(c + 1));
    }
  } else if constexpr (NV > 0) {
    float* dst = d_logits + static_cast<long long>(b) * C + first;
#pragma unroll
    for (int i = 0; i < kN; ++i)
      if (off(i) < left) dst[off(i)] = pr[i] * (g[i] - dot + zc);
  } else {
    for (int c = threadIdx.x; c < C; c += blockDim.x)
      d_logits[static_cast<long long>(b) * C + c] = p[c] * (dp[c] - dot + zc);
  }
}

// d_w[c,:] = sum_b d_logits[b,c] * pooled[b,:]; d_bias[c] = sum_b d_logits[b,c]; one warp per chapter, 8 batch rows of
// `pooled` staged in shared memory per pass.  Bound by latency and the store of d_w; V floats per access (4 where the width
// allows): 16 -> 9 us for 8 rows, 4,097 chapters, d 768.
template <int V>
__global__ void dweight_kernel(const float* __restrict__ d_logits, const float* __restrict__ pooled,
                               float* __restrict__ d_w, float* __restrict__ d_bias, int B, int d, int C) {
  using T = typename std::conditional<V == 4, float4, float>::type;
  extern __shared__ float4 sp4[];   // [8][d]
  T* sp = reinterpret_cast<T*>(sp4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, dv = d / V;
  const int c = blockIdx.x * (blockDim.x >> 5) + warp;
  float bsum = 0.f;
  for (int b0 = 0; b0 < B; b0 += 8) {
    const int nb = min(8, B - b0);
    float dz[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) dz[j] = (j < nb && c < C) ? d_logits[static_cast<long long>(b0 + j) * C + c] : 0.f;
    __syncthreads();
    // rows past the batch are zero-filled: they are multiplied by dz = 0 below, and 0 x stale NaN would be NaN
    const T* src = reinterpret_cast<const T*>(pooled + static_cast<long long>(b0) * d);
#pragma unroll 4
    for (int i = threadIdx.x; i < 8 * dv; i += blockDim.x) sp[i] = (i < nb * dv) ? src[i] : T{};
    __syncthreads();
    if (c >= C) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) bsum += dz[j];
    T* dst = reinterpret_cast<T*>(d_w + static_cast<long long>(c) * d);
    for (int k = lane; k < dv; k += 32) {
      T acc = (b0 == 0) ? T{} : dst[k];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const T v = sp[j * dv + k];
        if constexpr (V == 4) {
          acc.x = fmaf(dz[j], v.x, acc.x); acc.y = fmaf(dz[j], v.y, acc.y);
          acc.z = fmaf(dz[j], v.z, acc.z); acc.w = fmaf(dz[j], v.w, acc.w);
        } else {
          acc = fmaf(dz[j], v, acc);
        }
      }
      dst[k] = acc;
    }
  }
  if (c < C && lane == 0 && d_bias) d_bias[c] = bsum;
}

// partial[chunk][b][k] = sum over the chunk's chapters of d_logits[b,c] * w[c,k].  Bound by the latency of the weight rows,
// all of which a thread requests at once, V floats each: 17 -> 8 us for 8 rows, 4,097 chapters, d 768.
template <int V>
__global__ void __launch_bounds__(256)
dpooled_partial_kernel(const float* __restrict__ d_logits, const float* __restrict__ w, float* __restrict__ partial, int B,
                       int d, int C) {
  using T = typename std::conditional<V == 4, float4, float>::type;
  __shared__ float dz[kDpChunk][8];
  const int c0 = blockIdx.x * kDpChunk, dv = d / V;
  const int nc = min(kDpChunk, C - c0);
  for (int b0 = 0; b0 < B; b0 += 8) {
    const int nb = min(8, B - b0);
    __syncthreads();
    for (int i = threadIdx.x; i < 8 * kDpChunk; i += blockDim.x) {
      const int j = i / kDpChunk, cc = i - j * kDpChunk;
      dz[cc][j] = (cc < nc && j < nb) ? d_logits[static_cast<long long>(b0 + j) * C + c0 + cc] : 0.f;
    }
    for (int k = threadIdx.x; k < (dv + static_cast<int>(blockDim.x) - 1) / static_cast<int>(blockDim.x) * static_cast<int>(blockDim.x); k += blockDim.x) {
      T wv[kDpChunk];
#pragma unroll
      for (int cc = 0; cc < kDpChunk; ++cc)            // all loads first: they are independent
        wv[cc] = (cc < nc && k < dv) ? reinterpret_cast<const T*>(w + static_cast<long long>(c0 + cc) * d)[k] : T{};
      if (k < static_cast<int>(blockDim.x)) __syncthreads();      // first round: dz is there
      if (k >= dv) continue;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j >= nb) break;
        T acc = T{};
#pragma unroll
        for (int cc = 0; cc < kDpChunk; ++cc) {
          const float z = dz[cc][j];
          if constexpr (V == 4) {
            acc.x = fmaf(z, wv[cc].x, acc.x); acc.y = fmaf(z, wv[cc].y, acc.y);
            acc.z = fmaf(z, wv[cc].z, acc.z); acc.w = fmaf(z, wv[cc].w, acc.w);
          } else {
            acc = fmaf(z, wv[cc], acc);
          }
        }
        reinterpret_cast<T*>(partial + (static_cast<long long>(blockIdx.x) * B + b0 + j) * d)[k] = acc;
      }
    }
  }
}
__global__ void __launch_bounds__(256)
dpooled_finish_kernel(const float* __restrict__ partial, float* __restrict__ d_pooled, int nchunks, int total) {
  // eight warps share 32 outputs: each sums every eighth partial, then a fixed-order reduction
  __shared__ float red[8][32];
  const int sub = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (i < total) {
#pragma unroll 8
    for (int ch = sub; ch < nchunks; ch += 8) acc += partial[static_cast<long long>(ch) * total + i];
  }
  red[sub][lane] = acc;
  __syncthreads();
  if (sub == 0 && i < total)
    d_pooled[i] = ((red[0][lane] + red[1][lane]) + (red[2][lane] + red[3][lane])) +
                  ((red[4][lane] + red[5][lane]) + (red[6][lane] + red[7][lane]));
}
// d_h[b, t, :] (+)= d_pooled[b, :] / L; one thread per 8 consecutive columns of one row (d % 8 == 0),
// falling back to one element per thread otherwise
template <typename T>
__global__ void dh_broadcast_kernel(const float* __restrict__ d_pooled, T* __restrict__ d_h, int L, int d,
                                    long long rows, int accumulate) {
  const float invL = 1.f / static_cast<float>(L);
  if ((d & 7) == 0) {
    const int per_row = d >> 3;
    const long long total = rows * per_row;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
      const long long row = i / per_row;
      const int c = static_cast<int>(i - row * per_row) << 3;
      const int b = static_cast<int>(row / L);
      const float4 p0 = *reinterpret_cast<const float4*>(d_pooled + static_cast<long long>(b) * d + c);
      const float4 p1 = *reinterpret_cast<const float4*>(d_pooled + static_cast<long long>(b) * d + c + 4);
      float v[8] = {p0.x * invL, p0.y * invL, p0.z * invL, p0.w * invL, p1.x * invL, p1.y * invL, p1.z * invL, p1.w * invL};
      T* dst = d_h + row * d + c;
      if (accumulate) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += to_f32(dst[j]);
      }
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
      } else {
        uint4 o;
        o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
        o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
        *reinterpret_cast<uint4*>(dst) = o;
      }
    }
  } else {
    const long long total = rows * d;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
      const long long row = i / d;
      const int c = static_cast<int>(i - row * d);
      const int b = static_cast<int>(row / L);
      float v = d_pooled[static_cast<long long>(b) * d + c] * invL;
      if (accumulate) v += to_f32(d_h[i]);
      if constexpr (sizeof(T) == 4) d_h[i] = v; else d_h[i] = __float2bfloat16(v);
    }
  }
}

// kManyRows rows are enough to fill the chip with CTAs of 1,024 threads twice over; from there on smaller ones win
constexpr int kManyRows = 2 * 296;
constexpr int kRowSmemMost = 200 * 1024;          // what check_shape lets a row of chapters and its lists take
int launch_select(const float* logits, long long ld, const float* bias, float* probs, int64_t* idx, float* weights,
                  int* comb_idx, float* comb_w, float* row_stats, int B, int C, int k_sel, int S, float rho,
                  cudaStream_t stream) {
  const size_t sm = (static_cast<size_t>(C) + 2 * static_cast<size_t>(k_sel > 0 ? k_sel : 1)) * 4;
  // The row's values stay in registers: up to 9 a thread of 1,024 (64 registers leave room for no more), 33 of 256.  The
  // steps are a power of two of routed chapters and a few shared ones; rows beyond 8,192 and some go through shared memory.
  // 8,192 rows of 8,193 chapters: 435 us with 1,024 threads, 305 with 256 (1,024 rows: 62 and 50).
  const bool small = B >= kManyRows && C <= 33 * 256;
  auto kern = small ? (C <= 5 * 256 ? select_kernel<5, 256> : C <= 17 * 256 ? select_kernel<17, 256> : select_kernel<33, 256>)
              : C <= 2 * 1024 ? select_kernel<2, 1024> : C <= 5 * 1024 ? select_kernel<5, 1024>
              : C <= 9 * 1024 ? select_kernel<9, 1024> : select_kernel<0, 1024>;
  MOC_CUDA_OK(allow_shared(kern, sm, kRowSmemMost));
  kern<<<B, small ? 256 : 1024, sm, stream>>>(logits, ld, bias, probs, reinterpret_cast<long long*>(idx), weights, comb_idx,
                                              comb_w, row_stats, C, k_sel, S, rho);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

int launch_dlogits(const float* probs, const int64_t* idx, const float* weights, const float* comb_w, const float* row_stats,
                   const float* chapter_stats, const float* d_weights, const float* d_comb_w, const float* d_losses,
                   float* d_logits, __nv_bfloat16* terms, int ld, int B, int C, int k_sel, int S, float rho,
                   cudaStream_t stream) {
  const int cols = terms != nullptr ? ld : C;
  // In registers up to 18 values a thread of 256, 6 of 1,024.  More is no gain: with 34 of 256 the two CTAs an SM take as long
  // as the general kernel (8,192 rows of 8,193 chapters: 493 and 494 us; 1,024 rows: 61 and 49), with 9 of 1,024 too (8 rows:
  // 23 us either way).
  const bool small = B >= kManyRows && cols <= 18 * 256;
  const bool held = small || cols <= 6 * 1024;
  const size_t sm = (small ? 18 * 256 : held ? 6 * 1024 : static_cast<size_t>(C)) * 4;
  auto kern = terms != nullptr
                  ? (small ? dlogits_kernel<18, 256, true> : held ? dlogits_kernel<6, 1024, true> : dlogits_kernel<0, 1024, true>)
                  : (small ? dlogits_kernel<18, 256, false> : held ? dlogits_kernel<6, 1024, false> : dlogits_kernel<0, 1024, false>);
  MOC_CUDA_OK(allow_shared(kern, sm, kRowSmemMost));
  kern<<<B, small ? 256 : 1024, sm, stream>>>(probs, reinterpret_cast<const long long*>(idx), weights, comb_w, row_stats,
                                              chapter_stats, d_weights, d_comb_w, d_losses, d_logits, terms, ld, B, C, k_sel, S,
                                              rho);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

// Whether the one launch takes calls of this shape (see route_front_kernel), and that launch.  `done` says whether it was made: a
// device that cannot hold a cluster of 16 CTAs of 1,024 threads (a part of a GPU, say) leaves the call to the other kernels.
bool front_takes(const moc_router_shape* s, const void* h, const float* w, const float* pooled) {
  const int piece = s->h_dtype == MOC_F32 ? 4 : 8;
  return s->batch <= kFrontRows && s->seq <= kPoolSplits * kPoolOneMaxRows && s->hidden_dim % piece == 0 && s->hidden_dim % 4 == 0 &&
         s->hidden_dim <= 1024 && s->num_chapters <= kFrontChapters &&
         ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(pooled)) & 15) == 0;
}
template <typename T>
int launch_front(const T* h, const float* w, const float* bias, const FrontParams& p, cudaStream_t stream, bool* done) {
  const int nd = p.d <= 256 ? 0 : p.d <= 768 ? 1 : 2, nv = p.C <= 2 * 1024 ? 0 : p.C <= 5 * 1024 ? 1 : 2;
  using Kern = void (*)(const T*, const float*, const float*, FrontParams);
  static constexpr Kern kerns[3][3] = {
      {route_front_kernel<T, 2, 2>, route_front_kernel<T, 5, 2>, route_front_kernel<T, 9, 2>},
      {route_front_kernel<T, 2, 6>, route_front_kernel<T, 5, 6>, route_front_kernel<T, 9, 6>},
      {route_front_kernel<T, 2, 8>, route_front_kernel<T, 5, 8>, route_front_kernel<T, 9, 8>}};
  const Kern kern = kerns[nd][nv];
  const size_t part = static_cast<size_t>(kPoolSplits) * (32 * (16 / sizeof(T)) + 4) * 4;
  const size_t sel = (static_cast<size_t>(p.C) + 2 * static_cast<size_t>(p.k_sel > 0 ? p.k_sel : 1)) * 4;
  const size_t bytes = std::max(std::max(part, sel), static_cast<size_t>(p.B) * p.d * 4);
  MOC_CUDA_OK(allow_shared(kern, bytes, kFrontSmemMost));
  MOC_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  *done = resident_clusters(kern, 1024, static_cast<int>(bytes), kFrontCtas) > 0;
  if (!*done) return MOC_OK;
  const int more = ceil_div(ceil_div(p.q.n, 32), kFrontCtas);        // clusters for the projection; they wait for nobody
  MOC_CUDA_OK(launch_clustered(kern, dim3(kFrontCtas * (1 + more)), 1024, static_cast<int>(bytes), kFrontCtas, stream, h, w, bias, p));
  return MOC_OK;
}

inline int k_selected(const moc_router_shape* s) {
  int k = s->top_k;
  const int avail = s->num_chapters - s->num_shared;
  if (k > avail) k = avail;
  return k < 0 ? 0 : k;
}
// Scratch layout: [ pooling partials | d_pooled partials ] (they never live at once), then the loss partials.
// A call that neither pools (token rows, or pooled states handed in) nor produces d_pooled needs the loss part only.
inline size_t ws_floats(const moc_router_shape* s, bool pool, bool dpooled) {
  const size_t p = pool ? static_cast<size_t>(s->batch) * kPoolSplits * s->hidden_dim : 0;
  const size_t dp = dpooled ? static_cast<size_t>(ceil_div(s->num_chapters, kDpChunk)) * s->batch * s->hidden_dim : 0;
  return p > dp ? p : dp;
}
// row ranges of the loss statistics: one for the handful of rows of sequence-level routing, ~128 rows each otherwise
inline int loss_row_splits(const moc_router_shape* s) {
  return s->batch <= 256 ? 1 : (ceil_div(s->batch, 128) < 64 ? ceil_div(s->batch, 128) : 64);
}
inline size_t loss_floats(const moc_router_shape* s) {
  const int splits = loss_row_splits(s);
  // (the per-range records are float4: four floats of slack let the block start on a 16-byte boundary)
  const size_t rows_part = splits > 1 ? static_cast<size_t>(splits) * s->num_chapters * 4 + 4 : 0;
  return static_cast<size_t>(ceil_div(s->num_chapters, kLossChunk)) * 3 + rows_part;
}
inline size_t ws_bytes(const moc_router_shape* s) { return (ws_floats(s, true, true) + loss_floats(s)) * sizeof(float); }
inline int check_shape(const moc_router_shape* s) {
  MOC_REQUIRE(s != nullptr, "shape is NULL");
  MOC_REQUIRE(s->batch > 0 && s->seq > 0 && s->hidden_dim > 0, "empty router input");
  MOC_REQUIRE(s->num_chapters > 0, "num_chapters must be > 0");
  MOC_REQUIRE(s->top_k > 0 && s->top_k <= s->num_chapters, "top_k must be in [1, num_chapters]");
  MOC_REQUIRE(s->num_shared >= 0 && s->num_shared <= s->num_chapters, "exclude_prefix_chapters out of range");
  MOC_REQUIRE(s->top_k <= 1024, "top_k above 1024 is not supported");
  MOC_REQUIRE(s->h_dtype == MOC_F32 || s->h_dtype == MOC_BF16, "bad h_dtype");
  MOC_REQUIRE((static_cast<size_t>(s->num_chapters) + 2 * 1024) * 4 <= kRowSmemMost, "num_chapters too large");
  return MOC_OK;
}

void launch_losses(const moc_router_shape* s, const float* probs, const int64_t* idx, const float* row_stats,
                   float* chapter_stats, float* losses, float* loss_partial, cudaStream_t stream) {
  const int B = s->batch, C = s->num_chapters, k_sel = k_selected(s);
  const int nblk = ceil_div(C, kLossChunk);
  const int splits = loss_row_splits(s);
  if (splits > 1) {
    float* rows_part = reinterpret_cast<float*>(
        (reinterpret_cast<uintptr_t>(loss_partial + static_cast<size_t>(nblk) * 3) + 15) & ~uintptr_t(15));
    const int rows_per_split = ceil_div(B, splits);
    loss_rows_partial_kernel<<<dim3(nblk, splits), kLossChunk, 0, stream>>>(
        probs, reinterpret_cast<const long long*>(idx), rows_part, B, C, k_sel, rows_per_split);
    loss_rows_finish_kernel<<<nblk, kLossChunk, 0, stream>>>(rows_part, chapter_stats, loss_partial, B, C, splits);
  } else {
    loss_partial_kernel<<<nblk, kLossChunk, 0, stream>>>(probs, reinterpret_cast<const long long*>(idx),
                                                         chapter_stats, loss_partial, B, C, k_sel);
  }
  loss_finish_kernel<<<1, splits > 1 ? 1024 : 32, 0, stream>>>(loss_partial, row_stats, losses, nblk, B, C);
}

struct TokenSaved { __nv_bfloat16* w_terms; float *probs, *row_stats, *chapter_stats, *loss_ws; };
moc_router_shape token_shape(const moc_token_route_desc* s) {
  return moc_router_shape{s->rows, 1, s->hidden_dim, s->num_chapters, s->top_k, s->num_shared, 1.f, MOC_BF16};
}
int64_t carve(const moc_token_route_desc* s, TokenSaved* a) {
  const moc_router_shape r = token_shape(s);
  Carver c{static_cast<char*>(s->arena), 0};
  const int64_t C = s->num_chapters;
  a->w_terms = c.take<__nv_bfloat16>(3 * C * s->hidden_dim + 8 * s->hidden_dim);   // (a padded K reads a few rows further)
  a->probs = c.take<float>(s->rows * C);
  a->row_stats = c.take<float>(4 * static_cast<int64_t>(s->rows));
  a->chapter_stats = c.take<float>(2 * C);
  a->loss_ws = c.take<float>(static_cast<int64_t>(loss_floats(&r)));
  return c.off;
}
inline int64_t padded(int n) { return (n + 7) / 8 * 8; }

}  // namespace
}  // namespace moc

using namespace moc;

extern "C" int64_t moc_token_route_arena_bytes(const moc_token_route_desc* s) {
  TokenSaved a;
  return s ? carve(s, &a) : -1;
}
extern "C" int64_t moc_token_route_scratch_bytes(const moc_token_route_desc* s, int32_t backward) {
  if (!s) return -1;
  const int64_t cp = padded(s->num_chapters);
  return backward ? 3 * s->rows * cp * 2 + ceil_div(s->rows, kTermRows) * cp * 4 : s->rows * cp * 4;
}

extern "C" int moc_token_route_fwd(const moc_token_route_desc* s, void* scratch) {
  MOC_REQUIRE(s && s->h && s->w && s->weights && s->arena && scratch && s->status, "NULL token-router buffer");
  const moc_router_shape r = token_shape(s);
  int rc = check_shape(&r);
  if (rc != MOC_OK) return rc;
  MOC_REQUIRE(r.hidden_dim % 8 == 0, "the bf16 token router takes a width of a multiple of 8");
  TokenSaved a;
  carve(s, &a);
  cudaStream_t stream = static_cast<cudaStream_t>(s->stream);
  const int C = s->num_chapters, d = s->hidden_dim;
  const int64_t cp = padded(C);
  // bf16 activations are exact bf16 numbers: h (w0 + w1 + w2)^T as one product over three times the width, smallest term
  // first, carries the fp32 weight's 24 mantissa bits; nothing is added up outside the accumulator
  MOC_TRY(moc_split_bf16(s->w, a.w_terms, static_cast<int64_t>(C) * d, 3, stream));
  float* logits = static_cast<float*>(scratch);
  Gemm g(MOC_BF16, s->rows, C, d, true, true, MOC_F32);
  g.ldc = cp;
  g.extra.terms = 3; g.extra.b_term_rows = C;
  MOC_TRY(gemm_extra(g, s->h, a.w_terms, logits, s->status, stream));
  MOC_TRY(launch_select(logits, cp, s->bias, a.probs, s->idx, s->weights, nullptr, nullptr, a.row_stats, s->rows, C,
                        k_selected(&r), s->num_shared, 1.f, stream));
  if (s->losses != nullptr)
    launch_losses(&r, a.probs, s->idx, a.row_stats, a.chapter_stats, s->losses, a.loss_ws, stream);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" int moc_token_route_bwd(const moc_token_route_desc* s, const float* g_weights, const float* g_losses, void* d_h,
                                   float* d_w, float* d_bias, void* scratch) {
  MOC_REQUIRE(s && s->h && s->weights && s->arena && scratch && s->status, "NULL token-router buffer");
  const moc_router_shape r = token_shape(s);
  int rc = check_shape(&r);
  if (rc != MOC_OK) return rc;
  MOC_REQUIRE(d_w == nullptr || s->rows % 8 == 0, "a bf16 weight gradient takes the tokens in multiples of 8");
  TokenSaved a;
  carve(s, &a);
  cudaStream_t stream = static_cast<cudaStream_t>(s->stream);
  const int C = s->num_chapters, d = s->hidden_dim, rows = s->rows, k_sel = k_selected(&r);
  const int64_t cp = padded(C);
  __nv_bfloat16* terms = static_cast<__nv_bfloat16*>(scratch);
  float* partial = reinterpret_cast<float*>(terms + 3 * rows * cp);
  MOC_TRY(launch_dlogits(a.probs, s->idx, s->weights, nullptr, a.row_stats, a.chapter_stats, g_weights, nullptr, g_losses,
                         nullptr, terms, static_cast<int>(cp), rows, C, k_sel, s->num_shared, 1.f, stream));
  if (d_h != nullptr) {        // leaves in bf16: one product of the leading terms
    Gemm g(MOC_BF16, rows, d, cp, true, false, MOC_BF16);
    MOC_TRY(moc_gemm(&g, terms, a.w_terms, d_h, nullptr, nullptr, s->status, stream));
  }
  if (d_w != nullptr) {
    Gemm g(MOC_BF16, C, d, rows, false, false, MOC_F32);
    g.lda = cp;
    g.extra.terms = 3; g.extra.a_term_rows = rows;
    MOC_TRY(gemm_extra(g, terms, s->h, d_w, s->status, stream));
  }
  if (d_bias != nullptr) {
    const int chunks = ceil_div(rows, kTermRows);
    term_col_sum_kernel<<<dim3(ceil_div(static_cast<int>(cp), 64), chunks), 256, 0, stream>>>(terms, partial, rows,
                                                                                            static_cast<int>(cp));
    col_sum_kernel<<<ceil_div(C, 32), 256, 0, stream>>>(partial, d_bias, chunks, C, static_cast<int>(cp));
  }
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" size_t moc_router_workspace_bytes(const moc_router_shape* s) { return s ? ws_bytes(s) : 0; }
extern "C" size_t moc_router_workspace_bytes_parts(const moc_router_shape* s, int32_t fwd_parts, int32_t bwd_parts) {
  if (!s) return 0;
  const bool pool = (fwd_parts & 1) && !(fwd_parts & 8);
  return (ws_floats(s, pool, (bwd_parts & 4) != 0) + loss_floats(s)) * sizeof(float);
}

namespace moc {
int router_fwd_parts_impl(const moc_router_shape* s, const void* h, const float* w, const float* bias, float* pooled, float* logits,
                          float* probs, int64_t* idx, float* weights, int32_t* comb_idx, float* comb_w, float* row_stats,
                          float* chapter_stats, float* losses, void* workspace, size_t workspace_bytes, int32_t parts,
                          const RowsProduct* q, RouteRun* run, int32_t* status, void* stream_) {
  int rc = check_shape(s);
  if (rc != MOC_OK) return rc;
  const size_t front = ws_floats(s, (parts & 1) && !(parts & 8), false);
  MOC_REQUIRE(workspace_bytes >= (front + loss_floats(s)) * sizeof(float), "router workspace too small");
  MOC_REQUIRE((h || (parts & 8)) && w && pooled && logits && probs && comb_idx && comb_w && row_stats,
              "NULL router buffer");
  (void)status;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int B = s->batch, L = s->seq, d = s->hidden_dim, C = s->num_chapters, S = s->num_shared;
  const int k_sel = k_selected(s);
  MOC_REQUIRE(k_sel == 0 || (idx && weights), "NULL index / weight buffer");
  float* ws = static_cast<float*>(workspace);
  // the loss partials sit behind the front part of whatever layout the caller sized the workspace for
  float* loss_partial = ws + (workspace_bytes / sizeof(float) - loss_floats(s));

  dim3 pg(B, kPoolSplits);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  bool one_launch = false;
  if (q != nullptr && (parts & 1) && !(parts & (8 | 16)) && front_takes(s, h, w, pooled) &&
      cudaStreamIsCapturing(stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone) {
    FrontParams p{pooled, logits, probs, reinterpret_cast<long long*>(idx), weights, comb_idx, comb_w, row_stats, B, L, d, C, k_sel,
                  S, s->routed_scale, *q};
    MOC_TRY(s->h_dtype == MOC_F32 ? launch_front(static_cast<const float*>(h), w, bias, p, stream, &one_launch)
                                  : launch_front(static_cast<const __nv_bfloat16*>(h), w, bias, p, stream, &one_launch));
  }
  RouteRun did;
  did.q_done = one_launch;
  did.launches = one_launch ? 1 : 0;
  if ((parts & 1) && !one_launch) {
  did.launches = 1 + ((parts & 16) ? 0 : 1);
  if (!(parts & 8)) {      // bit 8: `pooled` already holds the pooled states (another pooling rule ran first)
  const int piece = s->h_dtype == MOC_F32 ? 4 : 8;
  const bool one = L <= kPoolSplits * kPoolOneMaxRows && d % piece == 0 && (reinterpret_cast<uintptr_t>(h) & 15) == 0;
  did.launches += one ? 1 : 2;
  const dim3 og(B, ceil_div(d, 8 * piece));
  if (one && s->h_dtype == MOC_F32)
    pool_mean_kernel<float><<<og, 8 * kPoolSplits, 0, stream>>>(static_cast<const float*>(h), pooled, L, d);
  else if (one)
    pool_mean_kernel<__nv_bfloat16><<<og, 8 * kPoolSplits, 0, stream>>>(static_cast<const __nv_bfloat16*>(h), pooled, L, d);
  else if (s->h_dtype == MOC_F32)
    pool_partial_kernel<float><<<pg, 256, 0, stream>>>(static_cast<const float*>(h), ws, L, d);
  else
    pool_partial_kernel<__nv_bfloat16><<<pg, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(h), ws, L, d);
  if (!one) pool_finish_kernel<<<ceil_div(B * d, 256), 256, 0, stream>>>(ws, pooled, L, d, B * d);
  }
  // bit 16: `logits` already holds pooled x W^T (a projection kernel ran); only the bias is missing
  const float* bias_left = (parts & 16) ? bias : nullptr;
  if (!(parts & 16)) {
    const size_t sm = static_cast<size_t>(8) * d * sizeof(float);
    if (d % 4 == 0 && d <= 1024 && ((reinterpret_cast<uintptr_t>(pooled) | reinterpret_cast<uintptr_t>(w)) & 15) == 0) {
      const bool few = B <= 8;
      auto kern = d <= 256 ? (few ? logits_rows_kernel<2, 1> : logits_rows_kernel<2, 4>)
                  : d <= 768 ? (few ? logits_rows_kernel<6, 1> : logits_rows_kernel<6, 4>)
                             : (few ? logits_rows_kernel<8, 1> : logits_rows_kernel<8, 4>);
      const size_t bytes = few ? sm : 2 * sm;
      MOC_CUDA_OK(allow_shared(kern, bytes, 2 * 8 * 1024 * 4));
      kern<<<ceil_div(C, few ? 8 : 32), 256, bytes, stream>>>(pooled, w, bias, logits, B, d, C);
    } else {
      MOC_CUDA_OK(allow_shared(logits_kernel, sm, kSharedMost));
      logits_kernel<<<ceil_div(C, 8), 256, sm, stream>>>(pooled, w, bias, logits, B, d, C);
    }
  }
  if ((rc = launch_select(logits, C, bias_left, probs, idx, weights, comb_idx, comb_w, row_stats, B, C, k_sel, S,
                          s->routed_scale, stream)) != MOC_OK) return rc;
  }
  if ((parts & 2) && losses != nullptr) {
    MOC_REQUIRE(chapter_stats != nullptr, "chapter_stats is NULL");
    launch_losses(s, probs, idx, row_stats, chapter_stats, losses, loss_partial, stream);
  }
  MOC_CUDA_OK(cudaGetLastError());
  if (run != nullptr) *run = did;
  return MOC_OK;
}

}  // namespace moc

extern "C" int moc_router_fwd_parts(const moc_router_shape* s, const void* h, const float* w, const float* bias,
                                    float* pooled, float* logits, float* probs, int64_t* idx, float* weights,
                                    int32_t* comb_idx, float* comb_w, float* row_stats, float* chapter_stats,
                                    float* losses, void* workspace, size_t workspace_bytes, int32_t parts,
                                    int32_t* status, void* stream) {
  return router_fwd_parts_impl(s, h, w, bias, pooled, logits, probs, idx, weights, comb_idx, comb_w, row_stats, chapter_stats,
                               losses, workspace, workspace_bytes, parts, nullptr, nullptr, status, stream);
}

extern "C" int moc_router_fwd(const moc_router_shape* s, const void* h, const float* w, const float* bias,
                              float* pooled, float* logits, float* probs, int64_t* idx, float* weights,
                              int32_t* comb_idx, float* comb_w, float* row_stats, float* chapter_stats,
                              float* losses, void* workspace, size_t workspace_bytes, int32_t* status,
                              void* stream_) {
  return moc_router_fwd_parts(s, h, w, bias, pooled, logits, probs, idx, weights, comb_idx, comb_w, row_stats,
                              chapter_stats, losses, workspace, workspace_bytes, 3, status, stream_);
}

extern "C" int moc_router_bwd_parts(const moc_router_shape* s, const float* w, const float* pooled,
                                    const float* probs, const int64_t* idx, const float* weights,
                                    const float* comb_w, const float* row_stats, const float* chapter_stats,
                                    const float* d_weights, const float* d_comb_w, const float* d_losses,
                                    float* d_logits, float* d_w, float* d_bias, float* d_pooled, void* d_h,
                                    int32_t accumulate_dh, void* workspace, size_t workspace_bytes, int32_t parts,
                                    int32_t* status, void* stream_) {
  int rc = check_shape(s);
  if (rc != MOC_OK) return rc;
  MOC_REQUIRE(workspace_bytes >= ws_floats(s, false, (parts & 4) != 0) * sizeof(float), "router workspace too small");
  MOC_REQUIRE(w && pooled && probs && comb_w && row_stats && d_logits && d_w && d_pooled, "NULL router buffer");
  MOC_REQUIRE(d_losses == nullptr || chapter_stats != nullptr, "loss gradients need chapter_stats");
  (void)status;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int B = s->batch, L = s->seq, d = s->hidden_dim, C = s->num_chapters, S = s->num_shared;
  const int k_sel = k_selected(s);
  float* ws = static_cast<float*>(workspace);
  if (parts & 1) {
    if ((rc = launch_dlogits(probs, idx, weights, comb_w, row_stats, chapter_stats, d_weights, d_comb_w, d_losses, d_logits,
                             nullptr, 0, B, C, k_sel, S, s->routed_scale, stream)) != MOC_OK) return rc;
  }
  if (parts & 2) {
    const size_t sm = static_cast<size_t>(8) * d * sizeof(float);
    const bool vec = d % 4 == 0 && ((reinterpret_cast<uintptr_t>(pooled) | reinterpret_cast<uintptr_t>(d_w)) & 15) == 0;
    auto kern = vec ? dweight_kernel<4> : dweight_kernel<1>;
    MOC_CUDA_OK(allow_shared(kern, sm, kSharedMost));
    kern<<<ceil_div(C, 8), 256, sm, stream>>>(d_logits, pooled, d_w, d_bias, B, d, C);
  }
  const int nchunks = ceil_div(C, kDpChunk);
  if (parts & 4) {
    const bool vec = d % 4 == 0 && ((reinterpret_cast<uintptr_t>(ws) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
    (vec ? dpooled_partial_kernel<4> : dpooled_partial_kernel<1>)<<<nchunks, 256, 0, stream>>>(d_logits, w, ws, B, d, C);
    dpooled_finish_kernel<<<ceil_div(B * d, 32), 256, 0, stream>>>(ws, d_pooled, nchunks, B * d);
  }
  if ((parts & 4) && d_h != nullptr) {
    const long long rows = static_cast<long long>(B) * L;
    const long long work = (d & 7) == 0 ? rows * (d >> 3) : rows * d;
    long long blocks = (work + 255) / 256;
    if (blocks > 148LL * 32) blocks = 148LL * 32;
    if (s->h_dtype == MOC_F32)
      dh_broadcast_kernel<float><<<static_cast<int>(blocks), 256, 0, stream>>>(d_pooled, static_cast<float*>(d_h), L, d, rows, accumulate_dh);
    else
      dh_broadcast_kernel<__nv_bfloat16><<<static_cast<int>(blocks), 256, 0, stream>>>(d_pooled, static_cast<__nv_bfloat16*>(d_h), L, d, rows, accumulate_dh);
  }
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" int moc_router_bwd(const moc_router_shape* s, const float* w, const float* pooled,
                              const float* probs, const int64_t* idx, const float* weights,
                              const float* comb_w, const float* row_stats, const float* chapter_stats,
                              const float* d_weights, const float* d_comb_w, const float* d_losses,
                              float* d_logits, float* d_w, float* d_bias, float* d_pooled, void* d_h,
                              int32_t accumulate_dh, void* workspace, size_t workspace_bytes,
                              int32_t* status, void* stream_) {
  return moc_router_bwd_parts(s, w, pooled, probs, idx, weights, comb_w, row_stats, chapter_stats, d_weights,
                              d_comb_w, d_losses, d_logits, d_w, d_bias, d_pooled, d_h, accumulate_dh, workspace,
                              workspace_bytes, 7, status, stream_);
}


extern "C" int moc_pool_weighted_fwd(const void* h, int32_t h_dtype, const float* pos_weight, float* pooled,
                                     int32_t batch, int32_t seq, int32_t dim, void* workspace,
                                     size_t workspace_bytes, void* stream_) {
  MOC_REQUIRE(h && pos_weight && pooled && workspace, "NULL buffer");
  MOC_REQUIRE(batch > 0 && seq > 0 && dim > 0, "empty input");
  MOC_REQUIRE(h_dtype == MOC_F32 || h_dtype == MOC_BF16, "bad h_dtype");
  MOC_REQUIRE(workspace_bytes >= static_cast<size_t>(batch) * kPoolSplits * dim * sizeof(float),
              "pooling workspace too small");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  float* ws = static_cast<float*>(workspace);
  dim3 pg(batch, kPoolSplits);
  if (h_dtype == MOC_F32)
    pool_weighted_partial_kernel<float><<<pg, 256, 0, stream>>>(static_cast<const float*>(h), pos_weight, ws, seq, dim);
  else
    pool_weighted_partial_kernel<__nv_bfloat16><<<pg, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(h),
                                                                        pos_weight, ws, seq, dim);
  pool_weighted_finish_kernel<<<ceil_div(batch * dim, 256), 256, 0, stream>>>(ws, pooled, dim, batch * dim);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" int moc_pool_weighted_bwd(const float* d_pooled, const float* pos_weight, void* d_h, int32_t h_dtype,
                                     int32_t batch, int32_t seq, int32_t dim, int32_t accumulate, void* stream_) {
  MOC_REQUIRE(d_pooled && pos_weight && d_h, "NULL buffer");
  MOC_REQUIRE(batch > 0 && seq > 0 && dim > 0, "empty input");
  MOC_REQUIRE(h_dtype == MOC_F32 || h_dtype == MOC_BF16, "bad h_dtype");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const long long total = static_cast<long long>(batch) * seq * dim;
  long long blocks = (total + 255) / 256;
  if (blocks > 148LL * 32) blocks = 148LL * 32;
  if (h_dtype == MOC_F32)
    pool_weighted_bwd_kernel<float><<<static_cast<int>(blocks), 256, 0, stream>>>(
        d_pooled, pos_weight, static_cast<float*>(d_h), seq, dim, total, accumulate);
  else
    pool_weighted_bwd_kernel<__nv_bfloat16><<<static_cast<int>(blocks), 256, 0, stream>>>(
        d_pooled, pos_weight, static_cast<__nv_bfloat16*>(d_h), seq, dim, total, accumulate);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}


extern "C" int moc_sum_terms(const float* src, const float* bias, float* dst, int64_t rows, int32_t cols, int32_t ld,
                             int32_t terms, void* stream_) {
  MOC_REQUIRE(src && dst && rows >= 0 && cols > 0 && ld >= cols && terms >= 1, "bad sum_terms arguments");
  if (rows == 0) return MOC_OK;
  long long blocks = (rows * cols + 255) / 256;
  if (blocks > 148LL * 32) blocks = 148LL * 32;
  sum_terms_kernel<<<static_cast<int>(blocks), 256, 0, static_cast<cudaStream_t>(stream_)>>>(src, bias, dst, rows, cols,
                                                                                             ld, terms);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" int moc_loss_total(const float* losses, const float* grad, float c0, float c1, float c2, float c3, float* out,
                              void* stream_) {
  MOC_REQUIRE(losses && out, "NULL buffer");
  loss_total_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream_)>>>(losses, grad, make_float4(c0, c1, c2, c3), out);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" int moc_col_sum(const float* x, float* out, int64_t rows, int32_t cols, void* stream_) {
  MOC_REQUIRE(x && out && rows > 0 && cols > 0, "bad column-sum arguments");
  col_sum_kernel<<<ceil_div(cols, 32), 256, 0, static_cast<cudaStream_t>(stream_)>>>(x, out, rows, cols, cols);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

extern "C" int moc_quotient_probe(const float* x, const float* d, float* y, int32_t n, void* stream) {
  MOC_REQUIRE(x && d && y && n > 0, "bad quotient probe");
  quotient_probe_kernel<<<ceil_div(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, d, y, n);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}
