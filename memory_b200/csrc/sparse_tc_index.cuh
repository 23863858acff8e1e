// Inverted index of the per-token chapter lists: key unit -> the (token, slot) pairs that selected it, cut into row
// tiles.  Included by sparse_tc.cu only.
//
// A listed block of `block_size` rows is U = block_size / KU units of KU keys (KU = 64 or 128, what one score tile
// holds).  Pairs are numbered p = (((b * TQ + t) * H + h) * S + s) * U + u, buckets (b * H + h) * M + unit.  A row of
// a tile is a (pair, query head of the group): the G = HQ / H query heads of a KV head share its keys, so a bucket of
// n pairs has n * G rows and a 128-row tile holds 128 / G pairs.
#pragma once
#include "moc_common.cuh"

namespace moc {
namespace sparse_tc {

struct Shape {
  int B, TQ, TK, HQ, H, G, S, U, KU, M;      // S: listed blocks per (token, KV head); M: units per (b, KV head)
  int ppt;                                    // pairs per tile
  int chunk;                                  // tiles per work item of the backward pass
  long long n_pairs, n_buckets;
  float scale, scale_log2;
};

struct Index {
  int *cnt, *cursor;                          // [n_buckets] each
  int *pair_off, *tile_off, *item_off, *part_off;   // [n_buckets + 1] each: exclusive scans
  int *entries;                               // [n_pairs] pairs grouped by bucket, ascending
  int *pos;                                   // [n_pairs] where a pair sits in `entries`, -1: bad chapter id
  int *tile_bucket, *tile_first, *tile_cnt;   // forward work: bucket, first entry, pairs
  int *item_bucket, *item_tile, *item_nt, *item_part;   // backward work: bucket, its tiles, partial slot or -1
  int *totals;                                // tiles, items, partial slots
};

inline long long max_tiles(const Shape& x) {
  return x.n_pairs / x.ppt + (x.n_buckets < x.n_pairs ? x.n_buckets : x.n_pairs);
}
inline long long max_items(const Shape& x) { return x.n_buckets + max_tiles(x) / x.chunk + 1; }
// a bucket is cut into several items only when it has more than `chunk` tiles: at most 2 * tiles / chunk such items
inline long long max_parts(const Shape& x) { return 2 * (max_tiles(x) / x.chunk) + 2; }

inline size_t carve(const Shape& x, int* ws, Index* ib) {
  int* p = ws;
  auto take = [&](long long n) { int* r = p; p += (n + 3) & ~3ll; return r; };
  const long long nb = x.n_buckets;
  ib->cnt = take(nb); ib->cursor = take(nb);
  ib->pair_off = take(nb + 1); ib->tile_off = take(nb + 1); ib->item_off = take(nb + 1); ib->part_off = take(nb + 1);
  ib->entries = take(x.n_pairs); ib->pos = take(x.n_pairs);
  const long long mt = max_tiles(x), mi = max_items(x);
  ib->tile_bucket = take(mt); ib->tile_first = take(mt); ib->tile_cnt = take(mt);
  ib->item_bucket = take(mi); ib->item_tile = take(mi); ib->item_nt = take(mi); ib->item_part = take(mi);
  ib->totals = take(4);
  return static_cast<size_t>(p - ws) * sizeof(int);
}

__global__ void index_count_kernel(const int* __restrict__ idx, Shape x, int* __restrict__ cnt, int* __restrict__ status) {
  const long long q = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;     // listed block
  if (q >= x.n_pairs / x.U) return;
  const long long bth = q / x.S;
  const int h = static_cast<int>(bth % x.H), b = static_cast<int>(bth / x.H / x.TQ);
  const int c = idx[q];
  if (c < 0 || c >= x.M / x.U) { atomicMax(status, MOC_DEV_BAD_INDEX); return; }
  int* dst = cnt + static_cast<long long>(b * x.H + h) * x.M + c * x.U;
  for (int u = 0; u < x.U; ++u) atomicAdd(dst + u, 1);
}

// exclusive scans over the buckets of {pairs, tiles, items, partial slots}; one CTA of 1,024 threads
__global__ void index_scan_kernel(Shape x, Index ib) {
  __shared__ int wt[4][32];
  const int n = static_cast<int>(x.n_buckets);
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int lo = threadIdx.x * per, hi = min(n, lo + per);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto sizes = [&](int i, int (&v)[4]) {
    v[0] = ib.cnt[i];
    v[1] = (v[0] + x.ppt - 1) / x.ppt;
    v[2] = max(1, (v[1] + x.chunk - 1) / x.chunk);    // an empty bucket keeps one item: it zero-fills its rows
    v[3] = v[2] > 1 ? v[2] : 0;
  };
  int s[4] = {0, 0, 0, 0}, v[4];
  for (int i = lo; i < hi; ++i) {
    sizes(i, v);
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] += v[j];
  }
  int inc[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    inc[j] = s[j];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc[j], o);
      if (lane >= o) inc[j] += t;
    }
    if (lane == 31) wt[j][warp] = inc[j];
  }
  __syncthreads();
  if (warp < 4) {
    int w = wt[warp][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    wt[warp][lane] = w;
  }
  __syncthreads();
  int e[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) e[j] = inc[j] - s[j] + (warp > 0 ? wt[j][warp - 1] : 0);
  for (int i = lo; i < hi; ++i) {
    ib.pair_off[i] = e[0]; ib.tile_off[i] = e[1]; ib.item_off[i] = e[2]; ib.part_off[i] = e[3];
    sizes(i, v);
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] += v[j];
  }
  if (threadIdx.x == 0) {
    ib.pair_off[n] = wt[0][31]; ib.tile_off[n] = wt[1][31]; ib.item_off[n] = wt[2][31]; ib.part_off[n] = wt[3][31];
    ib.totals[0] = wt[1][31]; ib.totals[1] = wt[2][31]; ib.totals[2] = wt[3][31];
  }
}

__global__ void index_fill_kernel(const int* __restrict__ idx, Shape x, Index ib) {
  const long long q = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (q >= x.n_pairs / x.U) return;
  const long long bth = q / x.S;
  const int h = static_cast<int>(bth % x.H), b = static_cast<int>(bth / x.H / x.TQ);
  const int c = idx[q];
  const bool bad = c < 0 || c >= x.M / x.U;
  for (int u = 0; u < x.U; ++u) {
    const long long p = q * x.U + u;
    if (bad) { ib.pos[p] = -1; continue; }
    const long long bkt = static_cast<long long>(b * x.H + h) * x.M + c * x.U + u;
    ib.entries[ib.pair_off[bkt] + atomicAdd(&ib.cursor[bkt], 1)] = static_cast<int>(p);
  }
}

// One CTA per bucket: its pairs in ascending order (the fill places them in arrival order; with this the sums of the
// backward pass do not depend on scheduling; buckets above kSortMax pairs stay in arrival order), their positions, and
// the bucket's entries of the two work tables.
constexpr int kSortMax = 2048;
__global__ void index_finish_kernel(Shape x, Index ib) {
  __shared__ int buf[kSortMax];
  const int bkt = blockIdx.x;
  const int first = ib.pair_off[bkt], n = ib.pair_off[bkt + 1] - first;
  if (n > 1 && n <= kSortMax) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) buf[i] = ib.entries[first + i];
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int v = buf[i];
      int rank = 0;
      for (int j = 0; j < n; ++j) rank += (buf[j] < v);
      ib.entries[first + rank] = v;
      ib.pos[v] = first + rank;
    }
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) ib.pos[ib.entries[first + i]] = first + i;
  }
  const int t0 = ib.tile_off[bkt], nt = ib.tile_off[bkt + 1] - t0;
  for (int t = threadIdx.x; t < nt; t += blockDim.x) {
    ib.tile_bucket[t0 + t] = bkt;
    ib.tile_first[t0 + t] = first + t * x.ppt;
    ib.tile_cnt[t0 + t] = min(x.ppt, n - t * x.ppt);
  }
  const int i0 = ib.item_off[bkt], ni = ib.item_off[bkt + 1] - i0;
  for (int i = threadIdx.x; i < ni; i += blockDim.x) {
    ib.item_bucket[i0 + i] = bkt;
    const int lo = static_cast<int>(static_cast<long long>(i) * nt / ni);        // the tiles in equal shares
    ib.item_tile[i0 + i] = lo;
    ib.item_nt[i0 + i] = static_cast<int>(static_cast<long long>(i + 1) * nt / ni) - lo;
    ib.item_part[i0 + i] = ni > 1 ? ib.part_off[bkt] + i : -1;
  }
}

inline int build_index(const int* idx, const Shape& x, const Index& ib, int* status, cudaStream_t stream) {
  MOC_CUDA_OK(cudaMemsetAsync(ib.cnt, 0, static_cast<size_t>(ib.pair_off - ib.cnt) * sizeof(int), stream));
  const int blocks = static_cast<int>((x.n_pairs / x.U + 255) / 256);
  index_count_kernel<<<blocks, 256, 0, stream>>>(idx, x, ib.cnt, status);
  index_scan_kernel<<<1, 1024, 0, stream>>>(x, ib);
  index_fill_kernel<<<blocks, 256, 0, stream>>>(idx, x, ib);
  index_finish_kernel<<<static_cast<int>(x.n_buckets), 128, 0, stream>>>(x, ib);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

}  // namespace sparse_tc
}  // namespace moc
