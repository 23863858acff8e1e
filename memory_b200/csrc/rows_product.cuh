// One column of a projection of a few bf16 rows, C [m <= ROWS, n] = A [m, k] W [n, k]^T, k <= 1,024, by one warp: what
// gemm_rows.cu does for up to eight rows a warp, with the same sums in the same order, where it runs beside something else.
#pragma once
#include "host_pass.cuh"

namespace moc {

__device__ __forceinline__ void unpack8(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
template <int ROWS>
__device__ __forceinline__ void rows_product_column(const RowsProduct& p, int col, int lane) {
  float acc[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) acc[r] = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int at = (lane + 32 * i) * 8;
    if (at >= p.k) break;
    float wf[8];
    unpack8(*reinterpret_cast<const uint4*>(p.w + col * p.ldb + at), wf);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      if (r < p.m) {
        float af[8];
        unpack8(*reinterpret_cast<const uint4*>(p.a + r * p.lda + at), af);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[r] = fmaf(af[j], wf[j], acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float t = warp_sum(acc[r]);
    if (lane == 0 && r < p.m) p.c[r * p.ldc + col] = __float2bfloat16(t);
  }
}

}  // namespace moc
