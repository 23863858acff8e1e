// Projection of a few rows, C [M <= 64, N] = A [M, K] W [N, K]^T with bf16 operands and fp32 accumulation: the query and
// output projections of a decoding step.  A 128-row tensor-core tile would leave all but a few SMs idle behind one serial
// chain of K steps (10 us at K 768 whatever M is); bound by latency, the work goes to a warp per column and eight rows, with
// the weight row in registers and the sums of the eight rows reduced together.  768 x 768: 9.5 -> 2.8 us for one row, 11 -> 10
// for 64.
#include "rows_product.cuh"

namespace moc {
namespace {

constexpr int kRows = 8, kCols = 8;
// NV: 16-byte pieces of a row per lane (K <= 256 NV)
template <int NV>
__global__ void __launch_bounds__(32 * kCols)
gemm_rows_kernel(const __nv_bfloat16* __restrict__ a, long long lda, const __nv_bfloat16* __restrict__ w, long long ldb,
                 void* __restrict__ c, long long ldc, int c_bf16, int m, int n, int k) {
  __shared__ float tile[kRows][kCols];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = min(static_cast<int>(blockIdx.x) * kCols + warp, n - 1), row0 = blockIdx.y * kRows;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 wv[NV], av[kRows][NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int p = (lane + 32 * i) * 8;
    wv[i] = p < k ? *reinterpret_cast<const uint4*>(w + col * ldb + p) : zero;
  }
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const __nv_bfloat16* src = a + min(row0 + r, m - 1) * lda;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int p = (lane + 32 * i) * 8;
      av[r][i] = p < k ? *reinterpret_cast<const uint4*>(src + p) : zero;
    }
  }
  float acc[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) acc[r] = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float wf[8];
    unpack8(wv[i], wf);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      float af[8];
      unpack8(av[r][i], af);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[r] = fmaf(af[j], wf[j], acc[r]);
    }
  }
  int o = 16;
#pragma unroll
  for (int h = kRows / 2; h > 0; h >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const float send = up ? acc[i] : acc[i + h];
      const float keep = up ? acc[i + h] : acc[i];
      acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    o >>= 1;
  }
  acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
  acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
  if ((lane & 3) == 0) tile[lane >> 2][warp] = acc[0];
  __syncthreads();
  const int r = threadIdx.x / kCols, j = threadIdx.x % kCols, oc = blockIdx.x * kCols + j;
  if (r < kRows && row0 + r < m && oc < n) {
    const long long at = (row0 + r) * ldc + oc;
    if (c_bf16) static_cast<__nv_bfloat16*>(c)[at] = __float2bfloat16(tile[r][j]);
    else static_cast<float*>(c)[at] = tile[r][j];
  }
}

}  // namespace

// Whether the kernel takes this projection: plain operands, rows of at most 1,024 (32 registers of operands a lane and row),
// and few enough of them: the work grows with M N while the tensor-core tiles stay at the length of their K chain until N
// fills the chip (64 x 1,536: 16 us here, 10 there).
bool gemm_rows_supported(const moc_gemm_desc* g, const float* row_scale, const int32_t* a_row_blocks,
                         const int32_t* b_row_blocks) {
  return g->m <= 64 && static_cast<long long>(g->m) * g->n <= 64 * 1024 && g->k <= 1024 && g->a_kmajor && g->b_kmajor && !g->accumulate && g->split_k <= 1 &&
         g->residual == nullptr && row_scale == nullptr && a_row_blocks == nullptr && b_row_blocks == nullptr;
}
int launch_gemm_rows(const moc_gemm_desc* g, const void* a, const void* b, void* c, cudaStream_t stream) {
  auto kern = g->k <= 256 ? gemm_rows_kernel<1> : g->k <= 512 ? gemm_rows_kernel<2>
              : g->k <= 768 ? gemm_rows_kernel<3> : gemm_rows_kernel<4>;
  kern<<<dim3(ceil_div(g->n, kCols), ceil_div(g->m, kRows)), 32 * kCols, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(a), g->lda, static_cast<const __nv_bfloat16*>(b), g->ldb, c, g->ldc,
      g->c_dtype == MOC_BF16, g->m, g->n, g->k);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

}  // namespace moc
