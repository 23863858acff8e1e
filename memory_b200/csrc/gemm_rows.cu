// Projection of a few rows, C [M <= 256, N] = A [M, K] W [N, K]^T with bf16 operands and fp32 accumulation: the query and
// output projections of a decoding step.  A 128-row tensor-core tile would leave all but a few SMs idle behind one serial
// chain of K steps (10 us at K 768 whatever M is).  Bound by latency: few outputs, and up to eight rows, go to a warp per column and
// eight rows, with the weight row in registers and the sums of the eight rows reduced together (768 x 768: 9.5 -> 2.8 us for one
// row); more of both, to CTAs of 16 columns and 32 rows on single-warp matrix instructions (64 rows: 7.9 -> 4.8 us, one behind the
// other; 10.6 -> 6 in a decoding step).  by_mma says which.
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

// Both operands come to shared memory whole (rows of K elements and 16 bytes, so that the eight rows of an ldmatrix
// meet no bank twice); eight warps take every eighth K step and their sums are added in warp order.
constexpr int kMmaRows = 32, kMmaCols = 16, kMmaWarps = 8;
__host__ __device__ inline int mma_stride(int k) { return (k + 15) / 16 * 32 + 16; }
__global__ void __launch_bounds__(32 * kMmaWarps)
gemm_rows_mma_kernel(const __nv_bfloat16* __restrict__ a, long long lda, const __nv_bfloat16* __restrict__ w, long long ldb,
                     void* __restrict__ c, long long ldc, int c_bf16, int m, int n, int k) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.y * kMmaRows, col0 = blockIdx.x * kMmaCols, stride = mma_stride(k), steps = (k + 15) / 16;
  const uint32_t a_s = smem_u32(smem), w_s = a_s + kMmaRows * stride;
  const int pieces = steps * 2;                       // 16-byte pieces of a row, the last one past K where K is an odd multiple of 8
  for (int i = threadIdx.x; i < (kMmaRows + kMmaCols) * pieces; i += 32 * kMmaWarps) {
    const int r = i / pieces, p = i - r * pieces;
    const bool is_a = r < kMmaRows;
    const bool valid = p * 8 < k && (is_a ? row0 + r < m : col0 + r - kMmaRows < n);
    const __nv_bfloat16* src = is_a ? a + (row0 + r) * lda + p * 8 : w + (col0 + r - kMmaRows) * ldb + p * 8;
    cp_async16_or_zero(a_s + r * stride + p * 16, valid ? src : a, valid);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  float acc[2][2][4];
#pragma unroll
  for (int t = 0; t < 8; ++t) acc[t >> 2][(t >> 1) & 1][0 + 2 * (t & 1)] = acc[t >> 2][(t >> 1) & 1][1 + 2 * (t & 1)] = 0.f;
  const uint32_t a_at = a_s + (lane & 15) * stride + (lane >> 4) * 16;
  const uint32_t w_at = w_s + ((lane & 7) + ((lane >> 4) << 3)) * stride + ((lane >> 3) & 1) * 16;
#pragma unroll 2
  for (int ks = warp; ks < steps; ks += kMmaWarps) {
    uint32_t b[4], x[4], y[4];
    ldsm4(b, w_at + ks * 32);
    ldsm4(x, a_at + ks * 32);
    ldsm4(y, a_at + 16 * stride + ks * 32);
    mma_16816(acc[0][0], x, b[0], b[1]); mma_16816(acc[0][1], x, b[2], b[3]);
    mma_16816(acc[1][0], y, b[0], b[1]); mma_16816(acc[1][1], y, b[2], b[3]);
  }
  __syncthreads();                                    // the operands are read; their place takes the warps' sums
  float* red = reinterpret_cast<float*>(smem);        // [warp][row][col]
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        *reinterpret_cast<float2*>(red + (warp * kMmaRows + 16 * i + (lane >> 2) + 4 * e) * kMmaCols + 8 * j + (lane & 3) * 2) =
            make_float2(acc[i][j][e], acc[i][j][e + 1]);
  __syncthreads();
  for (int i = threadIdx.x; i < kMmaRows * kMmaCols; i += 32 * kMmaWarps) {
    const int r = i / kMmaCols, j = i % kMmaCols;
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < kMmaWarps; ++q) t += red[q * kMmaRows * kMmaCols + i];
    if (row0 + r < m && col0 + j < n) {
      const long long at = (row0 + r) * ldc + col0 + j;
      if (c_bf16) static_cast<__nv_bfloat16*>(c)[at] = __float2bfloat16(t);
      else static_cast<float*>(c)[at] = t;
    }
  }
}

}  // namespace

// Whether the matrix instructions take a projection, us a warp a column and they: 24 x 768 3.6 and 4.8, 32 x 768 5.7 and 4.8, 24 x 1,536
// 6.0 and 4.9, 64 x 256 over K 1,024 5.3 and 5.6, 256 x 64 3.6 and 4.8 (tensor-core tiles: 9.0).  Up to eight rows they would be three
// quarters padding: 8 x 3,072 over K 256 / 512 / 768 / 1,024: 3.0 / 3.9 / 5.5 / 5.8 and 3.4 / 4.6 / 5.8 / 6.9.  Where fp32 FMAs of at most
// 64 rows ran before them, results in fp32 stay theirs: 6.6e-8 from fp64 (2-norm, K 768) against 1.07e-7; rounded to bf16 both are
// 1.65e-3 and agree to nine digits.  (The tensor-core tiles: 7.3e-7.)
constexpr int kWarpRows = 64;
constexpr long long kWarpOutputs = 64 * 1024, kMmaFrom = 24 * 1024;
bool by_warps(const moc_gemm_desc* g) { return g->m <= kWarpRows && static_cast<long long>(g->m) * g->n <= kWarpOutputs; }
bool by_mma(const moc_gemm_desc* g) {
  return g->m > kRows && static_cast<long long>(g->m) * g->n >= kMmaFrom && !(by_warps(g) && g->c_dtype == MOC_F32);
}

// Whether the kernels take this projection: plain operands, rows of at most 1,024 (32 registers of operands a lane and row),
// and few enough of them: their work grows with M N while the tensor-core tiles stay at the length of their K chain until N
// fills the chip.  The line is the CTAs of the matrix instructions, us there and here: 384 of them, 256 x 768 over K 768 9.8 and
// 7.5, over 1,024 11.5 and 11.5; 128 x 1,536 9.9 and 7.6, 11.5 and 11.5; 480, 160 x 1,536 over 768 10.0 and 10.4; 512, 16 x 8,192
// 9.8 and 10.4, 128 x 2,048 9.9 and 10.8; 1,024, 9 x 16,384 10.7 and 16.6.
constexpr int kMmaCtas = 384;
bool gemm_rows_supported(const moc_gemm_desc* g, const float* row_scale, const int32_t* a_row_blocks,
                         const int32_t* b_row_blocks) {
  const bool few = by_warps(g) || (g->m <= 256 && static_cast<long long>(ceil_div(g->m, kMmaRows)) * ceil_div(g->n, kMmaCols) <= kMmaCtas);
  return few && g->k <= 1024 && g->a_kmajor && g->b_kmajor && !g->accumulate && g->split_k <= 1 &&
         g->residual == nullptr && row_scale == nullptr && a_row_blocks == nullptr && b_row_blocks == nullptr;
}
int launch_gemm_rows(const moc_gemm_desc* g, const void* a, const void* b, void* c, cudaStream_t stream) {
  if (by_mma(g)) {
    const int sums = kMmaWarps * kMmaRows * kMmaCols * 4;
    const int bytes = std::max((kMmaRows + kMmaCols) * mma_stride(g->k), sums);
    MOC_CUDA_OK(allow_shared(gemm_rows_mma_kernel, bytes, (kMmaRows + kMmaCols) * mma_stride(1024)));
    gemm_rows_mma_kernel<<<dim3(ceil_div(g->n, kMmaCols), ceil_div(g->m, kMmaRows)), 32 * kMmaWarps, bytes, stream>>>(
        static_cast<const __nv_bfloat16*>(a), g->lda, static_cast<const __nv_bfloat16*>(b), g->ldb, c, g->ldc,
        g->c_dtype == MOC_BF16, g->m, g->n, g->k);
    MOC_CUDA_OK(cudaGetLastError());
    return MOC_OK;
  }
  auto kern = g->k <= 256 ? gemm_rows_kernel<1> : g->k <= 512 ? gemm_rows_kernel<2>
              : g->k <= 768 ? gemm_rows_kernel<3> : gemm_rows_kernel<4>;
  kern<<<dim3(ceil_div(g->n, kCols), ceil_div(g->m, kRows)), 32 * kCols, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(a), g->lda, static_cast<const __nv_bfloat16*>(b), g->ldb, c, g->ldc,
      g->c_dtype == MOC_BF16, g->m, g->n, g->k);
  MOC_CUDA_OK(cudaGetLastError());
  return MOC_OK;
}

}  // namespace moc
