// C[M,N] = A[M,K] * W[N,K]^T on CUDA cores in float32 (FFMA, no tensor cores,
// no reduced-precision mode), for the true 32-bit path and for weights that a
// checkpoint stores in 32-bit.  Weights keep the (out, in) layout of the
// checkpoint, y = x W^T (engine/layers.py:48-50).
//
// Every output element is one accumulator that walks k = 0..K-1 in ascending
// order, so a row's result does not depend on how many rows share the launch.
// A, W and C may each be float32 or bfloat16; products and sums are float32.
//
// A product of all float32 whose rows lie on 16 bytes goes to gemm_f32.cu, which reads W once at HBM speed for a few rows and
// keeps the multipliers busy for many; this kernel keeps mixed types and rows off that alignment.
#include "common.cuh"

int gemm_f32_takes(const void* A, const void* W, int K, int lda, int ldw);
int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream);

#define GS_BM 64
#define GS_BN 64
#define GS_BK 16
#define GS_THREADS 256

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(GS_THREADS) gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                                TC* __restrict__ C, int M, int N, int K, int lda,
                                                                int ldw, int ldc, long long a_batch, long long w_batch,
                                                                long long c_batch) {
  pdl_trigger();
  pdl_wait();
  A += (size_t)blockIdx.z * a_batch;      // a batch of independent products (blockIdx.z), each with its own offsets
  W += (size_t)blockIdx.z * w_batch;
  C += (size_t)blockIdx.z * c_batch;
  __shared__ float As[GS_BK][GS_BM + 4];
  __shared__ float Ws[GS_BK][GS_BN + 4];
  const int m0 = blockIdx.y * GS_BM, n0 = blockIdx.x * GS_BN;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;      // 16 x 16 threads, 4 x 4 outputs each
  const int lr = tid >> 2, lc = (tid & 3) * 4;  // loader: row 0..63, k offset 0,4,8,12
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += GS_BK) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + lc + u;
      const int am = m0 + lr, wn = n0 + lr;
      As[lc + u][lr] = (am < M && k < K) ? to_f32(A[(size_t)am * lda + k]) : 0.f;
      Ws[lc + u][lr] = (wn < N && k < K) ? to_f32(W[(size_t)wn * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GS_BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[(size_t)m * ldc + n] = from_f32<TC>(acc[i][j]);
    }
  }
}

template <typename TA, typename TW, typename TC>
static int launch_gemm(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc,
                       cudaStream_t stream, int batch = 1, long long a_batch = 0, long long w_batch = 0,
                       long long c_batch = 0) {
  dim3 grid((N + GS_BN - 1) / GS_BN, (M + GS_BM - 1) / GS_BM, batch);
  return launch_k(gemm_simt_kernel<TA, TW, TC>, grid, GS_THREADS, 0, stream, (const TA*)A, (const TW*)W, (TC*)C, M, N,
                  K, lda, ldw, ldc, a_batch, w_batch, c_batch);
}

extern "C" int ie_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype, int M,
                            int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return IE_OK;
  if (K <= 0) return IE_BAD_SIZE;
  const int code = a_dtype * 4 + w_dtype * 2 + c_dtype;
  switch (code) {
    case 0:
      if (gemm_f32_takes(A, W, K, lda, ldw))
        return gemm_f32((const float*)A, (const float*)W, (float*)C, M, N, K, lda, ldw, ldc, stream);
      return launch_gemm<float, float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    case 2: return launch_gemm<float, bf16, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    case 4: return launch_gemm<bf16, float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    case 5: return launch_gemm<bf16, float, bf16>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    case 6: return launch_gemm<bf16, bf16, float>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    case 7: return launch_gemm<bf16, bf16, bf16>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    default: return IE_BAD_DTYPE;
  }
}

// `batch` independent products in one launch: product b reads A + b * a_batch, W + b * w_batch and writes
// C + b * c_batch (offsets in elements).  A block-diagonal matrix applied to the rows of A is such a batch: block b
// reads columns b * K .. of A and writes columns b * N .. of C.
extern "C" int ie_gemm_simt_batched(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype, int M,
                                    int N, int K, int lda, int ldw, int ldc, int batch, long long a_batch,
                                    long long w_batch, long long c_batch, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return IE_OK;
  if (K <= 0 || batch > 65535) return IE_BAD_SIZE;
  const int code = a_dtype * 4 + w_dtype * 2 + c_dtype;
  switch (code) {
    case 0: return launch_gemm<float, float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream, batch, a_batch, w_batch, c_batch);
    case 2: return launch_gemm<float, bf16, float>(A, W, C, M, N, K, lda, ldw, ldc, stream, batch, a_batch, w_batch, c_batch);
    case 4: return launch_gemm<bf16, float, float>(A, W, C, M, N, K, lda, ldw, ldc, stream, batch, a_batch, w_batch, c_batch);
    case 6: return launch_gemm<bf16, bf16, float>(A, W, C, M, N, K, lda, ldw, ldc, stream, batch, a_batch, w_batch, c_batch);
    default: return IE_BAD_DTYPE;
  }
}

// four neighbouring elements as float32
__device__ __forceinline__ float4 rd_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 rd_load4(const bf16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// The same for a few rows (decode tokens): a warp an output column, its lanes stride k four at a time with one sum per row, then a
// tree over the lanes; the order is fixed by (n, k) alone.  The tile kernel gives 8 rows of 8 blocks of 256 x 256 to 32 thread
// blocks that walk K alone, 16 stages of loads one after the other (15.0 us; 4.9 here).
template <typename TA, typename TW>
__global__ void __launch_bounds__(256) gemm_diag_rows_kernel(const TA* __restrict__ A, const TW* __restrict__ W, float* __restrict__ C,
                                                             int M, int cols, int n, int K, int lda, int ldc) {
  constexpr int MR = 8;
  pdl_trigger();
  const int col = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_wait();
  if (col >= cols) return;
  const TW* w = W + (size_t)col * K;
  const TA* a = A + (size_t)(col / n) * K;
  for (int m0 = 0; m0 < M; m0 += MR) {
    float acc[MR] = {};
    for (int k = lane * 4; k < K; k += 128) {
      const float4 wv = rd_load4(w + k);
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        const float4 x = rd_load4(a + (size_t)min(m0 + r, M - 1) * lda + k);
        acc[r] = fmaf(x.w, wv.w, fmaf(x.z, wv.z, fmaf(x.y, wv.y, fmaf(x.x, wv.x, acc[r]))));
      }
    }
#pragma unroll
    for (int r = 0; r < MR; ++r) {
      const float total = warp_sum(acc[r]);
      if (lane == 0 && m0 + r < M) C[(size_t)(m0 + r) * ldc + col] = total;
    }
  }
}

// W [blocks, n, K]: block b maps columns b K .. of A to columns b n .. of C; rows of A and W start on four elements
extern "C" int ie_gemm_diag_rows(const void* A, int a_dtype, const void* W, int w_dtype, float* C, int M, int blocks, int n, int K,
                                 int lda, int ldc, cudaStream_t stream) {
  if (M <= 0 || n <= 0 || blocks <= 0) return IE_OK;
  if (K <= 0 || K % 4 || lda % 4 || (long long)blocks * n > 0x7fffffffLL) return IE_BAD_SIZE;
  if (((uintptr_t)A | (uintptr_t)W) & 15) return IE_BAD_ALIGN;
  const int cols = blocks * n;
  const unsigned grid = (unsigned)((cols + 7) / 8);
#define DR_GO(TA, TW) return launch_k(gemm_diag_rows_kernel<TA, TW>, grid, 256, 0, stream, (const TA*)A, (const TW*)W, C, M, cols, n, K, lda, ldc)
  if (a_dtype == IE_F32 && w_dtype == IE_F32) DR_GO(float, float);
  if (a_dtype == IE_F32 && w_dtype == IE_BF16) DR_GO(float, bf16);
  if (a_dtype == IE_BF16 && w_dtype == IE_F32) DR_GO(bf16, float);
  if (a_dtype == IE_BF16 && w_dtype == IE_BF16) DR_GO(bf16, bf16);
#undef DR_GO
  return IE_BAD_DTYPE;
}

// ------------------------------------------------------------------ few output columns (a router)
// C[m, n] = sum_k A[m, k] W[n, k] for N of a few dozen: the tile kernel above would give all of it to one block
// that walks K alone.  Here a block takes a row of A into shared memory and each of its eight warps takes outputs
// n = warp, warp + 8, ...: a lane takes four neighbouring k of every 128 with a sum for each (VEC; k = lane, lane + 32, ... where rows
// of W do not start on four elements), then a tree over the lanes.  The order is fixed by (n, k) alone, so a row's result
// does not depend on how many rows share the launch.  float32 arithmetic.  (2,048 rows of 17 outputs over 2,048 columns in
// a step: with four rows a block and two outputs a warp 38 us, eight rows and one output 41 us, a row a block 21:
// 17 outputs leave warps idle in the last round, and the more rows a block has the fewer blocks hide it.)
template <typename TA, typename TW, bool VEC>
__global__ void __launch_bounds__(256) gemm_rowdot_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                          float* __restrict__ C, int N, int K, int lda, int ldw, int ldc) {
  extern __shared__ __align__(16) float a_s[];
  pdl_trigger();
  pdl_wait();
  const int m = blockIdx.x;
  for (int k = threadIdx.x; k < K; k += blockDim.x) a_s[k] = to_f32(A[(size_t)m * lda + k]);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // blocks along y share a row's outputs in groups of eight (a few rows then still fill the device)
  for (int n = blockIdx.y * 8 + warp; n < N; n += 8 * gridDim.y) {
    const TW* w = W + (size_t)n * ldw;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (VEC) {
#pragma unroll 4
      for (int k = lane * 4; k < K; k += 128) {
        const float4 wv = rd_load4(w + k), x = *reinterpret_cast<const float4*>(a_s + k);
        acc[0] = fmaf(x.x, wv.x, acc[0]);
        acc[1] = fmaf(x.y, wv.y, acc[1]);
        acc[2] = fmaf(x.z, wv.z, acc[2]);
        acc[3] = fmaf(x.w, wv.w, acc[3]);
      }
    } else {
      int k = lane;
      for (; k + 96 < K; k += 128) {
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = fmaf(a_s[k + 32 * u], to_f32(w[k + 32 * u]), acc[u]);
      }
#pragma unroll
      for (int u = 0; u < 3; ++u)
        if (k + 32 * u < K) acc[u] = fmaf(a_s[k + 32 * u], to_f32(w[k + 32 * u]), acc[u]);
    }
    const float total = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
    if (lane == 0) C[(size_t)m * ldc + n] = total;
  }
}

extern "C" int ie_gemm_rowdot(const void* A, int a_dtype, const void* W, int w_dtype, float* C, int M, int N, int K,
                              int lda, int ldw, int ldc, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return IE_OK;
  if (K <= 0 || (size_t)K * sizeof(float) > 200 * 1024) return IE_BAD_SIZE;
  const bool vec = K % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)W & 15) == 0;
  const size_t smem = (size_t)K * sizeof(float);
  // few rows (decode tokens): a block a row and eight outputs, so that the weight rows stream through many blocks
  const dim3 grid(M, M <= 128 ? (N + 7) / 8 : 1);
#define RD_RUN(TA, TW, VEC)                                                                                        \
  {                                                                                                                \
    if (smem > 47 * 1024) {                                                                                        \
      cudaError_t e = cudaFuncSetAttribute(gemm_rowdot_kernel<TA, TW, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                           (int)smem);                                                             \
      if (e != cudaSuccess) return (int)e;                                                                         \
    }                                                                                                              \
    return launch_k(gemm_rowdot_kernel<TA, TW, VEC>, grid, 256, smem, stream, (const TA*)A, (const TW*)W, C, N, K, lda, ldw, \
                    ldc);                                                                                          \
  }
#define RD_GO(TA, TW)             \
  {                               \
    if (vec) RD_RUN(TA, TW, true); \
    RD_RUN(TA, TW, false);        \
  }
  if (a_dtype == IE_F32 && w_dtype == IE_F32) RD_GO(float, float);
  if (a_dtype == IE_F32 && w_dtype == IE_BF16) RD_GO(float, bf16);
  if (a_dtype == IE_BF16 && w_dtype == IE_F32) RD_GO(bf16, float);
  if (a_dtype == IE_BF16 && w_dtype == IE_BF16) RD_GO(bf16, bf16);
#undef RD_GO
#undef RD_RUN
  return IE_BAD_DTYPE;
}
