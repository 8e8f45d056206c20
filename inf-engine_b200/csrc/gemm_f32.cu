// C[M,N] = A[M,K] W[N,K]^T, all float32, for the true 32-bit path: FFMA only, no tensor cores (weights keep the (out, in)
// layout of the checkpoint, engine/layers.py:48-50).  Two kernels, one order of sums:
//
//   K is cut into GF_PARTS equal runs of k (multiples of GF_BK); within a run one accumulator takes the even k and one the
//   odd k, ascending, and the run's sum is even + odd; the result adds the runs in order.
//
// Both kernels follow it, so a row's result does not depend on how many rows share the launch nor on the kernel that took it.
// Even and odd k are the two lanes of fma.rn.f32x2 (two IEEE float32 products a lane pair and instruction): neighbouring k lie
// side by side in memory, so operands need neither a transpose nor a broadcast.
//
// stream: up to 16 rows.  The product is a read of W (4 bytes a weight): HBM bounds it.  (A tile kernel reads it at 6 to
//   14 % of HBM: tiles of 64 rows for 4, loads of 4 bytes, blocks that walk all of K alone.)  Warp w of a block or cluster owns run w
//   of K and streams its slice of 32 or 64 weight rows (and of the few activation rows, which come from L2) through a ring
//   of its own, 16 bytes a lane and copy; no barrier but one at the end of a group of rows.
// tile: more rows.  64 x 128 (or 32 x 128) outputs a block, 8 x 8 (4 x 8) a thread; FFMA bounds it (300 rows: 588 GFLOP for
//   a model whose layers hold 0.97 G weights, 7.9 ms at 74 TFLOP/s).  Where the tiles alone leave SMs idle, the eight runs of K
//   go to the eight blocks of a cluster, which add up through distributed shared memory in the same order.
//
// Measured on B200, us of a product, before (gemm_simt.cu's tile kernel) and now.  4 rows of 16,384 x 2,048: 325 and 30 (4.4
// TB/s), 128,256 x 2,048: 1,187 and 195 (5.4 TB/s).  300 rows of 16,384 x 2,048: 882 and 581 (35 TFLOP/s).  What holds the
// tile kernel at half of the FFMA rate: two warps a scheduler (128 sums a thread), which barriers and waits leave idle.
#include "common.cuh"

namespace {

constexpr int GF_PARTS = 8;
constexpr int GF_BK = 32;              // k of a stage: 128 bytes of a row
constexpr int GF_PITCH = 36;           // floats between staged rows: 16-byte reads of 8 consecutive rows hit 32 banks

typedef unsigned long long f2;         // two float32 side by side (k, k + 1)

__device__ __forceinline__ f2 ffma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float even_plus_odd(f2 v) {
  return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}
__device__ __forceinline__ uint32_t gf_saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes (or 16 zero bytes when `there` is false; the address is then not read)
__device__ __forceinline__ void gf_copy16(uint32_t dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void gf_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void gf_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
struct alignas(16) Pair2 { f2 lo, hi; };     // four consecutive k
__device__ __forceinline__ Pair2 gf_lds(uint32_t addr) {
  Pair2 v;
  asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];" : "=l"(v.lo), "=l"(v.hi) : "r"(addr));
  return v;
}

struct GfParams {
  const float* A;
  const float* W;
  float* C;
  int M, N, K, lda, ldw, ldc;
  int part;      // k of a run: the runs start at 0, part, 2 part, ... (the last ones may be short or empty)
};

// ------------------------------------------------------------------------------------------------ up to 16 rows
// A 16-byte read of shared memory costs its four cycles whether or not lanes read the same place, so what counts is reads
// per weight: lane (lane / 2, lane % 2) owns NR weight rows and MR activation rows, NR + MR reads for 16 NR rows of four k.
// The GF_PARTS runs lie with the warps of a cluster of CL blocks; block 0's share of the results is that of its rank.
template <int NR, int MR, int STAGES, int CL>
__global__ void __launch_bounds__(32 * (GF_PARTS / CL)) gemm_f32_stream_kernel(GfParams p) {
  extern __shared__ __align__(16) float gf_smem[];
  constexpr int W_ROWS = 16 * NR, X_ROWS = 2 * MR, ROWS = W_ROWS + X_ROWS, WARPS = GF_PARTS / CL;
  static_assert(W_ROWS * X_ROWS <= 2048 && ROWS % 2 == 0, "");
  __shared__ float red[2][WARPS][W_ROWS * X_ROWS];
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = CL > 1 ? (int)(blockIdx.x % CL) : 0;
  const int first_group = blockIdx.x / CL, group_step = gridDim.x / CL;
  const int run = rank * WARPS + warp;
  const int k_lo = min(p.K, run * p.part), k_hi = min(p.K, k_lo + p.part);
  const int chunks = (k_hi - k_lo + GF_BK - 1) / GF_BK;          // stages of this warp in a group of rows
  const int n_groups = (p.N + W_ROWS - 1) / W_ROWS;
  const int my_groups = (n_groups - first_group + group_step - 1) / group_step;
  const int total = my_groups * chunks;
  const uint32_t ring = gf_saddr(gf_smem) + (uint32_t)(warp * STAGES * ROWS * GF_PITCH) * 4;
  const int cr = lane >> 3, ck = (lane & 7) * 4;                 // copies: row cr + 4 i, k offset ck

  auto copy_w = [&](int slot, int g, int c) {
    const int k = k_lo + c * GF_BK + ck;
    const uint32_t dst = ring + (uint32_t)(slot * ROWS * GF_PITCH + cr * GF_PITCH + ck) * 4;
#pragma unroll
    for (int i = 0; i < W_ROWS / 4; ++i) {
      const int n = g * W_ROWS + cr + 4 * i;
      const bool there = n < p.N && k < k_hi;
      gf_copy16(dst + i * 4 * GF_PITCH * 4, p.W + (there ? (size_t)n * p.ldw + k : 0), there);
    }
  };
  auto copy_x = [&](int slot, int c) {
    const int k = k_lo + c * GF_BK + ck;
    const uint32_t dst = ring + (uint32_t)(slot * ROWS * GF_PITCH + (W_ROWS + cr) * GF_PITCH + ck) * 4;
#pragma unroll
    for (int i = 0; i < (X_ROWS + 3) / 4; ++i) {
      const int m = cr + 4 * i;
      const bool there = m < p.M && k < k_hi;
      if (X_ROWS % 4 == 0 || m < X_ROWS) gf_copy16(dst + i * 4 * GF_PITCH * 4, p.A + (there ? (size_t)m * p.lda + k : 0), there);
    }
  };
  int g_load = first_group, c_load = 0;                          // where the next stage's copies are
  auto advance = [&]() {
    if (++c_load == chunks) { c_load = 0; g_load += group_step; }
  };

  // the weights do not depend on the kernel ahead: the first ring of them is asked for before the wait
  {
    int g = g_load, c = c_load;
    for (int s = 0; s < STAGES; ++s) {
      if (s < total) copy_w(s, g, c);
      if (++c == chunks) { c = 0; g += group_step; }
    }
  }
  pdl_wait();
  for (int s = 0; s < STAGES; ++s) {
    if (s < total) copy_x(s, c_load);
    gf_commit();
    if (chunks) advance();
  }

  int slot = 0, it = 0, parity = 0;
  const int wr = lane >> 1, xr = lane & 1;
  for (int gi = 0; gi < my_groups; ++gi) {
    const int g = first_group + gi * group_step;
    f2 acc[NR][MR];
#pragma unroll
    for (int a = 0; a < NR; ++a)
#pragma unroll
      for (int b = 0; b < MR; ++b) acc[a][b] = 0ull;
    for (int c = 0; c < chunks; ++c) {
      gf_wait<STAGES - 1>();
      __syncwarp();
      const uint32_t base = ring + (uint32_t)(slot * ROWS * GF_PITCH) * 4;
      const uint32_t wa = base + (uint32_t)(wr * GF_PITCH) * 4, xa = base + (uint32_t)((W_ROWS + xr) * GF_PITCH) * 4;
#pragma unroll
      for (int k4 = 0; k4 < GF_BK / 4; ++k4) {
        Pair2 w[NR], x[MR];
#pragma unroll
        for (int a = 0; a < NR; ++a) w[a] = gf_lds(wa + (a * 16 * GF_PITCH + k4 * 4) * 4);
#pragma unroll
        for (int b = 0; b < MR; ++b) x[b] = gf_lds(xa + (b * 2 * GF_PITCH + k4 * 4) * 4);
#pragma unroll
        for (int a = 0; a < NR; ++a)
#pragma unroll
          for (int b = 0; b < MR; ++b) acc[a][b] = ffma2(x[b].lo, w[a].lo, acc[a][b]);
#pragma unroll
        for (int a = 0; a < NR; ++a)
#pragma unroll
          for (int b = 0; b < MR; ++b) acc[a][b] = ffma2(x[b].hi, w[a].hi, acc[a][b]);
      }
      __syncwarp();                       // every lane has read the slot
      if (it + STAGES < total) { copy_w(slot, g_load, c_load); copy_x(slot, c_load); advance(); }
      gf_commit();
      ++it;
      if (++slot == STAGES) slot = 0;
    }
    // this run's sums; one barrier a group, two buffers: what is written here was last read two barriers ago
#pragma unroll
    for (int a = 0; a < NR; ++a)
#pragma unroll
      for (int b = 0; b < MR; ++b) red[parity][warp][(xr + 2 * b) * W_ROWS + wr + 16 * a] = even_plus_odd(acc[a][b]);
    if (CL > 1) asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
    else __syncthreads();
    for (int i = rank * (32 * WARPS) + threadIdx.x; i < W_ROWS * X_ROWS; i += 32 * GF_PARTS) {
      const int m = i / W_ROWS, n = g * W_ROWS + i % W_ROWS;
      if (m < p.M && n < p.N) {
        float v[GF_PARTS];
#pragma unroll
        for (int q = 0; q < GF_PARTS; ++q) {
          if (CL > 1) {
            uint32_t there;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(gf_saddr(&red[parity][q % WARPS][i])), "r"(q / WARPS));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[q]) : "r"(there) : "memory");
          } else {
            v[q] = red[parity][q % WARPS][i];
          }
        }
        float sum = v[0];
#pragma unroll
        for (int q = 1; q < GF_PARTS; ++q) sum += v[q];
        p.C[(size_t)m * p.ldc + n] = sum;
      }
    }
    parity ^= 1;
  }
  gf_wait<0>();
  // no block leaves while another still reads its sums
  if (CL > 1) asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}

// ------------------------------------------------------------------------------------------------- more rows
// Warps 2 (m) x 2 (n), lanes 4 (m) x 8 (n): thread (tm, tn) holds rows tm + 8 i and columns tn + 16 j, so that a warp's reads
// touch consecutive staged rows.  8 x 8 outputs a thread: a 16-byte read of shared memory costs four cycles, the 8 products
// it then feeds as much (8 x 4 a thread ran at 37 TFLOP/s, bound by the reads).  SPLIT: the cluster's eight blocks take a run of K each.
constexpr int GF_BN = 128;
constexpr int GF_TILE_STAGES = 2;
constexpr int GF_TILE_THREADS = 128;

template <int TM, bool SPLIT>
__global__ void __launch_bounds__(GF_TILE_THREADS, 2) gemm_f32_tile_kernel(GfParams p) {
  constexpr int BM = 8 * TM, ROWS = BM + GF_BN, STAGE = ROWS * GF_PITCH;
  extern __shared__ __align__(16) float gf_smem[];       // the ring; then sums of finished runs (SPLIT: of this block's)
  pdl_trigger();
  float* const sums = gf_smem + GF_TILE_STAGES * STAGE;  // [BM][GF_BN]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tm = (warp & 1) * 4 + (lane & 3), tn = (warp >> 1) * 8 + (lane >> 2);
  const int rank = SPLIT ? (int)(blockIdx.x % GF_PARTS) : 0;
  const int tile = SPLIT ? blockIdx.x / GF_PARTS : blockIdx.x;
  const int m_tiles = (p.M + BM - 1) / BM;
  const int m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * GF_BN;   // neighbours share the weights' columns
  const uint32_t ring = gf_saddr(gf_smem);
  const int cr = tid >> 3, ck = (tid & 7) * 4;           // copies: row cr + 16 i

  auto copy_w = [&](int slot, int k, int k_hi) {
#pragma unroll
    for (int i = 0; i < GF_BN / 16; ++i) {
      const int n = n0 + cr + 16 * i;
      const bool there = n < p.N && k + ck < k_hi;
      gf_copy16(ring + (uint32_t)(slot * STAGE + (BM + cr + 16 * i) * GF_PITCH + ck) * 4,
                p.W + (there ? (size_t)n * p.ldw + k + ck : 0), there);
    }
  };
  auto copy_x = [&](int slot, int k, int k_hi) {
#pragma unroll
    for (int i = 0; i < BM / 16; ++i) {
      const int m = m0 + cr + 16 * i;
      const bool there = m < p.M && k + ck < k_hi;
      gf_copy16(ring + (uint32_t)(slot * STAGE + (cr + 16 * i) * GF_PITCH + ck) * 4,
                p.A + (there ? (size_t)m * p.lda + k + ck : 0), there);
    }
  };

  bool first = true, waited = false;
  for (int part = rank; part < GF_PARTS; part += SPLIT ? GF_PARTS : 1) {
    const int k_lo = min(p.K, part * p.part), k_hi = min(p.K, k_lo + p.part);
    const int chunks = (k_hi - k_lo + GF_BK - 1) / GF_BK;
    if (chunks == 0 && !(SPLIT || first)) break;
    f2 acc[TM][8];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
    if (chunks > 0) {
      copy_w(0, k_lo, k_hi);
      if (!waited) { pdl_wait(); waited = true; }
      copy_x(0, k_lo, k_hi);
    }
    gf_commit();
    for (int c = 0; c < chunks; ++c) {
      gf_wait<0>();
      __syncthreads();                    // stage c is there for all, and all have read stage c - 1
      if (c + 1 < chunks) {
        copy_w((c + 1) & 1, k_lo + (c + 1) * GF_BK, k_hi);
        copy_x((c + 1) & 1, k_lo + (c + 1) * GF_BK, k_hi);
        gf_commit();
      }
      const uint32_t base = ring + (uint32_t)((c & 1) * STAGE) * 4;
      const uint32_t xa = base + (uint32_t)(tm * GF_PITCH) * 4, wa = base + (uint32_t)((BM + tn) * GF_PITCH) * 4;
#pragma unroll 2
      for (int k4 = 0; k4 < GF_BK / 4; ++k4) {
        Pair2 w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = gf_lds(wa + (j * 16 * GF_PITCH + k4 * 4) * 4);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const Pair2 x = gf_lds(xa + (i * 8 * GF_PITCH + k4 * 4) * 4);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][j] = ffma2(x.lo, w[j].lo, acc[i][j]);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][j] = ffma2(x.hi, w[j].hi, acc[i][j]);
        }
      }
    }
    __syncthreads();                      // the next run copies into the stages again
    // the run's sum joins what earlier runs left (a place belongs to one thread: no barrier)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float* at = sums + (tm + 8 * i) * GF_BN + tn + 16 * j;
        const float v = even_plus_odd(acc[i][j]);
        *at = (SPLIT || first) ? v : *at + v;
      }
    first = false;
  }
  if (!waited) pdl_wait();

  if (SPLIT) {
    // block r of the cluster adds up rows r, r + 8, ... of the tile over the eight blocks, in order
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
    for (int e = tid; e < TM * GF_BN; e += GF_TILE_THREADS) {
      const int r = rank + 8 * (e / GF_BN), c = e % GF_BN;
      const uint32_t at = gf_saddr(sums + r * GF_BN + c);
      float part[GF_PARTS];
#pragma unroll
      for (int q = 0; q < GF_PARTS; ++q) {
        uint32_t there;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"(q));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part[q]) : "r"(there) : "memory");
      }
      float sum = part[0];
#pragma unroll
      for (int q = 1; q < GF_PARTS; ++q) sum += part[q];
      if (m0 + r < p.M && n0 + c < p.N) p.C[(size_t)(m0 + r) * p.ldc + n0 + c] = sum;
    }
    // no block leaves while another still reads its sums
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
  } else {
    __syncthreads();
    for (int e = tid; e < BM * GF_BN; e += GF_TILE_THREADS) {
      const int r = e / GF_BN, c = e % GF_BN;
      if (m0 + r < p.M && n0 + c < p.N) p.C[(size_t)(m0 + r) * p.ldc + n0 + c] = sums[e];
    }
  }
}

template <typename K>
int gf_allow_smem(K kernel, size_t smem) {
  return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

template <int NR, int MR, int STAGES, int CL>
int launch_stream(const GfParams& p, int max_clusters, cudaStream_t stream) {
  constexpr size_t smem = (size_t)(GF_PARTS / CL) * STAGES * (16 * NR + 2 * MR) * GF_PITCH * 4;
  static OncePerDevice once;
  const int ready = once([] { return gf_allow_smem(gemm_f32_stream_kernel<NR, MR, STAGES, CL>, smem); });
  if (ready) return ready;
  const int groups = (p.N + 16 * NR - 1) / (16 * NR);
  const int grid = (max_clusters > 0 && groups > max_clusters ? max_clusters : groups) * CL;
  if (CL > 1)
    return launch_k_cluster(gemm_f32_stream_kernel<NR, MR, STAGES, CL>, CL, grid, 32 * (GF_PARTS / CL), smem, stream, p);
  return launch_k(gemm_f32_stream_kernel<NR, MR, STAGES, CL>, grid, 32 * (GF_PARTS / CL), smem, stream, p);
}

template <int TM, bool SPLIT>
int launch_tile(const GfParams& p, int tiles, cudaStream_t stream) {
  constexpr size_t smem = ((size_t)GF_TILE_STAGES * (8 * TM + GF_BN) * GF_PITCH + 8 * TM * GF_BN) * 4;
  static OncePerDevice once;
  const int ready = once([] { return gf_allow_smem(gemm_f32_tile_kernel<TM, SPLIT>, smem); });
  if (ready) return ready;
  if (SPLIT) return launch_k_cluster(gemm_f32_tile_kernel<TM, SPLIT>, GF_PARTS, tiles * GF_PARTS, GF_TILE_THREADS, smem, stream, p);
  return launch_k(gemm_f32_tile_kernel<TM, SPLIT>, tiles, GF_TILE_THREADS, smem, stream, p);
}

}  // namespace

// 1 if the kernels of this file take the product, whatever M and N: rows of A and W in 16-byte pieces, and at least two stages
// in a run of K (below that nothing is on its way while a stage is multiplied, and such a product lasts as long as its launch
// on either side)
int gemm_f32_takes(const void* A, const void* W, int K, int lda, int ldw) {
  return (K >= 2 * GF_PARTS * GF_BK && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0) ? 1 : 0;
}

int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  const int n_sms = device_sms();
  if (n_sms <= 0) return IE_BAD_SIZE;
  GfParams p;
  p.A = A; p.W = W; p.C = C; p.M = M; p.N = N; p.K = K; p.lda = lda; p.ldw = ldw; p.ldc = ldc;
  p.part = (((K + GF_PARTS - 1) / GF_PARTS) + GF_BK - 1) / GF_BK * GF_BK;
  if (M <= 16) {
    // Many rows of weights: one block an SM walks over groups, its ring never empties.  Fewer: a cluster a group, so that
    // every SM has warps.
    const int groups = (N + 31) / 32;
    if (groups >= 4 * n_sms) {
      if (M <= 4) return launch_stream<2, 2, 5, 1>(p, n_sms, stream);
      if (M <= 8) return launch_stream<4, 4, 2, 1>(p, n_sms, stream);
      return launch_stream<2, 8, 3, 1>(p, n_sms, stream);
    }
    if (groups >= n_sms) {
      if (M <= 4) return launch_stream<2, 2, 5, 2>(p, 0, stream);
      if (M <= 8) return launch_stream<2, 4, 4, 2>(p, 0, stream);
      return launch_stream<2, 8, 4, 2>(p, 0, stream);
    }
    if (M <= 4) return launch_stream<2, 2, 8, 8>(p, 0, stream);
    if (M <= 8) return launch_stream<2, 4, 8, 8>(p, 0, stream);
    return launch_stream<2, 8, 6, 8>(p, 0, stream);
  }
  const bool low = M <= 32;
  const int bm = low ? 32 : 64;
  const long long tiles = (long long)((M + bm - 1) / bm) * ((N + GF_BN - 1) / GF_BN);
  if (tiles * GF_PARTS > 0x7fffffffLL) return IE_BAD_SIZE;
  // Two blocks an SM: below four tiles an SM the last round of tiles weighs too much, and the runs of K are spread instead
  // (640 tiles of 300 rows x 16,384: spread 591 us against 575; 80 tiles of 300 x 2,048 leave half the SMs idle unless spread)
  const bool split = tiles < 4LL * n_sms;
  if (low) return split ? launch_tile<4, true>(p, (int)tiles, stream) : launch_tile<4, false>(p, (int)tiles, stream);
  return split ? launch_tile<8, true>(p, (int)tiles, stream) : launch_tile<8, false>(p, (int)tiles, stream);
}
