// The gated delta rule: a recurrent mixer whose state is one DK x DV float32 matrix per (request, head).
//
// Per token and head, with the head's query q and key k (DK numbers; several heads may share one q/k head), its
// value v (DV numbers), a write strength beta = sigmoid(b_pre) and a decay g = exp(-exp(A_log) * softplus(a_pre +
// dt_bias)), both one number a head:
//     q <- q / sqrt(sum(q^2) + key_eps) * DK^-1/2,   k <- k / sqrt(sum(k^2) + key_eps)
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (o sees the token's own write)
// The head's o is divided by its root mean square over DV (norm_eps inside the root), multiplied by a gain of DV
// numbers that the heads share and by silu(gate), and written in the activation type for the output projection.
// Everything between the projections (q, k, v after their convolutions, b_pre, a_pre, gate) and that store is float32.
//
// DK and DV are compile-time constants (-DIE_GD_DK, -DIE_GD_DV): a library is built per pair when a model first asks.
// A block owns one (request, head).  Column j of S (value channel j) belongs to KS neighbouring threads, each with
// DK / KS of its rows in registers, so S^T k, the update and S^T q are sums inside a thread and a shuffle among
// those lanes.  The step's tokens of the request are walked in tiles of TT, whose q, k, v and gate are fetched into
// registers while the tile before is being run: (A) they go to shared memory as float32, a thread per token forms
// beta and g and a warp per token makes q and k unit vectors;
// (B) every thread runs the tile's tokens in order; (C) a warp per token norms and gates the outputs.  The order
// of every sum is fixed by the token and the channel alone, so this kernel's result does not depend on how the
// sequence was cut into steps or on what else the step holds.  A decode step is a tile of one token.  (The chunked form
// below sums in another order; the 32-bit path never takes it.)
#include <cfloat>
#include "common.cuh"

#if !defined(IE_GD_DK) || !defined(IE_GD_DV)
#error "gated_delta.cu is compiled per head size: -DIE_GD_DK=<key size> -DIE_GD_DV=<value size>"
#endif
#define GD_DK IE_GD_DK
#define GD_DV IE_GD_DV

constexpr int gd_pick_ks() {
  // the fewest lanes a column (1, 2, 4, 8) that leave a thread at most 32 rows; DK must split evenly
  for (int ks = 1; ks <= 8; ks *= 2)
    if (GD_DK % ks == 0 && GD_DK / ks <= 32 && GD_DV * ks <= 1024) return ks;
  for (int ks = 8; ks >= 1; ks /= 2)
    if (GD_DK % ks == 0 && GD_DV * ks <= 1024) return ks;
  return 1;
}
#define GD_KS (gd_pick_ks())
#define GD_DKP (GD_DK / GD_KS)                      // rows of a column in one thread
#define GD_THREADS (((GD_DV * GD_KS + 31) / 32) * 32)
#define GD_TT ((2 * GD_DK + 3 * GD_DV) <= 640 ? 16 : 8)
// the q and k vectors lie in shared memory part by part, each part GD_LD floats after the one before: the padding
// puts the parts that the KS lanes of a column read at once on different banks
#define GD_LD (GD_DKP + (GD_KS > 1 ? 4 : 0))
#define GD_ROW (GD_KS * GD_LD)
#define GD_VEC (GD_DKP % 4 == 0)

static_assert(GD_DK >= 1 && GD_DV >= 1 && GD_DV <= 1024, "value heads up to 1024 channels: one block a head");
static_assert(GD_DKP <= 128, "a thread keeps its rows of a state column in registers");
static_assert(GD_TT * (2 * GD_ROW + 3 * GD_DV + 3) * 4 <= 48 * 1024, "a tile's vectors must fit in shared memory");

struct GatedDeltaParams {
  const void* q;            // activation type, [N, *_stride]: columns of one buffer (after convolution and SiLU)
  const void* k;
  const void* v;
  int qk_stride, v_stride;
  const void* b_pre;        // activation type [N, ba_stride], one column a head
  const void* a_pre;
  int ba_stride;
  const void* gate;         // activation type [N, gate_stride], heads x DV
  int gate_stride;
  const void* a_log;        // weight type [H]
  const void* dt_bias;      // weight type [H]
  const void* out_gain;     // weight type [DV]
  float* state;             // [slots, H, DK, DV] float32
  void* out;                // activation type [N, out_stride]
  int out_stride;
  const int* q_start;       // [R + 1]
  const int* slots;         // [R], negative: a padding row without state
  int n_heads, n_kv_heads;
  float key_eps, norm_eps;
  int write_state;
};

// Loads of a tile's inputs that stay where they are written (volatile): they are issued before the tile ahead is run
// and used after it; left to itself the compiler moves them down to their use and the tile then waits for memory.
__device__ __forceinline__ float gd_ld_early(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float gd_ld_early(const bf16* p) {
  unsigned short v;
  asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return __uint_as_float((unsigned)v << 16);
}
#define GD_PQ ((GD_TT * GD_DK + GD_THREADS - 1) / GD_THREADS)   // elements of a tile's q (and k) a thread fetches
#define GD_PV ((GD_TT * GD_DV + GD_THREADS - 1) / GD_THREADS)   // of its v (and gate)

__device__ __forceinline__ int gd_place(int i) { return (i / GD_DKP) * GD_LD + (i % GD_DKP); }   // channel -> place
__device__ __forceinline__ float gd_column_sum(float v) {
#pragma unroll
  for (int o = 1; o < GD_KS; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename TA, typename TW>
__global__ void __launch_bounds__(GD_THREADS) gated_delta_kernel(GatedDeltaParams p) {
  __shared__ __align__(16) float sq[GD_TT][GD_ROW], sk[GD_TT][GD_ROW];
  __shared__ float sv[GD_TT][GD_DV], sg[GD_TT][GD_DV], so[GD_TT][GD_DV], sbeta[GD_TT], sdecay[GD_TT], sdecm1[GD_TT];
  pdl_trigger();
  pdl_wait();
  const int req = blockIdx.x, h = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int n_warps = GD_THREADS / 32;
  const int j = tid / GD_KS, part = tid - j * GD_KS;
  const bool active = j < GD_DV;
  const int row0 = part * GD_DKP, base = part * GD_LD;
  const int q0 = p.q_start[req], q1 = p.q_start[req + 1];
  const int slot = IE_SLOT(p.slots[req]);
  const int c = h / (p.n_heads / p.n_kv_heads);         // the q/k head this head reads
  TA* out = (TA*)p.out;
  if (slot < 0) {
    for (int idx = tid; idx < (q1 - q0) * GD_DV; idx += GD_THREADS)
      out[(size_t)(q0 + idx / GD_DV) * p.out_stride + h * GD_DV + idx % GD_DV] = from_f32<TA>(0.f);
    return;
  }
  const TA* Q = (const TA*)p.q + c * GD_DK;
  const TA* K = (const TA*)p.k + c * GD_DK;
  const TA* V = (const TA*)p.v + h * GD_DV;
  const TA* G = (const TA*)p.gate + h * GD_DV;
  const float rate = -expf(to_f32(((const TW*)p.a_log)[h]));
  const float dt_bias = to_f32(((const TW*)p.dt_bias)[h]);
  const TW* gain = (const TW*)p.out_gain;
  const float q_scale = rsqrtf((float)GD_DK);

  float S[GD_DKP];
  float* st = p.state + (((size_t)slot * p.n_heads + h) * GD_DK) * GD_DV;
#pragma unroll
  for (int i = 0; i < GD_DKP; ++i) S[i] = active ? st[(size_t)(row0 + i) * GD_DV + j] : 0.f;

  // a tile's inputs in registers, fetched while the tile ahead is being run
  float fq[GD_PQ], fk[GD_PQ], fv[GD_PV], fg[GD_PV];
  auto fetch = [&](int t0, int nt) {
#pragma unroll
    for (int u = 0; u < GD_PQ; ++u) {
      const int e = tid + u * GD_THREADS;
      const int tt = e / GD_DK, i = e - tt * GD_DK;
      if (tt < nt) {
        const size_t row = (size_t)(t0 + tt) * p.qk_stride + i;
        fq[u] = gd_ld_early(Q + row);
        fk[u] = gd_ld_early(K + row);
      }
    }
#pragma unroll
    for (int u = 0; u < GD_PV; ++u) {
      const int e = tid + u * GD_THREADS;
      const int tt = e / GD_DV, i = e - tt * GD_DV;
      if (tt < nt) {
        fv[u] = gd_ld_early(V + (size_t)(t0 + tt) * p.v_stride + i);
        fg[u] = gd_ld_early(G + (size_t)(t0 + tt) * p.gate_stride + i);
      }
    }
  };
  if (q0 < q1) fetch(q0, min(GD_TT, q1 - q0));

  for (int t0 = q0; t0 < q1; t0 += GD_TT) {
    const int nt = min(GD_TT, q1 - t0);
    // (A) the tile's vectors, the two numbers of every token, the unit vectors
#pragma unroll
    for (int u = 0; u < GD_PQ; ++u) {
      const int e = tid + u * GD_THREADS;
      const int tt = e / GD_DK, i = e - tt * GD_DK;
      if (tt < nt) {
        sq[tt][gd_place(i)] = fq[u];
        sk[tt][gd_place(i)] = fk[u];
      }
    }
#pragma unroll
    for (int u = 0; u < GD_PV; ++u) {
      const int e = tid + u * GD_THREADS;
      const int tt = e / GD_DV, i = e - tt * GD_DV;
      if (tt < nt) {
        sv[tt][i] = fv[u];
        sg[tt][i] = to_f32(gain[i]) * (fg[u] / (1.f + expf(-fg[u])));
      }
    }
    if (tid < nt) {
      const float b = to_f32(((const TA*)p.b_pre)[(size_t)(t0 + tid) * p.ba_stride + h]);
      const float a = to_f32(((const TA*)p.a_pre)[(size_t)(t0 + tid) * p.ba_stride + h]) + dt_bias;
      sbeta[tid] = 1.f / (1.f + expf(-b));
      // the decay, and the decay less one when it is above one half: a float32 decay of 1 - 2.5e-6 is off by up to a
      // hundredth of its distance from one, which a thousand tokens turn into the fifth digit of the state
      const float log_g = rate * (a > 20.f ? a : log1pf(expf(a)));
      sdecay[tid] = expf(log_g);
      sdecm1[tid] = log_g > -0.6931472f ? expm1f(log_g) : 0.f;
    }
    __syncthreads();
    for (int tt = warp; tt < nt; tt += n_warps) {
      float qq = 0.f, kk = 0.f;
      for (int i = lane; i < GD_DK; i += 32) {
        const float a = sq[tt][gd_place(i)], b = sk[tt][gd_place(i)];
        qq = fmaf(a, a, qq);
        kk = fmaf(b, b, kk);
      }
      const float qn = q_scale / sqrtf(warp_sum(qq) + p.key_eps), kn = 1.f / sqrtf(warp_sum(kk) + p.key_eps);
      for (int i = lane; i < GD_DK; i += 32) {
        sq[tt][gd_place(i)] *= qn;
        sk[tt][gd_place(i)] *= kn;
      }
    }
    __syncthreads();
    if (t0 + GD_TT < q1) fetch(t0 + GD_TT, min(GD_TT, q1 - t0 - GD_TT));     // lands while this tile runs
    // (B) the tile's tokens in order; this thread's rows of its column of the state
#pragma unroll 2
    for (int tt = 0; tt < nt; ++tt) {
      float kk[GD_DKP], qq[GD_DKP];
      if constexpr (GD_VEC) {
#pragma unroll
        for (int i = 0; i < GD_DKP; i += 4) {
          *reinterpret_cast<float4*>(&kk[i]) = *reinterpret_cast<const float4*>(&sk[tt][base + i]);
          *reinterpret_cast<float4*>(&qq[i]) = *reinterpret_cast<const float4*>(&sq[tt][base + i]);
        }
      } else {
#pragma unroll
        for (int i = 0; i < GD_DKP; ++i) {
          kk[i] = sk[tt][base + i];
          qq[i] = sq[tt][base + i];
        }
      }
      const float vj = active ? sv[tt][j] : 0.f;
      const float g = sdecay[tt], gm1 = sdecm1[tt], beta = sbeta[tt];
      float ks[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < GD_DKP; ++i) ks[i & 3] = fmaf(kk[i], S[i], ks[i & 3]);
      const float sk_old = gd_column_sum((ks[0] + ks[1]) + (ks[2] + ks[3]));
      float u;
      if (gm1 != 0.f) {                  // g S as S + (g - 1) S
        u = beta * (vj - fmaf(gm1, sk_old, sk_old));                                // (g S)^T k
#pragma unroll
        for (int i = 0; i < GD_DKP; ++i) S[i] = fmaf(kk[i], u, fmaf(gm1, S[i], S[i]));
      } else {
        u = beta * (vj - g * sk_old);
#pragma unroll
        for (int i = 0; i < GD_DKP; ++i) S[i] = fmaf(kk[i], u, g * S[i]);
      }
      float oo[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < GD_DKP; ++i) oo[i & 3] = fmaf(S[i], qq[i], oo[i & 3]);
      const float o = gd_column_sum((oo[0] + oo[1]) + (oo[2] + oo[3]));
      if (active && part == 0) so[tt][j] = o;
    }
    __syncthreads();
    // (C) norm over the head, gain, gate; a warp per token
    for (int tt = warp; tt < nt; tt += n_warps) {
      float ss = 0.f;
      for (int i = lane; i < GD_DV; i += 32) ss = fmaf(so[tt][i], so[tt][i], ss);
      const float rms = sqrtf(warp_sum(ss) / (float)GD_DV + p.norm_eps);
      for (int i = lane; i < GD_DV; i += 32)
        out[(size_t)(t0 + tt) * p.out_stride + h * GD_DV + i] = from_f32<TA>(so[tt][i] / rms * sg[tt][i]);
    }
    __syncthreads();
  }
  if (p.write_state && active) {
#pragma unroll
    for (int i = 0; i < GD_DKP; ++i) st[(size_t)(row0 + i) * GD_DV + j] = S[i];
  }
}

// ------------------------------------------------------------------------------------------ prompts, in chunks of tokens
// The kernel above is a chain: 2,048 tokens of one request took 1,713 us (0.84 us a token: two sums over the state and three
// trips through shared memory), on 32 of 148 SMs.  With the chunk's start state S0, L_t the sum (float64) of log g up to token
// t of the chunk, and (strictly lower) A[t][s] = beta_t exp(L_t - L_s) (k_t . k_s), the same recurrence reads
//     (I + A) U = diag(beta) V - diag(beta exp(L)) K S0        (row t of U is u_t)
//     o_t = exp(L_t) S0^T q_t + sum over s <= t of exp(L_t - L_s) (q_t . k_s) u_s
//     S_end = exp(L_end) S0 + sum over t of exp(L_end - L_t) k_t u_t^T
// so that all but two small products a chunk runs in parallel over chunks:
//   prepare  (block: chunk, head): unit vectors, the products k.k and q.k, and both right-hand sides solved against I + A by
//            forward substitution, a thread a column: Uv = (I + A)^-1 diag(beta) V and W = (I + A)^-1 diag(beta exp(L)) K
//   carry    (block: head, 16 value channels): chunk after chunk U = Uv - W S, S <- exp(L_end) S + Kd^T U, with the next
//            chunk's operands on their way; leaves S0 and U of every chunk
//   finish   (block: chunk, head): the outputs, their norm and gate
// All of it float32 products and sums; exponents are sums of log g, so a decay close to one keeps its digits
// (S + expm1(L_end) S).  Tokens beyond the request's last have beta = 0, log g = 0 and zero vectors.
// 2,048 tokens of 32 heads of 64: 1,221 us alone and 1,713 in a step token after token, 293 so
// (120 prepare, 85 carry, 69 finish).
#define GD_C 64
#define GD_CHUNKED (GD_DK % 16 == 0 && GD_DV % 16 == 0 && GD_DK >= 32 && GD_DK <= 128 && GD_DV >= 32 && GD_DV <= 128)
#if GD_CHUNKED

struct GatedDeltaChunks {
  GatedDeltaParams p;
  float* w;        // [slot, head][GD_C][DK]
  float* kd;       // [slot, head][DK][GD_C]   exp(L_end - L_t) k_t
  float* u;        // [slot, head][DV][GD_C]   Uv, then U
  float* qk;       // [slot, head][GD_C][GD_C] exp(L_t - L_s) (q_t . k_s), zero above the diagonal
  float* s0;       // [slot, head][DV][DK]
  float* tok;      // [slot, head][GD_C] what q_t is multiplied by, norm and exp(L_t) together; then [1] L_end
};
constexpr int GD_TOK = GD_C + 4;
constexpr int GD_CT = 256;                       // threads of the three kernels
constexpr int GD_PK = GD_DK + 4, GD_PC = GD_C + 4;   // row pitches in shared memory: 8 rows on 32 banks

// a request's chunk c lies at slot q0 / GD_C + req + c: requests follow one another in tokens, so slots never meet
__device__ __forceinline__ size_t gd_chunk(int q0, int req, int c, int h, int heads) {
  return (size_t)(q0 / GD_C + req + c) * heads + h;
}
constexpr float GD_LOG_FLOOR = -1e4f;
__device__ __forceinline__ float gd_log_decay(float rate, float a) { return rate * (a > 20.f ? a : log1pf(expf(a))); }

// acc[i][j] += sum over x of a[(r + 16 i)][x] b[(c + 16 j)][x], x in [x0, x1) (multiples of 4); four sums a thread run in order
template <int TM, int TN>
__device__ __forceinline__ void gd_product(float (&acc)[TM][TN], const float* a, int pa, const float* b, int pb, int x0, int x1,
                                           int a_step = 16, int b_step = 16) {
#pragma unroll 4
  for (int x = x0; x < x1; x += 4) {
    float4 av[TM], bv[TN];
#pragma unroll
    for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * a_step * pa + x);
#pragma unroll
    for (int j = 0; j < TN; ++j) bv[j] = *reinterpret_cast<const float4*>(b + j * b_step * pb + x);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        acc[i][j] = fmaf(av[i].x, bv[j].x, acc[i][j]);
        acc[i][j] = fmaf(av[i].y, bv[j].y, acc[i][j]);
        acc[i][j] = fmaf(av[i].z, bv[j].z, acc[i][j]);
        acc[i][j] = fmaf(av[i].w, bv[j].w, acc[i][j]);
      }
  }
}

template <typename TA, typename TW>
__global__ void __launch_bounds__(GD_CT, 2) gated_delta_prepare_kernel(GatedDeltaChunks d) {
  extern __shared__ __align__(16) float gd_smem[];
  float* const kn = gd_smem;                      // [GD_C][GD_PK] unit k
  float* const qn = kn + GD_C * GD_PK;            // [GD_C][GD_PK] unit q times DK^-1/2
  float* const at = qn + GD_C * GD_PK;            // [s][t] = A[t][s], pitch GD_PC
  __shared__ double sl[GD_C];                     // L_t: a difference of two keeps its digits however far the sum has run
  __shared__ float sbeta[GD_C], sqn[GD_C];
  const GatedDeltaParams& p = d.p;
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.y, req = blockIdx.z;
  const int q0 = p.q_start[req], q1 = p.q_start[req + 1];
  const int t0 = q0 + blockIdx.x * GD_C;
  if (t0 >= q1 || IE_SLOT(p.slots[req]) < 0) return;
  const int nt = min(GD_C, q1 - t0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = h / (p.n_heads / p.n_kv_heads);
  const TA* Q = (const TA*)p.q + c * GD_DK;
  const TA* K = (const TA*)p.k + c * GD_DK;
  const TA* V = (const TA*)p.v + h * GD_DV;
  const size_t slot = gd_chunk(q0, req, blockIdx.x, h, p.n_heads);

  if (warp == 0) {
    const float rate = -expf(to_f32(((const TW*)p.a_log)[h])), dt_bias = to_f32(((const TW*)p.dt_bias)[h]);
    double carry = 0.;
#pragma unroll
    for (int half = 0; half < GD_C / 32; ++half) {
      const int t = half * 32 + lane;
      double lg = 0.;
      float beta = 0.f;
      if (t < nt) {
        const float log_g = gd_log_decay(rate, to_f32(((const TA*)p.a_pre)[(size_t)(t0 + t) * p.ba_stride + h]) + dt_bias);
        // a log decay that overflowed would make differences of the sums NaN; from -104 down every exp is zero all the same
        lg = log_g < GD_LOG_FLOOR ? GD_LOG_FLOOR : log_g;
        beta = 1.f / (1.f + expf(-to_f32(((const TA*)p.b_pre)[(size_t)(t0 + t) * p.ba_stride + h])));
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, lg, o);
        if (lane >= o) lg += up;
      }
      lg += carry;
      sl[t] = lg;
      sbeta[t] = beta;
      carry = __shfl_sync(0xffffffffu, lg, 31);
    }
  }
  const float q_scale = rsqrtf((float)GD_DK);
  for (int t = warp; t < GD_C; t += GD_CT / 32) {
    constexpr int PER = (GD_DK + 31) / 32;
    float a[PER], b[PER], qq = 0.f, kk = 0.f;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = lane + 32 * u;
      const bool there = t < nt && i < GD_DK;
      a[u] = there ? to_f32(Q[(size_t)(t0 + t) * p.qk_stride + i]) : 0.f;
      b[u] = there ? to_f32(K[(size_t)(t0 + t) * p.qk_stride + i]) : 0.f;
      qq = fmaf(a[u], a[u], qq);
      kk = fmaf(b[u], b[u], kk);
    }
    const float fq = q_scale / sqrtf(warp_sum(qq) + p.key_eps), fk = 1.f / sqrtf(warp_sum(kk) + p.key_eps);
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = lane + 32 * u;
      if (i < GD_DK) {
        qn[t * GD_PK + i] = a[u] * fq;
        kn[t * GD_PK + i] = b[u] * fk;
      }
    }
    if (lane == 0) sqn[t] = fq;
  }
  __syncthreads();
  {
    const int r = tid >> 4, cc = tid & 15;       // rows t = r + 16 i, columns s = cc + 16 j
    float kk[4][4] = {}, qk[4][4] = {};
    gd_product<4, 4>(kk, kn + r * GD_PK, GD_PK, kn + cc * GD_PK, GD_PK, 0, GD_DK);
    gd_product<4, 4>(qk, qn + r * GD_PK, GD_PK, kn + cc * GD_PK, GD_PK, 0, GD_DK);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = r + 16 * i, s = cc + 16 * j;
        const float e = s <= t ? expf((float)(sl[t] - sl[s])) : 0.f;
        at[s * GD_PC + t] = s < t ? sbeta[t] * (e * kk[i][j]) : 0.f;
        d.qk[slot * (GD_C * GD_C) + t * GD_C + s] = s <= t ? e * qk[i][j] : 0.f;
      }
  }
  if (tid < GD_C) d.tok[slot * GD_TOK + tid] = sqn[tid] * expf((float)sl[tid]);
  if (tid == 0) d.tok[slot * GD_TOK + GD_C] = (float)sl[GD_C - 1];
  for (int idx = tid; idx < GD_C * GD_DK; idx += GD_CT) {
    const int i = idx / GD_C, t = idx % GD_C;
    d.kd[slot * (GD_C * GD_DK) + idx] = kn[t * GD_PK + i] * expf((float)(sl[GD_C - 1] - sl[t]));
  }
  __syncthreads();
  // a thread a column of the two right-hand sides
  for (int col = tid; col < GD_DV + GD_DK; col += GD_CT) {
    float x[GD_C];
    if (col < GD_DV) {
#pragma unroll
      for (int t = 0; t < GD_C; ++t) x[t] = t < nt ? to_f32(V[(size_t)(t0 + t) * p.v_stride + col]) : 0.f;
#pragma unroll
      for (int t = 0; t < GD_C; ++t) x[t] *= sbeta[t];
    } else {
#pragma unroll
      for (int t = 0; t < GD_C; ++t) x[t] = sbeta[t] * (expf((float)sl[t]) * kn[t * GD_PK + col - GD_DV]);
    }
#pragma unroll
    for (int s = 0; s < GD_C - 1; ++s) {
#pragma unroll
      for (int t4 = 0; t4 < GD_C; t4 += 4) {
        if (t4 + 3 <= s) continue;
        const float4 a = *reinterpret_cast<const float4*>(at + s * GD_PC + t4);
        if (t4 > s) x[t4] = fmaf(-a.x, x[s], x[t4]);
        if (t4 + 1 > s) x[t4 + 1] = fmaf(-a.y, x[s], x[t4 + 1]);
        if (t4 + 2 > s) x[t4 + 2] = fmaf(-a.z, x[s], x[t4 + 2]);
        if (t4 + 3 > s) x[t4 + 3] = fmaf(-a.w, x[s], x[t4 + 3]);
      }
    }
    if (col < GD_DV) {
      float4* dst = reinterpret_cast<float4*>(d.u + slot * (GD_C * GD_DV) + col * GD_C);
#pragma unroll
      for (int t = 0; t < GD_C; t += 4) dst[t / 4] = make_float4(x[t], x[t + 1], x[t + 2], x[t + 3]);
    } else {
#pragma unroll
      for (int t = 0; t < GD_C; ++t) d.w[slot * (GD_C * GD_DK) + t * GD_DK + col - GD_DV] = x[t];
    }
  }
}

__device__ __forceinline__ void gd_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

constexpr int GD_SLICE = 16;                      // value channels of a carry block
constexpr int GD_CARRY_STAGE = GD_C * GD_PK + GD_DK * GD_PC + GD_SLICE * GD_PC;

// Groups of 64 threads take an equal part of the inner length each (4 x 4 outputs a thread, 64 x 16 a group and pass).  A chunk is a
// chain of two short products and four barriers, so eight groups where DK allows (2,048 tokens of 32 heads: four groups 328 us
// for the three kernels, eight 293).
constexpr int GD_GROUPS = GD_DK % 32 == 0 ? 8 : 4;
constexpr int GD_CARRY_T = 64 * GD_GROUPS;
__global__ void __launch_bounds__(GD_CARRY_T) gated_delta_carry_kernel(GatedDeltaChunks d) {
  extern __shared__ __align__(16) float gd_smem[];
  float* const st = gd_smem + 2 * GD_CARRY_STAGE;             // [GD_SLICE][GD_PK] the state's columns
  float* const red = st + GD_SLICE * GD_PK;                   // [GD_GROUPS][64][GD_SLICE + 1]
  const GatedDeltaParams& p = d.p;
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.y, req = blockIdx.z, j0 = blockIdx.x * GD_SLICE;
  const int q0 = p.q_start[req], q1 = p.q_start[req + 1];
  const int slot_id = IE_SLOT(p.slots[req]);
  if (slot_id < 0 || q0 >= q1) return;
  const int tid = threadIdx.x;
  const int chunks = (q1 - q0 + GD_C - 1) / GD_C;
  float* const state = p.state + ((size_t)slot_id * p.n_heads + h) * GD_DK * GD_DV + j0;

  auto fetch = [&](int c) {
    if (c < chunks) {
      const size_t slot = gd_chunk(q0, req, c, h, p.n_heads);
      float* const w = gd_smem + (c & 1) * GD_CARRY_STAGE;
      float* const kd = w + GD_C * GD_PK;
      float* const u = kd + GD_DK * GD_PC;
      for (int i = tid; i < GD_C * GD_DK / 4; i += GD_CARRY_T) {
        gd_copy16(w + (i / (GD_DK / 4)) * GD_PK + (i % (GD_DK / 4)) * 4, d.w + slot * (GD_C * GD_DK) + i * 4);
        gd_copy16(kd + (i / (GD_C / 4)) * GD_PC + (i % (GD_C / 4)) * 4, d.kd + slot * (GD_C * GD_DK) + i * 4);
      }
      for (int i = tid; i < GD_SLICE * GD_C / 4; i += GD_CARRY_T)
        gd_copy16(u + (i / (GD_C / 4)) * GD_PC + (i % (GD_C / 4)) * 4, d.u + slot * (GD_C * GD_DV) + j0 * GD_C + i * 4);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);
  for (int i = tid; i < GD_DK * GD_SLICE; i += GD_CARRY_T)
    st[(i % GD_SLICE) * GD_PK + i / GD_SLICE] = state[(size_t)(i / GD_SLICE) * GD_DV + i % GD_SLICE];
  const int group = tid >> 6, r = (tid & 63) >> 2, jc = tid & 3;
  auto leave = [&](float (&acc)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) red[(group * 64 + r + 16 * i) * (GD_SLICE + 1) + jc + 4 * j] = acc[i][j];
  };
  auto total = [&](int row, int j) {
    const float* at = red + row * (GD_SLICE + 1) + j;
    constexpr int step = 64 * (GD_SLICE + 1);
    float v = (at[0] + at[step]) + (at[2 * step] + at[3 * step]);
    if (GD_GROUPS == 8) v += (at[4 * step] + at[5 * step]) + (at[6 * step] + at[7 * step]);
    return v;
  };
  for (int c = 0; c < chunks; ++c) {
    const size_t slot = gd_chunk(q0, req, c, h, p.n_heads);
    float* const w = gd_smem + (c & 1) * GD_CARRY_STAGE;
    float* const kd = w + GD_C * GD_PK;
    float* const u = kd + GD_DK * GD_PC;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                              // the chunk and the state are there, the other stage has been read
    fetch(c + 1);
    const float grow = expm1f(d.tok[slot * GD_TOK + GD_C]);
    // the start state, for the outputs
    for (int i = tid; i < GD_SLICE * GD_DK; i += GD_CARRY_T)
      d.s0[slot * (GD_DK * GD_DV) + j0 * GD_DK + i] = st[(i / GD_DK) * GD_PK + i % GD_DK];
    {
      float acc[4][4] = {};
      gd_product<4, 4>(acc, w + r * GD_PK, GD_PK, st + jc * GD_PK, GD_PK, group * (GD_DK / GD_GROUPS), (group + 1) * (GD_DK / GD_GROUPS), 16, 4);
      leave(acc);
    }
    __syncthreads();
    for (int i = tid; i < GD_SLICE * GD_C; i += GD_CARRY_T) {
      const int j = i / GD_C, t = i % GD_C;
      const float v = u[j * GD_PC + t] - total(t, j);
      u[j * GD_PC + t] = v;
      d.u[slot * (GD_C * GD_DV) + j0 * GD_C + i] = v;
    }
    __syncthreads();
#pragma unroll 1
    for (int i0 = 0; i0 < GD_DK; i0 += 64) {
      float acc[4][4] = {};
      // rows beyond DK (a size that 64 does not divide) read the rows that follow in shared memory and are dropped below
      gd_product<4, 4>(acc, kd + (i0 + r) * GD_PC, GD_PC, u + jc * GD_PC, GD_PC, group * (GD_C / GD_GROUPS), (group + 1) * (GD_C / GD_GROUPS), 16, 4);
      leave(acc);
      __syncthreads();
      for (int i = tid; i < GD_SLICE * 64; i += GD_CARRY_T) {
        const int j = i / 64, row = i % 64;
        if (i0 + row < GD_DK) {
          float* at = st + j * GD_PK + i0 + row;
          *at = fmaf(grow, *at, *at) + total(row, j);
        }
      }
      __syncthreads();
    }
  }
  if (p.write_state)
    for (int i = tid; i < GD_DK * GD_SLICE; i += GD_CARRY_T)
      state[(size_t)(i / GD_SLICE) * GD_DV + i % GD_SLICE] = st[(i % GD_SLICE) * GD_PK + i / GD_SLICE];
}

template <typename TA, typename TW>
__global__ void __launch_bounds__(GD_CT) gated_delta_finish_kernel(GatedDeltaChunks d) {
  extern __shared__ __align__(16) float gd_smem[];
  constexpr int TN = GD_DV / 16;
  float* const qs = gd_smem;                      // [GD_C][GD_PK] exp(L_t) q_t
  float* const s0 = qs + GD_C * GD_PK;            // [DV][GD_PK]
  float* const qk = s0 + GD_DV * GD_PK;           // [GD_C][GD_PC]
  float* const u = qk + GD_C * GD_PC;             // [DV][GD_PC]
  const GatedDeltaParams& p = d.p;
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.y, req = blockIdx.z;
  const int q0 = p.q_start[req], q1 = p.q_start[req + 1];
  const int t0 = q0 + blockIdx.x * GD_C;
  if (t0 >= q1) return;
  const int nt = min(GD_C, q1 - t0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  TA* out = (TA*)p.out;
  if (IE_SLOT(p.slots[req]) < 0) {
    for (int idx = tid; idx < nt * GD_DV; idx += GD_CT)
      out[(size_t)(t0 + idx / GD_DV) * p.out_stride + h * GD_DV + idx % GD_DV] = from_f32<TA>(0.f);
    return;
  }
  const size_t slot = gd_chunk(q0, req, blockIdx.x, h, p.n_heads);
  const TA* Q = (const TA*)p.q + (h / (p.n_heads / p.n_kv_heads)) * GD_DK;
  for (int i = tid; i < GD_DV * GD_DK / 4; i += GD_CT)
    gd_copy16(s0 + (i / (GD_DK / 4)) * GD_PK + (i % (GD_DK / 4)) * 4, d.s0 + slot * (GD_DK * GD_DV) + i * 4);
  for (int i = tid; i < GD_C * GD_C / 4; i += GD_CT)
    gd_copy16(qk + (i / (GD_C / 4)) * GD_PC + (i % (GD_C / 4)) * 4, d.qk + slot * (GD_C * GD_C) + i * 4);
  for (int i = tid; i < GD_DV * GD_C / 4; i += GD_CT)
    gd_copy16(u + (i / (GD_C / 4)) * GD_PC + (i % (GD_C / 4)) * 4, d.u + slot * (GD_C * GD_DV) + i * 4);
  asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll 8
  for (int idx = tid; idx < GD_C * GD_DK; idx += GD_CT) {
    const int t = idx / GD_DK, i = idx % GD_DK;
    qs[t * GD_PK + i] = t < nt ? to_f32(Q[(size_t)(t0 + t) * p.qk_stride + i]) * d.tok[slot * GD_TOK + t] : 0.f;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int r = tid >> 4, cc = tid & 15;
  float acc[4][TN];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  gd_product<4, TN>(acc, qs + r * GD_PK, GD_PK, s0 + cc * GD_PK, GD_PK, 0, GD_DK);
  // a token after t has weight zero for t, which hides it only while its u is a number: with an infinity or NaN in the chunk
  // the sum ends at t itself, so that a bad token spoils no earlier one
  bool bad = false;
  for (int i = tid; i < GD_DV * GD_C; i += GD_CT) bad |= !(fabsf(u[(i / GD_C) * GD_PC + i % GD_C]) <= FLT_MAX);
  if (__syncthreads_or(bad) == 0) {
    gd_product<4, TN>(acc, qk + r * GD_PC, GD_PC, u + cc * GD_PC, GD_PC, 0, GD_C);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
        for (int x = 0; x <= r + 16 * i; ++x) acc[i][j] = fmaf(qk[(r + 16 * i) * GD_PC + x], u[(cc + 16 * j) * GD_PC + x], acc[i][j]);
  }
  __syncthreads();
  float* const so = gd_smem;                      // [GD_C][GD_DV + 1], where the operands were (both products have read them)
  static_assert(GD_C * (GD_DV + 1) <= (GD_C + GD_DV) * (GD_PK + GD_PC), "the outputs take the place of the operands");
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) so[(r + 16 * i) * (GD_DV + 1) + cc + 16 * j] = acc[i][j];
  __syncthreads();
  const TA* G = (const TA*)p.gate + h * GD_DV;
  const TW* gain = (const TW*)p.out_gain;
  for (int t = warp; t < nt; t += GD_CT / 32) {
    float ss = 0.f;
    for (int i = lane; i < GD_DV; i += 32) ss = fmaf(so[t * (GD_DV + 1) + i], so[t * (GD_DV + 1) + i], ss);
    const float rms = sqrtf(warp_sum(ss) / (float)GD_DV + p.norm_eps);
    for (int i = lane; i < GD_DV; i += 32) {
      const float g = to_f32(G[(size_t)(t0 + t) * p.gate_stride + i]);
      out[(size_t)(t0 + t) * p.out_stride + h * GD_DV + i] =
          from_f32<TA>(so[t * (GD_DV + 1) + i] / rms * (to_f32(gain[i]) * (g / (1.f + expf(-g)))));
    }
  }
}

constexpr size_t GD_SLOT_FLOATS = (size_t)2 * GD_C * GD_DK + GD_C * GD_DV + GD_C * GD_C + GD_DK * GD_DV + GD_TOK;
constexpr size_t GD_PREPARE_SMEM = (size_t)(2 * GD_C * GD_PK + GD_C * GD_PC) * 4;
constexpr size_t GD_CARRY_SMEM = (size_t)(2 * GD_CARRY_STAGE + GD_SLICE * GD_PK + GD_GROUPS * 64 * (GD_SLICE + 1)) * 4;
constexpr size_t GD_FINISH_SMEM = (size_t)(GD_C * GD_PK + GD_DV * GD_PK + GD_C * GD_PC + GD_DV * GD_PC) * 4;

template <typename TA, typename TW>
static int gd_launch_chunks(const GatedDeltaChunks& d, int n_requests, int chunks, cudaStream_t stream) {
  static OncePerDevice once;
  const int ready = once([] {
    cudaError_t e = cudaFuncSetAttribute(gated_delta_prepare_kernel<TA, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GD_PREPARE_SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(gated_delta_carry_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GD_CARRY_SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(gated_delta_finish_kernel<TA, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GD_FINISH_SMEM);
    return e;
  });
  if (ready) return ready;
  const dim3 grid(chunks, d.p.n_heads, n_requests);
  int rc = launch_k(gated_delta_prepare_kernel<TA, TW>, grid, GD_CT, GD_PREPARE_SMEM, stream, d);
  if (!rc) rc = launch_k(gated_delta_carry_kernel, dim3(GD_DV / GD_SLICE, d.p.n_heads, n_requests), GD_CARRY_T, GD_CARRY_SMEM, stream, d);
  if (!rc) rc = launch_k(gated_delta_finish_kernel<TA, TW>, grid, GD_CT, GD_FINISH_SMEM, stream, d);
  return rc;
}
#endif  // GD_CHUNKED

// floats of scratch that the chunked form wants for a step of so many tokens and requests (0: this library has no such form)
extern "C" long long ie_gated_delta_scratch_floats(int n_tokens, int n_requests, int n_heads) {
#if GD_CHUNKED
  return (long long)(n_tokens / GD_C + n_requests + 1) * n_heads * (long long)GD_SLOT_FLOATS;
#else
  return 0;
#endif
}

extern "C" int ie_gated_delta_dims(int* dk, int* dv) {
  *dk = GD_DK;
  *dv = GD_DV;
  return IE_OK;
}

// scratch (16-byte aligned, ie_gated_delta_scratch_floats floats): the chunked form, for steps whose longest request brings
// max_q_len tokens of n_tokens in all; null: token after token.
extern "C" int ie_gated_delta(const void* q, const void* k, const void* v, int qk_stride, int v_stride,
                              const void* b_pre, const void* a_pre, int ba_stride, const void* gate, int gate_stride,
                              const void* a_log, const void* dt_bias, const void* out_gain, int w_dtype, float* state,
                              void* out, int out_stride, const int* q_start, const int* slots, int n_requests,
                              int n_heads, int n_kv_heads, int dk, int dv, float key_eps, float norm_eps,
                              int write_state, int act_dtype, float* scratch, int max_q_len, int n_tokens,
                              cudaStream_t stream) {
  if (n_requests <= 0 || n_heads <= 0) return IE_OK;
  if (dk != GD_DK || dv != GD_DV || n_kv_heads <= 0 || n_heads % n_kv_heads) return IE_BAD_SIZE;
  GatedDeltaParams p;
  p.q = q; p.k = k; p.v = v; p.qk_stride = qk_stride; p.v_stride = v_stride; p.b_pre = b_pre; p.a_pre = a_pre;
  p.ba_stride = ba_stride; p.gate = gate; p.gate_stride = gate_stride; p.a_log = a_log; p.dt_bias = dt_bias;
  p.out_gain = out_gain; p.state = state; p.out = out; p.out_stride = out_stride; p.q_start = q_start; p.slots = slots;
  p.n_heads = n_heads; p.n_kv_heads = n_kv_heads; p.key_eps = key_eps; p.norm_eps = norm_eps; p.write_state = write_state;
#if GD_CHUNKED
  if (scratch != nullptr) {
    if ((uintptr_t)scratch & 15) return IE_BAD_ALIGN;
    const int chunks = (max_q_len + GD_C - 1) / GD_C;
    if (chunks <= 0 || n_heads > 65535 || n_requests > 65535) return IE_BAD_SIZE;
    const size_t n = (size_t)(n_tokens / GD_C + n_requests + 1) * n_heads;
    GatedDeltaChunks d;
    d.p = p;
    d.w = scratch;
    d.kd = d.w + n * GD_C * GD_DK;
    d.u = d.kd + n * GD_C * GD_DK;
    d.qk = d.u + n * GD_C * GD_DV;
    d.s0 = d.qk + n * GD_C * GD_C;
    d.tok = d.s0 + n * GD_DK * GD_DV;
    if (act_dtype == IE_F32 && w_dtype == IE_F32) return gd_launch_chunks<float, float>(d, n_requests, chunks, stream);
    if (act_dtype == IE_F32 && w_dtype == IE_BF16) return gd_launch_chunks<float, bf16>(d, n_requests, chunks, stream);
    if (act_dtype == IE_BF16 && w_dtype == IE_F32) return gd_launch_chunks<bf16, float>(d, n_requests, chunks, stream);
    if (act_dtype == IE_BF16 && w_dtype == IE_BF16) return gd_launch_chunks<bf16, bf16>(d, n_requests, chunks, stream);
    return IE_BAD_DTYPE;
  }
#endif
  (void)scratch; (void)max_q_len; (void)n_tokens;
  dim3 grid(n_requests, n_heads);
  if (act_dtype == IE_F32 && w_dtype == IE_F32) return launch_k(gated_delta_kernel<float, float>, grid, GD_THREADS, 0, stream, p);
  if (act_dtype == IE_F32 && w_dtype == IE_BF16) return launch_k(gated_delta_kernel<float, bf16>, grid, GD_THREADS, 0, stream, p);
  if (act_dtype == IE_BF16 && w_dtype == IE_F32) return launch_k(gated_delta_kernel<bf16, float>, grid, GD_THREADS, 0, stream, p);
  if (act_dtype == IE_BF16 && w_dtype == IE_BF16) return launch_k(gated_delta_kernel<bf16, bf16>, grid, GD_THREADS, 0, stream, p);
  return IE_BAD_DTYPE;
}

IE_CHECK_API(gated_delta)
