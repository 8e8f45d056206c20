// The launches of a step through all layers of a plain pre-norm decoder (engine/llama_block.py:50-62), issued from here.
// Kernels, their order and their operands are those that the parts issue one by one; what this spares is the host's work around
// each launch.  A prompt of 61 tokens is 148 launches that keep the GPU busy for 1,040 us and took the host 2,030 us from Python
// (14 us a launch, 9 of them for a library product); from here 1,060.
//
// The kernels of other libraries and the library product come in as function pointers (they live in shared objects of their own).
#include "common.cuh"

extern "C" int ie_rmsnorm(float* residual, const void* delta, const void* gain, int gain_dtype, void* out, int act_dtype,
                          const int* row_index, int n_rows, int d, float eps, cudaStream_t stream);
extern "C" int ie_rope_kv_write(void* q, const void* k, const void* v, int q_stride, int kv_stride, const float* cos_t,
                                const float* sin_t, const int* positions, const int* slot_mapping, void* kpool, void* vpool,
                                int n_tokens, int n_heads, int n_kv_heads, int hd, int page_size, int write_kv, int act_dtype,
                                cudaStream_t stream);
extern "C" int ie_silu_mul(const void* in, void* out, int n_rows, int inter, int in_stride, int interleaved, int act_dtype,
                           cudaStream_t stream);

// one layer: all of it fixed once the model and its cache exist
struct IeLayer {
  const void *norm1, *qkv_w, *o_w, *norm2, *gate_up_w, *down_w;
  void *kpool, *vpool;
  float eps1, eps2;
  int gain1_dtype, gain2_dtype;
};

// the step: sizes, the buffers that the layers share, and how its requests attend
struct IeLayersStep {
  // cublasGemmEx: bfloat16 operands, float32 sums
  int (*gemm_ex)(void*, int, int, int, int, int, const void*, const void*, int, int, const void*, int, int, const void*, void*, int,
                 int, int, int);
  void* handle;
  int (*gemm_silu)(const void*, const void*, void*, int, int, int, int, int, int, int, int, int, int, float, float, float, float,
                   cudaStream_t);                          // null: the library product and silu_mul
  int (*attn_small)(const void*, void*, const void*, const void*, const int*, const int*, const int*, float*, int, int, int, int, int,
                    int, int, int, int, int, float, int, int, cudaStream_t);                       // null: no such requests
  int (*attn_tc)(const void*, void*, const void*, const void*, const int*, const int*, const int*, const int*, const int*, int, int,
                 int, int, int, int, int, int, int, float, const float*, const float*, const int*, cudaStream_t);
  int (*attn_mma)(const void*, void*, const void*, const void*, const int*, const int*, const int*, const int*, const int*, int, int,
                  int, int, int, int, int, int, int, float, int, cudaStream_t);
  float* residual;
  void *delta, *normed, *qkv, *attn_out, *mixer_out, *gate_up, *hidden, *ff_out;
  const float *cos_t, *sin_t;
  const int *positions, *slot_mapping, *block_table, *q_start, *ctx_before, *work_req, *work_pair0;
  float* scratch;
  int n, width, n_heads, n_kv_heads, hd, inter, page_size, table_stride, n_requests, n_pages, window, n_work, n_splits, split_keys,
      rotate_q, n_sms, mma_rows;
  float scale;
};

extern "C" int ie_prenorm_layers_sizes(int* layer, int* step) {
  *layer = (int)sizeof(IeLayer);
  *step = (int)sizeof(IeLayersStep);
  return IE_OK;
}

// `*launches` counts this package's kernels; the last layer's delta (`ff_out`) is not added to the residual
extern "C" int ie_prenorm_layers(const IeLayer* layers, int n_layers, const IeLayersStep* step, int* launches, cudaStream_t stream) {
  const IeLayersStep& s = *step;
  const float one = 1.f, zero = 0.f;
  int count = 0, rc = 0;
  const int qw = s.n_heads * s.hd, kw = s.n_kv_heads * s.hd, rows = qw + 2 * kw;
  // out [n, cols] = x [n, k] w [cols, k]^T: column-major w^T x of the library (CUDA_R_16BF 14, CUBLAS_COMPUTE_32F 68, operation T 1,
  // the default tensor-core heuristic 99)
  auto product = [&](const void* x, const void* w, void* out, int cols, int k) {
    if (rc) return;
    rc = s.gemm_ex(s.handle, 1, 0, cols, s.n, k, &one, w, 14, k, x, 14, k, &zero, out, 14, cols, 68, 99);
    if (rc) rc += 10000;                                   // a status of the library, not of CUDA
  };
  auto launched = [&](int status) {
    if (!rc) rc = status;
    ++count;
  };
  const void* delta = s.delta;
  for (int i = 0; i < n_layers && !rc; ++i) {
    const IeLayer& L = layers[i];
    launched(ie_rmsnorm(s.residual, delta, L.norm1, L.gain1_dtype, s.normed, IE_BF16, nullptr, s.n, s.width, L.eps1, stream));
    product(s.normed, L.qkv_w, s.qkv, rows, s.width);
    bf16* const q = (bf16*)s.qkv;
    if (!rc)
      launched(ie_rope_kv_write(q, q + qw, q + qw + kw, rows, rows, s.cos_t, s.sin_t, s.positions, s.slot_mapping, L.kpool, L.vpool, s.n,
                                s.n_heads, s.n_kv_heads, s.hd, s.page_size, 1 | (s.rotate_q ? 0 : 2), IE_BF16, stream));
    if (!rc && s.attn_small)
      launched(s.attn_small(q, s.attn_out, L.kpool, L.vpool, s.block_table, s.q_start, s.ctx_before, s.scratch, rows, qw, s.table_stride,
                            s.n_requests, s.n, s.n_heads, s.n_kv_heads, s.hd, s.page_size, s.window, s.scale, s.n_splits, s.split_keys,
                            stream));
    if (!rc && s.attn_tc)
      launched(s.attn_tc(q, s.attn_out, L.kpool, L.vpool, s.block_table, s.q_start, s.ctx_before, s.work_req, s.work_pair0, rows, qw,
                         s.table_stride, s.n_work, s.n_heads, s.n_kv_heads, s.hd, s.page_size, s.n_pages, s.scale,
                         s.rotate_q ? nullptr : s.cos_t, s.rotate_q ? nullptr : s.sin_t, s.rotate_q ? nullptr : s.positions, stream));
    if (!rc && s.attn_mma)
      launched(s.attn_mma(q, s.attn_out, L.kpool, L.vpool, s.block_table, s.q_start, s.ctx_before, s.work_req, s.work_pair0, rows, qw,
                          s.table_stride, s.n_work, s.n_heads, s.n_kv_heads, s.hd, s.page_size, s.window, s.scale, s.mma_rows, stream));
    product(s.attn_out, L.o_w, s.mixer_out, s.width, qw);
    if (!rc)
      launched(ie_rmsnorm(s.residual, s.mixer_out, L.norm2, L.gain2_dtype, s.normed, IE_BF16, nullptr, s.n, s.width, L.eps2, stream));
    if (s.gemm_silu) {
      if (!rc)
        launched(s.gemm_silu(s.normed, L.gate_up_w, s.hidden, s.n, 2 * s.inter, s.width, s.width, s.width, s.inter, 3, 256, s.n_sms, 0,
                             1.f, 0.f, 0.f, 0.f, stream));
    } else {
      product(s.normed, L.gate_up_w, s.gate_up, 2 * s.inter, s.width);
      if (!rc) launched(ie_silu_mul(s.gate_up, s.hidden, s.n, s.inter, 2 * s.inter, 1, IE_BF16, stream));
    }
    product(s.hidden, L.down_w, s.ff_out, s.width, s.inter);
    delta = s.ff_out;
  }
  *launches = count;
  return rc;
}
