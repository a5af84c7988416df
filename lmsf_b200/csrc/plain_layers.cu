// The layer loop of a plain pre-norm decoder (norm, attention, norm, gated feed-forward; bfloat16, no biases) for steps with
// more rows than the weight-streaming products take, launched by one call.
//
// What bounds short prompts is the host: the same launches made one by one from Python cost 15 to 20 us each, nine a layer, and
// the device waits for them (a prompt of 77 tokens of the 1B shape: 2.45 ms for 1.11 ms of kernels).  From here its 144 launches take
// the host 0.56 ms, 3.9 us each, the library's among them.  Host code only: the kernels are the other files' entry points, handed over as addresses, and the library's product is
// called with the handle that torch uses on the stream, with the arguments torch.mm gives it, so results are the same to the bit.
// Nothing is kept between calls: weights, caches and buffers are named anew by each.
#include <cublas_v2.h>

#include "common.cuh"

LMSF_DEFINE_LAST_ERROR(lmsf_plain_layers)

namespace {

typedef int (*NormFn)(void*, const void*, float*, const void*, int, int, float, int, int, int, void*);
typedef int (*RopeFn)(void*, const void*, const void*, long long, long long, long long, const int*, const int*, const int*, int, int,
                      void*, long long, const float*, int, int, int, int, int, int, int, int*, void*);
typedef int (*ActFn)(void*, const void*, int, int, long long, int, int, void*);
typedef int (*DecodeFn)(const void*, long long, void*, long long, const void*, long long, int, int, const int*, int, const int*, int,
                        int, const int*, const int*, float, int, int, int, int, int, void*, int, int, const float*, const float*,
                        const float*, int, int, const float*, const float*, int, float, void*);
typedef int (*PrefillFn)(const void*, long long, long long, void*, long long, const void*, long long, long long, int, int, const int*,
                         int, const int*, const int*, int, const int*, const int*, float, int, int, int, int*, int, int, const float*,
                         const float*, const float*, int, int, const float*, const float*, int, float, void*);
typedef int (*GatedFn)(void*, long long, const void*, long long, const void*, int, int, int, int, int*, void*);
typedef cublasStatus_t (*GemmFn)(cublasHandle_t, cublasOperation_t, cublasOperation_t, int, int, int, const void*, const void*,
                                 cudaDataType, int, const void*, cudaDataType, int, const void*, void*, cudaDataType, int,
                                 cublasComputeType_t, cublasGemmAlgo_t);
typedef cublasStatus_t (*GetModeFn)(cublasHandle_t, cublasMath_t*);
typedef cublasStatus_t (*SetModeFn)(cublasHandle_t, cublasMath_t);

}  // namespace

struct PlainStep {
  // entry points
  void *norm, *rope, *act, *decode, *prefill, *gated, *gemm, *get_mode, *set_mode, *handle, *stream;
  // buffers: x bfloat16 [tokens][hidden] what enters the first layer, y like it the pending branch (out: the last layer's), res
  // float32 of its shape, h like x, qkv, att [tokens][q width], gu [tokens][2 ff] (null: gate, up and activation are one kernel, gemm_gated_tc.cu),
  // m [tokens][ff]
  void *x, *y, *res, *h, *qkv, *att, *gu, *m;
  // the step's tables
  const int *positions, *token_seq, *block_table, *cu_q, *ctx_len, *decode_seq_ids, *tile_seq, *tile_q0;
  int* error_flag;
  void* scratch;
  long long page_stride, n_pages;
  int tokens, hidden, n_q_heads, n_kv_heads, head_dim, ff, max_blocks, block_size, n_decode, n_tiles, act_code, n_layers, n_seqs, splits, warps, pad;
};
struct PlainLayer {
  const void *norm1, *qkv, *o, *norm2, *gate_up, *down;
  void* cache;
  const float* inv_freq;
  int norm1_dtype, norm2_dtype, rot_dim, is_neox;
  float eps1, eps2, scale;
  int pad;
};

LMSF_API long long lmsf_plain_step_bytes() { return (long long)sizeof(PlainStep); }
LMSF_API long long lmsf_plain_layer_bytes() { return (long long)sizeof(PlainLayer); }

// Returns the launches made (the library's not among them), or minus the stage that failed, with its answer in *rc.
LMSF_API int lmsf_plain_layers_run(const PlainStep* sp, const PlainLayer* layers, int* rc) {
  const PlainStep& s = *sp;
  const auto handle = (cublasHandle_t)s.handle;
  const int T = s.tokens, D = s.hidden, q_size = s.n_q_heads * s.head_dim, kv_size = s.n_kv_heads * s.head_dim;
  const int qkv_w = q_size + 2 * kv_size;
  int launches = 0, stage = 0;
  *rc = 0;
  cublasMath_t mode = CUBLAS_DEFAULT_MATH;
  if (((GetModeFn)s.get_mode)(handle, &mode) != CUBLAS_STATUS_SUCCESS ||
      ((SetModeFn)s.set_mode)(handle, (cublasMath_t)(CUBLAS_DEFAULT_MATH | CUBLAS_MATH_DISALLOW_REDUCED_PRECISION_REDUCTION)) != CUBLAS_STATUS_SUCCESS) {
    *rc = 1;
    return -1;
  }
  // y [T][n] = in [T][k] w [n][k]^T, products added up in float32
  auto product = [&](void* y, const void* in, const void* w, int n, int k) {
    const float one = 1.f, zero = 0.f;
    *rc = (int)((GemmFn)s.gemm)(handle, CUBLAS_OP_T, CUBLAS_OP_N, n, T, k, &one, w, CUDA_R_16BF, k, in, CUDA_R_16BF, k, &zero, y,
                                CUDA_R_16BF, n, CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP);
    return *rc == 0;
  };
  auto ran = [&](int answer) {
    *rc = answer;
    ++launches;
    return answer == 0;
  };
  for (int i = 0; i < s.n_layers; ++i) {
    const PlainLayer& l = layers[i];
    unsigned char* qkv = (unsigned char*)s.qkv;
    stage = 2;
    if (!ran(((NormFn)s.norm)(s.h, i == 0 ? s.x : s.y, (float*)s.res, l.norm1, T, D, l.eps1, i == 0 ? 1 : 2, LMSF_BF16, l.norm1_dtype, s.stream))) break;
    stage = 1;
    if (!product(s.qkv, s.h, l.qkv, qkv_w, D)) break;
    stage = 3;
    if (!ran(((RopeFn)s.rope)(qkv, qkv + 2 * (size_t)q_size, qkv + 2 * (size_t)(q_size + kv_size), qkv_w, qkv_w, qkv_w, s.positions, s.token_seq,
                              s.block_table, s.max_blocks, s.block_size, l.cache, s.page_stride, l.inv_freq, l.rot_dim, l.is_neox, T,
                              s.n_q_heads, s.n_kv_heads, s.head_dim, LMSF_BF16, s.error_flag, s.stream))) break;
    if (s.n_decode > 0) {
      stage = 4;
      if (!ran(((DecodeFn)s.decode)(qkv, qkv_w, s.att, q_size, l.cache, s.page_stride, s.block_size, s.n_kv_heads, s.block_table, s.max_blocks,
                                    s.decode_seq_ids, s.n_decode, s.n_seqs, s.cu_q, s.ctx_len, l.scale, 0, s.n_q_heads, s.head_dim, s.splits,
                                    s.warps, s.scratch, 2, 0, nullptr, nullptr, nullptr, 0, 0, nullptr, nullptr, 0, 0.f, s.stream))) break;
    }
    if (s.n_tiles > 0) {
      stage = 5;
      if (!ran(((PrefillFn)s.prefill)(qkv, qkv_w, T, s.att, q_size, l.cache, s.page_stride, s.n_pages, s.block_size, s.n_kv_heads, s.block_table,
                                      s.max_blocks, s.tile_seq, s.tile_q0, s.n_tiles, s.cu_q, s.ctx_len, l.scale, 0, s.n_q_heads, s.head_dim,
                                      s.error_flag, 2, 0, nullptr, nullptr, nullptr, 0, 0, nullptr, nullptr, 0, 0.f, s.stream))) break;
    }
    stage = 1;
    if (!product(s.y, s.att, l.o, D, q_size)) break;
    stage = 2;
    if (!ran(((NormFn)s.norm)(s.h, s.y, (float*)s.res, l.norm2, T, D, l.eps2, 2, LMSF_BF16, l.norm2_dtype, s.stream))) break;
    if (!s.gu) {
      stage = 7;
      if (!ran(((GatedFn)s.gated)(s.m, s.ff, s.h, D, l.gate_up, T, s.ff, D, s.act_code, s.error_flag, s.stream))) break;
    } else {
      stage = 1;
      if (!product(s.gu, s.h, l.gate_up, 2 * s.ff, D)) break;
      stage = 6;
      if (!ran(((ActFn)s.act)(s.m, s.gu, T, s.ff, 2ll * s.ff, s.act_code, LMSF_BF16, s.stream))) break;
    }
    stage = 1;
    if (!product(s.y, s.m, l.down, D, s.ff)) break;
    stage = 0;
  }
  ((SetModeFn)s.set_mode)(handle, mode);
  return *rc ? -stage : launches;
}
