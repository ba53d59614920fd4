// The layers of a step in one call from the host: for a run of layers of one shape (sandwich or pre-norm blocks of paged
// attention and a gated feed-forward, bfloat16) the same launches, in the same order and by the same rules, as the
// parts make one by one (kernels/ops.py).  A launch from Python costs the host about 13 us, a quarter of which is the
// launch: the 186 of a Gemma 2 2B step of 13 tokens took 2.4 ms to issue and 1.65 to run.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

extern "C" {
int sb_residual_norm(float*, const void*, const void*, int, const void*, int, float, int, const void*, int, float, int, const int*,
                     void*, int, int, int, int*, cudaStream_t);
int sb_qkv_rope_skinny(const void*, const void*, int, int, const float*, const float*, float, void*, void*, const int*, int,
                       const int*, const int*, int, int, int, int, int, int*, int, cudaStream_t);
int sb_qkv_rope_stream_tc(const void*, const void*, int, int, const float*, const float*, float, void*, void*, const int*, int,
                          const int*, const int*, int, int, int, int, int, int*, int, int, cudaStream_t);
int sb_rope_cache_write(const void*, int, const float*, const float*, float, void*, void*, const int*, int, const int*,
                        const int*, int, int, int, int, int, int, int, int*, cudaStream_t);
int sb_gemm_skinny_bf16(const void*, const void*, void*, int, int, int, int, float, int, int, cudaStream_t);
int sb_gemm_stream_tc(const void*, const void*, void*, int, int, int, int, float, int, int, int, int*, cudaStream_t);
int sb_gemm_gated_tc(const void*, const void*, void*, int, int, int, int, float, int, int, int*, cudaStream_t);
int sb_gated_activation(const void*, int, void*, int, int, int, float, cudaStream_t);
int sb_gemm_library_bf16(const void*, const void*, void*, int, int, int, int, void*, long long, cudaStream_t);
}

// The host's mirrors of these structs are in kernels/layer_run.py.
struct SbRunLayer {
  const void *w_qkv, *w_o, *w_gate_up, *w_down;
  const void *pre_mixer, *post_mixer, *pre_ff, *post_ff;  // norm scales; no post norms: null
  void* cache;
  const int* block_table;
  const float *cos_t, *sin_t;
  const void* tensor_map;
  long long num_pages, max_pages, kind;  // kind: index of the layer's attention
};

typedef int (*SbPrefill)(const void*, const void*, const int*, int, const int*, const int*, void*, int, int, int, int, int, float,
                         int, const int*, int, int*, cudaStream_t);
typedef int (*SbDecode)(const void*, const void*, const int*, int, const int*, const int*, const int*, void*, int, int, int, int,
                        int, float, int, const int*, int, int, float*, float*, int*, int, const int*, const int*, int,
                        const void*, int, const float*, int, const float*, int, int, int*, cudaStream_t);

struct SbRunAttention {
  const int *prefill_items, *decode_items, *split_start, *split_count;
  float *part_o, *part_ml;
  int num_prefill, num_decode, chunk, rows_max, window, unused;
};

struct SbRunStep {
  const int *token_seq, *positions, *cu_q, *q_start;
  float* h;
  void *y, *qkv, *q, *attended, *mixed, *gate_up, *z, *down;
  void* library_workspace;
  long long library_bytes;
  int *work_counter, *err;
  SbPrefill prefill;
  SbDecode decode;
  int tokens, width, hidden, num_q_heads, num_kv_heads, head_dim, page_size, activation;
  int scales_f32, plus_one, older_keys_settled;
  int few_rows, mid_qkv, mid_gated, mid_plain, gated_tc_rows;  // the kernel table's lines between kernels
  float limit, q_scale, cap, eps;
};

// Bytes of a layer, an attention and a step, for the host's mirrors.
extern "C" int sb_layer_run_bytes(int which) {
  return (int)(which == 0 ? sizeof(SbRunLayer) : which == 1 ? sizeof(SbRunAttention) : sizeof(SbRunStep));
}

// A product that the library has no algorithm for: the caller runs it (layer, 0 qkv, 1 output, 2 gate and up, 3 down).
typedef int (*SbOtherProduct)(int, int);

// Returns 0 or a status; `launches` counts the kernels.
extern "C" int sb_layer_run(const SbRunLayer* layers, int count, const SbRunAttention* attentions, const SbRunStep* step,
                            SbOtherProduct other, int* launches, cudaStream_t stream) {
  const SbRunStep& s = *step;
  const int T = s.tokens, W = s.width, group_dim = s.num_q_heads * s.head_dim;
  const int qkv_rows = (s.num_q_heads + 2 * s.num_kv_heads) * s.head_dim;
  int done = 0;
#define SB_RUN(call)                \
  do {                              \
    const int rc_ = (call);         \
    if (rc_) {                      \
      *launches = done;             \
      return rc_;                   \
    }                               \
    ++done;                         \
  } while (0)
  auto library = [&](const void* x, const void* w, void* out, int n, int k, int layer, int which) {
    const int rc = sb_gemm_library_bf16(x, w, out, T, n, k, 0, s.library_workspace, s.library_bytes, stream);
    return rc == -9 ? other(layer, which) : rc;
  };
  auto linear = [&](const void* x, const void* w, void* out, int n, int k, int layer, int which) {
    int rc = -9;
    if (T <= s.few_rows) rc = sb_gemm_skinny_bf16(x, w, out, T, n, k, 0, 0.f, 0, 0, stream);
    else if (T <= s.mid_plain) rc = sb_gemm_stream_tc(x, w, out, T, n, k, 0, 0.f, 0, 0, 0, s.err, stream);
    return rc == -9 ? library(x, w, out, n, k, layer, which) : rc;
  };
  const void* branch = nullptr;
  const void* post = nullptr;
  for (int i = 0; i < count; ++i) {
    const SbRunLayer& l = layers[i];
    const SbRunAttention& a = attentions[l.kind];
    const int pages = (int)l.num_pages, table = (int)l.max_pages;
    SB_RUN(sb_residual_norm(s.h, branch, nullptr, SB_DTYPE_BF16, post, s.scales_f32, s.eps, s.plus_one, l.pre_mixer, s.scales_f32,
                            s.eps, s.plus_one, nullptr, s.y, T, W, T, s.err, stream));
    int rc = -9;
    if (T <= s.few_rows && s.head_dim % 32 == 0)
      rc = sb_qkv_rope_skinny(s.y, l.w_qkv, T, W, l.cos_t, l.sin_t, s.q_scale, s.q, l.cache, l.block_table, table, s.token_seq,
                              s.positions, s.num_q_heads, s.num_kv_heads, s.head_dim, s.page_size, pages, s.err, 0, stream);
    else if (T > s.few_rows && T <= s.mid_qkv && s.head_dim % 128 == 0)
      rc = sb_qkv_rope_stream_tc(s.y, l.w_qkv, T, W, l.cos_t, l.sin_t, s.q_scale, s.q, l.cache, l.block_table, table, s.token_seq,
                                 s.positions, s.num_q_heads, s.num_kv_heads, s.head_dim, s.page_size, pages, s.err, 0, 0, stream);
    if (rc != -9) {
      SB_RUN(rc);
    } else {
      SB_RUN(linear(s.y, l.w_qkv, s.qkv, qkv_rows, W, i, 0));
      SB_RUN(sb_rope_cache_write(s.qkv, SB_DTYPE_BF16, l.cos_t, l.sin_t, s.q_scale, s.q, l.cache, l.block_table, table,
                                 s.token_seq, s.positions, T, s.num_q_heads, s.num_kv_heads, s.head_dim, s.page_size, pages, 1,
                                 s.err, stream));
    }
    if (a.num_prefill)
      SB_RUN(s.prefill(s.q, l.cache, l.block_table, table, s.cu_q, s.q_start, s.attended, T, s.num_q_heads, s.num_kv_heads,
                       s.page_size, pages, s.cap, a.window, a.prefill_items, a.num_prefill, s.err, stream));
    if (a.num_decode) {
      SB_RUN(s.decode(s.q, l.cache, l.block_table, table, s.cu_q, s.q_start, s.token_seq, s.attended, T, s.num_q_heads,
                      s.num_kv_heads, s.page_size, pages, s.cap, a.window, a.decode_items, a.num_decode, a.chunk, a.part_o,
                      a.part_ml, s.work_counter, a.rows_max, a.split_start, a.split_count, 0, l.tensor_map,
                      s.older_keys_settled, nullptr, 0, nullptr, 0, 0, s.err, stream));
      ++done;  // (and the merge)
    }
    SB_RUN(linear(s.attended, l.w_o, s.mixed, W, group_dim, i, 1));
    SB_RUN(sb_residual_norm(s.h, s.mixed, nullptr, SB_DTYPE_BF16, l.post_mixer, s.scales_f32, s.eps, s.plus_one, l.pre_ff,
                            s.scales_f32, s.eps, s.plus_one, nullptr, s.y, T, W, T, s.err, stream));
    rc = -9;
    if (T <= s.few_rows)
      rc = sb_gemm_skinny_bf16(s.y, l.w_gate_up, s.z, T, 2 * s.hidden, W, 2, s.limit, s.activation, 0, stream);
    else if (T <= s.mid_gated)
      rc = sb_gemm_stream_tc(s.y, l.w_gate_up, s.z, T, 2 * s.hidden, W, 2, s.limit, s.activation, 0, 0, s.err, stream);
    if (rc == -9 && s.gated_tc_rows > 0 && T >= s.gated_tc_rows)
      rc = sb_gemm_gated_tc(s.y, l.w_gate_up, s.z, T, s.hidden, W, s.activation, s.limit, 0, 1, s.err, stream);
    if (rc != -9) {
      SB_RUN(rc);
    } else {
      SB_RUN(linear(s.y, l.w_gate_up, s.gate_up, 2 * s.hidden, W, i, 2));
      SB_RUN(sb_gated_activation(s.gate_up, SB_DTYPE_BF16, s.z, T, s.hidden, s.activation, s.limit, stream));
    }
    SB_RUN(linear(s.z, l.w_down, s.down, W, s.hidden, i, 3));
    branch = s.down;
    post = l.post_ff;
  }
#undef SB_RUN
  *launches = done;
  return 0;
}
