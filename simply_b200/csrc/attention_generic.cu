// Ragged paged attention, general form: any head size, page size, grouping and
// storage type.  One block of four warps per (token, query head); keys are visited in
// tiles of 32 that start at a multiple of 32 of the absolute key position, tile number i
// by warp i mod 4, and the warps' parts are merged in warp order, so a token's result is
// the same whatever else the step holds.  A prompt's tokens come 2, 4 or 8 to a block, which share every
// key and value that is fetched; each of them adds up in the order it has alone.  A block's tokens belong to one
// request: where requests meet inside a group of 2, 4 or 8 tokens, each has a block of its own, and a token alone in its
// block is walked as blocks of one token walk it (a group walked request by request, 16 heads of 128, us by blocks
// of one token, so, and now: 31 requests of one token and 4,000 keys beside a prompt of 600 1,452, 6,550, 1,368, 7 of 2,000 beside 256 439, 2,296, 232).
//
//   s = q . k                 (q is already rotated and scaled)
//   s = cap * tanh(s / cap)   if cap > 0          simply/model_lib.py:621-626
//   keep k_pos <= q_pos and, with a window W, q_pos - k_pos < W
//                                                 simply/model_lib.py:469-515
//   p = softmax(s) in float32, o = p . v          simply/model_lib.py:633-637
//   query head n reads kv head n / (Hq / Hkv)     simply/model_lib.py:2306-2310
//
// Options beyond that (`sb_paged_attention_general`): value heads of another size than key heads
// (a page then holds all its key rows, then all its value rows), and pooled blocks: with a
// window W and blocks of P tokens, position i also sees, ahead of its window and under the same
// softmax, one key and value per block c with c*P + P - 1 <= i - W, read from a second paged
// storage that holds one entry per P tokens in the page of the block's first token.  Blocks
// are visited in tiles of 32 by block number, before the tokens.  `tied`: an entry has one row of
// head_dim numbers whose first v_dim are its value as well (a cache of latents; a page then holds
// key rows only).  `sink`: one learned number per query head whose exponential joins the softmax's
// denominator; it has no key and no value.  `distance`: two learned numbers r1, r2 per query head
// ([2, heads]); the score of query i and key j loses r1 * log(1 + r2 * (i - j)) (float32, log1pf);
// with `linear` one number r1 per head ([heads]), and the score loses r1 * (i - j).  `chunk` C (without
// a window): a query sees the keys from (i / C) * C on, its own chunk's.  `keep` n (with a window): the sequence's
// first n keys stay visible too.
//
// This is the true 32-bit path's attention and the fallback of the bfloat16
// path for shapes its tensor-core kernels refuse.
#include <float.h>

#include <type_traits>

#include "common.cuh"

#define GEN_WARPS 4
#define GEN_MAX_DPL 16  // dims per lane: head_dim <= 512

template <typename T> struct Vec16;  // 16-byte vector loads of storage type T
template <> struct Vec16<float> {
  static constexpr int N = 4;
  __device__ static void load(const float* p, float* out) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  }
};
template <> struct Vec16<bf16> {
  static constexpr int N = 8;
  __device__ static void load(const bf16* p, float* out) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      out[2 * i] = __uint_as_float(w[i] << 16);
      out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};

// One tile of up to 32 keys, one per lane: scores, the running softmax, and the values' sum, for R queries.
// `kr` / `vr` are this lane's key and value rows (null where no query sees a key of this lane), `sees` has bit r set where
// query r sees it; query r's numbers stand in `qs` at r * head_dim.
template <typename KT, int R, int DPL>
__device__ __forceinline__ void gen_tile(const KT* kr, const KT* vr, unsigned sees, const float* qs, int head_dim, int v_dim,
                                         float cap, float minus, int lane, float* m_run, float* l_run, float (*acc)[DPL]) {
  constexpr int VN = Vec16<KT>::N;
  const float NEG = -0.5f * FLT_MAX;  // the reference's mask value, simply/utils/common.py:543-551
  float dot[R], p[R];
#pragma unroll
  for (int r = 0; r < R; ++r) dot[r] = 0.f;
  if (kr != nullptr) {
    int d = 0;
    if ((head_dim % VN) == 0) {
      for (; d < head_dim; d += VN) {
        float kf[VN];
        Vec16<KT>::load(kr + d, kf);
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int e = 0; e < VN; e += 4) {
            const float4 qf = *reinterpret_cast<const float4*>(qs + r * head_dim + d + e);
            dot[r] = fmaf(qf.x, kf[e], dot[r]);
            dot[r] = fmaf(qf.y, kf[e + 1], dot[r]);
            dot[r] = fmaf(qf.z, kf[e + 2], dot[r]);
            dot[r] = fmaf(qf.w, kf[e + 3], dot[r]);
          }
      }
    } else {
      for (; d < head_dim; ++d) {
        const float kf = to_f32<KT>(kr[d]);
#pragma unroll
        for (int r = 0; r < R; ++r) dot[r] = fmaf(qs[r * head_dim + d], kf, dot[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool valid = (sees >> r) & 1u;
    const float s = valid ? (cap > 0.f ? cap * tanhf(dot[r] / cap) : dot[r]) - minus : NEG;
    const float m_new = fmaxf(m_run[r], warp_max(s));
    const float alpha = expf(m_run[r] - m_new);
    p[r] = valid ? expf(s - m_new) : 0.f;
    l_run[r] = l_run[r] * alpha + warp_sum(p[r]);
    m_run[r] = m_new;
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[r][i] *= alpha;
  }
  const unsigned valid_mask = __ballot_sync(0xffffffffu, sees != 0);
  // Four keys at a time: their values are fetched together, then added in the keys' order (eight
  // at a time cost registers and were slower).  (A query adds nothing for a key that it does not see: p is 0 there,
  // and only what some query sees is read.)
  constexpr int KEYS = 4;
  for (int j0 = 0; j0 < 32; j0 += KEYS) {
    const unsigned four = (valid_mask >> j0) & ((1u << KEYS) - 1u);  // uniform over the warp
    if (!four) continue;
    const KT* vj[KEYS];
    float pj[R][KEYS];
    unsigned seen[KEYS];
#pragma unroll
    for (int u = 0; u < KEYS; ++u) {
      vj[u] = reinterpret_cast<const KT*>(__shfl_sync(0xffffffffu, (unsigned long long)vr, j0 + u));
      seen[u] = R > 1 ? __shfl_sync(0xffffffffu, sees, j0 + u) : (four >> u) & 1u;
#pragma unroll
      for (int r = 0; r < R; ++r) pj[r][u] = __shfl_sync(0xffffffffu, p[r], j0 + u);
    }
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
      const int d = lane + 32 * i;
      if (d < v_dim) {
        float x[KEYS];
#pragma unroll
        for (int u = 0; u < KEYS; ++u) x[u] = ((four >> u) & 1u) ? to_f32<KT>(vj[u][d]) : 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int u = 0; u < KEYS; ++u)
            if ((seen[u] >> r) & 1u) acc[r][i] = fmaf(pj[r][u], x[u], acc[r][i]);
      }
    }
  }
}

// R > 1: without pooled blocks, distances and kept first keys.  Its blocks: (a request but the first, query head), for the
// request's first tokens where those lie inside a group of R tokens, then (group of R tokens, query head), for the
// first request of the group: every run of one request's tokens within a group once.
template <typename T, int R, int DPL>
__global__ void __launch_bounds__(GEN_WARPS * 32)
paged_attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ cache,
                               const int* __restrict__ block_table, int max_pages,
                               const int* __restrict__ token_seq, const int* __restrict__ positions,
                               const int* __restrict__ cu_q, int num_seqs,
                               T* __restrict__ out, int num_tokens, int num_q_heads, int num_kv_heads,
                               int head_dim, int v_dim, int page_size, int num_pages, float cap, int window,
                               const T* __restrict__ pool, const int* __restrict__ pool_table,
                               int pool_max_pages, int pool_len, int pool_pages, int tied,
                               const float* __restrict__ sink, const float* __restrict__ distance, int linear,
                               int chunk, int keep, int* err) {
  const float r1 = distance != nullptr ? distance[blockIdx.x % num_q_heads] : 0.f;  // (weights: before the wait)
  const float r2 = distance != nullptr && !linear ? distance[num_q_heads + blockIdx.x % num_q_heads] : 0.f;
  pdl_wait_block();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x % num_q_heads;
  const int m = n / (num_q_heads / num_kv_heads);
  int t = blockIdx.x / num_q_heads, count = 1;
  if (R > 1) {
    const int others = num_seqs - 1, s = t + 1;
    if (t < others) {
      t = cu_q[s];
      if (t < 0 || t >= num_tokens || t % R == 0 || token_seq[t] != s) return;  // (a group's first token, or no new token)
    } else {
      t = (t - others) * R;
    }
    const int end = min(t / R * R + R, num_tokens);
    while (t + count < end && token_seq[t + count] == token_seq[t]) ++count;
  }
  const int b = token_seq[t];
  // The block's `count` tokens from t on, at most N; N * head_dim floats of q, then per query and warp its running
  // maximum, sum and v_dim partial results.
  extern __shared__ __align__(16) float smem[];
  auto attend = [&](auto most) {
    constexpr int N = decltype(most)::value;
    float* qs = smem;
    float* part = smem + N * head_dim;
    int pos[N], lo[N];
    int pos_all = 0, lo_all = 0;  // the highest and the lowest key that one of them sees
#pragma unroll
    for (int r = 0; r < N; ++r) {
      pos[r] = r < count ? positions[t + r] : -1;
      lo[r] = window > 0 ? max(pos[r] - window + 1, 0) : chunk > 0 ? max(pos[r], 0) / chunk * chunk : 0;
      if (r == 0 || (r < count && pos[r] > pos_all)) pos_all = pos[r];
      if (r == 0 || (r < count && lo[r] < lo_all)) lo_all = lo[r];
    }
#pragma unroll
    for (int r = 0; r < N; ++r) {
      const T* qp = q + ((size_t)(t + min(r, count - 1)) * num_q_heads + n) * head_dim;
      for (int d = threadIdx.x; d < head_dim; d += blockDim.x) qs[r * head_dim + d] = to_f32<T>(qp[d]);
    }
    __syncthreads();

    float m_run[N], l_run[N], acc[N][DPL];
#pragma unroll
    for (int r = 0; r < N; ++r) {
      m_run[r] = -0.5f * FLT_MAX;
      l_run[r] = 0.f;
#pragma unroll
      for (int i = 0; i < DPL; ++i) acc[r][i] = 0.f;
    }

    if (R == 1 && pool != nullptr && window > 0 && pool_len > 0) {
      // Blocks that lie wholly before the window: c * P + P - 1 <= pos - window.
      const int num_blocks = pos[0] - window + 1 > 0 ? (pos[0] - window + 1) / pool_len : 0;
      const int entries = (page_size + pool_len - 1) / pool_len;
      const size_t page_stride = (size_t)num_kv_heads * entries * (head_dim + v_dim);
      for (int tile = 32 * warp; tile < num_blocks; tile += 32 * GEN_WARPS) {  // tile i belongs to warp i % 4
        const int c = tile + lane;
        const T* kr = nullptr;
        const T* vr = nullptr;
        if (c < num_blocks) {
          const long long start = (long long)c * pool_len;
          const long long page = pool_table[(size_t)b * pool_max_pages + start / page_size];
          if (page < 0 || page >= pool_pages) {
            atomicOr(err, SB_ERR_BAD_PAGE);
          } else {
            const size_t row = (size_t)m * entries + (start % page_size) / pool_len;
            kr = pool + page * page_stride + row * head_dim;
            vr = pool + page * page_stride + (size_t)num_kv_heads * entries * head_dim + row * v_dim;
          }
        }
        gen_tile<T, N, DPL>(kr, vr, kr != nullptr, qs, head_dim, v_dim, cap, 0.f, lane, m_run, l_run, acc);
      }
    }

    const size_t page_stride = (size_t)num_kv_heads * page_size * (tied ? head_dim : head_dim + v_dim);
    const size_t value_base = (size_t)num_kv_heads * page_size * head_dim;
    // Tiles of kept first keys, then the tiles from the one that holds the lowest other key on.
    const int tile_lo = (lo_all / 32) * 32;
    for (int tile = keep > 0 ? 0 : tile_lo; tile <= pos_all; tile += 32) {
      if (tile < tile_lo && tile >= keep) tile = tile_lo;
      if (((tile >> 5) & (GEN_WARPS - 1)) != warp) continue;  // by the tile's absolute number
      const int j = tile + lane;
      const T* kr = nullptr;
      const T* vr = nullptr;
      unsigned sees = 0;
#pragma unroll
      for (int r = 0; r < N; ++r) sees |= (j >= lo[r] || j < keep) && j <= pos[r] ? 1u << r : 0u;
      if (sees) {
        const long long page = block_table[(size_t)b * max_pages + j / page_size];
        if (page < 0 || page >= num_pages) {
          atomicOr(err, SB_ERR_BAD_PAGE);
          sees = 0;
        } else {
          const size_t row = (size_t)m * page_size + j % page_size;
          kr = cache + page * page_stride + row * head_dim;
          vr = tied ? kr : cache + page * page_stride + value_base + row * v_dim;
        }
      }
      float minus = 0.f;
      if (R == 1 && distance != nullptr && j <= pos[0])
        minus = r1 * (linear ? (float)(pos[0] - j) : log1pf(r2 * (float)(pos[0] - j)));
      gen_tile<T, N, DPL>(kr, vr, sees, qs, head_dim, v_dim, cap, minus, lane, m_run, l_run, acc);
    }
    // The warps' parts meet in warp order (the same order whatever the step holds).
    const int stride = v_dim + 2;
#pragma unroll
    for (int r = 0; r < N; ++r) {
      float* mine = part + (size_t)(r * GEN_WARPS + warp) * stride;
      if (lane == 0) {
        mine[0] = m_run[r];
        mine[1] = l_run[r];
      }
#pragma unroll
      for (int i = 0; i < DPL; ++i) {
        const int d = lane + 32 * i;
        if (d < v_dim) mine[2 + d] = acc[r][i];
      }
    }
    __syncthreads();
    for (int r = warp; r < count; r += GEN_WARPS) {
      const float* parts = part + (size_t)r * GEN_WARPS * stride;
      float m_all = parts[0];
#pragma unroll
      for (int w = 1; w < GEN_WARPS; ++w) m_all = fmaxf(m_all, parts[(size_t)w * stride]);
      if (sink != nullptr) m_all = fmaxf(m_all, sink[n]);
      float scale[GEN_WARPS], l_all = 0.f;
#pragma unroll
      for (int w = 0; w < GEN_WARPS; ++w) {
        scale[w] = expf(parts[(size_t)w * stride] - m_all);
        l_all += parts[(size_t)w * stride + 1] * scale[w];
      }
      if (sink != nullptr) l_all += expf(sink[n] - m_all);
      T* op = out + ((size_t)(t + r) * num_q_heads + n) * v_dim;
      const float inv = 1.0f / l_all;
      for (int d = lane; d < v_dim; d += 32) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < GEN_WARPS; ++w) sum += parts[(size_t)w * stride + 2 + d] * scale[w];
        op[d] = from_f32<T>(sum * inv);
      }
    }
  };
  if (R == 1) {
    // (One turn.  Written as a loop: as straight code nvcc 12.9 fetches the values one by one here, 600 tokens of 16
    // heads of 128 864 us in place of 688, in bfloat16 1,057 in place of 562.)
    for (const int end = min(t + 1, num_tokens); t < end; ++t) {
      __syncthreads();
      attend(std::integral_constant<int, 1>{});
    }
  } else if (count == 1) {
    attend(std::integral_constant<int, 1>{});
  } else {
    attend(std::integral_constant<int, R>{});
  }
}

extern "C" int sb_paged_attention_general(const void* q, int dtype, const void* cache, const int* block_table,
                                          int max_pages, const int* token_seq, const int* positions,
                                          void* out, int num_tokens, int num_q_heads, int num_kv_heads,
                                          int head_dim, int v_dim, int page_size, int num_pages, float cap,
                                          int window, const void* pool, const int* pool_table,
                                          int pool_max_pages, int pool_len, int pool_pages, int tied,
                                          const float* sink, const float* distance, int linear, int chunk,
                                          int keep, const int* cu_q, int num_seqs, int together, int* err,
                                          cudaStream_t stream) {
  if (num_tokens == 0) return 0;
  if (distance != nullptr && pool != nullptr) return -13;
  if (chunk > 0 && (pool != nullptr || window > 0)) return -13;
  if (keep < 0 || (keep > 0 && (window <= 0 || pool != nullptr || tied))) return -13;
  if (tied && (pool != nullptr || v_dim > head_dim)) return -13;
  // (the values' sums live in registers, GEN_MAX_DPL per lane; a key row only passes through)
  if (head_dim <= 0 || head_dim > 4096 || v_dim <= 0 || v_dim > 32 * GEN_MAX_DPL) return -7;
  if (num_kv_heads <= 0 || num_q_heads % num_kv_heads) return -8;
  if (pool != nullptr || distance != nullptr || keep > 0 || dtype != SB_DTYPE_F32 || v_dim > 256) together = 1;
  if (v_dim > 128) together = min(together, 4);
  const int rows = together >= 8 ? 8 : together >= 4 ? 4 : together >= 2 ? 2 : 1;
  const long long items = ((long long)((num_tokens + rows - 1) / rows) + (rows > 1 ? num_seqs - 1 : 0)) * num_q_heads;
  if (items > 0x7fffffffLL) return -6;
  const unsigned blocks = (unsigned)items;
  const size_t smem = rows * ((size_t)head_dim + (size_t)GEN_WARPS * (v_dim + 2)) * sizeof(float);
#define SB_GENERIC(T_, R_, DPL_)                                                                                        \
  do {                                                                                                                  \
    auto kernel = paged_attention_generic_kernel<T_, R_, DPL_>;                                                         \
    if (smem > 48 * 1024) {                                                                                             \
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);       \
      if (e != cudaSuccess) return (int)e;                                                                              \
    }                                                                                                                   \
    sb_launch(kernel, blocks, GEN_WARPS * 32, smem, stream, (const T_*)q, (const T_*)cache, block_table, max_pages,     \
              token_seq, positions, cu_q, num_seqs, (T_*)out, num_tokens, num_q_heads, num_kv_heads, head_dim, v_dim,    \
              page_size, num_pages, cap, window, (const T_*)pool, pool_table, pool_max_pages, pool_len, pool_pages, tied, sink,    \
              distance, linear, chunk, keep, err);                                                                      \
  } while (0)
  if (dtype != SB_DTYPE_F32) SB_GENERIC(bf16, 1, GEN_MAX_DPL);
  else if (rows == 1) SB_GENERIC(float, 1, GEN_MAX_DPL);
  else if (v_dim > 128) { if (rows == 4) SB_GENERIC(float, 4, 8); else SB_GENERIC(float, 2, 8); }
  else if (rows == 8) SB_GENERIC(float, 8, 4);
  else if (rows == 4) SB_GENERIC(float, 4, 4);
  else SB_GENERIC(float, 2, 4);
#undef SB_GENERIC
  SB_LAUNCH_CHECK();
  return 0;
}

extern "C" int sb_paged_attention_generic(const void* q, int dtype, const void* cache, const int* block_table,
                                          int max_pages, const int* token_seq, const int* positions,
                                          void* out, int num_tokens, int num_q_heads, int num_kv_heads,
                                          int head_dim, int page_size, int num_pages, float cap, int window,
                                          const int* cu_q, int num_seqs, int together, int* err, cudaStream_t stream) {
  return sb_paged_attention_general(q, dtype, cache, block_table, max_pages, token_seq, positions, out, num_tokens,
                                    num_q_heads, num_kv_heads, head_dim, head_dim, page_size, num_pages, cap,
                                    window, nullptr, nullptr, 0, 0, 0, 0, nullptr, nullptr, 0, 0, 0, cu_q,
                                    num_seqs, together, err, stream);
}
