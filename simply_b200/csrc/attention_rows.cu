// Decode attention over the paged cache for single tokens and few keys (bfloat16 in, float32 arithmetic): one launch,
// no work list, compiled once per head size (-DSB_HEAD_DIM=N; head sizes 64, 128 and 256).
//
//   s = q . k, s = cap tanh(s / cap) if cap > 0, keep the window's keys, o = softmax(s) . v, as attention_mma.cu
//
// With a few hundred keys per request the split-key kernel of attention_mma.cu is bound by what comes one after the
// other: work items from a counter, a tile by TMA, matrix products, partial results through memory, a second launch
// that merges them.  Here a cluster of 1 to 16 blocks owns one (request, kv head).  A warp takes tiles of 4 keys (8 or 16
// of smaller heads): a lane copies 16 bytes of each key row and value row for itself alone, so that nothing but
// its own copies has to be waited for, two tiles ahead and the first ones before the kernel waits for its
// queries (tiles below the new token's are older than the step).  Scores are sums over lanes; weights stay in 32 bits.
// The warps' results meet in shared memory, the blocks' through the cluster's.
//
// Bound by latency, and where a block walks many keys by its instructions (about 280 per tile and warp).  Decode steps of
// Gemma 2 2B, us, the split-key kernel and this one: 1 request of 200 keys 1,493 and 1,372, 1,000 1,530 and 1,470,
// 4,000 1,614 and 1,570; 8 of 300 1,686 and 1,573, of 900 1,690 and 1,657; 32 of 300 2,566 and 2,320.  The line to
// the split-key kernel: attention_cluster in kernels/choices.py.  Tried: K and V in registers instead of the ring
// (1,000 keys 1,514: the second tile's trip is not hidden), 8 warps a block (1,517), 3 stages (as 2).
#include <math.h>

#include <atomic>

#include "common.cuh"
#include "tma_mbar.cuh"

#ifndef SB_HEAD_DIM
#define SB_HEAD_DIM 256
#endif

#define SB_CAT2(a, b) a##b
#define SB_CAT(a, b) SB_CAT2(a, b)
#define SB_FN(name) SB_CAT(name##_hd, SB_HEAD_DIM)

namespace {

constexpr int DH = SB_HEAD_DIM;
constexpr bool TAKES = DH == 64 || DH == 128 || DH == 256;
constexpr int WARPS = 16;
constexpr int LD = 4;      // copies per lane and tile, of keys and of values
constexpr int STAGES = 2;  // tiles on their way per warp: 128 KB a block
constexpr int RING_BYTES = STAGES * 2 * LD * WARPS * 32 * 16;
constexpr int MAX_CLUSTER = 16;
[[maybe_unused]] constexpr float LOG2E = 1.4426950408889634f;

struct RowsParams {
  const bf16* q;      // [B, Hq, DH]
  const bf16* cache;  // [P, 2, Hkv, page, DH]
  const int* block_table;
  const int* q_start;  // [B]: the new token's position
  bf16* out;           // [B, Hq * DH]
  int max_pages, num_kv_heads, page_shift, num_pages, window, older_keys_settled;
  float cap;
  int* err;
};

[[maybe_unused]] __device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
[[maybe_unused]] __device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
[[maybe_unused]] __device__ __forceinline__ float from_block(const float* mine, uint32_t rank) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(sbx::mapa_shared(sbx::smem_u32(mine), rank)) : "memory");
  return v;
}
[[maybe_unused]] __device__ __forceinline__ void unpack8(const uint4& v, float2 (&f)[4]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}
// Two FMAs in one instruction.
[[maybe_unused]] __device__ __forceinline__ void fma_pair(float2& acc, float2 a, float2 b) {
  unsigned long long* c = reinterpret_cast<unsigned long long*>(&acc);
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(*c)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
}

// G: query heads per kv head.
template <int G>
__global__ void __launch_bounds__(WARPS * 32, 1) attn_rows_kernel(const RowsParams p) {
  constexpr int LPK = DH / 8, KPI = 32 / LPK;  // lanes per key, keys per load of a warp
  constexpr int TK = LD * KPI;                 // keys per tile
  __shared__ float s_m[WARPS][G], s_l[WARPS][G];
  __shared__ float b_o[G * DH], b_m[G], b_l[G];  // the block's own result, which the cluster reads
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t size, rank;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(size));
  rank = sbx::cluster_ctarank();
  const int pair = blockIdx.x / size, b = pair / p.num_kv_heads, m = pair - b * p.num_kv_heads;
  const int qs = p.q_start[b], hi = qs + 1, lo = p.window > 0 ? max(hi - p.window, 0) : 0;
  const int tile0 = lo / TK, tiles = (hi - 1) / TK - tile0 + 1;
  const int step = (int)size * WARPS;
  const int chunk = (lane % LPK) * 8, sub = lane / LPK;
  const int page_size = 1 << p.page_shift;
  const size_t v_offset = (size_t)p.num_kv_heads * page_size * DH;
  extern __shared__ __align__(16) uint4 ring[];  // [STAGES][keys, values][LD][threads]
  float (*s_o)[G][DH] = reinterpret_cast<float (*)[G][DH]>(ring);  // [WARPS], once all tiles have been read
  static_assert(WARPS * 4 * DH * (int)sizeof(float) <= RING_BYTES, "the warps' results take the ring's place");
  auto place = [&](int stage, int value, int u) { return ring + (((stage * 2 + value) * LD + u) * (WARPS * 32)) + threadIdx.x; };
  const int* table = p.block_table + (size_t)b * p.max_pages;
  // (a tile lies in one page)
  auto page_of = [&](int tile) { return tile < tiles ? table[((tile0 + tile) * TK) >> p.page_shift] : 0; };
  auto copy = [&](int tile, int page, int stage) {
    const bool held = page >= 0 && page < p.num_pages;
    if (!held) atomicOr(p.err, SB_ERR_BAD_PAGE);
    const bf16* rows = p.cache + ((size_t)(held ? page : 0) * 2 * p.num_kv_heads + m) * page_size * DH + chunk;
#pragma unroll
    for (int u = 0; u < LD; ++u) {
      // (a tile's keys beyond the visible ones bring a visible one in their place, and count for nothing below)
      const int j = min(max((tile0 + tile) * TK + u * KPI + sub, lo), hi - 1) & (page_size - 1);
      const bf16* from = rows + (size_t)j * DH;
#pragma unroll
      for (int value = 0; value < 2; ++value)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sbx::smem_u32(place(stage, value, u))),
                     "l"(from + value * v_offset), "r"(held ? 16 : 0)
                     : "memory");
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;\n" ::: "memory"); };
  int tile = warp * (int)size + (int)rank;
  int pages[STAGES];
#pragma unroll
  for (int i = 0; i < STAGES; ++i) pages[i] = page_of(tile + i * step);
  int ahead = 0;  // tiles copied so far (only a request's last tile holds what this step writes: a warp's last one)
#pragma unroll
  for (int i = 0; i < STAGES; ++i)
    if (p.older_keys_settled && ahead == i && tile + i * step < tiles && (tile0 + tile + i * step + 1) * TK <= qs) {
      copy(tile + i * step, pages[i], i);
      commit();
      ahead = i + 1;
    }
  pdl_wait_block();
  pdl_launch_dependents();
#pragma unroll
  for (int i = 0; i < STAGES; ++i)
    if (i >= ahead) {
      if (tile + i * step < tiles) copy(tile + i * step, pages[i], i);
      commit();
    }
  int next_page = page_of(tile + STAGES * step);
  float2 q[G][4];
#pragma unroll
  for (int g = 0; g < G; ++g)
    unpack8(*reinterpret_cast<const uint4*>(p.q + ((size_t)(b * p.num_kv_heads + m) * G + g) * DH + chunk), q[g]);
  float2 o[G][4];
  float m_run[G], l_run[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m_run[g] = -INFINITY;
    l_run[g] = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) o[g][e] = make_float2(0.f, 0.f);
  }
  // The sums over a key's lanes: VALUES numbers (place u * G + g: key u, head g) are halved between two halves of the
  // lanes as long as a lane has more than one, so that a score is capped by one lane (two of a head of 64) and
  // then given to all.
  constexpr int VALUES = LD * G, HELD = VALUES > LPK ? VALUES / LPK : 1;
  int held = 0;  // the first place this lane ends up with
#pragma unroll
  for (int off = LPK / 2, n = VALUES / 2; off > 0 && n >= HELD && n > 0; off >>= 1, n >>= 1) held += lane & off ? n : 0;
  const float inv_cap = p.cap > 0.f ? 1.0f / p.cap : 0.f;
  for (int stage = 0; tile < tiles; tile += step, stage = stage + 1 == STAGES ? 0 : stage + 1) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 1) : "memory");
    uint4 k[LD], v[LD];
#pragma unroll
    for (int u = 0; u < LD; ++u) {
      k[u] = *place(stage, 0, u);
      v[u] = *place(stage, 1, u);
    }
    if (tile + STAGES * step < tiles) copy(tile + STAGES * step, next_page, stage);
    commit();
    next_page = page_of(tile + (STAGES + 1) * step);
    float s[VALUES];
#pragma unroll
    for (int u = 0; u < LD; ++u) {
      float2 f[4];
      unpack8(k[u], f);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float2 a = make_float2(0.f, 0.f);
#pragma unroll
        for (int e = 0; e < 4; ++e) fma_pair(a, q[g][e], f[e]);
        s[u * G + g] = a.x + a.y;
      }
    }
#pragma unroll
    for (int off = LPK / 2, n = VALUES / 2; off > 0; off >>= 1, n >>= 1) {
      if (n > 0) {
        const bool upper = lane & off;
#pragma unroll
        for (int i = 0; i < VALUES / 2; ++i)
          if (i < n) {
            const float mine = upper ? s[i + n] : s[i], other = upper ? s[i] : s[i + n];
            s[i] = mine + __shfl_xor_sync(0xffffffffu, other, off);
          }
      } else {
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], off);
      }
    }
    float x[HELD];
#pragma unroll
    for (int i = 0; i < HELD; ++i) {
      const int j = (tile0 + tile) * TK + (held + i) / G * KPI + sub;
      x[i] = p.cap > 0.f ? p.cap * tanh_fast(s[i] * inv_cap) : s[i];
      x[i] = j >= lo && j < hi ? x[i] * LOG2E : -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < VALUES; ++i) {
      int from = 0;
#pragma unroll
      for (int off = LPK / 2, n = VALUES / 2; off > 0 && n >= HELD && n > 0; off >>= 1, n >>= 1) from |= i & n ? off : 0;
      s[i] = __shfl_sync(0xffffffffu, x[i % HELD], sub * LPK + from);
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float mx = m_run[g];
#pragma unroll
      for (int u = 0; u < LD; ++u) mx = fmaxf(mx, s[u * G + g]);
      const float use = mx == -INFINITY ? 0.f : mx, keep = exp2_fast(m_run[g] - use);
      m_run[g] = mx;
      l_run[g] *= keep;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[g][e].x *= keep;
        o[g][e].y *= keep;
      }
#pragma unroll
      for (int u = 0; u < LD; ++u) {
        s[u * G + g] = exp2_fast(s[u * G + g] - use);
        l_run[g] += s[u * G + g];
      }
    }
#pragma unroll
    for (int u = 0; u < LD; ++u) {
      float2 f[4];
      unpack8(v[u], f);
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) fma_pair(o[g][e], make_float2(s[u * G + g], s[u * G + g]), f[e]);
    }
  }
  __syncthreads();  // (every warp has read its tiles: what meets below lies in their place)
  // The lanes that hold the same dims of other keys, then the warps, then the blocks.
#pragma unroll
  for (int g = 0; g < G; ++g) {
#pragma unroll
    for (int off = LPK; off < 32; off <<= 1) {
      const float other = __shfl_xor_sync(0xffffffffu, m_run[g], off), mx = fmaxf(m_run[g], other);
      const float use = mx == -INFINITY ? 0.f : mx, keep = exp2_fast(m_run[g] - use);
      l_run[g] *= keep;
      l_run[g] += __shfl_xor_sync(0xffffffffu, l_run[g], off);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[g][e].x *= keep;
        o[g][e].y *= keep;
        o[g][e].x += __shfl_xor_sync(0xffffffffu, o[g][e].x, off);
        o[g][e].y += __shfl_xor_sync(0xffffffffu, o[g][e].y, off);
      }
      m_run[g] = mx;
    }
    if (lane < LPK) {
      *reinterpret_cast<float4*>(&s_o[warp][g][chunk]) = make_float4(o[g][0].x, o[g][0].y, o[g][1].x, o[g][1].y);
      *reinterpret_cast<float4*>(&s_o[warp][g][chunk + 4]) = make_float4(o[g][2].x, o[g][2].y, o[g][3].x, o[g][3].y);
    }
    if (lane == 0) {
      s_m[warp][g] = m_run[g];
      s_l[warp][g] = l_run[g];
    }
  }
  __syncthreads();
  bf16* out = p.out + (size_t)(b * p.num_kv_heads + m) * G * DH;
  for (int i = threadIdx.x; i < G * DH; i += WARPS * 32) {
    const int g = i / DH, d = i % DH;
    float mx = -INFINITY, num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) mx = fmaxf(mx, s_m[w][g]);
    const float use = mx == -INFINITY ? 0.f : mx;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float scale = exp2_fast(s_m[w][g] - use);
      num = fmaf(scale, s_o[w][g][d], num);
      den = fmaf(scale, s_l[w][g], den);
    }
    if (size == 1) {
      out[i] = __float2bfloat16_rn(den > 0.f ? num / den : 0.f);
    } else {
      b_o[i] = num;
      if (d == 0) {
        b_m[g] = mx;
        b_l[g] = den;
      }
    }
  }
  if (size == 1) return;
  sbx::cluster_sync_all();
  for (int i = (int)rank * WARPS * 32 + threadIdx.x; i < G * DH; i += step * 32) {
    const int g = i / DH;
    float ms[MAX_CLUSTER], mx = -INFINITY, num = 0.f, den = 0.f;
#pragma unroll
    for (int r = 0; r < MAX_CLUSTER; ++r) {
      ms[r] = r < (int)size ? from_block(&b_m[g], r) : -INFINITY;
      mx = fmaxf(mx, ms[r]);
    }
    const float use = mx == -INFINITY ? 0.f : mx;
#pragma unroll
    for (int r = 0; r < MAX_CLUSTER; ++r)
      if (r < (int)size) {
        const float scale = exp2_fast(ms[r] - use);
        num = fmaf(scale, from_block(&b_o[i], r), num);
        den = fmaf(scale, from_block(&b_l[g], r), den);
      }
    out[i] = __float2bfloat16_rn(den > 0.f ? num / den : 0.f);
  }
  sbx::cluster_sync_all();  // (nobody leaves while its numbers may be read)
}

// How many clusters of this size the current device holds at once: 0 where it has no room for one (blocks of 128 KB
// and 16 warps need an SM each, all in one GPC) or cannot say.  Asked once per device and size.
template <int G>
int clusters_held(int cluster) {
  constexpr int DEVICES = 64;
  static std::atomic<int> known[DEVICES][MAX_CLUSTER + 1];  // one more than the number; 0: not asked yet
  int device = -1;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0) {
    cudaGetLastError();
    return 0;
  }
  if (device < DEVICES) {
    const int held = known[device][cluster].load(std::memory_order_relaxed);
    if (held > 0) return held - 1;
  }
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(cluster);
  config.blockDim = dim3(WARPS * 32);
  config.dynamicSmemBytes = RING_BYTES;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = cluster;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  int held = 0;
  if (cudaFuncSetAttribute(attn_rows_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES) != cudaSuccess ||
      (cluster > 8 &&
       cudaFuncSetAttribute(attn_rows_kernel<G>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
      cudaOccupancyMaxActiveClusters(&held, attn_rows_kernel<G>, &config) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (device < DEVICES) known[device][cluster].store(held + 1, std::memory_order_relaxed);
  return held;
}

template <int G>
int launch(const RowsParams& p, int blocks, int cluster, cudaStream_t stream) {
  if (clusters_held<G>(cluster) < 1) return -9;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(blocks);
  config.blockDim = dim3(WARPS * 32);
  config.dynamicSmemBytes = RING_BYTES;
  config.stream = stream;
  cudaLaunchAttribute attribute[2];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = cluster;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = sb_pdl_level() == 0 ? 1 : 2;
  const cudaError_t e = cudaLaunchKernelEx(&config, attn_rows_kernel<G>, p);
  if (e != cudaSuccess) return (int)e;
  SB_LAUNCH_CHECK();
  return 0;
}

}  // namespace

static bool cluster_size(int cluster) { return cluster == 1 || cluster == 2 || cluster == 4 || cluster == 8 || cluster == 16; }

// One token for each of `batch` requests, row b of q and out; cluster: blocks per (request, kv head), 1, 2, 4, 8 or 16.
// Returns -9 for what it does not take (other head sizes, groups other than 2 and 4, pages of no
// power of two or shorter than a tile of keys, clusters that the device has no room for).
extern "C" int SB_FN(sb_attn_rows)(const void* q, const void* cache, const int* block_table, int max_pages, const int* q_start,
                                   void* out, int batch, int num_q_heads, int num_kv_heads, int page_size, int num_pages,
                                   float cap, int window, int cluster, int older_keys_settled, int* err, cudaStream_t stream) {
  if constexpr (!TAKES) return -9;
  if (batch == 0) return 0;
  if (num_kv_heads <= 0 || num_q_heads % num_kv_heads) return -8;
  const int group = num_q_heads / num_kv_heads;
  if ((group != 2 && group != 4) || page_size <= 0 || page_size < LD * 256 / DH || (page_size & (page_size - 1)) ||
      !cluster_size(cluster) || ((uintptr_t)q & 15) || ((uintptr_t)cache & 15))
    return -9;
  int shift = 0;
  while (1 << shift < page_size) ++shift;
  const RowsParams p{(const bf16*)q, (const bf16*)cache, block_table, q_start, (bf16*)out, max_pages, num_kv_heads, shift,
                     num_pages, window, older_keys_settled, cap, err};
  const long long blocks = (long long)batch * num_kv_heads * cluster;
  if (blocks > 0x7fffffffLL) return -6;
  if constexpr (TAKES) {
    if (group == 2) return launch<2>(p, (int)blocks, cluster, stream);
    return launch<4>(p, (int)blocks, cluster, stream);
  }
  return -9;
}
