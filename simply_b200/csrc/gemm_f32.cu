// True 32-bit matrix product on CUDA cores: out[M, N] = x[M, K] . w[N, K]^T.
//
// No tensor-core mode, no reduced-precision staging: every product and sum is a
// float32 FMA.  Every output is the sum ((c0 + c1) + c2) + c3 of four chains of FMAs, one over each quarter of k
// (whole tiles of 32 long), whatever kernel computes it and whether the quarters are walked one after the other or
// side by side, so a token's result does not depend on what else is in the batch.
// Optional epilogue: soft cap (simply/model_lib.py:107-109) for the output layer.
//
// Bound by the FMA pipes for many rows, by the weights' bytes for a few.  Four tile shapes share the
// chains' order: 128 x 128 outputs (16 x 8 per thread, packed FMAs) for products of many tiles and long rows,
// 64 x 64 (8 x 4 per thread) where those fill the GPU, 32 x 32 (4 x 4 per thread) where they do not, and
// 8 x 16 or 16 x 8 (one output per thread) fed by a deep ring of asynchronous copies for up to 16 rows, where
// the weights only stream by.  sb_gemm_f32_tile has the lines between them; sb_gemm_f32_groups says whether a
// tile's quarters of k are four groups of a block's threads.
#include <type_traits>

#include "common.cuh"

// Two FMAs in one instruction, each rounded as fmaf rounds.
__device__ __forceinline__ void fma_pair(float2& acc, float2 a, float2 b) {
  unsigned long long* c = reinterpret_cast<unsigned long long*>(&acc);
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(*c)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
}

__device__ __forceinline__ float capped(float v, float cap) { return cap > 0.f ? cap * tanhf(v / cap) : v; }

// Four values of a row from k on (zeros beyond the matrix); `vec`: rows start on 16-byte boundaries.
__device__ __forceinline__ float4 row_quad(const float* __restrict__ p, bool in, int k, int K, bool vec) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!in) return v;
  if (vec) {
    if (k < K) v = *reinterpret_cast<const float4*>(p + k);
  } else {
    if (k < K) v.x = p[k];
    if (k + 1 < K) v.y = p[k + 1];
    if (k + 2 < K) v.z = p[k + 2];
    if (k + 3 < K) v.w = p[k + 3];
  }
  return v;
}

// ---------------------------------------------------------------------------
// Many rows: a BM x BN tile, TM x TN outputs per thread as TM / 2 pairs of rows.  Tiles of BK k stand
// turned round in shared memory ([k][row], so a thread reads its rows as one vector), twice: while
// one is multiplied the next one's values are on their way in registers.  Neighbouring lanes fetch a
// row's 16-byte quads; the rows of the four k of quad q are kept at places row ^ turn(q), so that the
// 32 values a warp stores at a time lie on 32 banks.
//
// GROUPS 4: four groups of threads take a quarter of k each, with tiles of their own in shared memory, and their
// chains meet there at the end; 1: one group walks the quarters in turn and keeps the sum so far there.
//
// What bounds it: a warp's reads of shared memory deliver 128 bytes a cycle and SM, so TM + TN cycles per
// k beside TM TN / 4 cycles of FMAs: 16 x 8 outputs per thread keep the FMA pipes the longer of the two,
// 8 x 8 are even, and 8 x 4 are half as long again as their FMAs.  64 x 64 of 8 x 4 all the same, whose blocks of
// 128 threads stand four to an SM: with 8 x 8 per thread 256 x 16,384 x 2,048 took 425 us (GROUPS 4: 467) in place of 351.
// One group walks all of k as one pipeline: a pipeline per quarter waited for its first tile four times (6,000 x 16,384 x
// 64 329 us in place of 308).  Four blocks to an SM only if the compiler is held to 128 registers: 3 blocks of 134 335 us.
// The sums so far pass through shared memory, at 256 bytes per thread and quarter: rows of a few tiles pay for it
// (6,000 x 2,048 x 100 81 us, as one chain 75; x 256 142 and 138; x 2,048 and longer nothing).
// ---------------------------------------------------------------------------
// A quarter of k, in whole tiles of 32.
__host__ __device__ __forceinline__ int f32_quarter(int K) { return (K + 127) / 128 * 32; }

template <int BM, int BN, int BK, int TM, int TN, int GROUPS>
__global__ void __launch_bounds__((BM / TM) * (BN / TN) * GROUPS, BM == 64 && GROUPS == 1 ? 4 : BM == 128 ? 1 : 0)
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, int M, int N,
                     int K, float cap, int vec) {
  constexpr int THREADS = (BM / TM) * (BN / TN), QUADS = BK / 4;  // (threads of a group)
  constexpr int TILE_FLOATS = 2 * BK * (BM + BN);  // a group's two tiles of x and of w
  static_assert(TILE_FLOATS >= BM * BN || GROUPS == 1, "a group's results take the place of its tiles");
  constexpr int XQ = BM * QUADS / THREADS, WQ = BN * QUADS / THREADS;  // quads a thread fetches per tile
  static_assert(BM * QUADS % THREADS == 0 && BN * QUADS % THREADS == 0, "whole quads per thread");
  static_assert(TM % 4 == 0 && TN % 4 == 0 && QUADS <= 8 && BM % 32 == 0 && BN % 32 == 0, "vectors of 4, places within a row");
  pdl_wait_block();
  pdl_launch_dependents();
  extern __shared__ __align__(16) float tile_smem[];
  const int group = GROUPS == 1 ? 0 : threadIdx.x / THREADS, tid = GROUPS == 1 ? threadIdx.x : threadIdx.x % THREADS;
  float (*xs)[BK][BM] = reinterpret_cast<float (*)[BK][BM]>(tile_smem + group * TILE_FLOATS);
  float (*ws)[BK][BN] = reinterpret_cast<float (*)[BK][BN]>(tile_smem + group * TILE_FLOATS + 2 * BK * BM);
  auto meet = [&]() {  // the threads of a group
    if (GROUPS == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;\n" ::"r"(group + 1), "n"(THREADS) : "memory");
  };
  // A warp is 4 groups of rows by 8 of columns: its vectors of a k are few and shared.
  const int lane = tid & 31, warp = tid >> 5;
  constexpr int WARP_COLS = BN / (8 * TN);
  // (a thread's columns: groups of 4, 32 apart, so that 8 lanes read 128 bytes in a row)
  const int mt = ((warp / WARP_COLS) * 4 + (lane >> 3)) * TM, nt = (warp % WARP_COLS) * 8 * TN + (lane & 7) * 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int quad = tid % QUADS, row = tid / QUADS;
  auto turn = [](int q) { return (q % 4) * 8 + (q / 4) * 4; };
  constexpr int STEP = THREADS / QUADS;  // rows between a thread's pieces
  float4 xq[XQ], wq[WQ];
  auto fetch = [&](int k0, int k_end) {
#pragma unroll
    for (int i = 0; i < XQ; ++i) {
      const int r = m0 + row + i * STEP;
      xq[i] = row_quad(x + (size_t)r * K, r < M, k0 + quad * 4, k_end, vec);
    }
#pragma unroll
    for (int i = 0; i < WQ; ++i) {
      const int r = n0 + row + i * STEP;
      wq[i] = row_quad(w + (size_t)r * K, r < N, k0 + quad * 4, k_end, vec);
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int i = 0; i < XQ; ++i) {
      const int r = (row + i * STEP) ^ turn(quad);
      xs[buf][quad * 4][r] = xq[i].x; xs[buf][quad * 4 + 1][r] = xq[i].y; xs[buf][quad * 4 + 2][r] = xq[i].z; xs[buf][quad * 4 + 3][r] = xq[i].w;
    }
#pragma unroll
    for (int i = 0; i < WQ; ++i) {
      const int r = (row + i * STEP) ^ turn(quad);
      ws[buf][quad * 4][r] = wq[i].x; ws[buf][quad * 4 + 1][r] = wq[i].y; ws[buf][quad * 4 + 2][r] = wq[i].z; ws[buf][quad * 4 + 3][r] = wq[i].w;
    }
  };
  float2 acc[TM / 2][TN];
  float* sums = tile_smem + TILE_FLOATS + tid;  // GROUPS 1: this thread's sums so far, THREADS apart
  const int quarter = f32_quarter(K);
  const int k_start = GROUPS == 1 ? 0 : min(group * quarter, K), k_end = GROUPS == 1 ? K : min(k_start + quarter, K);
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
  if (k_start < k_end) {
    fetch(k_start, k_end);
    put(0);
  }
  meet();
  int next_quarter = quarter;  // where the next chain begins
  auto add_sums = [&]() {
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float* at = sums + (i * TN + j) * 2 * THREADS;
        acc[i][j].x = at[0] + acc[i][j].x;
        acc[i][j].y = at[THREADS] + acc[i][j].y;
      }
  };
  for (int k0 = k_start, buf = 0; k0 < k_end; k0 += BK, buf ^= 1) {
    const bool more = k0 + BK < k_end;
    if (more) fetch(k0 + BK, k_end);
    float2 a[2][TM / 2];
    float b[2][TN];
    auto read = [&](int s, int k) {
      const int at = turn(k / 4);
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&xs[buf][k][(mt + i) ^ at]);
        a[s][i / 2] = make_float2(v.x, v.y);
        a[s][i / 2 + 1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&ws[buf][k][(nt + j * 8) ^ at]);
        b[s][j] = v.x; b[s][j + 1] = v.y; b[s][j + 2] = v.z; b[s][j + 3] = v.w;
      }
    };
    read(0, 0);
#pragma unroll
    for (int k = 0; k < BK; ++k) {  // (values beyond the end are zeros on both sides: the chain keeps its value)
      if (k + 1 < BK) read((k + 1) & 1, k + 1);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float2 bb = make_float2(b[k & 1][j], b[k & 1][j]);
#pragma unroll
        for (int i = 0; i < TM / 2; ++i) fma_pair(acc[i][j], a[k & 1][i], bb);
      }
    }
    if (GROUPS == 1 && more && k0 + BK == next_quarter) {  // (a chain has ended; the next tiles are on their way)
      if (next_quarter > quarter) add_sums();
#pragma unroll
      for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          float* at = sums + (i * TN + j) * 2 * THREADS;
          at[0] = acc[i][j].x;
          at[THREADS] = acc[i][j].y;
          acc[i][j] = make_float2(0.f, 0.f);
        }
      next_quarter += quarter;
    }
    if (more) put(buf ^ 1);
    meet();
  }
  if (GROUPS == 1 && next_quarter > quarter) add_sums();
  if (GROUPS == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gm = m0 + mt + i;
      if (gm >= M) break;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int gn = n0 + nt + (j / 4) * 32 + j % 4;
        if (gn < N) out[(size_t)gm * N + gn] = capped(i & 1 ? acc[i / 2][j].y : acc[i / 2][j].x, cap);
      }
    }
    return;
  }
  // The groups' chains meet: [BM][BN] each, in the place of a group's own tiles.
  float* mine = tile_smem + group * TILE_FLOATS;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; j += 4) {
      const float4 v = i & 1 ? make_float4(acc[i / 2][j].y, acc[i / 2][j + 1].y, acc[i / 2][j + 2].y, acc[i / 2][j + 3].y)
                             : make_float4(acc[i / 2][j].x, acc[i / 2][j + 1].x, acc[i / 2][j + 2].x, acc[i / 2][j + 3].x);
      *reinterpret_cast<float4*>(mine + (mt + i) * BN + nt + j * 8) = v;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < BM * BN; i += THREADS * GROUPS) {
    const int gm = m0 + i / BN, gn = n0 + i % BN;
    if (gm >= M || gn >= N) continue;
    float sum = tile_smem[i];
#pragma unroll
    for (int part = 1; part < GROUPS; ++part) sum += tile_smem[part * TILE_FLOATS + i];
    out[(size_t)gm * N + gn] = capped(sum, cap);
  }
}

// ---------------------------------------------------------------------------
// Up to 16 rows: one output per thread, 128 per block (ROWS x 128 / ROWS).  The weights' rows stream
// through a ring of asynchronous 16-byte copies (rows of 16-byte multiples only), several blocks per
// SM; a thread has the vectors of the next 16 k in registers while it multiplies these.  The four quarters' chains one
// after the other: side by side a stage held 32 k of each, and took longer although the FMAs wait less for one another
// (us, side by side and so: 1 x 16,384 x 2,048 44.8 and 42.2, x 2,048 x 8,192 49.2 and 45.3; 8 x 16,384 x 2,048 78.6 and
// 76; 9 117.8 and 121; 16 138 and 127.5, x 2,048 x 8,192 102.7 and 102.3).
// ---------------------------------------------------------------------------
#define F32_FEW 16        // most rows
#define F32_FEW_K 128     // k per stage
#define F32_FEW_STAGES 5
#define F32_FEW_LD (F32_FEW_K + 4)  // a row's start moves on by 4 banks

template <int ROWS>
__global__ void __launch_bounds__(128)
gemm_f32_few_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, int M, int N, int K,
                    float cap) {
  constexpr int COLS = 128 / ROWS, STAGE = (COLS + ROWS) * F32_FEW_LD, PIECES = F32_FEW_K / 4;
  extern __shared__ __align__(16) float few_smem[];  // stages of (weights [COLS][LD], x [ROWS][LD])
  const int n0 = blockIdx.x * COLS;
  const int steps = (K + F32_FEW_K - 1) / F32_FEW_K, quarter = f32_quarter(K);
  // A warp copies a row's 512 bytes at a time.  (Beyond the matrix: 0 bytes read, zeros written.)
  const int piece = (threadIdx.x % PIECES) * 4, first = threadIdx.x / PIECES;
  auto copy = [&](const float* from, int rows, int count, int step, float* to) {
    const int k = step * F32_FEW_K + piece;
    for (int r = first; r < count; r += 128 / PIECES) {
      const bool in = r < rows && k < K;
      const float* src = in ? from + (size_t)r * K + k : from;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                       (unsigned)__cvta_generic_to_shared(to + r * F32_FEW_LD + piece)), "l"(src), "r"(in ? 16 : 0));
    }
  };
  const float* wn = w + (size_t)n0 * K;
  // The weights of the first stages need nothing from the kernel before.
  for (int s = 0; s < F32_FEW_STAGES - 1; ++s)
    if (s < steps) copy(wn, N - n0, COLS, s, few_smem + s * STAGE);
  pdl_wait_block();
  pdl_launch_dependents();
  for (int s = 0; s < F32_FEW_STAGES - 1; ++s) {
    if (s < steps) copy(x, M, ROWS, s, few_smem + s * STAGE + COLS * F32_FEW_LD);
    asm volatile("cp.async.commit_group;\n");
  }
  const int m = threadIdx.x / COLS, n = threadIdx.x % COLS;
  float acc = 0.f, sum = 0.f;  // the chain that is walked, the ones that have ended
  int left = quarter;          // of this chain's k
  auto ended = [&]() {
    sum += acc;
    acc = 0.f;
    left = quarter;
  };
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(F32_FEW_STAGES - 2));
    __syncthreads();  // the stage has landed for all; the one read a turn ago is free
    const int next = s + F32_FEW_STAGES - 1;
    if (next < steps) {
      float* to = few_smem + (next % F32_FEW_STAGES) * STAGE;
      copy(wn, N - n0, COLS, next, to);
      copy(x, M, ROWS, next, to + COLS * F32_FEW_LD);
    }
    asm volatile("cp.async.commit_group;\n");
    if (m >= M) continue;
    const float* wr = few_smem + (s % F32_FEW_STAGES) * STAGE + n * F32_FEW_LD;
    const float* xr = few_smem + (s % F32_FEW_STAGES) * STAGE + (COLS + m) * F32_FEW_LD;
    auto walk = [&](auto count, int k0) {
      constexpr int COUNT = decltype(count)::value;
      float4 a[2][4], b[2][4];
      auto read = [&](int at, int k) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          a[at][q] = *reinterpret_cast<const float4*>(xr + k + 4 * q);
          b[at][q] = *reinterpret_cast<const float4*>(wr + k + 4 * q);
        }
      };
      read(0, k0);
#pragma unroll
      for (int k = 0; k < COUNT; k += 16) {
        const int at = (k / 16) & 1;
        if (k + 16 < COUNT) read(at ^ 1, k0 + k + 16);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc = fmaf(a[at][q].x, b[at][q].x, acc);
          acc = fmaf(a[at][q].y, b[at][q].y, acc);
          acc = fmaf(a[at][q].z, b[at][q].z, acc);
          acc = fmaf(a[at][q].w, b[at][q].w, acc);
        }
      }
      left -= COUNT;
    };
    if (left >= F32_FEW_K) {
      walk(std::integral_constant<int, F32_FEW_K>{}, 0);
      if (left == 0) ended();
    } else {  // a chain ends inside the stage (quarters are whole times 32)
      for (int k = 0; k < F32_FEW_K; k += 32) {
        walk(std::integral_constant<int, 32>{}, k);
        if (left == 0) ended();
      }
    }
  }
  if (m < M && n0 + n < N) out[(size_t)m * N + n0 + n] = capped(sum + acc, cap);
}

template <int ROWS>
static int launch_f32_few(const float* x, const float* w, float* out, int M, int N, int K, float cap, cudaStream_t stream) {
  constexpr int COLS = 128 / ROWS;
  constexpr size_t smem = (size_t)F32_FEW_STAGES * (COLS + ROWS) * F32_FEW_LD * sizeof(float);
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  sb_launch_early(gemm_f32_few_kernel<ROWS>, (N + COLS - 1) / COLS, 128, smem, stream, x, w, out, M, N, K, cap);
  SB_LAUNCH_CHECK();
  return 0;
}

template <int BM, int BN, int BK, int TM, int TN, int GROUPS>
static int launch_f32_tile(const float* x, const float* w, float* out, int M, int N, int K, float cap, int vec,
                           cudaStream_t stream) {
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return -6;
  constexpr size_t smem = sizeof(float) * (GROUPS * 2 * BK * (BM + BN) + (GROUPS == 1 ? BM * BN : 0));
  auto kernel = gemm_f32_tile_kernel<BM, BN, BK, TM, TN, GROUPS>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  sb_launch(kernel, grid, (BM / TM) * (BN / TN) * GROUPS, smem, stream, x, w, out, M, N, K, cap, vec);
  SB_LAUNCH_CHECK();
  return 0;
}

// Rows of the tile that a product takes; `vec`: rows of whole 16-byte pieces that start on their boundaries.
// A block of 128 x 128 fills an SM and its tile is long to set up and to store, so it needs many rounds of
// tiles and long rows (us, 128 x 128 against 64 x 64): 256 x 16,384 x 2,048 (256 tiles) 376 and 351; 4,000 x
// 3,100 x 2,048 (800) 1,075 and 1,024; 1,500 x 9,000 x 2,048 (852) 1,079 and 1,116, x 1,024 569 and 569, x 256
// 188 and 156; 2,048 x 16,384 x 2,048 (2,048) 2,467 and 2,678, x 512 716 and 702; 1,500 x 3,100 x 31 29.2 and 12.5.
extern "C" int sb_gemm_f32_tile(int M, int N, int K, int vec) {
  if (M <= F32_FEW && vec && K > 0) return M <= 8 ? 8 : 16;
  auto tiles = [&](int side) { return (long long)((N + side - 1) / side) * ((M + side - 1) / side); };
  if (tiles(128) >= 840 && K >= 1024) return 128;
  return tiles(64) >= 96 ? 64 : 32;
}

// Groups of threads a tile of 64 or 32 has for the quarters of k.  Four where the tiles alone leave SMs with too few
// warps and the quarters are long enough to share: an SM holds one block of 4 x 128 threads, or four of 128.  us, 1 group
// against 4, tiles of 64:
//   to one per SM   256 x 2,048 x 64 (128) 5.4 and 5.4, x 100 7.9 and 7.2, x 256 12.5 and 10.7, x 2,048 72 and 56, x 8,192 275 and 207
//   to two          44 x 16,384 x 512 (256) 31.2 and 32.0, x 2,048 110 and 107; 256 x 3,000 x 515 (188) 35.3 and 37.1;
//                   256 x 3,072 x 2,048 (192) 112 and 108; 600 x 1,600 x 1,024 (250) 58.6 and 57.9
//   beyond          600 x 2,048 x 100 (320) 16.5 and 16.9, x 256 27.6 and 26.8, x 512 50 and 46, x 2,048 185 and 158, x 8,192
//                   726 and 593; 600 x 3,072 x 2,048 (480) 209 and 208; 44 x 32,768 x 2,048 (512) 203 and 208;
//                   256 x 16,384 x 2,048 (1,024) 351 and 369
// and of 32: 44 x 2,048 x 2,048 56 and 26, x 8,192 230 and 96; 300 x 500 x 1,024 31 and 22; 20 x 2,048 x 64 4.5 and 3.8, x 32
// 3.6 and 3.6.
extern "C" int sb_gemm_f32_groups(int M, int N, int K, int tile) {
  const long long tiles = (long long)((N + 63) / 64) * ((M + 63) / 64);
  if (tile == 32) return K > 32 ? 4 : 1;
  if (tile != 64) return 1;
  return (tiles <= 148 ? K > 64 : tiles < 400 && K >= (tiles <= 296 ? 1024 : 256)) ? 4 : 1;
}

// `tile` and `groups`: 0 for the ones that the sizes choose (others are for tests).
extern "C" int sb_gemm_f32_nt_as(const float* x, const float* w, float* out, int M, int N, int K, float cap, int tile,
                                 int groups, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  const int vec = K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  if (tile == 0) tile = sb_gemm_f32_tile(M, N, K, vec);
  if (tile <= F32_FEW && (!vec || K <= 0 || M > tile)) return -9;
  if (groups == 0) groups = sb_gemm_f32_groups(M, N, K, tile);
  switch (tile) {
    case 8: return launch_f32_few<8>(x, w, out, M, N, K, cap, stream);
    case 16: return launch_f32_few<16>(x, w, out, M, N, K, cap, stream);
    case 128: return launch_f32_tile<128, 128, 16, 16, 8, 1>(x, w, out, M, N, K, cap, vec, stream);
    case 64:
      return groups == 4 ? launch_f32_tile<64, 64, 32, 8, 4, 4>(x, w, out, M, N, K, cap, vec, stream)
                         : launch_f32_tile<64, 64, 32, 8, 4, 1>(x, w, out, M, N, K, cap, vec, stream);
    case 32:
      return groups == 4 ? launch_f32_tile<32, 32, 32, 4, 4, 4>(x, w, out, M, N, K, cap, vec, stream)
                         : launch_f32_tile<32, 32, 32, 4, 4, 1>(x, w, out, M, N, K, cap, vec, stream);
    default: return -9;
  }
}

extern "C" int sb_gemm_f32_nt(const float* x, const float* w, float* out, int M, int N, int K, float cap,
                              cudaStream_t stream) {
  return sb_gemm_f32_nt_as(x, w, out, M, N, K, cap, 0, 0, stream);
}
