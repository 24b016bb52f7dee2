// C[M,N] = A[M,K] * W[N,K]^T in float32 on the CUDA cores: the products of the float32 engine.
//
// The order of a sum is the same in every kernel and tile here, so a row's result does not depend on the rest of the batch: the
// terms of an element go to eight chains by k (the group k / 4 mod 4, and k even or odd), each summed over ascending k with fused
// multiply-adds; a group's two chains are added, then the groups as (0 + 1) + (2 + 3).  Eight chains of K / 8 terms also stand
// closer to the exact sum than one of K.  Even and odd k are the two halves of a packed operand (fma.rn.f32x2: two products an
// instruction, from 16-byte pieces of rows as they lie in memory, with nothing to rearrange).
//
// gemm_f32_rows_kernel, up to 8 rows: bound by the weights' bytes.  A block owns 8 columns (with SiLU 8 of the gate and 8 of the
// up matrix) and requests their rows at once, before the kernel in front of it has ended; a lane sums one group of one column, a
// warp every fourth row of A.  One row at the 0.6B sizes (one B200, caches cold, before: 64 x 64 tiles, one value a load, one
// stage): q|k|v 115 -> 12 us, o_proj 221 -> 12, gate|up 268 -> 14, down_proj 328 -> 14, vocabulary 895 -> 109 (5.7 TB/s).
// gemm_f32_tile_kernel, more rows: bound by the multiply-adds.  Four warps, one for each group of k, work on the same tile of
// 4 TM x 8 TN, a thread on TM x TN of it: 16 bytes of each of TM + TN rows give 2 TM TN packed instructions, and the stride of 68
// floats lets eight neighbouring rows' pieces come from different banks; two to four blocks share an SM, so one's first loads and
// last sums run beside another's products.  613 rows: q|k|v 281 -> 150 us (34 TFLOP/s; registers alone sustain 61 with these
// instructions), o_proj 240 -> 88, gate|up 528 -> 209 (37 TFLOP/s), down_proj 355 -> 127.  One block of 256 threads an SM on tiles
// of 64 x 64 took 160 and 233 us for q|k|v and gate|up.
#include "f32x2.cuh"
#include "gemm_f32.cuh"
#include "mma_prims.cuh"

namespace {

__device__ __forceinline__ float silu_times(float g, float u) { return g / (1.0f + expf(-g)) * u; }

constexpr int ROWS_MAX = 8;             // rows of A that the rows kernel takes
constexpr int ROWS_SLICE = 1024;        // k a stage
constexpr int ROWS_THREADS = 128;

// Rows of a slice stand slice + 16 floats apart: two columns' four pieces come from all 32 banks.
template <int EPI, int MR>
__global__ void __launch_bounds__(ROWS_THREADS)
gemm_f32_rows_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ W, float* __restrict__ C, int64_t ldc, int M,
                     int N, int K, int slice, int stages) {
  using namespace mma_prims;
  constexpr int WR = EPI ? 16 : 8;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, col = lane >> 2, grp = lane & 3;
  const int n0 = blockIdx.x * 8, stride = slice + 16, stage_floats = (WR + M) * stride, slices = (K + slice - 1) / slice;
  auto load_w = [&](int s) {
    float* dst = smem + (s % stages) * stage_floats;
    const int k0 = s * slice, pieces = min(slice, K - k0) >> 2;
    for (int r = warp; r < WR; r += 4) {
      const float* src = W + ((int64_t)min(n0 + (r & 7), N - 1) + (r >> 3) * (int64_t)N) * K + k0;
      for (int p = lane; p < pieces; p += 32) cp_async16(dst + r * stride + 4 * p, src + 4 * p, true);
    }
  };
  auto load_a = [&](int s) {
    float* dst = smem + (s % stages) * stage_floats + WR * stride;
    const int k0 = s * slice, pieces = min(slice, K - k0) >> 2;
    for (int r = warp; r < M; r += 4)
      for (int p = lane; p < pieces; p += 32) cp_async16(dst + r * stride + 4 * p, A + (int64_t)r * lda + k0 + 4 * p, true);
  };
  const int ahead = min(stages, slices);
  for (int s = 0; s < ahead; ++s) load_w(s);
  pdl_wait();
  pdl_launch_dependents();
  for (int s = 0; s < ahead; ++s) {
    load_a(s);
    cp_async_commit();
  }
  for (int s = ahead; s < 3; ++s) cp_async_commit();      // three groups are under way, whatever the ring's depth
  f32x2 acc[MR] = {}, acu[EPI ? MR : 1] = {};
  for (int s = 0; s < slices; ++s) {
    if (stages >= 3) cp_async_wait<2>();
    else if (stages == 2) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncthreads();
    const float* st = smem + (s % stages) * stage_floats;
    const float* w = st + col * stride + 4 * grp;
    const float* a = st + (WR + warp) * stride + 4 * grp;
    const int len = min(slice, K - s * slice);
    if (warp < M) {
#pragma unroll 4
      for (int k = 0; k < len - 4 * grp; k += 16) {
        const ulonglong2 wv = pairs4(w + k);
        ulonglong2 uv;
        if (EPI) uv = pairs4(w + 8 * stride + k);
#pragma unroll
        for (int i = 0; i < MR; ++i) {
          if (i > 0 && warp + 4 * i >= M) break;
          const ulonglong2 av = pairs4(a + 4 * i * stride + k);
          fma2(acc[i], av.x, wv.x);
          fma2(acc[i], av.y, wv.y);
          if (EPI) {
            fma2(acu[i], av.x, uv.x);
            fma2(acu[i], av.y, uv.y);
          }
        }
      }
    }
    if (s + 1 < slices) {
      __syncthreads();                                    // the stage is free
      if (s + stages < slices) {
        load_w(s + stages);
        load_a(s + stages);
      }
      cp_async_commit();
    }
  }
#pragma unroll
  for (int i = 0; i < MR; ++i) {
    float v = half_sum(acc[i]), u = EPI ? half_sum(acu[EPI ? i : 0]) : 0.f;
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    if (EPI) {
      u += __shfl_xor_sync(0xffffffffu, u, 1);
      u += __shfl_xor_sync(0xffffffffu, u, 2);
      v = silu_times(v, u);
    }
    const int m = warp + 4 * i;
    if (grp == 0 && m < M && n0 + col < N) C[(int64_t)m * ldc + n0 + col] = v;
  }
}

constexpr int TILE_BK = 64, TILE_LD = TILE_BK + 4, TILE_THREADS = 128, TILE_STAGES = 4;
template <int TM, int TN> constexpr int tile_smem = TILE_STAGES * (4 * TM + 8 * TN) * TILE_LD * 4;

// EPI 1: a thread's first TN / 2 columns are the gate's, the others the same columns of the up matrix; 4 TN columns a block.
template <int TM, int TN, int EPI>
__global__ void __launch_bounds__(TILE_THREADS, TM * TN > 32 ? 2 : (TM * TN > 16 ? 3 : 4))
gemm_f32_tile_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ W, float* __restrict__ C, int64_t ldc, int M,
                     int N, int K) {
  using namespace mma_prims;
  constexpr int ROWS = 4 * TM, WROWS = 8 * TN, COLS = EPI ? WROWS / 2 : WROWS, STAGE = (ROWS + WROWS) * TILE_LD;
  static_assert(4 * ROWS * (WROWS + 4) * 4 <= tile_smem<TM, TN>, "the groups' sums fit the ring");
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, grp = tid >> 5, ty = (tid & 31) >> 3, tx = tid & 7;
  const int m0 = blockIdx.y * ROWS, n0 = blockIdx.x * COLS, stages = (K + TILE_BK - 1) / TILE_BK;
  const int lp = 4 * (tid & 15), lr = tid >> 4;           // a thread brings one piece of every 8th row
  // Inside the matrices a row's place is the thread's first one and a multiple of the same distance; only tiles and stages at an edge
  // look at each row.  (Each row's address for itself: 154 and 215 us where q|k|v and gate|up of 613 rows take 150 and 209.)
  const bool inner = m0 + ROWS <= M && n0 + COLS <= N;
  const float* w_first = W + (int64_t)(n0 + lr) * K + lp;
  const float* a_first = A + (int64_t)(m0 + lr) * lda + lp;
  const int64_t w_step = (int64_t)(TILE_THREADS / 16) * K, a_step = (TILE_THREADS / 16) * lda, to_up = ((int64_t)N - COLS) * K;
  auto load_w = [&](int s) {
    float* dst = smem + (s % TILE_STAGES) * STAGE + (ROWS + lr) * TILE_LD + lp;
    if (inner && (s + 1) * TILE_BK <= K) {
      const float* src = w_first + s * TILE_BK;
#pragma unroll
      for (int i = 0; i < WROWS * 16 / TILE_THREADS; ++i)
        cp_async16(dst + i * (TILE_THREADS / 16) * TILE_LD, src + i * w_step + (EPI && i * (TILE_THREADS / 16) >= COLS ? to_up : 0), true);
      return;
    }
    const int k = s * TILE_BK + lp;
#pragma unroll
    for (int i = 0; i < WROWS * 16 / TILE_THREADS; ++i) {
      const int r = lr + i * (TILE_THREADS / 16), c = EPI ? r % COLS : r, n = n0 + c;
      const bool ok = n < N && k < K;
      cp_async16(dst + i * (TILE_THREADS / 16) * TILE_LD, ok ? W + ((int64_t)n + (EPI && r >= COLS ? N : 0)) * K + k : W, ok);
    }
  };
  auto load_a = [&](int s) {
    float* dst = smem + (s % TILE_STAGES) * STAGE + lr * TILE_LD + lp;
    if (inner && (s + 1) * TILE_BK <= K) {
      const float* src = a_first + s * TILE_BK;
#pragma unroll
      for (int i = 0; i < ROWS * 16 / TILE_THREADS; ++i) cp_async16(dst + i * (TILE_THREADS / 16) * TILE_LD, src + i * a_step, true);
      return;
    }
    const int k = s * TILE_BK + lp;
#pragma unroll
    for (int i = 0; i < ROWS * 16 / TILE_THREADS; ++i) {
      const int r = lr + i * (TILE_THREADS / 16);
      const bool ok = m0 + r < M && k < K;
      cp_async16(dst + i * (TILE_THREADS / 16) * TILE_LD, ok ? A + (int64_t)(m0 + r) * lda + k : A, ok);
    }
  };
#pragma unroll
  for (int s = 0; s < TILE_STAGES - 1; ++s)
    if (s < stages) load_w(s);
  pdl_wait();
  pdl_launch_dependents();
#pragma unroll
  for (int s = 0; s < TILE_STAGES - 1; ++s) {
    if (s < stages) load_a(s);
    cp_async_commit();
  }
  f32x2 acc[TM][TN] = {};
  for (int s = 0; s < stages; ++s) {
    cp_async_wait<TILE_STAGES - 2>();
    __syncthreads();                                      // the stage has come; the one before it is free
    if (s + TILE_STAGES - 1 < stages) {
      load_w(s + TILE_STAGES - 1);
      load_a(s + TILE_STAGES - 1);
    }
    cp_async_commit();
    const float* a = smem + (s % TILE_STAGES) * STAGE + ty * TILE_LD + 4 * grp;
    const float* w = smem + (s % TILE_STAGES) * STAGE + (ROWS + tx) * TILE_LD + 4 * grp;
#pragma unroll
    for (int k = 0; k < TILE_BK; k += 16) {
      ulonglong2 av[TM], wv[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = pairs4(a + 4 * i * TILE_LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) wv[j] = pairs4(w + 8 * j * TILE_LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], av[i].x, wv[j].x);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], av[i].y, wv[j].y);
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  constexpr int LDS = WROWS + 4, GROUP = ROWS * LDS;      // the groups' sums, over the ring
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) smem[grp * GROUP + (ty + 4 * i) * LDS + tx + 8 * j] = half_sum(acc[i][j]);
  __syncthreads();
  auto total = [&](int at) { return (smem[at] + smem[GROUP + at]) + (smem[2 * GROUP + at] + smem[3 * GROUP + at]); };
  for (int idx = tid; idx < ROWS * COLS; idx += TILE_THREADS) {
    const int r = idx / COLS, c = idx - r * COLS;
    if (m0 + r >= M || n0 + c >= N) continue;
    const float v = total(r * LDS + c);
    C[(int64_t)(m0 + r) * ldc + n0 + c] = EPI ? silu_times(v, total(r * LDS + COLS + c)) : v;
  }
}

int raise_smem(const void* kernel, int bytes) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  ME_REQUIRE(e == cudaSuccess, "me_gemm_simt: cannot raise shared memory: %s", cudaGetErrorString(e));
  return 0;
}

constexpr int SMEM_MOST = 200 * 1024;

template <int EPI, int MR>
int launch_rows(const float* A, int64_t lda, const float* W, float* C, int64_t ldc, int M, int N, int K, cudaStream_t stream) {
  static const int raised = raise_smem((const void*)gemm_f32_rows_kernel<EPI, MR>, SMEM_MOST);
  if (raised) return raised;
  const int slice = K < ROWS_SLICE ? (K + 15) / 16 * 16 : ROWS_SLICE, slices = (K + slice - 1) / slice;
  const int stage = ((EPI ? 16 : 8) + M) * (slice + 16) * 4;
  const int fit = SMEM_MOST / stage, stages = slices < 3 ? (slices < fit ? slices : fit) : (fit < 3 ? fit : 3);
  me_launch(gemm_f32_rows_kernel<EPI, MR>, dim3((N + 7) / 8), dim3(ROWS_THREADS), (size_t)stages * stage, stream, A, lda, W, C, ldc, M, N,
            K, slice, stages);
  return 0;
}

template <int TM, int TN, int EPI>
int launch_tile(const float* A, int64_t lda, const float* W, float* C, int64_t ldc, int M, int N, int K, cudaStream_t stream) {
  static const int raised = raise_smem((const void*)gemm_f32_tile_kernel<TM, TN, EPI>, tile_smem<TM, TN>);
  if (raised) return raised;
  constexpr int COLS = EPI ? 4 * TN : 8 * TN, MOST = 65535 * 4 * TM;       // rows of a launch: the grid's y counts tiles of rows
  for (int m0 = 0; m0 < M; m0 += MOST) {
    const int rows = M - m0 < MOST ? M - m0 : MOST;
    me_launch(gemm_f32_tile_kernel<TM, TN, EPI>, dim3((N + COLS - 1) / COLS, (rows + 4 * TM - 1) / (4 * TM)), dim3(TILE_THREADS),
              (size_t)tile_smem<TM, TN>, stream, A + (int64_t)m0 * lda, lda, W, C + (int64_t)m0 * ldc, ldc, rows, N, K);
  }
  return 0;
}

template <int EPI>
int launch_f32(const float* A, int64_t lda, const float* W, float* C, int64_t ldc, int M, int N, int K, cudaStream_t stream) {
  // From 5 rows on the rows kernel is bound by what it reads of shared memory, and tiles are faster where there is one for every SM
  // (8 rows: 151,936 columns of 1,024 terms 272 us against 162 in tiles, 4,096 columns 19 us either way, 1,024 columns of 2,048 terms
  // 14.4 against 20.5); 9 to 16 rows took 22.6 to 37 us where the tiles take 18.5 to 20.5.
  const int64_t cols = (int64_t)N * (EPI ? 2 : 1);
  if (M <= 4) return launch_rows<EPI, 1>(A, lda, W, C, ldc, M, N, K, stream);
  if (M <= ROWS_MAX && (cols + 31) / 32 < me_sm_count()) return launch_rows<EPI, 2>(A, lda, W, C, ldc, M, N, K, stream);
  // The tile whose share of an SM costs least: TM x TN products and, at 0.6 of a product, the TM + TN pieces read for them.  (613 rows of
  // 1,024 terms: 4,096 columns 154, 156 and 168 us with the three tiles, 1,024 columns of 2,048 terms 104, 90 and 92; 32 rows, 1,024
  // columns: 43, 29 and 20.)
  auto cost = [&](int tm, int tn) {
    const int64_t tiles = (int64_t)((M + 4 * tm - 1) / (4 * tm)) * ((cols + 8 * tn - 1) / (8 * tn));
    return (tiles + me_sm_count() - 1) / me_sm_count() * (5 * tm * tn + 3 * (tm + tn));
  };
  const int64_t large = cost(8, 8), wide = cost(8, 4), small = cost(4, 4);
  if (large <= wide && large <= small) return launch_tile<8, 8, EPI>(A, lda, W, C, ldc, M, N, K, stream);
  if (wide <= small) return launch_tile<8, 4, EPI>(A, lda, W, C, ldc, M, N, K, stream);
  return launch_tile<4, 4, EPI>(A, lda, W, C, ldc, M, N, K, stream);
}

}  // namespace

bool gemm_f32_takes(const float* A, int64_t lda, const float* W, int K) {
  return K % 4 == 0 && lda % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
}

int gemm_f32(const float* A, int64_t lda, const float* W, float* C, int64_t ldc, int M, int N, int K, int epi, cudaStream_t stream) {
  return epi ? launch_f32<1>(A, lda, W, C, ldc, M, N, K, stream) : launch_f32<0>(A, lda, W, C, ldc, M, N, K, stream);
}
