// The mLSTM recurrence (mlstm.cu) for portions of prompts, a run of MLSTM_LC tokens at a time, all runs of a step side by side.  Within a
// run, with b_t the sum of its log forget gates up to t, x_t the largest gi_s - b_s of s <= t, and (S0, n0, m0) the state in front of it,
// unrolling the recurrence gives
//   m_t = b_t + max(m0, x_t)
//   S_t^T q_t = exp(b_t + m0 - m_t) S0^T q_t + sum_{s<=t} exp(b_t - b_s + gi_s - m_t) (k_s . q_t) v_s     (n_t . q_t likewise)
//   S_L = exp(b_L + m0 - m_L) S0 + exp(b_L + x_L - m_L) U,   U = sum_s exp(gi_s - b_s - x_L) k_s v_s^T    (n_L likewise)
// U and its sum of keys need nothing from in front of the run, so only the last line is walked in order.  All exponents are <= 0.
// Sums of gates are 64 bits, all else is float32; the results differ from the token-by-token kernel by the order of the sums.
//
//   ml_state_kernel   gates, b, x and U of every run: one block = one run x one head x 64 columns
//   ml_walk_kernel    per request, in order: states[c] <- the state in front of run c
//   ml_out_kernel     the outputs of a run: scores with their weights, times v, plus q S0, over the denominators
// What bounds it: float32 multiply-adds on the CUDA cores (D V for U, D V for q S0, 64 V for the weighted v and 64 D for the scores in each
// of the V / 64 blocks of a run's outputs: about 3 D V + 64 V a token and head, a quarter of it scores that one block could work out for
// all) and the states' way through memory (16 D V bytes a run and head: written, read and rewritten by the walk, read for the outputs).
// One kernel that walked a request's runs in order, a block for 16 columns of a head, worked the scores out in each of them and had as
// many steps behind one another as the longest prompt has runs: 3 prompts of 300 to 1,300 tokens, 8 heads of 128 x 256: 1,064 us, now
// 221 in all (under ncu, caches cold, 66 + 24 + 149).
#include "mlstm.cuh"
#include "vec4.cuh"

namespace {

constexpr int LC = MLSTM_LC, VT = 64, THREADS = 256;

struct MlRun {                  // a run and head
  double b[LC], w[LC], x[LC];   // b_t, gi_t - b_t and its largest up to t (beyond the last token: no further decay, gi -inf)
  float m0, m1, unused[2];      // the running maximum in front of the run and behind it
};

template <int VEC> __device__ __forceinline__ void ldv(const float* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) ld4(p, v);
  else v[0] = *p;
}
template <int VEC> __device__ __forceinline__ void stv(float* p, const float (&v)[VEC]) {
  if constexpr (VEC == 4) st4(p, v);
  else *p = v[0];
}

// rows x cols values of a matrix in global memory into shared memory, times f, zeros beyond n_rows and n_cols
template <int VEC>
__device__ __forceinline__ void fill(float* dst, int ld_dst, int rows, int cols, const float* src, int64_t ld_src, int n_rows, int n_cols, float f = 1.f) {
  const int per = cols / VEC;
#pragma unroll 4
  for (int i = threadIdx.x; i < rows * per; i += THREADS) {
    const int r = i / per, c = (i - r * per) * VEC;
    float v[VEC] = {};
    if (r < n_rows && c < n_cols) ldv<VEC>(src + (int64_t)r * ld_src + c, v);
#pragma unroll
    for (int j = 0; j < VEC; ++j) v[j] *= f;
    stv<VEC>(dst + r * ld_dst + c, v);
  }
}

// The first warp's work: the run's gates and their scans, two tokens a lane.  The sums of the gates are 64 bits: they go down to -64 caps,
// where a float is rounded to 6e-5 (cap 15), and the weights are exponentials of their differences.
__device__ __forceinline__ void run_gates(const MlstmArgs& a, int tok0, int L, int h, double* b_s, double* w_s, double* x_s) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  float gf[2], gi[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = 2 * lane + e;
    gf[e] = 0.f;
    gi[e] = -INFINITY;
    if (t < L) {
      const float* row = a.proj + (int64_t)(tok0 + t) * a.ld;
      gi[e] = mlstm_capped(row[a.off_i + h] + a.bias_i[h], a.cap);
      gf[e] = mlstm_log_sigmoid(mlstm_capped(row[a.off_f + h] + a.bias_f[h], a.cap));
    }
  }
  double run = (double)gf[0] + gf[1];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const double up = __shfl_up_sync(0xffffffffu, run, off);
    if (lane >= off) run += up;
  }
  const double b1 = run, b0 = run - gf[1], w0 = gi[0] - b0, w1 = gi[1] - b1;
  double mx = fmax(w0, w1);
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const double up = __shfl_up_sync(0xffffffffu, mx, off);
    if (lane >= off) mx = fmax(mx, up);
  }
  const double before = __shfl_up_sync(0xffffffffu, mx, 1);
  b_s[2 * lane] = b0;
  b_s[2 * lane + 1] = b1;
  w_s[2 * lane] = w0;
  w_s[2 * lane + 1] = w1;
  x_s[2 * lane] = lane > 0 ? fmax(before, w0) : w0;
  x_s[2 * lane + 1] = mx;
}

template <int VEC>
__global__ void __launch_bounds__(THREADS)
ml_state_kernel(MlstmArgs a, const int* __restrict__ tiles, float* __restrict__ states, float* __restrict__ key_sums, MlRun* __restrict__ runs) {
  extern __shared__ __align__(16) float smem[];
  __shared__ double b_s[LC], w_s[LC], x_s[LC];
  __shared__ float u_s[LC];                     // a token's weight in U
  const int D = a.D, V = a.V, Dp = (D + 63) / 64 * 64, ldk = Dp + 4;
  float* Kt = smem;                             // [LC][Dp + 4]
  float* Vc = Kt + LC * ldk;                    // [LC][VT], times a token's weight
  const int tid = threadIdx.x, h = blockIdx.y, v0 = blockIdx.z * VT;
  const int b = tiles[2 * blockIdx.x], q0 = tiles[2 * blockIdx.x + 1];
  const int tok0 = a.cu[b] + q0, L = min(LC, a.cu[b + 1] - tok0);
  pdl_wait();
  pdl_launch_dependents();
  if (L <= 0) return;
  run_gates(a, tok0, L, h, b_s, w_s, x_s);
  fill<VEC>(Kt, ldk, LC, Dp, a.proj + (int64_t)tok0 * a.ld + a.off_k + (int64_t)h * D, a.ld, L, D);
  __syncthreads();
  if (tid < LC) {
    u_s[tid] = tid < L ? expf((float)(w_s[tid] - x_s[LC - 1])) : 0.f;
    if (blockIdx.z == 0) {
      MlRun& run = runs[(int64_t)blockIdx.x * a.H + h];
      run.b[tid] = b_s[tid];
      run.w[tid] = w_s[tid];
      run.x[tid] = x_s[tid];
    }
  }
  __syncthreads();
  {
    const float* src = a.proj + (int64_t)tok0 * a.ld + a.off_v + (int64_t)h * V + v0;
    constexpr int per = VT / VEC;
#pragma unroll 4
    for (int i = tid; i < LC * per; i += THREADS) {
      const int r = i / per, c = (i - r * per) * VEC;
      float v[VEC] = {};
      if (r < L && v0 + c < V) ldv<VEC>(src + (int64_t)r * a.ld + c, v);
#pragma unroll
      for (int j = 0; j < VEC; ++j) v[j] *= u_s[r];
      stv<VEC>(Vc + r * VT + c, v);
    }
  }
  __syncthreads();
  // a thread: rows d0 + 4 ty .. + 3 and columns 4 tx .. + 3; one 16-byte load of each operand a token
  const int ty = tid / 16, tx = tid % 16;
  float* out = states + ((int64_t)blockIdx.x * a.H + h) * D * V;
  for (int d0 = 0; d0 < D; d0 += 64) {
    float acc[4][4] = {};
#pragma unroll 8
    for (int s = 0; s < LC; ++s) {              // (rows beyond L are zero)
      float kk[4], vv[4];
      ld4(Kt + s * ldk + d0 + 4 * ty, kk);
      ld4(Vc + s * VT + 4 * tx, vv);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(kk[i], vv[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = d0 + 4 * ty + i;
      if (d >= D) continue;
      float* row = out + (int64_t)d * V + v0 + 4 * tx;
      if constexpr (VEC == 4) {
        if (v0 + 4 * tx < V) st4(row, acc[i]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (v0 + 4 * tx + j < V) row[j] = acc[i][j];
      }
    }
  }
  if (blockIdx.z == 0) {
    for (int d = tid; d < D; d += THREADS) {
      float sum = 0.f;
#pragma unroll 8
      for (int s = 0; s < LC; ++s) sum = fmaf(u_s[s], Kt[s * ldk + d], sum);
      key_sums[((int64_t)blockIdx.x * a.H + h) * D + d] = sum;
    }
  }
}

// One block = one request (first_req + blockIdx.x) x one head x WALK VEC elements of S and, behind them, n; a thread walks VEC neighbours.
constexpr int WALK = 128;

template <int VEC>
__global__ void __launch_bounds__(WALK, 8)
ml_walk_kernel(MlstmArgs a, MlRun* runs, float* states, float* key_sums, const int* __restrict__ tiles, int n_tiles, int first_req) {
  __shared__ int first_tile;
  const int b = first_req + blockIdx.x, h = blockIdx.y, D = a.D, DV = a.D * a.V;
  const int e = (blockIdx.z * WALK + threadIdx.x) * VEC;
  const int slot = a.slots[b], tok0 = a.cu[b], n_tok = a.cu[b + 1] - tok0;
  if (threadIdx.x == 0) first_tile = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < n_tiles; i += WALK)              // a request's runs follow one another in the list
    if (tiles[2 * i] == b && tiles[2 * i + 1] == 0) first_tile = i;
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();
  const int c0 = first_tile;
  if (slot < 0 || n_tok <= 0 || c0 < 0 || e >= DV + D) return;
  const bool fresh = a.ctx[b] == n_tok, in_s = e < DV;           // (DV is a multiple of VEC)
  float* state = in_s ? a.S + ((int64_t)slot * a.H + h) * DV + e : a.n + ((int64_t)slot * a.H + h) * D + (e - DV);
  float* st = in_s ? states + ((int64_t)c0 * a.H + h) * DV + e : key_sums + ((int64_t)c0 * a.H + h) * D + (e - DV);
  const int64_t step = (int64_t)a.H * (in_s ? DV : D);
  float S[VEC] = {};
  if (!fresh) ldv<VEC>(state, S);
  float m0 = fresh ? 0.f : a.m[(int64_t)slot * a.H + h];
  const int n_runs = (n_tok + LC - 1) / LC;
  MlRun* run = runs + (int64_t)c0 * a.H + h;
  // The loads of the next AHEAD runs are on their way while these runs' states are stored.
  constexpr int AHEAD = 4;
  float u[2][AHEAD][VEC];
  double bl[2][AHEAD], xl[2][AHEAD];
  auto fetch = [&](int into, int c1) {
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      const int c = min(c1 + j, n_runs - 1);
      ldv<VEC>(st + c * step, u[into][j]);
      bl[into][j] = run[(int64_t)c * a.H].b[LC - 1];
      xl[into][j] = run[(int64_t)c * a.H].x[LC - 1];
    }
  };
  fetch(0, 0);
  for (int pair = 0; pair < n_runs; pair += 2 * AHEAD) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int c1 = pair + half * AHEAD;
      if (c1 >= n_runs) break;
      if (c1 + AHEAD < n_runs) fetch(half ^ 1, c1 + AHEAD);
#pragma unroll
      for (int j = 0; j < AHEAD; ++j) {
        if (c1 + j < n_runs) {
          stv<VEC>(st + (c1 + j) * step, S);
          const float m1 = (float)(bl[half][j] + fmax((double)m0, xl[half][j]));
          const float f = expf((float)(bl[half][j] + m0 - m1)), g = expf((float)(bl[half][j] + xl[half][j] - m1));
          if (e == 0) {
            run[(int64_t)(c1 + j) * a.H].m0 = m0;
            run[(int64_t)(c1 + j) * a.H].m1 = m1;
          }
#pragma unroll
          for (int k = 0; k < VEC; ++k) S[k] = fmaf(f, S[k], g * u[half][j][k]);
          m0 = m1;
        }
      }
    }
  }
  stv<VEC>(state, S);           // (m is stored by the next kernel: other blocks of this one still read it)
}

// states[c] and key_sums[c] hold the state in front of the run.
template <int VEC>
__global__ void __launch_bounds__(THREADS)
ml_out_kernel(MlstmArgs a, const int* __restrict__ tiles, const float* __restrict__ states, const float* __restrict__ key_sums,
              const MlRun* __restrict__ runs) {
  extern __shared__ __align__(16) float smem[];
  __shared__ double top_s[LC], w_s[LC];         // m_t - b_t, gi_t - b_t
  __shared__ float c_s[LC], em_s[LC], den_s[LC];
  constexpr int lda = LC + 4;
  const int D = a.D, V = a.V, D4 = (D + 3) / 4 * 4, ldq = D4 + 4;
  float* Q = smem;                              // [LC][ldq], times q_scale
  float* K = Q + LC * ldq;                      // [LC][ldq], later the state [D4][VT]
  float* A = K + max(LC * ldq, D4 * VT);        // [LC][lda]
  float* Vs = A + LC * lda;                     // [LC][VT]
  float* n_s = Vs + LC * VT;                    // [D4]
  const int tid = threadIdx.x, h = blockIdx.y, v0 = blockIdx.z * VT;
  const int b = tiles[2 * blockIdx.x], q0 = tiles[2 * blockIdx.x + 1], slot = a.slots[b];
  const int tok0 = a.cu[b] + q0, left = a.cu[b + 1] - tok0, L = min(LC, left);
  pdl_wait();
  pdl_launch_dependents();
  if (L <= 0 || slot < 0) return;
  const MlRun& run = runs[(int64_t)blockIdx.x * a.H + h];
  if (tid < LC) {
    const double top = fmax((double)run.m0, run.x[tid]);
    top_s[tid] = top;
    w_s[tid] = run.w[tid];
    c_s[tid] = expf((float)(run.m0 - top));
    em_s[tid] = expf(-(float)(run.b[tid] + top));
    if (tid == 0 && blockIdx.z == 0 && left <= LC) a.m[(int64_t)slot * a.H + h] = run.m1;
  }
  const float* rows = a.proj + (int64_t)tok0 * a.ld;
  fill<VEC>(Q, ldq, LC, D4, rows + a.off_q + (int64_t)h * D, a.ld, L, D, a.q_scale);
  fill<VEC>(K, ldq, LC, D4, rows + a.off_k + (int64_t)h * D, a.ld, L, D);
  fill<VEC>(Vs, VT, LC, VT, rows + a.off_v + (int64_t)h * V + v0, a.ld, L, V - v0);
  for (int d = tid; d < D4; d += THREADS) n_s[d] = d < D ? key_sums[((int64_t)blockIdx.x * a.H + h) * D + d] : 0.f;
  __syncthreads();
  const int ty = tid / 16, tx = tid % 16;
  {
    float sc[4][4] = {};
    for (int d = 0; d < D4; d += 4) {
      float x[4][4], y[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ld4(Q + (ty + 16 * i) * ldq + d, x[i]);
        ld4(K + (tx + 16 * i) * ldq + d, y[i]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k) sc[i][j] = fmaf(x[i][k], y[j][k], sc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = ty + 16 * i, s = tx + 16 * j;
        A[t * lda + s] = s <= t && t < L ? sc[i][j] * expf((float)(w_s[s] - top_s[t])) : 0.f;
      }
  }
  __syncthreads();                              // K is read, A is written
  fill<VEC>(K, VT, D4, VT, states + ((int64_t)blockIdx.x * a.H + h) * D * V + v0, V, D, V - v0);
  {   // the denominators: n_t . q_t = sum_s A[t][s] + c_t (q_t . n0), four threads a token
    const int t = tid / 4, part = tid % 4;
    float rs = 0.f, qn = 0.f;
    for (int s = part; s < LC; s += 4) rs += A[t * lda + s];
    for (int d = part; d < D4; d += 4) qn = fmaf(Q[t * ldq + d], n_s[d], qn);
    float nq = fmaf(c_s[t], qn, rs);
    nq += __shfl_xor_sync(0xffffffffu, nq, 1);
    nq += __shfl_xor_sync(0xffffffffu, nq, 2);
    if (part == 0) den_s[t] = fmaxf(fabsf(nq), em_s[t]) + 1e-6f;
  }
  __syncthreads();
  // a thread: rows ty + 16 i and columns 4 tx .. + 3; four terms a turn with 16-byte loads of both operands
  float acc[4][4] = {};
  auto product = [&](const float* X, int ldx, const float* Y, int n) {
#pragma unroll 2
    for (int c = 0; c < n; c += 4) {
      float xx[4][4], yy[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) ld4(X + (ty + 16 * i) * ldx + c, xx[i]);
#pragma unroll
      for (int k = 0; k < 4; ++k) ld4(Y + (c + k) * VT + 4 * tx, yy[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xx[i][k], yy[k][j], acc[i][j]);
    }
  };
  product(Q, ldq, K, D4);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] *= c_s[ty + 16 * i];
  product(A, lda, Vs, LC);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = ty + 16 * i;
    if (t >= L) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] /= den_s[t];
    float* row = a.o + (int64_t)(tok0 + t) * a.H * V + (int64_t)h * V + v0 + 4 * tx;
    if constexpr (VEC == 4) {
      if (v0 + 4 * tx < V) st4(row, acc[i]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (v0 + 4 * tx + j < V) row[j] = acc[i][j];
    }
  }
}

size_t state_smem(int D) { return sizeof(float) * ((size_t)LC * ((D + 63) / 64 * 64 + 4) + LC * VT); }
size_t out_smem(int D) {
  const size_t D4 = (D + 3) / 4 * 4, q = LC * (D4 + 4), s = D4 * VT;
  return sizeof(float) * (q + (q > s ? q : s) + LC * (LC + 4) + LC * VT + D4);
}

template <typename K>
int raise_smem(K kernel, size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  ME_REQUIRE(e == cudaSuccess, "me_mlstm_scan: cannot raise shared memory to %zu: %s", smem, cudaGetErrorString(e));
  return 0;
}

template <int VEC>
int launch_runs(const MlstmArgs& a, int first_req, int B, const int* tiles, int n_tiles, float* states, MlRun* runs, cudaStream_t stream) {
  const unsigned v_tiles = (a.V + VT - 1) / VT;
  float* key_sums = states + (int64_t)n_tiles * a.H * a.D * a.V;
  if (raise_smem(ml_state_kernel<VEC>, state_smem(a.D)) || raise_smem(ml_out_kernel<VEC>, out_smem(a.D))) return 1;
  me_launch(ml_state_kernel<VEC>, dim3(n_tiles, a.H, v_tiles), dim3(THREADS), state_smem(a.D), stream, a, tiles, states, key_sums, runs);
  ME_LAUNCH_CHECK("me_mlstm_scan (runs' states)");
  const int64_t elements = ((int64_t)a.D * a.V + a.D + VEC - 1) / VEC;
  me_launch(ml_walk_kernel<VEC>, dim3(B - first_req, a.H, (unsigned)((elements + WALK - 1) / WALK)), dim3(WALK), 0, stream, a, runs, states,
            key_sums, tiles, n_tiles, first_req);
  ME_LAUNCH_CHECK("me_mlstm_scan (walk)");
  me_launch(ml_out_kernel<VEC>, dim3(n_tiles, a.H, v_tiles), dim3(THREADS), out_smem(a.D), stream, a, tiles, states, key_sums, runs);
  ME_LAUNCH_CHECK("me_mlstm_scan (runs' outputs)");
  return 0;
}

}  // namespace

ME_API int me_mlstm_chunk_len() { return LC; }
ME_API int me_mlstm_run_bytes() { return (int)sizeof(MlRun); }      // what a run and head takes of ``runs_ws``

// (the state kernel's launch, and elements of S in an int)
bool mlstm_runs_take(const MlstmArgs& a) {
  return a.D <= 256 && (a.V + VT - 1) / VT <= 65535 && ((int64_t)a.D * a.V + a.D + WALK - 1) / WALK <= 65535;
}

int mlstm_runs(const MlstmArgs& a, int first_req, int B, const int* tiles, int n_tiles, float* states, void* runs, cudaStream_t stream) {
  ME_REQUIRE((uintptr_t)states % 16 == 0 && (uintptr_t)runs % 16 == 0, "me_mlstm_scan: the workspaces must start on 16 bytes");
  auto on = [](const float* p) { return (uintptr_t)p % 16 == 0; };
  const bool vec = a.D % 4 == 0 && a.V % 4 == 0 && a.ld % 4 == 0 && a.off_q % 4 == 0 && a.off_k % 4 == 0 && a.off_v % 4 == 0 && on(a.proj) &&
                   on(a.S) && on(a.n) && on(a.o);
  MlRun* r = reinterpret_cast<MlRun*>(runs);
  return vec ? launch_runs<4>(a, first_req, B, tiles, n_tiles, states, r, stream) : launch_runs<1>(a, first_req, B, tiles, n_tiles, states, r, stream);
}
