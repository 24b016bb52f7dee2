// The matrix-memory recurrence of xLSTM (mLSTM) with a state slot per request.
//
// Per head, with q (scaled), k of D values, v of V values, a log input gate gi and a log forget gate gf:
//   m_t = max(gf + m_(t-1), gi)
//   S_t = exp(gf + m_(t-1) - m_t) S_(t-1) + exp(gi - m_t) k v^T        (D x V)
//   n_t = exp(gf + m_(t-1) - m_t) n_(t-1) + exp(gi - m_t) k            (D)
//   o_t = S_t^T q / (max(|n_t . q|, exp(-m_t)) + 1e-6)                  (V)
// S, n and m start at zero (m at 0, not at minus infinity).  The gates are capped:
//   gi = cap tanh((x_i + b_i) / cap),   gf = logsigmoid(cap tanh((x_f + b_f) / cap)).
// The scan kernel walks a request's tokens of this step in order from the state its slot holds (from zero when the
// portion starts at position 0) and leaves the new state there; everything is float32, and a token's result does
// not depend on where the sequence was cut.  One block = one request x one head x MLSTM_VB (16) columns of S; the
// blocks of a head each keep n and m.  They are stored by a kernel behind (mlstm_norm_kernel), since blocks that start late
// still read what the slot held.  Portions of prompts run 64 tokens at a time, all runs of a step side by side (mlstm_runs.cu).
// A further kernel divides each head's o by its root mean square and applies the weight and the output gate.
#include "mlstm.cuh"

constexpr int MLSTM_VB = 16, MLSTM_DY = 16, MLSTM_THREADS = MLSTM_VB * MLSTM_DY;

__global__ void __launch_bounds__(MLSTM_THREADS)
mlstm_scan_kernel(const float* __restrict__ proj, int64_t ld, int off_q, int off_k, int off_v, int off_i, int off_f,
                  const float* __restrict__ bias_i, const float* __restrict__ bias_f, float cap,
                  float* __restrict__ S_state, float* __restrict__ n_state, float* __restrict__ m_state,
                  const int* __restrict__ cu_seqlens, const int* __restrict__ context_lens,
                  const int* __restrict__ state_slots, float* __restrict__ o, int H, int D, int V, float q_scale) {
  extern __shared__ float smem[];
  __shared__ float red[32];
  float* S = smem;                              // [D][MLSTM_VB + 1]
  float* q_s = S + D * (MLSTM_VB + 1);          // [D]
  float* k_s = q_s + D;                         // [D]
  float* n_s = k_s + D;                         // [D]
  float* parts = n_s + D;                       // [MLSTM_DY][MLSTM_VB]
  const int b = blockIdx.x, hd = blockIdx.y, v0 = blockIdx.z * MLSTM_VB;
  const int tid = threadIdx.x, vc = tid % MLSTM_VB, dy = tid / MLSTM_VB;
  const bool v_ok = v0 + vc < V;
  const float bi = bias_i[hd], bf_ = bias_f[hd];
  pdl_wait();
  pdl_launch_dependents();
  const int slot = state_slots[b];
  const int tok0 = cu_seqlens[b], n_tok = cu_seqlens[b + 1] - tok0;
  if (slot < 0 || n_tok <= 0) return;
  const bool fresh = context_lens[b] - n_tok == 0;
  float* Sg = S_state + ((int64_t)slot * H + hd) * D * V;
  float* ng = n_state + ((int64_t)slot * H + hd) * D;
  for (int d = dy; d < D; d += MLSTM_DY) S[d * (MLSTM_VB + 1) + vc] = (fresh || !v_ok) ? 0.f : Sg[(int64_t)d * V + v0 + vc];
  for (int d = tid; d < D; d += MLSTM_THREADS) n_s[d] = fresh ? 0.f : ng[d];
  float m = fresh ? 0.f : m_state[(int64_t)slot * H + hd];
  for (int i = 0; i < n_tok; ++i) {
    const float* row = proj + (int64_t)(tok0 + i) * ld;
    __syncthreads();                            // the token before is done with q_s, k_s, parts
    for (int d = tid; d < D; d += MLSTM_THREADS) {
      q_s[d] = row[off_q + hd * D + d] * q_scale;
      k_s[d] = row[off_k + hd * D + d];
    }
    const float gi = mlstm_capped(row[off_i + hd] + bi, cap), gf = mlstm_log_sigmoid(mlstm_capped(row[off_f + hd] + bf_, cap));
    const float m_new = fmaxf(gf + m, gi);
    const float fa = expf(gf + m - m_new), fb = expf(gi - m_new);
    const float vv = v_ok ? row[off_v + hd * V + v0 + vc] : 0.f;
    __syncthreads();
    float nq = 0.f;
    for (int d = tid; d < D; d += MLSTM_THREADS) {
      const float nn = fmaf(fa, n_s[d], fb * k_s[d]);
      n_s[d] = nn;
      nq = fmaf(nn, q_s[d], nq);
    }
    nq = block_sum(nq, red);
    float part = 0.f;
    for (int d = dy; d < D; d += MLSTM_DY) {
      const float s = fmaf(fa, S[d * (MLSTM_VB + 1) + vc], fb * k_s[d] * vv);
      S[d * (MLSTM_VB + 1) + vc] = s;
      part = fmaf(s, q_s[d], part);
    }
    parts[dy * MLSTM_VB + vc] = part;
    __syncthreads();
    if (dy == 0 && v_ok) {
      float tot = 0.f;
#pragma unroll
      for (int y = 0; y < MLSTM_DY; ++y) tot += parts[y * MLSTM_VB + vc];
      const float den = fmaxf(fabsf(nq), expf(-m_new)) + 1e-6f;
      o[(int64_t)(tok0 + i) * H * V + hd * V + v0 + vc] = tot / den;
    }
    m = m_new;
  }
  __syncthreads();
  if (v_ok)
    for (int d = dy; d < D; d += MLSTM_DY) Sg[(int64_t)d * V + v0 + vc] = S[d * (MLSTM_VB + 1) + vc];
}

// n and m behind the step's tokens: one block = one request x one head, a thread every 128th key channel.
__global__ void __launch_bounds__(128)
mlstm_norm_kernel(MlstmArgs a) {
  const int b = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, D = a.D;
  const float bi = a.bias_i[h], bf_ = a.bias_f[h];
  const int slot = a.slots[b], tok0 = a.cu[b], n_tok = a.cu[b + 1] - tok0;
  pdl_wait();
  pdl_launch_dependents();
  if (slot < 0 || n_tok <= 0) return;
  const bool fresh = a.ctx[b] == n_tok;
  float* ng = a.n + ((int64_t)slot * a.H + h) * D;
  const float m_old = fresh ? 0.f : a.m[(int64_t)slot * a.H + h];
  float m = m_old;
  for (int d = tid; d < D || d == tid; d += 128) {
    const bool on = d < D;
    float n = fresh || !on ? 0.f : ng[d];
    m = m_old;
    for (int i = 0; i < n_tok; ++i) {
      const float* row = a.proj + (int64_t)(tok0 + i) * a.ld;
      const float gi = mlstm_capped(row[a.off_i + h] + bi, a.cap), gf = mlstm_log_sigmoid(mlstm_capped(row[a.off_f + h] + bf_, a.cap));
      const float m_new = fmaxf(gf + m, gi);
      n = fmaf(expf(gf + m - m_new), n, expf(gi - m_new) * (on ? row[a.off_k + h * D + d] : 0.f));
      m = m_new;
    }
    if (on) ng[d] = n;
  }
  __syncthreads();                              // everyone has read m
  if (tid == 0) a.m[(int64_t)slot * a.H + h] = m;
}

// out[t, h*V + v] = o / sqrt(mean_v(o^2) + eps) * w[h*V + v] * sigmoid(g[t, h*V + v]); one warp a head.  ``w_shared``: the
// weight has V values that all heads share (w[v]); ``gate_mode`` 1: the gate is g * sigmoid(g) instead of sigmoid(g), 2: none.
// Rows of ``out`` lie out_ld elements apart.
template <typename TO>
__global__ void __launch_bounds__(128)
mlstm_out_kernel(const float* __restrict__ o, const float* __restrict__ proj, int64_t ld, int off_g,
                 const float* __restrict__ w, float eps, TO* __restrict__ out, int64_t out_ld, int H, int V, int w_shared, int gate_mode) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int hd = warp; hd < H; hd += nw) {
    const float* oo = o + ((int64_t)t * H + hd) * V;
    float ss = 0.f;
    for (int v = lane; v < V; v += 32) ss = fmaf(oo[v], oo[v], ss);
    const float r = 1.0f / sqrtf(warp_sum(ss) / (float)V + eps);
    for (int v = lane; v < V; v += 32) {
      float gate = 1.0f;
      if (gate_mode != 2) {
        const float g = proj[(int64_t)t * ld + off_g + hd * V + v];
        gate = (gate_mode ? g : 1.0f) / (1.0f + expf(-g));
      }
      out[(int64_t)t * out_ld + hd * V + v] = from_f<TO>(oo[v] * r * w[w_shared ? v : hd * V + v] * gate);
    }
  }
}

// The same sums with a head's values in registers, every 32nd of them a lane as above (V at most 32 CH), and one head a warp, so that
// everything is requested at once: a few rows take one round trip to memory instead of one a turn (8 heads of 256: 13.4 -> 4.2 us
// a launch, the mean of six launches of 3 rows and one of 2,787).  Four neighbouring values a lane would give other sums.
template <typename TO, int CH>
__global__ void __launch_bounds__(128)
mlstm_out_regs_kernel(const float* __restrict__ o, const float* __restrict__ proj, int64_t ld, int off_g,
                      const float* __restrict__ w, float eps, TO* __restrict__ out, int64_t out_ld, int H, int V, int w_shared, int gate_mode) {
  const int t = blockIdx.x, lane = threadIdx.x & 31, hd = blockIdx.y * 4 + (threadIdx.x >> 5);
  float ww[CH];
  if (hd < H)
#pragma unroll
    for (int c = 0; c < CH; ++c)
      if (lane + 32 * c < V) ww[c] = w[(w_shared ? 0 : hd * V) + lane + 32 * c];
  pdl_wait();
  pdl_launch_dependents();
  if (hd >= H) return;
  const float* oo = o + ((int64_t)t * H + hd) * V + lane;
  const float* gg = proj + (int64_t)t * ld + off_g + hd * V + lane;
  float x[CH], g[CH], ss = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c)
    if (lane + 32 * c < V) {
      x[c] = oo[32 * c];
      if (gate_mode != 2) g[c] = gg[32 * c];
    }
#pragma unroll
  for (int c = 0; c < CH; ++c)
    if (lane + 32 * c < V) ss = fmaf(x[c], x[c], ss);
  const float r = 1.0f / sqrtf(warp_sum(ss) / (float)V + eps);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    if (lane + 32 * c >= V) continue;
    const float gate = gate_mode == 2 ? 1.0f : (gate_mode ? g[c] : 1.0f) / (1.0f + expf(-g[c]));
    out[(int64_t)t * out_ld + hd * V + lane + 32 * c] = from_f<TO>(x[c] * r * ww[c] * gate);
  }
}

// proj: [T, ld] float32 rows holding q, k (H*D each), v, g (H*V each), i, f (H each) at the given column offsets.
// S_state [slots, H, D, V], n_state [slots, H, D], m_state [slots, H] float32.  o: [T, H*V] float32 work buffer.  Requests
// [0, num_decodes) are walked token by token.  The others too, unless ``tiles`` ([n_tiles, 2] int32: request and first token of every
// run of MLSTM_LC tokens of the requests from num_decodes on, a request's runs in order and side by side), ``states_ws`` (float32
// [n_tiles, H, D, V] and behind it [n_tiles, H, D]) and ``runs_ws`` (n_tiles * H times me_mlstm_run_bytes), both on 16 bytes, are given and D is at most 256.
ME_API int me_mlstm_scan(const float* proj, int64_t ld, int off_q, int off_k, int off_v, int off_i, int off_f,
                         const float* bias_i, const float* bias_f, float cap, float* S_state, float* n_state, float* m_state,
                         const int* cu_seqlens, const int* context_lens, const int* state_slots, float* o, int B, int H, int D,
                         int V, float q_scale, int num_decodes, const int* tiles, int n_tiles, float* states_ws, void* runs_ws, cudaStream_t stream) {
  if (B == 0) return 0;
  ME_REQUIRE(B > 0 && H > 0 && D > 0 && V > 0 && cap > 0.f, "me_mlstm_scan: bad sizes B=%d H=%d D=%d V=%d cap=%g", B, H, D, V, cap);
  ME_REQUIRE(H <= 65535, "me_mlstm_scan: too many heads");
  ME_REQUIRE(num_decodes >= 0 && num_decodes <= B, "me_mlstm_scan: %d single-token requests of %d", num_decodes, B);
  const MlstmArgs a = {proj, ld, off_q, off_k, off_v, off_i, off_f, bias_i, bias_f, cap, S_state, n_state, m_state, cu_seqlens, context_lens,
                       state_slots, o, H, D, V, q_scale};
  const bool runs = tiles && states_ws && runs_ws && n_tiles > 0 && num_decodes < B && mlstm_runs_take(a);
  const int n_scan = runs ? num_decodes : B;
  if (n_scan > 0) {
    const size_t smem = sizeof(float) * ((size_t)D * (MLSTM_VB + 1) + 3 * (size_t)D + MLSTM_DY * MLSTM_VB);
    ME_REQUIRE(smem <= 200 * 1024, "me_mlstm_scan: head size %d is too large", D);
    if (smem > 48 * 1024) {
      static bool attr_set = false;
      if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(mlstm_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        ME_REQUIRE(e == cudaSuccess, "me_mlstm_scan: cannot raise shared memory: %s", cudaGetErrorString(e));
        attr_set = true;
      }
    }
    me_launch(mlstm_scan_kernel, dim3(n_scan, H, (V + MLSTM_VB - 1) / MLSTM_VB), dim3(MLSTM_THREADS), smem, stream, proj, ld, off_q,
              off_k, off_v, off_i, off_f, bias_i, bias_f, cap, S_state, n_state, m_state, cu_seqlens, context_lens, state_slots, o,
              H, D, V, q_scale);
    ME_LAUNCH_CHECK("me_mlstm_scan");
    me_launch(mlstm_norm_kernel, dim3(n_scan, H), dim3(128), 0, stream, a);
    ME_LAUNCH_CHECK("me_mlstm_scan (n and m)");
  }
  if (runs) return mlstm_runs(a, num_decodes, B, tiles, n_tiles, states_ws, runs_ws, stream);
  return 0;
}

ME_API int me_mlstm_out(const float* o, const float* proj, int64_t ld, int off_g, const float* w, float eps, void* out,
                        int out_dtype, int64_t out_ld, int T, int H, int V, int w_shared, int gate_mode, cudaStream_t stream) {
  if (T == 0) return 0;
  ME_REQUIRE(T > 0 && H > 0 && V > 0 && out_ld >= (int64_t)H * V, "me_mlstm_out: bad sizes T=%d H=%d V=%d", T, H, V);
  ME_REQUIRE(gate_mode >= 0 && gate_mode <= 2 && (gate_mode == 2 || proj), "me_mlstm_out: gate mode %d", gate_mode);
  if (V <= 512 && (H + 3) / 4 <= 65535) {
#define MO_CASE(CH_)                                                                                                                  \
  me_launch(mlstm_out_regs_kernel<TO, CH_>, dim3(T, (H + 3) / 4), dim3(128), 0, stream, o, proj, ld, off_g, w, eps, (TO*)out, out_ld, H, V, \
            w_shared, gate_mode)
    ME_DISPATCH_DTYPE(out_dtype, TO, { if (V <= 128) MO_CASE(4); else if (V <= 256) MO_CASE(8); else MO_CASE(16); });
#undef MO_CASE
    ME_LAUNCH_CHECK("me_mlstm_out");
    return 0;
  }
  ME_DISPATCH_DTYPE(out_dtype, TO, me_launch(mlstm_out_kernel<TO>, dim3(T), dim3(128), 0, stream, o, proj, ld, off_g, w, eps,
                                             (TO*)out, out_ld, H, V, w_shared, gate_mode));
  ME_LAUNCH_CHECK("me_mlstm_out");
  return 0;
}
