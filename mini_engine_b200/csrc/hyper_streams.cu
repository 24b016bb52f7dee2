// Several residual streams ("hyper-connections") and the layer norm that reads them, in one pass over a token.
//
// A model may keep S copies x_1 .. x_S of the residual stream.  A sub-layer reads u = sum_s in[s] x_s, and its
// output y goes back into all streams at once: x'_r = sum_s mix[s, r] x_s + out[r] y.  The kernel applies the
// update that the sub-layer before left pending (if any), forms the next sub-layer's input u from the new
// streams and normalises it: (u - mean) / sqrt(var + eps) * w with var the mean squared deviation (a layer norm
// with a weight and no bias).  S = 1 with mix = out = in = 1 is the ordinary residual sum x += y.  With ``rows``
// only those tokens are read and nothing is written back (the model's last norm at the wanted places); without
// ``in`` every stream counts once (the sum of the streams).  Streams, sums and statistics are float32.
#include "common.cuh"
#include "vec4.cuh"

constexpr int HC_MAX_STREAMS = 16;

// NS: the number of streams the loops are unrolled for (S <= NS)
template <typename TY, typename TO, int NS>
__global__ void __launch_bounds__(256, 4)
hc_norm_kernel(float* __restrict__ x, int64_t stream_stride, int S, const TY* __restrict__ y,
               const float* __restrict__ mix, const float* __restrict__ outw, const float* __restrict__ inw,
               const float* __restrict__ normw, float eps, TO* __restrict__ out, const int* __restrict__ rows, int W,
               const float* __restrict__ conv_w, float* __restrict__ conv_state, const int* __restrict__ state_slots,
               const int* __restrict__ context_lens, int taps) {
  extern __shared__ float u_s[];               // the token's u, W floats
  __shared__ float red[32];
  __shared__ float c_mix[HC_MAX_STREAMS * HC_MAX_STREAMS], c_out[HC_MAX_STREAMS], c_in[HC_MAX_STREAMS];
  const int tid = threadIdx.x;
  for (int i = tid; i < S * S; i += blockDim.x) c_mix[i] = mix ? mix[i] : 0.f;
  for (int i = tid; i < S; i += blockDim.x) {
    c_out[i] = outw ? outw[i] : 0.f;
    c_in[i] = inw ? inw[i] : 1.f;
  }
  pdl_wait();
  pdl_launch_dependents();
  __syncthreads();
  const int r_out = blockIdx.x;
  const int64_t t = rows ? rows[r_out] : r_out;
  float sum = 0.f;
  for (int w = tid; w < W; w += blockDim.x) {
    float xs[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s)
      if (s < S) xs[s] = x[s * stream_stride + t * W + w];
    if (y != nullptr) {
      const float yy = to_f<TY>(y[t * W + w]);
      float nx[NS];
#pragma unroll
      for (int r = 0; r < NS; ++r) {
        if (r < S) {
          float a = 0.f;
#pragma unroll
          for (int s = 0; s < NS; ++s)
            if (s < S) a = fmaf(c_mix[s * S + r], xs[s], a);
          nx[r] = fmaf(c_out[r], yy, a);
        }
      }
#pragma unroll
      for (int r = 0; r < NS; ++r) {
        if (r < S) {
          xs[r] = nx[r];
          if (rows == nullptr) x[r * stream_stride + t * W + w] = nx[r];
        }
      }
    }
    float u = 0.f;
#pragma unroll
    for (int s = 0; s < NS; ++s)
      if (s < S) u = fmaf(c_in[s], xs[s], u);
    u_s[w] = u;
    sum += u;
  }
  if (normw == nullptr) return;                 // the update alone
  const float mean = block_sum(sum, red) / (float)W;
  float sq = 0.f;
  for (int w = tid; w < W; w += blockDim.x) {
    const float d = u_s[w] - mean;
    sq = fmaf(d, d, sq);
  }
  const float rstd = 1.0f / sqrtf(block_sum(sq, red) / (float)W + eps);
  if (conv_w == nullptr) {
    for (int w = tid; w < W; w += blockDim.x)
      out[(int64_t)r_out * W + w] = from_f<TO>((u_s[w] - mean) * rstd * normw[w]);
    return;
  }
  // Every request brings one token (token t is request t): the short convolution h + conv(h) of csrc/short_conv.cu
  // needs no other token of the step, only the request's state, which then moves up by one row and takes h.
  const int slot = state_slots[t], pos = context_lens[t] - 1;
  for (int w = tid; w < W; w += blockDim.x) {
    const float h = (u_s[w] - mean) * rstd * normw[w];
    float acc = h;
    if (slot >= 0 && taps > 1) {
      float* st = conv_state + (int64_t)slot * (taps - 1) * W + w;
      for (int j = 0; j < taps - 1; ++j) {
        const bool before_start = pos - (taps - 1) + j < 0;
        const float v = before_start ? 0.f : st[(int64_t)j * W];
        if (!before_start) acc = fmaf(conv_w[(int64_t)w * taps + j], v, acc);
        if (j > 0) st[(int64_t)(j - 1) * W] = v;
      }
      st[(int64_t)(taps - 2) * W] = h;
    }
    acc = fmaf(conv_w[(int64_t)w * taps + taps - 1], h, acc);
    out[(int64_t)r_out * W + w] = from_f<TO>(acc);
  }
}

// The same with a token's row in registers: a thread takes CH runs of four neighbouring values (W a multiple of 4, at most
// 4 CH threads of the block), so that everything a token needs (streams, y, the convolution's state) is requested at once, and the
// weights before the kernel in front has ended.  What it is bound by: one round trip to memory and two sums over the block for
// a few rows (3 rows of 2,048 in four streams with the convolution: 21.7 us with the kernel above, 7.4 with this one), the streams'
// bytes for many (2,787 rows: 68.7 -> 47.9 us, 4.5 TB/s).  TAPS: the convolution's taps (0: none; up to 4, else the kernel above).
template <typename TY, typename TO, int NS, int CH, int TAPS>
__global__ void __launch_bounds__(512)
hc_norm_vec_kernel(float* __restrict__ x, int64_t stream_stride, int S, const TY* __restrict__ y,
                   const float* __restrict__ mix, const float* __restrict__ outw, const float* __restrict__ inw,
                   const float* __restrict__ normw, float eps, TO* __restrict__ out, const int* __restrict__ rows, int W,
                   const float* __restrict__ conv_w, float* __restrict__ conv_state, const int* __restrict__ state_slots,
                   const int* __restrict__ context_lens) {
  __shared__ float red[32];
  __shared__ float c_mix[NS * NS], c_out[NS], c_in[NS];
  const int tid = threadIdx.x;
  for (int i = tid; i < S * S; i += blockDim.x) c_mix[i / S * NS + i % S] = mix ? mix[i] : 0.f;
  for (int i = tid; i < S; i += blockDim.x) {
    c_out[i] = outw ? outw[i] : 0.f;
    c_in[i] = inw ? inw[i] : 1.f;
  }
  int at[CH];
  float nw[CH][4], cw[TAPS ? TAPS : 1][CH][4];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    at[c] = 4 * (tid + c * blockDim.x);
    if (at[c] < W) {
      if (normw) ld4(normw + at[c], nw[c]);
      if (TAPS > 0)
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int j = 0; j < TAPS; ++j) cw[j][c][e] = conv_w[(int64_t)(at[c] + e) * TAPS + j];
    }
  }
  const int r_out = blockIdx.x;
  const int slot = TAPS > 0 ? state_slots[r_out] : -1, pos = TAPS > 0 ? context_lens[r_out] - 1 : 0;
  pdl_wait();
  pdl_launch_dependents();
  __syncthreads();
  const int64_t t = rows ? rows[r_out] : r_out;
  float xs[NS][CH][4], yy[CH][4], st[TAPS > 1 ? TAPS - 1 : 1][CH][4];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    if (at[c] < W) {
#pragma unroll
      for (int s = 0; s < NS; ++s)
        if (s < S) ld4(x + s * stream_stride + t * W + at[c], xs[s][c]);
      if (y != nullptr) ld4(y + t * W + at[c], yy[c]);
      if (TAPS > 1 && slot >= 0)
#pragma unroll
        for (int j = 0; j < TAPS - 1; ++j) {
          if (pos - (TAPS - 1) + j >= 0) ld4(conv_state + ((int64_t)slot * (TAPS - 1) + j) * W + at[c], st[j][c]);
          else st[j][c][0] = st[j][c][1] = st[j][c][2] = st[j][c][3] = 0.f;
        }
    }
  }
  float u[CH][4], sum = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    if (at[c] >= W) continue;
    if (y != nullptr) {
      float nx[NS][4];
#pragma unroll
      for (int r = 0; r < NS; ++r) {
        if (r < S) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float a = 0.f;
#pragma unroll
            for (int s = 0; s < NS; ++s)
              if (s < S) a = fmaf(c_mix[s * NS + r], xs[s][c][e], a);
            nx[r][e] = fmaf(c_out[r], yy[c][e], a);
          }
          if (rows == nullptr) st4(x + r * stream_stride + t * W + at[c], nx[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < NS; ++r)
        if (r < S)
#pragma unroll
          for (int e = 0; e < 4; ++e) xs[r][c][e] = nx[r][e];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float v = 0.f;
#pragma unroll
      for (int s = 0; s < NS; ++s)
        if (s < S) v = fmaf(c_in[s], xs[s][c][e], v);
      u[c][e] = v;
    }
    sum += (u[c][0] + u[c][1]) + (u[c][2] + u[c][3]);
  }
  if (normw == nullptr) return;                 // the update alone
  const float mean = block_sum_tree(sum, red) / (float)W;
  float sq = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c)
    if (at[c] < W) {
      const float d0 = u[c][0] - mean, d1 = u[c][1] - mean, d2 = u[c][2] - mean, d3 = u[c][3] - mean;
      sq += fmaf(d0, d0, d1 * d1) + fmaf(d2, d2, d3 * d3);
    }
  const float rstd = 1.0f / sqrtf(block_sum_tree(sq, red) / (float)W + eps);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    if (at[c] >= W) continue;
    float h[4], acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = h[e] = (u[c][e] - mean) * rstd * nw[c][e];
    if (TAPS > 0) {
      if (TAPS > 1 && slot >= 0) {
        float* dst = conv_state + (int64_t)slot * (TAPS - 1) * W + at[c];
#pragma unroll
        for (int j = 0; j < TAPS - 1; ++j) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[e] = fmaf(cw[j][c][e], st[j][c][e], acc[e]);
          if (j > 0) st4(dst + (int64_t)(j - 1) * W, st[j][c]);
        }
        st4(dst + (int64_t)(TAPS - 2) * W, h);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = fmaf(cw[TAPS ? TAPS - 1 : 0][c][e], h[e], acc[e]);
    }
    st4(out + (int64_t)r_out * W + at[c], acc);
  }
}

template <typename TY, typename TO, int NS, int CH, int TAPS>
static void launch_hc_norm_vec(float* x, int64_t stream_stride, int S, const void* y, const float* mix, const float* outw, const float* inw,
                               const float* normw, float eps, void* out, const int* rows, int n, int W, int threads, const float* conv_w,
                               float* conv_state, const int* state_slots, const int* context_lens, cudaStream_t stream) {
  me_launch(hc_norm_vec_kernel<TY, TO, NS, CH, TAPS>, dim3(n), dim3(threads), 0, stream, x, stream_stride, S, (const TY*)y, mix, outw, inw,
            normw, eps, (TO*)out, rows, W, conv_w, conv_state, state_slots, context_lens);
}

template <typename TY, typename TO, int NS>
static int launch_hc_norm(float* x, int64_t stream_stride, int S, const void* y, const float* mix, const float* outw,
                          const float* inw, const float* normw, float eps, void* out, const int* rows, int n, int W, int threads,
                          size_t smem, const float* conv_w, float* conv_state, const int* state_slots, const int* context_lens,
                          int taps, cudaStream_t stream) {
  if (smem > 48 * 1024) {
    static bool attr_set = false;
    if (!attr_set) {
      cudaError_t e = cudaFuncSetAttribute(hc_norm_kernel<TY, TO, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
      ME_REQUIRE(e == cudaSuccess, "me_hc_norm: cannot raise shared memory: %s", cudaGetErrorString(e));
      attr_set = true;
    }
  }
  me_launch(hc_norm_kernel<TY, TO, NS>, dim3(n), dim3(threads), smem, stream, x, stream_stride, S, (const TY*)y, mix, outw, inw,
            normw, eps, (TO*)out, rows, W, conv_w, conv_state, state_slots, context_lens, taps);
  return 0;
}

// x: [S, T, W] float32 (streams ``stream_stride`` elements apart).  y: [T, W] of y_dtype or null (no pending update;
// mix and outw are then unused).  inw: [S] or null (ones).  normw: [W] or null (no output).  out: [n, W] of out_dtype,
// n = number of rows if ``rows`` is given, else T.  conv_w [W, taps] (or null): every request brings one token, and the
// output is h + conv(h) with conv_state [slots, taps-1, W] renewed in place (state_slots and context_lens per request).
ME_API int me_hc_norm(float* x, int64_t stream_stride, int S, const void* y, int y_dtype, const float* mix,
                      const float* outw, const float* inw, const float* normw, float eps, void* out, int out_dtype,
                      const int* rows, int n, int W, const float* conv_w, float* conv_state, const int* state_slots,
                      const int* context_lens, int taps, cudaStream_t stream) {
  if (n == 0) return 0;
  ME_REQUIRE(S >= 1 && S <= HC_MAX_STREAMS, "me_hc_norm: %d streams (1 to %d are supported)", S, HC_MAX_STREAMS);
  ME_REQUIRE(n > 0 && W > 0, "me_hc_norm: bad sizes n=%d W=%d", n, W);
  ME_REQUIRE(y == nullptr || (mix != nullptr && outw != nullptr), "me_hc_norm: an update needs mix and out weights");
  ME_REQUIRE(normw == nullptr || out != nullptr, "me_hc_norm: a norm needs an output");
  ME_REQUIRE(conv_w == nullptr || (rows == nullptr && normw != nullptr && taps >= 1 && state_slots != nullptr && context_lens != nullptr
                                   && (taps == 1 || conv_state != nullptr)),
             "me_hc_norm: the convolution needs a norm, all rows, the requests' slots and lengths, and a state");
  // Rows of whole runs of four, up to 4,096 values and four streams, and up to four taps: a row in registers.  Threads: a run each
  // up to 1,024 values, two each beyond.
  if (W % 4 == 0 && W <= 4096 && S <= 4 && stream_stride % 4 == 0 && (conv_w == nullptr || (taps >= 2 && taps <= 4)) && on4(x, ME_F32) && on4(y, y_dtype) &&
      on4(normw, ME_F32) && on4(out, out_dtype) && on4(conv_state, ME_F32)) {
    const int ch = W > 1024 ? 2 : 1, threads = ((W / 4 + ch - 1) / ch + 31) / 32 * 32, tp = conv_w ? taps : 0;
#define HC_VEC(NS_, CH_, TAPS_)                                                                                                                \
  launch_hc_norm_vec<TY, TO, NS_, CH_, TAPS_>(x, stream_stride, S, y, mix, outw, inw, normw, eps, out, rows, n, W, threads, conv_w, conv_state, \
                                              state_slots, context_lens, stream)
#define HC_VEC_TAPS(NS_, CH_)                                                                                                                  \
  do { if (tp == 0) HC_VEC(NS_, CH_, 0); else if (tp == 2) HC_VEC(NS_, CH_, 2); else if (tp == 3) HC_VEC(NS_, CH_, 3); else HC_VEC(NS_, CH_, 4); } while (0)
    ME_DISPATCH_DTYPE(y_dtype, TY, ME_DISPATCH_DTYPE(out_dtype, TO, {
      if (S == 1) { if (ch == 1) HC_VEC_TAPS(1, 1); else HC_VEC_TAPS(1, 2); }
      else { if (ch == 1) HC_VEC_TAPS(4, 1); else HC_VEC_TAPS(4, 2); }
    }));
#undef HC_VEC_TAPS
#undef HC_VEC
    ME_LAUNCH_CHECK("me_hc_norm");
    return 0;
  }
  const size_t smem = sizeof(float) * (size_t)W;
  ME_REQUIRE(smem <= 160 * 1024, "me_hc_norm: width %d is too large", W);
  const int threads = W >= 1024 ? 256 : (W >= 256 ? 128 : 64);
  int rc = 0;
  ME_DISPATCH_DTYPE(y_dtype, TY, ME_DISPATCH_DTYPE(out_dtype, TO, {
    if (S == 1) rc = launch_hc_norm<TY, TO, 1>(x, stream_stride, S, y, mix, outw, inw, normw, eps, out, rows, n, W, threads, smem, conv_w, conv_state, state_slots, context_lens, taps, stream);
    else if (S == 2) rc = launch_hc_norm<TY, TO, 2>(x, stream_stride, S, y, mix, outw, inw, normw, eps, out, rows, n, W, threads, smem, conv_w, conv_state, state_slots, context_lens, taps, stream);
    else if (S <= 4) rc = launch_hc_norm<TY, TO, 4>(x, stream_stride, S, y, mix, outw, inw, normw, eps, out, rows, n, W, threads, smem, conv_w, conv_state, state_slots, context_lens, taps, stream);
    else if (S <= 8) rc = launch_hc_norm<TY, TO, 8>(x, stream_stride, S, y, mix, outw, inw, normw, eps, out, rows, n, W, threads, smem, conv_w, conv_state, state_slots, context_lens, taps, stream);
    else rc = launch_hc_norm<TY, TO, HC_MAX_STREAMS>(x, stream_stride, S, y, mix, outw, inw, normw, eps, out, rows, n, W, threads, smem, conv_w, conv_state, state_slots, context_lens, taps, stream);
  }));
  if (rc) return rc;
  ME_LAUNCH_CHECK("me_hc_norm");
  return 0;
}
