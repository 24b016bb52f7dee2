// PolyNorm activation over a token's vector z of F values:
//   out = a N(z) + b N(z^2) + c N(z^3) + e,   N(v) = v / sqrt(mean(v^2) + eps),
// powers taken element by element.  The three mean squares are mean(z^2), mean(z^4), mean(z^6); sums and
// factors are float32, the result is rounded once to the output's dtype.
#include "common.cuh"
#include "vec4.cuh"

template <typename TZ, typename TO>
__global__ void __launch_bounds__(256)
polynorm_kernel(const TZ* __restrict__ z, int64_t ldz, const float* __restrict__ coef, float eps, TO* __restrict__ out,
                int64_t ldo, int F) {
  __shared__ float red[32];
  const float a = coef[0], b = coef[1], c = coef[2], e = coef[3];
  pdl_wait();
  pdl_launch_dependents();
  const TZ* zr = z + (int64_t)blockIdx.x * ldz;
  float s2 = 0.f, s4 = 0.f, s6 = 0.f;
  for (int f = threadIdx.x; f < F; f += blockDim.x) {
    const float v = to_f<TZ>(zr[f]), v2 = v * v;
    s2 += v2;
    s4 = fmaf(v2, v2, s4);
    s6 = fmaf(v2 * v, v2 * v, s6);
  }
  const float r1 = 1.0f / sqrtf(block_sum(s2, red) / (float)F + eps);
  const float r2 = 1.0f / sqrtf(block_sum(s4, red) / (float)F + eps);
  const float r3 = 1.0f / sqrtf(block_sum(s6, red) / (float)F + eps);
  TO* o = out + (int64_t)blockIdx.x * ldo;
  for (int f = threadIdx.x; f < F; f += blockDim.x) {
    const float v = to_f<TZ>(zr[f]), v2 = v * v;
    o[f] = from_f<TO>(a * (v * r1) + b * (v2 * r2) + c * (v2 * v * r3) + e);
  }
}

// The same with the row in registers: up to CH runs of four neighbouring values a thread (F a multiple of 4), all requested before the
// first is used; the three sums cross the block together.  Rows of 8,192, float32 to bfloat16, the mean of six launches of 3 rows and one
// of 2,787 (137 MB): 20.9 -> 8.2 us.
template <typename TZ, typename TO, int CH>
__global__ void __launch_bounds__(512)
polynorm_vec_kernel(const TZ* __restrict__ z, int64_t ldz, const float* __restrict__ coef, float eps, TO* __restrict__ out,
                    int64_t ldo, int F) {
  __shared__ float red[3][16];
  const float a = coef[0], b = coef[1], c = coef[2], e = coef[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  pdl_wait();
  pdl_launch_dependents();
  const TZ* zr = z + (int64_t)blockIdx.x * ldz;
  float v[CH][4];
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const int f = 4 * (tid + i * blockDim.x);
    if (f < F) ld4(zr + f, v[i]);
    else v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.f;
  }
  float s2 = 0.f, s4 = 0.f, s6 = 0.f;
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    float x2[4], x3[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x2[k] = v[i][k] * v[i][k];
      x3[k] = x2[k] * v[i][k];
    }
    s2 += (x2[0] + x2[1]) + (x2[2] + x2[3]);
    s4 += fmaf(x2[0], x2[0], x2[1] * x2[1]) + fmaf(x2[2], x2[2], x2[3] * x2[3]);
    s6 += fmaf(x3[0], x3[0], x3[1] * x3[1]) + fmaf(x3[2], x3[2], x3[3] * x3[3]);
  }
  s2 = warp_sum(s2);
  s4 = warp_sum(s4);
  s6 = warp_sum(s6);
  if (lane == 0) {
    red[0][warp] = s2;
    red[1][warp] = s4;
    red[2][warp] = s6;
  }
  __syncthreads();
  s2 = warp_sum(lane < warps ? red[0][lane] : 0.f);
  s4 = warp_sum(lane < warps ? red[1][lane] : 0.f);
  s6 = warp_sum(lane < warps ? red[2][lane] : 0.f);
  const float r1 = 1.0f / sqrtf(s2 / (float)F + eps), r2 = 1.0f / sqrtf(s4 / (float)F + eps), r3 = 1.0f / sqrtf(s6 / (float)F + eps);
  TO* o = out + (int64_t)blockIdx.x * ldo;
#pragma unroll
  for (int i = 0; i < CH; ++i) {
    const int f = 4 * (tid + i * blockDim.x);
    if (f >= F) continue;
    float y[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float x = v[i][k], x2 = x * x;
      y[k] = a * (x * r1) + b * (x2 * r2) + c * (x2 * x * r3) + e;
    }
    st4(o + f, y);
  }
}

ME_API int me_polynorm(const void* z, int z_dtype, int64_t ldz, const float* coef, float eps, void* out, int out_dtype,
                       int64_t ldo, int T, int F, cudaStream_t stream) {
  if (T == 0) return 0;
  ME_REQUIRE(T > 0 && F > 0, "me_polynorm: bad sizes T=%d F=%d", T, F);
  if (F % 4 == 0 && F <= 16384 && ldz % 4 == 0 && ldo % 4 == 0 && on4(z, z_dtype) && on4(out, out_dtype)) {
    // four runs a thread up to 8,192 values (512 threads), eight beyond
    const int ch = F <= 2048 ? 2 : (F <= 8192 ? 4 : 8), threads = ((F / 4 + ch - 1) / ch + 31) / 32 * 32;
#define PN_CASE(CH_) me_launch(polynorm_vec_kernel<TZ, TO, CH_>, dim3(T), dim3(threads), 0, stream, (const TZ*)z, ldz, coef, eps, (TO*)out, ldo, F)
    ME_DISPATCH_DTYPE(z_dtype, TZ, ME_DISPATCH_DTYPE(out_dtype, TO, { if (ch == 2) PN_CASE(2); else if (ch == 4) PN_CASE(4); else PN_CASE(8); }));
#undef PN_CASE
    ME_LAUNCH_CHECK("me_polynorm");
    return 0;
  }
  const int threads = F >= 1024 ? 256 : 128;
  ME_DISPATCH_DTYPE(z_dtype, TZ, ME_DISPATCH_DTYPE(out_dtype, TO,
      me_launch(polynorm_kernel<TZ, TO>, dim3(T), dim3(threads), 0, stream, (const TZ*)z, ldz, coef, eps, (TO*)out, ldo, F)));
  ME_LAUNCH_CHECK("me_polynorm");
  return 0;
}
