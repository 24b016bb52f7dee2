// Portions of prompts through a latent on tcgen05 / tensor memory (bfloat16, latents of 64, 128, 192 or 256 values, rows of up to 320):
// the semantics of latent_attn_mma_kernel (latent_attention_mma.cu), tile by tile on the tensor core of this generation.
//
// One block = 128 rows = (128 / gp query tokens) x (gp heads), row r being token r / gp, head r % gp; key tiles of 64 cache rows at
// absolute multiples of 64, which serve as K (all C + R columns) and as V (the first C), for all of the block's heads.
//   warp 0: TMA, a box of 64 columns per page and column block with the 128-byte swizzle, into a ring of two or three tiles.
//   warp 1: tcgen05.mma.  S[128 x 64] = Q K^T into one of two S buffers in tensor memory, a tile ahead of the softmax; then
//     O[128 x C] += P V with P from tensor memory and V as an MN-major operand from K's own tile.  O stays in tensor memory.
//   warps 2..5: bring Q once, then a thread a row: scores from tensor memory, mask, maximum, exponentials; P (bfloat16, two a column)
//     goes over the S buffer it came from.  Where a row's maximum rises its row of O is rescaled in tensor memory.  At the end O leaves through Q's place in shared memory in whole rows.
// What bounds it: a tile's chain of waits, not the products (tensor pipe 22% of the active clocks at 256 + 64 values, 17% at 128 + 32).  Four
// warps read a row of S, reduce it, rescale O where the maximum rose, form and store P, and P V follows; only the next tile's Q K^T runs
// beside that: 1.5 us a tile with three tiles in the ring, 2.1 with two, where a load also waits for the P V two tiles before.  Q, 80 KB at
// 256 + 64, and three tiles of 40 KB take the SM; rows of up to 192 values and latents of up to 128 leave room for two blocks with two
// tiles each, which fill one another's waits.  Blocks are uneven (the last tokens of a prompt see all its keys): the rest of the time.
// Measured beside the mma.sync kernel (one B200, L2 flushed, 16 heads, us): 3 prompts of 400, 800 and 1,250 tokens, rows of 256 + 64 values
// 199 -> 61, 192 + 64 123 -> 54, 128 + 32 104 -> 53, 64 + 8 87 -> 47; one prompt of 4,000 tokens 1,038 -> 203 (256 + 64), 371 -> 170 (128 + 32),
// of 300 47 -> 25, 27 -> 22; 16 tokens behind 4,000 485 -> 109, 211 -> 144.  Steps of one key tile stay with that kernel (ops).
// All waits are bounded; a wait that gives up sets flag 1 of ``err`` and the block frees its tensor memory and exits.
#include "tcgen05.cuh"
#include "mma_prims.cuh"

namespace {

constexpr int LT_ROWS = 128, LT_KEYS = 64, LT_THREADS = 192, LT_RING = 3;
constexpr int LT_QBLOCK = LT_ROWS * 128, LT_KBLOCK = LT_KEYS * 128;      // bytes of 64 columns of Q and of a key tile
constexpr float LT_LOG2E = 1.4426950408889634f;

__device__ __forceinline__ void lt_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ float lt_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void lt_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tma::smem_addr(bar)) : "memory");
}

__global__ void __launch_bounds__(LT_THREADS, 2)
latent_attn_tcgen05_kernel(const bf16* __restrict__ q_abs, const bf16* __restrict__ q_rot, const __grid_constant__ CUtensorMap pool_map,
                           const int* __restrict__ block_tables, int bt_stride, const int* __restrict__ cu_seqlens,
                           const int* __restrict__ context_lens, const int* __restrict__ tiles, int num_tiles, const float* __restrict__ sink,
                           const float* __restrict__ gate, bf16* __restrict__ out, int T_total, int H, int C, int R, int page_size, int box_rows,
                           float scale_log2, int window, int gp, int ring, uint32_t tmem_cols, int* __restrict__ err) {
  extern __shared__ unsigned char lt_smem_raw[];
  __shared__ __align__(8) unsigned long long q_bar, k_full[LT_RING], k_empty[LT_RING], s_ready[2], p_ready[2], o_ready[2];
  __shared__ uint32_t tmem_slot;
  unsigned char* smem = lt_smem_raw + ((1024u - (tma::smem_addr(lt_smem_raw) & 1023u)) & 1023u);
  const int dk = C + R, blocks = (dk + 63) / 64, key_bytes = blocks * LT_KBLOCK;
  unsigned char* q_s = smem;                             // [blocks][128 rows][128 bytes]
  unsigned char* k_s = q_s + blocks * LT_QBLOCK;         // ring x [blocks][64 rows][128 bytes]
  const int warp = tc5::uniform_warp_index(), lane = threadIdx.x & 31;

  const int packs = (H + gp - 1) / gp, tq = LT_ROWS / gp;
  const int tile = num_tiles - 1 - (int)(blockIdx.x / packs), h0 = (int)(blockIdx.x % packs) * gp;   // (a request's last tiles, with the most keys, first)
  const int b = tiles[2 * tile], q0 = tiles[2 * tile + 1];
  const int tok0 = cu_seqlens[b], q_len = cu_seqlens[b + 1] - tok0;
  const int start = context_lens[b] - q_len;
  const int n_tok = min(tq, q_len - q0);
  const int p_lo = start + q0, p_hi = p_lo + n_tok - 1, hi = p_hi + 1;
  const int lo_seen = window > 0 ? max(0, p_lo - window + 1) : 0;        // keys below are seen by no row of the tile
  const int lo = lo_seen / LT_KEYS * LT_KEYS;
  const int n_tiles = (hi - lo + LT_KEYS - 1) / LT_KEYS;
  const int* bt = block_tables + (int64_t)b * bt_stride;

  if (threadIdx.x == 0) {
    tma::mbar_init(&q_bar, 128);
    for (int s = 0; s < LT_RING; ++s) {
      tma::mbar_init(&k_full[s], 1);
      tma::mbar_init(&k_empty[s], 1);
    }
    // Two barriers a kind, taken by the tile's parity.  A barrier counts arrivals, whoever makes them, and a wait names its phase by parity, so
    // between a tile and the next but one on the same barrier all must have passed:
    //   p_ready: a warp arrives for tile it + 2 behind S(it + 2), whose product is issued after the wait for P(it), all four arrivals.  So no
    //     warp arrives twice in a phase, and the issuing warp cannot miss one.  (On one barrier a warp that need not rescale O arrived for
    //     it + 1 in the place of one that was still rescaling for it.)
    //   s_ready: S(it + 2) is asked for after P(it), so every warp has passed its wait for S(it).
    //   o_ready: a wait for P V (it) stands behind S(it + 1), issued after P V (it - 1); the commit behind S covers all products before it, so
    //     P V (it - 2), the phase before, is over.  P V (it + 2) needs this warp's P(it + 2), so the phase is not passed over either.
    for (int i = 0; i < 2; ++i) {
      tma::mbar_init(&s_ready[i], 1);
      tma::mbar_init(&p_ready[i], 4);                     // one arrival per softmax warp
      tma::mbar_init(&o_ready[i], 1);
    }
    tma::mbar_fence_init();
    tma::prefetch_map(&pool_map);
  }
  if (warp == 1) tc5::tmem_alloc(&tmem_slot, tmem_cols);
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tmem_s = tmem_slot, tmem_o = tmem_slot + 2 * LT_KEYS;
  pdl_wait();                                             // the queries and the newest cache rows come from the kernels before
  bool ok = true;

  if (warp == 0) {
    const int pages = LT_KEYS / box_rows, boxes = pages * blocks;          // (a box is a page, or 64 rows of a longer one)
    for (int it = 0; it < n_tiles; ++it) {
      const int s = it % ring, kt = lo + it * LT_KEYS;
      ok = tc5::mbar_wait_warp(&k_empty[s], ((it / ring) & 1) ^ 1);
      if (!ok) break;
      int row = -1;
      const int j0 = kt + lane * box_rows;
      if (lane < pages && j0 < hi && j0 + box_rows > lo_seen) {
        const int pi = j0 / page_size, page = bt[pi];
        if (page >= 0) row = page * page_size + (j0 - pi * page_size);
      }
      const int n_boxes = __popc(__ballot_sync(0xffffffffu, row >= 0)) * blocks;
      if (lane == 0) tma::mbar_expect_tx(&k_full[s], (unsigned)(n_boxes * box_rows * 128));
      __syncwarp();
      for (int i0 = 0; i0 < boxes; i0 += 32) {
        const int i = i0 + lane, pg = i / blocks, c = i - pg * blocks;
        const int first_row = __shfl_sync(0xffffffffu, row, pg & 31);
        if (i < boxes && first_row >= 0)
          tma::load_2d(k_s + s * key_bytes + c * LT_KBLOCK + pg * box_rows * 128, &pool_map, c * 64, first_row, &k_full[s]);
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = tc5::instr_desc_bf16(LT_ROWS, LT_KEYS);
    const uint32_t idesc_o = tc5::instr_desc_bf16(LT_ROWS, C, true);
    const tc5::DescWords q_desc = tc5::words_of(tc5::smem_desc_k_major_sw128(q_s));
    const tc5::DescWords k_desc = tc5::words_of(tc5::smem_desc_k_major_sw128(k_s));
    const tc5::DescWords v_desc = tc5::words_of(tc5::smem_desc_mn_major_sw128(k_s, LT_KBLOCK));
    const int steps = (dk + 15) / 16;
    ok = tc5::mbar_wait_warp(&q_bar, 0);
    // S(it) goes into S buffer it % 2, which held S and then P of tile it - 2: P V (it - 2) was issued before this, and the tensor
    // core runs this warp's products in the order of their issue.
    auto issue_qk = [&](int it) -> bool {
      const int s = it % ring;
      if (!tc5::mbar_wait_warp(&k_full[s], (it / ring) & 1)) return false;
      tc5::fence_after_sync();
#pragma unroll 4
      for (int k = 0; k < steps; ++k)                     // (offsets in units of 16 bytes)
        tc5::mma_f16_elect(tmem_s + (it & 1) * LT_KEYS, q_desc, (k >> 2) * (LT_QBLOCK >> 4) + 2 * (k & 3), k_desc,
                           (s * key_bytes >> 4) + (k >> 2) * (LT_KBLOCK >> 4) + 2 * (k & 3), idesc_s, k > 0);
      tc5::commit_elect(&s_ready[it & 1]);
      return true;
    };
    if (ok) ok = issue_qk(0);
    for (int it = 0; it < n_tiles && ok; ++it) {
      const int s = it % ring;
      if (it + 1 < n_tiles) {
        ok = issue_qk(it + 1);
        if (!ok) break;
      }
      ok = tc5::mbar_wait_warp(&p_ready[it & 1], (it >> 1) & 1);         // P(it) is in tensor memory, O is rescaled if it had to be
      if (!ok) break;
      tc5::fence_after_sync();
      // A = P, 8 columns of tensor memory for 16 keys; B = V: 16 keys are 2048 bytes further in every 64-column block.
#pragma unroll
      for (int k = 0; k < LT_KEYS / 16; ++k)
        tc5::mma_f16_a_in_tmem_elect(tmem_o, tmem_s + (it & 1) * LT_KEYS + k * 8, v_desc, (s * key_bytes + k * 2048) >> 4, idesc_o,
                                     it > 0 || k > 0);
      tc5::commit_elect(&o_ready[it & 1]);
      tc5::commit_elect(&k_empty[s]);
    }
  } else {
    const int lane_base = (warp & 3) * 32, r = lane_base + lane;
    const uint32_t t_row = (uint32_t)lane_base << 16;
    {   // Q: eight neighbouring threads bring a row's pieces; zeros beyond dk, the tokens and the heads
      const int pieces = dk / 8, p0 = lane & 7;
      for (int row = (threadIdx.x - 64) >> 3; row < LT_ROWS; row += 16) {
        const int tk = row / gp, hd = h0 + row % gp;
        const bool real_row = tk < n_tok && hd < H;
        const int64_t tok = tok0 + q0 + tk;
        const bf16 *abs_row = q_abs + ((int64_t)hd * T_total + tok) * C, *rot_row = q_rot + (tok * H + hd) * R - C;
        unsigned char* dst = q_s + row * 128 + ((p0 ^ (row & 7)) << 4);
        for (int c = 0; c < blocks; ++c) {
          const int p = c * 8 + p0;
          const bool real = real_row && p < pieces;
          mma_prims::cp_async16(dst + c * LT_QBLOCK, real ? (p * 8 < C ? abs_row : rot_row) + p * 8 : q_abs, real);
        }
      }
      mma_prims::cp_async_commit();
      mma_prims::cp_async_wait<0>();
      lt_fence_async_smem();
      lt_arrive(&q_bar);
    }
    const int tk = r / gp, head = h0 + r % gp;
    const bool row_ok = tk < n_tok && head < H;
    const int pos = p_lo + tk;
    const int j_max = row_ok ? pos : -1, j_min = window > 0 ? pos - window + 1 : 0;      // the keys this row sees
    float m = -INFINITY, l0 = 0.f, l1 = 0.f;               // m: the row's maximum so far
    for (int it = 0; it < n_tiles && ok; ++it) {
      const int kt = lo + it * LT_KEYS;
      const uint32_t t_s = tmem_s + (it & 1) * LT_KEYS + t_row;
      ok = tc5::mbar_wait_warp(&s_ready[it & 1], (it >> 1) & 1);
      if (!ok) break;
      tc5::fence_after_sync();
      float s[64];
      tc5::ld_64cols(t_s, s);
      tc5::wait_ld();
      const int c_max = j_max - kt, c_min = j_min - kt;
      if (!__all_sync(0xffffffffu, c_max >= LT_KEYS - 1 && c_min <= 0)) {
#pragma unroll
        for (int c = 0; c < LT_KEYS; ++c)
          if (c > c_max || c < c_min) s[c] = -INFINITY;
      }
      float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int c = 4; c < LT_KEYS; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], s[c]);
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      // The reference follows the true maximum: a row's largest weight is then 1, which no rounding touches.  (Raised only by steps of
      // more than 2^8, rows were about 1% further from 64 bits.)
      float alpha = 1.f;
      if (mx > m) {
        alpha = lt_ex2((m - mx) * scale_log2);             // m = -inf gives 0
        m = mx;
        l0 *= alpha;
        l1 *= alpha;
      }
      if (it > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
        ok = tc5::mbar_wait_warp(&o_ready[(it - 1) & 1], ((it - 1) >> 1) & 1);          // after P V (it - 1)
        if (!ok) break;
        tc5::fence_after_sync();
        for (int c0 = 0; c0 < C; c0 += 32) {               // (the row of S is held meanwhile)
          float v[32];
          tc5::ld_32cols(tmem_o + t_row + c0, v);
          tc5::wait_ld();
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] *= alpha;
          tc5::st_32cols(tmem_o + t_row + c0, v);
        }
        tc5::wait_st();
      }
      if (kt + LT_KEYS > hi || kt < lo_seen) {
        // Rows of V that hold no key of this tile must be zero (0 * anything else would not be 0).  Q K^T (it) has read them.
        const int key = r & 63, j = kt + key;
        if (j >= hi || j < lo_seen) {
          for (int c = r >> 6; c < C / 64; c += 2) {
            uint4* row = reinterpret_cast<uint4*>(k_s + (it % ring) * key_bytes + c * LT_KBLOCK + key * 128);
#pragma unroll
            for (int q = 0; q < 8; ++q) row[q] = make_uint4(0, 0, 0, 0);
          }
        }
      }
      const float mu = m == -INFINITY ? 0.f : m;
#pragma unroll
      for (int c0 = 0; c0 < LT_KEYS; c0 += 32) {           // keys c .. c + 31 go to columns c / 2 .. of the S buffer, which is read already
        uint32_t pk[16];
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          const float p0 = lt_ex2((s[c0 + c] - mu) * scale_log2), p1 = lt_ex2((s[c0 + c + 1] - mu) * scale_log2);
          __nv_bfloat162 h2 = __floats2bfloat162_rn(p0, p1);
          pk[c >> 1] = *reinterpret_cast<uint32_t*>(&h2);
          // The sum is of the weights as P V sees them: a weight that stands alone then is 1 after the division, whatever the
          // reference rounds it to.  (With the unrounded weights' sum and a lagging reference rows of one large weight were 12% further
          // from 64 bits than the mma.sync kernel's.)
          l0 += __uint_as_float(pk[c >> 1] << 16);
          l1 += __uint_as_float(pk[c >> 1] & 0xffff0000u);
        }
        tc5::st_16cols(t_s + (c0 >> 1), pk);
      }
      tc5::wait_st();
      lt_fence_async_smem();                               // the zeroed rows of V were written by ordinary stores
      tc5::fence_before_sync();
      __syncwarp();
      if (lane == 0) lt_arrive(&p_ready[it & 1]);
    }
    // The last P V, and with it all before.  (P V (n - 3), the phase before on that barrier, is over: S(n - 1) was issued after it.)
    if (ok) ok = tc5::mbar_wait_warp(&o_ready[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1);
    if (ok) {
      tc5::fence_after_sync();
      float l = l0 + l1;
      if (sink != nullptr && row_ok) l += lt_ex2(sink[head] * LT_LOG2E - (m == -INFINITY ? 0.f : m) * scale_log2);   // joins the denominator once
      float f = l > 0.f ? 1.f / l : 0.f;
      if (gate != nullptr && row_ok) f *= gate[(int64_t)(tok0 + q0 + tk) * H + head];
      // Through Q's place (every product is over), 16-byte pieces swizzled by the row, so that rows leave whole.
      const int row_bytes = C * 2, per_row = C / 8;
      for (int c0 = 0; c0 < C; c0 += 32) {
        float v[32];
        tc5::ld_32cols(tmem_o + t_row + c0, v);
        tc5::wait_ld();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 pk;
          __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
          for (int e = 0; e < 4; ++e) h2[e] = __floats2bfloat162_rn(v[q * 8 + 2 * e] * f, v[q * 8 + 2 * e + 1] * f);
          *reinterpret_cast<uint4*>(q_s + r * row_bytes + (((c0 / 8 + q) ^ (r & 7)) << 4)) = pk;
        }
      }
      __syncwarp();
      for (int i = lane; i < 32 * per_row; i += 32) {
        const int rr = lane_base + i / per_row, piece = i % per_row;
        const int tk2 = rr / gp, hd2 = h0 + rr % gp;
        if (tk2 < n_tok && hd2 < H)
          *reinterpret_cast<uint4*>(out + ((int64_t)hd2 * T_total + tok0 + q0 + tk2) * C + piece * 8) =
              *reinterpret_cast<const uint4*>(q_s + rr * row_bytes + ((piece ^ (rr & 7)) << 4));
      }
    }
  }
  if (!ok) atomicOr(err + 1, 1);
  pdl_launch_dependents();
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 1) tc5::tmem_dealloc(tmem_slot, tmem_cols);
}

// Tiles in the ring: two where that lets two blocks share the SM's shared and tensor memory, else three.
int lt_ring(int C, int R) { return C <= 128 && C + R <= 192 ? 2 : LT_RING; }
size_t lt_smem(int C, int R) {
  const size_t blocks = (C + R + 63) / 64;
  return blocks * (LT_QBLOCK + (size_t)lt_ring(C, R) * LT_KBLOCK) + 1024;
}

}  // namespace

// Heads that share a block (which then covers 128 / that many query tokens); 0 where the kernel does not take the sizes: whole column
// blocks of V, O and the S buffers in tensor memory, Q and three key tiles in shared memory, pages that a box or whole boxes cover.
ME_API int me_latent_attention_tcgen05_heads_per_block(int H, int C, int R, int page_size) {
  const bool pages = page_size >= 8 && (page_size <= LT_KEYS ? LT_KEYS % page_size == 0 : page_size % LT_KEYS == 0);
  if (H < 1 || C < 64 || C > 256 || C % 64 || R < 0 || R % 8 || C + R > 320 || !pages) return 0;
  int gp = 1;
  while (gp < 16 && gp < H) gp *= 2;
  return gp;
}

// pool_map: the cache rows as [rows][C + R], boxes of min(page_size, 64) rows x 64 columns with the 128-byte swizzle.  ``tiles``: (request,
// first local query) per block, each 128 / heads_per_block query tokens.  The rest as for me_latent_attention_mma.
ME_API int me_latent_attention_tcgen05(const void* q_abs, const void* q_rot, const void* pool_map, const int* block_tables, int bt_stride,
                                       const int* cu_seqlens, const int* context_lens, const int* tiles, int num_tiles, const float* sink,
                                       const float* gate, void* out, int T_total, int H, int C, int R, int page_size, float scale, int window,
                                       int* err, cudaStream_t stream) {
  if (num_tiles == 0) return 0;
  const int gp = me_latent_attention_tcgen05_heads_per_block(H, C, R, page_size);
  ME_REQUIRE(gp > 0, "me_latent_attention_tcgen05: rows of %d + %d values, pages of %d are not taken", C, R, page_size);
  ME_REQUIRE(pool_map != nullptr && err != nullptr && scale > 0.f, "me_latent_attention_tcgen05: a tensor map, the error word and a positive scale are required");
  ME_REQUIRE((((uintptr_t)q_abs | (uintptr_t)q_rot | (uintptr_t)out) & 15) == 0, "me_latent_attention_tcgen05: operands must start on 16 bytes");
  const int64_t grid = (int64_t)((H + gp - 1) / gp) * num_tiles;
  ME_REQUIRE(grid <= 0x7fffffff, "me_latent_attention_tcgen05: too many blocks");
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(latent_attn_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lt_smem(256, 64));
    ME_REQUIRE(e == cudaSuccess, "me_latent_attention_tcgen05: cannot raise shared memory: %s", cudaGetErrorString(e));
    attr_set = true;
  }
  me_launch(latent_attn_tcgen05_kernel, dim3((unsigned)grid), dim3(LT_THREADS), lt_smem(C, R), stream, (const bf16*)q_abs, (const bf16*)q_rot,
            *reinterpret_cast<const CUtensorMap*>(pool_map), block_tables, bt_stride, cu_seqlens, context_lens, tiles, num_tiles, sink, gate,
            (bf16*)out, T_total, H, C, R, page_size, page_size < LT_KEYS ? page_size : LT_KEYS, scale * LT_LOG2E, window, gp, lt_ring(C, R),
            C > 128 ? 512u : 256u, err);
  ME_LAUNCH_CHECK("me_latent_attention_tcgen05");
  return 0;
}
