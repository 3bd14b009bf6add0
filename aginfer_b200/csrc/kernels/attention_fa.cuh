// Tensor-core attention for many query rows (prefill: 288 causal tokens with 128-wide heads; the vision
// tower: 512 patch tokens, 80-wide heads, block-diagonal windows).  Streaming-softmax formulation on
// warp-level MMAs, parallel over rows, keys and output columns:
//
//   * one block per (32 query rows, head): two groups of 16 rows, a warp per group and key tile, two loading warps;
//   * keys are visited in chunks of four or five 64-key tiles, staged row-major in shared memory by 16-byte
//     asynchronous copies: K by all warps, V by the loading warps while the others multiply Q with K (issuing the
//     copies takes as long as the bytes do, 35 B per clock, so V behind K in the same warps delayed the scores by 2 us);
//   * each warp of a group multiplies Q with one tile's keys, masks, and leaves the tile's row maxima in shared
//     memory; from the maxima of the tiles before it every warp knows the running maximum its tile would have met,
//     so it forms P = exp(S - m) and the tile's row sums at once and leaves them in shared memory too;
//   * each warp then adds P.V of the chunk's tiles, in order and with the streaming formulation's rescaling between
//     them, for its share of the head's columns: per output the same operations in the same order as one warp
//     walking the tiles one by one, which is what this replaced;
//   * only key tiles a block of rows can see are visited: the causal prefix, or the diagonal block(s).
//
// What bounds it: a chain of loading K, scores, P, P.V of about 2000 clocks each; scores and P.V run at the rate of the
// warp-level MMA (16 clocks each per scheduler).  288 causal tokens, 16 heads of 128:
// 12 us with 16 rows a warp and the tiles one after the other, now 8.3; 512 patches, windows of 64, 16 heads of 80:
// 11 us, now 6.
//
// Head width is a template parameter (16-element steps); grouped-query attention maps query head h to KV
// head h / (q_heads / kv_heads).  Pitch of the shared tiles = head_dim + 8 elements: rows stay 16-byte
// aligned and the eight rows of a fragment fall into different banks.
// grid = (ceil(q_rows / 32), q_heads), block = 64 * tiles + 64,
// dynamic shared memory = (256 * tiles + 64) * (head_dim + 8) + 4352 * tiles.
#pragma once

#include "attention.cuh"

namespace fa {

constexpr unsigned kKeyTile = 64, kRows = 32, kLoaders = 64;
// Key tiles of a chunk for 128-wide heads: five, so that up to 320 keys are one chunk.  One block per SM, as with four
// or three (165 and 126 KB).  Causal rows, us a launch with 2 (two blocks per SM) / 3 / 4 / 5 tiles, 16 query and 2 KV
// heads: 101 rows 5.5 / 5.0 / 5.4 / 5.4, 197: 9.1 / 7.2 / 6.5 / 6.9, 288: 11.4 / 8.9 / 9.8 / 8.5, 320: 13.1 / 12.1 / 13.8 /
// 12.4, 512: 18.8 / 21.3 / 21.7 / 22.6, 1024: 55.5 / 57.0 / 56.6 / 58.1; 28 and 4 heads: 101: 6.3 / 5.0 / 5.6 / 5.5, 288:
// 13.1 / 15.5 / 15.8 / 14.9, 1024: 77.8 / 88.1 / 88.5 / 89.5.  Of the one-block forms five is the best at 288 keys, level
// at 320 and up to 12 % behind three elsewhere; grids of more than a round would gain from two blocks per SM.
template <int HD16>
struct Shape {
  static constexpr unsigned kTiles = HD16 == 8 ? 5 : 4;
  static constexpr unsigned kCompute = kTiles * 64, kThreads = kCompute + kLoaders, kPerSm = HD16 == 8 ? 1 : 2;
};

template <int HD16>
__device__ __forceinline__ void attention_body(const bf16* q, const bf16* k, const bf16* v, bf16* o, unsigned q_rows,
                                               unsigned kv_rows, unsigned q_heads, unsigned kv_heads, unsigned q_stride,
                                               unsigned k_stride, unsigned v_stride, unsigned o_stride, float scale,
                                               unsigned mask_mode, unsigned mask_arg, unsigned* amax_bits = nullptr) {
  constexpr unsigned head_dim = HD16 * 16, pitch = head_dim + 8, vec_per_row = head_dim / 8;
  constexpr unsigned kTiles = Shape<HD16>::kTiles, kChunk = kKeyTile * kTiles, kCompute = Shape<HD16>::kCompute;
  constexpr int kCols = (2 * HD16 + int(kTiles) - 1) / int(kTiles);   // 8-column output tiles of a warp, the last may be absent
  auto block_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(Shape<HD16>::kThreads) : "memory"); };   // of both kinds of warps
  auto compute_sync = [] { asm volatile("bar.sync 2, %0;" ::"n"(Shape<HD16>::kCompute) : "memory"); };
  extern __shared__ __align__(16) unsigned char attn_smem[];
  bf16* k_chunk = reinterpret_cast<bf16*>(attn_smem);                         // [chunk][pitch]
  bf16* v_chunk = k_chunk + kChunk * pitch;                                   // [chunk][pitch]
  uint4* p_frag = reinterpret_cast<uint4*>(v_chunk + kChunk * pitch);         // [2 groups][tiles][4 16-key steps][32 lanes]
  float* maxima = reinterpret_cast<float*>(p_frag + 2 * kTiles * 4 * 32);     // [2][tiles][16 rows]
  float* sums = maxima + 2 * kTiles * 16;                                     // [2][tiles][16]
  bf16* q_rows_smem = reinterpret_cast<bf16*>(sums + 2 * kTiles * 16);        // [32][pitch]
  const bool q_vec = q_stride % 8 == 0 && (reinterpret_cast<size_t>(q) & 15) == 0;
  grid_dependency_wait();
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const unsigned group = warp / kTiles, own = warp % kTiles;                  // row group; tile (then columns) of this warp
  const unsigned head = blockIdx.y, kv_head = head / (q_heads / kv_heads);
  const unsigned row_base = blockIdx.x * kRows, warp_row = row_base + group * 16;
  const unsigned last_row = min(row_base + kRows, q_rows) - 1, warp_last = min(warp_row + 15, q_rows - 1);

  // keys this block of rows can see
  unsigned key_begin = 0, key_end = kv_rows;
  if (mask_mode == 1) key_end = min(kv_rows, last_row + mask_arg + 1);
  if (mask_mode == 2) {
    key_begin = (row_base / mask_arg) * mask_arg;
    key_end = min(kv_rows, (last_row / mask_arg + 1) * mask_arg);
  }
  const unsigned tiles_total = key_end > key_begin ? (key_end - key_begin + kKeyTile - 1) / kKeyTile : 0;

  auto stage = [&](bf16* dst, const bf16* src, unsigned stride, unsigned first_tile, unsigned thread, unsigned threads) {
    const unsigned keys = first_tile < tiles_total ? min(tiles_total - first_tile, kTiles) * kKeyTile : 0;
    const unsigned key0 = key_begin + first_tile * kKeyTile;
    for (unsigned i = thread; i < keys * vec_per_row; i += threads) {
      const unsigned j = i / vec_per_row, d = (i % vec_per_row) * 8;
      const unsigned key = key0 + j, src_row = min(key, kv_rows - 1), bytes = key < kv_rows ? 16u : 0u;  // zero-fill past the end
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                       static_cast<unsigned>(__cvta_generic_to_shared(dst + j * pitch + d))),
                   "l"(src + size_t(src_row) * stride + kv_head * head_dim + d), "r"(bytes) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // keys a row sees: [lo, hi); those of the group run from its first row's lo to its last row's hi
  auto lo_of = [&](unsigned row) { return mask_mode == 2 ? row / mask_arg * mask_arg : 0u; };
  auto hi_of = [&](unsigned row) {
    return mask_mode == 1 ? min(kv_rows, row + mask_arg + 1) : mask_mode == 2 ? min(kv_rows, (row / mask_arg + 1) * mask_arg) : kv_rows;
  };
  const unsigned group_lo = lo_of(warp_row), group_hi = warp_row < q_rows ? hi_of(warp_last) : 0u;
  auto visits = [&](unsigned tile) {   // does this group of rows see anything of a tile?
    const unsigned key0 = key_begin + tile * kKeyTile;
    return tile < tiles_total && key0 < group_hi && key0 + kKeyTile > group_lo;
  };
  if (warp >= 2 * kTiles) {   // loading warps: V of a chunk while the others multiply its K
    for (unsigned first = 0; first < tiles_total; first += kTiles) {
      block_sync();                                     // K has landed: V has the memory path to itself
      stage(v_chunk, v, v_stride, first, threadIdx.x - kCompute, kLoaders);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      block_sync();
      if (first + kTiles < tiles_total) block_sync();
    }
    return;
  }
  // Q as stored (zero past q_rows), with the first keys; the softmax scale is applied to the fp32 scores, so no second
  // rounding of Q.
  if (q_vec) {
    for (unsigned i = threadIdx.x; i < kRows * vec_per_row; i += kCompute) {
      const unsigned j = i / vec_per_row, d = (i % vec_per_row) * 8, row = min(row_base + j, q_rows - 1);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                       static_cast<unsigned>(__cvta_generic_to_shared(q_rows_smem + j * pitch + d))),
                   "l"(q + size_t(row) * q_stride + head * head_dim + d), "r"(row_base + j < q_rows ? 16u : 0u) : "memory");
    }
  } else {
    for (unsigned i = threadIdx.x; i < kRows * head_dim / 2; i += kCompute) {
      const unsigned j = i / (head_dim / 2), d = (i % (head_dim / 2)) * 2, row = min(row_base + j, q_rows - 1);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                       static_cast<unsigned>(__cvta_generic_to_shared(q_rows_smem + j * pitch + d))),
                   "l"(q + size_t(row) * q_stride + head * head_dim + d), "r"(row_base + j < q_rows ? 4u : 0u) : "memory");
    }
  }
  stage(k_chunk, k, k_stride, 0, threadIdx.x, kCompute);

  const unsigned lo[2] = {lo_of(warp_row + g), lo_of(warp_row + g + 8)}, hi[2] = {hi_of(warp_row + g), hi_of(warp_row + g + 8)};
  unsigned qa[HD16][4];

  float row_max[2] = {-3.0e38f, -3.0e38f}, row_sum[2] = {0.f, 0.f}, out[kCols][4];
#pragma unroll
  for (int c = 0; c < kCols; ++c)
#pragma unroll
    for (int i = 0; i < 4; ++i) out[c][i] = 0.f;

  for (unsigned first = 0; first < tiles_total; first += kTiles) {
    const bool more = first + kTiles < tiles_total;
    asm volatile("cp.async.wait_group 0;" ::: "memory");   // K of this chunk
    block_sync();
    if (first == 0) {   // Q fragments (A operand): rows g and g + 8 of this group's 16
      const unsigned q_addr = static_cast<unsigned>(__cvta_generic_to_shared(q_rows_smem + (group * 16 + (lane & 15)) * pitch + (lane >> 4) * 8));
#pragma unroll
      for (int ks = 0; ks < HD16; ++ks)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(qa[ks][0]), "=r"(qa[ks][1]), "=r"(qa[ks][2]), "=r"(qa[ks][3]) : "r"(q_addr + ks * 32));
    }

    // scores of this warp's tile, masked, and their row maxima
    const bool any = visits(first + own);
    const unsigned key0 = key_begin + (first + own) * kKeyTile;
    float s[8][4];
    if (any) {
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
      // lanes 0-7 | 8-15 | 16-23 | 24-31 address the 8 x 8 blocks (keys nt, depth 0) | (nt, 8) | (nt + 1, 0) | (nt + 1, 8)
      const unsigned k_addr = static_cast<unsigned>(__cvta_generic_to_shared(
          k_chunk + (own * kKeyTile + (lane >> 4) * 8 + (lane & 7)) * pitch + ((lane >> 3) & 1) * 8));
#pragma unroll
      for (int ks = 0; ks < HD16; ++ks)
#pragma unroll
        for (int nt = 0; nt < 8; nt += 2) {
          unsigned b0, b1, b2, b3;
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                       : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3) : "r"(k_addr + (nt * 8 * pitch + ks * 16) * 2));
          skinny_mma_bf16(s[nt], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
          skinny_mma_bf16(s[nt + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b2, b3);
        }
      // mask: c0,c1 belong to row g (keys 2t, 2t+1 of the 8-key tile), c2,c3 to row g + 8
#pragma unroll
      for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned key = key0 + nt * 8 + 2 * t + (i & 1);
          const bool visible = key >= lo[i >> 1] && key < hi[i >> 1];
          s[nt][i] = visible ? s[nt][i] * scale : -3.0e38f;
        }
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {   // hr 0: row g, hr 1: row g + 8
        float tile_max = -3.0e38f;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) tile_max = fmaxf(tile_max, fmaxf(s[nt][2 * hr], s[nt][2 * hr + 1]));
        tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 1));
        tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 2));
        if (t == 0) maxima[(group * kTiles + own) * 16 + g + hr * 8] = tile_max;
      }
    }
    compute_sync();                                     // maxima are there, K is no longer needed
    if (more) stage(k_chunk, k, k_stride, first + kTiles, threadIdx.x, kCompute);

    if (any) {
      unsigned pa[4][4];   // [16-key step][a0..a3]
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        float new_max = row_max[hr];   // the running maximum a walk over the tiles would have after this one
#pragma unroll
        for (unsigned i = 0; i < kTiles; ++i)
          if (i <= own && visits(first + i)) new_max = fmaxf(new_max, maxima[(group * kTiles + i) * 16 + g + hr * 8]);
        float tile_sum = 0.f;
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
          const float s0 = s[nt][2 * hr], s1 = s[nt][2 * hr + 1];
          const float e0 = __expf(s0 - new_max), e1 = __expf(s1 - new_max);
          const float p0 = s0 > -1.0e38f ? e0 : 0.f, p1 = s1 > -1.0e38f ? e1 : 0.f;
          tile_sum += p0 + p1;
          const bf162 pair = __floats2bfloat162_rn(p0, p1);
          // A operand of P.V for 16-key step nt / 2: a0/a1 = rows g / g + 8 of the first 8 keys, a2/a3 of the second
          pa[nt >> 1][(nt & 1) * 2 + hr] = *reinterpret_cast<const unsigned*>(&pair);
        }
        tile_sum += __shfl_xor_sync(0xffffffffu, tile_sum, 1);
        tile_sum += __shfl_xor_sync(0xffffffffu, tile_sum, 2);
        if (t == 0) sums[(group * kTiles + own) * 16 + g + hr * 8] = tile_sum;
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        p_frag[((group * kTiles + own) * 4 + kk) * 32 + lane] = make_uint4(pa[kk][0], pa[kk][1], pa[kk][2], pa[kk][3]);
    }
    block_sync();                                       // P, sums and V of this chunk are there

    // O += P (16 x 64 keys) . V (64 keys x this warp's columns), tile after tile; ldmatrix with transpose turns 8 x 8
    // blocks of row-major V into B fragments, two 16-key steps at a time
#pragma unroll 1
    for (unsigned i = 0; i < kTiles; ++i) {
      if (!visits(first + i)) continue;
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const float new_max = fmaxf(row_max[hr], maxima[(group * kTiles + i) * 16 + g + hr * 8]);
        const float rescale = new_max > -1.0e38f ? __expf(row_max[hr] - new_max) : 1.f;
        row_max[hr] = new_max;
        row_sum[hr] = row_sum[hr] * rescale + sums[(group * kTiles + i) * 16 + g + hr * 8];
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          out[c][2 * hr] *= rescale;
          out[c][2 * hr + 1] *= rescale;
        }
      }
#pragma unroll
      for (int kk = 0; kk < 4; kk += 2) {
        const uint4 pa = p_frag[((group * kTiles + i) * 4 + kk) * 32 + lane], pb = p_frag[((group * kTiles + i) * 4 + kk + 1) * 32 + lane];
        unsigned b[kCols][4];
#pragma unroll
        for (int c = 0; c < kCols; ++c) {
          const unsigned nt = own + c * kTiles;
          if (nt >= 2 * HD16) continue;
          const unsigned addr = static_cast<unsigned>(__cvta_generic_to_shared(v_chunk + (i * kKeyTile + kk * 16 + lane) * pitch + nt * 8));
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                       : "=r"(b[c][0]), "=r"(b[c][1]), "=r"(b[c][2]), "=r"(b[c][3]) : "r"(addr));
        }
#pragma unroll
        for (int c = 0; c < kCols; ++c)
          if (own + c * kTiles < 2 * HD16) skinny_mma_bf16(out[c], pa.x, pa.y, pa.z, pa.w, b[c][0], b[c][1]);
#pragma unroll
        for (int c = 0; c < kCols; ++c)
          if (own + c * kTiles < 2 * HD16) skinny_mma_bf16(out[c], pb.x, pb.y, pb.z, pb.w, b[c][2], b[c][3]);
      }
    }
    if (more) block_sync();                             // V, P, sums and maxima are free
  }

  if (tiles_total == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");   // Q is under way
  float best = 0.f;   // max |o| over this thread's outputs, for a following dynamic quantisation
#pragma unroll
  for (int hr = 0; hr < 2; ++hr) {
    const unsigned row = warp_row + g + hr * 8;
    if (row >= q_rows) continue;
    const float inv = row_sum[hr] > 0.f ? 1.f / row_sum[hr] : 0.f;
    bf16* dst = o + size_t(row) * o_stride + head * head_dim + 2 * t;
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
      const unsigned nt = own + c * kTiles;
      if (nt >= 2 * HD16) continue;
      const float a = out[c][2 * hr] * inv, b = out[c][2 * hr + 1] * inv;
      best = fmaxf(best, fmaxf(fabsf(a), fabsf(b)));
      *reinterpret_cast<bf162*>(dst + nt * 8) = __floats2bfloat162_rn(a, b);
    }
  }
  if (amax_bits != nullptr) {   // rounding is monotonic: the rounded maximum is the maximum of the rounded outputs
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, offset));
    if (lane == 0) atomicMax(amax_bits, __float_as_uint(__bfloat162float(__float2bfloat16_rn(best))));
  }
}

}  // namespace fa

#define AGI_ATTENTION_FA(NAME, HD16)                                                                                 \
  extern "C" __global__ void __launch_bounds__(fa::Shape<HD16>::kThreads, fa::Shape<HD16>::kPerSm)                                                                  \
  NAME(const bf16* q, const bf16* k, const bf16* v, bf16* o, unsigned q_rows, unsigned kv_rows, unsigned q_heads,    \
       unsigned kv_heads, unsigned head_dim, unsigned q_stride, unsigned k_stride, unsigned v_stride,               \
       unsigned o_stride, float scale, unsigned mask_mode, unsigned mask_arg) {                                      \
    fa::attention_body<HD16>(q, k, v, o, q_rows, kv_rows, q_heads, kv_heads, q_stride, k_stride, v_stride, o_stride, \
                             scale, mask_mode, mask_arg);                                                            \
  }
// the same, also folding max |o| into *amax_bits (a zero-initialised word)
#define AGI_ATTENTION_FA_AMAX(NAME, HD16)                                                                            \
  extern "C" __global__ void __launch_bounds__(fa::Shape<HD16>::kThreads, fa::Shape<HD16>::kPerSm)                                                                  \
  NAME(const bf16* q, const bf16* k, const bf16* v, bf16* o, unsigned q_rows, unsigned kv_rows, unsigned q_heads,    \
       unsigned kv_heads, unsigned head_dim, unsigned q_stride, unsigned k_stride, unsigned v_stride,               \
       unsigned o_stride, float scale, unsigned mask_mode, unsigned mask_arg, unsigned* amax_bits) {                 \
    fa::attention_body<HD16>(q, k, v, o, q_rows, kv_rows, q_heads, kv_heads, q_stride, k_stride, v_stride, o_stride, \
                             scale, mask_mode, mask_arg, amax_bits);                                                 \
  }
AGI_ATTENTION_FA_AMAX(agi_attention_fa_amax_bf16_d80, 5)
AGI_ATTENTION_FA_AMAX(agi_attention_fa_amax_bf16_d128, 8)
#undef AGI_ATTENTION_FA_AMAX
AGI_ATTENTION_FA(agi_attention_fa_bf16_d48, 3)
AGI_ATTENTION_FA(agi_attention_fa_bf16_d64, 4)
AGI_ATTENTION_FA(agi_attention_fa_bf16_d80, 5)
AGI_ATTENTION_FA(agi_attention_fa_bf16_d128, 8)
#undef AGI_ATTENTION_FA
