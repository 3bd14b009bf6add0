// Tensor-core GEMM for 33 tokens and up: Y[M, N] = epilogue(X[M, K] . W[N, K]^T), bf16 or E4M3 operands (row-major,
// or E4M3 in the packed layout of recipes/layout.py), fp32 accumulation in tensor memory.
//
// What bounds it.  At a few hundred tokens neither HBM nor the tensor pipe sets the time but the bytes each SM
// takes in from L2: every CTA reads its weight rows AND all of its tokens, at 50-60 bytes per clock and SM whatever
// the copy mechanism (measured: 16-byte cp.async 52, bulk copies of 16 KB and more 58).  So the tile is shaped to
// take in little and to use all 148 SMs at once:
//
//   * tokens are the MMA's A operand (128 rows an instruction, up to four such tiles in a CTA: 512 tokens), weights
//     the B operand with `NB` rows, any multiple of 16 up to 256.  NB divides N over the SMs in one wave (11008 rows:
//     138 CTAs of 80) where 128-row weight tiles leave a second wave nearly empty;
//   * clusters: the ranks of a thread-block cluster (grid z) share the K range, so that NB can be that much larger for
//     the same number of CTAs and the tokens are re-read less.  They meet through L2: each files its fp32 partial tiles
//     (coalesced, [run][column / 4][row]), the cluster barrier orders the writes, and every rank finishes a share of the
//     rows.  Through distributed shared memory the same exchange ran at 11 bytes per clock and SM (64 KB each way in a
//     cluster of 8: 2.9 us);
//   * how K is summed does not depend on the tile: it is cut into `runs` of `per_run` blocks, every run has an
//     accumulator of its own in tensor memory, and the runs are added in order.  A rank takes whole runs; without a
//     cluster one CTA keeps all of them.  Stacks of FP8 blocks need that: one flipped rounding in front of a per-tensor
//     amax moves the codes of a whole operand, so a tile chosen for speed must not change a single bit;
//   * the epilogue stages fp32 rows in the ring's memory so that outputs, residual and bias move in 16-byte vectors
//     along rows.  (Storing from the TMEM layout, a token per lane, each store touches 32 lines: 20k cycles for
//     288 x 80 outputs, four times the main loop.)  SwiGLU needs no further pass: with kFlagSwiglu a tile is NB / 2
//     gate rows beside the NB / 2 up rows of the same features, with kFlagMulSilu the gate comes from memory.
//     kFlagAmax folds max |y| for a following dynamic quantisation.
//
// Half of the warps bring in weights (they never wait for the previous kernel: under programmatic dependent launch the ring's
// weights land while it drains), the other half tokens, each on its own so that a slot is ready when both have
// arrived; the last warp issues the MMAs.  The issuing thread is chosen by elect.sync: issued under a lane comparison, an MMA costs
// ~99 cycles and a bulk copy ~54 in operand moves; elected, 39 and 17.  Row-major operands complete on the ring's
// mbarriers (cp.async.mbarrier.arrive), so the whole ring is in flight.
//
// Every mbarrier wait is bounded and reports through the status word; nobody waits for another CTA except at the
// cluster barrier.
#pragma once

#include "gemm_tc.cuh"

namespace tk {

using namespace tc;

constexpr unsigned kMaxRing = 8;
// kW weight warps, kW token warps (all of them: epilogue), 1 MMA warp.
constexpr unsigned kW = 4, kMmaWarp = 2 * kW, kEpilogue = 64 * kW, kThreads = kEpilogue + 32;

struct Part {
  const uint8_t* w;
  const bf16* bias;
  const float* scale;
  void* y;
  unsigned N, ldy;
};

// Arrives at `bar` once every cp.async this thread has issued so far has landed.
__device__ __forceinline__ void cp_async_arrive(unsigned long long* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_load16_nowait(unsigned addr, unsigned r[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_loads() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// What the epilogue of one thread needs to know about its part.
struct Out {
  void* y;
  const bf16* bias;
  const bf16* bias2;     // bias of the up matrix of kFlagSwiglu
  const bf16* other;     // residual, or the gate of kFlagMulSilu; row pitch ldy
  unsigned N, ldy, flags;
  float alpha, alpha2;   // alpha2: the up matrix of kFlagSwiglu
  bool vec;              // rows, bias and pointers allow 16-byte vectors
  bool one_run;          // K summed in one run: scale and bias are one fused multiply-add, otherwise two roundings
};

// How a tile is finished.  The modes that the recipes run have loops of their own without a flag test; everything
// else (activations, fp32 output, ragged or misaligned rows) takes the general one.
enum Finish { kScale, kScaleBias, kScaleResidual, kScaleBiasResidual, kGateUp, kTimesSilu, kGeneral };

// Rows [0, count) of the staged fp32 tile (P floats apart) are tokens m ... of features n0 ... n0 + 8 * groups - 1 (with
// kGateUp the up products follow the gate products in the row).  Eight features a thread, consecutive threads along a
// row.  Returns max |y| over what this thread stored, before rounding (rounding is monotonic), where it is asked for.
template <int kMode>
__device__ __forceinline__ float finish_tile(const float* tile, unsigned P, unsigned count, unsigned groups, unsigned m,
                                             unsigned n0, const Out& o) {
  constexpr bool kGen = kMode == kGeneral;
  constexpr bool kPairs = kMode == kGateUp;
  const unsigned step_r = kEpilogue / groups, step_c = kEpilogue % groups;
  unsigned r = threadIdx.x / groups, c = threadIdx.x % groups;
  const size_t base = size_t(m) * o.ldy + n0;
  const bool amax = (o.flags & kFlagAmax) != 0;
  float best = 0.f;
  while (r < count) {
    const unsigned n = n0 + c * 8, off = r * o.ldy + c * 8;
    const float* cell = tile + r * P + c * 8;
    if (n < o.N) {
      const float4 lo = *reinterpret_cast<const float4*>(cell), hi = *reinterpret_cast<const float4*>(cell + 4);
      float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w}, other[8], bias[8];
      const unsigned live = kGen ? min(8u, o.N - n) : 8u;
      const bool vec = !kGen || (o.vec && live == 8);
      if (kMode == kScaleResidual || kMode == kScaleBiasResidual || kMode == kTimesSilu || (kGen && (o.flags & (kFlagResidual | kFlagMulSilu)))) {
        const bf16* src = o.other + base + off;
        if (vec) unpack8(*reinterpret_cast<const Bf16x8*>(src), other);
        else
#pragma unroll
          for (int j = 0; j < 8; ++j) other[j] = unsigned(j) < live ? __bfloat162float(src[j]) : 0.f;
      }
      if (kMode == kScaleBias || kMode == kScaleBiasResidual || ((kGen || kPairs) && (o.flags & kFlagBias))) {
        if (vec) unpack8(*reinterpret_cast<const Bf16x8*>(o.bias + n), bias);
        else
#pragma unroll
          for (int j = 0; j < 8; ++j) bias[j] = unsigned(j) < live ? __bfloat162float(o.bias[n + j]) : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          v[j] = o.one_run ? fmaf(v[j], o.alpha, bias[j]) : __fadd_rn(__fmul_rn(v[j], o.alpha), bias[j]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __fmul_rn(v[j], o.alpha);
      }
      if (kPairs || (kGen && (o.flags & kFlagSwiglu))) {     // gate and up pass through bf16 as they would between launches
        const float* up = cell + groups * 8;
        const float4 ulo = *reinterpret_cast<const float4*>(up), uhi = *reinterpret_cast<const float4*>(up + 4);
        const float u[8] = {ulo.x, ulo.y, ulo.z, ulo.w, uhi.x, uhi.y, uhi.z, uhi.w};
        float ur[8], gr[8];
        if (o.flags & kFlagBias) {
          float bias2[8];
          if (vec) unpack8(*reinterpret_cast<const Bf16x8*>(o.bias2 + n), bias2);
          else
#pragma unroll
            for (int j = 0; j < 8; ++j) bias2[j] = unsigned(j) < live ? __bfloat162float(o.bias2[n + j]) : 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            ur[j] = o.one_run ? fmaf(u[j], o.alpha2, bias2[j]) : __fadd_rn(__fmul_rn(u[j], o.alpha2), bias2[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) ur[j] = __fmul_rn(u[j], o.alpha2);
        }
        unpack8(pack8(v), gr);
        unpack8(pack8(ur), ur);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = silu_bf16(gr[j]) * ur[j];
      } else if (kMode == kTimesSilu || (kGen && (o.flags & kFlagMulSilu))) {
        unpack8(pack8(v), v);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] *= silu_bf16(other[j]);
      } else {
        if (kGen && (o.flags & kFlagActMask)) {
#pragma unroll 1
          for (int j = 0; j < 8; ++j) v[j] = apply_activation(v[j], o.flags);
        }
        if (kMode == kScaleResidual || kMode == kScaleBiasResidual || (kGen && (o.flags & kFlagResidual))) {
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __fadd_rn(v[j], other[j]);
        }
      }
      if ((kGen || kPairs || kMode == kTimesSilu) && amax) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (!kGen || unsigned(j) < live) best = fmaxf(best, fabsf(v[j]));
      }
      if (kGen && (o.flags & kFlagOutF32)) {
        float* y = static_cast<float*>(o.y) + base + off;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (unsigned(j) < live) y[j] = v[j];
      } else {
        bf16* y = static_cast<bf16*>(o.y) + base + off;
        if (vec) *reinterpret_cast<Bf16x8*>(y) = pack8(v);
        else
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (unsigned(j) < live) y[j] = __float2bfloat16_rn(v[j]);
      }
    }
    r += step_r;
    c += step_c;
    if (c >= groups) { c -= groups; ++r; }
  }
  return best;
}

// Adds `runs` filed partial tiles, in order, over `count` rows and 4 * `quads` columns into the staged tile.  Item =
// (four columns, row), rows fastest; a thread's items are kEpilogue apart, kBatch at a time, and kRuns loads of each are
// in flight together (eight 16-byte loads a thread: more spill at the 96 registers that let two CTAs share an SM).
template <unsigned kBatch, unsigned kRuns>
__device__ __forceinline__ void add_runs(const float4* filed, float* tile, unsigned P, unsigned count, unsigned quads,
                                         unsigned R, unsigned runs) {
  if (count == 0) return;
  const unsigned items = count * quads, step_c = kEpilogue / count, step_r = kEpilogue % count;
  const unsigned run_step = quads * R;
  unsigned c4 = threadIdx.x / count, r = threadIdx.x % count;
  for (unsigned i0 = threadIdx.x; i0 < items; i0 += kEpilogue * kBatch) {
    float4 a[kBatch][kRuns];
    unsigned c = c4, q = r;
#pragma unroll
    for (unsigned b = 0; b < kBatch; ++b) {
      const float4* cell = filed + size_t(c) * R + q;
      const bool live = i0 + b * kEpilogue < items;
#pragma unroll
      for (unsigned z = 0; z < kRuns; ++z)
        if (live && z < runs) a[b][z] = __ldcg(cell + z * run_step);
      c += step_c;
      q += step_r;
      if (q >= count) { q -= count; ++c; }
    }
#pragma unroll
    for (unsigned b = 0; b < kBatch; ++b) {
      float4 sum = a[b][0];
#pragma unroll
      for (unsigned z = 1; z < kRuns; ++z)
        if (z < runs) { sum.x += a[b][z].x; sum.y += a[b][z].y; sum.z += a[b][z].z; sum.w += a[b][z].w; }
      if (i0 + b * kEpilogue < items) {
        for (unsigned z = kRuns; z < runs; ++z) {
          const float4 more = __ldcg(filed + size_t(c4) * R + r + z * run_step);
          sum.x += more.x; sum.y += more.y; sum.z += more.z; sum.w += more.w;
        }
        *reinterpret_cast<float4*>(tile + r * P + c4 * 4) = sum;
      }
      c4 += step_c;
      r += step_r;
      if (r >= count) { r -= count; ++c4; }
    }
  }
}

// grid = (weight tiles of all parts, token groups of `tg` rows, ranks); with kFlagGroupsFirst the first two change places, so that
// the groups of a weight tile run side by side (the builder's `groups_first` says when; gate and up of 90 MB for 288 tokens: 91 MB
// from DRAM, 173 with the tiles side by side).  block = kThreads.  NB: weight rows of a tile, a
// multiple of 16 (of 32 with kFlagSwiglu) up to 256; tg a multiple of 8, ceil(tg / 128) * NB' * (runs a rank takes) <=
// 512 with NB' = NB rounded up to 32.  Dynamic shared memory: 1024 + the larger of the ring, stages * (tg + NB) * 128 plus what the last
// slot's A tiles overhang (rows past the tokens are read by the MMA, never stored), and the epilogue's tile,
// min(tg, 128) (in a cluster: ceil(tg / (8 ranks)) * 8) * (NB + 4) * 4.  `partial` holds
// gridDim.x * gridDim.y * runs * NB * (tg rounded up to 32) floats for a cluster.
template <bool kFp8, bool kPacked, bool kCluster>
__device__ __forceinline__ void body(const uint8_t* x, const float* scale_a, const bf16* other, float* partial,
                                     unsigned* amax_bits, unsigned* status, unsigned M, unsigned K, unsigned ldx,
                                     unsigned flags, unsigned NB, unsigned stages, unsigned tg, unsigned runs,
                                     unsigned per_run, const Part& p0,
                                     const Part& p1, const Part& p2, unsigned tile) {
  constexpr unsigned kRowStep = 4 * kW;   // rows a copy pass covers
  extern __shared__ unsigned char dynamic_smem[];
  __shared__ __align__(8) unsigned long long full_bar[kMaxRing], empty_bar[kMaxRing], accum_bar;
  __shared__ unsigned tmem_slot;

  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned elem = kFp8 ? 1u : 2u;
  const bool swiglu = (flags & kFlagSwiglu) != 0;
  const unsigned nb_out = swiglu ? NB / 2 : NB;               // output features of a tile
  // which matrix this tile belongs to
  const unsigned t0 = (p0.N + nb_out - 1) / nb_out, t1 = swiglu ? 0u : (p1.N + nb_out - 1) / nb_out;
  Part part = p0;
  if (tile >= t0 + t1) { part = p2; tile -= t0 + t1; }
  else if (tile >= t0) { part = p1; tile -= t0; }
  const unsigned n0 = tile * nb_out;
  const unsigned m0 = ((flags & kFlagGroupsFirst) ? blockIdx.x : blockIdx.y) * tg, rows = min(tg, M - m0), m_tiles = (rows + 127) / 128;
  const unsigned rank = kCluster ? blockIdx.z : 0, ranks = kCluster ? gridDim.z : 1;
  const unsigned k_blocks = (K * elem) / kRowBytes;
  const unsigned run0 = rank * runs / ranks, my_runs = (rank + 1) * runs / ranks - run0;
  const unsigned kb0 = min(run0 * per_run, k_blocks), nkb = min((run0 + my_runs) * per_run, k_blocks) - kb0;
  const unsigned a_bytes = tg * kRowBytes, stage_bytes = a_bytes + NB * kRowBytes;
  const unsigned ring = (smem_u32(dynamic_smem) + 1023u) & ~1023u;
  const unsigned acc_cols = (NB + 31u) & ~31u;
  const unsigned run_cols = ((tg + 127) / 128) * acc_cols;      // tensor-memory columns of one run's accumulators
  const unsigned columns = tmem_columns_for((runs + ranks - 1) / ranks * run_cols);
  if (stages > kMaxRing) stages = kMaxRing;

  // ---- set-up; the first weights are requested before the block meets ----
  const unsigned r0 = (tid & (32 * kW - 1)) >> 3, chunk = tid & 7;     // row-major copies: 16-byte chunk of rows r0, r0 + kRowStep, ...
  const unsigned copy_off = r0 * kRowBytes + ((chunk ^ (r0 & 7)) << 4);
  const size_t w_pitch = kPacked ? 0 : size_t(K) * elem;
  const unsigned w_have = min(nb_out, part.N - n0);
  const uint8_t *w_src, *w_src2 = nullptr;
  if (kPacked) {
    const size_t from = (size_t(kb0) * (((part.N + 255u) / 256u) * 256u) + n0) * kRowBytes;
    w_src = part.w + from;
    if (swiglu) w_src2 = p1.w + from;
  } else {
    const size_t from = size_t(n0 + r0) * w_pitch + size_t(kb0) * kRowBytes + (chunk << 4);
    w_src = part.w + from;
    if (swiglu) w_src2 = p1.w + from;
  }
  const unsigned w_live = kPacked ? min(nb_out, ((part.N + 255u) / 256u) * 256u - n0) * kRowBytes
                                  : (r0 < w_have ? (w_have - r0 + kRowStep - 1) / kRowStep : 0);
  auto copy_weights = [&](unsigned s) {        // packed: one elected thread; row-major: the weight warps
    const unsigned dst = ring + s * stage_bytes + a_bytes;
    if (kPacked) {
      expect_bytes(&full_bar[s], swiglu ? 2 * w_live : w_live);
      bulk_copy(dst, w_src, w_live, &full_bar[s]);
      if (swiglu) bulk_copy(dst + nb_out * kRowBytes, w_src2, w_live, &full_bar[s]);
    } else {
#pragma unroll 4
      for (unsigned j = 0; j < w_live; ++j) cp_async_16(dst + copy_off + j * kRowStep * kRowBytes, w_src + j * kRowStep * w_pitch);
      if (swiglu) {
#pragma unroll 4
        for (unsigned j = 0; j < w_live; ++j)
          cp_async_16(dst + nb_out * kRowBytes + copy_off + j * kRowStep * kRowBytes, w_src2 + j * kRowStep * w_pitch);
      }
    }
  };
  const size_t w_block = kPacked ? size_t(((part.N + 255u) / 256u) * 256u) * kRowBytes : kRowBytes;   // to the next K block
  if (warp == 0) {
    if (elect_one()) {
      for (unsigned s = 0; s < stages; ++s) {
        mbar_init(&full_bar[s], kPacked ? 2 : kEpilogue);
        mbar_init(&empty_bar[s], 1);
      }
      mbar_init(&accum_bar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      if (kPacked && nkb > 0) copy_weights(0);
    }
    __syncwarp();
  }
  if (!kPacked && warp < kW && nkb > 0) copy_weights(0);
  if (warp == kMmaWarp) tmem_alloc(&tmem_slot, columns);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = tmem_slot;
  grid_dependency_release();

  // Row-major producers: every thread's copies of a K block arrive at the slot's barrier by themselves.
  auto produce = [&](auto copy) {
    unsigned s = 0, phase = 1;
    for (unsigned i = 0; i < nkb; ++i) {
      if (i >= stages) mbar_wait(&empty_bar[s], phase, status, kTimeoutEmpty | s);
      copy(i, s);
      cp_async_arrive(&full_bar[s]);
      if (++s == stages) { s = 0; phase ^= 1; }
    }
  };
  if (warp < kW) {
    // ---------------- weights ----------------
    if (kPacked) {
      if (warp == 0) {
        if (elect_one()) {
          unsigned s = 0, phase = 1;
          for (unsigned i = 0; i < nkb; ++i) {
            if (i >= stages) mbar_wait(&empty_bar[s], phase, status, kTimeoutEmpty | s);
            if (i != 0) copy_weights(s);
            w_src += w_block;
            w_src2 += w_block;
            if (++s == stages) { s = 0; phase ^= 1; }
          }
        }
        __syncwarp();
      }
    } else {
      produce([&](unsigned i, unsigned s) {
        if (i != 0) copy_weights(s);
        w_src += w_block;
        w_src2 += w_block;
      });
    }
    grid_dependency_only_wait();
  } else if (warp < kMmaWarp) {
    // ---------------- tokens ----------------
    grid_dependency_only_wait();
    if (kPacked) {
      if (warp == kW) {
        const unsigned live = ((rows + 7u) & ~7u) * kRowBytes;
        const size_t block = size_t(ldx) * kRowBytes;
        const uint8_t* src = x + size_t(kb0) * block + size_t(m0) * kRowBytes;
        if (elect_one()) {
          unsigned s = 0, phase = 1, dst = ring;
          for (unsigned i = 0; i < nkb; ++i) {
            if (i >= stages) mbar_wait(&empty_bar[s], phase, status, kTimeoutEmpty | s);
            expect_bytes(&full_bar[s], live);
            bulk_copy(dst, src, live, &full_bar[s]);
            src += block;
            dst += stage_bytes;
            if (++s == stages) { s = 0; phase ^= 1; dst = ring; }
          }
        }
        __syncwarp();
      }
    } else {
      const size_t row_bytes = size_t(ldx) * elem, step = kRowStep * row_bytes;
      const unsigned live = r0 < rows ? (rows - r0 + kRowStep - 1) / kRowStep : 0;
      const uint8_t* src = x + size_t(m0 + r0) * row_bytes + size_t(kb0) * kRowBytes + (chunk << 4);
      produce([&](unsigned, unsigned s) {
        const unsigned dst = ring + s * stage_bytes + copy_off;
#pragma unroll 4
        for (unsigned j = 0; j < live; ++j) cp_async_16(dst + j * kRowStep * kRowBytes, src + j * step);
        src += kRowBytes;
      });
    }
  } else {
    // ---------------- MMA warp: one elected lane walks the ring ----------------
    // (the whole loop is inside the election: elected anew in every round, an MMA costs ~110 cycles to issue)
    if (elect_one()) {
      const unsigned fmt = kFp8 ? 0u : 1u;
      const unsigned idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((NB >> 3) << 17) | (8u << 24);
      unsigned s = 0, phase = 0, in_run = 0, run_acc = tmem_base;
      unsigned long long a_desc = smem_descriptor(ring);
      const unsigned long long to_b = a_bytes >> 4, to_next = stage_bytes >> 4;
      for (unsigned i = 0; i < nkb; ++i) {
        mbar_wait(&full_bar[s], phase, status, kTimeoutFull | s);
        if (!kPacked) fence_async_shared();      // the copies were generic-proxy writes
        tc_fence_after();
        unsigned acc = run_acc;
        unsigned long long a = a_desc;
        const unsigned long long b_desc = a_desc + to_b;
        for (unsigned mt = 0; mt < m_tiles; ++mt) {
#pragma unroll
          for (unsigned k = 0; k < 4; ++k) mma<kFp8>(acc, a + 2 * k, b_desc + 2 * k, idesc, (in_run | k) != 0);
          acc += acc_cols;
          a += 16384u >> 4;
        }
        tc_commit(&empty_bar[s]);
        if (++in_run == per_run) { in_run = 0; run_acc += run_cols; }
        a_desc += to_next;
        if (++s == stages) { s = 0; phase ^= 1; a_desc = smem_descriptor(ring); }
      }
      tc_commit(&accum_bar);
    }
    __syncwarp();
  }

  // ---------------- epilogue: accumulators (or the filed sums) -> fp32 tile in the ring's memory -> rows of y ----------------
  // The ring is free once the last MMA has committed.  Tile rows are P floats apart: P * 4 = 16 mod 64 bytes keeps
  // both the row-per-lane writes and the row-wise reads free of bank conflicts.
  const unsigned P = NB + 4;
  float* const tile_rows = reinterpret_cast<float*>(dynamic_smem + (ring - smem_u32(dynamic_smem)));
  Out o;
  o.y = part.y; o.bias = part.bias; o.bias2 = p1.bias; o.other = other; o.N = part.N; o.ldy = part.ldy; o.flags = flags;
  o.alpha = o.alpha2 = 1.f;
  o.one_run = runs == 1;
  o.vec = (part.ldy & 7) == 0 && ((reinterpret_cast<size_t>(part.y) | reinterpret_cast<size_t>(part.bias) |
                                   reinterpret_cast<size_t>(p1.bias) | reinterpret_cast<size_t>(other)) & 15) == 0;   // unused pointers are arena-aligned
  float best = 0.f;
  const unsigned special = flags & (kFlagSwiglu | kFlagMulSilu);
  int mode = kGeneral;
  if (o.vec && (part.N & 7) == 0 && !(flags & (kFlagOutF32 | kFlagActMask))) {
    const unsigned plain = flags & (kFlagBias | kFlagResidual);
    if (special == kFlagSwiglu && !(plain & kFlagResidual)) mode = kGateUp;
    else if (special == kFlagMulSilu && plain == 0) mode = kTimesSilu;
    else if (special == 0 && !(flags & kFlagAmax)) mode = int(plain);     // kScale ... kScaleBiasResidual
  }
  auto finish = [&](unsigned count, unsigned m) {
    const unsigned groups = nb_out / 8;
    switch (mode) {
      case kScale: finish_tile<kScale>(tile_rows, P, count, groups, m, n0, o); break;
      case kScaleBias: finish_tile<kScaleBias>(tile_rows, P, count, groups, m, n0, o); break;
      case kScaleResidual: finish_tile<kScaleResidual>(tile_rows, P, count, groups, m, n0, o); break;
      case kScaleBiasResidual: finish_tile<kScaleBiasResidual>(tile_rows, P, count, groups, m, n0, o); break;
      case kGateUp: best = fmaxf(best, finish_tile<kGateUp>(tile_rows, P, count, groups, m, n0, o)); break;
      case kTimesSilu: best = fmaxf(best, finish_tile<kTimesSilu>(tile_rows, P, count, groups, m, n0, o)); break;
      default: best = fmaxf(best, finish_tile<kGeneral>(tile_rows, P, count, groups, m, n0, o)); break;
    }
  };
  const unsigned R = (tg + 31u) & ~31u;      // rows of a filed partial tile: [run][column / 4][row] float4
  float4* const filed = reinterpret_cast<float4*>(partial) +
                        size_t(blockIdx.y * gridDim.x + blockIdx.x) * runs * (NB / 4) * R;
  if (warp < kMmaWarp) {
    // warp w reads TMEM lanes 32 * (w % 4) ..., 16-column units w / 4, w / 4 + kW / 2, ...
    const unsigned quarter = warp & 3, half = warp >> 2, units = NB / 16;
    if (flags & kFlagScaled) {
      o.alpha = (*scale_a) * (*part.scale);
      if (swiglu) o.alpha2 = (*scale_a) * (*p1.scale);
    }
    if (nkb > 0) mbar_wait(&accum_bar, 0, status, kTimeoutAccum);
    tc_fence_after();
    for (unsigned mt = 0; mt < m_tiles; ++mt) {
      if (mt * 128 + quarter * 32 < rows) {        // not for a warp whose rows are all past the tokens
        const unsigned in_tile = quarter * 32 + lane, row = mt * 128 + in_tile;
        const unsigned addr = tmem_base + mt * acc_cols + ((quarter * 32u) << 16);
        for (unsigned c = half; c < units; c += kW / 2) {
          float v[16];
          for (unsigned q = 0; q < max(my_runs, 1u); ++q) {
            unsigned r[16];
            if (q * per_run < nkb) {
              tmem_load16_nowait(addr + q * run_cols + c * 16, r);
              tmem_wait_loads();
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) r[i] = 0u;
            }
            if (kCluster) {
              if (row < rows && q < my_runs) {
                float4* cell = filed + (size_t(run0 + q) * (NB / 4) + c * 4) * R + row;
#pragma unroll
                for (int h = 0; h < 4; ++h)
                  __stcg(cell + size_t(h) * R, make_float4(__uint_as_float(r[4 * h]), __uint_as_float(r[4 * h + 1]),
                                                           __uint_as_float(r[4 * h + 2]), __uint_as_float(r[4 * h + 3])));
              }
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i) v[i] = q == 0 ? __uint_as_float(r[i]) : v[i] + __uint_as_float(r[i]);
            }
          }
          if (!kCluster && row < rows) {        // the staging area holds the tokens' rows only
#pragma unroll
            for (int h = 0; h < 4; ++h)
              *reinterpret_cast<float4*>(tile_rows + in_tile * P + c * 16 + h * 4) =
                  make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
          }
        }
      }
      if (!kCluster) {
        asm volatile("bar.sync 1, %0;" ::"n"(kEpilogue) : "memory");
        finish(min(128u, rows - mt * 128), m0 + mt * 128);
        if (mt + 1 < m_tiles) asm volatile("bar.sync 1, %0;" ::"n"(kEpilogue) : "memory");
      }
    }
    tc_fence_before();
  }
  // Tensor memory goes back before this CTA waits for another one.  tcgen05.alloc blocks until columns are free: if a
  // CTA kept its columns across the cluster barrier, two clusters that share two SMs in opposite order would each hold
  // what the other's missing rank waits for.  The epilogue warps only arrive (their partial tiles are in L2, every
  // tcgen05.ld is complete) and do not wait for the release.
  if (warp == kMmaWarp) {
    asm volatile("bar.sync 2, %0;" ::"n"(kEpilogue + 32) : "memory");
    tc_fence_after();
    tmem_free(tmem_base, columns);
  } else {
    asm volatile("bar.arrive 2, %0;" ::"n"(kEpilogue + 32) : "memory");
  }
  if (kCluster) {
    cluster_arrive();     // release: this rank's partial tiles are filed
    cluster_wait();
  }
  if (kCluster && warp < kMmaWarp) {
    // ---------------- this rank adds the runs of its share of the rows, in order, and finishes them ----------------
    const unsigned share = ((rows + ranks * 8 - 1) / (ranks * 8)) * 8;
    const unsigned first = min(rank * share, rows), count = min(share, rows - first);
    const float4* from = filed + first;
    if (runs <= 2) add_runs<4, 2>(from, tile_rows, P, count, NB / 4, R, runs);
    else if (runs <= 4) add_runs<2, 4>(from, tile_rows, P, count, NB / 4, R, runs);
    else add_runs<1, 8>(from, tile_rows, P, count, NB / 4, R, runs);
    asm volatile("bar.sync 1, %0;" ::"n"(kEpilogue) : "memory");
    finish(count, m0 + first);
  }
  if ((flags & kFlagAmax) && warp < kMmaWarp) {
    best = warp_max(best);
    if (lane == 0) atomicMax(amax_bits, __float_as_uint(__bfloat162float(__float2bfloat16_rn(best))));
  }
}

}  // namespace tk

#define AGI_TK_KERNEL(NAME, CLUSTER, TYPE, FP8, PACKED, IN_CLUSTER)                                                   \
  extern "C" __global__ void CLUSTER __launch_bounds__(tk::kThreads, 2)                                              \
  NAME(const TYPE* x, const float* scale_a, const bf16* other, float* partial, unsigned* amax_bits,                  \
       unsigned* status, unsigned M, unsigned K, unsigned ldx, unsigned flags, unsigned NB, unsigned stages,         \
       unsigned tg, unsigned runs, unsigned per_run, const TYPE* w0, const bf16* bias0, const float* sw0, void* y0,   \
       unsigned N0, unsigned ldy0, const TYPE* w1, const bf16* bias1, const float* sw1, void* y1, unsigned N1,       \
       unsigned ldy1, const TYPE* w2, const bf16* bias2, const float* sw2, void* y2, unsigned N2, unsigned ldy2) {   \
    const tk::Part p0 = {reinterpret_cast<const uint8_t*>(w0), bias0, sw0, y0, N0, ldy0};                            \
    const tk::Part p1 = {reinterpret_cast<const uint8_t*>(w1), bias1, sw1, y1, N1, ldy1};                            \
    const tk::Part p2 = {reinterpret_cast<const uint8_t*>(w2), bias2, sw2, y2, N2, ldy2};                            \
    tk::body<FP8, PACKED, IN_CLUSTER>(reinterpret_cast<const uint8_t*>(x), scale_a, other, partial, amax_bits,       \
                                         status, M, K, ldx, flags, NB, stages, tg, runs, per_run, p0, p1, p2,         \
                                         (flags & kFlagGroupsFirst) ? blockIdx.y : blockIdx.x);                                      \
  }
// The ranks that share K: grid z = C.  Up to 15 clusters of 8, 33 of 4, 74 of 2 are resident at once.
#define AGI_TK_CLUSTER(NAME, TYPE, FP8, PACKED, C) AGI_TK_KERNEL(NAME##_c##C, __cluster_dims__(1, 1, C), TYPE, FP8, PACKED, true)
AGI_TK_KERNEL(agi_gemm_tk_bf16, , bf16, false, false, false)
AGI_TK_CLUSTER(agi_gemm_tk_bf16, bf16, false, false, 2)
AGI_TK_CLUSTER(agi_gemm_tk_bf16, bf16, false, false, 3)
AGI_TK_CLUSTER(agi_gemm_tk_bf16, bf16, false, false, 4)
AGI_TK_CLUSTER(agi_gemm_tk_bf16, bf16, false, false, 8)
AGI_TK_KERNEL(agi_gemm_tk_e4m3, , uint8_t, true, false, false)
AGI_TK_CLUSTER(agi_gemm_tk_e4m3, uint8_t, true, false, 2)
AGI_TK_CLUSTER(agi_gemm_tk_e4m3, uint8_t, true, false, 3)
AGI_TK_CLUSTER(agi_gemm_tk_e4m3, uint8_t, true, false, 4)
AGI_TK_CLUSTER(agi_gemm_tk_e4m3, uint8_t, true, false, 5)
AGI_TK_CLUSTER(agi_gemm_tk_e4m3, uint8_t, true, false, 6)
AGI_TK_CLUSTER(agi_gemm_tk_e4m3, uint8_t, true, false, 8)
// both operands packed
AGI_TK_KERNEL(agi_gemm_tcpk_e4m3, , uint8_t, true, true, false)
AGI_TK_CLUSTER(agi_gemm_tcpk_e4m3, uint8_t, true, true, 2)
AGI_TK_CLUSTER(agi_gemm_tcpk_e4m3, uint8_t, true, true, 3)
AGI_TK_CLUSTER(agi_gemm_tcpk_e4m3, uint8_t, true, true, 4)
AGI_TK_CLUSTER(agi_gemm_tcpk_e4m3, uint8_t, true, true, 6)
AGI_TK_CLUSTER(agi_gemm_tcpk_e4m3, uint8_t, true, true, 8)
// the names under which projections that share their input run as one launch (Q | K | V, gate | up)
AGI_TK_KERNEL(agi_gemm_tc_bf16_x3, , bf16, false, false, false)
AGI_TK_CLUSTER(agi_gemm_tc_bf16_x3, bf16, false, false, 2)
AGI_TK_CLUSTER(agi_gemm_tc_bf16_x3, bf16, false, false, 4)
AGI_TK_CLUSTER(agi_gemm_tc_bf16_x3, bf16, false, false, 8)
AGI_TK_KERNEL(agi_gemm_tc_e4m3_x3, , uint8_t, true, false, false)
AGI_TK_CLUSTER(agi_gemm_tc_e4m3_x3, uint8_t, true, false, 2)
AGI_TK_CLUSTER(agi_gemm_tc_e4m3_x3, uint8_t, true, false, 4)
AGI_TK_CLUSTER(agi_gemm_tc_e4m3_x3, uint8_t, true, false, 8)
#undef AGI_TK_CLUSTER
#undef AGI_TK_KERNEL

// Up to 16 independent bf16 GEMMs that share the activation matrix (the K and V projections of every cross-attention
// block over the context tokens, every block's AdaLN projection) as ONE launch: grid = (segments * ceil(N / NB), token groups), or the other way round;
// segment s multiplies by w[s], adds bias[s] and writes y + s * seg_stride elements.
extern "C" __global__ void __launch_bounds__(tk::kThreads, 2)
agi_gemm_tc_bf16_x16(const bf16* x, bf16* y, unsigned* status, unsigned M, unsigned N, unsigned K, unsigned ldx,
                     unsigned ldy, unsigned flags, unsigned NB, unsigned stages, unsigned tg, unsigned seg_stride,
                     const bf16* w0, const bf16* w1, const bf16* w2, const bf16* w3, const bf16* w4, const bf16* w5,
                     const bf16* w6, const bf16* w7, const bf16* w8, const bf16* w9, const bf16* w10,
                     const bf16* w11, const bf16* w12, const bf16* w13, const bf16* w14, const bf16* w15,
                     const bf16* b0, const bf16* b1, const bf16* b2, const bf16* b3, const bf16* b4, const bf16* b5,
                     const bf16* b6, const bf16* b7, const bf16* b8, const bf16* b9, const bf16* b10,
                     const bf16* b11, const bf16* b12, const bf16* b13, const bf16* b14, const bf16* b15) {
  const unsigned tiles = (N + NB - 1) / NB;
  const unsigned at = (flags & kFlagGroupsFirst) ? blockIdx.y : blockIdx.x, seg = at / tiles;
  const bf16 *w, *b;
  switch (seg) {
    case 0: w = w0; b = b0; break;    case 1: w = w1; b = b1; break;    case 2: w = w2; b = b2; break;
    case 3: w = w3; b = b3; break;    case 4: w = w4; b = b4; break;    case 5: w = w5; b = b5; break;
    case 6: w = w6; b = b6; break;    case 7: w = w7; b = b7; break;    case 8: w = w8; b = b8; break;
    case 9: w = w9; b = b9; break;    case 10: w = w10; b = b10; break; case 11: w = w11; b = b11; break;
    case 12: w = w12; b = b12; break; case 13: w = w13; b = b13; break; case 14: w = w14; b = b14; break;
    default: w = w15; b = b15; break;
  }
  const tk::Part part = {reinterpret_cast<const uint8_t*>(w), b, nullptr, y + size_t(seg) * seg_stride, N, ldy};
  tk::body<false, false, false>(reinterpret_cast<const uint8_t*>(x), nullptr, nullptr, nullptr, nullptr, status, M, K,
                               ldx, flags, NB, stages, tg, 1, K / 64, part, part, part, at % tiles);
}
