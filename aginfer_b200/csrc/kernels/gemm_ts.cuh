// Tensor-core GEMM for few tokens (up to 128): Y[M, N] = epilogue(X[M, K] . W[N, K]^T), bf16 or E4M3 operands, row-major,
// fp32 accumulation in tensor memory.
//
// What bounds it.  Such a product streams its weights once; in a chain of them neither HBM nor the tensor pipe sets the
// time but the chain of steps of each launch behind its dependency wait: tokens in, multiply, results out, and about 1 us
// until the next launch's wait returns (an empty launch of 148 CTAs repeats every 0.5 us, one that stores a word a CTA
// every 1.0 us; a barrier across the part inside one launch takes 1.3 us).  So everything is shaped to keep that chain
// short:
//
//   * weights are the MMA's A operand: 64 or 128 features x a K slice.  With 32 tokens an MMA takes 25 or 41 cycles (64
//     tokens: 33 or 49), so a CTA's slice of 4 - 16 blocks of 128 bytes is 0.2 - 0.8 us of multiplying.  Four warps
//     request as many of its weights as the ring holds before the dependency wait;
//   * K is cut over CTAs until the part is full, which also leaves each of them only its slice of the tokens to bring in
//     (17 x 1536 bf16 read by every CTA takes 0.6 - 0.8 us, a sixth of it 0.35);
//   * what the slices add up to is not gathered here where the next launch can do it: with kFlagSplit the slices leave
//     fp32 partial tiles, one bulk store each, and the norm launch that reads the result anyway adds them, in slice order,
//     on its way in.  The hand-over between launches is the barrier that a gather would need.  Where the next launch is
//     attention or another GEMM, the slices of a tile form a cluster, send each other their shares of the tokens by bulk
//     copies that complete on the receiver's mbarrier, and run the epilogue: scale, bias, activation, residual, SwiGLU;
//   * instructions are fetched cold in a chain of different kernels (16 KB of straight-line code: 2 us, 4 us once the
//     chain's kernels pass 64 KB) and a taken branch costs a lone warp 20 - 40 cycles, so loops are rolled, slots of the
//     ring are several K blocks deep, and the epilogue's one loop is kept from being cloned for each setting of its flags.
//
// Measured in the chain of a 17-token action head, from a launch's dependency wait to the next one's: 1536 x 1536 split
// (144 CTAs) 3.0 us, 1536 x 6144 split 5.4 (weight-streaming kernel of warp-level MMAs: 4.4 and 9.7); 6144 x 1536 with GELU
// in clusters of 3 6.4 (6.7).
//
// Every mbarrier wait is bounded and reports through the status word; nobody waits for another CTA except at the cluster
// barrier.
#pragma once

#include "gemm_tc.cuh"

namespace ts {

using namespace tc;

constexpr unsigned kMaxRing = 12, kCopy = 128;
constexpr unsigned kMmaWarp = 8, kEpilogue = 256, kThreads = kEpilogue + 32;   // 4 weight warps, 4 token warps (all: epilogue), MMA
constexpr unsigned kTimeoutTsFull = 0xB00, kTimeoutTsEmpty = 0xB10, kTimeoutTsAccum = 0xB20, kTimeoutTsGather = 0xB30;

struct Part {
  const uint8_t* w;
  const bf16* bias;
  const float* scale;
  void* y;
  unsigned N, ldy;
};

// Arrives at `bar` once every cp.async this thread has issued so far has landed.
__device__ __forceinline__ void arrive_async(unsigned bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Everything behind the sum over K, for four consecutive features of one token.  The code runs once a launch, cold: it is
// kept short (16 KB of straight-line code cost a launch 2 us), so activations share one expression: x * sigmoid(k(x)).
struct Finish {
  void* y;
  const bf16 *bias, *bias2, *other;
  unsigned N, ldy, flags;
  float alpha, alpha2;
  bool vec;            // rows, bias and pointers allow 8-byte vectors
};
__device__ __forceinline__ float4 load4(const bf16* p, unsigned live, bool vec) {
  if (vec) {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const bf162*>(&q.x)), b = __bfloat1622float2(*reinterpret_cast<const bf162*>(&q.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
  float v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = unsigned(j) < live ? __bfloat162float(p[j]) : 0.f;
  return make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ float scaled(float x, float alpha, float bias) { return __fadd_rn(__fmul_rn(x, alpha), bias); }
__device__ __forceinline__ float rounded(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
// `cell`: where the sums came from, as scratch for rows that take no vectors.
__device__ __forceinline__ float finish4(const float4& sum, const float4& up, const float4& bias, const float4& other, unsigned m,
                                         unsigned n, const Finish& o, float* cell) {
  const unsigned live = min(4u, o.N - n), act = o.flags & kFlagActMask;
  const bool swiglu = (o.flags & kFlagSwiglu) != 0;
  float v[4] = {scaled(sum.x, o.alpha, bias.x), scaled(sum.y, o.alpha, bias.y), scaled(sum.z, o.alpha, bias.z), scaled(sum.w, o.alpha, bias.w)};
  if (swiglu || act == kActSilu || act == kActGeluTanh) {
    // x * sigmoid(k): SiLU and SwiGLU with k = x, GELU with k = 2 u, as 0.5 x (1 + tanh(u)) = x / (1 + exp(-2 u)) (without
    // the cancellation of 1 + tanh for negative x).  Gate and up pass through bf16 as they would between launches.
    float u[4] = {1.f, 1.f, 1.f, 1.f};
    if (swiglu) {
      const float4 b = (o.flags & kFlagBias) ? load4(o.bias2 + n, live, o.vec) : make_float4(0.f, 0.f, 0.f, 0.f);
      u[0] = rounded(scaled(up.x, o.alpha2, b.x)); u[1] = rounded(scaled(up.y, o.alpha2, b.y));
      u[2] = rounded(scaled(up.z, o.alpha2, b.z)); u[3] = rounded(scaled(up.w, o.alpha2, b.w));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float x = swiglu ? rounded(v[j]) : v[j];
      const float k = act == kActGeluTanh ? 1.5957691216057308f * (x + 0.044715f * x * x * x) : x;
      v[j] = x / (1.f + __expf(-k)) * u[j];
    }
  }
  if (act == kActRelu) { v[0] = fmaxf(v[0], 0.f); v[1] = fmaxf(v[1], 0.f); v[2] = fmaxf(v[2], 0.f); v[3] = fmaxf(v[3], 0.f); }
  v[0] = __fadd_rn(v[0], other.x); v[1] = __fadd_rn(v[1], other.y); v[2] = __fadd_rn(v[2], other.z); v[3] = __fadd_rn(v[3], other.w);
  const size_t at = size_t(m) * o.ldy + n;
  float best = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  if (o.vec && !(o.flags & kFlagOutF32)) {
    const bf162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(static_cast<bf16*>(o.y) + at) =
        make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
  } else {
    *reinterpret_cast<float4*>(cell) = make_float4(v[0], v[1], v[2], v[3]);
    best = 0.f;
#pragma unroll 1
    for (unsigned j = 0; j < live; ++j) {
      const float r = cell[j];
      best = fmaxf(best, fabsf(r));
      if (o.flags & kFlagOutF32) static_cast<float*>(o.y)[at + j] = r;
      else static_cast<bf16*>(o.y)[at + j] = __float2bfloat16_rn(r);
    }
  }
  return best;
}

// grid = (feature tiles of all parts, 1, slices of K), block = kThreads.  A tile is TR = 64 or 128 weight rows (with
// kFlagSwiglu TR / 2 gate rows beside the up rows of the same features).  TN: accumulator columns, the tokens rounded up to 16 (64 weight rows: to 8), <= 64; a K block
// holds the tokens rounded up to 8 (an MMA's further columns read what follows).  kFlagSplit:
// the slices (any number) leave their partial tiles in `partial` [slice][tile][token][TR]; otherwise they are the kRanks CTAs
// of a cluster.  Dynamic shared memory: 1024 + stages * depth * (TR + ceil8(M)) * 128 + 1024 (at least M * TR * 4) and, without
// kFlagSplit, the gathered sums: kRanks * ceil(M / kRanks) * TR * 4.
template <bool kFp8, int kRanks>
__device__ __forceinline__ void body(const uint8_t* x, const float* scale_a, const bf16* other, float* partial,
                                     unsigned* amax_bits, unsigned* status, unsigned M, unsigned K, unsigned ldx,
                                     unsigned flags, unsigned TR, unsigned TN, unsigned stages, unsigned depth, const Part& p0, const Part& p1,
                                     const Part& p2) {
  extern __shared__ unsigned char dynamic_smem[];
  __shared__ __align__(8) unsigned long long full_bar[kMaxRing], empty_bar[kMaxRing], accum_bar, gather_bar;
  __shared__ unsigned tmem_slot;

  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned elem = kFp8 ? 1u : 2u;
  const bool swiglu = (flags & kFlagSwiglu) != 0, split = (flags & kFlagSplit) != 0;
  const unsigned out_rows = swiglu ? TR / 2 : TR;
  const unsigned t0 = (p0.N + out_rows - 1) / out_rows, t1 = swiglu ? 0u : (p1.N + out_rows - 1) / out_rows;
  unsigned tile = blockIdx.x;
  Part part = p0;
  if (tile >= t0 + t1) { part = p2; tile -= t0 + t1; }
  else if (tile >= t0) { part = p1; tile -= t0; }
  const unsigned n0 = tile * out_rows;
  const unsigned k_blocks = (K * elem) / kRowBytes, slice = blockIdx.z, slices = gridDim.z;
  const unsigned kb0 = slice * k_blocks / slices, nkb = (slice + 1) * k_blocks / slices - kb0;
  const unsigned weight_bytes = TR * kRowBytes, block_bytes = weight_bytes + ((M + 7) & ~7u) * kRowBytes, stage_bytes = depth * block_bytes;
  const unsigned ring = (smem_u32(dynamic_smem) + 1023u) & ~1023u;
  float* const ring_ptr = reinterpret_cast<float*>(dynamic_smem + (ring - smem_u32(dynamic_smem)));
  const unsigned columns = tmem_columns_for(TN);
  const unsigned share = (M + kRanks - 1) / kRanks;              // consecutive tokens that a rank finishes
  const unsigned first = min(slice * share, M), count = min(share, M - first);
  if (stages > kMaxRing) stages = kMaxRing;

  // ---- set-up; the first weights are requested before the block meets ----
  const unsigned r0 = (tid & (kCopy - 1)) >> 3, chunk = tid & 7;      // 16-byte chunk of rows r0, r0 + 16, ...
  const unsigned copy_off = r0 * kRowBytes + ((chunk ^ (r0 & 7)) << 4);
  const size_t w_pitch = size_t(K) * elem;
  const unsigned w_have = min(out_rows, part.N - n0);
  const size_t w_from = size_t(n0) * w_pitch + size_t(kb0) * kRowBytes + (chunk << 4);
  if (warp == 0) {
    if (elect_one()) {
      for (unsigned s = 0; s < stages; ++s) {
        mbar_init(&full_bar[s], 2 * kCopy);
        mbar_init(&empty_bar[s], 1);
      }
      mbar_init(&accum_bar, 1);
      if (kRanks > 1) mbar_init(&gather_bar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      if (kRanks > 1) expect_bytes(&gather_bar, kRanks * count * TR * 4);    // every rank's sums for this rank's tokens
    }
    __syncwarp();
  }
  // "This rank runs": said before tensor memory is asked for, which may block, and waited for before the first store
  // into a peer's shared memory.
  if (kRanks > 1 && !split) cluster_arrive();
  if (warp == kMmaWarp) tmem_alloc(&tmem_slot, columns);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = tmem_slot;
  grid_dependency_release();

  // Copies of one slot (`depth` K blocks) after the other, each thread's arriving at the slot's barrier by themselves.
  const unsigned slots = (nkb + depth - 1) / depth;
  auto produce = [&](unsigned to, auto copy) {
    unsigned s = 0, phase = 1, left = nkb;
#pragma unroll 1
    for (unsigned i = 0; i < slots; ++i) {
      if (i >= stages) mbar_wait(&empty_bar[s], phase, status, kTimeoutTsEmpty | s);
      unsigned dst = to + s * stage_bytes;
#pragma unroll 1
      for (unsigned n = min(left, depth); n != 0; --n, dst += block_bytes) copy(dst);
      arrive_async(smem_u32(&full_bar[s]));
      left -= depth;
      const bool wrap = s + 1 == stages;
      s = wrap ? 0 : s + 1;
      phase ^= wrap ? 1u : 0u;
    }
  };
  if (warp < 4) {
    // ---------------- weights (rows past N repeat the last one; their results are not stored) ----------------
    if (slots > stages && tid < w_have) {
      // what the ring has no room for yet is at least on its way to L2 (a row's blocks are contiguous)
      const size_t at = size_t(n0 + tid) * w_pitch + size_t(kb0 + stages * depth) * kRowBytes;
      const unsigned bytes = (nkb - stages * depth) * kRowBytes;
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(part.w + at), "r"(bytes) : "memory");
      if (swiglu) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p1.w + at), "r"(bytes) : "memory");
    }
    const uint8_t *base = part.w + w_from, *base2 = swiglu ? p1.w + w_from : base;
    const unsigned first_up = swiglu ? out_rows : TR;      // kFlagSwiglu: from this row of the tile on, rows of the up matrix
    produce(ring + copy_off, [&](unsigned dst) {
#pragma unroll 2
      for (unsigned r = r0; r < TR; r += 16, dst += 16 * kRowBytes) {
        const bool up = r >= first_up;
        cp_async_16(dst, (up ? base2 : base) + min(up ? r - first_up : r, w_have - 1) * w_pitch);
      }
      base += kRowBytes;
      base2 += kRowBytes;
    });
    grid_dependency_only_wait();
  } else if (warp < kMmaWarp) {
    // ---------------- tokens ----------------
    const size_t row_bytes = size_t(ldx) * elem, step = 16 * row_bytes;
    const uint8_t* src = x + size_t(r0) * row_bytes + size_t(kb0) * kRowBytes + (chunk << 4);
    const bool l0 = r0 < M, l1 = r0 + 16 < M, l2 = r0 + 32 < M, l3 = r0 + 48 < M;
    grid_dependency_only_wait();
    produce(ring + weight_bytes + copy_off, [&](unsigned dst) {
      if (l0) cp_async_16(dst, src);
      if (l1) cp_async_16(dst + 16 * kRowBytes, src + step);
      if (l2) cp_async_16(dst + 32 * kRowBytes, src + 2 * step);
      if (l3) cp_async_16(dst + 48 * kRowBytes, src + 3 * step);
      src += kRowBytes;
    });
  } else {
    // ---------------- MMA warp: one elected lane walks the ring ----------------
    if (elect_one()) {
      const unsigned fmt = kFp8 ? 0u : 1u;
      const unsigned idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((TN >> 3) << 17) | ((TR >> 4) << 24);
      const unsigned long long a0 = smem_descriptor(ring), to_b = weight_bytes >> 4, to_block = block_bytes >> 4, to_slot = stage_bytes >> 4;
      unsigned s = 0, phase = 0, more = 0, left = nkb;
      unsigned long long slot = a0;
#pragma unroll 1
      for (unsigned i = 0; i < slots; ++i) {
        mbar_wait(&full_bar[s], phase, status, kTimeoutTsFull | s);
        fence_async_shared();      // the copies were generic-proxy writes
        tc_fence_after();
        unsigned long long a = slot;
#pragma unroll 1
        for (unsigned n = min(left, depth); n != 0; --n, a += to_block) {
#pragma unroll
          for (unsigned k = 0; k < 4; ++k) mma<kFp8>(tmem_base, a + 2 * k, a + to_b + 2 * k, idesc, more | k);
          more = 1;
        }
        tc_commit(&empty_bar[s]);
        left -= depth;
        const bool wrap = s + 1 == stages;
        s = wrap ? 0 : s + 1;
        slot = wrap ? a0 : slot + to_slot;
        phase ^= wrap ? 1u : 0u;
      }
      tc_commit(&accum_bar);
    }
    __syncwarp();
  }

  // ---------------- accumulators: lane = feature, column = token ----------------
  // 128 rows: one a lane; 64 rows: 16 in the lower half of each warp's 32 lanes.
  float* const gathered = ring_ptr + stages * stage_bytes / 4;      // [rank][share][TR]
  if (kRanks > 1 && !split) cluster_wait();                         // every rank runs and expects its sums
  if (warp < kMmaWarp) {
    const unsigned row = (warp & 3) * (TR / 4) + lane;
    const bool live_lane = TR == 128 || lane < 16;
    mbar_wait(&accum_bar, 0, status, kTimeoutTsAccum);
    tc_fence_after();
    // into the ring's memory (every MMA has read it), a token's features side by side
#pragma unroll 1
    for (unsigned c = (warp >> 2) * 16; c < M; c += 32) {
      float v[16];
      tmem_load16(tmem_base + (((warp & 3) * 32u) << 16) + c, v);
      const unsigned live = live_lane ? M - c : 0u;
      unsigned cell = ring + (c * TR + row) * 4;
#pragma unroll
      for (unsigned j = 0; j < 16; ++j) {
        if (j < live) asm volatile("st.shared.f32 [%0], %1;" ::"r"(cell), "f"(v[j]) : "memory");
        cell += TR * 4;
      }
    }
    tc_fence_before();
    fence_async_shared();
    asm volatile("bar.sync 1, %0;" ::"n"(kEpilogue) : "memory");
    if (warp == 0) {
      if (split) {
        if (elect_one()) {
          // one bulk store of the tile (16 stores a thread, a token's row apart: 2900 cycles until they are complete; 1340 so)
          float* to = partial + (size_t(slice) * gridDim.x + blockIdx.x) * M * TR;
          asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(to), "r"(ring), "r"(M * TR * 4) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
        __syncwarp();
      } else if (kRanks > 1 && lane < unsigned(kRanks) && lane * share < M) {
        // lane z: rank z's tokens, to that rank
        const unsigned bytes = min(share, M - lane * share) * TR * 4, to = smem_u32(gathered) + slice * share * TR * 4;
        asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         peer_smem(to, lane)), "r"(ring + lane * share * TR * 4), "r"(bytes), "r"(peer_smem(smem_u32(&gather_bar), lane))
                     : "memory");
      }
    }
  }
  // Tensor memory goes back before this CTA waits for another one (tcgen05.alloc blocks until columns are free).
  if (warp == kMmaWarp) {
    asm volatile("bar.sync 2, %0;" ::"n"(kThreads) : "memory");
    tc_fence_after();
    tmem_free(tmem_base, columns);
  } else {
    asm volatile("bar.arrive 2, %0;" ::"n"(kThreads) : "memory");
  }
  if (split) return;

  // ---------------- this rank's tokens: sum over the ranks in order, epilogue ----------------
  const unsigned group_bits = 31 - __clz(out_rows / 4), groups = 1u << group_bits;
  Finish o;
  o.y = part.y; o.bias = part.bias; o.bias2 = p1.bias; o.other = other; o.N = part.N; o.ldy = part.ldy; o.flags = flags;
  o.alpha = o.alpha2 = 1.f;
  o.vec = ((part.ldy | part.N) & 3) == 0 && ((reinterpret_cast<size_t>(part.y) | reinterpret_cast<size_t>(part.bias) |
                                              reinterpret_cast<size_t>(p1.bias) | reinterpret_cast<size_t>(other)) & 7) == 0;
  if (flags & kFlagScaled) {
    o.alpha = (*scale_a) * (*part.scale);
    if (swiglu) o.alpha2 = (*scale_a) * (*p1.scale);
  }
  // bias and residual of this thread's first item are on their way while the ranks meet
  float4 bias, res;
  auto fetch = [&](unsigned item) {
    const unsigned m = first + (item >> group_bits), n = n0 + (item & (groups - 1)) * 4;
    bias = res = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n < part.N) {
      const unsigned live = min(4u, part.N - n);
      if (flags & kFlagBias) bias = load4(part.bias + n, live, o.vec);
      if (flags & kFlagResidual) res = load4(other + size_t(m) * part.ldy + n, live, o.vec);
    }
  };
  const unsigned items = warp < kMmaWarp ? count * groups : 0;
  if (tid < items) fetch(tid);
  if (kRanks > 1) {
    mbar_wait(&gather_bar, 0, status, kTimeoutTsGather);
    cluster_arrive();   // what this rank was sent has landed; the wait is at the end
  }
  float best = 0.f;
#pragma unroll 1
  for (unsigned item = tid; item < items; item += kEpilogue) {
    const unsigned t = item >> group_bits, g = item & (groups - 1), n = n0 + g * 4;
    asm volatile("" : "+r"(o.flags));      // one loop, not one for each setting of the flags
    if (item != tid) fetch(item);
    if (n >= part.N) continue;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f), up = v;
#pragma unroll
    for (unsigned z = 0; z < unsigned(kRanks); ++z) {
      const float4* cell = reinterpret_cast<const float4*>((kRanks == 1 ? ring_ptr : gathered) + (z * share + t) * TR + g * 4);
      const float4 a = cell[0];
      v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
      if (swiglu) {
        const float4 b = cell[TR / 8];
        up.x += b.x; up.y += b.y; up.z += b.z; up.w += b.w;
      }
    }
    best = fmaxf(best, finish4(v, up, bias, res, first + t, n, o, (kRanks == 1 ? ring_ptr : gathered) + t * TR + g * 4));
  }
  if ((flags & kFlagAmax) && warp < kMmaWarp) {
    best = warp_max(best);
    if (lane == 0) atomicMax(amax_bits, __float_as_uint(__bfloat162float(__float2bfloat16_rn(best))));
  }
  if (kRanks > 1) cluster_wait();     // nobody reads this CTA's shared memory any more
}

}  // namespace ts

// The parameters of agi_gemm_tk_*: NB = weight rows of a tile, tg = accumulator columns.  Three CTAs to an SM, so that a
// launch and its two successors fit: with 112 registers a thread the second successor's weights were requested late.
#define AGI_TS_KERNEL(NAME, CLUSTER, TYPE, FP8, RANKS)                                                                \
  extern "C" __global__ void CLUSTER __launch_bounds__(ts::kThreads, 3)                                              \
  NAME(const TYPE* x, const float* scale_a, const bf16* other, float* partial, unsigned* amax_bits,                  \
       unsigned* status, unsigned M, unsigned K, unsigned ldx, unsigned flags, unsigned NB, unsigned stages,         \
       unsigned tg, unsigned, unsigned depth, const TYPE* w0, const bf16* bias0, const float* sw0, void* y0, unsigned N0,   \
       unsigned ldy0, const TYPE* w1, const bf16* bias1, const float* sw1, void* y1, unsigned N1, unsigned ldy1,      \
       const TYPE* w2, const bf16* bias2, const float* sw2, void* y2, unsigned N2, unsigned ldy2) {                  \
    const ts::Part p0 = {reinterpret_cast<const uint8_t*>(w0), bias0, sw0, y0, N0, ldy0};                            \
    const ts::Part p1 = {reinterpret_cast<const uint8_t*>(w1), bias1, sw1, y1, N1, ldy1};                            \
    const ts::Part p2 = {reinterpret_cast<const uint8_t*>(w2), bias2, sw2, y2, N2, ldy2};                            \
    ts::body<FP8, RANKS>(reinterpret_cast<const uint8_t*>(x), scale_a, other, partial, amax_bits, status, M, K, ldx, \
                         flags, NB, tg, stages, depth, p0, p1, p2);                                                         \
  }
#define AGI_TS_CLUSTER(NAME, TYPE, FP8, C) AGI_TS_KERNEL(NAME##_c##C, __cluster_dims__(1, 1, C), TYPE, FP8, C)
AGI_TS_KERNEL(agi_gemm_ts_bf16, , bf16, false, 1)
AGI_TS_CLUSTER(agi_gemm_ts_bf16, bf16, false, 2)
AGI_TS_CLUSTER(agi_gemm_ts_bf16, bf16, false, 3)
AGI_TS_CLUSTER(agi_gemm_ts_bf16, bf16, false, 4)
AGI_TS_CLUSTER(agi_gemm_ts_bf16, bf16, false, 6)
AGI_TS_CLUSTER(agi_gemm_ts_bf16, bf16, false, 8)
// the names under which projections of few tokens that share their input run as one launch (Q | K | V, gate | up)
AGI_TS_CLUSTER(agi_gemm_tc_bf16_x3, bf16, false, 2)
AGI_TS_CLUSTER(agi_gemm_tc_bf16_x3, bf16, false, 4)
AGI_TS_CLUSTER(agi_gemm_tc_bf16_x3, bf16, false, 8)
#undef AGI_TS_CLUSTER
#undef AGI_TS_KERNEL
