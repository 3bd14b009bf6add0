// Shared device helpers for the sm_100a kernel bundle.
//
// Calling convention of every kernel in the bundle (AgInfer Kernel ABI 1.0,
// docs/kernel-abi-v1.md:39-53 in the reference): `extern "C" __global__`, parameters are
// device pointers, `unsigned` and `float` only, in plan-argument order; nothing is
// allocated, discovered or tuned on the device.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

// Epilogue / behaviour flags shared by the GEMM kernels (one `unsigned flags` parameter).
enum : unsigned {
  kFlagBias = 1u << 0,       // add bias[n]
  kFlagResidual = 1u << 1,   // add residual[m, n] (bf16, same leading dimension as the output)
  kFlagActMask = 0xFu << 4,  // activation applied after bias: 0 none, 1 GELU(tanh), 2 SiLU, 3 ReLU
  kActGeluTanh = 1u << 4,
  kActSilu = 2u << 4,
  kActRelu = 3u << 4,
  kFlagOutF32 = 1u << 8,     // write fp32 instead of bf16
  kFlagScaled = 1u << 9,     // multiply the accumulator by *scale_a * *scale_w (FP8 path)
  kFlagLayerNorm = 1u << 10, // fused prologue: LayerNorm (no affine) over each activation row before the GEMM
  kFlagLnModulate = 1u << 11, // ... followed by y * (1 + scale[k]) + shift[k] (AdaLN)
  kFlagSlab = 1u << 12,       // bulk-stream GEMM: whole K in one slot, rows unpadded, one copy per operand
  kFlagSwiglu = 1u << 13,     // the first two matrices are gate and up of the same width: y = silu(gate) * up
  kFlagMulSilu = 1u << 14,    // y = silu(gate[m, n]) * (...), the gate (bf16, pitch of y) in place of the residual
  kFlagAmax = 1u << 15,       // fold max |y| of the rounded outputs into a zero-initialised word
  kFlagGroupsFirst = 1u << 16,  // the token groups of a weight tile are neighbours in the grid (or walk), not the tiles of a group
};

// Programmatic dependent launch: when the loader launches with programmatic stream
// serialization, a kernel may start while its predecessor drains; `grid_dependency_wait`
// blocks until the predecessor's writes are visible.  Without that launch attribute both
// instructions do nothing.
// `grid_dependency_release` lets the successor's blocks be scheduled (they run their own prologue - barrier
// set-up, weight prefetch - and then block in their own wait until this grid has completed and flushed).
__device__ __forceinline__ void grid_dependency_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Wait first, release afterwards: the successor (and, transitively, everything after it) cannot start before this
// grid's predecessors have all completed.  Kernels that release before they wait let later grids cascade into
// their prologues while much earlier grids are still running, which is harmless for weights but not for data a
// prologue wants to read that an earlier grid of the same replay wrote; one launch of this kind between the
// writer and the readers restores the guarantee.
__device__ __forceinline__ void grid_dependency_wait_then_release() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void grid_dependency_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // release as early as possible, then wait
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void grid_dependency_only_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// True in exactly one lane of a converged warp, the same one every time.  The compiler knows it to be a single
// thread, so instructions that take warp-uniform operands (tcgen05.mma, cp.async.bulk) issue without the operand
// moves that a lane comparison costs: 39 instead of 99 cycles per MMA, 17 instead of 54 per bulk copy.
__device__ __forceinline__ bool elect_one() {
  unsigned p;
  asm volatile("{ .reg .pred q; elect.sync _|q, 0xffffffff; selp.u32 %0, 1, 0, q; }" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over a thread block of up to 1024 threads; every thread receives the result.  A second call in a kernel needs
// another scratch array (or a barrier in between).
__device__ __forceinline__ float block_sum(float v, float* scratch32) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  if (lane == 0) scratch32[warp] = v;
  __syncthreads();
  float total = lane < warps ? scratch32[lane] : 0.f;
  return warp_sum(total);
}
__device__ __forceinline__ float block_max(float v, float* scratch32) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch32[warp] = v;
  __syncthreads();
  float total = lane < warps ? scratch32[lane] : -3.0e38f;
  return warp_max(total);
}

// Maximum of non-negative floats over a warp (they order like their bit patterns) / over a block.
__device__ __forceinline__ float warp_max_nonneg(float v) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}
__device__ __forceinline__ float block_max_nonneg(float v, float* scratch32) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
  v = warp_max_nonneg(v);
  if (lane == 0) scratch32[warp] = v;
  __syncthreads();
  return warp_max_nonneg(lane < warps ? scratch32[lane] : 0.f);
}

__device__ __forceinline__ float e4m3_to_float(uint8_t b) {
  return __half2float(__half(__nv_cvt_fp8_to_halfraw(b, __NV_E4M3)));
}
// Round-to-nearest-even, saturating to +-448 (never NaN for finite input).
__device__ __forceinline__ uint8_t float_to_e4m3(float x) { return __nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3); }
// four of them, the first in the lowest byte; two values per conversion
__device__ __forceinline__ unsigned float4_to_e4m3x4(float a, float b, float c, float d) {
  return unsigned(__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3)) |
         unsigned(__nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3)) << 16;
}

__device__ __forceinline__ float gelu_tanh(float x) {
  const float inner = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.f + tanhf(inner));
}
__device__ __forceinline__ float silu(float x) { return x / (1.f + __expf(-x)); }

// Quotients by a reciprocal and one fused correction of the remainder (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990), shorter than the compiler's division, which was the larger part of a SwiGLU or
// quantisation (FP8 prefill of 288 rows packed 746 -> 694 us).  Used where the operands are few enough to compare every one of
// them with the division: silu in fp32 for all bf16 gates, E4M3 codes for all pairs of a bf16 value and a bf16 amax, the same
// bits.
__device__ __forceinline__ float corrected_quotient(float x, float y, float reciprocal) {
  const float q = x * reciprocal;
  return fmaf(fmaf(-q, y, x), reciprocal, q);
}
// silu of a value that is a bf16.  Below -40 both sides of the division are scaled so that the reciprocal stays a normal
// number; from 20 up 1 + exp(-x) is 1; below -88.7 it is infinite.
__device__ __forceinline__ float silu_bf16(float x) {
  const float s = x < -40.f ? 0x1p-64f : 1.f, y = (1.f + __expf(-x)) * s;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  r = fmaf(fmaf(-y, r, 1.f), r, r);
  const float q = corrected_quotient(x * s, y, r);
  return x > 20.f || x == 0.f ? x : x < -88.7f ? x * 0.f : q;
}
// E4M3 quantisation divides by scale = amax / 448: `Divisor` holds what all values share.  Scales outside the range where
// neither reciprocal nor remainder leaves the normal numbers take the division itself.
struct Divisor {
  float y, r;
  bool plain;
  __device__ __forceinline__ explicit Divisor(float scale)
      : y(scale), r(1.f / scale), plain(!(scale > 0x1p-80f && scale < 0x1p80f)) {}
  __device__ __forceinline__ float operator()(float x) const {      // for conversion to E4M3, which saturates at 448
    const float q = x * r;
    return fabsf(q) > 1e4f || q == 0.f ? q : corrected_quotient(x, y, r);
  }
};

__device__ __forceinline__ float apply_activation(float x, unsigned flags) {
  const unsigned act = flags & kFlagActMask;
  if (act == kActGeluTanh) return gelu_tanh(x);
  if (act == kActSilu) return silu(x);
  if (act == kActRelu) return fmaxf(x, 0.f);
  return x;
}

// 8 bf16 values <-> one 16-byte vector
struct alignas(16) Bf16x8 {
  bf162 v[4];
};
__device__ __forceinline__ void unpack8(const Bf16x8& p, float out[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(p.v[i]);
    out[2 * i] = f.x;
    out[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ Bf16x8 pack8(const float in[8]) {
  Bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(in[2 * i], in[2 * i + 1]);
  return p;
}
