// Row normalisations as warp-shuffle reductions: RMSNorm with gain, LayerNorm (no affine)
// with optional AdaLN modulation y = LN(x) * (1 + scale) + shift.
#pragma once

#include "common.cuh"

// One block per row, `cols` a multiple of 8.  y = bf16(x * rsqrt(mean(x^2) + eps) * gain).  With kAmax the
// kernel also folds max |y| (of the rounded outputs) into *amax_bits, which saves the separate pass of the
// dynamic quantisation that follows (rounding is monotonic, so the rounded maximum is the maximum of the
// rounded values).
// Bound by its chain of dependent steps (a row is 2.5 - 7 KB): with at most one vector per thread (rows up to 8192 wide)
// the row stays in registers between the passes and the gain, a weight, is fetched before the dependency wait.
template <bool kAmax>
__device__ __forceinline__ void rmsnorm_body(const bf16* x, const bf16* gain, bf16* y, unsigned rows, unsigned cols,
                                             unsigned x_stride, unsigned y_stride, float eps, unsigned* amax_bits) {
  __shared__ float scratch[32], scratch2[32];
  const unsigned row = blockIdx.x;
  if (row >= rows) return;
  const Bf16x8* xr = reinterpret_cast<const Bf16x8*>(x + size_t(row) * x_stride);
  const Bf16x8* gr = reinterpret_cast<const Bf16x8*>(gain);
  Bf16x8* yr = reinterpret_cast<Bf16x8*>(y + size_t(row) * y_stride);
  const unsigned vectors = cols / 8;
  float best = 0.f;
  if (vectors <= blockDim.x) {
    const bool live = threadIdx.x < vectors;
    Bf16x8 gv;
    if (live) gv = gr[threadIdx.x];
    grid_dependency_wait();
    float f[8], sumsq = 0.f;
    if (live) {
      unpack8(xr[threadIdx.x], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) sumsq += f[j] * f[j];
    }
    const float rstd = rsqrtf(block_sum(sumsq, scratch) / float(cols) + eps);
    if (live) {
      float g[8];
      unpack8(gv, g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        f[j] = f[j] * rstd * g[j];
        if (kAmax) best = fmaxf(best, fabsf(f[j]));
      }
      yr[threadIdx.x] = pack8(f);
    }
  } else {
    grid_dependency_wait();
    float sumsq = 0.f;
    for (unsigned i = threadIdx.x; i < vectors; i += blockDim.x) {
      float f[8];
      unpack8(xr[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) sumsq += f[j] * f[j];
    }
    const float rstd = rsqrtf(block_sum(sumsq, scratch) / float(cols) + eps);
    for (unsigned i = threadIdx.x; i < vectors; i += blockDim.x) {
      float f[8], g[8];
      unpack8(xr[i], f);
      unpack8(gr[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        f[j] = f[j] * rstd * g[j];
        if (kAmax) best = fmaxf(best, fabsf(f[j]));
      }
      yr[i] = pack8(f);
    }
  }
  if (kAmax) {
    best = block_max_nonneg(best, scratch2);
    if (threadIdx.x == 0) atomicMax(amax_bits, __float_as_uint(__bfloat162float(__float2bfloat16_rn(best))));
  }
}

extern "C" __global__ void agi_rmsnorm_bf16(const bf16* x, const bf16* gain, bf16* y, unsigned rows, unsigned cols,
                                             unsigned x_stride, unsigned y_stride, float eps) {
  rmsnorm_body<false>(x, gain, y, rows, cols, x_stride, y_stride, eps, nullptr);
}

extern "C" __global__ void agi_rmsnorm_amax_bf16(const bf16* x, const bf16* gain, bf16* y, unsigned rows, unsigned cols,
                                                  unsigned x_stride, unsigned y_stride, float eps, unsigned* amax_bits) {
  rmsnorm_body<true>(x, gain, y, rows, cols, x_stride, y_stride, eps, amax_bits);
}

// One block per row.  y = bf16(((x - mean) * rstd) * (1 + scale[c]) + shift[c]) when
// `modulated` != 0 (scale / shift are bf16 vectors of `cols` entries), else plain LayerNorm
// without affine parameters.  Variance is the biased one, computed as mean((x - mean)^2).
// Bit 1 of `modulated`: scale and shift were written before the last launch that released its successors only after its
// own wait, so they may be fetched ahead of the dependency wait.
extern "C" __global__ void agi_layernorm_bf16(const bf16* x, const bf16* scale, const bf16* shift, bf16* y,
                                               unsigned rows, unsigned cols, unsigned x_stride, unsigned y_stride,
                                               float eps, unsigned modulated) {
  __shared__ float scratch[32], scratch2[32];
  const unsigned row = blockIdx.x, vectors = cols / 8;
  if (row >= rows) return;
  const Bf16x8* xr = reinterpret_cast<const Bf16x8*>(x + size_t(row) * x_stride);
  const Bf16x8 *sc_v = reinterpret_cast<const Bf16x8*>(scale), *sh_v = reinterpret_cast<const Bf16x8*>(shift);
  Bf16x8* yr = reinterpret_cast<Bf16x8*>(y + size_t(row) * y_stride);
  auto finish = [&](float f[8], const Bf16x8& sc8, const Bf16x8& sh8, float mean, float rstd) {
    if (modulated) {
      float sc[8], sh[8];
      unpack8(sc8, sc);
      unpack8(sh8, sh);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = (f[j] - mean) * rstd * (1.f + sc[j]) + sh[j];
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = (f[j] - mean) * rstd;
    }
  };
  if (vectors <= blockDim.x) {      // one vector per thread: the row stays in registers
    const unsigned i = threadIdx.x;
    const bool live = i < vectors;
    Bf16x8 sc8, sh8;
    if (live && (modulated & 2u)) { sc8 = sc_v[i]; sh8 = sh_v[i]; }
    grid_dependency_wait();
    float f[8], sum = 0.f, var = 0.f;
    if (live) {
      unpack8(xr[i], f);
      if ((modulated & 3u) == 1u) { sc8 = sc_v[i]; sh8 = sh_v[i]; }
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += f[j];
    }
    const float mean = block_sum(sum, scratch) / float(cols);
    if (live) {
#pragma unroll
      for (int j = 0; j < 8; ++j) var += (f[j] - mean) * (f[j] - mean);
    }
    const float rstd = rsqrtf(block_sum(var, scratch2) / float(cols) + eps);
    if (live) {
      finish(f, sc8, sh8, mean, rstd);
      yr[i] = pack8(f);
    }
    return;
  }
  grid_dependency_wait();
  float sum = 0.f;
  for (unsigned i = threadIdx.x; i < vectors; i += blockDim.x) {
    float f[8];
    unpack8(xr[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += f[j];
  }
  const float mean = block_sum(sum, scratch) / float(cols);
  float var = 0.f;
  for (unsigned i = threadIdx.x; i < vectors; i += blockDim.x) {
    float f[8];
    unpack8(xr[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) var += (f[j] - mean) * (f[j] - mean);
  }
  const float rstd = rsqrtf(block_sum(var, scratch2) / float(cols) + eps);
  for (unsigned i = threadIdx.x; i < vectors; i += blockDim.x) {
    float f[8];
    unpack8(xr[i], f);
    finish(f, modulated ? sc_v[i] : Bf16x8(), modulated ? sh_v[i] : Bf16x8(), mean, rstd);
    yr[i] = pack8(f);
  }
}

// A row of x + the sum of a split product's partial tiles, and its normalisation, in one launch:
//   out[r] = bf16(sum over slices of partial[slice][r] + bias + residual[r]),   y[r] = norm(out[r]).
// The product in front (kFlagSplit) leaves its slices of K unadded, `partial` [slice][column / tile][row][tile]; this launch reads the row anyway and adds them in
// slice order.  One block per row, four columns a thread, every load of the row in flight at once; the statistics take one
// round of shuffles and one barrier (pairs of equal counts are merged: mean and centred squares, no second pass).
// cols a multiple of 128, <= 2048; blockDim = cols / 4; slices <= kNormSlices.
constexpr unsigned kNormSlices = 8;

__device__ __forceinline__ float4 bf16x4(const bf16* p) {
  const uint2 q = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const bf162*>(&q.x)), b = __bfloat1622float2(*reinterpret_cast<const bf162*>(&q.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
// Stores four rounded values and returns them as they were stored.
__device__ __forceinline__ float4 store_bf16x4(bf16* p, const float4& v) {
  const bf162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  uint2 q;
  q.x = *reinterpret_cast<const unsigned*>(&lo);
  q.y = *reinterpret_cast<const unsigned*>(&hi);
  *reinterpret_cast<uint2*>(p) = q;
  const float2 a = __bfloat1622float2(lo), b = __bfloat1622float2(hi);
  return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Four columns of one row: residual + bias + the slices' partial sums in order, rounded and stored.  Addresses are worked out
// ahead of the dependency wait.
struct RowSum {
  const float4* cell;
  size_t step;
  unsigned at, slices;
  __device__ __forceinline__ RowSum(const float* partial, unsigned rows, unsigned cols, unsigned slices, unsigned tile, unsigned row,
                                    unsigned col)
      : cell(reinterpret_cast<const float4*>(partial + (size_t(col / tile) * rows + row) * tile + col % tile)),
        step(size_t((cols + tile - 1) / tile) * rows * tile / 4), at(row * cols + col), slices(slices) {}
  __device__ __forceinline__ float4 operator()(const bf16* residual, bf16* out, const float4& b) const {
    float4 part[kNormSlices];
    const float4* p = cell;
#pragma unroll
    for (unsigned s = 0; s < kNormSlices; ++s, p += step)
      if (s < slices) part[s] = __ldcg(p);
    const float4 r = bf16x4(residual + at);
    float4 v = part[0];
#pragma unroll
    for (unsigned s = 1; s < kNormSlices; ++s)
      if (s < slices) { v.x += part[s].x; v.y += part[s].y; v.z += part[s].z; v.w += part[s].w; }
    v.x = v.x + b.x + r.x; v.y = v.y + b.y + r.y; v.z = v.z + b.z + r.z; v.w = v.w + b.w + r.w;
    return store_bf16x4(out + at, v);
  }
};

// flags: 1 bias, 2 scale and shift, 4 scale and shift may be fetched ahead of the dependency wait.
extern "C" __global__ void __launch_bounds__(512, 2)
agi_layernorm_sum_bf16(const bf16* residual, const float* partial, const bf16* bias, const bf16* scale, const bf16* shift, bf16* out,
                       bf16* y, unsigned rows, unsigned cols, unsigned slices, unsigned tile, float eps, unsigned flags) {
  __shared__ float2 warps_stat[16];
  const unsigned row = blockIdx.x, col = threadIdx.x * 4, warps = blockDim.x >> 5;
  if (row >= rows) return;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 b = zero, sc = zero, sh = zero;
  if (flags & 1u) b = bf16x4(bias + col);
  if ((flags & 6u) == 6u) { sc = bf16x4(scale + col); sh = bf16x4(shift + col); }
  const RowSum sum(partial, rows, cols, slices, tile, row, col);
  grid_dependency_wait();
  if ((flags & 6u) == 2u) { sc = bf16x4(scale + col); sh = bf16x4(shift + col); }
  const float4 v = sum(residual, out, b);
  float mean = 0.25f * ((v.x + v.y) + (v.z + v.w));
  float m2 = ((v.x - mean) * (v.x - mean) + (v.y - mean) * (v.y - mean)) + ((v.z - mean) * (v.z - mean) + (v.w - mean) * (v.w - mean));
  float n = 4.f;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float other = __shfl_xor_sync(0xffffffffu, mean, o), other2 = __shfl_xor_sync(0xffffffffu, m2, o), d = other - mean;
    m2 = m2 + other2 + d * d * (n * 0.5f);
    mean = 0.5f * (mean + other);
    n *= 2.f;
  }
  if ((threadIdx.x & 31) == 0) warps_stat[threadIdx.x >> 5] = make_float2(mean, m2);
  __syncthreads();
  // every warp adds up the (at most 16) warps' statistics for itself
  const unsigned lane = threadIdx.x & 15;
  const float2 mine = lane < warps ? warps_stat[lane] : make_float2(0.f, 0.f);
  mean = half_warp_sum(mine.x) / float(warps);
  const float d = mine.x - mean;
  const float squares = half_warp_sum(lane < warps ? mine.y + 128.f * d * d : 0.f);
  const float rstd = rsqrtf(squares / float(cols) + eps);
  float4 f = make_float4((v.x - mean) * rstd, (v.y - mean) * rstd, (v.z - mean) * rstd, (v.w - mean) * rstd);
  if (flags & 2u) f = make_float4(f.x * (1.f + sc.x) + sh.x, f.y * (1.f + sc.y) + sh.y, f.z * (1.f + sc.z) + sh.z, f.w * (1.f + sc.w) + sh.w);
  store_bf16x4(y + size_t(row) * cols + col, f);
}

// flags: 1 bias.
extern "C" __global__ void __launch_bounds__(512, 2)
agi_rmsnorm_sum_bf16(const bf16* residual, const float* partial, const bf16* bias, const bf16* gain, bf16* out, bf16* y,
                     unsigned rows, unsigned cols, unsigned slices, unsigned tile, float eps, unsigned flags) {
  __shared__ float warps_stat[16];
  const unsigned row = blockIdx.x, col = threadIdx.x * 4, warps = blockDim.x >> 5;
  if (row >= rows) return;
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (flags & 1u) b = bf16x4(bias + col);
  const float4 g = bf16x4(gain + col);
  const RowSum sum(partial, rows, cols, slices, tile, row, col);
  grid_dependency_wait();
  const float4 v = sum(residual, out, b);
  const float mine = warp_sum((v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w));
  if ((threadIdx.x & 31) == 0) warps_stat[threadIdx.x >> 5] = mine;
  __syncthreads();
  const unsigned lane = threadIdx.x & 15;
  const float squares = half_warp_sum(lane < warps ? warps_stat[lane] : 0.f);
  const float rstd = rsqrtf(squares / float(cols) + eps);
  store_bf16x4(y + size_t(row) * cols + col, make_float4(v.x * rstd * g.x, v.y * rstd * g.y, v.z * rstd * g.z, v.w * rstd * g.w));
}
