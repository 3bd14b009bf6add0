// The quotient helpers of the kernel bundle beside the divisions they stand for, with nothing rounded in between.
#include "elementwise.cuh"

// corrected[i], divided[i]: silu of x[i] both ways, in fp32.
extern "C" __global__ void probe_silu_f32(const bf16* x, float* corrected, float* divided, unsigned count) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const float v = __bfloat162float(x[i]);
    corrected[i] = silu_bf16(v);
    divided[i] = silu(v);
  }
}

// differ[b] = of the 65536 bf16 values x, held to +-amax, those whose E4M3 code of x / (amax / 448) is not the division's; amax
// is the bf16 with the bits first_amax + b, b this block.
extern "C" __global__ void probe_e4m3_codes(unsigned* differ, unsigned first_amax) {
  const float amax = __uint_as_float((first_amax + blockIdx.x) << 16);
  const float scale = amax > 0.f ? __fdiv_rn(amax, 448.f) : 1.f;
  const Divisor divide(scale);
  unsigned found = 0;
  for (unsigned v = threadIdx.x; v < 8192; v += blockDim.x) {
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float x = __uint_as_float((v * 8 + j) << 16);
      f[j] = fabsf(x) > amax ? copysignf(amax, x) : x;
    }
    const uint2 codes = quantize8(pack8(f), divide);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      found += uint8_t((j < 4 ? codes.x : codes.y) >> (j % 4 * 8)) != float_to_e4m3(__fdiv_rn(f[j], scale));
  }
  if (found != 0) atomicAdd(&differ[blockIdx.x], found);
}
