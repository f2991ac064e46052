// SRHT normalise-rotate of a query, for the stand-alone query preparation and the chain.  Fixed fp32 operation order, the
// same as the key coder's (keycode.cuh).
#pragma once
#include "common.cuh"

namespace pk {
namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ void unpack8(uint4 v, float* out) {
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    out[2 * i] = __uint_as_float(w[i] << 16);
    out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// x: dims [4*lane, 4*lane+4) of the group-mean query (bf16 values as floats); sg: their SRHT signs.
// Adjacent pairwise tree for the norm, butterflies in ascending distance, spread over 32 lanes.  Returns the bf16 norm.
__device__ __forceinline__ float rotate4(float (&x)[4], const float (&sg)[4], int lane) {
  float t0 = __fadd_rn(__fmul_rn(x[0], x[0]), __fmul_rn(x[1], x[1]));
  float t1 = __fadd_rn(__fmul_rn(x[2], x[2]), __fmul_rn(x[3], x[3]));
  float sum = __fadd_rn(t0, t1);
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, off));
  const float n = bfround(__fsqrt_rn(sum));
  const float den = fmaxf(n, bfround(1e-8f));
#pragma unroll
  for (int i = 0; i < 4; i++) x[i] = __fmul_rn(bfround(__fdiv_rn(x[i], den)), sg[i]);
  {  // h = 1, 2 inside the lane
    float a = x[0], b = x[1], c = x[2], d = x[3];
    x[0] = __fadd_rn(a, b), x[1] = __fsub_rn(a, b), x[2] = __fadd_rn(c, d), x[3] = __fsub_rn(c, d);
    a = x[0], b = x[1], c = x[2], d = x[3];
    x[0] = __fadd_rn(a, c), x[2] = __fsub_rn(a, c), x[1] = __fadd_rn(b, d), x[3] = __fsub_rn(b, d);
  }
#pragma unroll
  for (int bit = 1; bit < 32; bit <<= 1)  // h = 4 .. 64 across lanes
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float pv = __shfl_xor_sync(0xffffffffu, x[i], bit);
      x[i] = (lane & bit) ? __fsub_rn(pv, x[i]) : __fadd_rn(x[i], pv);
    }
#pragma unroll
  for (int i = 0; i < 4; i++) x[i] = bfround(__fmul_rn(x[i], 0.08838834764831845f));
  return n;
}

}  // namespace
}  // namespace pk
