// Coding of one key by four lanes, 32 dimensions (four 8-dim subspaces) per lane: SRHT normalise-rotate, 8-bit sign code,
// 4-bit (sign | 3-bit level) code, rerank weight.  The arithmetic of polar_cache.batch_encode
// (cache_hub/polar_cache.py:924-978) with its bf16 roundings, bit for bit.
//
// What bounds it is instruction issue, so everything runs two elements at a time: pair i of a lane holds its dimensions
// i and i + 16 in packed fp32 operations (every butterfly but one, all trees, two subspaces side by side), the levels and
// centre products run on packed bf16.  Four lanes per key instead of eight halve what every lane repeats (norm, addresses,
// stores) and leave two butterflies between lanes instead of three.  Three things need an argument:
//   * x / den rounded to bf16, with x and den bf16: a product with the approximate reciprocal gives the same bf16.  A
//     rounding boundary m has 9 significant bits, the last one set; x = m * den is impossible (m times an integer keeps at
//     least 9 significant bits, x has 8), and x - m * den is a multiple of the last place of m * den, which has 17 bits,
//     so the quotient stays 2^-17 (relative) away from every boundary.  The product is off by less than 2^-21.
//     (Quotients below 2^-126, with their coarser spacing, are outside this argument and of no effect on a rotated key.)
//   * square roots and weights rounded to bf16 are taken from approximate operations unless the result lies within a few
//     last places of a rounding boundary; then they are computed again with correctly rounded ones.
//   * the level search picks its next threshold by packed multiply-adds whose bf16 roundings land exactly on the
//     thresholds (checked over all bf16 values).
#pragma once
#include "common.cuh"

namespace pk {
namespace {

typedef unsigned long long f32x2;   // two fp32 values, the first in the low half

__device__ __forceinline__ f32x2 pair(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void split(f32x2 p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p)); }
__device__ __forceinline__ f32x2 add_2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul_2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma_2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// bf16 pair (hi << 16 | lo), rounded to nearest even
__device__ __forceinline__ uint32_t bf16_2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t bf16_2(f32x2 p) {
  float a, b;
  split(p, a, b);
  return bf16_2(a, b);
}
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
// packed bf16 operations on words
__device__ __forceinline__ uint32_t gt_b2(uint32_t a, uint32_t b) {   // 1.0 where a > b, else 0
  uint32_t r;
  asm("set.gt.bf16x2.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t fma_b2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__host__ __device__ constexpr uint32_t b2(uint32_t bits) { return bits | (bits << 16); }
// thresholds 0.0845 0.1699 0.2578 0.3496 0.4492 0.5586 0.6914 (bf16); the search needs T0, T1, T3 and the steps between them
constexpr uint32_t LV_T0 = b2(0x3dad), LV_T1 = b2(0x3e2e), LV_T3 = b2(0x3eb3);
constexpr uint32_t LV_D51 = b2(0x3ec7), LV_D40 = b2(0x3ebb), LV_D20 = b2(0x3e32), LV_D64 = b2(0x3d8c);   // T5-T1, T4-T0, T2-T0, (T6-T4)-(T2-T0)
// centres 0.0420 0.1270 0.2129 0.3027 0.3965 0.5 0.6172 0.7617 (bf16), low and high bytes of the eight
constexpr uint32_t CEN_LO0 = 0x9b5a022cu, CEN_LO1 = 0x431e00cbu, CEN_HI0 = 0x3e3e3e3du, CEN_HI1 = 0x3f3f3f3eu;

// levels of two magnitudes, in the low three bits of either half: 128 + level as bf16 has the level in the low bits of its pattern
__device__ __forceinline__ uint32_t level_b2(uint32_t a) {
  const uint32_t m1 = gt_b2(a, LV_T3);
  const uint32_t m2 = gt_b2(a, fma_b2(m1, LV_D51, LV_T1));
  const uint32_t m3 = gt_b2(a, fma_b2(m2, fma_b2(m1, LV_D64, LV_D20), fma_b2(m1, LV_D40, LV_T0)));
  return fma_b2(m1, b2(0x4080), fma_b2(m2, b2(0x4000), fma_b2(m3, b2(0x3f80), b2(0x4300))));
}
// centres of two levels l.lo, l.hi < 8, by byte permutes
__device__ __forceinline__ uint32_t centre_b2(uint32_t l) {
  const uint32_t sel = l | (l >> 12);   // three bits per nibble
  return __byte_perm(__byte_perm(CEN_LO0, CEN_LO1, sel), __byte_perm(CEN_HI0, CEN_HI1, sel), 0x5140);
}

struct KeyCode {
  uint32_t codes;    // sign codes of the lane's four subspaces, low byte first
  uint2 weights;     // their rerank weights, four bf16
  uint4 packed;      // their 4-bit codes
};

// What lane s of a key's four needs besides the key: sign masks of its dimensions (bits 15 and 31 of a word: the dimension is
// negated) and which side of the two cross-lane butterflies it is on.
__device__ __forceinline__ uint4 sign_mask(uint4 signs) {
  return make_uint4(signs.x & 0x80008000u, signs.y & 0x80008000u, signs.z & 0x80008000u, signs.w & 0x80008000u);
}
__device__ __forceinline__ uint4 flip(uint4 raw, uint4 mask) {
  return make_uint4(raw.x ^ mask.x, raw.y ^ mask.y, raw.z ^ mask.z, raw.w ^ mask.w);
}
struct RotateLane {
  f32x2 side[2];
  __device__ __forceinline__ explicit RotateLane(int s) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const float f = ((s >> i) & 1) ? -1.0f : 1.0f;
      side[i] = pair(f, f);
    }
  }
};

// adjacent pairwise tree over eight pairs, both halves at once
__device__ __forceinline__ f32x2 tree8(const f32x2* t) {
  return add_2(add_2(add_2(t[0], t[1]), add_2(t[2], t[3])), add_2(add_2(t[4], t[5]), add_2(t[6], t[7])));
}
// whether v, off by a few last places, might round to another bf16
template <int MARGIN>
__device__ __forceinline__ bool near_boundary(float v) {
  return ((__float_as_uint(v) & 0xffffu) - (0x8000u - MARGIN)) < 2u * MARGIN;
}
__device__ __forceinline__ float sqrt_approx(float x) {   // within 2 last places
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// key: the lane's 32 dimensions of the key (bf16), their signs applied; all 32 lanes of the warp take part (eight keys).
// Lanes that share a key are APART from each other.
template <int APART>
__device__ __forceinline__ KeyCode code_key(const uint4 (&key)[4], const RotateLane& rl) {
  uint32_t in[16];
#pragma unroll
  for (int i = 0; i < 4; i++) in[4 * i] = key[i].x, in[4 * i + 1] = key[i].y, in[4 * i + 2] = key[i].z, in[4 * i + 3] = key[i].w;
  f32x2 x[16], t[16];
#pragma unroll
  for (int j = 0; j < 8; j++) {   // pair i = dimensions i, i + 16; the sign flips do not change the norm
    const uint32_t a = in[j], b = in[j + 8];
    x[2 * j] = pair(lo_f(a), lo_f(b));
    x[2 * j + 1] = pair(hi_f(a), hi_f(b));
  }
#pragma unroll
  for (int i = 0; i < 16; i++) t[i] = mul_2(x[i], x[i]);
  float n;
  {
    float a, b;
    split(add_2(tree8(t), tree8(t + 8)), a, b);
    float sum = __fadd_rn(a, b);
#pragma unroll
    for (int off = 1; off < 4; off <<= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, off * APART));
    n = sqrt_approx(sum);
    if (near_boundary<8>(n)) n = __fsqrt_rn(sum);
    n = bfround(n);
  }
  {
    const float r = rcp_approx(fmaxf(n, bfround(1e-8f)));
    const f32x2 rr = pair(r, r);
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t q = bf16_2(mul_2(x[i], rr));
      x[i] = pair(lo_f(q), hi_f(q));
    }
  }
  // Hadamard butterflies h = 1, 2, 4, 8 between pairs, h = 16 inside a pair, h = 32, 64 between lanes
  const f32x2 minus = pair(-1.0f, -1.0f);
#pragma unroll
  for (int h = 1; h < 16; h <<= 1)
#pragma unroll
    for (int i = 0; i < 16; i++)
      if ((i & h) == 0) {
        const f32x2 a = x[i], b = x[i + h];
        x[i] = add_2(a, b);
        x[i + h] = fma_2(b, minus, a);
      }
#pragma unroll
  for (int i = 0; i < 16; i++) {
    float a, b;
    split(x[i], a, b);
    x[i] = pair(__fadd_rn(a, b), __fsub_rn(a, b));
  }
#pragma unroll
  for (int st = 0; st < 2; st++)
#pragma unroll
    for (int i = 0; i < 16; i++) {
      float a, b;
      split(x[i], a, b);
      const f32x2 p = pair(__shfl_xor_sync(0xffffffffu, a, APART << st), __shfl_xor_sync(0xffffffffu, b, APART << st));
      x[i] = fma_2(x[i], rl.side[st], p);   // x + p on one side, p - x on the other
    }
  // per half of the pairs (i < 8: subspaces 0 and 2 of the lane, i >= 8: 1 and 3)
  uint32_t pk[4], code[4];
  float r[4], al[4], w[4];
  const f32x2 sc = pair(0.08838834764831845f, 0.08838834764831845f), zero = pair(0.0f, 0.0f);
#pragma unroll
  for (int g = 0; g < 2; g++) {
    // scaled and rounded coordinates; word i = dimensions i and i + 16.  Adding +0 turns -0 into +0, which counts as
    // non-negative
    uint32_t y[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      y[i] = bf16_2(fma_2(x[8 * g + i], sc, zero));
      x[8 * g + i] = pair(lo_f(y[i]), hi_f(y[i]));
      t[i] = mul_2(x[8 * g + i], x[8 * g + i]);
    }
    {
      float s0, s1;
      split(tree8(t), s0, s1);
      float r0 = sqrt_approx(s0), r1 = sqrt_approx(s1);
      if (near_boundary<8>(r0) || near_boundary<8>(r1)) r0 = __fsqrt_rn(s0), r1 = __fsqrt_rn(s1);
      r[g] = bfround(r0), r[g + 2] = bfround(r1);
    }
    const f32x2 ri = pair(rcp_approx(fmaxf(r[g], bfround(1e-8f))), rcp_approx(fmaxf(r[g + 2], bfround(1e-8f))));
    uint32_t u[4];   // per two dimensions: bytes 0 and 2 hold the nibble pairs of the two subspaces
#pragma unroll
    for (int j = 0; j < 4; j++) {
      uint32_t lv[2], au[2];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int i = 2 * j + k;
        const uint32_t a = au[k] = bf16_2(mul_2(x[8 * g + i], ri)) & 0x7fff7fffu;
        lv[k] = (level_b2(a) & 0x00070007u) | ((~y[i] >> 12) & 0x00080008u);   // sign | level nibbles
      }
      const uint32_t nib = lv[0] | (lv[1] << 8);
      u[j] = nib | (nib >> 4);
      // centres of the four levels by byte permutes (selector: three bits per nibble), then centre x magnitude in bf16
      const uint32_t sel = (nib | (nib >> 12)) & 0x7777u;
      const uint32_t cl = __byte_perm(CEN_LO0, CEN_LO1, sel), ch = __byte_perm(CEN_HI0, CEN_HI1, sel);
      const uint32_t p0 = fma_b2(__byte_perm(cl, ch, 0x5140), au[0], b2(0x8000)), p1 = fma_b2(__byte_perm(cl, ch, 0x7362), au[1], b2(0x8000));
      t[2 * j] = pair(lo_f(p0), hi_f(p0));
      t[2 * j + 1] = pair(lo_f(p1), hi_f(p1));
    }
    split(tree8(t), al[g], al[g + 2]);
    const uint32_t p01 = __byte_perm(u[0], u[1], 0x6240), p23 = __byte_perm(u[2], u[3], 0x6240);
    pk[g] = __byte_perm(p01, p23, 0x5410), pk[g + 2] = __byte_perm(p01, p23, 0x7632);
  }
  bool near = false;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    al[i] = fmaxf(al[i], 1e-6f);
    w[i] = __fmul_rn(__fmul_rn(r[i], rcp_approx(al[i])), n);
    near = near || near_boundary<16>(w[i]);
    uint32_t v = (pk[i] >> 3) & 0x11111111u;   // bit 3 of every nibble, gathered: the sign code
    v = (v | (v >> 3)) & 0x03030303u;
    v = (v | (v >> 6)) & 0x000f000fu;
    code[i] = (v | (v >> 12)) & 0xffu;
  }
  if (near)
#pragma unroll
    for (int i = 0; i < 4; i++) w[i] = __fmul_rn(__fdiv_rn(r[i], al[i]), n);
  KeyCode out;
  out.codes = code[0] | (code[1] << 8) | (code[2] << 16) | (code[3] << 24);
  out.weights = make_uint2(bf16_2(w[0], w[1]), bf16_2(w[2], w[3]));
  out.packed = make_uint4(pk[0], pk[1], pk[2], pk[3]);
  return out;
}

}  // namespace
}  // namespace pk
