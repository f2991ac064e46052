// Device pieces of the retrieval chain that its kernels share: query preparation, ranking of the clusters of a subspace,
// tier tables and look-ups, the candidate list, the 4-bit rerank.
#pragma once
#include "common.cuh"
#include "kernels.cuh"
#include "rotate.cuh"

namespace pk {
namespace {

// byte k (0..3) of w, zero-extended: one PRMT
__device__ __forceinline__ unsigned byte_of(uint32_t w, int k) { return __byte_perm(w, 0, 0x4440 | k); }

// Sorts the 128 keys of a warp (4 per lane, element index e = 4 * lane + r) into DESCENDING order of e with a
// bitonic network: exchanges at distance < 4 stay inside a lane, the others are xor shuffles.  Keys are distinct.
// The merges run as loops over two small bodies: fully unrolled the network is long code that every warp runs
// once, and a kernel that starts with it waits for instruction fetches (a third of its stalls, measured).
// A block that has to end ascending is sorted as complements, so every exchange inside a lane is one max and one min.
__device__ __forceinline__ void lane_exchange(unsigned (&v)[4], int r, int l, bool up) {
  const unsigned a = v[r], b = v[l], mx = max(a, b), mn = min(a, b);
  v[r] = up ? mx : mn;
  v[l] = up ? mn : mx;
}
__device__ __forceinline__ void warp_sort_desc_128(unsigned (&v)[4], int lane) {
  lane_exchange(v, 0, 1, true);
  lane_exchange(v, 2, 3, false);
#pragma unroll 1
  for (int k = 4; k <= 128; k <<= 1) {
    const unsigned flip = ((lane << 2) & k) ? 0xffffffffu : 0u;   // blocks with this bit set end ascending
#pragma unroll
    for (int r = 0; r < 4; r++) v[r] ^= flip;
#pragma unroll 1
    for (int lj = k >> 3; lj > 0; lj >>= 1) {
      const bool take_max = (lane & lj) == 0;   // the lower element of a pair keeps the maximum
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const unsigned o = __shfl_xor_sync(0xffffffffu, v[r], lj);
        v[r] = take_max ? max(v[r], o) : min(v[r], o);
      }
    }
    lane_exchange(v, 0, 2, true), lane_exchange(v, 1, 3, true);
    lane_exchange(v, 0, 1, true), lane_exchange(v, 2, 3, true);
#pragma unroll
    for (int r = 0; r < 4; r++) v[r] ^= flip;
  }
}

// Ranks the 256 clusters of a subspace by (score descending, id ascending), the scores being the sums of +-q over the
// bits of the cluster id.  The complement of an id has exactly the negated score, so the order is its own mirror image:
// with a cluster at position e its complement is at position 255 - e, ties included (equal scores are ascending in the ids,
// their negatives in the complements read backwards; of the scores that are zero the ids below 128 come first).  Only the
// first 128 positions are sorted, one cluster of every pair: that of the positive score, or the lower id.  On return
// position e = 4 * lane + r is cluster 255 - (key[r] & 255), position 255 - e cluster key[r] & 255.
// Register r of a lane starts with cluster c = 32 * r + lane: the first five terms of the score (bits 0..4 of c) are the
// lane's, the next two the register's, bit 7 is clear; the sum is taken in the order j = 0..7.
__device__ __forceinline__ void rank_subspace(unsigned (&key)[4], const float* q8, int lane) {
  float qv[8];
#pragma unroll
  for (int j = 0; j < 8; j++) qv[j] = q8[j];
  float s5 = 0.0f;
#pragma unroll
  for (int j = 0; j < 5; j++) s5 = __fadd_rn(s5, ((lane >> j) & 1) ? qv[j] : -qv[j]);
#pragma unroll
  for (int rr = 0; rr < 4; rr++) {
    float sc = s5;
#pragma unroll
    for (int j = 5; j < 7; j++) sc = __fadd_rn(sc, ((rr >> (j - 5)) & 1) ? qv[j] : -qv[j]);
    const unsigned bits = f2bf(__fadd_rn(sc, -qv[7])), mag = bits & 0x7fffu;   // a zero of either sign counts as positive
    const unsigned c = 32 * rr + lane, id = (bits & 0x8000u) && mag ? 255u - c : c;
    key[rr] = (mag << 8) | (255u - id);
  }
  warp_sort_desc_128(key, lane);
}

// Sixteen times the sum over the 16 subspaces of a key of the tier count of its code.  lut: [16][128] bytes, entry c of a
// subspace is nibble c >> 7 of byte c & 127: 128 bytes, one word per bank, so the 32 look-ups of a warp never conflict.
// The integer ALU bounds this (half rate on sm_100a): eight of its instructions per four look-ups.  The four table
// bytes are joined by multiply-adds, which run on the FMA pipe; c256 = 256 comes from a kernel argument, because
// the compiler turns a multiplication by a known power of two into ALU shifts.
__device__ __forceinline__ unsigned tier_sum16(uint4 cw, const uint8_t* lut, unsigned c256) {
  const uint32_t w4[4] = {cw.x, cw.y, cw.z, cw.w};
  unsigned acc = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t w = w4[i], at = w & 0x7f7f7f7fu;
    const uint8_t* t = lut + 4 * i * 128;
    const unsigned b0 = t[byte_of(at, 0)], b1 = t[128 + byte_of(at, 1)], b2 = t[256 + byte_of(at, 2)], b3 = t[384 + byte_of(at, 3)];
    const uint32_t v = ((b3 * c256 + b2) * c256 + b1) * c256 + b0;
    uint32_t high;   // 0xff where the code is 128 or more: its nibble is the high one (the intrinsic drops the sign mode)
    asm("prmt.b32 %0, %1, %2, 0xba98;" : "=r"(high) : "r"(w), "r"(0u));
    // the wanted nibble of every byte in place, times 16 (low) or 1 (high)
    acc = __dp4a(v & (high ^ 0x0f0f0f0fu), (high & 0x01010101u) | (~high & 0x10101010u), acc);
  }
  return acc;
}

// The tier counts of four codes of ONE subspace, one per byte; lut: its 128 bytes (see tier_sum16).
__device__ __forceinline__ uint32_t tier_bytes(uint32_t w, const uint8_t* t, unsigned c256) {
  const uint32_t at = w & 0x7f7f7f7fu;
  const unsigned b0 = t[byte_of(at, 0)], b1 = t[byte_of(at, 1)], b2 = t[byte_of(at, 2)], b3 = t[byte_of(at, 3)];
  const uint32_t v = ((b3 * c256 + b2) * c256 + b1) * c256 + b0;
  uint32_t high;
  asm("prmt.b32 %0, %1, %2, 0xba98;" : "=r"(high) : "r"(w), "r"(0u));
  return (((v >> 4) & high) | (v & ~high)) & 0x0f0f0f0fu;
}

__device__ __forceinline__ void unpack4(uint2 v, float* out) {
  out[0] = __uint_as_float(v.x << 16), out[1] = __uint_as_float(v.x & 0xffff0000u);
  out[2] = __uint_as_float(v.y << 16), out[3] = __uint_as_float(v.y & 0xffff0000u);
}

struct RerankSmem {
  float lev[16][32];  // lev[nibble][lane]
  float q[128];
};

__device__ __forceinline__ void rerank_setup(RerankSmem& sm, const RerankArgs& a, int64_t bh, int tid, int nthreads) {
  for (int i = tid; i < 16 * 32; i += nthreads) {
    const int nib = i >> 5;
    const float c = bf2f(a.centers[nib & 7]);
    sm.lev[nib][i & 31] = (nib & 8) ? c : -c;
  }
  for (int i = tid; i < 128; i += nthreads) sm.q[i] = bf2f(a.q_blocks[bh * 128 + i]);
}

// FAST: key-major, 16-byte aligned records.  Returns the fp32 score of key `key`.
template <bool FAST>
__device__ __forceinline__ float rerank_one(const RerankSmem& sm, const RerankArgs& a, const uint8_t* k4,
                                            const uint16_t* w, int64_t key, float qn, int lane, uint16_t* v4b_row,
                                            int64_t v4b_sub_stride) {
  uint32_t code[16];
  uint32_t wt[8];
  if (FAST) {
    const uint4* cp = reinterpret_cast<const uint4*>(k4 + key * a.k4_l);
    const uint4* wp = reinterpret_cast<const uint4*>(w + key * a.w_l);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint4 v = cp[i];
      code[4 * i] = v.x, code[4 * i + 1] = v.y, code[4 * i + 2] = v.z, code[4 * i + 3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint4 v = wp[i];
      wt[4 * i] = v.x, wt[4 * i + 1] = v.y, wt[4 * i + 2] = v.z, wt[4 * i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int s = 0; s < 16; s++) {
      const uint8_t* cp = k4 + s * a.k4_s + key * a.k4_l;
      code[s] = (uint32_t)cp[0] | ((uint32_t)cp[1] << 8) | ((uint32_t)cp[2] << 16) | ((uint32_t)cp[3] << 24);
    }
#pragma unroll
    for (int s = 0; s < 8; s++)
      wt[s] = (uint32_t)w[(2 * s) * a.w_s + key * a.w_l] | ((uint32_t)w[(2 * s + 1) * a.w_s + key * a.w_l] << 16);
  }
  float acc = 0.0f;
#pragma unroll
  for (int s = 0; s < 16; s++) {
    const float4 q0 = *reinterpret_cast<const float4*>(&sm.q[8 * s]);
    const float4 q1 = *reinterpret_cast<const float4*>(&sm.q[8 * s + 4]);
    const float qv[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    float dot = 0.0f;
    float lv[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      lv[j] = sm.lev[(code[s] >> (4 * j)) & 0xFu][lane];
      dot = __fmaf_rn(lv[j], qv[j], dot);
    }
    if (v4b_row) {
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; j++) o[j] = (uint32_t)f2bf(lv[2 * j]) | ((uint32_t)f2bf(lv[2 * j + 1]) << 16);
      *reinterpret_cast<uint4*>(v4b_row + s * v4b_sub_stride) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    const float wf = __uint_as_float((s & 1) ? (wt[s >> 1] & 0xffff0000u) : (wt[s >> 1] << 16));
    acc = __fmaf_rn(dot, wf, acc);
  }
  return __fmul_rn(acc, qn);
}

// The rerank of one candidate from its key-major record, for kernels that rank many candidates per block.
// Levels are looked up two at a time: entry v of lev2 holds the bf16 levels of the nibbles v & 15 and v >> 4, one copy
// per lane (word v * 32 + lane: never a bank conflict), so a record costs 64 look-ups instead of 128.  Levels and query are
// bf16 and go into the fp32 multiply-adds as they are (fma.rn.f32.bf16: the exact product, one rounding), every subspace with
// its own chain over j, then acc = fma(dot, w_b, acc) over b ascending, so the result has the bits of rerank_one.
// c128 = 128 comes from a kernel argument, because a multiplication by a known power of two becomes a shift on the integer ALU
// (half rate).  What bounds it: shared-memory wavefronts, 64 for the look-ups, 32 for the query, 24 for the record, some 30
// for the fetch of the next.
// Four lanes per candidate (whole sectors per load, the query in registers) measured 15 % slower: passing the sum from
// lane to lane costs more instructions than the query's shared-memory reads.
constexpr int LEV2_BYTES = 256 * 32 * 4;

__device__ __forceinline__ void build_lev2(uint32_t* lev2, const uint16_t* centers, int tid, int nthreads) {
  for (int v = tid >> 5; v < 256; v += nthreads >> 5) {   // (tid < 0: a warp that leaves it to the others)
    if (tid < 0) break;
    const uint32_t a = centers[v & 7], b = centers[(v >> 4) & 7];
    lev2[v * 32 + (tid & 31)] = ((v & 8) ? a : a ^ 0x8000u) | (((v & 0x80) ? b : b ^ 0x8000u) << 16);
  }
}
__device__ __forceinline__ float rerank_record(const uint4 (&rec)[6], const uint32_t* lev2, const uint4* q, float qn, int lane, unsigned c128) {
  const uint32_t code[16] = {rec[0].x, rec[0].y, rec[0].z, rec[0].w, rec[1].x, rec[1].y, rec[1].z, rec[1].w,
                             rec[2].x, rec[2].y, rec[2].z, rec[2].w, rec[3].x, rec[3].y, rec[3].z, rec[3].w};
  const uint32_t wt[8] = {rec[4].x, rec[4].y, rec[4].z, rec[4].w, rec[5].x, rec[5].y, rec[5].z, rec[5].w};
  const uint8_t* base = reinterpret_cast<const uint8_t*>(lev2) + lane * 4;
  float acc = 0.0f;
#pragma unroll
  for (int s = 0; s < 16; s++) {
    const uint4 qs = q[s];   // the eight dimensions of the subspace
    const uint32_t qw[4] = {qs.x, qs.y, qs.z, qs.w};
    float dot = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++)
      dot = fma_bf16x2(*reinterpret_cast<const uint32_t*>(base + byte_of(code[s], i) * c128), qw[i], dot);
    acc = __fmaf_rn(dot, __uint_as_float((s & 1) ? (wt[s >> 1] & 0xffff0000u) : (wt[s >> 1] << 16)), acc);
  }
  return __fmul_rn(acc, qn);
}

// ---- stages that the one-launch chain and its several-launch form share; blocks of CH_THREADS threads ------------------
constexpr int CH_THREADS = 512;
constexpr int CH_WARPS = CH_THREADS / 32;
constexpr int CH_CBINS = 129;                      // counts 0 .. 16 subspaces x 8 tiers
constexpr int CH_HIST_BYTES = CH_CBINS * 32 * 4;   // count histogram, one replica per lane: a warp's atomics never conflict
// A warp's 32 staged records: 96 bytes each, 16 more after every fourth.  Record r starts at unit 6 r + r / 4 of 16 bytes, so
// the eight lanes of a quarter-warp read fall into eight different groups of four banks.
constexpr int CH_STAGE_WARP = 16 * (6 * 32 + 8);
constexpr int CH_STAGE = CH_WARPS * CH_STAGE_WARP;

struct PreparedQuery {
  float x[4], avg[4], n;   // warp 0: the lane's dimensions of the rotated and of the mean query, the norm
};
// What warp 0 reads for it, issued ahead of everything that waits: eight queries of the group, the signs.
struct QueryLoads {
  uint2 raw[8], signs;
};
__device__ __forceinline__ void load_queries(QueryLoads& ql, const ChainQuery& cq, int b, int h, int G, int g0) {
  const uint16_t* q = cq.queries + ((int64_t)b * cq.Hq + (int64_t)h * G) * 128 + 4 * (threadIdx.x & 31);
#pragma unroll
  for (int k = 0; k < 8; k++) ql.raw[k] = *reinterpret_cast<const uint2*>(q + min(g0 + k, G - 1) * 128);
}
__device__ __forceinline__ void load_query(QueryLoads& ql, const ChainQuery& cq, int b, int h, int G) {
  if (threadIdx.x >= 32) return;
  load_queries(ql, cq, b, h, G, 0);
  ql.signs = *reinterpret_cast<const uint2*>(cq.signs + 4 * threadIdx.x);
}
// Warp 0 averages the group's queries, normalises and rotates the mean into s_q.
__device__ __forceinline__ void prepare_query(PreparedQuery& pq, QueryLoads& ql, const ChainQuery& cq, int b, int h, int G,
                                              float inv_g, float* s_q, float* s_qnorm) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x >= 32) return;
  float sg[4], acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  unpack4(ql.signs, sg);
  for (int g0 = 0; g0 < G; g0 += 8) {  // fp32 sum over the group, g ascending
    if (g0) load_queries(ql, cq, b, h, G, g0);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      if (g0 + k >= G) break;
      float v[4];
      unpack4(ql.raw[k], v);
#pragma unroll
      for (int i = 0; i < 4; i++) acc[i] = __fadd_rn(acc[i], v[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) pq.x[i] = pq.avg[i] = bfround(__fmul_rn(acc[i], inv_g));
  pq.n = rotate4(pq.x, sg, lane);
#pragma unroll
  for (int i = 0; i < 4; i++) s_q[4 * lane + i] = pq.x[i];
  if (lane == 0) *s_qnorm = pq.n;
}
__device__ __forceinline__ void publish_query(const PreparedQuery& pq, const ChainQuery& cq, int64_t bh) {   // warp 0 of one block
  const int lane = threadIdx.x & 31;
  auto words = [](const float* v) {
    return make_uint2((uint32_t)f2bf(v[0]) | ((uint32_t)f2bf(v[1]) << 16), (uint32_t)f2bf(v[2]) | ((uint32_t)f2bf(v[3]) << 16));
  };
  if (cq.query_avg) *reinterpret_cast<uint2*>(cq.query_avg + bh * 128 + 4 * lane) = words(pq.avg);
  if (cq.q_blocks) *reinterpret_cast<uint2*>(cq.q_blocks + bh * 128 + 4 * lane) = words(pq.x);
  if (cq.q_norm && lane == 0) cq.q_norm[bh] = f2bf(pq.n);
}
__device__ __forceinline__ void load_tiers(const ChainQuery& cq, long long N, unsigned* s_tiers, int t) {   // threads t = 0 .. 8
  const int n = cq.n_dev ? cq.sched.n_tiers : cq.n_tiers;
  if (t < n) s_tiers[t] = cq.n_dev ? zone_tier(cq.sched, N, t) : cq.tiers[t];
  if (t == 8) s_tiers[8] = (unsigned)n;
}
// Tier table of one subspace by a warp: the lane's four of the 128 bytes (see tier_sum16).  sizes: 256 words with the cluster
// sizes (overwritten); key: the order made by rank_subspace.
__device__ __forceinline__ uint32_t tier_table(const unsigned (&key)[4], unsigned* sizes, const unsigned* s_tiers) {
  const int lane = threadIdx.x & 31;
  const int n_tiers = (int)s_tiers[8];
  unsigned tier[8], front[4], back[4], n_front = 0, n_back = 0;
#pragma unroll
  for (int t = 0; t < 8; t++) tier[t] = t < n_tiers ? s_tiers[t] : 0u;
#pragma unroll
  for (int r = 0; r < 4; r++) {   // sizes at positions e and 255 - e
    const unsigned id = key[r] & 255u;
    front[r] = sizes[255u - id], back[r] = sizes[id];
    n_front += front[r], n_back += back[r];
  }
  unsigned inc_f = n_front, inc_b = n_back;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned f = __shfl_up_sync(0xffffffffu, inc_f, off), g = __shfl_up_sync(0xffffffffu, inc_b, off);
    if (lane >= off) inc_f += f, inc_b += g;
  }
  // keys before position e, and up to position 255 - e
  unsigned before = inc_f - n_front;
  unsigned upto = __shfl_sync(0xffffffffu, inc_f, 31) + __shfl_sync(0xffffffffu, inc_b, 31) - (inc_b - n_back);
  __syncwarp();   // the sizes have been read: the same words take the tier counts, packed to nibbles below
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const unsigned id = key[r] & 255u;
    unsigned wf = 0, wb = 0;
    upto -= back[r];   // keys before position 255 - e
#pragma unroll
    for (int t = 0; t < 8; t++) wf += (before < tier[t]) ? 1u : 0u, wb += (upto < tier[t]) ? 1u : 0u;   // absent tiers are 0: never above a prefix sum
    sizes[255u - id] = wf, sizes[id] = wb;
    before += front[r];
  }
  __syncwarp();
  // entries i (low nibble) and i + 128 of byte i: four bytes per lane
  const uint4 e0 = *reinterpret_cast<const uint4*>(sizes + lane * 4), e1 = *reinterpret_cast<const uint4*>(sizes + 128 + lane * 4);
  return (e0.x | (e1.x << 4)) | ((e0.y | (e1.y << 4)) << 8) | ((e0.z | (e1.z << 4)) << 16) | ((e0.w | (e1.w << 4)) << 24);
}

// Ordered candidate list of a block's n_keys counts (cnt8, overwritten; the first `skip` < 16 are not keys): those above
// T, and ties at T while the zone-wide quota lasts, of which lower blocks have met eq_base.  put(position, offset of the
// key) for positions below `limit`; returns the length of the list.  warp_a / warp_b: CH_WARPS words of scratch.
template <class Put>
__device__ __forceinline__ int list_candidates(uint8_t* cnt8, int n_keys, int skip, unsigned T, unsigned quota,
                                               unsigned eq_base, int64_t limit, unsigned* warp_a, unsigned* warp_b, Put put) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wspan = ((n_keys + CH_WARPS - 1) / CH_WARPS + 15) / 16 * 16;
  const int k0 = min(n_keys, warp * wspan), k1 = min(n_keys, k0 + wspan);
  // the top bit of every byte: count above / not below T (T <= 128, counts <= 128: no carry between bytes)
  const uint32_t add_gt = T < 128u ? (127u - T) * 0x01010101u : 0u, keep_gt = T < 128u ? 0x80808080u : 0u;
  const uint32_t add_ge = T ? (128u - T) * 0x01010101u : 0u, all_ge = T ? 0u : 0x80808080u;
  // the top bits of 16 bytes, in order: dot products place eight of them side by side, 128 times as large
  auto gather = [](uint32_t a, uint32_t b, uint32_t c, uint32_t d) -> unsigned {
    return (__dp4a(b, 0x80402010u, __dp4a(a, 0x08040201u, 0u)) >> 7) | (__dp4a(d, 0x80402010u, __dp4a(c, 0x08040201u, 0u)) << 1);
  };
  unsigned n_gt = 0, n_eq = 0;
#pragma unroll 1
  for (int k = k0 + 16 * lane; k < k1; k += 512) {   // 16 keys -> masks of counts above / at the threshold, kept in their place
    const uint4 v = *reinterpret_cast<const uint4*>(cnt8 + k);
    auto above = [&](uint32_t w) -> uint32_t { return (w + add_gt) & keep_gt; };
    auto not_below = [&](uint32_t w) -> uint32_t { return ((w + add_ge) | all_ge) & 0x80808080u; };
    unsigned gt = gather(above(v.x), above(v.y), above(v.z), above(v.w));
    unsigned eq = gather(not_below(v.x), not_below(v.y), not_below(v.z), not_below(v.w)) & ~gt;
    if (k1 - k < 16) gt &= (1u << (k1 - k)) - 1u, eq &= (1u << (k1 - k)) - 1u;
    if (k < skip) gt &= ~0u << skip, eq &= ~0u << skip;
    *reinterpret_cast<unsigned*>(cnt8 + k) = gt | (eq << 16);
    n_gt += __popc(gt), n_eq += __popc(eq);
  }
  n_gt = __reduce_add_sync(0xffffffffu, n_gt), n_eq = __reduce_add_sync(0xffffffffu, n_eq);
  if (lane == 0) warp_a[warp] = n_gt, warp_b[warp] = n_eq;
  __syncthreads();
  unsigned g = 0, e = eq_base, g_all = 0, e_all = eq_base;
#pragma unroll
  for (int w = 0; w < CH_WARPS; w++) {
    const unsigned a = warp_a[w], c = warp_b[w];
    if (w < warp) g += a, e += c;
    g_all += a, e_all += c;
  }
  const unsigned eq_before = min(eq_base, quota);
  int n_list = (int)(g_all + min(e_all, quota) - eq_before);
  n_list = (int)max((int64_t)0, min((int64_t)n_list, limit));   // a no-op with consistent histograms
#pragma unroll 1
  for (int k = k0; k < k1; k += 512) {
    const unsigned m = k + 16 * lane < k1 ? *reinterpret_cast<const unsigned*>(cnt8 + k + 16 * lane) : 0u;
    const unsigned gt = m & 0xffffu, eq = m >> 16;
    const unsigned mine = ((unsigned)__popc(gt) << 16) | (unsigned)__popc(eq);
    unsigned inc = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned o = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += o;
    }
    const unsigned total = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned eg = g + ((inc - mine) >> 16), ee = e + ((inc - mine) & 0xffffu);
    const int room = (int)quota - (int)ee;   // ties this lane may still take
    unsigned take = eq;
    if (room < (int)__popc(eq))
      for (int drop = (int)__popc(eq) - max(room, 0); drop > 0; drop--) take &= ~(1u << (31 - __clz(take)));
    take |= gt;
    int pos = (int)(eg + min(ee, quota) - eq_before);
    while (take) {
      const int j = __ffs(take) - 1;
      take &= take - 1;
      if (pos < n_list) put(pos, k + 16 * lane + j);
      pos++;
    }
    g += total >> 16, e += total & 0xffffu;
  }
  return n_list;
}

// 4-bit rerank of a list by one block, from key-major records: key_at(i) -> sink(i, key, score).  ids: the keys of the first
// n_ids candidates in shared memory (all of them, or a multiple of 32); q: the rotated query, 128 bf16 in shared memory;
// after_round(): called by whole warps behind each of their rounds.
// A warp takes 32 consecutive candidates per round.  The records of its next round are on their way to its staging buffer by
// cp.async while it works on this one, which it has read into registers, one record per lane: 24 lanes fetch four records per
// instruction, six 16-byte pieces each.
// What bounds it: the wavefronts of rerank_record, 162 a round and SM, and HBM in units of 128 bytes (the records of a
// candidate in two arrays are two).  128 blocks with 6000 candidates each on B200: 54 us with the records through registers
// and packed fp32 products (264 wavefronts, 593 instructions a round), 33 like this (493 instructions).  16 sequences of
// 16 - 32K keys 232.6 -> 219.5 us a step of two layers, adaptive budgets of 8 sequences 155.1 -> 147.1, 1M keys 135.0 -> 132.1.
// A second buffer per warp, two candidates per lane and the TMA's four-row gather were no faster.
template <class KeyAt, class Sink, class AfterRound>
__device__ __forceinline__ void rerank_list(int n_list, const int* ids, int n_ids, const RerankArgs& a, const uint8_t* k4, const uint16_t* w,
                                            uint8_t* stage, const uint32_t* lev2, const uint4* q, float qn, unsigned c128, KeyAt key_at,
                                            Sink sink, AfterRound after_round) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int ROUND = CH_WARPS * 32;
  const int sub = (lane * 43) >> 8, piece = lane - 6 * sub;   // lane / 6 and the rest
  const uint8_t* src = piece < 4 ? k4 + 16 * piece : reinterpret_cast<const uint8_t*>(w) + 16 * (piece - 4);
  const unsigned step = (unsigned)(piece < 4 ? a.k4_l : 2 * a.w_l);   // bytes from key to key
  const unsigned dst = (unsigned)__cvta_generic_to_shared(stage) + 16 * lane;
  const int n_whole = min(n_list, n_ids);
  auto copy = [&](int i, int key) {   // records 4 i .. 4 i + 3 of the round
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 400 * i), "l"(src + (uint64_t)(unsigned)key * step) : "memory");
  };
  auto fetch = [&](int base) {
    if (base < n_list && lane < 24) {
      if (base + 32 <= n_whole) {
#pragma unroll
        for (int i = 0; i < 8; i++) copy(i, ids[base + 4 * i + sub]);
      } else {   // past the end: the list's last candidate again
#pragma unroll 1
        for (int i = 0; i < 8; i++) copy(i, key_at(min(base + 4 * i + sub, n_list - 1)));
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(warp * 32);
#pragma unroll 1
  for (int base = warp * 32; base < n_list; base += ROUND) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    uint4 rec[6];
#pragma unroll
    for (int i = 0; i < 6; i++) rec[i] = *reinterpret_cast<const uint4*>(stage + (6 * lane + (lane >> 2) + i) * 16);
    __syncwarp();
    fetch(base + ROUND);
    const float v = rerank_record(rec, lev2, q, qn, lane, c128);
    const int i = base + lane;
    if (i < n_list) sink(i, key_at(i), v);
    __syncwarp();
    after_round();
  }
}

}  // namespace
}  // namespace pk
