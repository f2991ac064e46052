// Key coding (SRHT normalise-rotate, sign code, 4-bit code, rerank weight; keycode.cuh), prompt ingestion, cluster
// histograms, query preparation and the append of a decode token.  One key is coded by 4 lanes, 32 dimensions (four
// 8-dim subspaces) per lane.  Every fp32 operation rounds to nearest in a fixed order, so results do not depend on the
// mapping.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <atomic>

#include "common.cuh"
#include "keycode.cuh"
#include "rotate.cuh"

namespace pk {
namespace {

struct EncodeParams {
  const uint16_t* keys;
  int64_t k_b, k_h, k_l;
  const uint16_t* signs;
  uint8_t* codes;
  int64_t c_b, c_h, c_s, c_l;
  uint16_t* w;
  int64_t w_b, w_h, w_s, w_l;
  uint8_t* pk;
  int64_t p_b, p_h, p_s, p_l;
  int32_t* counts;
  int H;
  int64_t L, chunk;
};

constexpr int EN_THREADS = 256;
constexpr int EN_KEYS = EN_THREADS / 4;   // keys per block and round

__device__ __forceinline__ void load_key32(uint4 (&raw)[4], const uint16_t* row, int s) {
#pragma unroll
  for (int i = 0; i < 4; i++) raw[i] = reinterpret_cast<const uint4*>(row + 32 * s)[i];
}

// KEY_MAJOR: records stored key by key (contiguous over subspaces), so a lane's share of a record is one store; otherwise
// any strides.
template <bool KEY_MAJOR>
__global__ void __launch_bounds__(EN_THREADS, 2) encode_kernel(EncodeParams p) {
  __shared__ int hist[16 * 256];
  const int tid = threadIdx.x, s = tid & 3, grp = tid >> 2;
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
  if (p.counts) {
    for (int i = tid; i < 16 * 256; i += EN_THREADS) hist[i] = 0;
    __syncthreads();
  }
  const RotateLane rl(s);
  uint4 mask[4];
  load_key32(mask, p.signs, s);
#pragma unroll
  for (int i = 0; i < 4; i++) mask[i] = sign_mask(mask[i]);
  const int64_t begin = (int64_t)blockIdx.y * p.chunk;
  const int64_t end = min(p.L, begin + p.chunk);
  const uint16_t* kbase = p.keys + b * p.k_b + h * p.k_h;
  uint4 raw[4], nxt[4];
  load_key32(raw, kbase + min(begin + grp, end - 1) * p.k_l, s);
#pragma unroll
  for (int i = 0; i < 4; i++) raw[i] = flip(raw[i], mask[i]);
  for (int64_t k0 = begin; k0 < end; k0 += EN_KEYS) {  // uniform per block: shuffles need whole warps
    const int64_t key = k0 + grp;
    load_key32(nxt, kbase + min(key + EN_KEYS, end - 1) * p.k_l, s);   // in flight during the arithmetic
    const KeyCode kc = code_key<1>(raw, rl);
#pragma unroll
    for (int i = 0; i < 4; i++) raw[i] = flip(nxt[i], mask[i]);   // (behind the coding: 8 heads x 131072 keys 221.1 -> 208.7 us on B200)
    if (key >= end) continue;
    if (KEY_MAJOR) {
      *reinterpret_cast<uint32_t*>(p.codes + b * p.c_b + h * p.c_h + key * 16 + 4 * s) = kc.codes;
      *reinterpret_cast<uint2*>(p.w + b * p.w_b + h * p.w_h + key * p.w_l + 4 * s) = kc.weights;
      *reinterpret_cast<uint4*>(p.pk + b * p.p_b + h * p.p_h + key * p.p_l + 16 * s) = kc.packed;
    } else {
      const uint32_t pk4[4] = {kc.packed.x, kc.packed.y, kc.packed.z, kc.packed.w};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int sub = 4 * s + i;
        const uint32_t wt = i < 2 ? kc.weights.x : kc.weights.y;
        p.codes[b * p.c_b + h * p.c_h + sub * p.c_s + key * p.c_l] = (uint8_t)(kc.codes >> (8 * i));
        p.w[b * p.w_b + h * p.w_h + sub * p.w_s + key * p.w_l] = (uint16_t)((i & 1) ? wt >> 16 : wt);
        uint8_t* pp = p.pk + b * p.p_b + h * p.p_h + sub * p.p_s + key * p.p_l;
        if ((reinterpret_cast<uintptr_t>(pp) & 3) == 0) {
          *reinterpret_cast<uint32_t*>(pp) = pk4[i];
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) pp[j] = (uint8_t)(pk4[i] >> (8 * j));
        }
      }
    }
    if (p.counts)
#pragma unroll
      for (int i = 0; i < 4; i++) atomicAdd(&hist[(4 * s + i) * 256 + ((kc.codes >> (8 * i)) & 0xffu)], 1);
  }
  if (p.counts) {
    __syncthreads();
    int32_t* dst = p.counts + (int64_t)bh * 16 * 256;
    for (int i = tid; i < 16 * 256; i += EN_THREADS)
      if (hist[i]) atomicAdd(dst + i, hist[i]);
  }
}

// ---- a prompt into the cache, one launch per sample ---------------------------------------------------------------
// Token t of the prompt is a window row (the first `sink` tokens and the last `local` ones; all of them where the prompt
// is not longer than both together) or zone row t - sink.  Every row is read once: its K and V go to the window or to the
// store (K row and V row of a key next to each other), its key is coded into the staging arrays or the zone records, ||v||
// and the cluster histogram come with it.  A head's tokens are cut into tiles of 96, the zone rows first and the window
// rows behind them; a block takes consecutive tiles, the heads of a token range side by side in the grid, since they are
// neighbours in memory (prefill_kernel; short prompts, and those that cannot be described to the TMA unit: prefill_rows_kernel).
// Tiles of zone rows come by TMA into one of two stages of shared memory and go to the store from there, K and V, four
// instructions of one thread each way; the warps only read the keys, lane l of a warp 32 dimensions (quarter l / 8) of its key
// l % 8, so that with the copies' 128-byte swizzle the eight lanes of a quarter-warp read fall into eight different groups of
// four banks.  Window rows are loaded and stored row by row.
// What bounds it: issue slots of the coding, 70 - 75 % of them taken (integer ALU 60 %, DRAM 67 - 80 %), with 24 warps per SM.
// 131072 tokens x 8 heads on B200: 2003 us as coding, interleaving and copy launches; 262 as one launch that carries the rows
// through registers, 16 warps per SM (prefill_rows_kernel); 211 as this one: 5.6 TB/s of 1136 bytes per key.  A block's tiles are an even
// share of one wave: two waves of half the size take 229.  (Single rows by bulk copies took 450: the copy engine takes a row
// per instruction no faster than a tile.)
struct PrefillMaps {
  CUtensorMap k, v;         // [P][H][128] by 64 dimensions x 1 head x 96 tokens
  CUtensorMap store;        // [H][N][256] by 64 x 96 rows x 1 head
  int heads_inner;          // the heads are the middle dimension of k and v, not the outer one
};
struct PrefillParams {
  const uint16_t* k;        // [P][H][128] of one sample
  const uint16_t* v;
  int64_t k_l, k_h, v_l, v_h;
  const uint16_t* signs;
  uint16_t* wk;             // window rows of the sample: head h at h * w_h, rows 128 apart
  uint16_t* wv;
  int64_t w_h;
  uint8_t* win_codes;       // staging records of the sample: [H][cap_w][16], [H][cap_w][16], [H][cap_w][64], [H][cap_w]
  uint16_t* win_w;
  uint8_t* win_pk;
  float* win_vnorm;
  uint8_t* z_codes;         // zone records of the sample: [H][cap_z][16], [H][cap_z][16 of z_wl], [H][cap_z][64 of z_pl], [H][cap_z] or null
  uint16_t* z_w;
  uint8_t* z_pk;
  float* z_vnorm;
  int64_t z_wl, z_pl;       // weights (elements) and 4-bit codes (bytes) from one key to the next
  int32_t* counts;          // [H][16][256], zero at launch
  uint16_t* store;          // [H][store_cap][2][128]
  int32_t* state;           // the layer's words
  int64_t P, N, cap_z, store_cap;
  int64_t zone_tiles, n_tiles, tiles_per_block;   // prefill_kernel: tiles of a head, those of zone rows and all
  int64_t chunk;                                  // prefill_rows_kernel: tokens of a block
  int H, cap_w, sink, n_window, b;
};

constexpr int PF_THREADS = 384, PF_WARPS = PF_THREADS / 32;
constexpr int PF_TILE = 8 * PF_WARPS;             // tokens
constexpr int PF_HALF = PF_TILE * 128;            // bytes of 64 dimensions of a tile's K or V rows
constexpr int PF_STAGE = 4 * PF_HALF;             // K, V; two halves each
constexpr int PF_HIST = 16 * 256 * 4;
constexpr int PF_SMEM = 2 * PF_STAGE + PF_HIST + 256 + 32;
constexpr int PF_WAIT_LIMIT = 4000000;            // polls of a barrier before giving up

// Ahead of a prompt: its histogram, and with a layer's first sample the error word that all samples share.  A launch of its own,
// so that the word is clear before any block may set it; with a later sample it would take the report of an earlier one away.
// In the place of a memset of the histogram, and 0.15 us faster; it costs the host 0.6 us more, so that prefill_rows_kernel, which
// reports nothing, clears the word itself behind a memset.
__global__ void __launch_bounds__(1024) prefill_clear_kernel(int32_t* counts, int32_t* error) {
  counts[(int64_t)blockIdx.x * 1024 + threadIdx.x] = 0;
  if (error && blockIdx.x == 0 && threadIdx.x == 0) *error = 0;
}

__device__ __forceinline__ bool pf_wait(unsigned mbar, unsigned parity) {
  unsigned done = 0;
  for (int it = 0; it < PF_WAIT_LIMIT && !done; it++)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
  return done != 0;
}

__global__ void __launch_bounds__(PF_THREADS, 2) prefill_kernel(const __grid_constant__ PrefillParams p, const __grid_constant__ PrefillMaps m) {
  extern __shared__ __align__(1024) unsigned char pf_smem[];   // (no static shared memory: the stages start on 1024 bytes)
  int* hist = reinterpret_cast<int*>(pf_smem + 2 * PF_STAGE);
  uint32_t* masks = reinterpret_cast<uint32_t*>(pf_smem + 2 * PF_STAGE + PF_HIST);
  const unsigned smem0 = (unsigned)__cvta_generic_to_shared(pf_smem);
  const unsigned full0 = smem0 + 2 * PF_STAGE + PF_HIST + 256, empty0 = full0 + 16;   // one barrier per stage: filled, read by all warps
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, s = lane >> 3;
  const int h = blockIdx.x;
  const int64_t first = (int64_t)blockIdx.y * p.tiles_per_block;
  const int n = (int)min(p.tiles_per_block, p.n_tiles - first);                       // tiles of this block
  const int n_tma = (int)min((int64_t)n, max((int64_t)0, p.zone_tiles - first));      // the leading ones come by TMA
  if (tid == 0)
#pragma unroll
    for (int i = 0; i < 2; i++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n\tmbarrier.init.shared::cta.b64 [%1], %2;" ::"r"(full0 + 8 * i), "r"(empty0 + 8 * i),
                   "r"(PF_WARPS)
                   : "memory");
  if (tid == 0) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  for (int i = tid; i < 16 * 256; i += PF_THREADS) hist[i] = 0;
  if (tid < 64) masks[tid] = reinterpret_cast<const uint32_t*>(p.signs)[tid] & 0x80008000u;
  if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) {
    p.state[0] = p.n_window, p.state[1] = 0, p.state[2] = 0;   // (state[3]: see prefill_clear_kernel)
    p.state[4 + p.b] = (int32_t)p.N;
  }
  __syncthreads();
  auto load_tile = [&](int j) {   // (thread 0)
    const unsigned dst = smem0 + (j & 1) * PF_STAGE, bar = full0 + 8 * (j & 1);
    const int t = (int)(p.sink + (first + j) * PF_TILE), c1 = m.heads_inner ? h : t, c2 = m.heads_inner ? t : h;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(PF_STAGE) : "memory");
#pragma unroll
    for (int i = 0; i < 4; i++)
      asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                       dst + i * PF_HALF),
                   "l"(i < 2 ? &m.k : &m.v), "r"((i & 1) * 64), "r"(c1), "r"(c2), "r"(bar)
                   : "memory");
  };
  auto store_tile = [&](int j) {   // (thread 0)
    const unsigned src = smem0 + (j & 1) * PF_STAGE;
    const int z = (int)((first + j) * PF_TILE);
#pragma unroll
    for (int i = 0; i < 4; i++)
      asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(&m.store), "r"(i * 64), "r"(z),
                   "r"(h), "r"(src + i * PF_HALF)
                   : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  };
  if (tid == 0) {
    if (n_tma > 0) load_tile(0);
    if (n_tma > 1) load_tile(1);
  }
  const RotateLane rl(s);
  const uint16_t* kb = p.k + h * p.k_h;
  const uint16_t* vb = p.v + h * p.v_h;
  bool lost = false;
#pragma unroll 1
  for (int j = 0; j < n; j++) {
    const int row = warp * 8 + (lane & 7);   // the lane's key in the tile
    const unsigned stage = smem0 + (j & 1) * PF_STAGE;
    uint4 key[4];
    int64_t t;       // the lane's token; P: none
    if (j < n_tma) {
      lost = __any_sync(0xffffffffu, lost || !pf_wait(full0 + 8 * (j & 1), (unsigned)(j >> 1) & 1u));
      if (lost) {    // a copy that never landed: reported, and once more waited for, since it writes into this block's memory
        if (lane == 0) atomicExch(p.state + 3, 1);
        for (int i = j; i < min(n_tma, j + 2); i++) pf_wait(full0 + 8 * (i & 1), (unsigned)(i >> 1) & 1u);
        break;
      }
      if (tid == 0) store_tile(j);
      t = p.sink + (first + j) * PF_TILE + row;
      if (t >= p.sink + p.N) t = p.P;
      const unsigned at = stage + (s >> 1) * PF_HALF + row * 128;
#pragma unroll
      for (int i = 0; i < 4; i++)
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(key[i].x), "=r"(key[i].y), "=r"(key[i].z), "=r"(key[i].w)
                     : "r"(at + ((((s & 1) * 4 + i) ^ (lane & 7)) << 4)));
    } else {
      const int64_t q = (first + j - p.zone_tiles) * PF_TILE + row;   // window row
      t = q < p.n_window ? (q >= p.sink ? q + p.N : q) : p.P;
#pragma unroll
      for (int i = 0; i < 4; i++) key[i] = reinterpret_cast<const uint4*>(kb + min(t, p.P - 1) * p.k_l + 32 * s)[i];
    }
    const int64_t z = t - p.sink;   // zone row, if 0 <= z < N; window row t or t - N otherwise
    const bool zone = z >= 0 && z < p.N;
    const int64_t wrow = z < p.N ? t : t - p.N;
    if (j >= n_tma && t < p.P) {
      uint4* dst = reinterpret_cast<uint4*>(p.wk + h * p.w_h + wrow * 128) + 4 * s;
#pragma unroll
      for (int i = 0; i < 4; i++) dst[i] = key[i];
    }
    // V: a half warp takes a row (16 bytes per lane), a warp the rows 2i, 2i + 1 of its eight in step i; those that TMA copies
    // are looked at for their norms only
    if (j >= n_tma || p.z_vnorm) {
#pragma unroll 1
      for (int i = 0; i < 4; i++) {
        const int64_t tv = __shfl_sync(0xffffffffu, t, 2 * i + (lane >> 4)), zv = tv - p.sink;
        const int64_t wv = zv < p.N ? tv : tv - p.N;
        const bool in_zone = zv >= 0 && zv < p.N;
        const int l = lane & 15;
        uint4 raw;
        if (j < n_tma) {
          const int r = warp * 8 + 2 * i + (lane >> 4);
          const unsigned at = stage + (2 + (l >> 3)) * PF_HALF + r * 128 + (((l & 7) ^ (r & 7)) << 4);
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(raw.x), "=r"(raw.y), "=r"(raw.z), "=r"(raw.w) : "r"(at));
        } else {
          raw = reinterpret_cast<const uint4*>(vb + min(tv, p.P - 1) * p.v_l)[l];
          if (tv < p.P) reinterpret_cast<uint4*>(p.wv + h * p.w_h + wv * 128)[l] = raw;
        }
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
        float a = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; k++) a = fmaf(lo_f(w[k]), lo_f(w[k]), fmaf(hi_f(w[k]), hi_f(w[k]), a));
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        if (tv < p.P && l == 0) {
          if (!in_zone) p.win_vnorm[(int64_t)h * p.cap_w + wv] = sqrtf(a);
          else if (p.z_vnorm) p.z_vnorm[(int64_t)h * p.cap_z + zv] = sqrtf(a);
        }
      }
    }
    if (j < n_tma) {
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty0 + 8 * (j & 1)) : "memory");
    }
#pragma unroll
    for (int i = 0; i < 4; i++) key[i] = flip(key[i], reinterpret_cast<const uint4*>(masks)[4 * s + i]);
    const KeyCode kc = code_key<8>(key, rl);
    if (t < p.P) {
      const int64_t rec = zone ? (int64_t)h * p.cap_z + z : (int64_t)h * p.cap_w + wrow;
      *reinterpret_cast<uint32_t*>((zone ? p.z_codes : p.win_codes) + rec * 16 + 4 * s) = kc.codes;
      *reinterpret_cast<uint2*>((zone ? p.z_w + rec * p.z_wl : p.win_w + rec * 16) + 4 * s) = kc.weights;
      *reinterpret_cast<uint4*>((zone ? p.z_pk + rec * p.z_pl : p.win_pk + rec * 64) + 16 * s) = kc.packed;
      if (zone)
#pragma unroll
        for (int i = 0; i < 4; i++) atomicAdd(&hist[(4 * s + i) * 256 + ((kc.codes >> (8 * i)) & 0xffu)], 1);
    }
    if (tid == 0 && j + 2 < n_tma) {   // the stage goes to tile j + 2 once all warps have read it and the stores have
      lost = !pf_wait(empty0 + 8 * (j & 1), (unsigned)(j >> 1) & 1u);
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      if (!lost) load_tile(j + 2);
    }
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncthreads();
  int32_t* dst = p.counts + (int64_t)h * 16 * 256;
  for (int i = tid; i < 16 * 256; i += PF_THREADS)
    if (hist[i]) atomicAdd(dst + i, hist[i]);
}

// The same row by row: the heads of a token range side by side in the grid, block (h, chunk) a head's consecutive tokens, the next
// round's rows in flight in registers while a round is coded.  Short prompts, which the setup of the other form takes longer than,
// and whatever cannot be described to the TMA unit (K and V in different orders of tokens and heads, heads that share their rows).
// What bounds it: issue slots of the coding, with 16 warps per SM.  B200, us, this form | prefill_kernel with all rows loaded where
// they are used, no round in flight: 300 tokens x 8 heads 7.8 | 10.4, 2000 x 8 11.5 | 16.7, 131072 x 8 with K and V in different
// orders 261 | 359.
__global__ void __launch_bounds__(EN_THREADS, 2) prefill_rows_kernel(PrefillParams p) {
  __shared__ int hist[16 * 256];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, s = tid & 3, grp = tid >> 2;
  const int h = blockIdx.x;
  for (int i = tid; i < 16 * 256; i += EN_THREADS) hist[i] = 0;
  if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) {
    p.state[0] = p.n_window, p.state[1] = 0, p.state[2] = 0;
    if (p.b == 0) p.state[3] = 0;   // (a later sample's launch would take the report of an earlier one away)
    p.state[4 + p.b] = (int32_t)p.N;
  }
  __syncthreads();
  const RotateLane rl(s);
  uint4 mask[4];
  load_key32(mask, p.signs, s);
#pragma unroll
  for (int i = 0; i < 4; i++) mask[i] = sign_mask(mask[i]);
  const int64_t begin = (int64_t)blockIdx.y * p.chunk, end = min(p.P, begin + p.chunk);
  const uint16_t* kb = p.k + h * p.k_h;
  const uint16_t* vb = p.v + h * p.v_h;
  // V is only copied: a half warp takes a row (16 bytes per lane), a warp the rows 2i, 2i + 1 of its eight in step i
  uint4 kr[4], kn[4], vr[4];
  auto load_v = [&](int64_t t0) {
#pragma unroll
    for (int i = 0; i < 4; i++)
      vr[i] = reinterpret_cast<const uint4*>(vb + min(t0 + warp * 8 + 2 * i + (lane >> 4), end - 1) * p.v_l)[lane & 15];
  };
  load_key32(kr, kb + min(begin + grp, end - 1) * p.k_l, s);
  load_v(begin);
  for (int64_t t0 = begin; t0 < end; t0 += EN_KEYS) {
    load_key32(kn, kb + min(t0 + EN_KEYS + grp, end - 1) * p.k_l, s);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int64_t t = t0 + warp * 8 + 2 * i + (lane >> 4), z = t - p.sink;
      const bool zone = z >= 0 && z < p.N;
      if (!zone || p.z_vnorm) {   // uniform over the half warp of a row
        const uint32_t w[4] = {vr[i].x, vr[i].y, vr[i].z, vr[i].w};
        float a = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; j++) a = fmaf(lo_f(w[j]), lo_f(w[j]), fmaf(hi_f(w[j]), hi_f(w[j]), a));
        const unsigned half = 0xffffu << (lane & 16);
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) a += __shfl_xor_sync(half, a, off);
        if (t < end && (lane & 15) == 0) {
          if (zone) p.z_vnorm[(int64_t)h * p.cap_z + z] = sqrtf(a);
          else p.win_vnorm[(int64_t)h * p.cap_w + (z < p.N || p.N == 0 ? t : t - p.N)] = sqrtf(a);
        }
      }
      if (t < end) {
        if (zone) __stcs(reinterpret_cast<uint4*>(p.store + ((int64_t)h * p.store_cap + z) * 256 + 128) + (lane & 15), vr[i]);
        else reinterpret_cast<uint4*>(p.wv + h * p.w_h + (z < p.N || p.N == 0 ? t : t - p.N) * 128)[lane & 15] = vr[i];
      }
    }
    load_v(t0 + EN_KEYS);
    const int64_t t = t0 + grp, z = t - p.sink;   // zone row, if 0 <= z < N; window row t or t - N otherwise
    const bool zone = z >= 0 && z < p.N;
    const int64_t wrow = z < p.N || p.N == 0 ? t : t - p.N;
    if (t < end) {
      uint4* dst = reinterpret_cast<uint4*>(zone ? p.store + ((int64_t)h * p.store_cap + z) * 256 : p.wk + h * p.w_h + wrow * 128) + 4 * s;
#pragma unroll
      for (int i = 0; i < 4; i++) dst[i] = kr[i];
    }
#pragma unroll
    for (int i = 0; i < 4; i++) kr[i] = flip(kr[i], mask[i]);
    const KeyCode kc = code_key<1>(kr, rl);
    if (t < end) {
      if (zone) {
        const int64_t rec = (int64_t)h * p.cap_z + z;
        *reinterpret_cast<uint32_t*>(p.z_codes + rec * 16 + 4 * s) = kc.codes;
        *reinterpret_cast<uint2*>(p.z_w + rec * p.z_wl + 4 * s) = kc.weights;
        *reinterpret_cast<uint4*>(p.z_pk + rec * p.z_pl + 16 * s) = kc.packed;
#pragma unroll
        for (int i = 0; i < 4; i++) atomicAdd(&hist[(4 * s + i) * 256 + ((kc.codes >> (8 * i)) & 0xffu)], 1);
      } else {
        const int64_t rec = (int64_t)h * p.cap_w + wrow;
        *reinterpret_cast<uint32_t*>(p.win_codes + rec * 16 + 4 * s) = kc.codes;
        *reinterpret_cast<uint2*>(p.win_w + rec * 16 + 4 * s) = kc.weights;
        *reinterpret_cast<uint4*>(p.win_pk + rec * 64 + 16 * s) = kc.packed;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) kr[i] = kn[i];
  }
  __syncthreads();
  int32_t* dst = p.counts + (int64_t)h * 16 * 256;
  for (int i = tid; i < 16 * 256; i += EN_THREADS)
    if (hist[i]) atomicAdd(dst + i, hist[i]);
}

__global__ void __launch_bounds__(256) count_kernel(const uint8_t* codes, int64_t c_b, int64_t c_h,
                                                    int64_t c_s, int64_t c_l, int H, int B, int64_t N,
                                                    int64_t chunk, int32_t* counts) {
  extern __shared__ int hist[];
  const int tid = threadIdx.x;
  const int bh = blockIdx.y, b = bh / H, h = bh % H;
  for (int i = tid; i < B * 256; i += 256) hist[i] = 0;
  __syncthreads();
  const int64_t begin = (int64_t)blockIdx.x * chunk, end = min(N, begin + chunk);
  const uint8_t* base = codes + b * c_b + h * c_h;
  for (int64_t k = begin + tid; k < end; k += 256)
    for (int s = 0; s < B; s++) atomicAdd(&hist[s * 256 + base[s * c_s + k * c_l]], 1);
  __syncthreads();
  int32_t* dst = counts + (int64_t)bh * B * 256;
  for (int i = tid; i < B * 256; i += 256)
    if (hist[i]) atomicAdd(dst + i, hist[i]);
}

// One warp per (batch, KV head), four dims per lane.  What bounds it is the latency of its loads: those of eight queries go
// out together (16 serial sums in 8 lanes before: 5.6 us for 8 heads of 4 queries on B200, 2.6 now).
__global__ void __launch_bounds__(32) query_prep_kernel(const uint16_t* queries, int Hq, int H, int G, float inv_g,
                                                        const uint16_t* signs, uint16_t* q_blocks,
                                                        uint16_t* q_norm, uint16_t* query_avg) {
  const int lane = threadIdx.x;
  const int bh = blockIdx.x, b = bh / H, h = bh % H;
  const uint16_t* q = queries + ((int64_t)b * Hq + (int64_t)h * G) * 128 + 4 * lane;
  pdl_wait();
  pdl_trigger();
  float x[4], sg[4], acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int i = 0; i < 4; i++) sg[i] = bf2f(signs[4 * lane + i]);
  for (int g0 = 0; g0 < G; g0 += 8) {   // fp32 sum over the group, g ascending
    uint16_t raw[8][4];
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
      for (int i = 0; i < 4; i++) raw[k][i] = q[min(g0 + k, G - 1) * 128 + i];
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (g0 + k < G) acc[i] = __fadd_rn(acc[i], bf2f(raw[k][i]));
  }
  auto store = [&](uint16_t* out) {
#pragma unroll
    for (int i = 0; i < 4; i++) out[(int64_t)bh * 128 + 4 * lane + i] = f2bf(x[i]);
  };
#pragma unroll
  for (int i = 0; i < 4; i++) x[i] = bfround(__fmul_rn(acc[i], inv_g));
  if (query_avg) store(query_avg);
  const float n = rotate4(x, sg, lane);
  store(q_blocks);
  if (lane == 0) q_norm[bh] = f2bf(n);
}

// ---- append one decode token: window row, key coding, and the flush of a full update buffer, one launch ----------
// Device-side state per layer (int32): [0] rows in the window, [1] arrival counter, [2] flushes done, [3] error flag,
// [4 + b] searchable keys of sample b.  One block per (batch, KV head):
//   * the K and V row go to window row `pos`, the key is coded (the arithmetic of encode_kernel) and its codes, the rerank
//     weights, the 4-bit codes and ||v|| go to the window-aligned staging arrays, so every key is coded exactly once, when
//     it arrives;
//   * if that row filled the window, the oldest `interval` rows behind the sink are PUBLISHED: their staged records
//     are copied to zone records [N, N + interval), their codes are added to the cluster histogram, their K/V rows go
//     to the store (device or pinned host memory), and the rest of the window slides down;
//   * the block that arrives last advances the state words.
// Everything a later kernel needs (window length, zone length) is read from the state words, so the launch arguments
// never change and one captured CUDA graph serves the whole generation, flushes included.
struct AppendParams {
  const uint16_t* k_row;
  const uint16_t* v_row;
  int64_t kr_b, kr_h, vr_b, vr_h;   // element strides of the [bs,1,H,128] rows
  const uint16_t* signs;
  uint16_t* wk;
  uint16_t* wv;
  int64_t w_b, w_h;                 // window strides (elements); rows are 128 apart
  uint8_t* win_codes;               // [bs*H][cap_w][16]
  uint16_t* win_w;                  // [bs*H][cap_w][16]
  uint8_t* win_pk;                  // [bs*H][cap_w][64]
  float* win_vnorm;                 // [bs*H][cap_w]
  uint8_t* z_codes;                 // [bs*H][cap_z][16]   key-major zone records
  uint16_t* z_w;                    // [bs*H][cap_z][16 of z_wl]
  uint8_t* z_pk;                    // [bs*H][cap_z][64 of z_pl]
  int64_t z_wl, z_pl;               // weights (elements) and 4-bit codes (bytes) from one key to the next
  float* z_vnorm;                   // [bs*H][cap_z] or null
  int32_t* counts;                  // [bs*H][16][256]
  uint16_t* store;                  // [bs*H][cap_s][2][128]
  int32_t* state;
  int H, cap_w, sink, interval;
  int64_t cap_z, cap_s;
};

// One key by a whole warp, four dimensions per lane: the same bits as code_key, which codes eight keys in the same time.  For
// a single key the latency counts, and that of fetching the instructions: a fifth of code_key's.
struct LaneCode {
  uint32_t packed;   // the lane's four 4-bit codes
  uint32_t code;     // even lanes: the sign code of subspace lane / 2
  uint16_t weight;   // even lanes: its rerank weight
};
__device__ __forceinline__ LaneCode code_key_warp(uint2 raw, uint2 signs, int lane) {
  float x[4] = {lo_f(raw.x), hi_f(raw.x), lo_f(raw.y), hi_f(raw.y)};
  const float sg[4] = {lo_f(signs.x), hi_f(signs.x), lo_f(signs.y), hi_f(signs.y)};
  const float n = rotate4(x, sg, lane);
  float t[4];
#pragma unroll
  for (int i = 0; i < 4; i++) x[i] = __fadd_rn(x[i], 0.0f), t[i] = __fmul_rn(x[i], x[i]);   // -0 counts as non-negative
  // adjacent pairwise tree over the eight dimensions of a subspace: two lanes
  auto tree = [&](const float (&v)[4]) -> float {
    const float s4 = __fadd_rn(__fadd_rn(v[0], v[1]), __fadd_rn(v[2], v[3]));
    return __fadd_rn(s4, __shfl_xor_sync(FULL, s4, 1));
  };
  const float r = bfround(__fsqrt_rn(tree(t)));
  const float ri = rcp_approx(fmaxf(r, bfround(1e-8f)));
  uint32_t nib[2], p[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {   // dimensions 2 k, 2 k + 1 of the lane
    const uint32_t au = bf16_2(__fmul_rn(x[2 * k], ri), __fmul_rn(x[2 * k + 1], ri)) & 0x7fff7fffu;
    const uint32_t l = level_b2(au) & 0x00070007u;
    p[k] = fma_b2(centre_b2(l), au, b2(0x8000));
    const uint32_t v = l | (~bf16_2(x[2 * k], x[2 * k + 1]) >> 12 & 0x00080008u);   // sign | level
    nib[k] = (v | (v >> 12)) & 0xffu;
  }
  const float pr[4] = {lo_f(p[0]), hi_f(p[0]), lo_f(p[1]), hi_f(p[1])};
  const float al = fmaxf(tree(pr), 1e-6f);
  LaneCode out;
  out.packed = nib[0] | (nib[1] << 8);
  uint32_t v = (out.packed >> 3) & 0x1111u;   // bit 3 of every nibble, gathered
  v = (v | (v >> 3)) & 0x0303u;
  v = (v | (v >> 6)) & 0xfu;
  out.code = v | (__shfl_xor_sync(FULL, v, 1) << 4);
  out.weight = f2bf(__fmul_rn(__fdiv_rn(r, al), n));
  return out;
}

// What bounds it is the latency of dependent steps: the state words and the rows (one round trip), the coding, the stores.
// Warp 0 codes the key, warp 1 copies the rows and takes ||v||.  The blocks arrive as soon as they have read the state words,
// while the key is coded, not behind their writes: the new words are for the kernels that wait for all of this one.  On B200,
// a step of four layers, against warp 0 doing everything with code_key and the arrival at the end: 10K keys in host memory
// 178.3 -> 168.9 us, 128K keys 221.9 -> 212.4, a KV head of eight sequences 214.5 -> 208.0; two layers with adaptive budgets
// of eight sequences 144.7 -> 136.0.
__global__ void __launch_bounds__(256) append_encode_kernel(AppendParams p) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t bh = blockIdx.x;
  const int b = (int)(bh / p.H), h = (int)(bh % p.H);
  pdl_wait();     // the rows to append and the state words come from the kernels before this one
  pdl_trigger();
  const int pos = p.state[0];
  const int64_t N = p.state[4 + b];
  uint16_t* wk = p.wk + b * p.w_b + h * p.w_h;
  uint16_t* wv = p.wv + b * p.w_b + h * p.w_h;
  uint8_t* wc = p.win_codes + bh * p.cap_w * 16;
  uint16_t* ww = p.win_w + bh * p.cap_w * 16;
  uint8_t* wp = p.win_pk + bh * p.cap_w * 64;
  float* wn = p.win_vnorm + bh * p.cap_w;
  const uint16_t* kr = p.k_row + b * p.kr_b + h * p.kr_h;
  const uint16_t* vr = p.v_row + b * p.vr_b + h * p.vr_h;
  uint2 key, sg;
  uint4 row;
  if (warp == 0) {
    key = reinterpret_cast<const uint2*>(kr)[lane], sg = reinterpret_cast<const uint2*>(p.signs)[lane];
  } else if (warp == 1) {   // lanes 0-15 carry K, lanes 16-31 carry V
    row = reinterpret_cast<const uint4*>(lane < 16 ? kr : vr)[lane & 15];
  }
  // every thread has its words when it passes (the vote uses them)
  const bool ok = __syncthreads_and(pos >= 0 && pos < p.cap_w && N >= 0) != 0;
  const int I = p.interval, sink = p.sink;
  const bool flush = ok && pos + 1 == p.cap_w;
  const bool room = N >= 0 && N + I <= p.cap_z && N + I <= p.cap_s;
  if (tid == 64) {   // the block that arrives last advances the state: every block has read it
    __threadfence();
    if (atomicAdd(reinterpret_cast<unsigned*>(p.state + 1), 1u) + 1u == gridDim.x) {
      if (!ok || (flush && !room)) {
        p.state[3] = 1;   // window overrun or zone full: the host checks this word
      } else if (flush) {
        p.state[0] = p.cap_w - I;
        p.state[2] += 1;
        const int bs = (int)(gridDim.x / p.H);
        for (int i = 0; i < bs; i++) p.state[4 + i] += I;
      } else {
        p.state[0] = pos + 1;
      }
      p.state[1] = 0;
    }
  }
  if (warp == 0) {
    const LaneCode kc = code_key_warp(key, sg, lane);
    if (ok) {
      reinterpret_cast<uint16_t*>(wp + (int64_t)pos * 64)[lane] = (uint16_t)kc.packed;
      if (!(lane & 1)) {
        wc[(int64_t)pos * 16 + (lane >> 1)] = (uint8_t)kc.code;
        ww[(int64_t)pos * 16 + (lane >> 1)] = kc.weight;
      }
    }
  } else if (warp == 1) {
    // ||v||: fp32, pairwise tree over adjacent dimensions
    float y[8];
    unpack8(row, y);
#pragma unroll
    for (int i = 0; i < 8; i++) y[i] = __fmul_rn(y[i], y[i]);
#pragma unroll
    for (int w = 8; w > 1; w >>= 1)
#pragma unroll
      for (int i = 0; i < w / 2; i++) y[i] = __fadd_rn(y[2 * i], y[2 * i + 1]);
    float vs = y[0];
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) vs = __fadd_rn(vs, __shfl_xor_sync(FULL, vs, off));
    if (ok) {
      reinterpret_cast<uint4*>((lane < 16 ? wk : wv) + (int64_t)pos * 128)[lane & 15] = row;
      if (lane == 16) wn[pos] = __fsqrt_rn(vs);
    }
  }
  if (flush && room) {
    __syncthreads();   // the new row and its records
    // publish rows [sink, sink + I): staged records -> zone records [N, N + I), K/V rows -> store, histogram
    const uint4* sc = reinterpret_cast<const uint4*>(wc + (int64_t)sink * 16);
    const uint4* sp = reinterpret_cast<const uint4*>(wp + (int64_t)sink * 64);
    const uint4* sw = reinterpret_cast<const uint4*>(ww + (int64_t)sink * 16);
    uint4* zc = reinterpret_cast<uint4*>(p.z_codes + (bh * p.cap_z + N) * 16);
    uint8_t* zp = p.z_pk + (bh * p.cap_z + N) * p.z_pl;
    uint16_t* zw = p.z_w + (bh * p.cap_z + N) * p.z_wl;
    for (int i = tid; i < I; i += 256) zc[i] = sc[i];
    for (int i = tid; i < 4 * I; i += 256) reinterpret_cast<uint4*>(zp + (i >> 2) * p.z_pl)[i & 3] = sp[i];
    for (int i = tid; i < 2 * I; i += 256) reinterpret_cast<uint4*>(zw + (i >> 1) * p.z_wl)[i & 1] = sw[i];
    if (p.z_vnorm)
      for (int i = tid; i < I; i += 256) p.z_vnorm[bh * p.cap_z + N + i] = wn[sink + i];
    uint4* st = reinterpret_cast<uint4*>(p.store + (bh * p.cap_s + N) * 256);
    const uint4* rk = reinterpret_cast<const uint4*>(wk + (int64_t)sink * 128);
    const uint4* rv = reinterpret_cast<const uint4*>(wv + (int64_t)sink * 128);
    for (int i = tid; i < 32 * I; i += 256) {
      const int row = i >> 5, c = i & 31;
      st[i] = c < 16 ? rk[row * 16 + c] : rv[row * 16 + (c - 16)];
    }
    int32_t* cnt = p.counts + bh * 16 * 256;
    for (int i = tid; i < 16 * I; i += 256) atomicAdd(cnt + (i & 15) * 256 + wc[(int64_t)sink * 16 + i], 1);
    __syncthreads();
    // slide rows [sink + I, cap_w) down to [sink, ...): chunks of at most I rows, in order, so a chunk's destination
    // only ever overlaps the sources of chunks already moved
    const int keep = p.cap_w - sink - I;
    const int R = min(I, 32);
    for (int r0 = 0; r0 < keep; r0 += R) {
      const int rows = min(R, keep - r0);
      for (int i = tid; i < rows * 39; i += 256) {
        const int row = r0 + i / 39, c = i % 39;
        const int64_t src = sink + I + row, dst = sink + row;
        if (c < 16) reinterpret_cast<uint4*>(wk + dst * 128)[c] = reinterpret_cast<const uint4*>(wk + src * 128)[c];
        else if (c < 32) reinterpret_cast<uint4*>(wv + dst * 128)[c - 16] = reinterpret_cast<const uint4*>(wv + src * 128)[c - 16];
        else if (c < 36) reinterpret_cast<uint4*>(wp + dst * 64)[c - 32] = reinterpret_cast<const uint4*>(wp + src * 64)[c - 32];
        else if (c < 38) reinterpret_cast<uint4*>(ww + dst * 16)[c - 36] = reinterpret_cast<const uint4*>(ww + src * 16)[c - 36];
        else reinterpret_cast<uint4*>(wc + dst * 16)[0] = reinterpret_cast<const uint4*>(wc + src * 16)[0];
      }
      for (int i = tid; i < rows; i += 256) wn[sink + r0 + i] = wn[sink + I + r0 + i];
      __syncthreads();
    }
  }
}

}  // namespace

// Keys per block: about eight blocks per SM over the whole launch (two waves of what is resident), whole rounds of 64 keys,
// at most 4096 so that the blocks stay many; at least 64, so that clearing and adding a block's 16 KB histogram does not
// outweigh the coding.
static int64_t encode_chunk(int64_t L, int64_t heads) {
  const int64_t target = (int64_t)sm_count() * 8;
  int64_t chunk = ((L * heads + target - 1) / target + EN_KEYS - 1) / EN_KEYS * EN_KEYS;
  if (chunk < 64) chunk = 64;
  if (chunk > 4096) chunk = 4096;
  while ((L + chunk - 1) / chunk > 65535) chunk *= 2;
  return chunk;
}

// Host launchers shared with the fused retrieval entry point.
int launch_query_prep(const uint16_t* queries, int bs, int Hq, int H, const uint16_t* signs,
                      uint16_t* q_blocks, uint16_t* q_norm, uint16_t* query_avg, cudaStream_t st) {
  const int G = Hq / H;
  StageTimer tm(ST_QUERY_PREP, st);
  launch_chain(query_prep_kernel, dim3(bs * H), dim3(32), 0, st, queries, Hq, H, G, 1.0f / (float)G, signs, q_blocks, q_norm,
               query_avg);
  return check_launch("query_prep");
}

}  // namespace pk

using namespace pk;

extern "C" int pk_encode_keys(const pk_tensor* keys, const pk_tensor* signs, const pk_tensor* codebook,
                              const pk_tensor* block_weight, const pk_tensor* packed_4bit,
                              const pk_tensor* cluster_counts, void* stream) {
  PK_CHECK_TENSOR(keys, PK_BF16, 4);
  PK_CHECK_TENSOR(signs, PK_BF16, 1);
  PK_CHECK_TENSOR(codebook, PK_U8, 4);
  PK_CHECK_TENSOR(block_weight, PK_BF16, 4);
  PK_CHECK_TENSOR(packed_4bit, PK_U8, 5);
  const int64_t bs = keys->shape[0], H = keys->shape[1], L = keys->shape[2];
  PK_REQUIRE(keys->shape[3] == 128 && signs->shape[0] == 128, "head_dim must be 128");
  PK_REQUIRE(keys->stride[3] == 1 && signs->stride[0] == 1, "keys/signs must have last stride 1");
  PK_REQUIRE((reinterpret_cast<uintptr_t>(keys->data) & 15) == 0 && keys->stride[0] % 8 == 0 &&
                 keys->stride[1] % 8 == 0 && keys->stride[2] % 8 == 0,
             "key rows must be 16-byte aligned");
  PK_REQUIRE((reinterpret_cast<uintptr_t>(signs->data) & 15) == 0, "signs must be 16-byte aligned");
  PK_REQUIRE(codebook->shape[0] == bs && codebook->shape[1] == H && codebook->shape[2] == 16 &&
                 codebook->shape[3] == L,
             "codebook must be [bs,H,16,L]");
  PK_REQUIRE(block_weight->shape[0] == bs && block_weight->shape[1] == H && block_weight->shape[2] == 16 &&
                 block_weight->shape[3] == L,
             "block_weight must be [bs,H,16,L]");
  PK_REQUIRE(packed_4bit->shape[0] == bs && packed_4bit->shape[1] == H && packed_4bit->shape[2] == 16 &&
                 packed_4bit->shape[3] == L && packed_4bit->shape[4] == 4 && packed_4bit->stride[4] == 1,
             "packed_4bit must be [bs,H,16,L,4] with last stride 1");
  if (cluster_counts) {
    PK_CHECK_TENSOR(cluster_counts, PK_I32, 4);
    PK_REQUIRE(is_contig(cluster_counts) && cluster_counts->shape[0] == bs && cluster_counts->shape[1] == H &&
                   cluster_counts->shape[2] == 16 && cluster_counts->shape[3] == 256,
               "cluster_counts must be contiguous [bs,H,16,256]");
  }
  if (bs * H * L == 0) return PK_OK;
  EncodeParams p;
  p.keys = (const uint16_t*)keys->data;
  p.k_b = keys->stride[0], p.k_h = keys->stride[1], p.k_l = keys->stride[2];
  p.signs = (const uint16_t*)signs->data;
  p.codes = (uint8_t*)codebook->data;
  p.c_b = codebook->stride[0], p.c_h = codebook->stride[1], p.c_s = codebook->stride[2], p.c_l = codebook->stride[3];
  p.w = (uint16_t*)block_weight->data;
  p.w_b = block_weight->stride[0], p.w_h = block_weight->stride[1], p.w_s = block_weight->stride[2],
  p.w_l = block_weight->stride[3];
  p.pk = (uint8_t*)packed_4bit->data;
  p.p_b = packed_4bit->stride[0], p.p_h = packed_4bit->stride[1], p.p_s = packed_4bit->stride[2],
  p.p_l = packed_4bit->stride[3];
  p.counts = cluster_counts ? (int32_t*)cluster_counts->data : nullptr;
  p.H = (int)H;
  p.L = L;
  p.chunk = encode_chunk(L, bs * H);
  const bool key_major = p.c_s == 1 && p.c_l == 16 && p.w_s == 1 && p.p_s == 4 && (reinterpret_cast<uintptr_t>(p.codes) & 3) == 0 &&
                         (reinterpret_cast<uintptr_t>(p.w) & 7) == 0 && (reinterpret_cast<uintptr_t>(p.pk) & 15) == 0 &&
                         ((p.c_b | p.c_h | p.w_b | p.w_h | p.w_l) & 3) == 0 && ((p.p_b | p.p_h | p.p_l) & 15) == 0;
  dim3 grid((unsigned)(bs * H), (unsigned)((L + p.chunk - 1) / p.chunk));
  PK_REQUIRE(grid.y <= 65535, "too many keys for one call");
  StageTimer tm(ST_ENCODE, (cudaStream_t)stream);
  if (key_major) encode_kernel<true><<<grid, EN_THREADS, 0, (cudaStream_t)stream>>>(p);
  else encode_kernel<false><<<grid, EN_THREADS, 0, (cudaStream_t)stream>>>(p);
  return check_launch("encode_keys");
}

// ---- tensor maps of the prompt's copies ----
// The driver's encoder, through the runtime, so that the library does not link to the driver.  Asked for until it is found: a lookup
// that fails once does not keep the process on the other form.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static std::atomic<PFN_cuTensorMapEncodeTiled_v12000> found{nullptr};
  if (const auto fn = found.load(std::memory_order_relaxed)) return fn;
  void* f = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
    return cudaGetLastError(), nullptr;
  found.store((PFN_cuTensorMapEncodeTiled_v12000)f, std::memory_order_relaxed);
  return (PFN_cuTensorMapEncodeTiled_v12000)f;
}
// 64 elements x box1 x box2 of a bf16 tensor [d2][d1][inner] in device memory; strides in elements, a multiple of 8.
static bool row_map(CUtensorMap* m, const void* base, int64_t inner, int64_t d1, int64_t s1, int64_t d2, int64_t s2, int box1, int box2) {
  const auto encode = tensor_map_encoder();
  cudaPointerAttributes at;
  if (!encode || s1 <= 0 || s2 <= 0 || s1 >= (1ll << 38) || s2 >= (1ll << 38) || d1 >= (1ll << 31) || d2 >= (1ll << 31)) return false;
  if (cudaPointerGetAttributes(&at, base) != cudaSuccess || at.type != cudaMemoryTypeDevice) return cudaGetLastError(), false;
  const cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)d1, (cuuint64_t)d2}, strides[2] = {(cuuint64_t)s1 * 2, (cuuint64_t)s2 * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)box1, (cuuint32_t)box2}, steps[3] = {1, 1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The maps of a prompt with zone rows; false: the kernel copies row by row.  K and V share the order of their dimensions.
static bool prefill_maps(PrefillMaps& m, const PrefillParams& p) {
  const int64_t kh = p.H == 1 ? p.P * p.k_l : p.k_h, vh = p.H == 1 ? p.P * p.v_l : p.v_h;
  m.heads_inner = p.H > 1 && kh < p.k_l;
  if (m.heads_inner != (p.H > 1 && vh < p.v_l)) return false;
  auto prompt = [&](CUtensorMap* map, const uint16_t* x, int64_t sl, int64_t sh) {
    return m.heads_inner ? row_map(map, x, 128, p.H, sh, p.P, sl, 1, PF_TILE) : row_map(map, x, 128, p.P, sl, p.H, sh, PF_TILE, 1);
  };
  return prompt(&m.k, p.k, p.k_l, kh) && prompt(&m.v, p.v, p.v_l, vh) &&
         row_map(&m.store, p.store, 256, p.N, 256, p.H, p.store_cap * 256, PF_TILE, 1);
}

// The tensors of one cache layer that pk_append_encode and pk_prefill_sample share.
struct CacheLayer {
  int64_t bs, H, cap_w, cap_z, w_b, w_h, z_wl, z_pl;
  float* z_vnorm;
};
static int check_cache_layer(CacheLayer* c, const pk_tensor* window_k, const pk_tensor* window_v, const pk_tensor* win_codes,
                             const pk_tensor* win_weight, const pk_tensor* win_4bit, const pk_tensor* win_vnorm,
                             const pk_tensor* codebook, const pk_tensor* block_weight, const pk_tensor* packed_4bit,
                             const pk_tensor* value_norm, const pk_tensor* cluster_counts, const pk_tensor* state) {
  PK_CHECK_TENSOR(window_k, PK_BF16, 4);
  PK_CHECK_TENSOR(window_v, PK_BF16, 4);
  PK_CHECK_TENSOR(win_codes, PK_U8, 4);
  PK_CHECK_TENSOR(win_weight, PK_BF16, 4);
  PK_CHECK_TENSOR(win_4bit, PK_U8, 5);
  PK_CHECK_TENSOR(win_vnorm, PK_F32, 3);
  PK_CHECK_TENSOR(codebook, PK_U8, 4);
  PK_CHECK_TENSOR(block_weight, PK_BF16, 4);
  PK_CHECK_TENSOR(packed_4bit, PK_U8, 5);
  PK_CHECK_TENSOR(cluster_counts, PK_I32, 4);
  PK_CHECK_TENSOR(state, PK_I32, 1);
  const int64_t bs = window_k->shape[0], H = window_k->shape[1], cap_w = window_k->shape[2];
  PK_REQUIRE(bs >= 1 && H >= 1 && bs * H < (1ll << 31), "window_k must be [bs,H,cap,128]");
  PK_REQUIRE(window_k->shape[3] == 128 && window_k->stride[3] == 1 && window_k->stride[2] == 128 &&
                 (reinterpret_cast<uintptr_t>(window_k->data) & 15) == 0 && (reinterpret_cast<uintptr_t>(window_v->data) & 15) == 0,
             "window_k must be [bs,H,cap,128] with rows 128 elements apart, 16-byte aligned");
  for (int i = 0; i < 4; i++)
    PK_REQUIRE(window_v->shape[i] == window_k->shape[i] && (window_k->shape[i] == 1 || window_v->stride[i] == window_k->stride[i]),
               "window_k and window_v must have the same shape and strides");
  PK_REQUIRE(window_k->stride[0] % 8 == 0 && window_k->stride[1] % 8 == 0, "window strides must be multiples of 8 elements");
  // staging arrays: contiguous, window-aligned
  PK_REQUIRE(is_contig(win_codes) && win_codes->shape[0] == bs && win_codes->shape[1] == H && win_codes->shape[2] == cap_w &&
                 win_codes->shape[3] == 16 && is_contig(win_weight) && numel(win_weight) == bs * H * cap_w * 16 &&
                 is_contig(win_4bit) && numel(win_4bit) == bs * H * cap_w * 64 && is_contig(win_vnorm) &&
                 numel(win_vnorm) == bs * H * cap_w,
             "staging arrays must be contiguous [bs,H,cap,16] u8, [bs,H,cap,16] bf16, [bs,H,cap,16,4] u8, [bs,H,cap] f32");
  for (const pk_tensor* t : {win_codes, win_weight, win_4bit})
    PK_REQUIRE((reinterpret_cast<uintptr_t>(t->data) & 15) == 0, "staging arrays must be 16-byte aligned");
  // zone records: logical [bs,H,16,cap_z(,4)], stored key-major and contiguous
  const int64_t cap_z = codebook->shape[3];
  PK_REQUIRE(codebook->shape[0] == bs && codebook->shape[1] == H && codebook->shape[2] == 16 && codebook->stride[2] == 1 &&
                 codebook->stride[3] == 16 && codebook->stride[1] == cap_z * 16 && (bs == 1 || codebook->stride[0] == H * cap_z * 16),
             "codebook must be the key-major [bs,H,16,cap] view of a contiguous [bs,H,cap,16] buffer");
  const int64_t wl = block_weight->stride[3], pl = packed_4bit->stride[3];   // from key to key; the heads follow each other
  PK_REQUIRE(block_weight->shape[3] == cap_z && block_weight->shape[2] == 16 && block_weight->stride[2] == 1 && wl >= 16 &&
                 wl % 8 == 0 && block_weight->stride[1] == cap_z * wl && (bs == 1 || block_weight->stride[0] == H * cap_z * wl),
             "block_weight must be the key-major [bs,H,16,cap] view of [bs,H,cap] records of at least 16 elements, a multiple of 8");
  PK_REQUIRE(packed_4bit->shape[3] == cap_z && packed_4bit->shape[2] == 16 && packed_4bit->shape[4] == 4 &&
                 packed_4bit->stride[4] == 1 && packed_4bit->stride[2] == 4 && pl >= 64 && pl % 16 == 0 &&
                 packed_4bit->stride[1] == cap_z * pl && (bs == 1 || packed_4bit->stride[0] == H * cap_z * pl),
             "packed_4bit must be the key-major [bs,H,16,cap,4] view of [bs,H,cap] records of at least 64 bytes, a multiple of 16");
  for (const pk_tensor* t : {codebook, block_weight, packed_4bit})
    PK_REQUIRE((reinterpret_cast<uintptr_t>(t->data) & 15) == 0, "zone records must be 16-byte aligned");
  float* zv = nullptr;
  if (value_norm) {
    PK_CHECK_TENSOR(value_norm, PK_F32, 3);
    PK_REQUIRE(is_contig(value_norm) && value_norm->shape[0] == bs && value_norm->shape[1] == H && value_norm->shape[2] == cap_z,
               "value_norm must be contiguous [bs,H,cap] with the zone's capacity");
    zv = (float*)value_norm->data;
  }
  PK_REQUIRE(is_contig(cluster_counts) && cluster_counts->shape[0] == bs && cluster_counts->shape[1] == H &&
                 cluster_counts->shape[2] == 16 && cluster_counts->shape[3] == 256,
             "cluster_counts must be contiguous [bs,H,16,256]");
  PK_REQUIRE(state->stride[0] == 1 && state->shape[0] >= 4 + bs, "state must hold 4 + bs int32 words");
  c->bs = bs, c->H = H, c->cap_w = cap_w, c->cap_z = cap_z, c->z_vnorm = zv, c->z_wl = wl, c->z_pl = pl;
  c->w_b = bs == 1 ? 0 : window_k->stride[0], c->w_h = H == 1 ? 0 : window_k->stride[1];
  return PK_OK;
}

extern "C" int pk_prefill_sample(const pk_tensor* k, const pk_tensor* v, const pk_tensor* signs, const pk_tensor* window_k,
                                 const pk_tensor* window_v, const pk_tensor* win_codes, const pk_tensor* win_weight,
                                 const pk_tensor* win_4bit, const pk_tensor* win_vnorm, const pk_tensor* codebook,
                                 const pk_tensor* block_weight, const pk_tensor* packed_4bit, const pk_tensor* value_norm,
                                 const pk_tensor* cluster_counts, const pk_tensor* rows, const pk_tensor* state, int64_t b,
                                 int64_t sink, int64_t local, void* stream) {
  PK_CHECK_TENSOR(k, PK_BF16, 3);
  PK_CHECK_TENSOR(v, PK_BF16, 3);
  PK_CHECK_TENSOR(signs, PK_BF16, 1);
  PK_CHECK_TENSOR(cluster_counts, PK_I32, 4);
  PK_CHECK_TENSOR(state, PK_I32, 1);
  const int64_t P = k->shape[0], H = k->shape[1];
  for (const pk_tensor* t : {k, v})
    PK_REQUIRE(t->shape[0] == P && t->shape[1] == H && t->shape[2] == 128 && t->stride[2] == 1 &&
                   (reinterpret_cast<uintptr_t>(t->data) & 15) == 0 && (P == 1 || t->stride[0] % 8 == 0) && (H == 1 || t->stride[1] % 8 == 0),
               "k / v must be [P,H,128] with last stride 1 and 16-byte aligned rows");
  PK_REQUIRE(signs->shape[0] == 128 && signs->stride[0] == 1 && (reinterpret_cast<uintptr_t>(signs->data) & 15) == 0,
             "signs must be a 16-byte aligned [128]");
  CacheLayer c;
  int rc = check_cache_layer(&c, window_k, window_v, win_codes, win_weight, win_4bit, win_vnorm, codebook, block_weight,
                             packed_4bit, value_norm, cluster_counts, state);
  if (rc) return rc;
  PK_REQUIRE(c.H == H && b >= 0 && b < c.bs, "k / v and the cache disagree on the heads, or sample %lld does not exist", (long long)b);
  PK_REQUIRE(P >= 1 && sink >= 0 && local >= 0 && sink + local <= c.cap_w, "need at least one token and sink + local rows of window");
  const int64_t N = P > sink + local ? P - sink - local : 0;
  PK_REQUIRE(N > 0 || P <= c.cap_w, "a prompt without zone rows must fit the window");
  PK_REQUIRE(N <= c.cap_z, "the zone records hold %lld keys, %lld needed", (long long)c.cap_z, (long long)N);
  if (N > 0) {
    PK_CHECK_TENSOR(rows, PK_BF16, 4);
    PK_REQUIRE(rows->shape[0] == H && rows->shape[1] >= N && rows->shape[2] == 2 && rows->shape[3] == 128 && rows->stride[3] == 1 &&
                   rows->stride[2] == 128 && rows->stride[1] == 256 && (H == 1 || rows->stride[0] % 256 == 0) &&
                   (reinterpret_cast<uintptr_t>(rows->data) & 15) == 0,
               "rows must be [H,n,2,128] with n >= %lld, a head's rows contiguous", (long long)N);
  }
  cudaStream_t st = (cudaStream_t)stream;
  PrefillParams p = {};
  p.k = (const uint16_t*)k->data, p.v = (const uint16_t*)v->data;
  p.k_l = k->stride[0], p.k_h = k->stride[1], p.v_l = v->stride[0], p.v_h = v->stride[1];
  p.signs = (const uint16_t*)signs->data;
  p.wk = (uint16_t*)window_k->data + b * c.w_b, p.wv = (uint16_t*)window_v->data + b * c.w_b, p.w_h = c.w_h;
  const int64_t wr = b * H * c.cap_w, zr = b * H * c.cap_z;
  p.win_codes = (uint8_t*)win_codes->data + wr * 16, p.win_w = (uint16_t*)win_weight->data + wr * 16;
  p.win_pk = (uint8_t*)win_4bit->data + wr * 64, p.win_vnorm = (float*)win_vnorm->data + wr;
  p.z_codes = (uint8_t*)codebook->data + zr * 16, p.z_w = (uint16_t*)block_weight->data + zr * c.z_wl;
  p.z_pk = (uint8_t*)packed_4bit->data + zr * c.z_pl, p.z_wl = c.z_wl, p.z_pl = c.z_pl, p.z_vnorm = c.z_vnorm ? c.z_vnorm + zr : nullptr;
  p.counts = (int32_t*)cluster_counts->data + b * H * 16 * 256;
  p.state = (int32_t*)state->data;
  p.P = P, p.N = N, p.cap_z = c.cap_z;
  if (N > 0) p.store = (uint16_t*)rows->data, p.store_cap = H == 1 ? rows->shape[1] : rows->stride[0] / 256;
  p.H = (int)H, p.cap_w = (int)c.cap_w, p.sink = (int)sink, p.n_window = (int)(N > 0 ? sink + local : P), p.b = (int)b;
  // By TMA: one wave of two blocks per SM, an even share of the tiles for each; where that makes less than 4/3 of a block per SM (one
  // or two tiles a block, half the warps that an SM has room for), row by row.  B200, us on the device, row by row | by TMA: 8 heads
  // of 2000 tokens (176 blocks) 11.2 | 13.3, 2400 (200) 14.5 | 13.4, 3500 (296) 16.6 | 14.1, 4000 (168) 18.1 | 21.2, 4500 (192)
  // 18.6 | 20.4, 5000 (216) 22.4 | 18.4, 8000 (224) 30.0 | 26.8; 4 heads of 8000 (168) 18.4 | 20.7, of 12000 (252) 24.7 | 20.7; one
  // head of 16000 (167) 10.8 | 13.4, of 24000 (250) 16.9 | 13.1, of 32768 (171) 17.8 | 20.8, of 48000 (250) 24.3 | 18.9.  The host's
  // share of a call (three tensors described, one launch more) is 1.5 - 2 us more by TMA, and hidden at these sizes.
  p.zone_tiles = (N + PF_TILE - 1) / PF_TILE;
  p.n_tiles = p.zone_tiles + (p.n_window + PF_TILE - 1) / PF_TILE;
  const int64_t fit = 2 * (int64_t)sm_count() / H;
  p.tiles_per_block = fit > 1 ? (p.n_tiles + fit - 1) / fit : p.n_tiles;
  while ((p.n_tiles + p.tiles_per_block - 1) / p.tiles_per_block > 65535) p.tiles_per_block *= 2;
  const int64_t blocks = (p.n_tiles + p.tiles_per_block - 1) / p.tiles_per_block;   // of a head
  PrefillMaps maps;
  if (N == 0 || 3 * blocks * H < 4 * (int64_t)sm_count() || !prefill_maps(maps, p)) {
    p.chunk = encode_chunk(P, H);
    if (cudaMemsetAsync(p.counts, 0, (size_t)(H * 16 * 256 * 4), st) != cudaSuccess) return check_launch("prefill memset", 0);
    StageTimer tm(ST_ENCODE, st);
    prefill_rows_kernel<<<dim3((unsigned)H, (unsigned)((P + p.chunk - 1) / p.chunk)), EN_THREADS, 0, st>>>(p);
    return check_launch("prefill");
  }
  static PerDevice smem_attr;
  if (const unsigned long long bit = first_on_device(smem_attr)) {
    if (cudaFuncSetAttribute(prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM) != cudaSuccess) return check_launch("prefill smem", 0);
    mark_on_device(smem_attr, bit);
  }
  prefill_clear_kernel<<<(unsigned)(H * 4), 1024, 0, st>>>(p.counts, b == 0 ? p.state + 3 : nullptr);
  if (const int rc_clear = check_launch("prefill clear")) return rc_clear;
  StageTimer tm(ST_ENCODE, st);
  prefill_kernel<<<dim3((unsigned)H, (unsigned)blocks), PF_THREADS, PF_SMEM, st>>>(p, maps);
  return check_launch("prefill");
}

extern "C" int pk_copy_rows(const pk_tensor* src, const pk_tensor* dst, void* stream) {
  PK_REQUIRE(src && dst && src->data && dst->data, "src / dst is null");
  PK_REQUIRE(src->dtype == dst->dtype && src->ndim == dst->ndim && src->ndim >= 2, "src and dst must have the same type and shape");
  int64_t inner = elem_size(src->dtype);
  for (int i = src->ndim - 1; i >= 0; i--) {
    PK_REQUIRE(src->shape[i] == dst->shape[i], "src and dst must have the same shape");
    if (i == 0) break;
    for (const pk_tensor* t : {src, dst})
      PK_REQUIRE(t->shape[i] == 1 || t->stride[i] * elem_size(t->dtype) == inner, "everything behind the first dimension must be contiguous");
    inner *= src->shape[i];
  }
  const int64_t H = src->shape[0];
  if (H * inner == 0) return PK_OK;
  const int64_t sp = H == 1 ? inner : src->stride[0] * elem_size(src->dtype), dp = H == 1 ? inner : dst->stride[0] * elem_size(dst->dtype);
  PK_REQUIRE(sp >= inner && dp >= inner, "the blocks overlap");
  if (cudaMemcpy2DAsync(dst->data, (size_t)dp, src->data, (size_t)sp, (size_t)inner, (size_t)H, cudaMemcpyDefault,
                        (cudaStream_t)stream) != cudaSuccess)
    return check_launch("copy_rows", 0);
  return PK_OK;
}

extern "C" int pk_count_clusters(const pk_tensor* codebook, const pk_tensor* counts, int accumulate,
                                 void* stream) {
  PK_CHECK_TENSOR(codebook, PK_U8, 4);
  PK_CHECK_TENSOR(counts, PK_I32, 4);
  const int64_t bs = codebook->shape[0], H = codebook->shape[1], B = codebook->shape[2], N = codebook->shape[3];
  PK_REQUIRE(B >= 1 && B <= 32, "subspaces must be in 1..32");
  PK_REQUIRE(is_contig(counts) && counts->shape[0] == bs && counts->shape[1] == H && counts->shape[2] == B &&
                 counts->shape[3] == 256,
             "counts must be contiguous [bs,H,B,256]");
  cudaStream_t st = (cudaStream_t)stream;
  if (!accumulate) {
    if (cudaMemsetAsync(counts->data, 0, (size_t)(bs * H * B * 256 * 4), st) != cudaSuccess)
      return check_launch("count_clusters memset", 0);
  }
  if (bs * H * N == 0) return PK_OK;
  int64_t target = (int64_t)sm_count() * 4;
  int64_t chunk = (N * bs * H + target - 1) / target;
  if (chunk < 256) chunk = 256;
  if (chunk > 8192) chunk = 8192;
  dim3 grid((unsigned)((N + chunk - 1) / chunk), (unsigned)(bs * H));
  StageTimer tm(ST_COUNT, st);
  count_kernel<<<grid, 256, (size_t)B * 256 * 4, st>>>((const uint8_t*)codebook->data, codebook->stride[0],
                                                       codebook->stride[1], codebook->stride[2],
                                                       codebook->stride[3], (int)H, (int)B, N, chunk,
                                                       (int32_t*)counts->data);
  return check_launch("count_clusters");
}

extern "C" int pk_query_prep(const pk_tensor* queries, const pk_tensor* signs, const pk_tensor* q_blocks,
                             const pk_tensor* q_norm, const pk_tensor* query_avg, void* stream) {
  PK_CHECK_TENSOR(queries, PK_BF16, 4);
  PK_CHECK_TENSOR(signs, PK_BF16, 1);
  PK_CHECK_TENSOR(q_blocks, PK_BF16, 4);
  PK_CHECK_TENSOR(q_norm, PK_BF16, 3);
  const int64_t bs = queries->shape[0], Hq = queries->shape[2], H = q_blocks->shape[1];
  PK_REQUIRE(queries->shape[1] == 1 && queries->shape[3] == 128 && is_contig(queries),
             "queries must be contiguous [bs,1,Hq,128]");
  PK_REQUIRE(H > 0 && Hq % H == 0, "query heads (%lld) must be a multiple of KV heads (%lld)", (long long)Hq,
             (long long)H);
  PK_REQUIRE(is_contig(q_blocks) && q_blocks->shape[0] == bs && q_blocks->shape[2] == 16 && q_blocks->shape[3] == 8,
             "q_blocks must be contiguous [bs,H,16,8]");
  PK_REQUIRE(is_contig(q_norm) && q_norm->shape[0] == bs && q_norm->shape[1] == H && q_norm->shape[2] == 1,
             "q_norm must be contiguous [bs,H,1]");
  PK_REQUIRE(signs->shape[0] == 128 && signs->stride[0] == 1, "signs must be [128]");
  uint16_t* qa = nullptr;
  if (query_avg) {
    PK_CHECK_TENSOR(query_avg, PK_BF16, 3);
    PK_REQUIRE(is_contig(query_avg) && query_avg->shape[0] == bs && query_avg->shape[1] == H &&
                   query_avg->shape[2] == 128,
               "query_avg must be contiguous [bs,H,128]");
    qa = (uint16_t*)query_avg->data;
  }
  if (bs * H == 0) return PK_OK;
  return launch_query_prep((const uint16_t*)queries->data, (int)bs, (int)Hq, (int)H, (const uint16_t*)signs->data,
                           (uint16_t*)q_blocks->data, (uint16_t*)q_norm->data, qa, (cudaStream_t)stream);
}

extern "C" int pk_append_encode(const pk_tensor* k_row, const pk_tensor* v_row, const pk_tensor* signs,
                                const pk_tensor* window_k, const pk_tensor* window_v, const pk_tensor* win_codes,
                                const pk_tensor* win_weight, const pk_tensor* win_4bit, const pk_tensor* win_vnorm,
                                const pk_tensor* codebook, const pk_tensor* block_weight, const pk_tensor* packed_4bit,
                                const pk_tensor* value_norm, const pk_tensor* cluster_counts, const pk_tensor* store_kv,
                                const pk_tensor* state, int64_t sink, int64_t interval, void* stream) {
  PK_CHECK_TENSOR(k_row, PK_BF16, 4);
  PK_CHECK_TENSOR(v_row, PK_BF16, 4);
  PK_CHECK_TENSOR(signs, PK_BF16, 1);
  PK_CHECK_TENSOR(store_kv, PK_BF16, 5);
  CacheLayer c;
  int rc = check_cache_layer(&c, window_k, window_v, win_codes, win_weight, win_4bit, win_vnorm, codebook, block_weight,
                             packed_4bit, value_norm, cluster_counts, state);
  if (rc) return rc;
  const int64_t bs = c.bs, H = c.H, cap_w = c.cap_w, cap_z = c.cap_z;
  float* zv = c.z_vnorm;
  PK_REQUIRE(k_row->shape[0] == bs && k_row->shape[1] == 1 && k_row->shape[2] == H && k_row->shape[3] == 128 &&
                 k_row->stride[3] == 1 && v_row->shape[0] == bs && v_row->shape[1] == 1 && v_row->shape[2] == H &&
                 v_row->shape[3] == 128 && v_row->stride[3] == 1,
             "k_row / v_row must be [bs,1,H,128] with last stride 1");
  for (const pk_tensor* t : {k_row, v_row})
    PK_REQUIRE((reinterpret_cast<uintptr_t>(t->data) & 15) == 0 && (t->shape[0] == 1 || t->stride[0] % 8 == 0) &&
                   (t->shape[2] == 1 || t->stride[2] % 8 == 0),
               "k_row / v_row rows must be 16-byte aligned");
  PK_REQUIRE(signs->shape[0] == 128 && signs->stride[0] == 1 && (reinterpret_cast<uintptr_t>(signs->data) & 15) == 0,
             "signs must be a 16-byte aligned [128]");
  PK_REQUIRE(sink >= 0 && interval >= 1 && sink + interval <= cap_w, "need sink + interval <= window capacity");
  PK_REQUIRE(is_contig(store_kv) && store_kv->shape[0] == bs && store_kv->shape[1] == H && store_kv->shape[3] == 2 &&
                 store_kv->shape[4] == 128 && (reinterpret_cast<uintptr_t>(store_kv->data) & 15) == 0,
             "store_kv must be contiguous, 16-byte aligned [bs,H,cap,2,128] (device or pinned host memory)");
  AppendParams p;
  p.k_row = (const uint16_t*)k_row->data, p.v_row = (const uint16_t*)v_row->data;
  p.kr_b = k_row->shape[0] == 1 ? 0 : k_row->stride[0], p.kr_h = k_row->shape[2] == 1 ? 0 : k_row->stride[2];
  p.vr_b = v_row->shape[0] == 1 ? 0 : v_row->stride[0], p.vr_h = v_row->shape[2] == 1 ? 0 : v_row->stride[2];
  p.signs = (const uint16_t*)signs->data;
  p.wk = (uint16_t*)window_k->data, p.wv = (uint16_t*)window_v->data;
  p.w_b = c.w_b, p.w_h = c.w_h;
  p.win_codes = (uint8_t*)win_codes->data, p.win_w = (uint16_t*)win_weight->data, p.win_pk = (uint8_t*)win_4bit->data;
  p.win_vnorm = (float*)win_vnorm->data;
  p.z_codes = (uint8_t*)codebook->data, p.z_w = (uint16_t*)block_weight->data, p.z_pk = (uint8_t*)packed_4bit->data;
  p.z_wl = c.z_wl, p.z_pl = c.z_pl, p.z_vnorm = zv;
  p.counts = (int32_t*)cluster_counts->data;
  p.store = (uint16_t*)store_kv->data;
  p.state = (int32_t*)state->data;
  p.H = (int)H, p.cap_w = (int)cap_w, p.sink = (int)sink, p.interval = (int)interval;
  p.cap_z = cap_z, p.cap_s = store_kv->shape[2];
  StageTimer tm(ST_APPEND, (cudaStream_t)stream);
  launch_chain(append_encode_kernel, dim3((unsigned)(bs * H)), dim3(256), 0, (cudaStream_t)stream, p);
  return check_launch("append_encode");
}
