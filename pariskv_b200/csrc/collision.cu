// Cluster ranking, tier look-up tables and the weighted multi-tier collision count.
//
// The six cumulative tier bitsets of a subspace collapse into one 256-entry byte table (number of tiers a
// cluster belongs to), 4 KB per (batch, head) in shared memory at a link-time address, so one look-up is a
// byte extract, a byte load with an immediate offset and an add.  Codes are streamed with 128-bit loads,
// every thread keeps 256 bytes in flight before it starts counting.
#include <mutex>

#include "chain.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "rotate.cuh"

namespace pk {
namespace {

struct Tiers {
  long long t[8];
  int n;
};

// ---- table builders -----------------------------------------------------------------------------

// From a given cluster order (the collision_fused op): one block per (batch, head, subspace).
template <typename IdT>
__global__ void __launch_bounds__(256) lut_from_sorted_kernel(const IdT* ids, const int32_t* counts, int NC, Tiers tiers,
                                                              uint32_t* lut) {
  __shared__ long long warp_tot[8];
  __shared__ unsigned mask[256];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t blk = blockIdx.x;
  mask[tid] = 0;
  pdl_wait();
  pdl_trigger();
  long long id = -1;
  long long cnt = 0;
  if (tid < NC) {
    id = (long long)ids[blk * NC + tid];
    if (id >= 0 && id < NC) cnt = counts[blk * NC + id];
  }
  long long incl = cnt;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    long long v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  long long base = 0;
  for (int w = 0; w < warp; w++) base += warp_tot[w];
  const long long excl = base + incl - cnt;
  unsigned bits = 0;
  for (int t = 0; t < tiers.n; t++)
    if (excl < tiers.t[t]) bits |= 1u << t;
  if (id >= 0 && id < NC && bits) atomicOr(&mask[id], bits);
  __syncthreads();
  if (tid < 64) {
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) w |= (uint32_t)__popc(mask[tid * 4 + i]) << (8 * i);
    lut[blk * 64 + tid] = w;
  }
}

// The explicit order of the clusters (rank_clusters op): one block per (batch, head, subspace), thread c owns cluster c.
// score_c = bf16(sum_j +-q_j), fp32 sum j ascending; order: score descending, id ascending.
__global__ void __launch_bounds__(256) rank_kernel(const uint16_t* q_blocks, int64_t* sorted_ids) {
  __shared__ __align__(16) unsigned keys[256];   // (ordered bf16 score) << 8 | (255 - id)
  __shared__ float s_q[8];
  const int c = threadIdx.x;
  const int64_t blk = blockIdx.x;  // (b*H + h)*16 + subspace
  pdl_wait();
  pdl_trigger();
  if (c < 8) s_q[c] = bf2f(q_blocks[blk * 8 + c]);
  __syncthreads();
  float s = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const float qv = s_q[j];
    s = __fadd_rn(s, ((c >> j) & 1) ? qv : -qv);
  }
  // order of (score descending, id ascending) as one unsigned compare; -0 counts as +0 like a float compare
  unsigned bits = f2bf(s);
  if (bits == 0x8000u) bits = 0u;
  const unsigned ord = (bits & 0x8000u) ? (~bits & 0xFFFFu) : (bits | 0x8000u);
  const unsigned my_key = (ord << 8) | (unsigned)(255 - c);
  keys[c] = my_key;
  __syncthreads();
  unsigned rank = 0;
  const uint4* k4 = reinterpret_cast<const uint4*>(keys);
#pragma unroll 16
  for (int o = 0; o < 64; o++) {
    const uint4 k = k4[o];  // four keys per 128-bit read (a broadcast: every thread reads the same words)
    rank += (unsigned)(k.x > my_key) + (unsigned)(k.y > my_key) + (unsigned)(k.z > my_key) + (unsigned)(k.w > my_key);
  }
  sorted_ids[blk * 256 + rank] = c;
}

// ---- the streaming count --------------------------------------------------------------------------

struct CollParams {
  const uint8_t* codes;          // element (b,h,s,k) at codes[b*c_b + h*c_h + s*c_s + k*c_l]
  int64_t c_b, c_h, c_s, c_l;
  const uint32_t* lut;           // [bs*H][B][64] words = 256 byte entries per subspace (stand-alone op)
  int32_t* out_i32;              // [bs*H][N]            (stand-alone op)
  uint8_t* out_u8;               // [bs*H][u8_stride], indexed by virtual key (chain kernel)
  uint32_t* chunk_hist;          // [bs*H][n_chunks][256] (chain kernel)
  int64_t u8_stride;
  int H, B;
  int64_t N;                     // keys per head
  int mis;                       // virtual key v = key + mis; loads are 16-byte aligned in v
  int64_t chunk_keys;            // virtual keys per block
  int64_t n_hist;                // histogram rows per (batch, head) of chunk_hist (chain kernel)
  ChainQuery q;                  // chain kernel: the table is built in the block from the query
  int G;
  float inv_g;
  unsigned c256;                 // 256 (see tier_sum16)
};

// The stand-alone op (tier table from global memory, int32 counts out), 256 threads.
// LAYOUT 0: plane-major ([.., 16, N], key stride 1): a thread owns 16 consecutive keys.
// LAYOUT 1: key-major ([.., N, 16], subspace stride 1): a warp owns 512 consecutive keys, lane-strided.
// LAYOUT 2: any strides, any B <= 32: a thread owns one key at a time.
template <int LAYOUT>
__global__ void __launch_bounds__(256, 2) collision_kernel(CollParams p) {
  __shared__ __align__(16) uint8_t s_lut[32 * 256];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bh = blockIdx.y, b = bh / p.H, h = bh % p.H;
  const int64_t N = p.N;
  const int64_t Nv = N + p.mis;
  const int64_t v_begin = (int64_t)blockIdx.x * p.chunk_keys;
  const int64_t v_end = min(Nv, v_begin + p.chunk_keys);
  const uint8_t* base = p.codes + b * p.c_b + h * p.c_h - p.mis * p.c_l;
  pdl_wait();
  pdl_trigger();
  int32_t* out32 = p.out_i32 + (int64_t)bh * p.N;

  // the first batch of code loads is issued before the table is staged, so both latencies overlap
  uint4 r[16];
  if (LAYOUT == 1) {
    const int64_t w0 = v_begin + 512 * (int64_t)warp;
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const int64_t v = w0 + 32 * j + lane;
      r[j] = (v < v_end) ? *reinterpret_cast<const uint4*>(base + v * 16) : make_uint4(0, 0, 0, 0);
    }
  } else if (LAYOUT == 0) {
    const int64_t v0 = v_begin + 16 * (int64_t)tid;
#pragma unroll
    for (int s = 0; s < 16; s++)
      r[s] = (v0 < v_end) ? *reinterpret_cast<const uint4*>(base + s * p.c_s + v0) : make_uint4(0, 0, 0, 0);
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(p.lut + (int64_t)bh * p.B * 64);
    uint4* dst = reinterpret_cast<uint4*>(s_lut);
    for (int i = tid; i < p.B * 16; i += 256) dst[i] = src[i];
  }
  __syncthreads();

  if (LAYOUT == 0) {
    for (int64_t t0 = v_begin; t0 < v_end; t0 += 16 * 256) {  // block-uniform trip count (the warp votes below)
      const int64_t v0 = t0 + 16 * (int64_t)tid;
      const bool live = v0 < v_end;
      int cnt[16];
#pragma unroll
      for (int k = 0; k < 16; k++) cnt[k] = 0;
#pragma unroll
      for (int s = 0; s < 16; s++) {
        const uint32_t w4[4] = {r[s].x, r[s].y, r[s].z, r[s].w};
#pragma unroll
        for (int k = 0; k < 16; k++) cnt[k] += s_lut[s * 256 + byte_of(w4[k >> 2], k & 3)];
      }
      const int64_t vn = v0 + 16 * 256;
      if (vn < v_end) {
#pragma unroll
        for (int s = 0; s < 16; s++) r[s] = *reinterpret_cast<const uint4*>(base + s * p.c_s + vn);
      }
      const int64_t key0 = v0 - p.mis;
      if (live) {
        if (key0 >= 0 && key0 + 16 <= N && ((reinterpret_cast<uintptr_t>(out32 + key0) & 15) == 0)) {
#pragma unroll
          for (int q = 0; q < 4; q++)
            *reinterpret_cast<int4*>(out32 + key0 + 4 * q) =
                make_int4(cnt[4 * q], cnt[4 * q + 1], cnt[4 * q + 2], cnt[4 * q + 3]);
        } else {
#pragma unroll
          for (int k = 0; k < 16; k++)
            if (key0 + k >= 0 && key0 + k < N) out32[key0 + k] = cnt[k];
        }
      }
    }
  } else if (LAYOUT == 1) {
    for (int64_t w0 = v_begin + 512 * (int64_t)warp; w0 < v_end; w0 += 512 * 8) {
      int cnt[16];
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const uint32_t w4[4] = {r[j].x, r[j].y, r[j].z, r[j].w};
        int c = 0;
#pragma unroll
        for (int s = 0; s < 16; s++) c += s_lut[s * 256 + byte_of(w4[s >> 2], s & 3)];
        cnt[j] = c;
      }
      const int64_t wn = w0 + 512 * 8;
      if (wn < v_end) {
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const int64_t v = wn + 32 * j + lane;
          r[j] = (v < v_end) ? *reinterpret_cast<const uint4*>(base + v * 16) : make_uint4(0, 0, 0, 0);
        }
      }
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const int64_t v = w0 + 32 * j + lane;
        if (v < v_end) {
          out32[v] = cnt[j];
        }
      }
    }
  } else {
    for (int64_t v = v_begin + tid; v < v_end; v += 256) {
      const int64_t key = v - p.mis;
      if (key < 0) continue;
      int cnt = 0;
      for (int s = 0; s < p.B; s++) cnt += s_lut[s * 256 + base[s * p.c_s + v * p.c_l]];
      out32[key] = cnt;
    }
  }
}

// ---- the collision kernel of the chain's several-launch form ---------------------------------------------------------
// One block per SM.  While its first code loads are in flight every block builds the tier tables itself (query, ranking,
// prefix sums; chain.cuh), then counts its keys: one u8 per virtual key and one histogram row per block, from which
// the selection kernel derives thresholds and output offsets.
// What bounds it: 7 us of prologue, then the half-rate integer ALU, 28 cycles per 32 keys and SM.  8 heads x 1M keys on B200:
// 64 us with byte tables (bank conflicts), 35 now; the codes alone take 20 at the copy rate.
// LAYOUT 1: key-major records; 0: plane-major ([.., 16, N], a thread owns 16 consecutive keys); 2: any strides.
template <int LAYOUT>
__global__ void __launch_bounds__(CH_THREADS, 1) collide_kernel(CollParams p) {
  __shared__ __align__(16) uint8_t s_lut[16 * 128];
  __shared__ __align__(16) unsigned region[CH_HIST_BYTES / 4];   // count histogram
  __shared__ __align__(16) unsigned s_sizes[16 * 256];           // cluster sizes, then tier counts
  __shared__ __align__(16) float s_q[128];
  __shared__ float s_qnorm;
  __shared__ unsigned s_tiers[9];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bh = blockIdx.y, b = bh / p.H, h = bh % p.H;
  const ChainQuery& cq = p.q;
  PreparedQuery pq;
  QueryLoads ql;
  unsigned key[4];
  const bool early = cq.early_query != 0;
  if (early) {   // the queries were complete before the kernel before this one started
    load_query(ql, cq, b, h, p.G);
    prepare_query(pq, ql, cq, b, h, p.G, p.inv_g, s_q, &s_qnorm);
    __syncthreads();
    rank_subspace(key, s_q + warp * 8, lane);
  }
  if (cq.n_dev || !cq.early_loads) pdl_wait();  // the zone length may have been written by the kernel just before this one
  const int64_t N = cq.n_dev ? min(max((int64_t)cq.n_dev[b], (int64_t)1), p.N) : p.N;
  const int64_t Nv = N + p.mis;
  const int64_t chunk_keys = cq.n_dev ? chain_chunk(Nv, p.n_hist, p.chunk_keys) : p.chunk_keys;
  const int64_t v_begin = (int64_t)blockIdx.x * chunk_keys;
  if (v_begin >= Nv) {  // beyond this sample's zone (whole block, before any barrier but the early one)
    pdl_wait();
    pdl_trigger();
    return;
  }
  const int n_keys = (int)(min(Nv, v_begin + chunk_keys) - v_begin);   // virtual keys of this block
  const uint8_t* base = p.codes + b * p.c_b + h * p.c_h + (v_begin - p.mis) * p.c_l;
  uint8_t* out8 = p.out_u8 + (int64_t)bh * p.u8_stride + v_begin;
  // the first code loads are issued before the tables are built
  constexpr int STEP = CH_WARPS * 128;   // LAYOUT 1: a warp takes 128 consecutive keys (four per lane) of every STEP
  uint4 r0[4], r1[4];
  auto load_codes = [&](uint4 (&r)[4], int v0) {
#pragma unroll
    for (int j = 0; j < 4; j++)   // past the end: the last key again, its count unused
      r[j] = reinterpret_cast<const uint4*>(base)[min(v0 + 32 * j, n_keys - 1)];
  };
  if (LAYOUT == 1) {
    load_codes(r0, warp * 128 + lane);
    load_codes(r1, warp * 128 + lane + STEP);
  }
  pdl_wait();
  pdl_trigger();
  if (!early) load_query(ql, cq, b, h, p.G);
  {
    const int4* cp = reinterpret_cast<const int4*>(cq.counts + ((int64_t)bh * 16 + warp) * 256 + lane * 8);
    const int4 c0 = cp[0], c1 = cp[1];   // cluster sizes of this warp's subspace
    unsigned* my = s_sizes + warp * 256;
    if (!early) prepare_query(pq, ql, cq, b, h, p.G, p.inv_g, s_q, &s_qnorm);
    if (warp == 0 && blockIdx.x == 0) publish_query(pq, cq, bh);
    if (tid >= 32 && tid < 41) load_tiers(cq, (long long)N, s_tiers, tid - 32);
    *reinterpret_cast<int4*>(my + lane * 8) = c0;
    *reinterpret_cast<int4*>(my + lane * 8 + 4) = c1;
    for (int i = tid; i < CH_CBINS * 32; i += CH_THREADS) region[i] = 0;
    __syncthreads();
    if (!early) rank_subspace(key, s_q + warp * 8, lane);
    reinterpret_cast<uint32_t*>(s_lut + warp * 128)[lane] = tier_table(key, my, s_tiers);
    __syncthreads();
  }
  if (LAYOUT == 1) {
    auto count_round = [&](uint4 (&r)[4], int v0) {   // counts four keys and puts the loads of the round after next in their place
      unsigned c[4];
#pragma unroll
      for (int j = 0; j < 4; j++) c[j] = tier_sum16(r[j], s_lut, p.c256);
      load_codes(r, v0 + 2 * STEP);
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (v0 + 32 * j < n_keys) {
          out8[v0 + 32 * j] = (uint8_t)(c[j] >> 4);
          atomicAdd(&region[c[j] * 2 + lane], 1u);   // c is a multiple of 16: word 32 per bin
        }
    };
#pragma unroll 1
    for (int v0 = warp * 128 + lane; v0 - lane < n_keys; v0 += 2 * STEP) {
      count_round(r0, v0);
      if (v0 - lane + STEP < n_keys) count_round(r1, v0 + STEP);
    }
  } else if (LAYOUT == 0) {
    // 16 consecutive keys of a thread, one 16-byte load per subspace; four counts per word, added as bytes
#pragma unroll 1
    for (int v0 = 16 * tid; v0 < n_keys; v0 += 16 * CH_THREADS) {
      uint32_t acc[4] = {0, 0, 0, 0};
#pragma unroll 4
      for (int s = 0; s < 16; s++) {
        const uint4 w = *reinterpret_cast<const uint4*>(base + s * p.c_s + v0);
        acc[0] += tier_bytes(w.x, s_lut + s * 128, p.c256), acc[1] += tier_bytes(w.y, s_lut + s * 128, p.c256);
        acc[2] += tier_bytes(w.z, s_lut + s * 128, p.c256), acc[3] += tier_bytes(w.w, s_lut + s * 128, p.c256);
      }
      *reinterpret_cast<uint4*>(out8 + v0) = make_uint4(acc[0], acc[1], acc[2], acc[3]);
      const int64_t key0 = v_begin + v0 - p.mis;
#pragma unroll
      for (int k = 0; k < 16; k++)
        if (key0 + k >= 0 && key0 + k < N && v0 + k < n_keys)
          atomicAdd(&region[byte_of(acc[k >> 2], k & 3) * 32 + lane], 1u);
    }
  } else {
    for (int v = tid; v < n_keys; v += CH_THREADS) {
      if (v_begin + v - p.mis < 0) continue;
      unsigned cnt = 0;
      for (int s = 0; s < 16; s++) {
        const unsigned c = base[s * p.c_s + v * p.c_l];
        cnt += (s_lut[s * 128 + (c & 127u)] >> (c >> 7 << 2)) & 15u;
      }
      out8[v] = (uint8_t)cnt;
      atomicAdd(&region[cnt * 32 + lane], 1u);
    }
  }
  __syncthreads();
  uint32_t* row = p.chunk_hist + ((int64_t)bh * p.n_hist + blockIdx.x) * 256;
  for (int bin = warp; bin < 256; bin += CH_WARPS) {
    const unsigned t = bin < CH_CBINS ? __reduce_add_sync(0xffffffffu, region[bin * 32 + lane]) : 0u;
    if (lane == 0) row[bin] = t;
  }
}

// Unfused single-tier op: codes are int32 [bs,H,N,B] contiguous; one thread per key.
__global__ void __launch_bounds__(256) collision_i32_kernel(const int32_t* __restrict__ codes,
                                                            const uint32_t* __restrict__ lut_g, int B, int NC,
                                                            int64_t N, int32_t* __restrict__ out) {
  extern __shared__ uint32_t lut_w[];
  const uint8_t* lut = reinterpret_cast<const uint8_t*>(lut_w);
  const int bh = blockIdx.y;
  for (int i = threadIdx.x; i < B * 64; i += 256) lut_w[i] = lut_g[(int64_t)bh * B * 64 + i];
  __syncthreads();
  for (int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x; k < N; k += (int64_t)gridDim.x * 256) {
    const int32_t* row = codes + ((int64_t)bh * N + k) * B;
    int cnt = 0;
    for (int s = 0; s < B; s++) {
      const int32_t c = row[s];
      if (c >= 0 && c < NC) cnt += lut[s * 256 + c];
    }
    out[(int64_t)bh * N + k] = cnt;
  }
}

// single-tier table from (sorted ids, how many leading clusters are selected)
__global__ void __launch_bounds__(256) lut_single_kernel(const int32_t* __restrict__ ids,
                                                         const int32_t* __restrict__ topk_cnt, int NC,
                                                         uint32_t* __restrict__ lut) {
  __shared__ unsigned sel[256];
  const int tid = threadIdx.x;
  const int64_t blk = blockIdx.x;
  sel[tid] = 0;
  __syncthreads();
  if (tid < NC && tid < topk_cnt[blk]) {
    const int id = ids[blk * NC + tid];
    if (id >= 0 && id < NC) sel[id] = 1;
  }
  __syncthreads();
  if (tid < 64) {
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) w |= sel[tid * 4 + i] << (8 * i);
    lut[blk * 64 + tid] = w;
  }
}

Tiers make_tiers(const int64_t* tier_counts, int n) {
  Tiers t;
  t.n = n;
  for (int i = 0; i < 8; i++) t.t[i] = i < n ? (long long)tier_counts[i] : 0;
  return t;
}

}  // namespace

int64_t collision_chunk_keys(int64_t bs_h, int64_t Nv) {
  // one block = 8 warps x 512 keys per pass; about two blocks per SM over the whole grid
  int64_t n_chunks = (2 * (int64_t)sm_count()) / (bs_h > 0 ? bs_h : 1);
  if (n_chunks < 1) n_chunks = 1;
  int64_t chunk = (Nv + n_chunks - 1) / n_chunks;
  chunk = ((chunk + 4095) / 4096) * 4096;
  if (chunk > 32768) chunk = 32768;  // long rows: more blocks, so that the last wave is short
  return chunk;
}

// Launch geometry of the several-launch chain: about one block per SM over the whole grid, one histogram row each; both
// the collision and the selection kernel take chunk_keys virtual keys per block, a multiple of 512 (fewer where the zone's
// length on the device asks for less, see chain_chunk); at most what the selection kernel holds in shared memory.
void chain_geometry(int64_t bs_h, int64_t Nv, int64_t* chunk_keys, int64_t* n_hist) {
  int64_t target = (int64_t)sm_count() / (bs_h > 0 ? bs_h : 1);
  if (target < 1) target = 1;
  int64_t chunk = ((Nv + target - 1) / target + 511) / 512 * 512;
  if (chunk < CHAIN_CHUNK_MIN) chunk = CHAIN_CHUNK_MIN;
  if (chunk > CHAIN_CHUNK_MAX) chunk = CHAIN_CHUNK_MAX;
  *chunk_keys = chunk;
  *n_hist = (Nv + chunk - 1) / chunk;
}

// The stand-alone op: streams the codes of N keys per (batch, head) and writes int32 counts; table from `lut`.
int launch_collision(const pk_tensor* codebook, const uint32_t* lut, int32_t* out_i32, cudaStream_t st) {
  const int64_t bs = codebook->shape[0], H = codebook->shape[1], B = codebook->shape[2], N = codebook->shape[3];
  CollParams p = {};
  p.codes = (const uint8_t*)codebook->data;
  p.c_b = codebook->stride[0], p.c_h = codebook->stride[1], p.c_s = codebook->stride[2], p.c_l = codebook->stride[3];
  p.lut = lut;
  p.out_i32 = out_i32;
  p.H = (int)H, p.B = (int)B, p.N = N;
  const uintptr_t addr = reinterpret_cast<uintptr_t>(p.codes);
  int layout = 2, mis = 0;
  if (B == 16 && p.c_l == 1 && p.c_s % 16 == 0 && p.c_h % 16 == 0 && p.c_b % 16 == 0) {
    layout = 0;
    mis = (int)(addr & 15);
  } else if (B == 16 && p.c_s == 1 && p.c_l == 16 && (addr & 15) == 0 && p.c_h % 16 == 0 && p.c_b % 16 == 0) {
    layout = 1;
  }
  p.mis = mis;
  const int64_t Nv = N + mis;
  p.chunk_keys = collision_chunk_keys(bs * H, Nv);
  const int64_t n_chunks = (Nv + p.chunk_keys - 1) / p.chunk_keys;
  dim3 grid((unsigned)n_chunks, (unsigned)(bs * H));
  StageTimer tm(ST_COLLISION, st);
  if (layout == 0) launch_chain(collision_kernel<0>, grid, dim3(256), 0, st, p);
  else if (layout == 1) launch_chain(collision_kernel<1>, grid, dim3(256), 0, st, p);
  else launch_chain(collision_kernel<2>, grid, dim3(256), 0, st, p);
  return check_launch("collision");
}

// First launch of the several-launch chain: u8 counts per virtual key and one 256-bin histogram row per chunk_keys keys.
int launch_chain_collision(const pk_tensor* codebook, const ChainQuery& cq, uint8_t* counts_u8, int64_t u8_stride,
                           uint32_t* chunk_hist, int* mis_out, int64_t* chunk_keys_out, int64_t* n_hist_out, cudaStream_t st) {
  const int64_t bs = codebook->shape[0], H = codebook->shape[1], B = codebook->shape[2], N = codebook->shape[3];
  if (B != 16) return fail(PK_ERR_ARG, "the fused chain supports 16 subspaces");
  CollParams p = {};
  p.codes = (const uint8_t*)codebook->data;
  p.c_b = codebook->stride[0], p.c_h = codebook->stride[1], p.c_s = codebook->stride[2], p.c_l = codebook->stride[3];
  p.out_u8 = counts_u8;
  p.chunk_hist = chunk_hist;
  p.u8_stride = u8_stride;
  p.H = (int)H, p.B = 16, p.N = N;
  p.q = cq;
  p.G = H > 0 ? cq.Hq / (int)H : 1;
  p.inv_g = 1.0f / (float)p.G;
  p.c256 = 256;
  int layout = 2;
  *mis_out = p.mis = chain_layout(codebook, &layout);
  chain_geometry(bs * H, N + p.mis, &p.chunk_keys, &p.n_hist);
  *chunk_keys_out = p.chunk_keys, *n_hist_out = p.n_hist;
  dim3 grid((unsigned)p.n_hist, (unsigned)(bs * H));
  StageTimer tm(ST_COLLISION, st);
  if (layout == 0) launch_chain(collide_kernel<0>, grid, dim3(CH_THREADS), 0, st, p);
  else if (layout == 1) launch_chain(collide_kernel<1>, grid, dim3(CH_THREADS), 0, st, p);
  else launch_chain(collide_kernel<2>, grid, dim3(CH_THREADS), 0, st, p);
  return check_launch("chain collision");
}

// Which code path a codebook view takes in the chain kernel (0 plane-major, 1 key-major, 2 generic) and, for the
// plane-major one, how many bytes its first key lies past a 16-byte boundary.
int chain_layout(const pk_tensor* codebook, int* layout) {
  const int64_t c_b = codebook->stride[0], c_h = codebook->stride[1], c_s = codebook->stride[2], c_l = codebook->stride[3];
  const uintptr_t addr = reinterpret_cast<uintptr_t>(codebook->data);
  *layout = 2;
  if (c_l == 1 && c_s % 16 == 0 && c_h % 16 == 0 && c_b % 16 == 0) {
    *layout = 0;
    return (int)(addr & 15);
  }
  if (c_s == 1 && c_l == 16 && (addr & 15) == 0 && c_h % 16 == 0 && c_b % 16 == 0) *layout = 1;
  return 0;
}

namespace {
// One block per (batch, head): bin `tid` summed over the chunks.
__global__ void __launch_bounds__(256) hist_reduce_kernel(const uint32_t* chunk_hist, int64_t n_chunks, uint32_t* local_hist) {
  const int64_t bh = blockIdx.x;
  const int tid = threadIdx.x;
  pdl_wait();
  pdl_trigger();
  const uint32_t* hp = chunk_hist + bh * n_chunks * 256 + tid;
  unsigned t = 0;
  int64_t c = 0;
  for (; c + 8 <= n_chunks; c += 8) {
    unsigned v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = hp[(c + i) * 256];
#pragma unroll
    for (int i = 0; i < 8; i++) t += v[i];
  }
  for (; c < n_chunks; c++) t += hp[c * 256];
  local_hist[bh * 256 + tid] = t;
}
}  // namespace

int launch_hist_reduce(const uint32_t* chunk_hist, int64_t bs_h, int64_t n_chunks, uint32_t* local_hist, cudaStream_t st) {
  StageTimer tm(ST_HIST_REDUCE, st);
  launch_chain(hist_reduce_kernel, dim3((unsigned)bs_h), dim3(256), 0, st, chunk_hist, n_chunks, local_hist);
  return check_launch("shard histogram");
}

}  // namespace pk

using namespace pk;

extern "C" int64_t pk_collision_workspace_bytes(int64_t bs, int64_t H, int64_t B, int64_t NC) {
  (void)NC;
  return bs * H * B * 64 * 4;
}

extern "C" int pk_rank_clusters(const pk_tensor* q_blocks, const pk_tensor* sorted_ids, void* stream) {
  PK_CHECK_TENSOR(q_blocks, PK_BF16, 4);
  PK_CHECK_TENSOR(sorted_ids, PK_I64, 4);
  const int64_t bs = q_blocks->shape[0], H = q_blocks->shape[1];
  PK_REQUIRE(is_contig(q_blocks) && q_blocks->shape[2] == 16 && q_blocks->shape[3] == 8,
             "q_blocks must be contiguous [bs,H,16,8]");
  PK_REQUIRE(is_contig(sorted_ids) && sorted_ids->shape[0] == bs && sorted_ids->shape[1] == H &&
                 sorted_ids->shape[2] == 16 && sorted_ids->shape[3] == 256,
             "sorted_ids must be contiguous [bs,H,16,256]");
  if (bs * H == 0) return PK_OK;
  StageTimer tm(ST_RANK, (cudaStream_t)stream);
  launch_chain(rank_kernel, dim3((unsigned)(bs * H * 16)), dim3(256), 0, (cudaStream_t)stream, (const uint16_t*)q_blocks->data,
               (int64_t*)sorted_ids->data);
  return check_launch("rank_clusters");
}

extern "C" int pk_collision_fused(const pk_tensor* sorted_cluster_ids, const pk_tensor* cluster_key_counts,
                                  const pk_tensor* codebook, const int64_t* tier_counts, int n_tiers,
                                  const pk_tensor* cache_cnt, void* workspace, int64_t workspace_bytes,
                                  void* stream) {
  PK_REQUIRE(sorted_cluster_ids && sorted_cluster_ids->data, "sorted_cluster_ids is null");
  PK_REQUIRE(sorted_cluster_ids->dtype == PK_I64 || sorted_cluster_ids->dtype == PK_I32,
             "sorted_cluster_ids must be int64 or int32");
  PK_REQUIRE(sorted_cluster_ids->ndim == 4, "sorted_cluster_ids must be 4-D");
  PK_CHECK_TENSOR(cluster_key_counts, PK_I32, 4);
  PK_CHECK_TENSOR(codebook, PK_U8, 4);
  PK_CHECK_TENSOR(cache_cnt, PK_I32, 3);
  const int64_t bs = codebook->shape[0], H = codebook->shape[1], B = codebook->shape[2], N = codebook->shape[3];
  const int64_t NC = sorted_cluster_ids->shape[3];
  PK_REQUIRE(n_tiers >= 1 && n_tiers <= 8 && tier_counts, "n_tiers must be in 1..8");
  PK_REQUIRE(B >= 1 && B <= 32, "subspaces must be in 1..32, got %lld", (long long)B);
  PK_REQUIRE(NC >= 1 && NC <= 256, "clusters per subspace must be in 1..256, got %lld", (long long)NC);
  PK_REQUIRE(B * n_tiers <= 255, "subspaces x tiers must not exceed 255");
  PK_REQUIRE(is_contig(sorted_cluster_ids) && sorted_cluster_ids->shape[0] == bs && sorted_cluster_ids->shape[1] == H &&
                 sorted_cluster_ids->shape[2] == B,
             "sorted_cluster_ids must be contiguous [bs,H,B,NC]");
  PK_REQUIRE(is_contig(cluster_key_counts) && cluster_key_counts->shape[0] == bs && cluster_key_counts->shape[1] == H &&
                 cluster_key_counts->shape[2] == B && cluster_key_counts->shape[3] == NC,
             "cluster_key_counts must be contiguous [bs,H,B,NC]");
  PK_REQUIRE(is_contig(cache_cnt) && cache_cnt->shape[0] == bs && cache_cnt->shape[1] == H && cache_cnt->shape[2] == N,
             "cache_cnt must be contiguous [bs,H,N]");
  if (bs * H * N == 0) return PK_OK;
  if (!workspace || workspace_bytes < pk_collision_workspace_bytes(bs, H, B, NC))
    return fail(PK_ERR_WORKSPACE, "collision workspace too small: %lld < %lld", (long long)workspace_bytes,
                (long long)pk_collision_workspace_bytes(bs, H, B, NC));
  cudaStream_t st = (cudaStream_t)stream;
  uint32_t* lut = (uint32_t*)workspace;
  Tiers tiers = make_tiers(tier_counts, n_tiers);
  const unsigned nblk = (unsigned)(bs * H * B);
  int rc;
  {
    StageTimer tm(ST_RANK, st);
    if (sorted_cluster_ids->dtype == PK_I64)
      launch_chain(lut_from_sorted_kernel<int64_t>, dim3(nblk), dim3(256), 0, st, (const int64_t*)sorted_cluster_ids->data,
                   (const int32_t*)cluster_key_counts->data, (int)NC, tiers, lut);
    else
      launch_chain(lut_from_sorted_kernel<int32_t>, dim3(nblk), dim3(256), 0, st, (const int32_t*)sorted_cluster_ids->data,
                   (const int32_t*)cluster_key_counts->data, (int)NC, tiers, lut);
    rc = check_launch("collision table");
  }
  if (rc) return rc;
  return launch_collision(codebook, lut, (int32_t*)cache_cnt->data, st);
}

extern "C" int pk_collision(const pk_tensor* sorted_cluster_ids, const pk_tensor* topk_cluster_cnt,
                            const pk_tensor* code_book, const pk_tensor* cache_cnt, void* workspace,
                            int64_t workspace_bytes, void* stream) {
  PK_CHECK_TENSOR(sorted_cluster_ids, PK_I32, 4);
  PK_CHECK_TENSOR(topk_cluster_cnt, PK_I32, 3);
  PK_CHECK_TENSOR(code_book, PK_I32, 4);
  PK_CHECK_TENSOR(cache_cnt, PK_I32, 3);
  const int64_t bs = code_book->shape[0], H = code_book->shape[1], N = code_book->shape[2], B = code_book->shape[3];
  const int64_t NC = sorted_cluster_ids->shape[3];
  PK_REQUIRE(B >= 1 && B <= 32 && NC >= 1 && NC <= 256, "need B <= 32 and NC <= 256");
  PK_REQUIRE(is_contig(sorted_cluster_ids) && is_contig(topk_cluster_cnt) && is_contig(code_book) && is_contig(cache_cnt),
             "all tensors must be contiguous");
  PK_REQUIRE(sorted_cluster_ids->shape[0] == bs && sorted_cluster_ids->shape[1] == H && sorted_cluster_ids->shape[2] == B &&
                 topk_cluster_cnt->shape[0] == bs && topk_cluster_cnt->shape[1] == H && topk_cluster_cnt->shape[2] == B &&
                 cache_cnt->shape[0] == bs && cache_cnt->shape[1] == H && cache_cnt->shape[2] == N,
             "shape mismatch: ids [bs,H,B,NC], cnt [bs,H,B], code_book [bs,H,N,B], cache_cnt [bs,H,N]");
  if (bs * H * N == 0) return PK_OK;
  if (!workspace || workspace_bytes < pk_collision_workspace_bytes(bs, H, B, NC))
    return fail(PK_ERR_WORKSPACE, "collision workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  uint32_t* lut = (uint32_t*)workspace;
  lut_single_kernel<<<(unsigned)(bs * H * B), 256, 0, st>>>((const int32_t*)sorted_cluster_ids->data,
                                                            (const int32_t*)topk_cluster_cnt->data, (int)NC, lut);
  int rc = check_launch("collision table");
  if (rc) return rc;
  int64_t gx = (N + 255) / 256;
  int64_t cap = (int64_t)sm_count() * 8 / (bs * H) + 1;
  if (gx > cap) gx = cap;
  collision_i32_kernel<<<dim3((unsigned)gx, (unsigned)(bs * H)), 256, (size_t)B * 64 * 4, st>>>(
      (const int32_t*)code_book->data, lut, (int)B, (int)NC, N, (int32_t*)cache_cnt->data);
  return check_launch("collision");
}

// ---------------------------------------------------------------------------------------------------------
// Collision count for callers that may not allocate.
//
// pk_collision_fused needs a scratch table from its caller.  Some callers have nowhere to get one: a plugin
// loaded into a serving process whose runtime has already claimed nearly all of HBM for its own pool (a
// cudaMalloc from the plugin then fails or fragments the pool), a real-time decode thread that is forbidden to
// touch the device allocator because an allocation can stall the whole device, or code that was handed raw
// input / output pointers and nothing else.  For them the table lives in the array below, which is part of
// the library image: every GPU that loads the library holds these 256 KB until the process exits.
// ---------------------------------------------------------------------------------------------------------
namespace {
constexpr int64_t kStaticTableBytes = 256 * 1024;  // tables for up to 1024 (batch x head x subspace) triples
static __device__ __align__(256) unsigned char g_static_tier_table[kStaticTableBytes];

// Device address of the array, looked up once per device.  The array's name is only a host-side handle here;
// a kernel must be given the address that cudaGetSymbolAddress returns for the device that is current.
static std::mutex g_static_mu;
static void* g_static_ptr[64] = {nullptr};

int static_table_address(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return fail(PK_ERR_CUDA, "cannot identify the current device");
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (!g_static_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_static_tier_table);
    if (e != cudaSuccess || p == nullptr) {
      cudaGetLastError();
      return fail(PK_ERR_CUDA, "cudaGetSymbolAddress(static tier table): %s", cudaGetErrorString(e));
    }
    g_static_ptr[dev] = p;
  }
  *out = g_static_ptr[dev];
  return PK_OK;
}
}  // namespace

extern "C" int64_t pk_collision_fused_static_max_triples(void) { return kStaticTableBytes / 256; }

extern "C" int pk_collision_fused_static(const pk_tensor* sorted_cluster_ids, const pk_tensor* cluster_key_counts,
                                         const pk_tensor* codebook, const int64_t* tier_counts, int n_tiers,
                                         const pk_tensor* cache_cnt, void* stream) {
  PK_CHECK_TENSOR(codebook, PK_U8, 4);
  PK_CHECK_TENSOR(cluster_key_counts, PK_I32, 4);
  PK_CHECK_TENSOR(cache_cnt, PK_I32, 3);
  PK_REQUIRE(sorted_cluster_ids && sorted_cluster_ids->data && sorted_cluster_ids->ndim == 4,
             "sorted_cluster_ids must be a 4-D tensor");
  const int64_t triples = codebook->shape[0] * codebook->shape[1] * codebook->shape[2];
  if (triples * 256 > kStaticTableBytes)
    return fail(PK_ERR_WORKSPACE,
                "pk_collision_fused_static handles at most %lld (batch x head x subspace) triples, got %lld; use "
                "pk_collision_fused with caller-provided scratch for larger problems",
                (long long)(kStaticTableBytes / 256), (long long)triples);
  void* table = nullptr;
  const int rc = static_table_address(&table);
  if (rc) return rc;
  // The table kernel rewrites every word that the counting kernel reads (64 words per triple), so nothing left
  // over from an earlier call can leak into this one and nothing has to be cleared.
  return pk_collision_fused(sorted_cluster_ids, cluster_key_counts, codebook, tier_counts, n_tiers, cache_cnt, table,
                            kStaticTableBytes, stream);
}

