// Split-K sparse decode attention with the UVA fetch of the selected rows fused in.
//
// Per (batch, KV head) the attended rows are the selected rows of the big K/V store, which may live in pinned host
// memory, followed by the first n_window rows of the GPU window ([sink | local | update buffer]): with the selected
// rows first, their indices can be loaded before the row counts are known.  The rows are cut into tiles of 64 or 128; a block
// takes one tile, or several consecutive ones that it streams through its staging buffers, and stages a tile with TMA bulk copies (cp.async.bulk, one
// 512-byte copy per selected key where its K and V rows are adjacent, completion counted on an mbarrier), so a whole
// grid keeps megabytes outstanding on the host link.  An online softmax over the staged rows runs on the tensor
// cores for up to eight query heads per KV head (on 16 groups of 8 lanes, four heads at a time, for more), and the block
// has one partial (m, l, o) per head.
// Where the blocks of a (batch, KV head) fit a thread-block cluster they merge their partials through distributed shared
// memory, otherwise the block that finishes last merges them from records in the workspace and writes the output: one launch,
// no second kernel, no waiting on blocks that may not be resident.  Scores are kept in the log2 domain.
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace pk {
namespace {

constexpr int ATT_TILE = 64;    // rows of a tile of the streaming form
constexpr int ATT_GQ = 4;       // query heads per pass of the scalar form, and per step of the merge
// Query heads per KV head that the tensor-core form takes in its one pass: the rows 0 .. 7 of its A operand.  Batch 8 of one
// KV head with eight query heads, 2180 rows each: 45 us a launch with the scalar form (two passes), 20 with this one.
constexpr int ATT_MQ = 8;
constexpr int ATT_HEAD_TILES = 5;  // tiles of 128 rows that a block of the cluster form takes at most (see head_tiles)
constexpr int ATT_HEAD_BUFS = 3;   // tiles of 128 rows that a block of the cluster form has in flight: 198 KB
constexpr int ATT_CLUSTER_MAX = 16;
constexpr int ATT_CHAINS = 4;   // accumulators of a score's k-steps; eight spill in the streaming form and cost 1 % there
constexpr int ATT_REC = 132;    // floats per partial: o[128], m, l, pad, pad
constexpr int ATT_WAIT_LIMIT = 4000000;  // polls of the copy barrier before giving up
// Elements (bf16) between two staged rows [K 128 | V 128 | pad].  The tensor-core form pads a row by 16 bytes, so that
// the eight rows of an 8x8 fragment fall into eight different groups of four banks.
template <bool MMA> struct AttRow { static constexpr int stride = MMA ? 264 : 256; };

struct AttParams {
  const uint16_t* q;  // [bs][Hq][128]
  const uint16_t* wk;
  const uint16_t* wv;
  int64_t w_b, w_h, w_l;  // window strides (elements)
  int64_t n_window;       // host value; an upper bound when n_window_dev is set
  const int32_t* n_window_dev;  // optional: actual window rows = n_window_dev[0] + n_window_add (device memory)
  int64_t n_window_add;
  const uint16_t* sk;
  const uint16_t* sv;
  int64_t cap_s;          // rows per (b,h) of the store
  int64_t s_b, s_h, s_l;  // store strides in elements (batch, head, row); K and V share them
  int kv_pair;            // the V row of a store key directly follows its K row: one 512-byte copy fetches both
  const int64_t* sel;     // selected rows of (b,h) at sel[b*sel_b + h*sel_h + j]
  int64_t sel_b, sel_h;
  const int32_t* n_sel;   // [bs*H] or null
  int64_t K, index_offset;
  int H, Hq, G, n_qgroups;
  int tiles_per_block;    // consecutive tiles of a (batch, KV head) that one block streams at most; the grid has ceil(tiles / it) groups
  float scale_log2;
  unsigned* counters;     // [bs*H] arrival counters, zero between calls
  int* status;            // set to 1 if a copy barrier was never completed
  float* ws;              // [bs*Hq][groups][ATT_REC]
  uint16_t* out;          // [bs][Hq][128]
  float* lse;             // optional [bs][Hq]: log2 of the softmax denominator (scaled scores, log2 domain)
};

__device__ __forceinline__ void unpack8f(uint4 v, float* out) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    out[2 * i] = __uint_as_float(w[i] << 16);
    out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 x = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&x);
}

// 2^x for x <= 0: the unit's own instruction, results below 2^-126 are zero.  For the rows of a warp of the tensor-core form only: the
// partials are merged with exp2f, a factor below 2^-126 as it is, because a partial may hold an infinite value.
__device__ __forceinline__ float exp2_neg(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two fp32 operations in one instruction
__device__ __forceinline__ void mul2(float& a, float& b, float f) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(f));
}
__device__ __forceinline__ void add2(float& a, float& b, float c, float d) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(c), "f"(d));
}

__device__ __forceinline__ bool mbar_wait(unsigned mb, unsigned parity, int limit) {
  unsigned done = 0;
  for (int it = 0; it < limit && !done; it++)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(mb), "r"(parity)
        : "memory");
  return done != 0;
}

__device__ __forceinline__ void mbar_arrive(unsigned mb) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mb) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect(unsigned mb, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(bytes) : "memory");
}

// One block takes `tiles_per_block` consecutive tiles of a (batch, KV head) and streams them through two staging
// buffers: while the online softmax runs over tile j, the copies of tile j + 1 are in flight.  With few tiles in the
// whole launch (one sequence) every block has one tile and all copies of the launch are outstanding at once, which is
// what the host link wants; with many (a batch of sequences, rows in HBM) a block amortises its fixed costs - index
// loads, the partial record, the fence and the arrival - over its tiles and the grid is a single wave.
//
// MMA: the scores and the weighted sum of a tile run on the tensor cores (mma.sync m16n8k16, bf16 in, fp32 out) in the
// arrangement of a flash-attention step with the query heads of the KV head as the 16 rows of the A operand (rows
// 0 .. 7): a warp takes 16 rows of the tile, S[head][row] = Q K^T is two n-tiles of eight k-steps, its C fragments ARE the
// A fragments of P for O[head][dim] += P V (sixteen n-tiles over the 128 dims), V^T comes from ldmatrix.trans.
// Neither product gives up precision for the tensor cores:
//   P is split into two bf16 numbers, itself rounded and what the rounding left.  The head's row of A carries the first,
//   the otherwise empty row g + 8 the second, and the two rows of O are added at the end: 17 bits for no further product.
//   The k-steps of a score run in four accumulators, added pairwise: the unit truncates each time it adds to one.
// Against 64 bits, 2180 rows of eight heads a KV head, on B200: 0.88 % of the bf16 outputs not the nearest with P rounded
// and one accumulator, 0.03 like this, 0.04 in the scalar form; rms error of log2 of the denominator 4.4e-6, 1.8e-6, 1.8e-6.
// Packed fp32 arithmetic and the plain ex2 instruction pay for it: a step of two layers with 16 sequences of 16 - 32K keys
// 228 -> 229 us, adaptive budgets of 8 sequences 152 -> 151, 10K keys in host memory 177 -> 175.5.
//
// WARPS: a warp takes 16 rows of a tile.  Four: the streaming form.  Eight: launches that are one tile of 128 rows per
// SM at most; there only latency counts: the same number of records, but one tile instead of two in a row, and twice the
// warps to merge them.  8 heads of 2180 rows in HBM: 9.8 -> 9.3 us alone and 61 -> 58 us for the layer step in a graph;
// batch 8 of one KV head with eight query heads 60 -> 53 us for the step.
//
// CLUSTER: the blocks of a head are a thread-block cluster.  Each has up to three of its tiles of 128 rows in flight, and the
// blocks' partials meet through distributed shared memory: every block merges a share of the outputs.  What this saves is the
// way over L2, 4.4 us from the last product to the end (partial record, fence, atomic, records back into one SM, all in a row;
// 7.3 with eight query heads); 1.6 like this.  B200, a step of four layers with this form switched off -> on, all else the
// same: 10K keys in host memory 156.4 -> 145.1 us, 128K keys 198.4 -> 191.7, one KV head of eight sequences with eight query heads each
// 182.5 -> 176.3.
template <bool MMA, int WARPS, bool CLUSTER>
__global__ void __launch_bounds__(32 * WARPS, WARPS > 4 ? 1 : 3) sparse_attention_kernel(AttParams p) {
  static_assert(!CLUSTER || (MMA && WARPS == 8), "the cluster form");
  constexpr int THREADS = 32 * WARPS, TILE = 16 * WARPS;
  constexpr int NBUF = CLUSTER ? ATT_HEAD_BUFS : WARPS > 4 ? 1 : 2;   // one buffer: one tile per block
  constexpr int RS = AttRow<MMA>::stride;  // elements per staged row
  extern __shared__ __align__(128) unsigned char dyn[];
  uint16_t* KVs = reinterpret_cast<uint16_t*>(dyn);                          // [2 buffers][64][RS]: K row, V row of a key
  constexpr int PQ = MMA ? ATT_MQ : ATT_GQ;   // query heads of a pass
  constexpr int PG = MMA ? WARPS : 16;   // groups of a block that hold partials of them
  // Floats between the partials of two heads: with 8 more than 128 the float2 stores of a half warp (four heads, four lanes of
  // each) fall into all 32 banks, without them into eight.
  constexpr int OS = MMA ? 136 : 128;
  // [PG][PQ][OS], over the LAST buffer (CLUSTER: the first): used when that buffer is idle
  float* obuf = reinterpret_cast<float*>(dyn + (CLUSTER ? 0 : NBUF - 1) * 2 * TILE * RS);
  static_assert(PG * PQ * OS * 4 <= 2 * TILE * RS && WARPS * ATT_GQ * 128 * 4 <= 2 * TILE * RS, "partials fit a buffer");
  __shared__ __align__(8) unsigned long long mbar[NBUF > 2 ? NBUF : 2];
  __shared__ float s_m[PG][PQ], s_l[PG][PQ];
  __shared__ unsigned char s_valid[NBUF][TILE];
  __shared__ int s_last;
  const int tid = threadIdx.x;
  const int h = blockIdx.y, b = blockIdx.z;
  const int64_t bh = (int64_t)b * p.H + h;
  const int n_groups = (int)gridDim.x;
  int tpb = p.tiles_per_block, t_first = (int)blockIdx.x * tpb;
  const unsigned mb0 = (unsigned)__cvta_generic_to_shared(&mbar[0]);
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < (NBUF > 2 ? NBUF : 2); i++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mb0 + 8 * i), "r"(THREADS) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // index of this thread's row of tile t: loaded a tile ahead of the copy that needs it, the first with the row counts
  auto index_of = [&](int t) -> int64_t {
    const int r = t * TILE + (tid >> 1);
    return r < p.K ? p.sel[b * p.sel_b + h * p.sel_h + r] : 0;
  };
  pdl_wait();  // the selected indices and the per-head row counts come from the kernels before this one
  pdl_trigger();
  int64_t ahead = index_of(t_first), later[ATT_HEAD_BUFS - 1];
  if (CLUSTER)
#pragma unroll
    for (int i = 0; i < ATT_HEAD_BUFS - 1; i++) later[i] = i + 1 < tpb ? index_of(t_first + i + 1) : 0;
  const int n_sel = (int)(p.n_sel ? min((int64_t)p.n_sel[bh], p.K) : p.K);   // (a call has at most 65536 rows)
  const int n_window = (int)(p.n_window_dev ? min(p.n_window, max((int64_t)0, (int64_t)p.n_window_dev[0] + p.n_window_add)) : p.n_window);
  const int n_rows = max(0, n_window + n_sel);   // (a count far below zero, which the caller's word may hold, is no row at all)
  // The launch is sized for the most rows there can be; where a block's share of those that there are is a tile less, they are
  // spread evenly over all blocks of the head.  (The indices are then asked for again: their first read was for another tile.)
  // Adaptive budgets select 1024 of the 4096 rows that a launch has room for: two of six blocks a head had all the work.  B200, the
  // launch alone, some 1000 of 4096 rows: 64 heads 25.9 -> 13.9 us, 8 heads 10.5 -> 7.3, of 2048 rows: 96 heads 22.0 -> 16.4; with all of 2048 rows the
  // look at the counts costs 64 heads 0.2 of 17.4, 128 heads 0.5 of 32.9.
  const int n_tiles = (n_rows + TILE - 1) / TILE;
  if (n_tiles <= (tpb - 1) * n_groups) {
    tpb = max(1, (int)((unsigned)(n_tiles + n_groups - 1) / (unsigned)n_groups));
    t_first = (int)blockIdx.x * tpb;
    ahead = index_of(t_first);
    if (CLUSTER)
#pragma unroll
      for (int i = 0; i < ATT_HEAD_BUFS - 1; i++) later[i] = i + 1 < tpb ? index_of(t_first + i + 1) : 0;
  }

  // ---- stage a tile: thread t copies row t/2, K for even t and V for odd t; where the store keeps the V row of a
  // key right behind its K row, the even thread fetches both with one 512-byte copy (half as many requests on the
  // host link).  Every thread arrives on the tile's barrier exactly once, the copying ones with their byte count ----
  auto tile_rows = [&](int t) -> int {
    return max(0, min(TILE, n_rows - t * TILE));
  };
  auto issue = [&](int t, int buf) {
    const int i = tid >> 1;
    const bool is_v = tid & 1;
    const uint16_t* src = nullptr;
    bool ok = i < tile_rows(t), paired = false;
    if (ok) {
      const int r = t * TILE + i;
      if (r >= n_sel) {
        src = (is_v ? p.wv : p.wk) + b * p.w_b + h * p.w_h + (r - n_sel) * p.w_l;
      } else {
        const int64_t row = ahead + p.index_offset;
        ok = row >= 0 && row < p.cap_s;
        paired = p.kv_pair != 0;
        src = ((is_v && !paired) ? p.sv : p.sk) + b * p.s_b + h * p.s_h + (ok ? row : 0) * p.s_l;
      }
    }
    if (!is_v) s_valid[buf][i] = ok;
    const unsigned mb = mb0 + 8 * buf;
    if (ok && !(paired && is_v)) {
      const unsigned dst =
          (unsigned)__cvta_generic_to_shared(KVs + buf * (TILE * RS) + i * RS + ((is_v && !paired) ? 128 : 0));
      mbar_arrive_expect(mb, paired ? 512u : 256u);
      if (paired)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 512, [%2];" ::"r"(dst),
                     "l"(src), "r"(mb)
                     : "memory");
      else
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 256, [%2];" ::"r"(dst),
                     "l"(src), "r"(mb)
                     : "memory");
    } else {
      if (MMA && !ok) {  // a row without a copy is an operand of the matrix products all the same: make it zero
        uint4* z = reinterpret_cast<uint4*>(KVs + buf * (TILE * RS) + i * RS + (is_v ? 128 : 0));
#pragma unroll
        for (int k = 0; k < 16; k++) z[k] = make_uint4(0, 0, 0, 0);
      }
      mbar_arrive(mb);
    }
    if (!CLUSTER) ahead = index_of(t + 1);
  };
  issue(t_first, 0);
  if (CLUSTER) {
#pragma unroll
    for (int i = 0; i < ATT_HEAD_BUFS - 1; i++)
      if (i + 1 < tpb) ahead = later[i], issue(t_first + i + 1, i + 1);
    if (ATT_HEAD_BUFS < tpb) ahead = index_of(t_first + ATT_HEAD_BUFS);
  }

  bool dead = false;  // a copy barrier never completed: reported, the remaining tiles count as empty
  // Called by every thread once per tile j of the block: starts the copies of tile j + 1 (its buffer was released by
  // the barrier that ends tile j - 1), waits for tile j, returns its live rows.
  // The copies never completed: report it, give them (and those of the tile just issued) one more bounded chance to
  // land, and go on with EMPTY tiles (partials m = -inf, l = 0), so that this block still arrives on the counter of
  // its (batch, KV head), the merge runs and the counter returns to zero.  The host must treat a raised status word
  // as fatal.
  auto acquire = [&](int j) -> int {
    if (CLUSTER) {
      if (!dead && !__syncthreads_and(mbar_wait(mb0 + 8 * (j % ATT_HEAD_BUFS), (unsigned)(j / ATT_HEAD_BUFS & 1), ATT_WAIT_LIMIT))) {
        if (tid == 0) atomicExch(p.status, 1);
        for (int i = j; i < min(tpb, j + ATT_HEAD_BUFS); i++) mbar_wait(mb0 + 8 * (i % ATT_HEAD_BUFS), (unsigned)(i / ATT_HEAD_BUFS & 1), ATT_WAIT_LIMIT);
        dead = true;
      }
      return dead ? 0 : tile_rows(t_first + j);
    }
    const int buf = j & 1;
    if (NBUF > 1 && j + 1 < tpb && !dead) issue(t_first + j + 1, buf ^ 1);
    if (!dead && !__syncthreads_and(mbar_wait(mb0 + 8 * buf, (unsigned)((j >> 1) & 1), ATT_WAIT_LIMIT))) {
      if (tid == 0) atomicExch(p.status, 1);
      mbar_wait(mb0 + 8 * buf, (unsigned)((j >> 1) & 1), ATT_WAIT_LIMIT);
      if (j + 1 < tpb) mbar_wait(mb0 + 8 * (buf ^ 1), (unsigned)(((j + 1) >> 1) & 1), ATT_WAIT_LIMIT);
      dead = true;
    }
    return dead ? 0 : tile_rows(t_first + j);
  };
  // Partial record of this block for up to PQ query heads from the groups' (m, l, o) in shared memory.
  auto block_partial = [&](int qg, int n_heads) {
    const int dim = tid & 127;
#pragma unroll 2
    for (int g = tid >> 7; g < n_heads; g += THREADS / 128) {
      float M = -INFINITY;
#pragma unroll 4
      for (int t = 0; t < PG; t++) M = fmaxf(M, s_m[t][g]);
      float L = 0.0f, O = 0.0f;
#pragma unroll 4
      for (int t = 0; t < PG; t++) {
        const float f = (s_m[t][g] == -INFINITY) ? 0.0f : exp2f(s_m[t][g] - M);
        L += s_l[t][g] * f;
        O += obuf[(t * PQ + g) * OS + dim] * f;
      }
      float* rec = p.ws + (((int64_t)b * p.Hq + h * p.G + qg * PQ + g) * n_groups + blockIdx.x) * ATT_REC;
      __stcg(rec + dim, O);
      if (dim == 0) {
        __stcg(rec + 128, M);
        __stcg(rec + 129, L);
      }
    }
  };

  if constexpr (MMA) {
    // ---- tensor-core form: one pass, at most ATT_MQ query heads per KV head ----
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const bool head_ok = g < p.G;
    uint32_t qa[8][2];  // A fragments of Q for the eight k-steps: rows g (a0, a2); rows g + 8 are zero (a1, a3)
    {
      const uint32_t* qrow = reinterpret_cast<const uint32_t*>(p.q + ((int64_t)b * p.Hq + h * p.G + (head_ok ? g : 0)) * 128);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        qa[k][0] = head_ok ? qrow[8 * k + t] : 0u;
        qa[k][1] = head_ok ? qrow[8 * k + 4 + t] : 0u;
      }
    }
    float oacc[16][4];
#pragma unroll
    for (int n = 0; n < 16; n++) oacc[n][0] = oacc[n][1] = oacc[n][2] = oacc[n][3] = 0.0f;
    float m_run = -INFINITY, l_run = 0.0f;  // head g; l is this lane's share, summed over the four lanes at the end
    const int r0 = warp * 16;               // this warp's rows of every tile
    for (int j = 0; j < tpb; j++) {
      const int buf = CLUSTER ? j % ATT_HEAD_BUFS : j & 1;
      const int n_live = acquire(j);
      const uint16_t* tile = KVs + buf * (TILE * RS);
      if (r0 < n_live) {  // warp-uniform
        // S[head][row] = Q K^T over the warp's 16 rows: two n-tiles of eight rows
        float sc[2][2];
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
          float acc[ATT_CHAINS][4] = {};
          const uint32_t* krow = reinterpret_cast<const uint32_t*>(tile + (r0 + nt * 8 + g) * RS);
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const uint32_t b0 = krow[8 * k + t], b1 = krow[8 * k + 4 + t];
            float (&a)[4] = acc[k % ATT_CHAINS];
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                : "+f"(a[0]), "+f"(a[1]), "+f"(a[2]), "+f"(a[3])
                : "r"(qa[k][0]), "r"(0u), "r"(qa[k][1]), "r"(0u), "r"(b0), "r"(b1));
          }
#pragma unroll
          for (int w = ATT_CHAINS / 2; w > 0; w >>= 1)
#pragma unroll
            for (int c = 0; c < w; c++) add2(acc[c][0], acc[c][1], acc[c + w][0], acc[c + w][1]);
          sc[nt][0] = acc[0][0], sc[nt][1] = acc[0][1];
        }
        // online softmax of head g over the rows this lane holds: n-tile nt, columns 2t and 2t + 1
        float v[2][2], mx = -INFINITY;
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int row = r0 + nt * 8 + 2 * t + e;
            const bool live = row < n_live && s_valid[buf][row];
            v[nt][e] = live ? sc[nt][e] * p.scale_log2 : -INFINITY;
            mx = fmaxf(mx, v[nt][e]);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float m_new = fmaxf(m_run, mx);
        const bool none = m_new == -INFINITY;  // no live row so far
        const float corr = none ? 1.0f : exp2_neg(m_run - m_new);
        float pr[2][2];
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
          for (int e = 0; e < 2; e++) pr[nt][e] = none ? 0.0f : exp2_neg(v[nt][e] - m_new);
        l_run = l_run * corr + (pr[0][0] + pr[0][1]) + (pr[1][0] + pr[1][1]);
        m_run = m_new;
#pragma unroll
        for (int n = 0; n < 16; n++) mul2(oacc[n][0], oacc[n][1], corr), mul2(oacc[n][2], oacc[n][3], corr);
        // P as the A operand of the second product: rows g hold the probabilities rounded to bf16, rows g + 8 what is left
        uint32_t pa[4];   // registers 0, 2: row g; 1, 3: row g + 8
#pragma unroll
        for (int nt = 0; nt < 2; nt++) {
          const uint32_t h = pack_bf16(pr[nt][0], pr[nt][1]);
          pa[2 * nt] = h;
          pa[2 * nt + 1] = pack_bf16(pr[nt][0] - __uint_as_float(h << 16), pr[nt][1] - __uint_as_float(h & 0xffff0000u));
        }
        // O[head][dim] += P V: sixteen n-tiles of eight dims, two per ldmatrix (V^T fragments)
        const int mi = lane >> 3;
        const uint16_t* vrow = tile + (r0 + (mi & 1) * 8 + (lane & 7)) * RS + 128 + (mi >> 1) * 8;
#pragma unroll
        for (int np = 0; np < 8; np++) {
          uint32_t b0, b1, b2, b3;
          const unsigned addr = (unsigned)__cvta_generic_to_shared(vrow + np * 16);
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                       : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                       : "r"(addr));
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
              : "+f"(oacc[2 * np][0]), "+f"(oacc[2 * np][1]), "+f"(oacc[2 * np][2]), "+f"(oacc[2 * np][3])
              : "r"(pa[0]), "r"(pa[1]), "r"(pa[2]), "r"(pa[3]), "r"(b0), "r"(b1));
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
              : "+f"(oacc[2 * np + 1][0]), "+f"(oacc[2 * np + 1][1]), "+f"(oacc[2 * np + 1][2]), "+f"(oacc[2 * np + 1][3])
              : "r"(pa[0]), "r"(pa[1]), "r"(pa[2]), "r"(pa[3]), "r"(b2), "r"(b3));
        }
      }
      __syncthreads();  // the tile has been consumed: its buffer may be refilled (after the last tile obuf is free)
      if (CLUSTER && j + ATT_HEAD_BUFS < tpb && !dead) {
        issue(t_first + j + ATT_HEAD_BUFS, buf);
        ahead = index_of(t_first + j + ATT_HEAD_BUFS + 1);
      }
    }
    // the four warps are the groups of the block-level merge
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    // the two parts of O; where a value row is infinite the first alone (the rest may be zero, and 0 x inf is not a number)
    auto join = [](float o, float rest) { return fabsf(o) < INFINITY ? o + rest : o; };
    if (head_ok) {
#pragma unroll
      for (int n = 0; n < 16; n++)
        *reinterpret_cast<float2*>(obuf + (warp * PQ + g) * OS + 8 * n + 2 * t) = make_float2(join(oacc[n][0], oacc[n][2]), join(oacc[n][1], oacc[n][3]));
      if (t == 0) s_m[warp][g] = m_run, s_l[warp][g] = l_run;
    }
    if constexpr (CLUSTER) {
      // Unit u: dims 4 (u & 31) .. + 3 of head u >> 5.  The warps' partials become the block's, a thread per unit; behind the
      // cluster barrier every block takes consecutive units, eight lanes a unit, each of them every eighth block's partial.
      cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
      __shared__ __align__(16) float4 s_o[ATT_MQ * 32];
      __shared__ float2 s_ml[ATT_MQ];
      const int units = p.G * 32;
      __syncthreads();
      if (tid < units) {
        const int hd = tid >> 5;
        float M = -INFINITY, L = 0.0f;
        float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int w = 0; w < WARPS; w++) M = fmaxf(M, s_m[w][hd]);
#pragma unroll
        for (int w = 0; w < WARPS; w++) {
          const float f = s_m[w][hd] == -INFINITY ? 0.0f : exp2f(s_m[w][hd] - M);
          const float4 v = reinterpret_cast<const float4*>(obuf + (w * PQ + hd) * OS)[lane];
          L += s_l[w][hd] * f, o.x += v.x * f, o.y += v.y * f, o.z += v.z * f, o.w += v.w * f;
        }
        s_o[tid] = o;
        if (lane == 0) s_ml[hd] = make_float2(M, L);
      }
      cluster.sync();
      constexpr int MB = ATT_CLUSTER_MAX / 8;
      const int per = (units + n_groups - 1) / n_groups, sub = lane & 7;
      const int u1 = min(units, ((int)blockIdx.x + 1) * per);
      for (int u0 = blockIdx.x * per; u0 < u1; u0 += THREADS / 8) {
        const int u = u0 + (tid >> 3), hd = u < u1 ? u >> 5 : 0;
        float2 ml[MB];
        float4 v[MB];
#pragma unroll
        for (int i = 0; i < MB; i++) {
          ml[i] = make_float2(-INFINITY, 0.0f), v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (u < u1 && sub + 8 * i < n_groups)
            ml[i] = *cluster.map_shared_rank(&s_ml[hd], sub + 8 * i), v[i] = *cluster.map_shared_rank(&s_o[u], sub + 8 * i);
        }
        float m = -INFINITY, l = 0.0f;
        float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < MB; i++) m = fmaxf(m, ml[i].x);
#pragma unroll
        for (int i = 0; i < MB; i++) {
          const float f = ml[i].x == -INFINITY ? 0.0f : exp2f(ml[i].x - m);
          l += ml[i].y * f, o.x += v[i].x * f, o.y += v[i].y * f, o.z += v[i].z * f, o.w += v[i].w * f;
        }
        float M = m;
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
        const float f = m == -INFINITY ? 0.0f : exp2f(m - M);
        l *= f, o.x *= f, o.y *= f, o.z *= f, o.w *= f;
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) {
          l += __shfl_xor_sync(0xffffffffu, l, off);
          o.x += __shfl_xor_sync(0xffffffffu, o.x, off), o.y += __shfl_xor_sync(0xffffffffu, o.y, off);
          o.z += __shfl_xor_sync(0xffffffffu, o.z, off), o.w += __shfl_xor_sync(0xffffffffu, o.w, off);
        }
        if (u < u1 && sub == 0) {
          const int64_t bq = (int64_t)b * p.Hq + h * p.G + hd;
          const bool any = l > 0.0f;
          *reinterpret_cast<uint2*>(p.out + bq * 128 + 4 * (u & 31)) =
              any ? make_uint2(pack_bf16(o.x / l, o.y / l), pack_bf16(o.z / l, o.w / l)) : make_uint2(0u, 0u);
          if (p.lse && (u & 31) == 0) p.lse[bq] = any ? M + log2f(l) : -INFINITY;
        }
      }
      cluster.sync();   // shared memory must outlive the other blocks' reads
      return;
    }
    __syncthreads();
    block_partial(0, p.G);
  } else {
    const int s = tid & 7, grp = tid >> 3;
    for (int qg = 0; qg < p.n_qgroups; qg++) {  // more than one pass only for more than four query heads per KV head,
                                                // and then a block has a single tile, which stays staged
      const int n_heads = min(ATT_GQ, p.G - qg * ATT_GQ);
      float qf[ATT_GQ][16];
#pragma unroll
      for (int g = 0; g < ATT_GQ; g++) {
        if (g < n_heads) {
          const uint4* qp =
              reinterpret_cast<const uint4*>(p.q + ((int64_t)b * p.Hq + h * p.G + qg * ATT_GQ + g) * 128 + 16 * s);
          unpack8f(qp[0], qf[g]);
          unpack8f(qp[1], qf[g] + 8);
        } else {
#pragma unroll
          for (int i = 0; i < 16; i++) qf[g][i] = 0.0f;
        }
      }
      float m[ATT_GQ], lsum[ATT_GQ], o[ATT_GQ][16];
#pragma unroll
      for (int g = 0; g < ATT_GQ; g++) {
        m[g] = -INFINITY;
        lsum[g] = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; i++) o[g][i] = 0.0f;
      }
      for (int j = 0; j < tpb; j++) {
        const int buf = j & 1;
        const int n_live = qg == 0 ? acquire(j) : (dead ? 0 : tile_rows(t_first + j));
        const uint16_t* tile = KVs + buf * (TILE * RS);
        for (int i = grp; i < TILE; i += 16) {  // uniform trip count per warp: shuffles need all lanes
          const bool live = i < n_live && s_valid[buf][i];
          float kf[16], vf[16];
          if (live) {
            const uint4* kp = reinterpret_cast<const uint4*>(tile + i * RS + 16 * s);
            const uint4* vp = reinterpret_cast<const uint4*>(tile + i * RS + 128 + 16 * s);
            unpack8f(kp[0], kf);
            unpack8f(kp[1], kf + 8);
            unpack8f(vp[0], vf);
            unpack8f(vp[1], vf + 8);
          } else {
#pragma unroll
            for (int jj = 0; jj < 16; jj++) kf[jj] = 0.0f, vf[jj] = 0.0f;
          }
#pragma unroll
          for (int g = 0; g < ATT_GQ; g++) {
            float d = 0.0f;
#pragma unroll
            for (int jj = 0; jj < 16; jj++) d = fmaf(kf[jj], qf[g][jj], d);
            d += __shfl_xor_sync(0xffffffffu, d, 1);
            d += __shfl_xor_sync(0xffffffffu, d, 2);
            d += __shfl_xor_sync(0xffffffffu, d, 4);
            if (live) {
              const float sc = d * p.scale_log2;
              const float mn = fmaxf(m[g], sc);
              const float corr = exp2f(m[g] - mn);  // m = -inf on the first row gives 0
              const float pr = exp2f(sc - mn);
              lsum[g] = lsum[g] * corr + pr;
#pragma unroll
              for (int jj = 0; jj < 16; jj++) o[g][jj] = o[g][jj] * corr + pr * vf[jj];
              m[g] = mn;
            }
          }
        }
        __syncthreads();  // the tile has been consumed: its buffer may be refilled (and, after the last tile or
                          // between passes, obuf / s_m / s_l are free)
      }
#pragma unroll
      for (int g = 0; g < ATT_GQ; g++) {
#pragma unroll
        for (int jj = 0; jj < 16; jj++) obuf[(grp * PQ + g) * OS + 16 * s + jj] = o[g][jj];
        if (s == 0) {
          s_m[grp][g] = m[g];
          s_l[grp][g] = lsum[g];
        }
      }
      __syncthreads();
      block_partial(qg, n_heads);
      __syncthreads();  // obuf / s_m / s_l have been consumed before the next pass writes them
    }
  }

  // ---- the block that arrives last for this (batch, KV head) merges all tiles ----
  __syncthreads();
  if (tid == 0) {   // one thread's fences order the whole block's records (the barriers carry them to and from it)
    __threadfence();
    s_last = atomicAdd(p.counters + bh, 1u) + 1u == (unsigned)n_groups;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  if (tid == 0) p.counters[bh] = 0;  // ready for the next call on this stream (behind the fence: nobody waits for it)
  // ATT_GQ query heads are merged by all warps, up to twice as many by half of the warps each.  The warps take the records in
  // turn, a lane four dims of each; the records of MB steps are in flight together, (m, l) with the values, because nothing in
  // this tail but their latency costs time: 36 records of four heads took 6.6 us with a pass for the scale factors and 16
  // single floats in flight per thread, 4.4 like this with four warps.  The warps' sums meet in shared memory.
  const int warp = tid >> 5, lane = tid & 31;
  auto merge = [&](auto n_parts, int q0) {
    constexpr int parts = decltype(n_parts)::value, nw = WARPS / parts, MB = MMA && nw <= 4 ? 5 : 3;
    const int n_heads = min(parts * ATT_GQ, p.G - q0);
    const int first = warp / nw * ATT_GQ, mine = min(ATT_GQ, n_heads - first);   // this warp's heads
    const int64_t bq0 = (int64_t)b * p.Hq + h * p.G + q0;
    float m[ATT_GQ], l[ATT_GQ];
    float4 o[ATT_GQ];
#pragma unroll
    for (int g = 0; g < ATT_GQ; g++) m[g] = -INFINITY, l[g] = 0.0f, o[g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int t0 = warp % nw; t0 < n_groups; t0 += nw * MB) {
      float4 v[MB][ATT_GQ];
      float2 ml[MB][ATT_GQ];
#pragma unroll
      for (int i = 0; i < MB; i++)
#pragma unroll
        for (int g = 0; g < ATT_GQ; g++) {
          const int t = t0 + nw * i;
          ml[i][g] = make_float2(-INFINITY, 0.0f), v[i][g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (t < n_groups && g < mine) {
            const float* rec = p.ws + ((bq0 + first + g) * n_groups + t) * ATT_REC;
            ml[i][g] = __ldcg(reinterpret_cast<const float2*>(rec + 128));
            v[i][g] = __ldcg(reinterpret_cast<const float4*>(rec) + lane);
          }
        }
#pragma unroll
      for (int g = 0; g < ATT_GQ; g++) {
        float mn = m[g];
#pragma unroll
        for (int i = 0; i < MB; i++) mn = fmaxf(mn, ml[i][g].x);
        if (mn == -INFINITY) continue;   // no live row so far
        const float c = exp2f(m[g] - mn);
        m[g] = mn, l[g] *= c, o[g].x *= c, o[g].y *= c, o[g].z *= c, o[g].w *= c;
#pragma unroll
        for (int i = 0; i < MB; i++) {
          const float f = exp2f(ml[i][g].x - mn);
          l[g] += ml[i][g].y * f;
          o[g].x += v[i][g].x * f, o[g].y += v[i][g].y * f, o[g].z += v[i][g].z * f, o[g].w += v[i][g].w * f;
        }
      }
    }
    if (q0) __syncthreads();            // the sums of the previous heads have been consumed
#pragma unroll
    for (int g = 0; g < ATT_GQ; g++) {
      if (lane == 0) s_m[warp][g] = m[g], s_l[warp][g] = l[g];
      reinterpret_cast<float4*>(obuf + (warp * ATT_GQ + g) * 128)[lane] = o[g];
    }
    __syncthreads();
    for (int g = tid >> 7; g < n_heads; g += THREADS / 128) {
      const int w0 = g / ATT_GQ * nw, gg = g % ATT_GQ;   // the warps that merged this head
      float M = -INFINITY, L = 0.0f, O = 0.0f;
#pragma unroll
      for (int w = 0; w < nw; w++) M = fmaxf(M, s_m[w0 + w][gg]);
#pragma unroll
      for (int w = 0; w < nw; w++) {
        const float f = s_m[w0 + w][gg] == -INFINITY ? 0.0f : exp2f(s_m[w0 + w][gg] - M);
        L += s_l[w0 + w][gg] * f;
        O += obuf[((w0 + w) * ATT_GQ + gg) * 128 + (tid & 127)] * f;
      }
      p.out[(bq0 + g) * 128 + (tid & 127)] = f2bf(L > 0.0f ? O / L : 0.0f);
      if (p.lse && (tid & 127) == 0) p.lse[bq0 + g] = L > 0.0f ? M + log2f(L) : -INFINITY;
    }
  };
  for (int q0 = 0; q0 < p.G;) {
    if (p.G - q0 > ATT_GQ) merge(std::integral_constant<int, 2>(), q0), q0 += 2 * ATT_GQ;
    else merge(std::integral_constant<int, 1>(), q0), q0 += ATT_GQ;
  }
}

template <bool MMA, int WARPS>
int launch_attention(const AttParams& p, dim3 grid, cudaStream_t st) {
  const int smem = (WARPS > 4 ? 1 : 2) * 16 * WARPS * AttRow<MMA>::stride * 2;
  static PerDevice smem_attr;   // the opt-in to more than 48 KB of dynamic shared memory is per kernel and device
  if (const unsigned long long bit = first_on_device(smem_attr)) {
    if (cudaFuncSetAttribute(sparse_attention_kernel<MMA, WARPS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return check_launch("sparse_attention smem");
    mark_on_device(smem_attr, bit);
  }
  StageTimer tm(ST_ATTENTION, st);
  launch_chain(sparse_attention_kernel<MMA, WARPS, false>, grid, dim3(32 * WARPS), (size_t)smem, st, p);
  return check_launch("sparse_attention");
}

// ---- the cluster form ----
int head_smem(int tiles) { return (tiles < ATT_HEAD_BUFS ? tiles : ATT_HEAD_BUFS) * 128 * AttRow<true>::stride * 2; }
cudaLaunchConfig_t head_config(cudaLaunchAttribute* attr, dim3 grid, int tiles, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid, cfg.blockDim = dim3(256), cfg.dynamicSmemBytes = (size_t)head_smem(tiles), cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = grid.x, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cfg;
}
// Clusters of a size, with a number of tiles per block, that fit the device at once; asked once per device.
struct HeadCapacity {
  int active[ATT_HEAD_BUFS + 1][ATT_CLUSTER_MAX + 1];
};
const HeadCapacity* head_capacity() {
  static HeadCapacity cap[64];
  static PerDevice asked;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (const unsigned long long bit = first_on_device(asked)) {
    auto kern = sparse_attention_kernel<true, 8, true>;
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, head_smem(ATT_HEAD_BUFS)) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    for (int tiles = 1; tiles <= ATT_HEAD_BUFS; tiles++)   // several threads may ask at the same time: they write the same numbers
      for (int cs = 1; cs <= ATT_CLUSTER_MAX; cs++) {
        cudaLaunchAttribute attr[2];
        cudaLaunchConfig_t cfg = head_config(attr, dim3(cs, 64), tiles, nullptr);
        cfg.numAttrs = 1;
        int n = 0;
        cap[dev].active[tiles][cs] = ok && cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess ? n : 0;
      }
    cudaGetLastError();
    mark_on_device(asked, bit);
  }
  return &cap[dev];
}
// Tiles of 128 rows per block of the cluster form, or 0 where it does not apply: as few as make a cluster that is resident for
// every head at once, at most ATT_HEAD_TILES.  On B200, us per launch of four query heads per KV head, the other forms -> this
// one, at one to six tiles: 8 heads of 700 rows 7.4 -> 5.0; of 2244 rows 8 heads 7.7 -> 6.6, 16 heads 11.7 -> 8.6, 24 heads
// 12.7 -> 11.1, 32 heads 14.3 -> 13.5, 40 heads 15.9 -> 16.2.  Beyond, three blocks of four warps per SM stream faster than one of eight.
int head_tiles(int64_t n_halves, int64_t heads) {
  const HeadCapacity* cap = head_capacity();
  for (int64_t cs = n_halves < ATT_CLUSTER_MAX ? n_halves : ATT_CLUSTER_MAX; cap && cs >= 1; cs--) {
    const int64_t tiles = (n_halves + cs - 1) / cs;
    if (tiles > ATT_HEAD_TILES) break;
    if (heads <= cap->active[tiles < ATT_HEAD_BUFS ? tiles : ATT_HEAD_BUFS][(n_halves + tiles - 1) / tiles]) return (int)tiles;
  }
  return 0;
}
int launch_head_attention(const AttParams& p, dim3 grid, cudaStream_t st) {
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = head_config(attr, grid, p.tiles_per_block, st);
  StageTimer tm(ST_ATTENTION, st);
  if (cudaLaunchKernelEx(&cfg, sparse_attention_kernel<true, 8, true>, p) != cudaSuccess) return check_launch("sparse_attention cluster", 0);
  return check_launch("sparse_attention");
}

}  // namespace
}  // namespace pk

using namespace pk;

namespace {
inline int64_t att_header_bytes(int64_t bs, int64_t H) { return (bs * H * 4 + 4 + 255) / 256 * 256; }
}  // namespace

extern "C" int64_t pk_attention_workspace_bytes(int64_t bs, int64_t Hq, int64_t max_rows) {
  // header (arrival counters + status word, sized for one KV head per query head) followed by the partials
  const int64_t tiles = (max_rows + ATT_TILE - 1) / ATT_TILE;
  return att_header_bytes(bs, Hq) + bs * Hq * (tiles > 0 ? tiles : 1) * ATT_REC * 4;
}

extern "C" int pk_sparse_attention(const pk_tensor* queries, const pk_tensor* window_k, const pk_tensor* window_v,
                                   int64_t n_window, const pk_tensor* n_window_dev, int64_t n_window_add,
                                   const pk_tensor* store_k, const pk_tensor* store_v,
                                   const pk_tensor* selected, const pk_tensor* n_sel, int64_t index_offset,
                                   float scale, const pk_tensor* out, const pk_tensor* lse, void* workspace,
                                   int64_t workspace_bytes, void* stream) {
  PK_CHECK_TENSOR(queries, PK_BF16, 4);
  PK_CHECK_TENSOR(out, PK_BF16, 4);
  const int64_t bs = queries->shape[0], Hq = queries->shape[2];
  PK_REQUIRE(queries->shape[1] == 1 && queries->shape[3] == 128 && is_contig(queries) &&
                 (reinterpret_cast<uintptr_t>(queries->data) & 15) == 0,
             "queries must be contiguous, 16-byte aligned [bs,1,Hq,128]");
  PK_REQUIRE(is_contig(out) && out->shape[0] == bs && out->shape[1] == 1 && out->shape[2] == Hq && out->shape[3] == 128,
             "out must be contiguous [bs,1,Hq,128]");
  AttParams p = {};
  int64_t H = 0;
  if (n_window > 0) {
    PK_CHECK_TENSOR(window_k, PK_BF16, 4);
    PK_CHECK_TENSOR(window_v, PK_BF16, 4);
    H = window_k->shape[1];
    PK_REQUIRE(window_k->shape[0] == bs && window_k->shape[3] == 128 && window_k->stride[3] == 1 &&
                   window_k->shape[2] >= n_window,
               "window_k must be [bs,H,cap>=n_window,128] with last stride 1");
    for (int i = 0; i < 4; i++)
      PK_REQUIRE(window_k->shape[i] == window_v->shape[i] &&
                     (window_k->shape[i] == 1 || window_k->stride[i] == window_v->stride[i]),
                 "window_k and window_v must have the same shape and strides");
    PK_REQUIRE((reinterpret_cast<uintptr_t>(window_k->data) & 15) == 0 && (reinterpret_cast<uintptr_t>(window_v->data) & 15) == 0 &&
                   window_k->stride[0] % 8 == 0 && window_k->stride[1] % 8 == 0 && window_k->stride[2] % 8 == 0,
               "window rows must be 16-byte aligned");
    p.wk = (const uint16_t*)window_k->data, p.wv = (const uint16_t*)window_v->data;
    p.w_b = window_k->stride[0], p.w_h = window_k->stride[1], p.w_l = window_k->stride[2];
  }
  int64_t K = 0;
  if (selected) {
    PK_CHECK_TENSOR(selected, PK_I64, 3);
    PK_CHECK_TENSOR(store_k, PK_BF16, 4);
    PK_CHECK_TENSOR(store_v, PK_BF16, 4);
    K = selected->shape[2];
    PK_REQUIRE(H == 0 || store_k->shape[1] == H, "window and store disagree on the number of KV heads");
    H = store_k->shape[1];
    PK_REQUIRE(store_k->shape[0] == bs && store_k->shape[3] == 128 && store_v->shape[0] == bs && store_v->shape[1] == H &&
                   store_v->shape[2] == store_k->shape[2] && store_v->shape[3] == 128 && store_k->stride[3] == 1 &&
                   store_v->stride[3] == 1,
               "store_k / store_v must be [bs,H,cap,128] with last stride 1");
    for (int i = 0; i < 3; i++) {
      PK_REQUIRE(store_k->shape[i] == 1 || store_k->stride[i] == store_v->stride[i], "store_k and store_v must have the same strides");
      PK_REQUIRE(store_k->shape[i] == 1 || store_k->stride[i] % 8 == 0, "store rows must be 16-byte aligned");
    }
    PK_REQUIRE((reinterpret_cast<uintptr_t>(store_k->data) & 15) == 0 && (reinterpret_cast<uintptr_t>(store_v->data) & 15) == 0,
               "store rows must be 16-byte aligned");
    p.s_b = store_k->shape[0] == 1 ? 0 : store_k->stride[0];
    p.s_h = store_k->shape[1] == 1 ? 0 : store_k->stride[1];
    p.s_l = store_k->shape[2] == 1 ? 128 : store_k->stride[2];
    PK_REQUIRE(selected->shape[0] == bs && selected->shape[1] == H && (K <= 1 || selected->stride[2] == 1),
               "selected must be [bs,H,K] with last stride 1");
    p.sel_b = selected->stride[0], p.sel_h = selected->stride[1];
    p.sk = (const uint16_t*)store_k->data, p.sv = (const uint16_t*)store_v->data;
    p.kv_pair = (p.sv == p.sk + 128 && p.s_l >= 256) ? 1 : 0;
    p.cap_s = store_k->shape[2];
    p.sel = (const int64_t*)selected->data;
    if (n_sel) {
      PK_CHECK_TENSOR(n_sel, PK_I32, 2);
      PK_REQUIRE(is_contig(n_sel) && n_sel->shape[0] == bs && n_sel->shape[1] == H, "n_sel must be contiguous [bs,H]");
      p.n_sel = (const int32_t*)n_sel->data;
    }
  }
  PK_REQUIRE(H > 0 && Hq % H == 0, "need at least one of window / selected rows, and Hq a multiple of H");
  PK_REQUIRE(n_window >= 0, "n_window must be non-negative");
  if (bs == 0) return PK_OK;
  const int64_t max_rows = n_window + K;
  const int64_t n_tiles = max_rows > 0 ? (max_rows + ATT_TILE - 1) / ATT_TILE : 1;
  PK_REQUIRE(n_tiles <= 1024, "too many rows for one call: %lld (limit 65536)", (long long)max_rows);
  if (!workspace || workspace_bytes < pk_attention_workspace_bytes(bs, Hq, max_rows))
    return fail(PK_ERR_WORKSPACE, "attention workspace too small: %lld < %lld", (long long)workspace_bytes,
                (long long)pk_attention_workspace_bytes(bs, Hq, max_rows));
  p.q = (const uint16_t*)queries->data;
  p.n_window = n_window;
  if (n_window_dev) {
    PK_CHECK_TENSOR(n_window_dev, PK_I32, 1);
    PK_REQUIRE(n_window_dev->shape[0] >= 1, "n_window_dev must hold one int32");
    p.n_window_dev = (const int32_t*)n_window_dev->data;
    p.n_window_add = n_window_add;
  }
  p.K = K, p.index_offset = index_offset;
  p.H = (int)H, p.Hq = (int)Hq, p.G = (int)(Hq / H);
  p.n_qgroups = (p.G + ATT_GQ - 1) / ATT_GQ;
  // Blocks per (batch, KV head): one per 128 rows when the whole launch is then a block per SM at most (every copy of the
  // launch outstanding at once), otherwise one per two tiles of 64 rows - a block copies two at once - but no more than
  // ONE wave of three blocks per SM, each streaming several tiles.  Before either the cluster form is tried (see head_tiles).
  // The scalar form needs the staged tile for several
  // passes: one tile per block then.
  const bool mma = p.G <= ATT_MQ;   // at most ATT_MQ query heads per KV head: one pass on the tensor cores
  const int64_t halves = (n_tiles + 1) / 2;
  const bool wide = mma && halves * H * bs <= sm_count();
  int64_t groups = n_tiles;
  p.tiles_per_block = 1;
  const int in_cluster = mma && (reinterpret_cast<uintptr_t>(out->data) & 7) == 0 ? head_tiles(halves, H * bs) : 0;   // (it stores four outputs at once)
  if (in_cluster) {
    p.tiles_per_block = in_cluster;
    groups = (halves + in_cluster - 1) / in_cluster;
  } else if (wide) {
    groups = halves;
  } else if (mma) {
    const int64_t fit = (int64_t)sm_count() * 3 / (H * bs);
    groups = fit < 1 ? 1 : (fit < halves ? fit : halves);
    p.tiles_per_block = (int)((n_tiles + groups - 1) / groups);
    groups = (n_tiles + p.tiles_per_block - 1) / p.tiles_per_block;
  }
  p.scale_log2 = scale * 1.4426950408889634f;
  PK_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & 15) == 0, "workspace must be 16-byte aligned");
  p.counters = (unsigned*)workspace;
  p.status = (int*)workspace + bs * Hq;
  p.ws = (float*)((char*)workspace + att_header_bytes(bs, Hq));
  p.out = (uint16_t*)out->data;
  if (lse) {
    PK_CHECK_TENSOR(lse, PK_F32, 2);
    PK_REQUIRE(is_contig(lse) && lse->shape[0] == bs && lse->shape[1] == Hq, "lse must be contiguous [bs,Hq]");
    p.lse = (float*)lse->data;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid((unsigned)groups, (unsigned)H, (unsigned)bs);
  if (in_cluster) return launch_head_attention(p, grid, st);
  if (wide) return launch_attention<true, 8>(p, grid, st);
  return mma ? launch_attention<true, 4>(p, grid, st) : launch_attention<false, 4>(p, grid, st);
}
