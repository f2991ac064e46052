// 4-bit RaBitQ rerank, stand-alone and fused with candidate selection.
//
// One thread per candidate.  With key-major storage a candidate is one 64-byte record of nibbles
// plus one 32-byte record of bf16 weights (three DRAM sectors); with the reference's plane-major
// storage it is 16 + 16 scattered words (correct, but 32 sectors).  The 16 signed magnitude levels sit
// in shared memory replicated once per lane (bank = lane), the query blocks are read as broadcasts.
// fp32 order (shared with the CPU oracle): per subspace dot = fma chain over j ascending,
// acc = fma(dot, w_b, acc) over b ascending, score = acc * ||q||.
#include "chain.cuh"
#include "common.cuh"
#include "kernels.cuh"

namespace pk {
namespace {

constexpr int RR_THREADS = 128;
constexpr int SEL_LIST_MAX = 16384;   // candidates of a block kept in shared memory

template <bool FAST>
__global__ void __launch_bounds__(RR_THREADS) rerank_kernel(RerankArgs a, uint16_t* scores_bf16, float* scores_f32,
                                                            uint16_t* v4b) {
  __shared__ RerankSmem sm;
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t bh = blockIdx.y;
  const int b = (int)(bh / a.H), h = (int)(bh % a.H);
  pdl_wait();
  pdl_trigger();
  rerank_setup(sm, a, bh, tid, RR_THREADS);
  __syncthreads();
  const float qn = bf2f(a.q_norm[bh]);
  const uint8_t* k4 = a.k4 + b * a.k4_b + h * a.k4_h;
  const uint16_t* w = a.w + b * a.w_b + h * a.w_h;
  for (int64_t c = (int64_t)blockIdx.x * RR_THREADS + tid; c < a.C; c += (int64_t)gridDim.x * RR_THREADS) {
    const int64_t key = a.cand[bh * a.C + c];
    uint16_t* vrow = v4b ? v4b + (bh * 16 * a.C + c) * 8 : nullptr;  // [bh][16][C][8]
    const float s = rerank_one<FAST>(sm, a, k4, w, key, qn, lane, vrow, a.C * 8);
    if (scores_bf16) scores_bf16[bh * a.C + c] = f2bf(s);
    if (scores_f32) scores_f32[bh * a.C + c] = s;
  }
}

// ---- candidate selection from u8 counts and rerank of the selected keys, one launch ----------------------------------
// One block per (chunk of keys, batch*head), one block per SM.  The histogram rows written by the collision kernel
// give every block the global threshold count, the tie quota and its own output offset, so the candidate
// list comes out in ascending key order with no atomics and no second pass.
// What bounds it at 8 heads x 1M keys, 33 us on B200: 4 for the threshold, 7 for the list (issue: some 190 instructions per 512
// counts and warp), 20 for the rerank, 840 K candidates of which HBM reads 128 bytes each: 5.4 TB/s.  (50 us with codes and
// weights in two arrays, 226 bytes a candidate, and the rerank through registers.)  With the final top-K by the last block of a
// head inside it (one SM per head) 8 heads x 1M keys took 129 us where this and the top-k launch now take 52.
struct SelParams {
  SelectArgs s;
  int list_cap;            // candidates whose keys fit in shared memory; the others are read back from cand_out
  unsigned c128;           // 128 (see rerank_record)
};

template <bool FAST>
__global__ void __launch_bounds__(CH_THREADS, 1) select_rerank_kernel(RerankArgs a, SelParams pp) {
  extern __shared__ __align__(16) unsigned char dyn[];
  const SelectArgs& p = pp.s;
  uint32_t* lev2 = reinterpret_cast<uint32_t*>(dyn);                  // FAST: pair levels; otherwise RerankSmem
  uint8_t* cnt8 = dyn + LEV2_BYTES;
  uint8_t* stage = cnt8 + (threadIdx.x >> 5) * CH_STAGE_WARP;        // the counts are done with when records are staged
  int* ids = reinterpret_cast<int*>(cnt8 + max((int)p.chunk_keys, CH_STAGE));
  __shared__ unsigned tot[2][CH_CBINS + 3], pre[2][CH_CBINS + 3];
  __shared__ unsigned s_warp[CH_WARPS], s_pwarp[CH_WARPS];
  __shared__ unsigned s_res[6];   // threshold, quota, keys above it before this block, ties before it, candidates of this shard
  __shared__ __align__(16) uint4 s_qb[16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t bh = blockIdx.y, chunk = blockIdx.x;
  const int b = (int)(bh / a.H), h = (int)(bh % a.H);
  if (FAST && p.early_loads) build_lev2(lev2, a.centers, tid, CH_THREADS);
  pdl_wait();  // counts, histograms and query blocks come from the collision kernel
  pdl_trigger();
  if (FAST && !p.early_loads) build_lev2(lev2, a.centers, tid, CH_THREADS);
  const int64_t N = p.n_dev ? min(max((int64_t)p.n_dev[b], (int64_t)1), p.N) : p.N;
  const int64_t Nv = N + p.mis;
  const int64_t chunk_keys = p.n_dev ? chain_chunk(Nv, p.n_chunks, p.chunk_keys) : p.chunk_keys;   // as the collision kernel has it
  const int64_t v_begin = chunk * chunk_keys;
  if (v_begin >= Nv) return;  // beyond this sample's zone (whole block, before any barrier)
  const int n_keys = (int)(min(Nv, v_begin + chunk_keys) - v_begin);
  const int64_t live_chunks = (Nv + chunk_keys - 1) / chunk_keys;
  // candidates wanted over the whole zone (all shards together)
  const int64_t C_want = p.n_dev ? min((int64_t)zone_candidates(p.sched, N), p.C) : p.C_want;
  // this block's counts, straight into shared memory, under the latency of the histogram rows
  {
    const uint8_t* src = p.counts_u8 + bh * p.u8_stride + v_begin;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(cnt8);
    for (int k = 16 * tid; k < n_keys; k += 16 * CH_THREADS)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + k), "l"(src + k) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (!FAST) {
    rerank_setup(*reinterpret_cast<RerankSmem*>(dyn), a, bh, tid, CH_THREADS);
  } else if (tid < 128) {
    reinterpret_cast<uint16_t*>(s_qb)[tid] = a.q_blocks[bh * 128 + tid];
  }
  // Bin totals over the rows: the block's two halves take alternate rows, eight loads in flight per thread.  Bins 0 .. 128
  // are the only ones: the halves' threads 0 .. 128.
  {
    const int bin = tid & 255, par = tid >> 8;
    if (bin < CH_CBINS) {
      const uint32_t* hp = p.chunk_hist + bh * p.n_chunks * 256 + bin;
      unsigned t = 0, pr = 0;
      for (int64_t c0 = par; c0 < live_chunks; c0 += 16) {
        unsigned v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = (c0 + 2 * i < live_chunks) ? __ldcg(hp + (c0 + 2 * i) * 256) : 0u;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          t += v[i];
          if (c0 + 2 * i < chunk) pr += v[i];
        }
      }
      tot[par][bin] = t, pre[par][bin] = pr;
    }
  }
  if (tid < 6) s_res[tid] = 0;
  __syncthreads();
  // threshold bin: suffix sums over the bins (thread t: bin t)
  unsigned mine = 0, mine_pre = 0, g_tot = 0, g_before = 0;   // this shard's bin; all shards' and the lower shards'
  if (tid < CH_CBINS) {
    mine = tot[0][tid] + tot[1][tid], mine_pre = pre[0][tid] + pre[1][tid];
    g_tot = mine;
    if (p.shard_hist) {
      g_tot = 0;
      const int64_t rows = (int64_t)gridDim.y;  // bs*H
      for (int r = 0; r < p.world; r++) {
        const unsigned v = p.shard_hist[((int64_t)r * rows + bh) * 256 + tid];
        g_tot += v;
        if (r < p.rank) g_before += v;
      }
    }
  }
  unsigned suf = g_tot, psuf = mine_pre, lsuf = mine;   // inclusive suffixes: all shards, before this block, this shard
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned o = __shfl_down_sync(0xffffffffu, suf, off), q = __shfl_down_sync(0xffffffffu, psuf, off),
                   l = __shfl_down_sync(0xffffffffu, lsuf, off);
    if (lane + off < 32) suf += o, psuf += q, lsuf += l;
  }
  if (warp < 5 && lane == 0) s_warp[warp] = suf, s_pwarp[warp] = psuf, s_warp[8 + warp] = lsuf;
  __syncthreads();
  if (tid < CH_CBINS) {
    for (int w = warp + 1; w < 5; w++) suf += s_warp[w], psuf += s_pwarp[w], lsuf += s_warp[8 + w];
    const unsigned above = suf - g_tot;
    if (g_tot && suf >= (unsigned)C_want && above < (unsigned)C_want) {
      // ties of the threshold count taken over the whole zone; a shard takes what the shards before it left
      const unsigned q_all = (unsigned)C_want - above, left = q_all > g_before ? q_all - g_before : 0u;
      const unsigned quota = p.shard_hist ? min(left, mine) : q_all;
      s_res[0] = (unsigned)tid, s_res[1] = quota;
      s_res[2] = psuf - mine_pre, s_res[3] = mine_pre;
      s_res[4] = (lsuf - mine) + min(mine, quota);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const unsigned T = s_res[0], quota = s_res[1], eq_base = s_res[3];
  const int64_t C_here = min((int64_t)s_res[4], p.C);   // candidates of this (batch, head) held by this shard
  const int64_t row_base = bh * p.C, out_pos = (int64_t)s_res[2] + min(eq_base, quota);
  const int64_t key0 = v_begin - p.mis;
  const int n_list = list_candidates(cnt8, n_keys, chunk == 0 ? p.mis : 0, T, quota, eq_base, C_here - out_pos, s_warp, s_pwarp, [&](int pos, int off) {
    p.cand_out[row_base + out_pos + pos] = key0 + off;
    if (pos < pp.list_cap) ids[pos] = (int)(key0 + off);
  });
  __syncthreads();
  auto key_at = [&](int i) -> int { return i < pp.list_cap ? ids[i] : (int)p.cand_out[row_base + out_pos + i]; };
  const float qn = bf2f(a.q_norm[bh]);
  const uint8_t* k4 = a.k4 + b * a.k4_b + h * a.k4_h;
  const uint16_t* w = a.w + b * a.w_b + h * a.w_h;
  float* scores = p.scores_f32 + row_base + out_pos;
  if (FAST) {
    rerank_list(n_list, ids, pp.list_cap, a, k4, w, stage, lev2, s_qb, qn, pp.c128, key_at, [&](int i, int, float v) { scores[i] = v; }, []() {});
  } else {
    for (int i = tid; i < n_list; i += CH_THREADS)
      scores[i] = rerank_one<false>(*reinterpret_cast<RerankSmem*>(dyn), a, k4, w, key_at(i), qn, lane, nullptr, 0);
  }
  if (chunk == 0) {
    if (tid == 0) p.n_cand_out[bh] = (int32_t)C_here;
    // per-sample lengths: rows are longer than this candidate list; the tail gets (score -inf, key 0), so
    // a consumer that walks whole rows (the adaptive selection) gives those entries no weight
    if (p.fill_tail)
      for (int64_t i = C_here + tid; i < p.C; i += CH_THREADS) {
        p.scores_f32[row_base + i] = -INFINITY;
        p.cand_out[row_base + i] = 0;
      }
  }
}

}  // namespace

bool rerank_fast_layout(const RerankArgs& a) {
  return a.k4_s == 4 && a.k4_l >= 0 && a.k4_l < (1 << 30) && a.k4_l % 16 == 0 && a.w_s == 1 && a.w_l >= 0 && a.w_l < (1 << 30) && a.w_l % 8 == 0 && (reinterpret_cast<uintptr_t>(a.k4) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(a.w) & 15) == 0 && a.k4_b % 16 == 0 && a.k4_h % 16 == 0 && a.w_b % 8 == 0 &&
         a.w_h % 8 == 0;
}

int fill_rerank_args(RerankArgs* a, const pk_tensor* key_4bit, const pk_tensor* key_block_weight) {
  PK_CHECK_TENSOR(key_4bit, PK_U8, 5);
  PK_CHECK_TENSOR(key_block_weight, PK_BF16, 4);
  PK_REQUIRE(key_4bit->shape[2] == 16 && key_4bit->shape[4] == 4 && key_4bit->stride[4] == 1,
             "key_4bit must be [bs,H,16,N,4] with last stride 1");
  PK_REQUIRE(key_block_weight->shape[2] == 16 && key_block_weight->shape[0] == key_4bit->shape[0] &&
                 key_block_weight->shape[1] == key_4bit->shape[1] && key_block_weight->shape[3] == key_4bit->shape[3],
             "key_block_weight must be [bs,H,16,N]");
  a->k4 = (const uint8_t*)key_4bit->data;
  a->k4_b = key_4bit->stride[0], a->k4_h = key_4bit->stride[1], a->k4_s = key_4bit->stride[2], a->k4_l = key_4bit->stride[3];
  a->w = (const uint16_t*)key_block_weight->data;
  a->w_b = key_block_weight->stride[0], a->w_h = key_block_weight->stride[1], a->w_s = key_block_weight->stride[2],
  a->w_l = key_block_weight->stride[3];
  a->H = (int)key_4bit->shape[1];
  return PK_OK;
}

int launch_rerank(const RerankArgs& a, int64_t bs_h, uint16_t* scores_bf16, float* scores_f32, uint16_t* v4b,
                  cudaStream_t st) {
  int64_t gx = (a.C + RR_THREADS - 1) / RR_THREADS;
  dim3 grid((unsigned)gx, (unsigned)bs_h);
  StageTimer tm(ST_RERANK, st);
  if (rerank_fast_layout(a))
    launch_chain(rerank_kernel<true>, grid, dim3(RR_THREADS), 0, st, a, scores_bf16, scores_f32, v4b);
  else
    launch_chain(rerank_kernel<false>, grid, dim3(RR_THREADS), 0, st, a, scores_bf16, scores_f32, v4b);
  return check_launch("rerank");
}

int launch_select_rerank(const RerankArgs& a, int64_t bs_h, const SelectArgs& sa, cudaStream_t st) {
  SelParams p;
  p.s = sa;
  p.c128 = 128;
  if (sa.C >= (1ll << 31) || sa.N >= (1ll << 31)) return fail(PK_ERR_ARG, "zone too long for the selection kernel");
  const int64_t body = sa.chunk_keys > CH_STAGE ? sa.chunk_keys : CH_STAGE;
  int64_t list = ((sa.C < sa.chunk_keys ? sa.C : sa.chunk_keys) + 31) / 32 * 32;
  if (list > SEL_LIST_MAX) list = SEL_LIST_MAX;
  p.list_cap = (int)list;
  const int smem = (int)(LEV2_BYTES + body + 4 * list);
  constexpr int smem_max = LEV2_BYTES + (CHAIN_CHUNK_MAX > CH_STAGE ? (int)CHAIN_CHUNK_MAX : CH_STAGE) + 4 * SEL_LIST_MAX;
  const bool fast = rerank_fast_layout(a);
  static PerDevice smem_attr;
  if (const unsigned long long bit = first_on_device(smem_attr)) {
    if (cudaFuncSetAttribute(select_rerank_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max) != cudaSuccess ||
        cudaFuncSetAttribute(select_rerank_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max) != cudaSuccess)
      return check_launch("select_rerank smem");
    mark_on_device(smem_attr, bit);
  }
  dim3 grid((unsigned)sa.n_chunks, (unsigned)bs_h);
  StageTimer tm(ST_SELECT_RERANK, st);
  if (fast) launch_chain(select_rerank_kernel<true>, grid, dim3(CH_THREADS), (size_t)smem, st, a, p);
  else launch_chain(select_rerank_kernel<false>, grid, dim3(CH_THREADS), (size_t)smem, st, a, p);
  return check_launch("select_rerank");
}

}  // namespace pk

using namespace pk;

extern "C" int pk_rerank(const pk_tensor* coarse_indices, const pk_tensor* key_4bit,
                         const pk_tensor* key_block_weight, const pk_tensor* q_blocks, const pk_tensor* q_norm,
                         const pk_tensor* mag_centers, const pk_tensor* approx_scores, const pk_tensor* scores_f32,
                         const pk_tensor* v4b, void* stream) {
  PK_CHECK_TENSOR(coarse_indices, PK_I64, 3);
  PK_CHECK_TENSOR(q_blocks, PK_BF16, 4);
  PK_CHECK_TENSOR(q_norm, PK_BF16, 3);
  PK_CHECK_TENSOR(mag_centers, PK_BF16, 1);
  RerankArgs a;
  int rc = fill_rerank_args(&a, key_4bit, key_block_weight);
  if (rc) return rc;
  const int64_t bs = key_4bit->shape[0], H = key_4bit->shape[1], C = coarse_indices->shape[2];
  PK_REQUIRE(is_contig(coarse_indices) && coarse_indices->shape[0] == bs && coarse_indices->shape[1] == H,
             "coarse_indices must be contiguous [bs,H,C]");
  PK_REQUIRE(is_contig(q_blocks) && q_blocks->shape[0] == bs && q_blocks->shape[1] == H && q_blocks->shape[2] == 16 &&
                 q_blocks->shape[3] == 8,
             "q_blocks must be contiguous [bs,H,16,8] (only B == 16, m == 8 is supported)");
  PK_REQUIRE(is_contig(q_norm) && numel(q_norm) == bs * H, "q_norm must be contiguous [bs,H,1]");
  PK_REQUIRE(mag_centers->shape[0] == 8 && mag_centers->stride[0] == 1, "mag_centers must be [8]");
  uint16_t* sbf = nullptr;
  float* s32 = nullptr;
  uint16_t* v = nullptr;
  if (approx_scores) {
    PK_CHECK_TENSOR(approx_scores, PK_BF16, 3);
    PK_REQUIRE(is_contig(approx_scores) && approx_scores->shape[0] == bs && approx_scores->shape[1] == H &&
                   approx_scores->shape[2] == C,
               "approx_scores must be contiguous [bs,H,C]");
    sbf = (uint16_t*)approx_scores->data;
  }
  if (scores_f32) {
    PK_CHECK_TENSOR(scores_f32, PK_F32, 3);
    PK_REQUIRE(is_contig(scores_f32) && scores_f32->shape[0] == bs && scores_f32->shape[1] == H &&
                   scores_f32->shape[2] == C,
               "scores_f32 must be contiguous [bs,H,C]");
    s32 = (float*)scores_f32->data;
  }
  if (v4b) {
    PK_CHECK_TENSOR(v4b, PK_BF16, 5);
    PK_REQUIRE(is_contig(v4b) && v4b->shape[0] == bs && v4b->shape[1] == H && v4b->shape[2] == 16 &&
                   v4b->shape[3] == C && v4b->shape[4] == 8 && (reinterpret_cast<uintptr_t>(v4b->data) & 15) == 0,
               "v4b must be contiguous [bs,H,16,C,8]");
    v = (uint16_t*)v4b->data;
  }
  PK_REQUIRE(sbf || s32, "at least one of approx_scores / scores_f32 is required");
  if (bs * H * C == 0) return PK_OK;
  a.cand = (const int64_t*)coarse_indices->data;
  a.q_blocks = (const uint16_t*)q_blocks->data;
  a.q_norm = (const uint16_t*)q_norm->data;
  a.centers = (const uint16_t*)mag_centers->data;
  a.C = C;
  return launch_rerank(a, bs * H, sbf, s32, v, (cudaStream_t)stream);
}

