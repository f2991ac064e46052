// The retrieval chain of one decode step as ONE launch: a thread-block cluster per (batch, KV head) takes the query to
// the final top-K without leaving the chip.
//
// Every CTA of the cluster owns a contiguous slice of the zone's keys.  It prepares the query and the tier tables itself
// (behind its first code loads), counts the collisions of its keys into shared memory, and from there on only histograms
// and a few hundred scores cross the cluster (distributed shared memory):
//   count histogram  -> threshold count, tie quota, this CTA's offset in the candidate list
//   4-bit rerank of its own candidates, scores in shared memory
//   final top-K over the cluster (cluster_select.cuh).
//
// Why this split: as two launches (count | select + rerank + final top-K by the last block of a head) the final stage ran
// on one SM per head, 12 us of 48 at 128K keys, and counts and scores went through L2.  Time line of a CTA on B200
// (8 heads x 131004 keys, 10 CTAs each; query and ranking, 2.4 us, before the wait): tables 1.9 us, counting 13 K keys 6.8, threshold
// 1.5, list 2.2, rerank of 1310 candidates 5.9, final selection 6.7: 25 behind the wait.  Graph-replayed layer step, two launches -> one: 16
// sequences of 16 - 32K keys (one CTA per head, no exchange at all) 155 -> 116 us, 8 heads x 128K keys 70 -> 60, 10K keys 27 -> 19
// for the chain.
// What bounds it: the serial chain of exchanges for small zones; for long ones instruction issue in the counting (85
// instructions per 32 keys, 28 cycles of an SM) and, with every SM at it, HBM in the rerank (16 sequences: 80 MB in 15 us).
#include "chain.cuh"
#include "cluster_select.cuh"
#include "common.cuh"
#include "kernels.cuh"

namespace pk {
namespace {

static_assert(CH_THREADS == SEL_THREADS, "one block shape");
constexpr int FR_LIST_MAX = 8192;           // candidates a CTA keeps in shared memory; more spill to the workspace
constexpr int FR_SPAN_MAX = 40 * 1024;      // keys of a CTA: beyond it three launches over all SMs are faster
constexpr int FR_WORDS = LEV2_BYTES / 8;    // ballots of the final selection, over the level table
static_assert(FR_SPAN_MAX / 32 <= FR_WORDS && FR_SPAN_MAX < 65536, "one ballot per 32 candidates, 16 bits for a bin's count");
static_assert(CH_HIST_BYTES >= SEL_REGION && CH_STAGE >= 16 * 256 * 4, "areas that serve two stages");

struct FusedParams {
  const uint8_t* codes;   // key-major records of 16 bytes; (b,h) at b*c_b + h*c_h
  int64_t c_b, c_h;
  RerankArgs a;
  ChainQuery q;
  int H, G;
  float inv_g;
  int64_t N;              // keys per head of the view (upper bound when q.n_dev is set)
  int64_t C, C_want, K;   // row stride of the candidate arrays, candidates wanted (q.n_dev == null), final top-K
  int fill_tail;
  int span_cap, list_cap; // shared memory: keys and candidates per CTA
  int64_t* cand_out;      // [bs*H][C] or null
  float* scores_out;      // [bs*H][C] or null
  unsigned c128, c256;    // 128 and 256 (see tier_sum16, rerank_record)
  int64_t* ws_cand;       // the same arrays for what does not fit in shared memory (never null)
  float* ws_scores;
  int64_t* final_out;     // [bs*H][K]
  int32_t* n_sel_out;
  int32_t* n_cand_out;
};

template <int CS>
__global__ void __launch_bounds__(CH_THREADS, 1) retrieve_fused_kernel(FusedParams p) {
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ SelShared s;
  __shared__ unsigned s_tiers[9];
  __shared__ float s_qnorm;
  __shared__ __align__(16) float s_q[128];        // rotated query
  __shared__ __align__(16) uint4 s_qb[16];        // the same, its bf16 values as such
  __shared__ __align__(16) uint8_t s_lut[16 * 128];
  unsigned* region = reinterpret_cast<unsigned*>(dyn);
  unsigned* inbox = reinterpret_cast<unsigned*>(dyn + CH_HIST_BYTES);
  uint32_t* lev2 = reinterpret_cast<uint32_t*>(dyn + CH_HIST_BYTES + sel_inbox_bytes(CS));
  uint8_t* cnt8 = dyn + CH_HIST_BYTES + sel_inbox_bytes(CS) + LEV2_BYTES;
  uint8_t* stage = cnt8 + (threadIdx.x >> 5) * CH_STAGE_WARP;   // the counts are done with when records are staged
  int* ids = reinterpret_cast<int*>(cnt8 + max(p.span_cap, CH_STAGE));
  float* sc = reinterpret_cast<float*>(ids + p.list_cap);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned rank = CS == 1 ? 0u : cluster.block_rank();
  const int64_t bh = blockIdx.y;
  const int b = (int)(bh / p.H), h = (int)(bh % p.H);
  const ChainQuery& cq = p.q;
  PreparedQuery pq;
  QueryLoads ql;
  unsigned key[4];
  for (int i = tid; i < CH_CBINS * 32; i += CH_THREADS) region[i] = 0;
  const bool early = cq.early_query != 0;
  // the level table is left to the warps that do not prepare the query
  if (cq.early_loads) build_lev2(lev2, p.a.centers, tid - 32, CH_THREADS - 32);
  if (CS > 1) cluster.barrier_arrive();   // a CTA has to run before the others may write into it
  // Both orders (queries before the wait or behind it) run through one copy of the preparation and the ranking: a CTA fetches its
  // code as it goes, and with two copies of them and longer unrolls in the selection a step with 128K keys took 195.8 us against
  // 191.9, one KV head of eight sequences 170.7 against 167.4.
  if (!early) {
    pdl_wait();
    pdl_trigger();
  }
  load_query(ql, cq, b, h, p.G);
  // A word written by the kernel before this one takes over a microsecond to arrive: the cluster sizes, the zone length and
  // (where they may not be read earlier) the queries are asked for together.  Then the code loads: a warp takes 128
  // consecutive keys (four per lane) every CH_WARPS * 128; two rounds are in flight, the first ones during the prologue.
  int4 c0, c1;   // cluster sizes of this warp's subspace
  int64_t N, begin;
  int n_keys;
  const uint8_t* codes;
  uint4 r0[4], r1[4];
  constexpr int STEP = CH_WARPS * 128;
  auto load_codes = [&](uint4 (&r)[4], int v0) {
    if (n_keys > 0)
#pragma unroll
      for (int j = 0; j < 4; j++)   // past the end: the last key again, its count unused
        r[j] = reinterpret_cast<const uint4*>(codes)[min(v0 + 32 * j, n_keys - 1)];
  };
  // In a large cluster a CTA makes the tables of its share of the subspaces only, a warp each, and writes them into all CTAs:
  // sixteen warps at the tier counts are bound by the integer ALU, and the exchange costs less than that (sort and tables of 10K
  // keys on 10 CTAs 3.6 -> 2.7 us; on one or two CTAs there is nothing to gain).  The chain alone in a graph, every CTA all tables |
  // shared: 16 heads of 12K keys, six CTAs each, 15.3 | 14.5, 32 heads, four each, 16.1 | 15.3, 24 heads of 40K 21.8 | 21.3.  With the
  // level table left to the warps that do not prepare the query, a histogram that four threads a bin add up, and 512 bins in the
  // selection: 8 heads of 10K keys 15.4 -> 14.0, of 131K 29.4 -> 28.4, eight sequences of one head of 65K 21.7 -> 20.5, 128 heads of
  // 33K 49.0 -> 48.2.  All pairs of clusters compared by all threads instead of the sort took longer: reads of shared memory.
  constexpr bool SHARED_TABLES = CS >= 4;
  const int sub = SHARED_TABLES ? (int)rank + CS * warp : warp;
  const bool ranks = sub < 16;
  auto load_zone = [&]() {
    if (ranks) {
      const int4* sizes = reinterpret_cast<const int4*>(cq.counts + ((int64_t)bh * 16 + sub) * 256 + lane * 8);
      c0 = sizes[0], c1 = sizes[1];
    }
    N = cq.n_dev ? min(max((int64_t)cq.n_dev[b], (int64_t)1), p.N) : p.N;
    const int span = (int)(((N + CS - 1) / CS + 15) / 16 * 16);
    begin = (int64_t)rank * span;
    n_keys = (int)max((int64_t)0, min((int64_t)span, N - begin));
    codes = p.codes + b * p.c_b + h * p.c_h + begin * 16;
    load_codes(r0, warp * 128 + lane);
    load_codes(r1, warp * 128 + lane + STEP);
  };
  if (!early) load_zone();
  prepare_query(pq, ql, cq, b, h, p.G, p.inv_g, s_q, &s_qnorm);
  if (!cq.early_loads) build_lev2(lev2, p.a.centers, tid - 32, CH_THREADS - 32);
  __syncthreads();
  if (ranks) rank_subspace(key, s_q + sub * 8, lane);
  if (early) {   // the queries were complete before the kernel before this one started
    pdl_wait();
    pdl_trigger();
    load_zone();
  }
  const int64_t C_want = cq.n_dev ? min((int64_t)zone_candidates(cq.sched, N), p.C) : p.C_want;
  {
    if (warp == 0 && rank == 0) publish_query(pq, cq, bh);
    if (tid >= CH_THREADS - 32 && tid < CH_THREADS - 23) load_tiers(cq, (long long)N, s_tiers, tid - (CH_THREADS - 32));
    if (tid < 128) reinterpret_cast<uint16_t*>(s_qb)[tid] = f2bf(s_q[tid]);
    unsigned* my = reinterpret_cast<unsigned*>(cnt8) + warp * 256;   // the counts are not there yet
    if (ranks) {
      *reinterpret_cast<int4*>(my + lane * 8) = c0;
      *reinterpret_cast<int4*>(my + lane * 8 + 4) = c1;
    }
    __syncthreads();
    uint32_t table = 0;
    if (ranks) table = tier_table(key, my, s_tiers);
    uint32_t* at = reinterpret_cast<uint32_t*>(s_lut + sub * 128) + lane;
    if (SHARED_TABLES) {
      cluster.barrier_wait();
      if (ranks) put_everywhere<CS>(cluster, at, table);
      cluster.sync();
    } else {
      *at = table;
      __syncthreads();   // the tables are complete, the sizes are done with
    }
  }
  const float qn = s_qnorm;

  // ---- collision counts of this CTA's keys ----
  auto count_round = [&](uint4 (&r)[4], int v0) {   // counts four keys and puts the loads of the round after next in their place
    unsigned c[4];
#pragma unroll
    for (int j = 0; j < 4; j++) c[j] = tier_sum16(r[j], s_lut, p.c256);
    load_codes(r, v0 + 2 * STEP);
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (v0 + 32 * j < n_keys) {
        cnt8[v0 + 32 * j] = (uint8_t)(c[j] >> 4);
        atomicAdd(&region[c[j] * 2 + lane], 1u);   // c is a multiple of 16: word 32 per bin
      }
  };
#pragma unroll 1
  for (int v0 = warp * 128 + lane; v0 - lane < n_keys; v0 += 2 * STEP) {
    count_round(r0, v0);
    if (v0 - lane + STEP < n_keys) count_round(r1, v0 + STEP);
  }
  if (CS > 1 && !SHARED_TABLES) cluster.barrier_wait();
  __syncthreads();
  {   // bin totals into the inboxes of all CTAs: four threads a bin, each with eight replicas (in turns, so that banks differ)
    const int bin = tid >> 2, q = tid & 3;
    unsigned t = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) t += region[bin * 32 + q * 8 + ((i + bin) & 7)];
    t += __shfl_xor_sync(0xffffffffu, t, 1);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    static_assert(CH_CBINS == CH_THREADS / 4 + 1, "four threads a bin, and the last bin");
    unsigned last = 0;
    if (warp == 0) last = __reduce_add_sync(0xffffffffu, region[(CH_CBINS - 1) * 32 + lane]);
#pragma unroll
    for (int r = 0; r < CS; r += 4)
      if (r + q < CS) {
        unsigned* at = inbox + rank * SEL_WORDS;
        if (CS > 1) at = cluster.map_shared_rank(at, r + q);
        at[bin] = t;
        if (tid < 4) at[CH_CBINS - 1] = last;
      }
  }
  sync_cluster<CS>(cluster);
  cluster_threshold<CS, CH_CBINS>(s, inbox, rank, (unsigned)C_want);
  const unsigned T = s.res[0], quota = (unsigned)C_want - s.res[1];
  const unsigned gt_base = s.res[3], eq_base = s.res[4];
  const int64_t C_here = min(C_want, p.C);

  // ---- ordered candidate list of this CTA: counts above T, and ties at T while the quota lasts ----
  const int64_t row_base = bh * p.C;
  const int64_t out_pos = (int64_t)gt_base + min(eq_base, quota);
  const int n_list = list_candidates(cnt8, n_keys, 0, T, quota, eq_base, C_here - out_pos, s.warp_a, s.warp_b, [&](int pos, int off) {
    if (pos < p.list_cap) ids[pos] = (int)begin + off;
    else p.ws_cand[row_base + out_pos + pos] = begin + off;
  });
  __syncthreads();

  // ---- rerank ----
  auto id_at = [&](int i) -> int { return i < p.list_cap ? ids[i] : (int)p.ws_cand[row_base + out_pos + i]; };
  auto score_at = [&](int i) -> float { return i < p.list_cap ? sc[i] : p.ws_scores[row_base + out_pos + i]; };
  unsigned kmin = 0xffffffffu, kmax = 0u;
  // The bins of the final selection lie between the extremes of the scores of every warp's first round, so that their exchange
  // passes under the other rounds.
  bool published = p.K <= 0;
  auto publish = [&]() {
    if (published) return;
    published = true;
    publish_range<CS, CH_WARPS>(cluster, inbox, rank, kmin, kmax);
    if (CS > 1) cluster.barrier_arrive();
  };
  {
    const uint8_t* k4 = p.a.k4 + b * p.a.k4_b + h * p.a.k4_h;
    const uint16_t* w = p.a.w + b * p.a.w_b + h * p.a.w_h;
    rerank_list(n_list, ids, p.list_cap, p.a, k4, w, stage, lev2, s_qb, qn, p.c128, id_at, [&](int i, int k, float v) {
      const int64_t at = row_base + out_pos + i;
      if (i < p.list_cap) sc[i] = v;
      else p.ws_scores[at] = v;
      if (p.scores_out) p.scores_out[at] = v;
      if (p.cand_out) p.cand_out[at] = k;
      const unsigned u = ord_key(v);
      kmin = min(kmin, u), kmax = max(kmax, u);
    }, publish);
    publish();   // warps without candidates
    if (p.fill_tail && p.scores_out && p.cand_out)
      for (int64_t i = C_here + (int64_t)rank * CH_THREADS + tid; i < p.C; i += CS * CH_THREADS) {
        p.scores_out[row_base + i] = -INFINITY;
        p.cand_out[row_base + i] = 0;
      }
  }
  const int K_here = (int)min(p.K, C_here);
  if (rank == 0 && tid == 0) {
    if (p.n_cand_out) p.n_cand_out[bh] = (int32_t)C_here;
    if (p.n_sel_out && p.K > 0) p.n_sel_out[bh] = K_here;
  }
  if (p.K <= 0) return;

  // ---- final top-K over the cluster ----
  __syncthreads();   // the scores are complete; the level table and the histogram region are free
  cluster_select<CS, F32Row<512>, false, CH_THREADS>(
      cluster, s, region, inbox, lev2, FR_WORDS, rank, n_list, K_here, p.final_out + bh * p.K,
      [&](int i) -> uint32_t { return __float_as_uint(score_at(i)); }, [&](int i) -> int64_t { return id_at(i); }, kmin, kmax, true);
}

// Clusters that fit the device at once, per size in CLUSTER_SIZES (0: the size cannot be launched).
struct Capacity {
  int active[N_CLUSTER_SIZES];
};

template <int CS>
int active_clusters() {
  auto kern = retrieve_fused_kernel<CS>;
  const int smem = CH_HIST_BYTES + sel_inbox_bytes(CS) + LEV2_BYTES + (FR_SPAN_MAX > CH_STAGE ? FR_SPAN_MAX : CH_STAGE) + 8 * FR_LIST_MAX;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return cudaGetLastError(), 0;
  if (CS > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return cudaGetLastError(), 0;
  if (CS == 1) return sm_count();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CS, 64), cfg.blockDim = dim3(CH_THREADS), cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) return cudaGetLastError(), 0;
  return n;
}

// Asked once per device: the answers and the shared-memory opt-ins belong to it.
const Capacity* capacity() {
  static Capacity cap[64];
  static PerDevice asked;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (const unsigned long long bit = first_on_device(asked)) {
    for (int i = 0; i < N_CLUSTER_SIZES; i++)   // several threads may ask at the same time: they write the same numbers
      with_cluster_size(CLUSTER_SIZES[i], [&](auto cs) { cap[dev].active[i] = active_clusters<cs.value>(); });
    mark_on_device(asked, bit);
  }
  return &cap[dev];
}

int span_of(int64_t N, int cs) { return (int)(((N + cs - 1) / cs + 15) / 16 * 16); }

template <int CS>
cudaError_t launch_cs(dim3 grid, size_t smem, cudaStream_t st, const FusedParams& p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid, cfg.blockDim = dim3(CH_THREADS), cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (CS > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = CS, attr[n].val.clusterDim.y = 1, attr[n].val.clusterDim.z = 1;
    n++;
  }
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    n++;
  }
  cfg.attrs = attr, cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, retrieve_fused_kernel<CS>, p);
}

}  // namespace

// CTAs per (batch, head), or 0 where the fused kernel does not apply (the codebook must be key-major, and a CTA's slice of the
// zone at most FR_SPAN_MAX keys) or the several-launch form is faster.
// Both forms are a fixed time and a share of the work; fitted on B200 to 1 .. 128 heads of 8 .. 400 K keys with 5 and 10 % of
// candidates.  This one: waves x (16 us + 0.66 ns a key and 3.9 a candidate of a CTA's slice); without the final top-K 11 us,
// 0.59 and 2.8.  The other: 22 us + 0.74 ns a key and 1.6 a candidate of an SM's share + 2.8 a candidate of a CTA's slice in the
// top-k launch; without it 13 us.  It uses all SMs, so it wins where a cluster would leave most of them idle (one head) or the
// heads are more than one wave.  (Fitted before the tables were shared and the top-k had 1024 threads; both forms have become up to 2 us
// faster since, and the rule takes the faster one at all of these but for the margin.)  us measured with the present kernels, alone in a
// graph, 10 % of candidates, this form | the other: 8 heads of 10K keys 14.0 | 19.1, of 131K 28.4 | 30.7, of 200K 36.8 | 38.6, of
// 400K 57.4 | 54.7; one head of 131K 22.7 | 23.4, of 400K 41.7 | 28.9; 16 heads of 262K 85.2 | 61.6; 128 heads of 33K 48.3 | 63.3;
// without top-K 8 heads of 66K 15.5 | 16.1, of 131K 22.7 | 20.1, one head of 400K 34.6 | 18.3.  The other form has to win by 8 us
// of a full zone: its further launches cost a program that calls eagerly, and is bound by its host, up to 5 (one layer of two heads,
// adaptive budget, 91K keys 77.3 us a step with this form, 81.5 with the other), and a zone that is nearly empty 4 on the device.
// A captured call has no such host time and pays the margin all the same: 8 heads of 400K keys take the 57.4 us.
int fused_cluster_size(const pk_tensor* codebook, const RerankArgs& a, int64_t bs_h, int64_t N, int64_t C, int64_t K) {
  int layout = 0;
  chain_layout(codebook, &layout);
  if (layout != 1 || !rerank_fast_layout(a) || N >= (1ll << 30) || bs_h > 65535) return 0;
  const Capacity* cap = capacity();
  if (!cap) return 0;
  int best = 0, whole = 1;   // whole: the largest cluster that is resident for every head at once
  double best_us = 0.0;
  const double fixed = K > 0 ? 16.0 : 11.0, work = (K > 0 ? 0.00066 : 0.00059) * (double)N + (K > 0 ? 0.0039 : 0.0028) * (double)C;
  for (int i = 0; i < N_CLUSTER_SIZES; i++) {
    const int cs = CLUSTER_SIZES[i];
    if (bs_h <= cap->active[i]) whole = cs;
    if (cap->active[i] <= 0 || span_of(N, cs) > FR_SPAN_MAX) continue;
    const double waves = (double)((bs_h + cap->active[i] - 1) / cap->active[i]);
    const double us = waves * (fixed + work / cs);
    if (!best || us < 0.98 * best_us) best = cs, best_us = us;
  }
  const double spread = (0.00074 * (double)N + 0.0016 * (double)C) * (double)bs_h / sm_count();
  const double other = K > 0 ? 22.0 + spread + 0.0028 * (double)C / whole : 13.0 + spread;
  return !best || other + 8.0 < best_us ? 0 : best;
}

int launch_fused_retrieve(int cs, const pk_tensor* codebook, const RerankArgs& a, const ChainQuery& cq, const SelectArgs& sa,
                          int64_t* cand_out, float* scores_out, int64_t* ws_cand, float* ws_scores, cudaStream_t st) {
  const int64_t bs = codebook->shape[0], H = codebook->shape[1];
  FusedParams p = {};
  p.codes = (const uint8_t*)codebook->data, p.c_b = codebook->stride[0], p.c_h = codebook->stride[1];
  p.a = a, p.q = cq, p.H = (int)H, p.G = cq.Hq / (int)H, p.inv_g = 1.0f / (float)p.G;
  p.N = sa.N, p.C = sa.C, p.C_want = sa.C_want, p.K = sa.K, p.fill_tail = sa.fill_tail;
  p.c128 = 128, p.c256 = 256;
  p.cand_out = cand_out, p.scores_out = scores_out, p.ws_cand = ws_cand, p.ws_scores = ws_scores;
  p.final_out = sa.final_out, p.n_sel_out = sa.n_sel_out, p.n_cand_out = sa.n_cand_out;
  p.span_cap = span_of(sa.N, cs);
  // twice an even share of the candidates: slices differ, and what does not fit goes through the workspace
  int64_t list = (2 * sa.C / cs + 512 + 31) / 32 * 32;
  if (list > p.span_cap + 32) list = (p.span_cap + 63) / 32 * 32;
  p.list_cap = (int)(list < FR_LIST_MAX ? list : FR_LIST_MAX);
  const size_t smem = (size_t)CH_HIST_BYTES + sel_inbox_bytes(cs) + LEV2_BYTES + (p.span_cap > CH_STAGE ? p.span_cap : CH_STAGE) + 8 * (size_t)p.list_cap;
  const dim3 grid((unsigned)cs, (unsigned)(bs * H));
  StageTimer tm(ST_RETRIEVE, st);
  cudaError_t e = cudaErrorInvalidValue;
  with_cluster_size(cs, [&](auto c) { e = launch_cs<c.value>(grid, smem, st, p); });
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(PK_ERR_CUDA, "retrieve: %s", cudaGetErrorString(e));
  }
  return check_launch("retrieve");
}

}  // namespace pk
