// Launchers shared between translation units of the pariskv_b200 library (host side only).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/pariskv_b200.h"

namespace pk {

// encode.cu
int launch_query_prep(const uint16_t* queries, int bs, int Hq, int H, const uint16_t* signs,
                      uint16_t* q_blocks, uint16_t* q_norm, uint16_t* query_avg, cudaStream_t st);

// ---- zone plan: tier thresholds and candidate count as functions of the zone length ------------------------------
// Same arithmetic on the host and on the device (IEEE double products, left to right, then ceil), which is what the
// reference's Python computes: int(math.ceil(N * collision_ratio * r)) and max(1, ceil(N * candidate_ratio))
// (cache_hub/polar_cache.py:1221-1222, :1239-1240) with the ratios picked by zone length (:1113-1124).
__host__ __device__ inline int zone_row(const pk_zone_schedule& s, long long N) {
  int row = s.n_rows - 1;
  for (int i = s.n_rows - 2; i >= 0; i--)
    if (N < s.bound[i]) row = i;
  return row;
}
__host__ __device__ inline unsigned zone_tier(const pk_zone_schedule& s, long long N, int t) {
  double x = ceil((double)N * s.collision_ratio[zone_row(s, N)] * s.tier_ratio[t]);
  if (!(x > 0.0)) x = 0.0;
  if (x > 4294967295.0) x = 4294967295.0;
  return (unsigned)x;
}
__host__ __device__ inline long long zone_candidates(const pk_zone_schedule& s, long long N) {
  const double x = ceil((double)N * s.candidate_ratio[zone_row(s, N)]);
  const long long c = (long long)x;
  return c < 1 ? 1 : (c > N ? N : c);
}

// collision.cu
int64_t collision_chunk_keys(int64_t bs_h, int64_t Nv);

// The query side of the fused chain: the collision kernel prepares the query, ranks the clusters of every subspace
// and builds the tier table itself, in every block, while its first code loads are in flight.
struct ChainQuery {
  const uint16_t* queries;    // [bs][Hq][128]
  const uint16_t* signs;      // [128]
  int Hq;
  uint16_t* q_blocks;         // [bs*H][128]  written by the first block of every (batch, head)
  uint16_t* q_norm;           // [bs*H]
  uint16_t* query_avg;        // [bs*H][128] or null
  const int32_t* counts;      // [bs*H][16][256] cluster histogram
  unsigned tiers[8];          // thresholds when n_dev == null
  int n_tiers;
  const int32_t* n_dev;       // [bs] searchable keys per sample (device), or null: all N keys of the view
  pk_zone_schedule sched;     // thresholds = zone_tier(sched, n_dev[b], t) when n_dev is set
  int early_query;            // the queries were complete before the previous kernel on the stream started
  int early_loads;            // see pdl_early()
};
int launch_collision(const pk_tensor* codebook, const uint32_t* lut, int32_t* out_i32, cudaStream_t st);
int chain_layout(const pk_tensor* codebook, int* layout);
constexpr int64_t CHAIN_CHUNK_MAX = 64 * 1024;   // keys per block of the several-launch chain
void chain_geometry(int64_t bs_h, int64_t Nv, int64_t* chunk_keys, int64_t* n_hist);
constexpr int64_t CHAIN_CHUNK_MIN = 2048;        // every block of the selection reads the histogram rows of its whole head
// Keys per block for a zone of Nv keys: the launch has blocks for the capacity of the zone; where the length comes from the
// device, what the zone holds is spread over all of them.
__host__ __device__ inline int64_t chain_chunk(int64_t Nv, int64_t n_blocks, int64_t at_most) {
  const int64_t even = ((Nv + n_blocks - 1) / n_blocks + 511) / 512 * 512;
  const int64_t c = even < CHAIN_CHUNK_MIN ? CHAIN_CHUNK_MIN : even;
  return c < at_most ? c : at_most;
}
int launch_chain_collision(const pk_tensor* codebook, const ChainQuery& cq, uint8_t* counts_u8, int64_t u8_stride,
                           uint32_t* chunk_hist, int* mis_out, int64_t* chunk_keys_out, int64_t* n_hist_out,
                           cudaStream_t st);
// local_hist[bh][bin] = sum over chunks of chunk_hist[bh][chunk][bin]
int launch_hist_reduce(const uint32_t* chunk_hist, int64_t bs_h, int64_t n_chunks, uint32_t* local_hist, cudaStream_t st);

// topk.cu: exact top-k of rows of 32-bit values; out[row][i] = map ? map[row*map_stride + pos] : pos.  n_dev: valid elements
// of every row, read on the device (null: L); n_out: [rows] min(k, valid elements), or null.
int launch_topk(const void* in, bool is_float, int64_t rows, int64_t row_stride, int64_t L, int64_t k, const int32_t* n_dev,
                int64_t* out, int32_t* n_out, const int64_t* map, int64_t map_stride, int order, cudaStream_t st, int stage);

// rerank.cu
struct RerankArgs {
  const int64_t* cand;   // [bs*H][C] or nullptr when candidates come from a per-block list
  const uint8_t* k4;     // element (b,h,s,k,i) at k4[b*k4_b + h*k4_h + s*k4_s + k*k4_l + i]
  int64_t k4_b, k4_h, k4_s, k4_l;
  const uint16_t* w;     // element (b,h,s,k) at w[b*w_b + h*w_h + s*w_s + k*w_l]
  int64_t w_b, w_h, w_s, w_l;
  const uint16_t* q_blocks;  // [bs*H][128]
  const uint16_t* q_norm;    // [bs*H]
  const uint16_t* centers;   // [8]
  int H;
  int64_t C;
};
bool rerank_fast_layout(const RerankArgs& a);   // key-major, 16-byte aligned records
int fill_rerank_args(RerankArgs* a, const pk_tensor* key_4bit, const pk_tensor* key_block_weight);
int launch_rerank(const RerankArgs& a, int64_t bs_h, uint16_t* scores_bf16, float* scores_f32, uint16_t* v4b,
                  cudaStream_t st);

// Candidate selection from u8 counts + per-block histograms and the rerank of the selected keys in one kernel.
struct SelectArgs {
  const uint8_t* counts_u8;      // [bs*H][u8_stride] virtual keys
  int64_t u8_stride;
  const uint32_t* chunk_hist;    // [bs*H][n_chunks][256]
  int64_t n_chunks, chunk_keys;
  int mis;
  int64_t N;                     // keys per head of the view (upper bound when n_dev is set)
  int64_t C;                     // row stride (and capacity) of cand_out / scores_f32
  int64_t C_want;                // candidates wanted per head over the whole zone, all shards together (n_dev == null)
  int64_t K;                     // final top-K (one-launch chain); 0 = stop after the rerank
  int fill_tail;                 // rows may be longer than the candidate list: the tail gets (score -inf, key 0)
  int early_loads;               // see pdl_early()
  const int32_t* n_dev;          // [bs] searchable keys per sample, or null
  pk_zone_schedule sched;        // candidates = zone_candidates(sched, n_dev[b]) when n_dev is set
  const uint32_t* shard_hist;    // [world][bs*H][256] histograms of every shard (exact sequence-sharded selection)
  int world, rank;
  int64_t* cand_out;             // [bs*H][C]
  float* scores_f32;             // [bs*H][C]
  int64_t* final_out;            // [bs*H][K] ascending key index (one-launch chain, K > 0)
  int32_t* n_sel_out;            // [bs*H] or null: entries of final_out that are valid = min(K, candidates)
  int32_t* n_cand_out;           // [bs*H] or null: candidates of this (batch, head)
};
int launch_select_rerank(const RerankArgs& a, int64_t bs_h, const SelectArgs& s, cudaStream_t st);

// retrieve_fused.cu: the whole chain in one launch, one cluster of `cs` CTAs per (batch, head)
int fused_cluster_size(const pk_tensor* codebook, const RerankArgs& a, int64_t bs_h, int64_t N, int64_t C, int64_t K);
// cand_out / scores_out: [bs*H][C] or null; ws_cand / ws_scores: the same arrays in the workspace
int launch_fused_retrieve(int cs, const pk_tensor* codebook, const RerankArgs& a, const ChainQuery& cq, const SelectArgs& sa,
                          int64_t* cand_out, float* scores_out, int64_t* ws_cand, float* ws_scores, cudaStream_t st);

}  // namespace pk
