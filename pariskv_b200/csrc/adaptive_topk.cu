// Fused adaptive-k: window logits, joint max, exp * ||v|| benefits, the K_out largest in order, chunked prefix sums and
// threshold search, index gather.  One block of 1024 threads per (batch, head).  Every fp32 step follows a fixed order
// (stated inline) that the CPU oracle repeats.
//
// What bounds it: latency (a dependent gather of value norms, then a dozen block-wide steps over a few thousand values);
// one block per head keeps every step inside one SM.  Selection and sort are one bucket pass: 8192 buckets, linear in
// the benefits' bit patterns (so about logarithmic in their values), hold a candidate or two each, and a candidate's
// rank is its bucket's offset plus its rank among the few of its bucket.  B200, 64 heads, 3.3 - 6.6K candidates, K_out 4096:
// 47 us with a radix select, a 78-level bitonic sort and atomics of every row that reaches the threshold; 14 now.
#include "common.cuh"
#include "kernels.cuh"

namespace pk {
namespace {

constexpr int AK_THREADS = 1024;
constexpr int AK_ITEMS = 8;                  // candidates per thread whose loads are in flight together
constexpr int AK_BINS = 8192;
constexpr int AK_BIN_MAX = 128;              // fuller buckets (benefits equal, or spread over very many octaves) take the radix path
constexpr int AK_CACHE_MAX = 32 * 1024;      // benefits kept in shared memory; longer lists are recomputed per pass

struct AkParams {
  float* sl_logits;        // read, or written when q_avg is set
  int64_t sl_b, sl_h;
  const float* sl_vnorm;
  int64_t sv_b, sv_h;
  const uint16_t* q_avg;   // bf16 [bs*H,128] or null: the window logits are given
  const uint16_t* win_k;   // rows of 128 bf16
  int64_t wk_b, wk_h;
  const int32_t* n_window; // rows filled (device), or null: all S
  const void* cand;        // f32 or bf16
  int cand_bf16, round_bf16;   // round_bf16: f32 scores are rounded to bf16 first
  int64_t c_b, c_h;
  float scale;
  const int64_t* cand_idx;
  int64_t ci_b, ci_h;
  const float* cand_vnorm;  // or null
  int64_t cv_b, cv_h;
  const float* value_norm;  // used when cand_vnorm is null
  int64_t vn_b, vn_h;
  int64_t sink;
  int H;
  int64_t S, C, K_out, min_k, max_k;
  int K_pad, n_sort;     // power of two >= K_out; slots of the sort area
  int cache_c;           // benefits kept in shared memory (C when they fit, else 0: recomputed per pass)
  float threshold;
  const int32_t* n_cand; // or null: caps the result
  int64_t* ak_out;
  int64_t* topk_out;
  int32_t* n_sel_out;    // or null
};

// Two sums over the 1024 per-thread partials (thread id = leaf), each an adjacent pairwise tree, and the extremes of `lo`, `hi`.
__device__ __forceinline__ void tree_sums_1024(float& a, float& b, unsigned& lo, unsigned& hi, uint4* s_red, int tid) {
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, off));
    b = __fadd_rn(b, __shfl_xor_sync(0xffffffffu, b, off));
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((tid & 31) == 0) s_red[tid >> 5] = make_uint4(__float_as_uint(a), __float_as_uint(b), lo, hi);
  __syncthreads();
  const uint4 v = s_red[tid & 31];
  a = __uint_as_float(v.x), b = __uint_as_float(v.y);
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, off));
    b = __fadd_rn(b, __shfl_xor_sync(0xffffffffu, b, off));
  }
  lo = __reduce_min_sync(0xffffffffu, v.z);
  hi = __reduce_max_sync(0xffffffffu, v.w);
}

// Exclusive prefix sum over the block; `sum` receives the total.
__device__ __forceinline__ unsigned block_scan_1024(unsigned v, unsigned* s_scan, int tid, unsigned* sum) {
  const int lane = tid & 31, warp = tid >> 5;
  unsigned incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned o = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += o;
  }
  if (lane == 31) s_scan[warp] = incl;
  __syncthreads();
  const unsigned w = s_scan[lane];
  *sum = __reduce_add_sync(0xffffffffu, w);
  return incl - v + __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
}

__device__ __forceinline__ float dot8(const uint4& a, const uint4& b, float acc) {
  const unsigned x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    acc = fmaf(__uint_as_float(x[i] << 16), __uint_as_float(y[i] << 16), acc);
    acc = fmaf(__uint_as_float(x[i] & 0xffff0000u), __uint_as_float(y[i] & 0xffff0000u), acc);
  }
  return acc;
}

__global__ void __launch_bounds__(AK_THREADS) adaptive_topk_kernel(AkParams p) {
  extern __shared__ __align__(16) unsigned char dyn[];
  unsigned* hist = reinterpret_cast<unsigned*>(dyn);                                       // AK_BINS
  unsigned long long* sk = reinterpret_cast<unsigned long long*>(hist + AK_BINS);          // n_sort composite keys
  float* sb = reinterpret_cast<float*>(sk + p.n_sort);                                     // sorted benefits, a word of padding per 32
  float* bcache = sb + p.K_pad + (p.K_pad >> 5) + 1;                                       // cache_c benefits
  __shared__ uint4 s_red[32];
  __shared__ float s_max[32];
  __shared__ unsigned s_scan[32];
  __shared__ unsigned s_res[3];
  __shared__ unsigned s_counter;
  __shared__ int s_fk;
  __shared__ float chunk_base[130];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t bh = blockIdx.x;
  const int b = (int)(bh / p.H), h = (int)(bh % p.H);
  const int C = (int)p.C, S = (int)p.S, K_out = (int)p.K_out;
  float* sll = p.sl_logits + b * p.sl_b + h * p.sl_h;
  const float* slv = p.sl_vnorm + b * p.sv_b + h * p.sv_h;
  const int64_t* ci = p.cand_idx + b * p.ci_b + h * p.ci_h;
  const float* cvn = p.cand_vnorm ? p.cand_vnorm + b * p.cv_b + h * p.cv_h : nullptr;
  const float* vn = p.value_norm ? p.value_norm + b * p.vn_b + h * p.vn_h + p.sink : nullptr;
  const float* cf = p.cand_bf16 ? nullptr : (const float*)p.cand + b * p.c_b + h * p.c_h;
  const uint16_t* cb = p.cand_bf16 ? (const uint16_t*)p.cand + b * p.c_b + h * p.c_h : nullptr;
  auto score = [&](int c) -> float { return cb ? bf2f(cb[c]) : cf[c]; };
  auto scaled = [&](float s) -> float { return __fmul_rn(p.round_bf16 ? bfround(s) : s, p.scale); };
  auto vnorm = [&](int c) -> float { return cvn ? cvn[c] : vn[ci[c]]; };
  pdl_wait();
  pdl_trigger();

  // 1. joint max.  The first AK_ITEMS candidates of a thread stay in registers, their norms on the way meanwhile
  float lg[AK_ITEMS], nv[AK_ITEMS];
  {
    int64_t at[AK_ITEMS];
#pragma unroll
    for (int j = 0; j < AK_ITEMS; j++) {   // past the end: the last candidate again, unused below
      const int c = min(tid + AK_THREADS * j, C - 1);
      lg[j] = score(c);
      at[j] = cvn ? c : ci[c];
    }
#pragma unroll
    for (int j = 0; j < AK_ITEMS; j++) nv[j] = cvn ? cvn[at[j]] : vn[at[j]];
  }
  int n_win = S;
  float m = -3.402823466e+38f;
  if (p.q_avg) {
    // window logits: eight lanes per row of 128, fp32 sums rounded to bf16 (the reference's dense product), then scaled
    if (p.n_window) n_win = min(max(*p.n_window, 0), S);
    const int l8 = lane & 7;
    const uint4* q = reinterpret_cast<const uint4*>(p.q_avg + bh * 128);
    const uint4 q0 = q[l8], q1 = q[l8 + 8];
    const uint4* rows = reinterpret_cast<const uint4*>(p.win_k + b * p.wk_b + h * p.wk_h);
#pragma unroll 2
    for (int s0 = warp * 4; s0 < S; s0 += AK_THREADS / 8) {
      const int s = s0 + (lane >> 3);
      const uint4* r = rows + (int64_t)min(s, max(n_win - 1, 0)) * 16;
      float d = dot8(r[l8 + 8], q1, dot8(r[l8], q0, 0.0f));
#pragma unroll
      for (int off = 1; off < 8; off <<= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
      d = s < n_win ? __fmul_rn(bfround(d), p.scale) : -INFINITY;
      m = fmaxf(m, d);
      if (l8 == 0 && s < S) sll[s] = d;
    }
  } else {
    for (int s = tid; s < S; s += AK_THREADS) m = fmaxf(m, sll[s]);
  }
#pragma unroll
  for (int j = 0; j < AK_ITEMS; j++) lg[j] = scaled(lg[j]), m = fmaxf(m, lg[j]);
#pragma unroll 4
  for (int c = tid + AK_THREADS * AK_ITEMS; c < C; c += AK_THREADS) m = fmaxf(m, scaled(score(c)));
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  if (lane == 0) s_max[warp] = m;
#pragma unroll
  for (int i = 0; i < AK_BINS / AK_THREADS; i++) hist[tid + AK_THREADS * i] = 0u;
  __syncthreads();
  float gmax = s_max[lane];
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, off));
  auto compute_benefit = [&](float logit, float norm) -> float { return __fmul_rn(pinned_expf(__fsub_rn(logit, gmax)), norm); };
  const bool cached = p.cache_c > 0;
  auto benefit = [&](int c) -> float { return cached ? bcache[c] : compute_benefit(scaled(score(c)), vnorm(c)); };

  // 2./3. benefit sums: strided sequential partials, then the pairwise tree
  float sl_ben = 0.0f, total = 0.0f;
  for (int s = tid; s < n_win; s += AK_THREADS)
    sl_ben = __fadd_rn(sl_ben, __fmul_rn(pinned_expf(__fsub_rn(sll[s], gmax)), slv[s]));
  unsigned umin = 0xffffffffu, umax = 0u;   // bit patterns of the benefits above zero
  auto note = [&](int c, float bn) {
    if (cached) bcache[c] = bn;
    total = __fadd_rn(total, bn);
    const unsigned u = __float_as_uint(bn);
    if (u) umin = min(umin, u), umax = max(umax, u);
  };
#pragma unroll
  for (int j = 0; j < AK_ITEMS; j++)
    if (tid + AK_THREADS * j < C) note(tid + AK_THREADS * j, compute_benefit(lg[j], nv[j]));
#pragma unroll 4
  for (int c = tid + AK_THREADS * AK_ITEMS; c < C; c += AK_THREADS) note(c, compute_benefit(scaled(score(c)), vnorm(c)));
  tree_sums_1024(sl_ben, total, umin, umax, s_red, tid);
  total = __fadd_rn(sl_ben, total);

  // 4. buckets, highest benefits first (bit patterns of non-negative floats are ordered); zeros are kept out of them
  const float inv = (float)(AK_BINS - 1) / (__uint2float_rn(umax - umin) + 1.0f);   // unused when no benefit is above zero
  auto bucket = [&](unsigned u) -> int { return min((int)(__uint2float_rn(umax - u) * inv), AK_BINS - 1); };
  for (int c = tid; c < C; c += AK_THREADS)
    if (const unsigned u = __float_as_uint(benefit(c))) atomicAdd(&hist[bucket(u)], 1u);
  __syncthreads();
  unsigned nnz, n_bin[AK_BINS / AK_THREADS], sum = 0;
  {
    const uint4* src = reinterpret_cast<const uint4*>(hist) + tid * (AK_BINS / AK_THREADS / 4);
#pragma unroll
    for (int i = 0; i < AK_BINS / AK_THREADS / 4; i++) {
      const uint4 v = src[i];
      n_bin[4 * i] = v.x, n_bin[4 * i + 1] = v.y, n_bin[4 * i + 2] = v.z, n_bin[4 * i + 3] = v.w;
      sum += v.x + v.y + v.z + v.w;
    }
  }
  unsigned at = block_scan_1024(sum, s_scan, tid, &nnz);
  bool full = false;
#pragma unroll
  for (int i = 0; i < AK_BINS / AK_THREADS; i++) {
    full |= n_bin[i] > AK_BIN_MAX && at < (unsigned)K_out;
    hist[tid * (AK_BINS / AK_THREADS) + i] = at;   // a bucket's first slot; the scatter turns it into its end
    at += n_bin[i];
  }
  int64_t* out = p.topk_out + bh * p.K_out;
  auto slot_of = [](unsigned i) -> unsigned { return i + (i >> 5); };
  if (!__syncthreads_or(full)) {
    // 5. scatter into the buckets.  Buckets that start below K_out end below n_sort = K_out + AK_BIN_MAX
    for (int c = tid; c < C; c += AK_THREADS)
      if (const unsigned u = __float_as_uint(benefit(c))) {
        const unsigned slot = atomicAdd(&hist[bucket(u)], 1u);
        if (slot < (unsigned)p.n_sort) sk[slot] = ((unsigned long long)u << 32) | (0xffffffffu - (unsigned)c);
      }
    __syncthreads();
    // 6. rank inside the bucket: benefit descending, then lower position first
    for (unsigned i = tid; i < min(nnz, (unsigned)p.n_sort); i += AK_THREADS) {
      const unsigned long long key = sk[i];
      const int bk = bucket((unsigned)(key >> 32));
      unsigned r = bk ? hist[bk - 1] : 0u;
      const unsigned end = min(hist[bk], (unsigned)p.n_sort);
      if (r < (unsigned)K_out) {
        for (unsigned j = r; j < end; j++) r += sk[j] > key;
        if (r < (unsigned)K_out) {
          sb[slot_of(r)] = __uint_as_float((unsigned)(key >> 32));
          out[r] = ci[0xffffffffu - (unsigned)key];
        }
      }
    }
    if (nnz < (unsigned)K_out) {   // zeros fill up by ascending position
      const int span = (C + AK_THREADS - 1) / AK_THREADS, lo = min(C, tid * span), hi = min(C, lo + span);
      unsigned n = 0, all;
      for (int c = lo; c < hi; c++) n += __float_as_uint(benefit(c)) == 0u;
      __syncthreads();   // (s_scan)
      unsigned r = nnz + block_scan_1024(n, s_scan, tid, &all);
      for (int c = lo; c < hi && r < (unsigned)K_out; c++)
        if (__float_as_uint(benefit(c)) == 0u) {
          sb[slot_of(r)] = 0.0f;
          out[r++] = ci[c];
        }
    }
    __syncthreads();
  } else {
    // 5. exact radix select of the K_out-th largest: 11-bit digits from the top; stops when a whole digit bin is taken
    unsigned prefix = 0u, pmask = 0u, rem = (unsigned)K_out;
    for (int hi = 31; hi >= 0; hi -= 11) {
      const int lo = max(hi - 10, 0);
      const unsigned dm = ((hi == 31 ? 0u : (1u << (hi + 1))) - (1u << lo));
      hist[tid] = 0;
      hist[tid + 1024] = 0;
      __syncthreads();
      for (int c = tid; c < C; c += AK_THREADS) {
        const unsigned u = __float_as_uint(benefit(c));
        if (((u ^ prefix) & pmask) == 0) atomicAdd(&hist[2047u - ((u & dm) >> lo)], 1u);
      }
      __syncthreads();
      const unsigned v0 = hist[2 * tid], v1 = hist[2 * tid + 1];  // thread t owns digits 2047 - 2t, 2046 - 2t
      unsigned all_here;
      const unsigned before = block_scan_1024(v0 + v1, s_scan, tid, &all_here);
      if (before < rem && before + v0 >= rem) s_res[0] = 2047u - 2 * tid, s_res[1] = before, s_res[2] = v0;
      else if (before + v0 < rem && before + v0 + v1 >= rem) s_res[0] = 2046u - 2 * tid, s_res[1] = before + v0, s_res[2] = v1;
      __syncthreads();
      prefix |= s_res[0] << lo;
      pmask |= dm;
      rem -= s_res[1];
      const bool all = s_res[2] == rem;
      __syncthreads();
      if (all) break;  // undecided bits of prefix stay zero: the rest of the bin compares >= prefix
    }
    const unsigned T = prefix;  // take all benefits > T and the first `rem` (by position) equal to T
    // collect: ties by ascending position need an ordered scan; slots are arbitrary, the sort fixes order
    for (int i = tid; i < p.K_pad; i += AK_THREADS) sk[i] = 0ull;
    if (tid == 0) s_counter = 0;
    const int span = (C + AK_THREADS - 1) / AK_THREADS;
    const int my_b = min(C, tid * span), my_e = min(C, my_b + span);
    unsigned n_eq = 0, all_eq;
    for (int c = my_b; c < my_e; c++) n_eq += (__float_as_uint(benefit(c)) == T);
    unsigned eq_run = block_scan_1024(n_eq, s_scan, tid, &all_eq);
    for (int c = my_b; c < my_e; c++) {
      const unsigned u = __float_as_uint(benefit(c));
      bool take = u > T;
      if (u == T) {
        take = eq_run < rem;
        eq_run++;
      }
      if (take) {
        const unsigned slot = atomicAdd(&s_counter, 1u);
        if (slot < (unsigned)K_out) sk[slot] = ((unsigned long long)u << 32) | (0xffffffffu - (unsigned)c);
      }
    }
    __syncthreads();
    // 6. bitonic sort, descending (benefit, then lower position first)
    for (int sz = 2; sz <= p.K_pad; sz <<= 1)
      for (int st = sz >> 1; st > 0; st >>= 1) {
        for (int i = tid; i < p.K_pad / 2; i += AK_THREADS) {
          const int l = 2 * i - (i & (st - 1)), r = l + st;
          const bool desc = ((l / sz) & 1) == 0;
          const unsigned long long a = sk[l], c2 = sk[r];
          if (desc ? (a < c2) : (a > c2)) {
            sk[l] = c2;
            sk[r] = a;
          }
        }
        __syncthreads();
      }
    for (int i = tid; i < K_out; i += AK_THREADS) {
      sb[slot_of(i)] = __uint_as_float((unsigned)(sk[i] >> 32));
      const unsigned pos = 0xffffffffu - (unsigned)(sk[i] & 0xffffffffu);
      out[i] = pos < (unsigned)C ? ci[pos] : 0;
    }
    __syncthreads();
  }

  // 7. prefix sums in chunks of 32 (sequential inside a chunk, sequential over chunk totals)
  const int n_chunks = (K_out + 31) / 32;
  if (tid < n_chunks) {
    float loc = 0.0f;
    float* mine = sb + tid * 33;
    const int n = min(32, K_out - tid * 32);
#pragma unroll 8
    for (int i = 0; i < n; i++) {
      loc = __fadd_rn(loc, mine[i]);
      mine[i] = loc;
    }
    chunk_base[tid + 1] = loc;
  }
  if (tid == 0) s_fk = K_out;
  __syncthreads();
  if (tid == 0) {
    float base = 0.0f;
#pragma unroll 8
    for (int c = 0; c < n_chunks; c++) {
      const float t = chunk_base[c + 1];
      chunk_base[c] = base;
      base = __fadd_rn(base, t);
    }
  }
  __syncthreads();
  if (total <= 0.0f) {
    if (tid == 0) s_fk = 1;
  } else {
    const float tgt = __fmul_rn(p.threshold, total);
    unsigned first = (unsigned)K_out;
    for (int i = tid; i < K_out; i += AK_THREADS) {
      const float cs = __fadd_rn(chunk_base[i >> 5], sb[slot_of(i)]);
      if (__fadd_rn(sl_ben, cs) >= tgt) first = min(first, (unsigned)i + 1u);
    }
    first = __reduce_min_sync(0xffffffffu, first);
    if (lane == 0) atomicMin(&s_fk, (int)first);
  }
  __syncthreads();
  if (tid == 0) {
    int64_t fk = s_fk;
    if (p.max_k > 0) {
      fk = max(fk, p.min_k);
      fk = min(fk, p.max_k);
      fk = min(fk, p.K_out);
    }
    if (p.n_cand) fk = min(fk, (int64_t)p.n_cand[bh]);
    p.ak_out[bh] = fk;
    if (p.n_sel_out) p.n_sel_out[bh] = (int)fk;
  }
}

}  // namespace
}  // namespace pk

using namespace pk;

namespace {

// `win`: the window logits are computed here (query_avg, window_k, n_window) and sl_logits is an output.
struct AkWindow {
  const pk_tensor *query_avg, *window_k, *n_window, *n_cand, *n_sel;
};

int run_adaptive(const pk_tensor* sl_logits, const pk_tensor* cand_scores, float cand_scale,
                 const pk_tensor* sl_vnorm, const pk_tensor* cand_indices, const pk_tensor* cand_vnorm,
                 const pk_tensor* value_norm, int64_t sink_size, float threshold, int64_t K_out, int64_t min_k,
                 int64_t max_k, const pk_tensor* adaptive_k, const pk_tensor* topk_indices, const AkWindow* win,
                 void* stream) {
  PK_CHECK_TENSOR(sl_logits, PK_F32, 3);
  PK_CHECK_TENSOR(sl_vnorm, PK_F32, 3);
  PK_CHECK_TENSOR(cand_indices, PK_I64, 3);
  PK_CHECK_TENSOR(adaptive_k, PK_I64, 2);
  PK_CHECK_TENSOR(topk_indices, PK_I64, 3);
  PK_REQUIRE(cand_scores && cand_scores->data && cand_scores->ndim == 3 &&
                 (cand_scores->dtype == PK_F32 || cand_scores->dtype == PK_BF16),
             "cand_scores must be a 3-D float32 or bfloat16 tensor");
  const int64_t bs = sl_logits->shape[0], H = sl_logits->shape[1], S = sl_logits->shape[2], C = cand_scores->shape[2];
  PK_REQUIRE(sl_logits->stride[2] == 1 && sl_vnorm->stride[2] == 1 && cand_scores->stride[2] == 1 &&
                 cand_indices->stride[2] == 1,
             "inputs must have last stride 1");
  PK_REQUIRE(sl_vnorm->shape[0] == bs && sl_vnorm->shape[1] == H && sl_vnorm->shape[2] == S, "sl_vnorm must be [bs,H,S]");
  PK_REQUIRE(cand_scores->shape[0] == bs && cand_scores->shape[1] == H && cand_indices->shape[0] == bs &&
                 cand_indices->shape[1] == H && cand_indices->shape[2] == C,
             "cand_scores / cand_indices must be [bs,H,C]");
  PK_REQUIRE(K_out >= 1 && K_out <= C && K_out <= 4096, "K_out must be in 1..min(C,4096), got %lld", (long long)K_out);
  PK_REQUIRE(threshold > 0.0f && threshold <= 1.0f, "threshold must be in (0,1]");
  PK_REQUIRE(is_contig(adaptive_k) && adaptive_k->shape[0] == bs && adaptive_k->shape[1] == H,
             "adaptive_k must be contiguous [bs,H]");
  PK_REQUIRE(is_contig(topk_indices) && topk_indices->shape[0] == bs && topk_indices->shape[1] == H &&
                 topk_indices->shape[2] == K_out,
             "topk_indices must be contiguous [bs,H,K_out]");
  AkParams p = {};
  if (cand_vnorm) {
    PK_CHECK_TENSOR(cand_vnorm, PK_F32, 3);
    PK_REQUIRE(cand_vnorm->shape[0] == bs && cand_vnorm->shape[1] == H && cand_vnorm->shape[2] == C &&
                   cand_vnorm->stride[2] == 1,
               "cand_vnorm must be [bs,H,C] with last stride 1");
    p.cand_vnorm = (const float*)cand_vnorm->data;
    p.cv_b = cand_vnorm->stride[0], p.cv_h = cand_vnorm->stride[1];
  } else {
    PK_CHECK_TENSOR(value_norm, PK_F32, 3);
    PK_REQUIRE(value_norm->shape[0] == bs && value_norm->shape[1] == H && value_norm->stride[2] == 1,
               "value_norm must be [bs,H,cap] with last stride 1");
    p.value_norm = (const float*)value_norm->data;
    p.vn_b = value_norm->stride[0], p.vn_h = value_norm->stride[1];
    p.sink = sink_size;
  }
  if (bs * H == 0) return PK_OK;
  p.sl_logits = (float*)sl_logits->data, p.sl_b = sl_logits->stride[0], p.sl_h = sl_logits->stride[1];
  p.sl_vnorm = (const float*)sl_vnorm->data, p.sv_b = sl_vnorm->stride[0], p.sv_h = sl_vnorm->stride[1];
  p.cand = cand_scores->data, p.cand_bf16 = cand_scores->dtype == PK_BF16;
  p.c_b = cand_scores->stride[0], p.c_h = cand_scores->stride[1];
  p.scale = cand_scale;
  p.cand_idx = (const int64_t*)cand_indices->data, p.ci_b = cand_indices->stride[0], p.ci_h = cand_indices->stride[1];
  p.H = (int)H, p.S = S, p.C = C, p.K_out = K_out, p.min_k = min_k, p.max_k = max_k;
  int kp = 2;
  while (kp < K_out) kp <<= 1;
  p.K_pad = kp;
  p.threshold = threshold;
  p.ak_out = (int64_t*)adaptive_k->data;
  p.topk_out = (int64_t*)topk_indices->data;
  PK_REQUIRE(S < (1ll << 30) && C < (1ll << 30), "adaptive top-k: rows too long");
  if (win) {
    PK_CHECK_TENSOR(win->query_avg, PK_BF16, 3);
    PK_CHECK_TENSOR(win->window_k, PK_BF16, 4);
    const pk_tensor& w = *win->window_k;
    PK_REQUIRE(is_contig(win->query_avg) && numel(win->query_avg) == bs * H * 128, "query_avg must be contiguous [bs,H,128]");
    PK_REQUIRE(w.shape[0] == bs && w.shape[1] == H && w.shape[2] >= S && w.shape[3] == 128 && w.stride[2] == 128 &&
                   w.stride[3] == 1 && w.stride[0] % 8 == 0 && w.stride[1] % 8 == 0 && ((uintptr_t)w.data & 15) == 0,
               "window_k must be [bs,H,>=S,128] with contiguous, 16-byte aligned rows");
    PK_REQUIRE(cand_scores->dtype == PK_F32, "cand_scores must be float32");
    p.q_avg = (const uint16_t*)win->query_avg->data;
    p.win_k = (const uint16_t*)w.data, p.wk_b = w.stride[0], p.wk_h = w.stride[1];
    p.round_bf16 = 1;
    if (win->n_window) {
      PK_REQUIRE(win->n_window->data && win->n_window->dtype == PK_I32 && numel(win->n_window) >= 1, "n_window must be an i32 word");
      p.n_window = (const int32_t*)win->n_window->data;
    }
    if (win->n_cand) {
      PK_CHECK_TENSOR(win->n_cand, PK_I32, 2);
      PK_REQUIRE(is_contig(win->n_cand) && numel(win->n_cand) == bs * H, "n_cand must be contiguous i32 [bs,H]");
      p.n_cand = (const int32_t*)win->n_cand->data;
    }
    PK_CHECK_TENSOR(win->n_sel, PK_I32, 2);
    PK_REQUIRE(is_contig(win->n_sel) && numel(win->n_sel) == bs * H, "n_sel must be contiguous i32 [bs,H]");
    p.n_sel_out = (int32_t*)win->n_sel->data;
  }
  p.cache_c = C <= AK_CACHE_MAX ? (int)C : 0;
  p.n_sort = (int)(kp > K_out + AK_BIN_MAX ? kp : K_out + AK_BIN_MAX);
  auto bytes = [](int64_t k_pad, int64_t n_sort, int64_t cache) {
    return (size_t)(AK_BINS * 4 + n_sort * 8 + (k_pad + k_pad / 32 + 1) * 4 + cache * 4);
  };
  static PerDevice smem_attr;
  if (const unsigned long long bit = first_on_device(smem_attr)) {
    if (cudaFuncSetAttribute(adaptive_topk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)bytes(4096, 4096 + AK_BIN_MAX, AK_CACHE_MAX)) != cudaSuccess)
      return check_launch("adaptive_topk smem");
    mark_on_device(smem_attr, bit);
  }
  StageTimer timer(ST_ADAPTIVE, (cudaStream_t)stream);
  launch_chain(adaptive_topk_kernel, dim3((unsigned)(bs * H)), dim3(AK_THREADS), bytes(kp, p.n_sort, p.cache_c),
               (cudaStream_t)stream, p);
  return check_launch("adaptive_topk");
}

}  // namespace

extern "C" int pk_adaptive_topk(const pk_tensor* sl_logits, const pk_tensor* cand_scores, float cand_scale,
                                const pk_tensor* sl_vnorm, const pk_tensor* cand_indices, const pk_tensor* cand_vnorm,
                                const pk_tensor* value_norm, int64_t sink_size, float threshold, int64_t K_out,
                                int64_t min_k, int64_t max_k, const pk_tensor* adaptive_k,
                                const pk_tensor* topk_indices, void* stream) {
  return run_adaptive(sl_logits, cand_scores, cand_scale, sl_vnorm, cand_indices, cand_vnorm, value_norm, sink_size,
                      threshold, K_out, min_k, max_k, adaptive_k, topk_indices, nullptr, stream);
}

extern "C" int pk_adaptive_select(const pk_tensor* query_avg, const pk_tensor* window_k, const pk_tensor* n_window,
                                  const pk_tensor* sl_logits, const pk_tensor* cand_scores, const pk_tensor* n_cand,
                                  float scale, const pk_tensor* sl_vnorm, const pk_tensor* cand_indices,
                                  const pk_tensor* value_norm, float threshold, int64_t K_out, int64_t min_k,
                                  int64_t max_k, const pk_tensor* adaptive_k, const pk_tensor* topk_indices,
                                  const pk_tensor* n_sel, void* stream) {
  const AkWindow win = {query_avg, window_k, n_window, n_cand, n_sel};
  return run_adaptive(sl_logits, cand_scores, scale, sl_vnorm, cand_indices, nullptr, value_norm, 0, threshold, K_out,
                      min_k, max_k, adaptive_k, topk_indices, &win, stream);
}
