// Exact top-K of a row that is spread over the CTAs of a thread-block cluster (each holds a contiguous slice):
// first K of (value descending, position ascending), emitted in ascending position.
//
//   extremes of the row                      -> 512 bins: linear in the value for floats, about equally filled; the top
//                                               nine bits of (key - lowest key) for whole numbers, exact at any size
//   histogram of the bins, summed over ranks -> the bin of the K-th largest, this CTA's share above it and in it
//   the elements of that bin, gathered by every CTA, cut once more into 64 sub-bins and ranked -> the exact threshold
//   ordered emission of this CTA's elements at its offset, a warp per 32 elements.
// Where more than SEL_TIES elements share the bin (flat rows, equal counts), further levels bin their ordered keys; if
// that many are equal, the lowest positions win.  Three exchanges in the usual case: what a CTA knows it WRITES into the
// shared memory of all CTAs, then comes a cluster barrier, and everything is read at home.  (Reading from the others behind the
// barrier adds a round trip over the cluster to each, two for the members, and a barrier before a CTA may leave.)  A caller
// that makes the values itself can have the extremes exchanged while it still does (see `published`).
// What bounds it is the latency of these steps and three passes over the slice.  On B200 the last stage of the chain takes 7.2
// us with 1310 scores on each of 10 CTAs (9.7 with remote reads, the emission a word per lane and every rank counted in
// sub-bins), 6.1 with 655 (9.5), 7 - 10 with some 5000 on one CTA (10 - 13), all with 256 bins of 32 bits.  512 bins halve the members
// of the threshold bin and what ranking them takes (1.9 -> 1.5 us of the 7.2, with fewer than 129 a warp has four lanes for each);
// as words of 32 bits their exchange would take as much longer (10 CTAs: 1.1 -> 1.6 us), as halves it does not.
#pragma once
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"

namespace pk {
namespace {

namespace cg = cooperative_groups;

// Threads of a block: 512, or twice as many for long slices (see topk.cu).
constexpr int SEL_THREADS = 512;
constexpr int SEL_WARPS_MAX = 32;
constexpr int SEL_WORDS = 256;   // words of a histogram: 512 bins of 16 bits for slices below 65536 elements, 256 of 32 bits for longer ones
constexpr int SEL_SUB = 64;
constexpr int SEL_TIES = 1024;
constexpr int SEL_REGION = 2 * SEL_TIES * 8;   // bytes of dynamic shared memory
// What the CTAs of a cluster write into each other, at the same offset of dynamic shared memory in every CTA and used by nothing
// else: histograms [rank][SEL_WORDS], extremes [rank][warp].
__host__ __device__ constexpr int sel_inbox_bytes(int cs, int threads = SEL_THREADS) { return cs * (SEL_WORDS * 4 + threads / 32 * 8); }

// Rows of a type: the ordered key of an element, and the level-0 bins between the extremes of the row's keys.  A bin is
// monotone in the key; sub() cuts a bin into SEL_SUB parts, monotone as well; single(): a bin holds one value.
template <int N_BINS>
struct F32Row {
  static constexpr int BINS = N_BINS;
  static __device__ __forceinline__ uint32_t key(uint32_t u) { return ord_key(__uint_as_float(u)); }
  static __device__ __forceinline__ float from_key(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k); }
  // Counted down from the row's highest value: a NaN, which the conversion makes zero, then shares the highest bin with what lies
  // above the range.  Its key is the highest there is where arithmetic made it; one with the sign bit set, the lowest key there
  // is, has to lie within the range (which then has no scale).
  struct Bins {
    float vmax, scale;
    __device__ __forceinline__ Bins(uint32_t kmin, uint32_t kmax) {
      vmax = from_key(kmax);
      scale = (float)(BINS - 1) / (vmax - from_key(kmin));
      if (!(scale > 0.0f) || !(scale < INFINITY)) scale = 0.0f;   // flat or non-finite: one bin, the key levels decide
    }
    __device__ __forceinline__ unsigned of(uint32_t u) const {
      return BINS - 1 - min((unsigned)(BINS - 1), __float2uint_rz((vmax - __uint_as_float(u)) * scale));   // (above vmax: the last)
    }
    __device__ __forceinline__ unsigned sub(uint32_t k, unsigned bin) const {
      const float down = (vmax - from_key(k)) * scale - (float)(BINS - 1 - bin);   // of the bin, from its upper end
      return SEL_SUB - 1 - min((unsigned)(SEL_SUB - 1), __float2uint_rz(down * (float)SEL_SUB));
    }
    __device__ __forceinline__ bool single() const { return false; }
  };
};
// From the keys themselves: as floats, whole numbers above 2^24 would share a bin that single() takes for one value.
template <int N_BINS>
struct I32Row {
  static constexpr int BINS = N_BINS;
  static __device__ __forceinline__ uint32_t key(uint32_t u) { return ord_key((int32_t)u); }
  struct Bins {
    uint32_t kmin;
    int shift;   // (kmax - kmin) >> shift < BINS
    __device__ __forceinline__ Bins(uint32_t kmin_, uint32_t kmax) : kmin(kmin_) { shift = max(0, (BINS == 512 ? 23 : 24) - __clz(kmax - kmin)); }
    __device__ __forceinline__ unsigned of(uint32_t u) const { return (key(u) - kmin) >> shift; }
    __device__ __forceinline__ unsigned sub(uint32_t k, unsigned bin) const { return (k - kmin - (bin << shift)) >> max(0, shift - 6); }
    __device__ __forceinline__ bool single() const { return shift == 0; }
  };
};
static_assert(SEL_SUB == 64, "the shifts of I32Row::Bins");

struct SelShared {               // static: small block-wide results
  unsigned n_members;            // local elements of the threshold bin
  unsigned thr_key, thr_pos;     // the last element taken from the threshold bin
  unsigned lower_sel;            // elements taken from the threshold bin by lower ranks
  unsigned res[5];               // threshold bin, elements above it, elements in it, the same two of lower ranks
  unsigned warp_a[SEL_WARPS_MAX], warp_b[SEL_WARPS_MAX];
  unsigned sub[SEL_SUB], n_few;
};

// Cluster sizes that kernels are built for.  A cluster lies within one GPC; with a CTA per SM 148 / 74 / 45 / 33 / 26 /
// 22 / 15 / 11 / 7 of these sizes are resident at once on B200, and no size above 10 does better than 7.
constexpr int CLUSTER_SIZES[] = {1, 2, 3, 4, 5, 6, 8, 10, 16};
constexpr int N_CLUSTER_SIZES = sizeof(CLUSTER_SIZES) / sizeof(int);
// f(integral_constant<int, cs>) for a size of the table.
template <int I = 0, class F>
void with_cluster_size(int cs, F&& f) {
  if constexpr (I < N_CLUSTER_SIZES) {
    if (CLUSTER_SIZES[I] == cs) f(std::integral_constant<int, CLUSTER_SIZES[I]>());
    else with_cluster_size<I + 1>(cs, f);
  }
}

template <int CS>
__device__ __forceinline__ void sync_cluster(cg::cluster_group& cluster) {
  if (CS == 1) __syncthreads();
  else cluster.sync();
}

// value -> *at in CTA r of the cluster, for all r: lane r of a warp (all lanes hold the value), or a thread for all CTAs
template <int CS, class T>
__device__ __forceinline__ void put_by_lanes(cg::cluster_group& cluster, T* at, T value, int lane) {
  if (CS == 1) {
    if (lane == 0) *at = value;
  } else if (lane < CS) {
    *cluster.map_shared_rank(at, lane) = value;
  }
}
template <int CS, class T>
__device__ __forceinline__ void put_everywhere(cg::cluster_group& cluster, T* at, T value) {
  if (CS == 1) {
    *at = value;
  } else {
#pragma unroll
    for (int r = 0; r < CS; r++) *cluster.map_shared_rank(at, r) = value;
  }
}

// Threshold of a histogram spread over the cluster, after the barrier that completes hists ([CS][SEL_WORDS], one row per CTA;
// two bins of 16 bits in a word where there are 512):
// thread t sums bin t, a block-wide suffix scan finds the highest bin with (elements in bins >= it) >= want; see
// SelShared::res.  Returns after the result is visible to the block.
template <int CS, int BINS>
__device__ __forceinline__ void cluster_threshold(SelShared& s, const unsigned* hists, unsigned rank, unsigned want) {
  static_assert(BINS <= SEL_THREADS && (BINS <= SEL_WORDS || BINS == 2 * SEL_WORDS), "one bin per thread");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned tot = 0, pre = 0;
  if (tid < BINS) {
#pragma unroll
    for (int r = 0; r < CS; r++) {
      const unsigned v = BINS <= SEL_WORDS ? hists[r * SEL_WORDS + tid] : (unsigned)reinterpret_cast<const uint16_t*>(hists + r * SEL_WORDS)[tid];
      tot += v;
      if ((unsigned)r < rank) pre += v;
    }
  }
  unsigned suf = tot, psuf = pre;   // inclusive suffix over the lanes
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned o = __shfl_down_sync(0xffffffffu, suf, off), q = __shfl_down_sync(0xffffffffu, psuf, off);
    if (lane + off < 32) suf += o, psuf += q;
  }
  if (lane == 0) s.warp_a[warp] = suf, s.warp_b[warp] = psuf;
  __syncthreads();
  const bool later = lane > warp && lane < (BINS + 31) / 32;   // the sums of the warps behind this one
  suf += __reduce_add_sync(0xffffffffu, later ? s.warp_a[lane] : 0u), psuf += __reduce_add_sync(0xffffffffu, later ? s.warp_b[lane] : 0u);
  const unsigned above = suf - tot;
  if (tot && above < want && suf >= want)
    s.res[0] = (unsigned)tid, s.res[1] = above, s.res[2] = tot, s.res[3] = psuf - pre, s.res[4] = pre;
  __syncthreads();
}

// A warp's extremes into the inboxes of all CTAs.
template <int CS, int WARPS>
__device__ __forceinline__ void publish_range(cg::cluster_group& cluster, unsigned* inbox, unsigned rank, unsigned kmin, unsigned kmax) {
  uint2* extremes = reinterpret_cast<uint2*>(inbox + CS * SEL_WORDS);
  kmin = __reduce_min_sync(0xffffffffu, kmin), kmax = __reduce_max_sync(0xffffffffu, kmax);
  put_by_lanes<CS>(cluster, extremes + rank * WARPS + (threadIdx.x >> 5), make_uint2(kmin, kmax), threadIdx.x & 31);
}

// n: elements of this slice; at(i): raw 32 bits of element i; out_of(i): the 64-bit value to emit for it.
// kmin / kmax: this thread's share of the extremes of the slice's ordered keys (~0 / 0 without any).  published: every warp has
// called publish_range() with the extremes of some of the slice's elements, and every thread has arrived at a cluster barrier
// (CS > 1) behind it; the level-0 bins then lie between those extremes, elements outside fall into the first and the last one.
// V::BINS: 512 where no CTA's slice has more than 65535 elements, otherwise 256.
// region: SEL_REGION bytes, inbox: sel_inbox_bytes(CS, THREADS), at the same offsets in all CTAs; words: 2 * words_cap words of this
// CTA's shared memory for ballots (longer slices are evaluated again instead).  All CTAs of the cluster call this with the same
// K (>= 1, at most the row's length), after a cluster barrier, none of them still using its region for anything else.
// LISTED: the elements are listed in shared memory before out_of() is asked for them, all at once: for values that have to be
// fetched from global memory.
template <int CS, class V, bool LISTED, int THREADS, class At, class OutOf>
__device__ __forceinline__ void cluster_select(cg::cluster_group& cluster, SelShared& s, unsigned* region, unsigned* inbox,
                                               unsigned* words, int words_cap, unsigned rank, int n, int K, int64_t* __restrict__ out, At at,
                                               OutOf out_of, unsigned kmin, unsigned kmax, bool published = false) {
  constexpr int BINS = V::BINS, WARPS = THREADS / 32;
  static_assert(BINS == SEL_WORDS || BINS == 2 * SEL_WORDS, "one word or half a word per bin");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned* hists = inbox;
  uint2* extremes = reinterpret_cast<uint2*>(inbox + CS * SEL_WORDS);
  auto exchange_range = [&](bool published) {   // extremes over the cluster, to kmin and kmax of every thread; clears the histogram replicas
    for (int i = tid; i < 4 * BINS; i += THREADS) region[i] = 0;
    if (published) {
      if (CS > 1) cluster.barrier_wait();
      __syncthreads();
      kmin = 0xffffffffu, kmax = 0u;
    } else {
      publish_range<CS, WARPS>(cluster, inbox, rank, kmin, kmax);
      sync_cluster<CS>(cluster);
    }
#pragma unroll
    for (int i = 0; i < (CS * WARPS + 31) / 32; i++) {
      const uint2 e = extremes[min(i * 32 + lane, CS * WARPS - 1)];
      kmin = min(kmin, e.x), kmax = max(kmax, e.y);
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin), kmax = __reduce_max_sync(0xffffffffu, kmax);
  };
  unsigned* my_hist = region + (lane & 3) * BINS;
  auto exchange_hist = [&]() {
    __syncthreads();
    if (tid < SEL_WORDS) {
      unsigned word = 0;
#pragma unroll
      for (int i = 0; i < 4; i++) {   // (16 bits a bin: the halves' sums stay below 65536)
        if (BINS == SEL_WORDS) {
          word += region[i * BINS + tid];
        } else {
          const uint2 v = reinterpret_cast<const uint2*>(region + i * BINS)[tid];
          word += v.x | (v.y << 16);
        }
      }
      put_everywhere<CS>(cluster, hists + rank * SEL_WORDS + tid, word);
    }
    sync_cluster<CS>(cluster);
  };
  // ---- level 0: bins over the range of the row ----
  exchange_range(published);
  const typename V::Bins bins(kmin, kmax);
  auto bin0 = [&](uint32_t u) -> unsigned { return bins.of(u); };
#pragma unroll 4
  for (int i = tid; i < n; i += THREADS) atomicAdd(&my_hist[bin0(at(i))], 1u);
  exchange_hist();
  cluster_threshold<CS, BINS>(s, hists, rank, (unsigned)K);
  const unsigned T0 = s.res[0];
  unsigned rem = (unsigned)K - s.res[1], in_bin = s.res[2], pre_above = s.res[3], pre_in = s.res[4];
  // ---- key levels: ordered keys of the members between their extremes ----
  unsigned lo = 0u, hi = 0xffffffffu;
  while (in_bin > (unsigned)SEL_TIES && lo != hi) {
    kmin = 0xffffffffu, kmax = 0u;
#pragma unroll 1
    for (int i = tid; i < n; i += THREADS) {
      const uint32_t u = at(i), k = V::key(u);
      if (bin0(u) == T0 && k >= lo && k <= hi) kmin = min(kmin, k), kmax = max(kmax, k);
    }
    __syncthreads();   // s.res and the replicas have been read
    exchange_range(false);
    const unsigned base = kmin, top = kmax;
    if (base == top) {
      lo = hi = base;
      break;
    }
    const int shift = max(0, (BINS == 512 ? 23 : 24) - __clz(top - base));   // (top - base) >> shift < BINS
#pragma unroll 1
    for (int i = tid; i < n; i += THREADS) {
      const uint32_t u = at(i), k = V::key(u);
      if (bin0(u) == T0 && k >= base && k <= top) atomicAdd(&my_hist[(k - base) >> shift], 1u);
    }
    exchange_hist();
    cluster_threshold<CS, BINS>(s, hists, rank, rem);
    lo = base + (s.res[0] << shift);
    hi = lo + min((1u << shift) - 1u, top - lo);   // the sum may not pass the highest key there is
    rem -= s.res[1], in_bin = s.res[2], pre_above += s.res[3], pre_in = s.res[4];
  }
  const bool level0 = lo == 0u && hi == 0xffffffffu;
  // the threshold bin holds equal keys only: the lowest positions win, rank by rank (whole numbers in a small range have a
  // bin each)
  const bool flat = in_bin > (unsigned)SEL_TIES || (level0 && bins.single());

  // ---- where every element stands: above the threshold bin, in it, below; one bit per element ----
  auto standing = [&](uint32_t u, bool& above, bool& member) {
    const unsigned bn = bin0(u);
    above = bn > T0, member = bn == T0;
    if (!level0 && member) {
      const unsigned k = V::key(u);
      above = k > hi, member = k >= lo && k <= hi;
    }
  };
  // The members of all CTAs, in rank order: (key, rank and position).  The histograms say how many the lower ranks have, so
  // every CTA writes its own to their place in all of them.  (The histogram replicas there are done with in every CTA: the
  // barrier of the last histogram lies behind.)
  uint2* all = reinterpret_cast<uint2*>(region);
  const uint2* own = all + pre_in;
  const int n_words = (n + 31) / 32;
  const bool kept = n_words <= words_cap;          // otherwise the words are made window by window, after the threshold
  unsigned* above_w = words;
  unsigned* member_w = words + words_cap;
  if (tid == 0) s.n_members = 0, s.lower_sel = 0, s.n_few = 0;
  if (tid < SEL_SUB) s.sub[tid] = 0;
  __syncthreads();
  if (kept || !flat) {
#pragma unroll 2
    for (int w = warp; w < n_words; w += WARPS) {   // a warp takes every WARPS-th group of 32 elements
      const int i = w * 32 + lane;
      bool above = false, member = false;
      const uint32_t u = at(min(i, n - 1));
      if (i < n) standing(u, above, member);
      const unsigned aw = __ballot_sync(0xffffffffu, above), mw = __ballot_sync(0xffffffffu, member);
      if (kept && lane == 0) above_w[w] = aw, member_w[w] = flat ? mw : 0u;
      if (!flat && mw) {
        unsigned slot = 0;
        if (lane == 0) slot = atomicAdd(&s.n_members, (unsigned)__popc(mw));
        slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(mw & ((1u << lane) - 1u));
        if (member && pre_in + slot < (unsigned)SEL_TIES) put_everywhere<CS>(cluster, all + pre_in + slot, make_uint2(V::key(u), (rank << 27) | (unsigned)i));
      }
    }
  }
  unsigned thr_key = 0u, thr_pos = 0xffffffffu, lower_sel = min(pre_in, rem);
  if (!flat) {
    sync_cluster<CS>(cluster);
    const unsigned before_me = pre_in, n_all = min(in_bin, (unsigned)SEL_TIES);
    if (n_all <= THREADS / 4) {   // four lanes rank a member
      const unsigned t = tid >> 2;
      const uint2 me = t < n_all ? all[t] : make_uint2(0u, 0u);
      unsigned rk = 0;
#pragma unroll 2
      for (unsigned j = tid & 3; j < n_all; j += 4) {
        const uint2 o = all[j];
        rk += (o.x > me.x || (o.x == me.x && o.y < me.y)) ? 1u : 0u;
      }
      rk += __shfl_xor_sync(0xffffffffu, rk, 1);
      rk += __shfl_xor_sync(0xffffffffu, rk, 2);
      if (t < n_all && (tid & 3) == 0) {
        if (rk < rem && t < before_me) atomicAdd(&s.lower_sel, 1u);
        if (rk + 1 == rem) s.thr_key = me.x, s.thr_pos = me.y;
      }
    } else {
      // the members' place within the threshold bin: ranks have to be counted out only in the sub-bin of the last one taken
      auto sub_of = [&](unsigned k) -> unsigned { return level0 ? bins.sub(k, T0) : 0u; };
      for (unsigned t = tid; t < n_all; t += THREADS) atomicAdd(&s.sub[sub_of(all[t].x)], 1u);
      __syncthreads();
      if (warp == 0) {   // lane l: sub-bins 2l, 2l + 1
        const unsigned c0 = s.sub[2 * lane], c1 = s.sub[2 * lane + 1];
        unsigned suf = c0 + c1;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const unsigned o = __shfl_down_sync(0xffffffffu, suf, off);
          if (lane + off < 32) suf += o;
        }
        const unsigned above1 = suf - c0 - c1, above0 = above1 + c1;
        if (above1 < rem && above0 >= rem) s.res[0] = 2 * lane + 1, s.res[1] = above1;
        else if (above0 < rem && suf >= rem) s.res[0] = 2 * lane, s.res[1] = above0;
      }
      __syncthreads();
      const unsigned S = s.res[0], need = rem - s.res[1];
      uint2* few = all + SEL_TIES;   // the sub-bin's elements; bit 31 of the position: held by a lower rank
      for (unsigned t = tid; t < n_all; t += THREADS) {
        const uint2 m = all[t];
        const unsigned ms = sub_of(m.x);
        if (ms == S) few[atomicAdd(&s.n_few, 1u)] = make_uint2(m.x, m.y | (t < before_me ? 0x80000000u : 0u));
        else if (ms > S && t < before_me) atomicAdd(&s.lower_sel, 1u);
      }
      __syncthreads();
      const unsigned n_few = s.n_few;
#pragma unroll 1
      for (unsigned t = warp; t < n_few; t += WARPS) {   // a warp ranks an element
        const uint2 me = few[t];
        const unsigned pos = me.y & 0x7fffffffu;
        unsigned rk = 0;
        for (unsigned j = lane; j < n_few; j += 32) {
          const uint2 o = few[j];
          rk += (o.x > me.x || (o.x == me.x && (o.y & 0x7fffffffu) < pos)) ? 1u : 0u;
        }
        rk = __reduce_add_sync(0xffffffffu, rk);
        if (lane == 0) {
          if (rk < need && (me.y >> 31)) atomicAdd(&s.lower_sel, 1u);
          if (rk + 1 == need) s.thr_key = me.x, s.thr_pos = pos;
        }
      }
    }
    __syncthreads();
    thr_key = s.thr_key, thr_pos = s.thr_pos, lower_sel = s.lower_sel;
  }

  // ---- ordered emission: a warp takes a word of 32 elements at a time, a lane an element ----
  auto taken = [&](unsigned k, unsigned pos) -> bool { return k > thr_key || (k == thr_key && pos <= thr_pos); };
  if (kept && !flat) {   // members that are taken join the elements above
    const unsigned m = min(s.n_members, (unsigned)SEL_TIES - min(pre_in, (unsigned)SEL_TIES));
    for (unsigned t = tid; t < m; t += THREADS) {
      const uint2 me = own[t];
      const unsigned i = me.y & 0x07ffffffu;
      if (taken(me.x, me.y)) atomicOr(&above_w[i >> 5], 1u << (i & 31));
    }
  }
  const unsigned room = flat && rem > lower_sel ? rem - lower_sel : 0u;   // flat bin: members this CTA may still take
  const unsigned pos0 = pre_above + lower_sel;
  unsigned g = pos0, e = 0;   // entries of the final list, and members, before the window
  int* list = reinterpret_cast<int*>(region);   // (the members are done with at the next barrier)
  constexpr unsigned LIST = LISTED ? SEL_REGION / 4 : 0;
  for (int w0 = 0; w0 < n_words; w0 += words_cap) {
    const int nw = min(n_words - w0, words_cap);
    if (!kept) {
      __syncthreads();   // the words of the window before have been read
      for (int w = warp; w < nw; w += WARPS) {
        const int i = (w0 + w) * 32 + lane;
        bool above = false, member = false;
        const uint32_t u = at(min(i, n - 1));
        if (i < n) standing(u, above, member);
        above = above || (!flat && member && taken(V::key(u), (rank << 27) | (unsigned)i));
        const unsigned aw = __ballot_sync(0xffffffffu, above), mw = __ballot_sync(0xffffffffu, member);
        if (lane == 0) above_w[w] = aw, member_w[w] = flat ? mw : 0u;
      }
    }
    __syncthreads();
    const int per = (nw + WARPS - 1) / WARPS;   // a warp's consecutive words
    const int a0 = min(nw, warp * per), a1 = min(nw, a0 + per);
    unsigned na = 0, nm = 0;
    for (int w = a0 + lane; w < a1; w += 32) na += __popc(above_w[w]), nm += __popc(member_w[w]);
    na = __reduce_add_sync(0xffffffffu, na), nm = __reduce_add_sync(0xffffffffu, nm);
    if (lane == 0) s.warp_a[warp] = na, s.warp_b[warp] = nm;
    __syncthreads();
    unsigned gw, ew;
    {
      const unsigned x = lane < WARPS ? s.warp_a[lane] : 0u, y = lane < WARPS ? s.warp_b[lane] : 0u;
      gw = g + __reduce_add_sync(0xffffffffu, lane < warp ? x : 0u), ew = e + __reduce_add_sync(0xffffffffu, lane < warp ? y : 0u);
      g += __reduce_add_sync(0xffffffffu, x), e += __reduce_add_sync(0xffffffffu, y);
    }
    for (int wb = a0; wb < a1; wb += 32) {
      const int w = wb + lane;
      const unsigned aw = w < a1 ? above_w[w] : 0u, mw = w < a1 ? member_w[w] : 0u;
      const unsigned mine = ((unsigned)__popc(aw) << 16) | (unsigned)__popc(mw);   // at most 1024 of either in 32 words
      unsigned inc = mine;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned o = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += o;
      }
      const unsigned total = __shfl_sync(0xffffffffu, inc, 31);
      const unsigned e0 = ew + ((inc - mine) & 0xffffu), g0 = gw + ((inc - mine) >> 16);   // before the lane's word
#pragma unroll 1
      for (int j = 0; j < min(32, a1 - wb); j++) {
        const unsigned a = __shfl_sync(0xffffffffu, aw, j), below = (1u << lane) - 1u;
        unsigned pos = __shfl_sync(0xffffffffu, g0, j) + __popc(a & below);
        bool take = (a >> lane) & 1u;
        if (flat) {
          const unsigned m = __shfl_sync(0xffffffffu, mw, j), e = __shfl_sync(0xffffffffu, e0, j) + __popc(m & below);
          take = take || (((m >> lane) & 1u) && e < room);
          pos += min(e, room);
        }
        if (take && pos < (unsigned)K) {
          const int i = (w0 + wb + j) * 32 + lane;
          if (pos - pos0 < LIST) list[pos - pos0] = i;
          else out[pos] = out_of(i);
        }
      }
      gw += total >> 16, ew += total & 0xffffu;
    }
  }
  if (!LISTED) return;
  __syncthreads();
  const unsigned last = min((unsigned)K, g + min(e, room)), n_list = last > pos0 ? min(last - pos0, LIST) : 0u;
  for (unsigned t = tid; t < n_list; t += THREADS) out[pos0 + t] = out_of(list[t]);
}

}  // namespace
}  // namespace pk
