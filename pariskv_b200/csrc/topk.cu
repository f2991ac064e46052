// Exact, deterministic top-k of rows of 32-bit values (int32 counts or fp32 scores): one thread-block cluster per row
// (cluster_select.cuh).  Selected set: first k of (value descending, index ascending), emitted in ascending index.
//
// What bounds it: the latency of the selection's exchanges for rows of up to some 10 K elements, three to five passes over
// a CTA's slice (shared memory where it fits) beyond.  On B200, us per launch before (a cluster kernel with five
// bisected levels and per-thread spans; one CTA per row up to 16384 elements) -> now: 8 rows of 32768 counts, k 4096
// 16.7 -> 10.0; 8 rows of 4096 scores, k 256 9.6 -> 8.7.  The operators' nine launches, two of them these: 68.1 -> 65.2 us with
// the exchanges by remote stores.  Rows read four elements a load, six loads in flight: 8 rows of 105K scores, the last launch of
// a step with 1M keys, 114.2 -> 112.7 us a step.  Slices of 4096 elements and more take 1024 threads: that step 114.2 -> 109.3, the
// operators over 8 x 131072 keys with 20000 candidates 243.7 -> 235.3, 32 x 50000 keys 234.0 -> 226.4, 8 x 60000 (slices of 6000) 95.1 ->
// 92.6; shorter slices (8 x 32768 keys, 3300 a slice) lost 1 us to them, 1250 a slice 3.  (Called one after the other with nothing
// between, where a block of 512 threads shares an SM with the call before, slices of 4 - 10 K elements lose about 1 us: 8 x 60000
// 10.5 | 11.5.)  More rows than fit at once keep 512 threads: see launch_rows.
#include "cluster_select.cuh"
#include "common.cuh"
#include "kernels.cuh"

namespace pk {
namespace {

constexpr int TK_WORDS = 1024;              // ballots kept per kind: slices of up to 32 K elements
constexpr int TK_CACHE = 32 * TK_WORDS;     // elements of a slice kept in shared memory; longer ones are read again from L2
constexpr int TK_THREADS_LONG = 1024;       // threads of a block for slices of at least TK_LONG elements
constexpr int TK_LONG = 4096;
constexpr int64_t SM_SMEM = 228 << 10;      // shared memory of an SM
constexpr int TK_STATIC = 2048;             // of a block besides the dynamic: SelShared, and 1 KB of the system's
__host__ __device__ constexpr int tk_fixed(int cs, int threads) { return SEL_REGION + 2 * TK_WORDS * 4 + sel_inbox_bytes(cs, threads); }

struct TopkParams {
  const uint32_t* in;
  int64_t row_stride, L, k;
  const int32_t* n_dev;      // valid elements of every row (device), or null: L
  int64_t* out;              // [rows][k]
  const int64_t* map;        // the value to emit for an element of the row, or null: its index
  int64_t map_stride;
  int32_t* n_out;            // [rows] min(k, valid elements), or null
  int cache;                 // elements of a slice kept in shared memory: all of them, or 0
};

template <int CS, template <int> class Row, int THREADS>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) topk_kernel(TopkParams p) {
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ SelShared s;
  unsigned* region = reinterpret_cast<unsigned*>(dyn);
  unsigned* words = region + SEL_REGION / 4;
  unsigned* inbox = words + 2 * TK_WORDS;
  uint32_t* cache = inbox + sel_inbox_bytes(CS, THREADS) / 4;
  const int tid = threadIdx.x;
  const unsigned rank = CS == 1 ? 0u : cluster.block_rank();
  const int64_t row = blockIdx.y;
  if (CS > 1) cluster.barrier_arrive();   // a CTA has to run before the others may write into it
  pdl_wait();
  pdl_trigger();
  const int64_t L = p.n_dev ? min((int64_t)max(p.n_dev[row], 0), p.L) : p.L;
  const int K = (int)min(p.k, L);
  if (p.n_out && rank == 0 && tid == 0) p.n_out[row] = K;
  if (K <= 0) {   // the same for all CTAs of the row
    if (CS > 1) cluster.barrier_wait();
    return;
  }
  const int64_t slice = ((L + CS - 1) / CS + 31) / 32 * 32, begin = min(L, (int64_t)rank * slice);
  const int n = (int)(min(L, begin + slice) - begin);
  const uint32_t* in = p.in + row * p.row_stride + begin;
  const bool cached = p.cache > 0;   // the same for all CTAs of the row
  unsigned kmin = 0xffffffffu, kmax = 0u;
  int done = 0;
  if (cached && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {   // whole groups of four: up to six such loads in flight per thread
    const int groups = n >> 2;
    const uint4* in4 = reinterpret_cast<const uint4*>(in);
    for (int base = tid; base < groups; base += 6 * THREADS) {
      uint4 u[6];
#pragma unroll
      for (int j = 0; j < 6; j++) u[j] = in4[min(base + j * THREADS, groups - 1)];
#pragma unroll
      for (int j = 0; j < 6; j++) {   // (past the end: the last group again, which changes nothing)
        reinterpret_cast<uint4*>(cache)[min(base + j * THREADS, groups - 1)] = u[j];
        const unsigned k0 = Row<512>::key(u[j].x), k1 = Row<512>::key(u[j].y), k2 = Row<512>::key(u[j].z), k3 = Row<512>::key(u[j].w);
        kmin = min(min(kmin, min(k0, k1)), min(k2, k3)), kmax = max(max(kmax, max(k0, k1)), max(k2, k3));
      }
    }
    done = groups * 4;
  }
  for (int base = done + tid; base < n; base += 8 * THREADS) {   // eight loads in flight per thread
    uint32_t u[8];
#pragma unroll
    for (int j = 0; j < 8; j++) u[j] = in[min(base + j * THREADS, n - 1)];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int i = base + j * THREADS;
      if (i < n) {
        if (cached) cache[i] = u[j];
        const unsigned k = Row<512>::key(u[j]);
        kmin = min(kmin, k), kmax = max(kmax, k);
      }
    }
  }
  if (CS > 1) cluster.barrier_wait();
  const int64_t* map = p.map ? p.map + row * p.map_stride + begin : nullptr;
  auto out_of = [&](int i) -> int64_t { return map ? map[i] : begin + i; };
  if (cached)
    cluster_select<CS, Row<512>, true, THREADS>(cluster, s, region, inbox, words, TK_WORDS, rank, n, K, p.out + row * p.k,
                            [&](int i) -> uint32_t { return cache[i]; }, out_of, kmin, kmax);
  else
    cluster_select<CS, Row<256>, true, THREADS>(cluster, s, region, inbox, words, TK_WORDS, rank, n, K, p.out + row * p.k,
                            [&](int i) -> uint32_t { return in[i]; }, out_of, kmin, kmax);
}

template <int CS, template <int> class Row, int THREADS>
int topk_active() {   // clusters that fit the device at once; also opts in to the shared memory
  auto kern = topk_kernel<CS, Row, THREADS>;
  const int smem = tk_fixed(CS, THREADS) + TK_CACHE * 4;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return cudaGetLastError(), 0;
  if (CS > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return cudaGetLastError(), 0;
  if (CS == 1) return sm_count();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CS, 64), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) return cudaGetLastError(), 0;
  return n;
}
struct TopkCapacity {
  int active[N_CLUSTER_SIZES];
};
template <template <int> class Row>
const TopkCapacity* topk_capacity() {
  static TopkCapacity cap[64];
  static PerDevice asked;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (const unsigned long long bit = first_on_device(asked)) {
    for (int i = 0; i < N_CLUSTER_SIZES; i++)   // several threads may ask at the same time: they write the same numbers
      with_cluster_size(CLUSTER_SIZES[i], [&](auto cs) {
        const int a = topk_active<cs.value, Row, SEL_THREADS>(), b = topk_active<cs.value, Row, TK_THREADS_LONG>();
        cap[dev].active[i] = a < b ? a : b;
      });
    mark_on_device(asked, bit);
  }
  return &cap[dev];
}

template <int CS, template <int> class Row, int THREADS>
cudaError_t launch_topk_cs(int64_t rows, size_t smem, cudaStream_t st, const TopkParams& p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CS, (unsigned)rows), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = smem, cfg.stream = st;
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
  return cudaLaunchKernelEx(&cfg, topk_kernel<CS, Row, THREADS>, p);
}

template <template <int> class Row>
int launch_rows(TopkParams p, int64_t rows, cudaStream_t st) {
  const TopkCapacity* cap = topk_capacity<Row>();
  if (!cap) return fail(PK_ERR_CUDA, "topk: cannot identify the device");
  // CTAs per row: as many as are resident at once with at least 512 elements each (less does not pay for the exchanges);
  // a CTA numbers its elements with 27 bits
  int best = 0, best_i = 0;
  for (int i = 0; i < N_CLUSTER_SIZES; i++) {
    const int cs = CLUSTER_SIZES[i];
    if (cap->active[i] <= 0) continue;
    const bool fits = rows <= cap->active[i] && p.L >= 512LL * cs;
    if (best == 0 || fits || (p.L + best - 1) / best >= (1LL << 27)) best = cs, best_i = i;
  }
  const int64_t slice = ((p.L + best - 1) / best + 31) / 32 * 32;
  if (slice >= (1LL << 27)) return fail(PK_ERR_ARG, "topk: row too long");
  p.cache = slice <= TK_CACHE ? (int)slice : 0;
  // 1024 threads, of which an SM takes one block, unless the rows are more than fit at once and two blocks of 512 threads would share
  // an SM.  B200, us, 512 | 1024 threads: 300 rows of 5000 counts 14.0 | 19.6, of 16384 33.2 | 36.7, of 22000 43.8 | 45.6; of 24000, of
  // which an SM takes one block either way, 58.6 | 48.6; of 60000, read again from L2, 197 | 170; 128 rows of 16384 15.3 | 13.3.
  const bool pair = p.cache > 0 && 2 * (tk_fixed(best, SEL_THREADS) + (int64_t)p.cache * 4 + TK_STATIC) <= SM_SMEM;
  const bool is_long = slice >= TK_LONG && (rows <= cap->active[best_i] || !pair);
  const size_t smem = tk_fixed(best, is_long ? TK_THREADS_LONG : SEL_THREADS) + (size_t)p.cache * 4;
  for (int64_t r0 = 0; r0 < rows; r0 += 65535) {   // grid.y limit
    TopkParams q = p;
    const int64_t nr = rows - r0 < 65535 ? rows - r0 : 65535;
    q.in += r0 * p.row_stride, q.out += r0 * p.k;
    if (q.map) q.map += r0 * p.map_stride;
    if (q.n_dev) q.n_dev += r0;
    if (q.n_out) q.n_out += r0;
    cudaError_t e = cudaErrorInvalidValue;
    with_cluster_size(best, [&](auto c) {
      e = is_long ? launch_topk_cs<c.value, Row, TK_THREADS_LONG>(nr, smem, st, q) : launch_topk_cs<c.value, Row, SEL_THREADS>(nr, smem, st, q);
    });
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(PK_ERR_CUDA, "topk: %s", cudaGetErrorString(e));
    }
    const int rc = check_launch("topk");
    if (rc) return rc;
  }
  return PK_OK;
}

// Reorders an emitted top-k list by (value descending, index ascending): one block per row, k <= 4096.
__global__ void __launch_bounds__(1024) sort_by_value_kernel(const uint32_t* in, int is_float, int64_t row_stride,
                                                             int64_t k, int kp, int64_t* out) {
  extern __shared__ unsigned long long sk[];  // (key << 32) | ~idx  sorted descending
  const int tid = threadIdx.x;
  const int64_t row_id = blockIdx.x;
  const uint32_t* row = in + row_id * row_stride;
  int64_t* o = out + row_id * k;
  for (int i = tid; i < kp; i += 1024) {
    unsigned long long v = 0;
    if (i < k) {
      const int64_t idx = o[i];
      v = ((unsigned long long)(is_float ? F32Row<512>::key(row[idx]) : I32Row<512>::key(row[idx])) << 32) | (0xffffffffu - (unsigned)idx);
    }
    sk[i] = v;
  }
  __syncthreads();
  for (int sz = 2; sz <= kp; sz <<= 1)
    for (int st = sz >> 1; st > 0; st >>= 1) {
      for (int i = tid; i < kp / 2; i += 1024) {
        const int l = 2 * i - (i & (st - 1)), r = l + st;
        const bool desc = ((l / sz) & 1) == 0;
        const unsigned long long a = sk[l], b = sk[r];
        if (desc ? (a < b) : (a > b)) {
          sk[l] = b;
          sk[r] = a;
        }
      }
      __syncthreads();
    }
  for (int i = tid; i < k; i += 1024) o[i] = (int64_t)(0xffffffffu - (unsigned)(sk[i] & 0xffffffffu));
}

}  // namespace

int launch_topk(const void* in, bool is_float, int64_t rows, int64_t row_stride, int64_t L, int64_t k, const int32_t* n_dev,
                int64_t* out, int32_t* n_out, const int64_t* map, int64_t map_stride, int order, cudaStream_t st, int stage) {
  StageTimer tm(stage, st);
  TopkParams p = {};
  p.in = (const uint32_t*)in;
  p.row_stride = row_stride, p.L = L, p.k = k, p.n_dev = n_dev;
  p.out = out, p.n_out = n_out, p.map = map, p.map_stride = map_stride;
  const int rc = is_float ? launch_rows<F32Row>(p, rows, st) : launch_rows<I32Row>(p, rows, st);
  if (rc || order == 0) return rc;
  int kp = 1;
  while (kp < k) kp <<= 1;
  sort_by_value_kernel<<<(unsigned)rows, 1024, (size_t)kp * 8, st>>>(p.in, is_float ? 1 : 0, row_stride, k, kp, out);
  return check_launch("topk sort");
}

}  // namespace pk

using namespace pk;

extern "C" int pk_topk(const pk_tensor* input, int64_t k, const pk_tensor* out, int order, void* stream) {
  PK_REQUIRE(input && input->data, "input is null");
  PK_REQUIRE(input->dtype == PK_I32 || input->dtype == PK_F32, "input must be int32 or float32");
  PK_REQUIRE(input->ndim == 2, "input must be [rows, L]");
  PK_CHECK_TENSOR(out, PK_I64, 2);
  const int64_t rows = input->shape[0], L = input->shape[1];
  PK_REQUIRE(input->stride[1] == 1, "input must have last stride 1");
  PK_REQUIRE(k > 0 && k <= L, "k must be in 1..L (k=%lld, L=%lld)", (long long)k, (long long)L);
  PK_REQUIRE(L < (1ll << 31), "row too long");
  PK_REQUIRE(is_contig(out) && out->shape[0] == rows && out->shape[1] == k, "out must be contiguous [rows,k]");
  PK_REQUIRE(order == 0 || (order == 1 && k <= 4096), "order 1 (sorted by value) needs k <= 4096");
  if (rows == 0) return PK_OK;
  return launch_topk(input->data, input->dtype == PK_F32, rows, input->stride[0], L, k, nullptr, (int64_t*)out->data,
                     nullptr, nullptr, 0, order, (cudaStream_t)stream, ST_TOPK);
}

extern "C" int pk_final_topk(const pk_tensor* scores, const pk_tensor* cand, int64_t K, const pk_tensor* out,
                             void* stream) {
  PK_CHECK_TENSOR(scores, PK_F32, 3);
  PK_CHECK_TENSOR(cand, PK_I64, 3);
  PK_CHECK_TENSOR(out, PK_I64, 3);
  const int64_t bs = scores->shape[0], H = scores->shape[1], C = scores->shape[2];
  PK_REQUIRE(is_contig(scores) && is_contig(cand) && is_contig(out), "scores, cand and out must be contiguous");
  PK_REQUIRE(cand->shape[0] == bs && cand->shape[1] == H && cand->shape[2] == C, "cand must be [bs,H,C]");
  PK_REQUIRE(K > 0 && K <= C, "K must be in 1..C");
  PK_REQUIRE(out->shape[0] == bs && out->shape[1] == H && out->shape[2] == K, "out must be [bs,H,K]");
  if (bs * H == 0) return PK_OK;
  return launch_topk(scores->data, true, bs * H, C, C, K, nullptr, (int64_t*)out->data, nullptr,
                     (const int64_t*)cand->data, C, 0, (cudaStream_t)stream, ST_FINAL_TOPK);
}
