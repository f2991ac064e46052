// The elementwise steps of a decoder layer that sit between the projections and the cache calls of a decode step:
// q/k RMS-norm + rotate-half RoPE, residual add + RMS-norm, and the gated activation.  One launch each, rows of one
// token per sequence.  They are not retrieval operators (the reference takes them from its attention library,
// model_hub/qwen.py:381 silu_and_mul, :405 and :429 rmsnorm, :482 the rotary embedding); they are here because a
// decode step of 36 layers is launch-latency bound outside the host-link fetch, and every separate elementwise
// launch between two cache calls costs as much as the collision count itself.
#include <type_traits>

#include "common.cuh"

namespace pk {
namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// One warp per (sequence, head) of the first Hq + Hk heads of a fused q/k/v row; lane L holds dims 4L .. 4L+3, whose
// rotate-half partners (d xor 64) sit in lane L xor 16.
//   y   = bf16( x * rsqrt(mean(x^2) + eps) * w[head] )
//   out = bf16( y * cos + y[d xor 64] * sin )            (the sign of rotate-half is folded into sin by the caller)
__global__ void __launch_bounds__(128) qk_norm_rope_kernel(const uint16_t* qkv, int64_t row_stride, const uint16_t* w,
                                                           const uint16_t* cosv, const uint16_t* sinv, int64_t cs_stride, uint16_t* out, int heads, int64_t n_warps, float eps) {
  pdl_wait();
  pdl_trigger();
  const int64_t wid = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (wid >= n_warps) return;
  const int lane = threadIdx.x & 31;
  const int64_t b = wid / heads;
  const int hd = (int)(wid % heads);
  const uint2 raw = *reinterpret_cast<const uint2*>(qkv + b * row_stride + (int64_t)hd * 128 + 4 * lane);
  const uint2 wr = *reinterpret_cast<const uint2*>(w + (int64_t)hd * 128 + 4 * lane);
  const uint2 cr = *reinterpret_cast<const uint2*>(cosv + b * cs_stride + 4 * lane);
  const uint2 sr = *reinterpret_cast<const uint2*>(sinv + b * cs_stride + 4 * lane);
  float x[4] = {__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                __uint_as_float(raw.y & 0xffff0000u)};
  const float ss = warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]);
  const float rstd = rsqrtf(ss * (1.0f / 128.0f) + eps);
  const float wf[4] = {__uint_as_float(wr.x << 16), __uint_as_float(wr.x & 0xffff0000u), __uint_as_float(wr.y << 16),
                       __uint_as_float(wr.y & 0xffff0000u)};
  float y[4], yr[4];
#pragma unroll
  for (int i = 0; i < 4; i++) y[i] = bfround(x[i] * rstd * wf[i]);
#pragma unroll
  for (int i = 0; i < 4; i++) yr[i] = __shfl_xor_sync(0xffffffffu, y[i], 16);
  const float cf[4] = {__uint_as_float(cr.x << 16), __uint_as_float(cr.x & 0xffff0000u), __uint_as_float(cr.y << 16),
                       __uint_as_float(cr.y & 0xffff0000u)};
  const float sf[4] = {__uint_as_float(sr.x << 16), __uint_as_float(sr.x & 0xffff0000u), __uint_as_float(sr.y << 16),
                       __uint_as_float(sr.y & 0xffff0000u)};
  uint16_t o[4];
#pragma unroll
  for (int i = 0; i < 4; i++) o[i] = f2bf(fmaf(y[i], cf[i], yr[i] * sf[i]));
  uint2 ov;
  ov.x = (uint32_t)o[0] | ((uint32_t)o[1] << 16);
  ov.y = (uint32_t)o[2] | ((uint32_t)o[3] << 16);
  *reinterpret_cast<uint2*>(out + wid * 128 + 4 * lane) = ov;
}

// One block per row: h = bf16(a + r) (r optional), x = bf16( h * rsqrt(mean(h^2) + eps) * w ).
// Latency: loads, the sum over the block, stores.  What a thread takes first stays in registers, outside the loops over the rest (a
// choice inside them cost the longer rows more than it saved), and three blocks per SM leave it enough of them.  B200, us, every
// value read again | so: 1 x 4096 1.87 | 1.77, 1 x 12288 3.28 | 3.29, 300 x 4096 3.11 | 2.69.
__global__ void __launch_bounds__(512, 3) add_rmsnorm_kernel(const uint16_t* a, const uint16_t* r, const uint16_t* w,
                                                          uint16_t* h_out, uint16_t* x_out, int n, float eps) {
  pdl_wait();
  pdl_trigger();
  const int tid = threadIdx.x;
  const int64_t base = (int64_t)blockIdx.x * n;
  __shared__ float s_part[16];
  __shared__ float s_rstd;
  float ss = 0.0f;
  const uint4 w0 = tid * 8 < n ? *reinterpret_cast<const uint4*>(w + tid * 8) : make_uint4(0, 0, 0, 0);   // under the reduction
  auto add = [&](int i) -> uint4 {
    const uint4 av = *reinterpret_cast<const uint4*>(a + base + i);
    const uint4 rv = r ? *reinterpret_cast<const uint4*>(r + base + i) : make_uint4(0, 0, 0, 0);
    const uint32_t aw[4] = {av.x, av.y, av.z, av.w}, rw[4] = {rv.x, rv.y, rv.z, rv.w};
    uint32_t ow[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint16_t lo = f2bf(__uint_as_float(aw[k] << 16) + __uint_as_float(rw[k] << 16));
      const uint16_t hi = f2bf(__uint_as_float(aw[k] & 0xffff0000u) + __uint_as_float(rw[k] & 0xffff0000u));
      const float fl = bf2f(lo), fh = bf2f(hi);
      ss += fl * fl + fh * fh;
      ow[k] = (uint32_t)lo | ((uint32_t)hi << 16);
    }
    const uint4 hv = make_uint4(ow[0], ow[1], ow[2], ow[3]);
    *reinterpret_cast<uint4*>(h_out + base + i) = hv;
    return hv;
  };
  uint4 h0 = make_uint4(0, 0, 0, 0);
  if (tid * 8 < n) h0 = add(tid * 8);
  for (int i = tid * 8 + 512 * 8; i < n; i += 512 * 8) add(i);
  ss = warp_sum(ss);
  if ((tid & 31) == 0) s_part[tid >> 5] = ss;
  __syncthreads();
  if (tid < 32) {
    float v = tid < 16 ? s_part[tid] : 0.0f;
    v = warp_sum(v);
    if (tid == 0) s_rstd = rsqrtf(v / (float)n + eps);
  }
  __syncthreads();
  const float rstd = s_rstd;
  auto scale = [&](int i, const uint4 hv, const uint4 wv) {
    const uint32_t hw[4] = {hv.x, hv.y, hv.z, hv.w}, ww[4] = {wv.x, wv.y, wv.z, wv.w};
    uint32_t ow[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint16_t lo = f2bf(__uint_as_float(hw[k] << 16) * rstd * __uint_as_float(ww[k] << 16));
      const uint16_t hi = f2bf(__uint_as_float(hw[k] & 0xffff0000u) * rstd * __uint_as_float(ww[k] & 0xffff0000u));
      ow[k] = (uint32_t)lo | ((uint32_t)hi << 16);
    }
    *reinterpret_cast<uint4*>(x_out + base + i) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
  };
  if (tid * 8 < n) scale(tid * 8, h0, w0);
  for (int i = tid * 8 + 512 * 8; i < n; i += 512 * 8)   // of rows longer than 4096 a thread re-reads what it wrote itself
    scale(i, *reinterpret_cast<const uint4*>(h_out + base + i), *reinterpret_cast<const uint4*>(w + i));
}

// out[row][i] = bf16( bf16(silu(g[row][i])) * u[row][i] ), g = gu[row][0:F], u = gu[row][F:2F]
__global__ void __launch_bounds__(256) silu_mul_kernel(const uint16_t* gu, uint16_t* out, int F) {
  pdl_wait();
  pdl_trigger();
  const int64_t row = blockIdx.y;
  const int i = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (i >= F) return;
  const uint4 gv = *reinterpret_cast<const uint4*>(gu + row * 2 * F + i);
  const uint4 uv = *reinterpret_cast<const uint4*>(gu + row * 2 * F + F + i);
  const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
  uint32_t ow[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const float g0 = __uint_as_float(gw[k] << 16), g1 = __uint_as_float(gw[k] & 0xffff0000u);
    const float a0 = bfround(g0 / (1.0f + __expf(-g0))), a1 = bfround(g1 / (1.0f + __expf(-g1)));
    ow[k] = (uint32_t)f2bf(a0 * __uint_as_float(uw[k] << 16)) | ((uint32_t)f2bf(a1 * __uint_as_float(uw[k] & 0xffff0000u)) << 16);
  }
  *reinterpret_cast<uint4*>(out + row * F + i) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace
}  // namespace pk

using namespace pk;

extern "C" int pk_qk_norm_rope(const pk_tensor* qkv, const pk_tensor* weight, const pk_tensor* cos, const pk_tensor* sin,
                               const pk_tensor* out, double eps, void* stream) {
  PK_CHECK_TENSOR(qkv, PK_BF16, 2);
  PK_CHECK_TENSOR(weight, PK_BF16, 2);
  PK_CHECK_TENSOR(cos, PK_BF16, 2);
  PK_CHECK_TENSOR(sin, PK_BF16, 2);
  PK_CHECK_TENSOR(out, PK_BF16, 3);
  const int64_t B = qkv->shape[0], heads = weight->shape[0];
  PK_REQUIRE(weight->shape[1] == 128 && is_contig(weight), "weight must be contiguous bf16 [heads,128]");
  PK_REQUIRE(qkv->stride[1] == 1 && qkv->shape[1] >= heads * 128 && qkv->stride[0] % 8 == 0,
             "qkv must be bf16 [B, >= heads*128] with unit inner stride and a row stride that is a multiple of 8");
  PK_REQUIRE(out->shape[0] == B && out->shape[1] == heads && out->shape[2] == 128 && is_contig(out),
             "out must be contiguous bf16 [B,heads,128]");
  PK_REQUIRE((cos->shape[0] == 1 || cos->shape[0] == B) && cos->shape[1] == 128 && is_contig(cos) &&
                 sin->shape[0] == cos->shape[0] && sin->shape[1] == 128 && is_contig(sin),
             "cos / sin must be contiguous bf16 [1 or B,128]");
  PK_REQUIRE(aligned16(qkv->data) && aligned16(weight->data) && aligned16(cos->data) && aligned16(sin->data) &&
                 aligned16(out->data),
             "tensors must be 16-byte aligned");
  const int64_t n_warps = B * heads;
  if (n_warps == 0) return PK_OK;
  PK_REQUIRE(heads < (1 << 20) && n_warps < (1LL << 31), "sizes out of range");
  StageTimer timer(ST_GLUE, (cudaStream_t)stream);
  launch_chain(qk_norm_rope_kernel, dim3((unsigned)((n_warps + 3) / 4)), dim3(128), 0, (cudaStream_t)stream,
      (const uint16_t*)qkv->data, qkv->stride[0], (const uint16_t*)weight->data, (const uint16_t*)cos->data,
      (const uint16_t*)sin->data, cos->shape[0] == 1 ? 0 : 128, (uint16_t*)out->data, (int)heads, n_warps, (float)eps);
  return check_launch("qk_norm_rope");
}

extern "C" int pk_add_rmsnorm(const pk_tensor* a, const pk_tensor* residual, const pk_tensor* weight, const pk_tensor* h_out,
                              const pk_tensor* x_out, double eps, void* stream) {
  PK_CHECK_TENSOR(a, PK_BF16, 2);
  PK_CHECK_TENSOR(weight, PK_BF16, 1);
  PK_CHECK_TENSOR(h_out, PK_BF16, 2);
  PK_CHECK_TENSOR(x_out, PK_BF16, 2);
  const int64_t B = a->shape[0], n = a->shape[1];
  PK_REQUIRE(is_contig(a) && is_contig(h_out) && is_contig(x_out) && is_contig(weight), "tensors must be contiguous");
  PK_REQUIRE(h_out->shape[0] == B && h_out->shape[1] == n && x_out->shape[0] == B && x_out->shape[1] == n &&
                 weight->shape[0] == n,
             "h_out / x_out must be [B,n] like a, weight [n]");
  PK_REQUIRE(n % 8 == 0 && n < (1 << 30) && B < 65536LL * 32768, "row length must be a multiple of 8");
  const uint16_t* r = nullptr;
  if (residual) {
    PK_CHECK_TENSOR(residual, PK_BF16, 2);
    PK_REQUIRE(is_contig(residual) && residual->shape[0] == B && residual->shape[1] == n, "residual must be [B,n] like a");
    r = (const uint16_t*)residual->data;
    PK_REQUIRE(aligned16(r), "tensors must be 16-byte aligned");
  }
  PK_REQUIRE(aligned16(a->data) && aligned16(weight->data) && aligned16(h_out->data) && aligned16(x_out->data),
             "tensors must be 16-byte aligned");
  if (B * n == 0) return PK_OK;
  StageTimer timer(ST_GLUE, (cudaStream_t)stream);
  launch_chain(add_rmsnorm_kernel, dim3((unsigned)B), dim3(512), 0, (cudaStream_t)stream, (const uint16_t*)a->data, r,
               (const uint16_t*)weight->data, (uint16_t*)h_out->data, (uint16_t*)x_out->data, (int)n, (float)eps);
  return check_launch("add_rmsnorm");
}

extern "C" int pk_silu_mul(const pk_tensor* gate_up, const pk_tensor* out, void* stream) {
  PK_CHECK_TENSOR(gate_up, PK_BF16, 2);
  PK_CHECK_TENSOR(out, PK_BF16, 2);
  const int64_t B = gate_up->shape[0], F = out->shape[1];
  PK_REQUIRE(is_contig(gate_up) && is_contig(out) && out->shape[0] == B && gate_up->shape[1] == 2 * F,
             "gate_up must be contiguous bf16 [B,2F], out [B,F]");
  PK_REQUIRE(F % 8 == 0 && F < (1 << 30) && B < 65536, "F must be a multiple of 8, B < 65536");
  PK_REQUIRE(aligned16(gate_up->data) && aligned16(out->data), "tensors must be 16-byte aligned");
  if (B * F == 0) return PK_OK;
  StageTimer timer(ST_GLUE, (cudaStream_t)stream);
  launch_chain(silu_mul_kernel, dim3((unsigned)((F / 8 + 255) / 256), (unsigned)B), dim3(256), 0, (cudaStream_t)stream,
               (const uint16_t*)gate_up->data, (uint16_t*)out->data, (int)F);
  return check_launch("silu_mul");
}

// ---- matrix-vector products of a decode step (one token): y = W x, W bf16 [O, I] row-major, fp32 accumulation ------
// HBM-bound: the weights are read once.  A block per SM takes an even share of the rows; its warps share the columns
// (GvSplit::k_warps of them; where rows are short several rows are taken side by side), so that a warp keeps its part
// of x in registers for all rows, and every lane has two steps of up to ten weight loads in flight, by pointers that move on.
// What is lost to the copy rate is the start of each launch.  A block takes nearly all registers of an SM: it starts when its SM's
// block of such a launch before it has ended, beside other kernels at once, and asks for the first 48 KB of its rows by one
// prefetch to L2 before it waits.
// B200, us, in a graph: 6144 x 4096 9.5, 4096 x 12288 15.9, gate and up of 12288 x 4096 32.5, 7168 x 5120 12.6 (two rows per warp, 256
// threads and a grid of 1.2 to 5.2 waves: 10.9, 18.1, 33.7, 15.2; indexes multiplied out for each load and one row of 5120 a step: 9.7,
// 17.1, 32.8, 13.9).  The prefetch: a dense pass of two layers, hidden 4096, feed-forward 12288, 143.1 with it, 146.4 without (16, 32,
// 64, 128 KB 145.1, 143.4, 143.7, 146.4).
// Rows in one range per block up to GV_TURNS steps a block; from there on they are dealt out a step at a time, so that all SMs read one
// window of memory (a last step that only some blocks have costs less than an eighth).  One range | in turn: 151936 x 4096 176.0 | 174.1,
// 32768 x 4096 42.0 | 41.1, 10240 x 4096 14.3 | 14.1, 20480 x 8192 52.1 | 50.1, gate and up of 28672 x 8192 135.1 | 132.5.
// GATED: the rows are (o, o + F) of a stacked [gate; up] matrix and the output is silu(gate) * up, rounded like the
// separate launches would (bf16 after the product, after silu, after the multiply).
namespace pk {
namespace {

constexpr int GV_THREADS = 512, GV_WARPS = GV_THREADS / 32;
constexpr int GV_CHUNKS = 6;               // 16-byte pieces of a row that a lane takes at most
constexpr int GV_PANEL = 128;              // rows whose partial sums are kept at a time
constexpr unsigned GV_PREFETCH = 48 << 10; // bytes
constexpr int GV_TURNS = 8;                // steps of a block from which on its rows are dealt out in turn

// How the columns are split: 1 << k_log warps over a row, `chunks` pieces for a lane.
struct GvSplit {
  int k_log, chunks;
};
// The split that leaves the fewest lanes without a piece, of those with as many warps on a row as possible.
GvSplit gemv_split(int64_t I) {
  const int64_t n = I / 8;
  GvSplit best = {0, 0};
  double used = 0.0;
  for (int k_log = 4; k_log >= 0; k_log--) {
    const int64_t per_warp = (n + (1 << k_log) - 1) >> k_log, chunks = (per_warp + 31) / 32;
    const double u = (double)n / (double)((chunks * 32) << k_log);
    if (chunks <= GV_CHUNKS && u > used + 0.02) best = {k_log, (int)chunks}, used = u;
  }
  return best;
}

// Sums of N (a power of two) values over the lanes of a warp; every lane gets that of value sum_of<N>(lane).
template <int N>
__device__ __forceinline__ float warp_sums(float (&v)[N], int lane) {
  int off = 16;
#pragma unroll
  for (int n = N / 2; n >= 1; n /= 2, off /= 2) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < n; i++) {
      const float keep = up ? v[i + n] : v[i], give = up ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
#pragma unroll
  for (; off > 0; off /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
  return v[0];
}
template <int N>
__device__ __forceinline__ int sum_of(int lane) { return lane * N / 32; }

// Outputs of a warp per step, of U rows of CH pieces each: up to ten loads a lane.
__host__ __device__ constexpr int gv_outputs(int U, int CH) {
  return CH * U >= 6 || (U == 2 && CH >= 3) ? 1 : CH * U >= 3 ? 2 : 8 / (CH * U);
}

// CH: pieces of a row per lane
template <bool GATED, int CH>
__global__ void __launch_bounds__(GV_THREADS, 1) gemv_kernel(const uint16_t* W, const uint16_t* x, uint16_t* out, int n_out, int I, int k_log, int share, int extra, bool early) {
  constexpr int U = GATED ? 2 : 1;                                            // rows of W per output
  constexpr int RB = gv_outputs(U, CH);                                       // outputs of a warp per step
  constexpr int NV = RB * U;
  static_assert(NV == 1 || NV == 2 || NV == 4 || NV == 8, "warp_sums");
  __shared__ float part[GV_PANEL * U][GV_WARPS + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k_warps = 1 << k_log, kw = warp & (k_warps - 1), side = GV_WARPS >> k_log, group = warp >> k_log;
  static_assert((RB & (RB - 1)) == 0, "shifts");
  const int step_log = 4 - k_log + (RB >= 8 ? 3 : RB >= 4 ? 2 : RB >= 2 ? 1 : 0), per_step = 1 << step_log;   // RB * side outputs
  // step s of the block: outputs first + s * stride .. + per_step - 1, those below `end`
  const bool in_turn = share == 0;
  const int block = (int)blockIdx.x, first = in_turn ? block * per_step : block * share + min(block, extra);
  const int end = in_turn ? n_out : first + share + (block < extra);
  const int stride = in_turn ? (int)gridDim.x * per_step : per_step;
  int steps = (end - first + per_step - 1) >> step_log;
  if (in_turn) steps = (int)((unsigned)(steps + (int)gridDim.x - 1) / gridDim.x);
  const int n = I >> 3, c0 = (int)((int64_t)n * kw >> k_log) + lane, c1 = (int)((int64_t)n * (kw + 1) >> k_log);
  if (tid == 0) {   // what this block reads first, on its way to L2 while it waits (a hint: no value is taken before the wait)
    const int64_t bytes = (int64_t)(in_turn ? min(per_step, end - first) : end - first) * I * 2;
    const unsigned size = (unsigned)min(bytes, (int64_t)(GV_PREFETCH / U));
#pragma unroll
    for (int u = 0; u < U; u++)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(W + ((int64_t)first + (int64_t)u * n_out) * I), "r"(size) : "memory");
  }
  struct Step {
    uint4 w[RB][U][CH];
  };
  const uint4* at = reinterpret_cast<const uint4*>(W + (int64_t)(first + group) * I) + c0;   // of the step that is loaded next
  const int64_t next_row = (int64_t)side * n, next_step = (int64_t)stride * n, up = (int64_t)n_out * n;
  int left = end - first - group;   // rows of the block from that step's first of this group on
  auto load = [&](Step& s) {
#pragma unroll
    for (int i = 0; i < RB; i++)
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int j = 0; j < CH; j++)
          s.w[i][u][j] = i * side < left && c0 + 32 * j < c1 ? __ldcs(at + i * next_row + u * up + 32 * j) : make_uint4(0, 0, 0, 0);
    at += next_step, left -= stride;
  };
  Step a, b;
  if (!early) pdl_wait();
  load(a);
  pdl_wait();
  pdl_trigger();
  constexpr bool KEEP_X = CH * U < 12;   // (otherwise the registers do not hold it beside two steps: from L1 each time)
  auto load_x = [&](int j) -> uint4 { return c0 + 32 * j < c1 ? reinterpret_cast<const uint4*>(x)[c0 + 32 * j] : make_uint4(0, 0, 0, 0); };
  uint4 xs[CH];
  if (KEEP_X)
#pragma unroll
    for (int j = 0; j < CH; j++) xs[j] = load_x(j);
  const int panel = GV_PANEL >> step_log;
  auto flush = [&](int step, int n_steps) {   // the outputs of a panel of n_steps steps
    __syncthreads();
    const int o = first + (step + (tid >> step_log)) * stride + (tid & (per_step - 1));
    if (tid < n_steps << step_log && o < end) {
      float y[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        y[u] = 0.0f;
        for (int k = 0; k < k_warps; k++) y[u] += part[tid * U + u][k];
      }
      if (GATED) {
        const float g = bfround(y[0]), up = bfround(y[U - 1]);
        out[o] = f2bf(bfround(g / (1.0f + __expf(-g))) * up);
      } else {
        out[o] = f2bf(y[0]);
      }
    }
  };
  auto use = [&](const Step& s, int in_panel) {
    float v[NV];
#pragma unroll
    for (int i = 0; i < RB; i++)
#pragma unroll
      for (int u = 0; u < U; u++) {
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < CH; j++) {
          const uint4 w = s.w[i][u][j], v8 = KEEP_X ? xs[j] : load_x(j);
          acc = fma_bf16x2(w.x, v8.x, acc), acc = fma_bf16x2(w.y, v8.y, acc);
          acc = fma_bf16x2(w.z, v8.z, acc), acc = fma_bf16x2(w.w, v8.w, acc);
        }
        v[i * U + u] = acc;
      }
    const float sum = warp_sums(v, lane);
    const int at = sum_of<NV>(lane), r = (in_panel * RB + at / U) * side + group;
    if (lane % (32 / NV) == 0) part[r * U + at % U][kw] = sum;
  };
  int in_panel = 0, panel_first = 0;
  auto step_done = [&]() {
    if (++in_panel == panel) {
      flush(panel_first, panel);
      __syncthreads();
      in_panel = 0, panel_first += panel;
    }
  };
#pragma unroll 1
  for (int step = 0; step < steps; step += 2) {
    if (step + 1 < steps) load(b);
    use(a, in_panel);
    step_done();
    if (step + 1 < steps) {
      if (step + 2 < steps) load(a);
      use(b, in_panel);
      step_done();
    }
  }
  if (in_panel) flush(panel_first, in_panel);
}

}  // namespace
}  // namespace pk

extern "C" int pk_gemv(const pk_tensor* weight, const pk_tensor* x, const pk_tensor* out, int gated, void* stream) {
  PK_CHECK_TENSOR(weight, PK_BF16, 2);
  PK_CHECK_TENSOR(x, PK_BF16, 2);
  PK_CHECK_TENSOR(out, PK_BF16, 2);
  const int64_t O = weight->shape[0], I = weight->shape[1];
  PK_REQUIRE(is_contig(weight) && is_contig(x) && is_contig(out) && x->shape[0] == 1 && x->shape[1] == I && out->shape[0] == 1,
             "weight must be contiguous bf16 [O,I], x [1,I], out [1,O] (or [1,O/2] when gated)");
  PK_REQUIRE(I % 8 == 0 && I >= 8 && I <= 24576 && O >= 1 && O < (1LL << 30), "I must be a multiple of 8, at most 24576");
  PK_REQUIRE(gated ? (O % 2 == 0 && out->shape[1] == O / 2) : out->shape[1] == O,
             "out must have O columns (O/2 when gated, with O even)");
  PK_REQUIRE(aligned16(weight->data) && aligned16(x->data), "weight and x must be 16-byte aligned");
  const GvSplit split = gemv_split(I);
  const int64_t n_out = gated ? O / 2 : O;
  const unsigned grid = (unsigned)(n_out < sm_count() ? n_out : sm_count());
  StageTimer timer(ST_GEMV, (cudaStream_t)stream);
  auto launch = [&](auto chunks) {
    constexpr int CH = decltype(chunks)::value;
    const uint16_t *w = (const uint16_t*)weight->data, *in = (const uint16_t*)x->data;
    uint16_t* y = (uint16_t*)out->data;
    const int per_step = gv_outputs(gated ? 2 : 1, CH) * (GV_WARPS >> split.k_log), in_turn = n_out >= (int64_t)GV_TURNS * per_step * grid;
    const int share = in_turn ? 0 : (int)(n_out / grid), extra = (int)(n_out % grid);
    if (gated) launch_chain(gemv_kernel<true, CH>, dim3(grid), dim3(GV_THREADS), 0, (cudaStream_t)stream, w, in, y, (int)n_out, (int)I, split.k_log, share, extra, pdl_early());
    else launch_chain(gemv_kernel<false, CH>, dim3(grid), dim3(GV_THREADS), 0, (cudaStream_t)stream, w, in, y, (int)n_out, (int)I, split.k_log, share, extra, pdl_early());
  };
  switch (split.chunks) {
    case 1: launch(std::integral_constant<int, 1>()); break;
    case 2: launch(std::integral_constant<int, 2>()); break;
    case 3: launch(std::integral_constant<int, 3>()); break;
    case 4: launch(std::integral_constant<int, 4>()); break;
    case 5: launch(std::integral_constant<int, 5>()); break;
    default: launch(std::integral_constant<int, 6>());
  }
  return check_launch("gemv");
}
