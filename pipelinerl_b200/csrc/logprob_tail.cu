// Hot path (2b, generic-model variant): per-token log-probability and exact entropy
// from MATERIALISED fp32 logits, single pass, plus the backward.
//
// Replaces pipelinerl/finetune/rl/__init__.py:207-233: the reference makes a
// `/temperature` copy, a gather, a logsumexp and a 38-chunk entropy loop (>= 3
// full passes over 608 KB/token of logits, plus softmax again in backward).
// Here: forward reads each logit once (online max / sum / sum(e*z)), backward
// reads once and writes once.  The fused-head kernel (lm_head.cu) removes the
// logits from HBM altogether; this kernel serves models that hand us logits
// (any torch module, as rl_step's contract allows).
//
//   z = logits / temperature
//   lse = logsumexp(z);  new_lp = z[next] - lse
//   H = -sum p log p = lse - sum(p * z)
//   dz_v = g_lp (1[v==next] - p_v) - g_H p_v (log p_v + H)
#include "prl_common.cuh"
#include <math.h>

namespace prl {
namespace {

constexpr int kThreads = 512;

struct Online {
  float m, s, u;  // running max, sum exp(z-m), sum exp(z-m)*z
};
// A group of n values joins: one comparison and at most one rescale for all of them.  Value by value, the branch of a new
// maximum kept the loads of a row from staying in flight: 2000 x 151936 logits 257 us (4.7 TB/s), 198 now.
template <int n>
__device__ __forceinline__ void online_add(Online& a, const float (&z)[n]) {
  float m = z[0];
#pragma unroll
  for (int e = 1; e < n; ++e) m = fmaxf(m, z[e]);
  if (m > a.m) {
    const float r = __expf(a.m - m);  // exp(-inf) = 0 for the first group
    a.s *= r;
    a.u *= r;
    a.m = m;
  }
  const float base = a.m == -INFINITY ? 0.f : a.m;   // nothing but -inf so far: their exponentials are zeros
#pragma unroll
  for (int e = 0; e < n; ++e) {
    const float x = __expf(z[e] - base);
    a.s += x;
    a.u = fmaf(x, z[e], a.u);
  }
}
__device__ __forceinline__ Online online_merge(const Online& a, const Online& b) {
  Online o;
  o.m = fmaxf(a.m, b.m);
  const float ra = (a.m == -INFINITY) ? 0.f : __expf(a.m - o.m);
  const float rb = (b.m == -INFINITY) ? 0.f : __expf(b.m - o.m);
  o.s = a.s * ra + b.s * rb;
  o.u = a.u * ra + b.u * rb;
  return o;
}

__global__ void __launch_bounds__(kThreads) tail_fwd_kernel(const float* __restrict__ logits, int64_t V,
                                                           int64_t row_stride, const int64_t* __restrict__ ids,
                                                           float inv_temp, float* __restrict__ new_lp,
                                                           float* __restrict__ entropy, float* __restrict__ lse_out) {
  const int64_t row = blockIdx.x;
  const float* z = logits + row * row_stride;
  Online acc{-INFINITY, 0.f, 0.f};
  const bool vec = ((reinterpret_cast<uintptr_t>(z) & 15) == 0);
  const int64_t v4 = vec ? (V / 4) : 0;
  constexpr int kAhead = 4;           // 16-byte loads in flight per thread
  int64_t i = threadIdx.x;
  for (; i + (kAhead - 1) * kThreads < v4; i += kAhead * kThreads) {
    float4 x[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) x[k] = ld_stream_f4(reinterpret_cast<const float4*>(z) + i + k * kThreads);
    float v[4 * kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      v[4 * k] = x[k].x * inv_temp; v[4 * k + 1] = x[k].y * inv_temp;
      v[4 * k + 2] = x[k].z * inv_temp; v[4 * k + 3] = x[k].w * inv_temp;
    }
    online_add(acc, v);
  }
  for (; i < v4; i += kThreads) {
    const float4 x = ld_stream_f4(reinterpret_cast<const float4*>(z) + i);
    const float v[4] = {x.x * inv_temp, x.y * inv_temp, x.z * inv_temp, x.w * inv_temp};
    online_add(acc, v);
  }
  for (i = v4 * 4 + threadIdx.x; i < V; i += kThreads) {
    const float v[1] = {z[i] * inv_temp};
    online_add(acc, v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Online other;
    other.m = __shfl_xor_sync(0xffffffffu, acc.m, o);
    other.s = __shfl_xor_sync(0xffffffffu, acc.s, o);
    other.u = __shfl_xor_sync(0xffffffffu, acc.u, o);
    acc = online_merge(acc, other);
  }
  __shared__ Online s_w[kThreads / kWarp];
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    Online t = s_w[0];
    for (int w = 1; w < kThreads / kWarp; ++w) t = online_merge(t, s_w[w]);
    const float lse = t.m + logf(t.s);
    const int64_t nxt = ids[row + 1];
    float lp = NAN;  // out-of-vocabulary ids surface through the non-finite check, as an index error would
    if (nxt >= 0 && nxt < V) lp = z[nxt] * inv_temp - lse;
    new_lp[row] = lp;
    if (entropy) entropy[row] = lse - t.u / t.s;
    if (lse_out) lse_out[row] = lse;
  }
}

// d logits: reads 4 bytes and writes 4 per logit, or writes alone where a row has no gradient (prompts): 2001 x 151936, HBM-bound, 390 us,
// 332 with a third of the rows masked.  Rows go from the last to the first, whose logits the forward has left in L2.  g_loss (device memory,
// or NULL: 1) scales the gradients; where it is 1 the last rows_done rows are left alone: they hold d logits of that scale already.
__global__ void __launch_bounds__(kThreads) tail_bwd_kernel(const float* __restrict__ logits, int64_t V,
                                                           int64_t row_stride, int64_t n_rows,
                                                           const int64_t* __restrict__ ids, float inv_temp,
                                                           const float* __restrict__ lse_in,
                                                           const float* __restrict__ entropy,
                                                           const float* __restrict__ g_lp,
                                                           const float* __restrict__ g_ent,
                                                           const float* __restrict__ g_loss, int rows_done,
                                                           float* __restrict__ dlogits, int64_t d_stride) {
  const float gs = g_loss ? *g_loss : 1.f;
  if ((int)blockIdx.x < rows_done && gs == 1.f) return;
  const int64_t row = (int64_t)gridDim.x - 1 - blockIdx.x;
  float* d = dlogits + row * d_stride;
  const bool has_target = row < n_rows;  // the last position has none (logits[:, :-1])
  const float gl = has_target && g_lp ? g_lp[row] * gs : 0.f, ge = has_target && g_ent ? g_ent[row] * gs : 0.f;
  // no gradient: zeros, without a look at the logits where the statistics say that they are numbers; a logit that is not one (entropy or
  // log-sum-exp are none either) makes the row's gradient none, masked or not, as the formula has it
  if (gl == 0.f && ge == 0.f && (!has_target || (entropy && isfinite(lse_in[row]) && isfinite(entropy[row])))) {
    const int64_t v4 = (reinterpret_cast<uintptr_t>(d) & 15) == 0 ? V / 4 : 0;
    for (int64_t i = threadIdx.x; i < v4; i += kThreads) st_stream_f4(reinterpret_cast<float4*>(d) + i, make_float4(0.f, 0.f, 0.f, 0.f));
    for (int64_t i = v4 * 4 + threadIdx.x; i < V; i += kThreads) d[i] = 0.f;
    return;
  }
  const float* z = logits + row * row_stride;
  const float lse = lse_in[row];
  const float H = (g_ent && entropy) ? entropy[row] : 0.f;
  const int64_t nxt = ids[row + 1];
  const bool vec = ((reinterpret_cast<uintptr_t>(z) & 15) == 0) && ((reinterpret_cast<uintptr_t>(d) & 15) == 0);
  const int64_t v4 = vec ? (V / 4) : 0;
  auto one = [&](float zi, int64_t idx) -> float {
    const float lp = zi * inv_temp - lse;
    const float p = __expf(lp);
    float g = -gl * p - ge * p * (lp + H);
    if (idx == nxt) g += gl;
    return g * inv_temp;
  };
  for (int64_t i = threadIdx.x; i < v4; i += kThreads) {
    const float4 x = ld_stream_f4(reinterpret_cast<const float4*>(z) + i);
    float4 o;
    o.x = one(x.x, i * 4); o.y = one(x.y, i * 4 + 1); o.z = one(x.z, i * 4 + 2); o.w = one(x.w, i * 4 + 3);
    st_stream_f4(reinterpret_cast<float4*>(d) + i, o);
  }
  for (int64_t i = v4 * 4 + threadIdx.x; i < V; i += kThreads) d[i] = one(z[i], i);
}

// ---- head backward over the rows that have a gradient (the tokens of prompts have none: their labels are masked) -------------------
// Order of the `count` rows with a gradient: slot c holds row rows[c], row r's slot is place[r], or -1.  A row below `count` keeps its own
// slot and the others fill the slots of rows without one, in turn: d logits of a row can then take the place of the logits it is made
// from.  One block: 2048 rows of two columns are 16 KB.
__global__ void __launch_bounds__(1024) live_rows_kernel(const float* __restrict__ g_lp, const float* __restrict__ g_ent,
                                                         const float* __restrict__ lse, const float* __restrict__ entropy, int n,
                                                         int32_t* rows, int32_t* place, int32_t* open, int32_t* __restrict__ count) {
  __shared__ int s_warp[2][32];
  __shared__ int s_total;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_total = 0;
  __syncthreads();
  int mine = 0;
  for (int r = threadIdx.x; r < n; r += 1024) {
    // a gradient that is not a number is one, too, and so is none on a row of which a logit is not a number
    const bool live = (g_lp && !(g_lp[r] == 0.f)) || (g_ent && !(g_ent[r] == 0.f)) || !isfinite(lse[r]) || !isfinite(entropy[r]);
    place[r] = live ? r : -1;
    mine += live;
  }
  atomicAdd(&s_total, mine);
  __syncthreads();
  const int total = s_total;
  int n_open = 0, n_moved = 0;             // slots without a row, rows without a slot: as many of either
  for (int r0 = 0; r0 < n; r0 += 1024) {
    const int r = r0 + (int)threadIdx.x;
    const bool live = r < n && place[r] >= 0, is_open = r < total && !live, moved = live && r >= total;
    const unsigned mo = __ballot_sync(0xffffffffu, is_open), mm = __ballot_sync(0xffffffffu, moved);
    if (lane == 0) { s_warp[0][warp] = __popc(mo); s_warp[1][warp] = __popc(mm); }
    __syncthreads();
    int at_open = n_open + __popc(mo & ((1u << lane) - 1u)), at_moved = n_moved + __popc(mm & ((1u << lane) - 1u));
    for (int w = 0; w < 32; ++w) {
      if (w < warp) { at_open += s_warp[0][w]; at_moved += s_warp[1][w]; }
      n_open += s_warp[0][w];
      n_moved += s_warp[1][w];
    }
    if (is_open) open[at_open] = r;
    if (moved) place[r] = n + at_moved;    // until every open slot is known
    if (live && r < total) rows[r] = r;
    __syncthreads();
  }
  for (int r = threadIdx.x; r < n; r += 1024) {
    const int p = place[r];
    if (p >= n) {
      const int slot = open[p - n];
      rows[slot] = r;
      place[r] = slot;
    }
  }
  if (threadIdx.x == 0) *count = total;
}

// xc[c] = x[rows[c]], and zeros in both operands of dW up to the k-block's end (rows count .. the next multiple of 64).
// Rows are K channels (a multiple of 8) wide.
__global__ void __launch_bounds__(256) gather_rows_kernel(const uint4* __restrict__ x, const int32_t* __restrict__ rows,
                                                          const int32_t* __restrict__ count, int64_t k8, uint4* __restrict__ xc,
                                                          __nv_bfloat16* __restrict__ dz, int64_t dz_rows, int64_t V, int64_t ld_dz) {
  const int c = blockIdx.x, n = *count;
  if (c >= (n + 63) / 64 * 64) return;
  if (c < n) {
    const uint4* src = x + (int64_t)rows[c] * k8;
    for (int64_t i = threadIdx.x; i < k8; i += 256) xc[c * k8 + i] = src[i];
    return;
  }
  for (int64_t i = threadIdx.x; i < k8; i += 256) xc[c * k8 + i] = make_uint4(0u, 0u, 0u, 0u);
  if (c >= dz_rows) return;
  __nv_bfloat16* d = dz + c * ld_dz;
  if ((reinterpret_cast<uintptr_t>(d) & 15) == 0 && (V & 7) == 0)
    for (int64_t i = threadIdx.x; i < V / 8; i += 256) reinterpret_cast<uint4*>(d)[i] = make_uint4(0u, 0u, 0u, 0u);
  else
    for (int64_t i = threadIdx.x; i < V; i += 256) d[i] = __float2bfloat16_rn(0.f);
}

// out[r] = src[place[r]], or zeros
__global__ void __launch_bounds__(256) spread_rows_kernel(const uint4* __restrict__ src, const int32_t* __restrict__ place, int64_t k8,
                                                          uint4* __restrict__ out) {
  const int64_t r = blockIdx.x;
  const int c = place[r];
  for (int64_t i = threadIdx.x; i < k8; i += 256) out[r * k8 + i] = c >= 0 ? src[c * k8 + i] : make_uint4(0u, 0u, 0u, 0u);
}

// d logits (bf16) of the rows with a gradient from logits that the forward kept: the formula of the head's GEMM epilogue, whose
// products these are, so the bits of a recomputation.  They take the place of the logits, slot c = the first half of row c, so that no second buffer is
// needed: a piece is written once all threads have read theirs, and lies in a part of the row that was read by then.
// Reads 4 bytes and writes 2 per logit: HBM-bound.
constexpr int kKept = 16;                  // logits per thread and piece
__device__ __forceinline__ float4 ld_rw_f4(const float4* p) {      // not the read-only path: this launch writes there
  float4 r;
  asm volatile("ld.global.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "l"(p) : "memory");
  return r;
}
__global__ void __launch_bounds__(kThreads) dlogits_kept_kernel(float* logits, int64_t ld, int64_t V, const int32_t* __restrict__ rows,
                                                                const int32_t* __restrict__ count, const int64_t* __restrict__ targets,
                                                                float inv_temp, const float* __restrict__ lse_in,
                                                                const float* __restrict__ entropy, const float* __restrict__ g_lp,
                                                                const float* __restrict__ g_ent) {
  const int64_t c = blockIdx.x;
  if (c >= *count) return;
  const int64_t row = rows[c];
  const float4* z = reinterpret_cast<const float4*>(logits + row * ld);
  uint4* d = reinterpret_cast<uint4*>(logits + c * ld);
  const float lse = lse_in[row], gl = g_lp ? g_lp[row] : 0.f, ge = g_ent ? g_ent[row] : 0.f;
  const float H = (g_ent && entropy) ? entropy[row] : 0.f;
  const int64_t tgt = targets[row];
  const int64_t v8 = V / 8;
  constexpr int kP = kKept / 8;
  auto load = [&](int64_t i0, float4 (&x)[2 * kP]) {
#pragma unroll
    for (int k = 0; k < kP; ++k) {
      const int64_t i = i0 + k * kThreads + threadIdx.x;
      if (i < v8) { x[2 * k] = ld_rw_f4(z + 2 * i); x[2 * k + 1] = ld_rw_f4(z + 2 * i + 1); }
    }
  };
  float4 next[2 * kP];
  load(0, next);
  for (int64_t i0 = 0; i0 < v8; i0 += kP * kThreads) {
    float4 x[2 * kP];
#pragma unroll
    for (int k = 0; k < 2 * kP; ++k) x[k] = next[k];
    load(i0 + kP * kThreads, next);
    uint4 h[kP];
#pragma unroll
    for (int k = 0; k < kP; ++k) {
      const int64_t rel = tgt - 8 * (i0 + k * kThreads + threadIdx.x);
      const float v[8] = {x[2 * k].x, x[2 * k].y, x[2 * k].z, x[2 * k].w, x[2 * k + 1].x, x[2 * k + 1].y, x[2 * k + 1].z, x[2 * k + 1].w};
      uint32_t u[4];
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        float o[2];
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          const float lp = v[e + f] * inv_temp - lse;
          const float pr = __expf(lp);
          float w = -gl * pr - ge * pr * (lp + H);
          if (rel == e + f) w += gl;
          o[f] = w * inv_temp;
        }
        const __nv_bfloat162 p = __floats2bfloat162_rn(o[0], o[1]);
        u[e / 2] = *reinterpret_cast<const uint32_t*>(&p);
      }
      h[k] = make_uint4(u[0], u[1], u[2], u[3]);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kP; ++k) {
      const int64_t i = i0 + k * kThreads + threadIdx.x;
      if (i < v8) d[i] = h[k];
    }
  }
}

}  // namespace
}  // namespace prl

using namespace prl;

extern "C" int prl_logprob_tail_fwd(const float* logits, int64_t T, int64_t V, int64_t row_stride,
                                    const int64_t* input_ids, float temperature, float* new_logprobs,
                                    float* entropy, float* lse, prl_stream_t stream_) {
  PRL_CHECK_ARG(T >= 1 && V >= 1 && row_stride >= V, "prl_logprob_tail_fwd: bad shape T=%lld V=%lld stride=%lld",
                (long long)T, (long long)V, (long long)row_stride);
  PRL_CHECK_ARG(temperature > 0.f, "prl_logprob_tail_fwd: temperature must be > 0");
  if (T == 1) return PRL_OK;
  PRL_CHECK_ARG(logits && input_ids && new_logprobs, "prl_logprob_tail_fwd: NULL argument");
  tail_fwd_kernel<<<(unsigned)(T - 1), kThreads, 0, (cudaStream_t)stream_>>>(
      logits, V, row_stride, input_ids, 1.f / temperature, new_logprobs, entropy, lse);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

extern "C" int prl_logprob_tail_bwd(const float* logits, int64_t T, int64_t V, int64_t row_stride,
                                    const int64_t* input_ids, float temperature, const float* lse,
                                    const float* entropy, const float* g_logprobs, const float* g_entropy,
                                    float* dlogits, int64_t dlogits_stride, prl_stream_t stream_) {
  PRL_CHECK_ARG(T >= 1 && V >= 1 && row_stride >= V && dlogits_stride >= V, "prl_logprob_tail_bwd: bad shape");
  PRL_CHECK_ARG(temperature > 0.f, "prl_logprob_tail_bwd: temperature must be > 0");
  PRL_CHECK_ARG(logits && input_ids && lse && dlogits, "prl_logprob_tail_bwd: NULL argument");
  PRL_CHECK_ARG(!g_entropy || entropy, "prl_logprob_tail_bwd: g_entropy needs the forward entropy");
  tail_bwd_kernel<<<(unsigned)T, kThreads, 0, (cudaStream_t)stream_>>>(
      logits, V, row_stride, T - 1, input_ids, 1.f / temperature, lse, entropy, g_logprobs, g_entropy, nullptr, 0, dlogits,
      dlogits_stride);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

// prl_logprob_tail_bwd with the gradients scaled by *g_loss (device memory); where that is 1 the last rows_done rows are not written
extern "C" int prl_logprob_tail_bwd_scaled(const float* logits, int64_t T, int64_t V, int64_t row_stride, const int64_t* input_ids,
                                           float temperature, const float* lse, const float* entropy, const float* g_logprobs,
                                           const float* g_entropy, const float* g_loss, int32_t rows_done, float* dlogits,
                                           int64_t dlogits_stride, prl_stream_t stream_) {
  PRL_CHECK_ARG(T >= 1 && V >= 1 && row_stride >= V && dlogits_stride >= V, "prl_logprob_tail_bwd_scaled: bad shape");
  PRL_CHECK_ARG(temperature > 0.f, "prl_logprob_tail_bwd_scaled: temperature must be > 0");
  PRL_CHECK_ARG(logits && input_ids && lse && g_loss && dlogits, "prl_logprob_tail_bwd_scaled: NULL argument");
  PRL_CHECK_ARG(!g_entropy || entropy, "prl_logprob_tail_bwd_scaled: g_entropy needs the forward entropy");
  PRL_CHECK_ARG(rows_done >= 0 && rows_done <= T, "prl_logprob_tail_bwd_scaled: bad rows_done");
  tail_bwd_kernel<<<(unsigned)T, kThreads, 0, (cudaStream_t)stream_>>>(logits, V, row_stride, T - 1, input_ids, 1.f / temperature, lse, entropy,
                                                                       g_logprobs, g_entropy, g_loss, rows_done, dlogits, dlogits_stride);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

// Backward over an explicit (row, target) list: rows of a recomputed logits CHUNK (the fused head's backward
// recomputes logits chunk by chunk instead of keeping 608 KB/token alive between forward and backward).
extern "C" int prl_logprob_rows_bwd(const float* logits, int64_t n_rows, int64_t V, int64_t row_stride,
                                    const int64_t* targets, float temperature, const float* lse, const float* entropy,
                                    const float* g_logprobs, const float* g_entropy, float* dlogits,
                                    int64_t dlogits_stride, prl_stream_t stream_) {
  PRL_CHECK_ARG(n_rows >= 1 && V >= 1 && row_stride >= V && dlogits_stride >= V, "prl_logprob_rows_bwd: bad shape");
  PRL_CHECK_ARG(temperature > 0.f, "prl_logprob_rows_bwd: temperature must be > 0");
  PRL_CHECK_ARG(logits && targets && lse && dlogits, "prl_logprob_rows_bwd: NULL argument");
  PRL_CHECK_ARG(!g_entropy || entropy, "prl_logprob_rows_bwd: g_entropy needs the forward entropy");
  // the kernel reads ids[row + 1]: bias the pointer by one element so that it sees targets[row]
  tail_bwd_kernel<<<(unsigned)n_rows, kThreads, 0, (cudaStream_t)stream_>>>(
      logits, V, row_stride, n_rows, targets - 1, 1.f / temperature, lse, entropy, g_logprobs, g_entropy, nullptr, 0,
      dlogits, dlogits_stride);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

// Rows of [n] gradient columns that are not zero, or of statistics that are no numbers: slot c < *count holds row rows[c], row r has slot place[r] or -1; a row below *count
// has its own.  index: room for 3 n + 1 (rows, places, scratch, count).
extern "C" int prl_live_rows(const float* g_logprobs, const float* g_entropy, const float* lse, const float* entropy, int64_t n,
                             int32_t* index, prl_stream_t stream_) {
  PRL_CHECK_ARG(index && (g_logprobs || g_entropy) && lse && entropy, "prl_live_rows: NULL argument");
  PRL_CHECK_ARG(n >= 1 && n < (1ll << 30), "prl_live_rows: bad row count %lld", (long long)n);
  live_rows_kernel<<<1, 1024, 0, (cudaStream_t)stream_>>>(g_logprobs, g_entropy, lse, entropy, (int)n, index, index + n, index + 2 * n, index + 3 * n);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

// xc[c] = x[rows[c]] (c < *count, bf16 rows of K); xc and dz are zeroed from there up to the next multiple of 64 rows, dz to its last row
// (dz_rows) at most.  xc has room for n rounded up to 64 rows.
extern "C" int prl_gather_live_rows(const void* x, int64_t n, int64_t K, const int32_t* rows, const int32_t* count, void* xc, void* dz,
                                    int64_t dz_rows, int64_t V, int64_t ld_dz, prl_stream_t stream_) {
  PRL_CHECK_ARG(x && rows && count && xc && dz, "prl_gather_live_rows: NULL argument");
  PRL_CHECK_ARG(n >= 1 && K >= 8 && K % 8 == 0 && V >= 1 && ld_dz >= V, "prl_gather_live_rows: bad shape");
  PRL_CHECK_ARG((((uintptr_t)x | (uintptr_t)xc) & 15) == 0, "prl_gather_live_rows: rows must be 16-byte aligned");
  gather_rows_kernel<<<(unsigned)((n + 63) / 64 * 64), 256, 0, (cudaStream_t)stream_>>>((const uint4*)x, rows, count, K / 8, (uint4*)xc,
                                                                                         (__nv_bfloat16*)dz, dz_rows, V, ld_dz);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

// out[r] = src[place[r]] for n bf16 rows of K, zeros where place[r] is -1
extern "C" int prl_spread_rows(const void* src, const int32_t* place, int64_t n, int64_t K, void* out, prl_stream_t stream_) {
  PRL_CHECK_ARG(src && place && out, "prl_spread_rows: NULL argument");
  PRL_CHECK_ARG(n >= 1 && K >= 8 && K % 8 == 0, "prl_spread_rows: bad shape");
  PRL_CHECK_ARG((((uintptr_t)src | (uintptr_t)out) & 15) == 0, "prl_spread_rows: rows must be 16-byte aligned");
  spread_rows_kernel<<<(unsigned)n, 256, 0, (cudaStream_t)stream_>>>((const uint4*)src, place, K / 8, (uint4*)out);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

// d loss / d logits (bf16) of row rows[c] into the first half of row c of the logits that prl_head_logprob_keep left: a [n, V] matrix of
// row stride 2 ld_logits
extern "C" int prl_head_dlogits_kept(float* logits, int64_t ld_logits, int64_t n, int64_t V, float temperature, const int32_t* rows,
                                     const int32_t* count, const int64_t* targets, const float* lse, const float* entropy,
                                     const float* g_logprobs, const float* g_entropy, prl_stream_t stream_) {
  PRL_CHECK_ARG(logits && rows && count && targets && lse, "prl_head_dlogits_kept: NULL argument");
  PRL_CHECK_ARG(n >= 1 && V >= 8 && V % 8 == 0 && ld_logits >= V && ld_logits % 4 == 0 && ((uintptr_t)logits & 15) == 0 && temperature > 0.f,
                "prl_head_dlogits_kept: bad shape (rows of a multiple of 8 logits that start on 16 bytes)");
  PRL_CHECK_ARG(!g_entropy || entropy, "prl_head_dlogits_kept: g_entropy needs the forward entropy");
  dlogits_kept_kernel<<<(unsigned)n, kThreads, 0, (cudaStream_t)stream_>>>(logits, ld_logits, V, rows, count, targets, 1.f / temperature,
                                                                           lse, entropy, g_logprobs, g_entropy);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}
