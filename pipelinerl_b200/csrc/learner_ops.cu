// Row-wise kernels of the learner body (hot path 2): everything between the GEMMs of the Qwen2 forward / backward
// that the reference runs as HF eager modules under autograd (pipelinerl/finetune/rl/__init__.py:190-207 reached
// through transformers' Qwen2RMSNorm / apply_rotary_pos_emb / Qwen2MLP; backward finetune_loop.py:716-725).
// All of them are HBM-bound: one pass over the activations, bf16 in / bf16 out, fp32 arithmetic, 16-byte accesses.
// Reductions over the token dimension (RMSNorm gain, qkv bias) are two-stage with a FIXED order: per-block partial
// rows in a workspace, then one pass that adds them into the fp32 gradient arena -> bitwise reproducible.
#include "prl_common.cuh"
#include "tc_ptx.cuh"

namespace prl {
namespace {

constexpr int kRowThreads = 256;
constexpr int kMaxVec = 4;          // 8-element vectors per thread -> rows of up to 8192 elements
constexpr int kPartialBlocks = 148 * 8; // most blocks of a persistent row kernel = rows of the partial workspace

struct Vec8 { float v[8]; };

__device__ __forceinline__ Vec8 load8(const __nv_bfloat16* p) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
  Vec8 r;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = __bfloat1622float2(h[e]);
    r.v[2 * e] = f.x;
    r.v[2 * e + 1] = f.y;
  }
  return r;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const Vec8& r) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(r.v[2 * e], r.v[2 * e + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}

__device__ __forceinline__ Vec8 unpack8(const uint4& u) {
  Vec8 r;
  const uint32_t h[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    r.v[2 * e] = __uint_as_float(h[e] << 16);
    r.v[2 * e + 1] = __uint_as_float(h[e] & 0xFFFF0000u);
  }
  return r;
}
// sum over the block; the caller alternates between two s_red buffers, so one barrier serves
__device__ __forceinline__ float block_sum(float v, float* s_red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int w = 0; w < kRowThreads / 32; ++w) t += w < (int)(blockDim.x >> 5) ? s_red[w] : 0.f;
  return t;
}

// The row kernels are bound by HBM.  A block walks its rows with the next row already asked for (registers, raw bf16) while the
// current one goes through its block sum: without that the reads stop at every row's barrier (16384 x 3584: backward 170 us,
// 0.42 of the copy rate).  A narrow row's block has just the threads that it fills (row_threads), and the grid
// just the blocks that are resident at once.  With the faster column sums below: 16384 x 3584 forward 49 -> 47 us, backward
// 214 -> 87 us (5.4 TB/s, cold L2); 4096 x 5120 27 -> 21, 150 -> 44; 16384 x 1024 25 -> 21, 79 -> 38.
template <int kVec>
__device__ __forceinline__ void load_row(const __nv_bfloat16* __restrict__ p, int64_t row, int H, uint4 (&r)[kVec]) {
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < (H >> 3)) r[i] = ld_stream_u4(reinterpret_cast<const uint4*>(p + row * H) + v);
  }
}

// The backward's rows of up to three matrices on their way into shared memory, `slots` rows of the block's walk ahead: a thread asks for whole rows
// (bulk copies), so what is under way does not hang on the registers (one row ahead: 48 KB an SM).  A row's slot is asked for again
// once the block's sum has brought all threads past their reads.
struct RowRing {
  uint32_t data, bars;
  uint32_t row_bytes, slot_bytes;
  int slots, mats;
  const __nv_bfloat16* src[3];
  __device__ __forceinline__ void ask(int64_t row, int H, int s) const {        // one thread
    const uint32_t bar = bars + 8u * (uint32_t)s;
    ptx::mbar_arrive_expect_tx(bar, row_bytes * (uint32_t)mats);
    for (int m = 0; m < mats; ++m)
      ptx::bulk_load_1d(data + (uint32_t)s * slot_bytes + (uint32_t)m * row_bytes, src[m] + row * H, row_bytes, bar, ptx::kEvictFirst);
  }
  __device__ __forceinline__ void start(int64_t T, int H) const {
    if (threadIdx.x == 0) {
      for (int s = 0; s < slots; ++s) ptx::mbar_init(bars + 8u * (uint32_t)s, 1);
      ptx::fence_barrier_init();
      ptx::fence_proxy_async();
      int64_t row = blockIdx.x;
      for (int s = 0; s < slots && row < T; ++s, row += gridDim.x) ask(row, H, s);
    }
    __syncthreads();
  }
  template <int kVec>
  __device__ __forceinline__ void get(int s, int m, int nvec, uint4 (&r)[kVec]) const {
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (v < nvec)
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[i].x), "=r"(r[i].y), "=r"(r[i].z), "=r"(r[i].w)
                     : "r"(data + (uint32_t)s * slot_bytes + (uint32_t)m * row_bytes + (uint32_t)v * 16u) : "memory");
    }
  }
};
__device__ __forceinline__ RowRing row_ring(uint8_t* raw, int H, int slots, int mats) {
  RowRing r;
  const uint32_t base = (ptx::smem_u32(raw) + 127u) & ~127u;
  r.bars = base;
  r.data = base + 128u;
  r.row_bytes = 2u * (uint32_t)H;
  r.slot_bytes = r.row_bytes * (uint32_t)mats;
  r.slots = slots;
  r.mats = mats;
  return r;
}

// y = bf16(x * rstd) * gamma  (the rounding order of HF's Qwen2RMSNorm); rstd kept for the backward
template <int kVec>
__global__ void __launch_bounds__(kRowThreads) rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                                  const __nv_bfloat16* __restrict__ gamma, int64_t T,
                                                                  int H, float eps, __nv_bfloat16* __restrict__ y,
                                                                  float* __restrict__ rstd) {
  __shared__ float s_red[2][kRowThreads / 32];
  const int nvec = H >> 3;
  uint4 g[kVec], next[kVec];
  load_row<kVec>(gamma, 0, H, g);
  load_row<kVec>(x, blockIdx.x, H, next);
  int buf = 0;
  for (int64_t row = blockIdx.x; row < T; row += gridDim.x, buf ^= 1) {
    uint4 xr[kVec];
#pragma unroll
    for (int i = 0; i < kVec; ++i) xr[i] = next[i];
    if (row + gridDim.x < T) load_row<kVec>(x, row + gridDim.x, H, next);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      if (threadIdx.x + i * blockDim.x < nvec) {
        const Vec8 xv = unpack8(xr[i]);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += xv.v[e] * xv.v[e];
      }
    }
    const float r = rsqrtf(block_sum(ss, s_red[buf]) / (float)H + eps);
    if (threadIdx.x == 0) rstd[row] = r;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        const Vec8 xv = unpack8(xr[i]), gv = unpack8(g[i]);
        Vec8 o;
#pragma unroll
        for (int e = 0; e < 8; ++e) o.v[e] = __bfloat162float(__float2bfloat16(xv.v[e] * r)) * gv.v[e];
        store8(y + row * H + v * 8, o);
      }
    }
  }
}

// dx = dres + rstd * (dy*gamma - xhat * mean(dy*gamma*xhat));  partial[block][c] = sum over this block's rows of dy*xhat
template <int kVec, bool kRing>
__global__ void __launch_bounds__(kRowThreads, kVec == 1 ? 4 : (kVec == 2 ? 2 : 1))
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma, const float* __restrict__ rstd,
                   const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ dres, int64_t T, int H,
                   __nv_bfloat16* __restrict__ dx, float* __restrict__ partial, int slots) {
  extern __shared__ uint8_t row_raw[];
  __shared__ float s_red[2][kRowThreads / 32];
  const int nvec = H >> 3;
  uint4 g[kVec], xn[kVec], dn[kVec], sn[kVec];
  Vec8 acc[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    sn[i] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[i].v[e] = 0.f;
  }
  RowRing ring = row_ring(row_raw, H, slots, dres ? 3 : 2);
  ring.src[0] = x;
  ring.src[1] = dy;
  ring.src[2] = dres;
  if (kRing) ring.start(T, H);
  load_row<kVec>(gamma, 0, H, g);
  if (!kRing) {
    load_row<kVec>(x, blockIdx.x, H, xn);
    load_row<kVec>(dy, blockIdx.x, H, dn);
    if (dres) load_row<kVec>(dres, blockIdx.x, H, sn);
  }
  float rn = rstd[blockIdx.x];
  int buf = 0, slot = 0;
  uint32_t ph = 0;
  for (int64_t row = blockIdx.x; row < T; row += gridDim.x, buf ^= 1) {
    uint4 xr[kVec], dr[kVec], sr[kVec];
    const float r = rn;
    const int64_t nx = row + gridDim.x;
    if constexpr (kRing) {
#pragma unroll
      for (int i = 0; i < kVec; ++i) sr[i] = sn[i];
      if (nx < T) rn = rstd[nx];
      ptx::mbar_wait(ring.bars + 8u * (uint32_t)slot, ph);
      ring.get<kVec>(slot, 0, nvec, xr);
      ring.get<kVec>(slot, 1, nvec, dr);
      if (dres) ring.get<kVec>(slot, 2, nvec, sr);
    } else {
#pragma unroll
      for (int i = 0; i < kVec; ++i) { xr[i] = xn[i]; dr[i] = dn[i]; sr[i] = sn[i]; }
      if (nx < T) {
        load_row<kVec>(x, nx, H, xn);
        load_row<kVec>(dy, nx, H, dn);
        if (dres) load_row<kVec>(dres, nx, H, sn);
        rn = rstd[nx];
      }
    }
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      if (threadIdx.x + i * blockDim.x < nvec) {
        const Vec8 xv = unpack8(xr[i]), dv = unpack8(dr[i]), gv = unpack8(g[i]);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = xv.v[e] * r;
          acc[i].v[e] += dv.v[e] * xh;
          dot += dv.v[e] * gv.v[e] * xh;
        }
      }
    }
    const float m = block_sum(dot, s_red[buf]) / (float)H;
    if constexpr (kRing) {
      const int64_t ahead = row + (int64_t)ring.slots * gridDim.x;
      if (threadIdx.x == 0 && ahead < T) ring.ask(ahead, H, slot);
      if (++slot == ring.slots) { slot = 0; ph ^= 1u; }
    }
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        const Vec8 xv = unpack8(xr[i]), dv = unpack8(dr[i]), gv = unpack8(g[i]), sv = unpack8(sr[i]);
        Vec8 o;
#pragma unroll
        for (int e = 0; e < 8; ++e)    // contracted by hand, so that the bits don't hang on how the loop is compiled
          o.v[e] = __fmul_rn(r, fmaf(-(xv.v[e] * r), m, dv.v[e] * gv.v[e]));
        if (dres) {
#pragma unroll
          for (int e = 0; e < 8; ++e) o.v[e] = __fadd_rn(o.v[e], sv.v[e]);
        }
        store8(dx + row * H + v * 8, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      float* pp = partial + (int64_t)blockIdx.x * H + v * 8;
      *reinterpret_cast<float4*>(pp) = make_float4(acc[i].v[0], acc[i].v[1], acc[i].v[2], acc[i].v[3]);
      *reinterpret_cast<float4*>(pp + 4) = make_float4(acc[i].v[4], acc[i].v[5], acc[i].v[6], acc[i].v[7]);
    }
  }
}

template <int kVec>
__global__ void __launch_bounds__(kRowThreads) colsum_kernel(const __nv_bfloat16* __restrict__ x, int64_t ld, int64_t T,
                                                             int Cc, float* __restrict__ partial) {
  const int nvec = Cc >> 3;
  Vec8 acc[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[i].v[e] = 0.f;
  for (int64_t row = blockIdx.x; row < T; row += gridDim.x) {
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int v = threadIdx.x + i * kRowThreads;
      if (v < nvec) {
        const Vec8 d = load8(x + row * ld + v * 8);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[i].v[e] += d.v[e];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int v = threadIdx.x + i * kRowThreads;
    if (v < nvec) {
      float* pp = partial + (int64_t)blockIdx.x * Cc + v * 8;
      *reinterpret_cast<float4*>(pp) = make_float4(acc[i].v[0], acc[i].v[1], acc[i].v[2], acc[i].v[3]);
      *reinterpret_cast<float4*>(pp + 4) = make_float4(acc[i].v[4], acc[i].v[5], acc[i].v[6], acc[i].v[7]);
    }
  }
}

// out[c] += sum_b partial[b][c]: warp w of a block adds rows w, w + 16, ... of the block's 32 columns, then the warps' sums are
// added in order (one fixed order).  One thread per column walking all the rows took 36 us for 592 x 3584.
constexpr int kReduceWarps = 16;
__global__ void __launch_bounds__(32 * kReduceWarps) partial_reduce_kernel(const float* __restrict__ partial, int n_blocks, int Cc,
                                                                          float* __restrict__ out) {
  __shared__ float s_sum[kReduceWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 32 + lane;
  pdl_wait();
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < Cc) {
    int b = warp;
    for (; b + 3 * kReduceWarps < n_blocks; b += 4 * kReduceWarps) {
#pragma unroll
      for (int k = 0; k < 4; ++k) s[k] += partial[(int64_t)(b + k * kReduceWarps) * Cc + c];
    }
    for (; b < n_blocks; b += kReduceWarps) s[0] += partial[(int64_t)b * Cc + c];
  }
  s_sum[warp][lane] = (s[0] + s[1]) + (s[2] + s[3]);
  __syncthreads();
  if (warp == 0 && c < Cc) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kReduceWarps; ++w) t += s_sum[w][lane];
    out[c] += t;
  }
}

// in-place rotation of the first n_heads heads of each row: (x1, x2) -> (x1 cos - s x2 sin, x2 cos + s x1 sin)
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, int64_t ld, int64_t T, int n_heads, int head_dim,
                            const int32_t* __restrict__ pos, const float* __restrict__ inv_freq, float sign) {
  extern __shared__ float s_cs[];  // [half] cos, [half] sin
  const int half = head_dim >> 1;
  const int per_head = half >> 3;  // threads per head (8 pairs each)
  for (int64_t row = blockIdx.x; row < T; row += gridDim.x) {
    __syncthreads();
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
      float sn, cs;
      sincosf((float)pos[row] * inv_freq[i], &sn, &cs);
      s_cs[i] = cs;
      s_cs[half + i] = sn * sign;
    }
    __syncthreads();
    for (int w = threadIdx.x; w < n_heads * per_head; w += blockDim.x) {
      const int head = w / per_head, i0 = (w % per_head) * 8;
      __nv_bfloat16* p = x + row * ld + (int64_t)head * head_dim + i0;
      const Vec8 a = load8(p), b = load8(p + half);
      Vec8 oa, ob;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float cs = s_cs[i0 + e], sn = s_cs[half + i0 + e];
        oa.v[e] = a.v[e] * cs - b.v[e] * sn;
        ob.v[e] = b.v[e] * cs + a.v[e] * sn;
      }
      store8(p, oa);
      store8(p + half, ob);
    }
  }
}

// kLines: eight rows of at most 256 features per block, a warp each; else a row per block or blocks
template <bool kLines>
__global__ void __launch_bounds__(256) silu_mul_fwd_kernel(const __nv_bfloat16* __restrict__ gu, int64_t T, int I,
                                                           __nv_bfloat16* __restrict__ act) {
  const int64_t row = kLines ? (int64_t)blockIdx.x * 8 + threadIdx.y : blockIdx.x;   // no division per element
  if (kLines && row >= T) return;
  const __nv_bfloat16* gp = gu + row * 2 * I;
  for (int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8; c < I; c += gridDim.y * blockDim.x * 8) {
    const Vec8 g = unpack8(ld_stream_u4(reinterpret_cast<const uint4*>(gp + c)));
    const Vec8 u = unpack8(ld_stream_u4(reinterpret_cast<const uint4*>(gp + I + c)));
    Vec8 o;
#pragma unroll
    for (int e = 0; e < 8; ++e) o.v[e] = div_ge1(g.v[e], 1.f + __expf(-g.v[e])) * u.v[e];
    store8(act + row * I + c, o);
  }
}

// kAct: the forward's activation is made again beside it (the operand of down_proj's weight gradient), in place of d act: read through
// the coherent path, each piece by the thread that writes it.  HBM-bound either way, with one reading of gate_up
// less: 4096 x 18944, forward and backward in two launches 201.6 us, in one 149.9 (6.2 TB/s; the backward alone 125.3).
template <bool kLines, bool kAct>
__global__ void __launch_bounds__(256) silu_mul_bwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* dact, int64_t T, int I,
                                                           __nv_bfloat16* __restrict__ dgu) {
  const int64_t row = kLines ? (int64_t)blockIdx.x * 8 + threadIdx.y : blockIdx.x;
  if (kLines && row >= T) return;
  const __nv_bfloat16* gp = gu + row * 2 * I;
  for (int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8; c < I; c += gridDim.y * blockDim.x * 8) {
    const Vec8 g = unpack8(ld_stream_u4(reinterpret_cast<const uint4*>(gp + c)));
    const Vec8 u = unpack8(ld_stream_u4(reinterpret_cast<const uint4*>(gp + I + c)));
    __nv_bfloat16* dp = dact + row * I + c;
    uint4 dr;
    if constexpr (kAct)
      asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(dr.x), "=r"(dr.y), "=r"(dr.z), "=r"(dr.w) : "l"(dp) : "memory");
    else
      dr = ld_stream_u4(reinterpret_cast<const uint4*>(dp));
    const Vec8 d = unpack8(dr);
    Vec8 dg, du, o;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float b = 1.f + __expf(-g.v[e]), s = div_ge1(1.f, b);
      const float silu = g.v[e] * s;
      du.v[e] = d.v[e] * silu;
      dg.v[e] = d.v[e] * u.v[e] * (s + silu * (1.f - s));
      if (kAct) o.v[e] = div_ge1(g.v[e], b) * u.v[e];      // the forward's rounding, not that of `silu`
    }
    store8(dgu + row * 2 * I + c, dg);
    store8(dgu + row * 2 * I + I + c, du);
    if (kAct) store8(dp, o);
  }
}

__global__ void __launch_bounds__(256) embed_gather_kernel(const __nv_bfloat16* __restrict__ table,
                                                           const int64_t* __restrict__ ids, int64_t T, int H,
                                                           __nv_bfloat16* __restrict__ out) {
  const int nvec = H >> 3;
  for (int64_t row = blockIdx.x; row < T; row += gridDim.x) {
    const int64_t id = ids[row];
    for (int v = threadIdx.x; v < nvec; v += blockDim.x)
      *reinterpret_cast<uint4*>(out + row * H + v * 8) = *reinterpret_cast<const uint4*>(table + id * H + v * 8);
  }
}

// kVec: four sums per access, on tables that start on 16 bytes (rows of a multiple of 8 numbers keep that); else one by one
template <bool kVec>
__global__ void __launch_bounds__(256) embed_scatter_kernel(float* __restrict__ dtable, const int64_t* __restrict__ ids,
                                                            const __nv_bfloat16* __restrict__ dh, int64_t T, int H) {
  const int nvec = H >> 3;
  for (int64_t row = blockIdx.x; row < T; row += gridDim.x) {
    const int64_t id = ids[row];
    for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
      const Vec8 d = load8(dh + row * H + v * 8);
      float* to = dtable + id * H + v * 8;
      if constexpr (kVec) {
        atomicAdd(reinterpret_cast<float4*>(to), make_float4(d.v[0], d.v[1], d.v[2], d.v[3]));
        atomicAdd(reinterpret_cast<float4*>(to + 4), make_float4(d.v[4], d.v[5], d.v[6], d.v[7]));
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) atomicAdd(to + e, d.v[e]);
      }
    }
  }
}

__global__ void __launch_bounds__(256) quotient_kernel(const float* __restrict__ a, const float* __restrict__ b, int64_t n,
                                                       float* __restrict__ q) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) q[i] = div_ge1(a[i], b[i]);
}

// rows of up to a warp's 32 pieces share a block: with a block each, 16384 rows of 128 features took 9.7 us forward, so 4.8
bool silu_lines(int64_t I) { return I <= 256; }
int silu_threads(int64_t I) {
  const int64_t n = (I + 7) / 8;
  return n >= 256 ? 256 : (int)((n + 31) / 32 * 32);
}
dim3 silu_grid(int64_t T, int64_t I) {   // a block per row; few rows are cut, so that eight blocks per SM are there
  const int64_t pieces = (I / 8 + silu_threads(I) - 1) / silu_threads(I), want = ((int64_t)num_sms() * 8 + T - 1) / T;
  return dim3((unsigned)T, (unsigned)(want < pieces ? want : pieces));
}
int row_grid(int64_t T) { return (int)(T < kPartialBlocks / 2 ? T : kPartialBlocks / 2); }
int row_vecs(int64_t H) { return (int)((H / 8 + kRowThreads - 1) / kRowThreads); }                       // 16-byte pieces per thread
// Threads of a row's block: as many as one piece each needs, all of them where a thread holds several.  Thread t then adds pieces
// t, t + 256, ... whatever the width, so a row's sum has one order.  With 224 threads for 3584 (two pieces each, none idle) the
// last bit of some rstd moved, and with it single bf16 values of everything behind the norm.
int row_threads(int64_t H) { return row_vecs(H) > 1 ? kRowThreads : (int)((H / 8 + 31) / 32 * 32); }
// resident blocks of the backward: two of 256 threads with 128 registers each per SM, or the threads' worth of narrow rows
int row_bwd_grid(int64_t T, int64_t H) {
  const int per_sm = row_vecs(H) == 1 ? 1024 / row_threads(H) : (row_vecs(H) == 2 ? 2 : 1);
  const int64_t n = (int64_t)num_sms() * (per_sm < 8 ? per_sm : 8);
  const int64_t most = n < kPartialBlocks ? n : kPartialBlocks;
  return (int)(T < most ? T : most);
}
// Slots of the backward's ring: what an SM's shared memory holds beside its other blocks, 16 at most; 0: rows through registers.  The ring pays
// where a block has many rows to be ahead of (it costs a start, and the SM another split of its L1) and rows are whole lines.  Rows, registers /
// ring, us: 3584 channels (two blocks an SM) 4096 25.0 / 27.9, 8192 43.5 / 43.9, 12000 63.9 / 62.0, 16384 84.0 / 81.0, 32768 158 / 150; 5120 (one) 4096 35.1 / 37.2,
// 6000 51.6 / 49.5, 16384 132 / 118; 2048 (four) 4096 20.8 / 20.9, 6000 26.9 / 26.0, 16384 55.8 / 51.9; 128 12000 18.7 / 16.7; 2056 16384 65.6 / 67.8; 4096,
// where two blocks have four slots each, 32768 173 / 177; 384 and 512 (two warps a block) 14000 19.5 / 20.7 and 20.1 / 21.2, 24000 27.1 / 28.5 and
// 28.2 / 28.8, 60000 55.9 / 56.2 and 62.7 / 57.0; 640 (three) 14000 24.4 / 24.6, 24000 35.3 / 34.4; 1024 (four) 14000 29.4 / 28.3.
// The forward lost throughout (16384 x 3584 43.4 / 46.1): one row in flight a block was enough.
int ring_slots(int64_t T, int64_t H, int64_t grid, int mats) {
  const int vecs = row_vecs(H), warps = row_threads(H) / 32;
  if (H % 64 != 0 || T < (vecs > 1 ? 40 : warps == 2 ? 50 : warps == 3 ? 20 : 10) * grid) return 0;
  const int64_t per_sm = (grid + num_sms() - 1) / num_sms(), n = (216 * 1024 / per_sm - 1536) / (2 * H * mats);
  return (int)(n < (vecs == 2 ? 5 : 4) ? 0 : n > 16 ? 16 : n);
}
int ring_bytes(int64_t H, int slots, int mats) { return slots ? (int)(256 + 2 * H * mats * slots) : 0; }
cudaError_t launch_partial_reduce(const float* ws, int blocks, int64_t cols, float* out, cudaStream_t stream) {
  return launch_pdl(partial_reduce_kernel, dim3((unsigned)((cols + 31) / 32)), dim3(32 * kReduceWarps), 0, stream, ws, blocks, (int)cols, out);
}

}  // namespace
}  // namespace prl

using namespace prl;

extern "C" size_t prl_rowops_workspace_bytes(int64_t cols) { return (size_t)kPartialBlocks * (size_t)cols * sizeof(float); }

#define PRL_ROW_ARGS(name, H)                                                                                       \
  PRL_CHECK_ARG((H) >= 8 && (H) % 8 == 0 && (H) <= kRowThreads * kMaxVec * 8, name ": row length must be a multiple " \
                "of 8 in [8, 8192] (got %lld)", (long long)(H))

extern "C" int prl_rmsnorm_fwd(const void* x, const void* gamma, int64_t T, int64_t H, float eps, void* y, float* rstd,
                               prl_stream_t stream) {
  PRL_CHECK_ARG(x && gamma && y && rstd && T >= 1, "prl_rmsnorm_fwd: bad argument");
  PRL_ROW_ARGS("prl_rmsnorm_fwd", H);
  const int threads = row_threads(H);
  const int64_t most = (int64_t)num_sms() * (row_vecs(H) == 4 ? 3 : 1024 / threads);   // resident at once: 80 registers a thread for four pieces
  const unsigned grid = (unsigned)(T < most ? T : most);
#define PRL_FWD(V) rmsnorm_fwd_kernel<V><<<grid, threads, 0, (cudaStream_t)stream>>>( \
      (const __nv_bfloat16*)x, (const __nv_bfloat16*)gamma, T, (int)H, eps, (__nv_bfloat16*)y, rstd)
  switch (row_vecs(H)) { case 1: PRL_FWD(1); break; case 2: PRL_FWD(2); break; case 3: PRL_FWD(3); break; default: PRL_FWD(4); }
#undef PRL_FWD
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

extern "C" int prl_rmsnorm_bwd(const void* x, const void* gamma, const float* rstd, const void* dy, const void* dres,
                               int64_t T, int64_t H, void* dx, float* dgamma, void* workspace, size_t workspace_bytes,
                               prl_stream_t stream) {
  PRL_CHECK_ARG(x && gamma && rstd && dy && dx && dgamma && workspace && T >= 1, "prl_rmsnorm_bwd: bad argument");
  PRL_ROW_ARGS("prl_rmsnorm_bwd", H);
  PRL_CHECK_ARG(workspace_bytes >= prl_rowops_workspace_bytes(H), "prl_rmsnorm_bwd: workspace too small");
  const int g = row_bwd_grid(T, H), threads = row_threads(H);
  const int mats = dres ? 3 : 2;
  const int slots = ring_slots(T, H, g, mats), smem = ring_bytes(H, slots, mats);
#define PRL_BWD_(V, RING)                                                                                                         \
  do {                                                                                                                            \
    static SmemAttr attr = {};                                                                                                    \
    if (RING) PRL_CUDA(ensure_smem((rmsnorm_bwd_kernel<V, RING>), smem, attr));                                                   \
    rmsnorm_bwd_kernel<V, RING><<<g, threads, smem, (cudaStream_t)stream>>>(                                                      \
        (const __nv_bfloat16*)x, (const __nv_bfloat16*)gamma, rstd, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)dres, T,      \
        (int)H, (__nv_bfloat16*)dx, (float*)workspace, slots);                                                                    \
  } while (0)
#define PRL_BWD(V) do { if (slots) PRL_BWD_(V, true); else PRL_BWD_(V, false); } while (0)
  switch (row_vecs(H)) { case 1: PRL_BWD(1); break; case 2: PRL_BWD(2); break; case 3: PRL_BWD(3); break; default: PRL_BWD(4); }
#undef PRL_BWD
#undef PRL_BWD_
  PRL_LAUNCH_CHECK();
  PRL_CUDA(launch_partial_reduce((const float*)workspace, g, H, dgamma, (cudaStream_t)stream));
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

extern "C" int prl_colsum_bf16(const void* x, int64_t ld, int64_t T, int64_t cols, float* out, void* workspace,
                               size_t workspace_bytes, prl_stream_t stream) {
  PRL_CHECK_ARG(x && out && workspace && T >= 1 && ld >= cols && ld % 8 == 0, "prl_colsum_bf16: bad argument");
  PRL_ROW_ARGS("prl_colsum_bf16", cols);
  PRL_CHECK_ARG(workspace_bytes >= prl_rowops_workspace_bytes(cols), "prl_colsum_bf16: workspace too small");
  const int g = row_grid(T);
#define PRL_CS(V) colsum_kernel<V><<<g, kRowThreads, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, ld, T, (int)cols, \
                                                                            (float*)workspace)
  if (cols <= 2048) PRL_CS(1); else if (cols <= 4096) PRL_CS(2); else PRL_CS(4);
#undef PRL_CS
  PRL_LAUNCH_CHECK();
  PRL_CUDA(launch_partial_reduce((const float*)workspace, g, cols, out, (cudaStream_t)stream));
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

extern "C" int prl_rope_inplace(void* x, int64_t ld, int64_t T, int32_t n_heads, int32_t head_dim, const int32_t* pos,
                                const float* inv_freq, float sign, prl_stream_t stream) {
  PRL_CHECK_ARG(x && pos && inv_freq && T >= 1 && n_heads >= 1, "prl_rope_inplace: bad argument");
  PRL_CHECK_ARG(head_dim >= 16 && head_dim % 16 == 0 && head_dim <= 512 && ld % 8 == 0 && ld >= (int64_t)n_heads * head_dim,
                "prl_rope_inplace: head_dim must be a multiple of 16 and ld a multiple of 8 covering the rotated heads");
  int threads = n_heads * (head_dim / 16);
  threads = threads > 256 ? 256 : ((threads + 31) / 32 * 32);
  rope_kernel<<<(unsigned)(T < 4 * kPartialBlocks ? T : 4 * kPartialBlocks), threads, (size_t)head_dim * sizeof(float),
                (cudaStream_t)stream>>>((__nv_bfloat16*)x, ld, T, n_heads, head_dim, pos, inv_freq, sign);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

extern "C" int prl_silu_mul_fwd(const void* gate_up, int64_t T, int64_t I, void* act, prl_stream_t stream) {
  PRL_CHECK_ARG(gate_up && act && T >= 1 && I >= 8 && I % 8 == 0, "prl_silu_mul_fwd: bad argument (I %% 8 == 0)");
  if (silu_lines(I))
    silu_mul_fwd_kernel<true><<<(unsigned)((T + 7) / 8), dim3(32, 8), 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)gate_up, T, (int)I,
                                                                                                 (__nv_bfloat16*)act);
  else
    silu_mul_fwd_kernel<false><<<silu_grid(T, I), silu_threads(I), 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)gate_up, T, (int)I,
                                                                                              (__nv_bfloat16*)act);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

template <bool kAct>
static int silu_mul_bwd_impl(const void* gate_up, void* dact, int64_t T, int64_t I, void* dgate_up, prl_stream_t stream) {
  PRL_CHECK_ARG(gate_up && dact && dgate_up && T >= 1 && I >= 8 && I % 8 == 0, "prl_silu_mul_bwd: bad argument");
  const auto kernel = silu_lines(I) ? silu_mul_bwd_kernel<true, kAct> : silu_mul_bwd_kernel<false, kAct>;
  const dim3 grid = silu_lines(I) ? dim3((unsigned)((T + 7) / 8)) : silu_grid(T, I), block = silu_lines(I) ? dim3(32, 8) : dim3(silu_threads(I));
  kernel<<<grid, block, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)gate_up, (__nv_bfloat16*)dact, T, (int)I, (__nv_bfloat16*)dgate_up);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}
extern "C" int prl_silu_mul_bwd(const void* gate_up, const void* dact, int64_t T, int64_t I, void* dgate_up,
                                prl_stream_t stream) {
  return silu_mul_bwd_impl<false>(gate_up, const_cast<void*>(dact), T, I, dgate_up, stream);
}
extern "C" int prl_silu_mul_bwd_act(const void* gate_up, void* dact, int64_t T, int64_t I, void* dgate_up, prl_stream_t stream) {
  return silu_mul_bwd_impl<true>(gate_up, dact, T, I, dgate_up, stream);
}

extern "C" int prl_embed_gather(const void* table, const int64_t* ids, int64_t T, int64_t H, void* out,
                                prl_stream_t stream) {
  PRL_CHECK_ARG(table && ids && out && T >= 1 && H >= 8 && H % 8 == 0, "prl_embed_gather: bad argument");
  embed_gather_kernel<<<(unsigned)(T < 4096 ? T : 4096), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)table, ids, T,
                                                                                         (int)H, (__nv_bfloat16*)out);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

extern "C" int prl_embed_scatter_add(float* dtable, const int64_t* ids, const void* dh, int64_t T, int64_t H,
                                     prl_stream_t stream) {
  PRL_CHECK_ARG(dtable && ids && dh && T >= 1 && H >= 8 && H % 8 == 0, "prl_embed_scatter_add: bad argument");
  PRL_CHECK_ARG(((uintptr_t)dtable & 3) == 0 && ((uintptr_t)dh & 15) == 0, "prl_embed_scatter_add: dh must start on 16 bytes, dtable on 4");
  const auto kernel = ((uintptr_t)dtable & 15) == 0 ? embed_scatter_kernel<true> : embed_scatter_kernel<false>;
  kernel<<<(unsigned)(T < 4096 ? T : 4096), 256, 0, (cudaStream_t)stream>>>(dtable, ids, (const __nv_bfloat16*)dh, T, (int)H);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}

extern "C" int prl_debug_quotient(const float* a, const float* b, int64_t n, float* q, prl_stream_t stream) {
  PRL_CHECK_ARG(a && b && q && n >= 1, "prl_debug_quotient: bad argument");
  quotient_kernel<<<(unsigned)(n < 256 * 4096 ? (n + 255) / 256 : 4096), 256, 0, (cudaStream_t)stream>>>(a, b, n, q);
  PRL_LAUNCH_CHECK();
  return PRL_OK;
}
