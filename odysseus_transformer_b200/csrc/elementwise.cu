// Memory-bound hot ops for sm_100a: RMSNorm(+residual) fwd/bwd, RoPE, SwiGLU fwd/bwd, cross-entropy
// fwd / in-place bwd, fused AdamW over flat shards, attention partial-result merge.
//
// The reference gets these from unfused ATen elementwise kernels inside HF Llama, a Triton loss from
// flash-attn and torch.optim.AdamW (reference train.py:167,173; decoder/odysseus.py:210-213,293-295).
// Every kernel here moves 16 bytes per thread per access and touches each operand once.
#include <float.h>
#include <string.h>

#include <atomic>

#include "common.cuh"
#include "launch.cuh"
#include "ody_kernels.h"
#include "sm100.cuh"

namespace ody {

// ------------------------------------------------------------------------------------------- RMSNorm

template <int NV>
__global__ void __launch_bounds__(256) rmsnorm_fwd_k(const bf16* __restrict__ x, const bf16* __restrict__ delta,
                                                     const bf16* __restrict__ w, bf16* __restrict__ sum_out,
                                                     bf16* __restrict__ y, float* __restrict__ rstd, int dim,
                                                     float eps) {
  after_previous_kernel(x, delta, w);
  __shared__ float red[33];
  const int64_t row = blockIdx.x;
  const bf16* xr = x + row * dim;
  float vals[NV][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 8;
    if (c < dim) {
      bf16x8 p = ld8(xr + c);
      if (delta != nullptr) {
        float a[8], b[8];
        unpack8(p, a);
        unpack8(ld8(delta + row * dim + c), b);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] += b[j];
        p = pack8(a);  // the residual stream is stored in bf16; the norm sees the stored value
        st8(sum_out + row * dim + c, p);
      }
      unpack8(p, vals[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += vals[i][j] * vals[i][j];
    }
  }
  ss = block_sum(ss, red);
  const float rs = rsqrtf(ss / (float)dim + eps);
  if (threadIdx.x == 0) rstd[row] = rs;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 8;
    if (c < dim) {
      float wv[8], o[8];
      unpack8(ld8(w + c), wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = vals[i][j] * rs * wv[j];
      st8(y + row * dim + c, pack8(o));
    }
  }
}

// Rows wider than the ring kernel's (below): one row per iteration, one barrier (the warps' partial dot products go through a
// double-buffered shared array that every thread sums itself).  The row stays in registers as packed bf16 and is unpacked
// a second time for the output: with fp32 copies 16384 columns would spill.
template <int NV>
__global__ void __launch_bounds__(256, 1) rmsnorm_bwd_k(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                                     const bf16* __restrict__ w, const float* __restrict__ rstd,
                                                     const bf16* __restrict__ ds, bf16* __restrict__ dx,
                                                     float* __restrict__ dw_partial, int64_t rows, int dim) {
  after_previous_kernel(dy, x, w, rstd, ds);
  __shared__ __align__(16) float red[2][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float wv[NV][8], acc[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    if (c < dim) unpack8(ld8(w + c), wv[i]);
  }
  const float inv_dim = 1.f / (float)dim;
  int par = 0;
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x, par ^= 1) {
    const float rs = rstd[row];
    bf16x8 pa[NV], px[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (threadIdx.x + i * blockDim.x) * 8;
      if (c < dim) {
        pa[i] = ld8(dy + row * dim + c);
        px[i] = ld8(x + row * dim + c);
      }
    }
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (threadIdx.x + i * blockDim.x) * 8;
      if (c < dim) {
        float a[8], xh[8];
        unpack8(pa[i], a);
        unpack8(px[i], xh);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[j] *= rs;
          acc[i][j] += a[j] * xh[j];
          dot += a[j] * wv[i][j] * xh[j];
        }
      }
    }
    dot = warp_sum(dot);
    if (lane == 0) red[par][wid] = dot;
    __syncthreads();
    const float4 lo = *reinterpret_cast<const float4*>(&red[par][0]), hi = *reinterpret_cast<const float4*>(&red[par][4]);
    dot = ((lo.x + lo.y) + (lo.z + lo.w) + (hi.x + hi.y) + (hi.z + hi.w)) * inv_dim;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (threadIdx.x + i * blockDim.x) * 8;
      if (c < dim) {
        float a[8], xh[8], o[8];
        unpack8(pa[i], a);
        unpack8(px[i], xh);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (a[j] * wv[i][j] - xh[j] * rs * dot) * rs;
        if (ds != nullptr) {
          float s[8];
          unpack8(ld8(ds + row * dim + c), s);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += s[j];
        }
        st8(dx + row * dim + c, pack8(o));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 8;
    if (c < dim) {
      float* p = dw_partial + (int64_t)blockIdx.x * dim + c;
      *reinterpret_cast<float4*>(p) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      *reinterpret_cast<float4*>(p + 4) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
    }
  }
}

// Up to 8192 columns: rows fetched ahead through a ring of STAGES rows of dy, x and ds per block, filled with 16-byte asynchronous
// copies.  A thread copies exactly the elements it reads itself, so the ring needs no barrier of its own, and the loads of the
// next rows are in flight while a row's dot product waits at its barrier - which bounds a kernel that loads a row when it gets
// to it.  With the column sum below, alone: 95 -> 62 us at [8192, 4096] with ds (four 64 MB streams, 41 us at the copy rate),
// 140 -> 69 at [4096, 8192], 17 -> 15 at [512, 1024].
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int NORM_STAGES = 4;
template <int NV, bool DS>
__global__ void __launch_bounds__(256, NV <= 2 ? 2 : 1) rmsnorm_bwd_ring_k(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                                          const bf16* __restrict__ w, const float* __restrict__ rstd,
                                                          const bf16* __restrict__ ds, bf16* __restrict__ dx,
                                                          float* __restrict__ dw_partial, int64_t rows, int dim) {
  after_previous_kernel(dy, x, w, rstd, ds);
  extern __shared__ __align__(16) uint8_t ring_raw[];
  constexpr int NT = DS ? 3 : 2;
  bf16x8* ring = reinterpret_cast<bf16x8*>(ring_raw);          // [STAGES][NT][NV][256]
  __shared__ __align__(16) float red[2][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float wv[NV][8], acc[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * 256) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = wv[i][j] = 0.f;
    if (c < dim) unpack8(ld8(w + c), wv[i]);
  }
  auto fetch = [&](int64_t row, int stage) {
    if (row < rows) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = (threadIdx.x + i * 256) * 8;
        if (c < dim) {
          bf16x8* dst = ring + ((stage * NT) * NV + i) * 256 + threadIdx.x;
          cp_async16(dst, dy + row * dim + c);
          cp_async16(dst + NV * 256, x + row * dim + c);
          if (DS) cp_async16(dst + 2 * NV * 256, ds + row * dim + c);
        }
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < NORM_STAGES - 1; ++s) fetch(blockIdx.x + (int64_t)s * gridDim.x, s);
  const float inv_dim = 1.f / (float)dim;
  int par = 0, stage = 0;
  float rs = (int64_t)blockIdx.x < rows ? rstd[blockIdx.x] : 0.f;
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x, par ^= 1) {
    const int64_t next = row + gridDim.x;
    const float rs_next = next < rows ? rstd[next] : 0.f;
    cp_async_wait<NORM_STAGES - 2>();
    const bf16x8* src = ring + stage * NT * NV * 256 + threadIdx.x;
    bf16x8 pa[NV], px[NV], pd[NV];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (threadIdx.x + i * 256) * 8;
      if (c < dim) {
        pa[i] = src[i * 256];
        px[i] = src[(NV + i) * 256];
        if (DS) pd[i] = src[(2 * NV + i) * 256];
        float a[8], xh[8];
        unpack8(pa[i], a);
        unpack8(px[i], xh);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[j] *= rs;
          acc[i][j] += a[j] * xh[j];
          dot += a[j] * wv[i][j] * xh[j];
        }
      }
    }
    // the slot of the row before this one: this thread has it in registers since the last iteration
    fetch(row + (int64_t)(NORM_STAGES - 1) * gridDim.x, stage == 0 ? NORM_STAGES - 1 : stage - 1);
    dot = warp_sum(dot);
    if (lane == 0) red[par][wid] = dot;
    __syncthreads();
    const float4 lo = *reinterpret_cast<const float4*>(&red[par][0]), hi = *reinterpret_cast<const float4*>(&red[par][4]);
    dot = ((lo.x + lo.y) + (lo.z + lo.w) + (hi.x + hi.y) + (hi.z + hi.w)) * inv_dim;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = (threadIdx.x + i * 256) * 8;
      if (c < dim) {
        float a[8], xh[8], o[8];
        unpack8(pa[i], a);
        unpack8(px[i], xh);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (a[j] * wv[i][j] - xh[j] * rs * dot) * rs;
        if (DS) {
          float t[8];
          unpack8(pd[i], t);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += t[j];
        }
        st8(dx + row * dim + c, pack8(o));
      }
    }
    rs = rs_next;
    if (++stage == NORM_STAGES) stage = 0;
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * 256) * 8;
    if (c < dim) {
      float* p = dw_partial + (int64_t)blockIdx.x * dim + c;
      *reinterpret_cast<float4*>(p) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      *reinterpret_cast<float4*>(p + 4) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
    }
  }
}

// out[c] = sum over the nblocks rows of partial[nblocks, dim].  Block = 32 columns x 32 row slices: the grid has dim / 32
// blocks, and a thread adds about ten of the 296 rows - with 8 slices its chain of dependent loads was four times as long:
// 7.8 -> 3.3 us at dim 1024, 10.6 -> 4.9 at 4096.
// OUT: fp32, or bf16 for a gradient that goes straight to where the optimizer reads it.
__device__ __forceinline__ void store_sum(float* p, float v) { *p = v; }
__device__ __forceinline__ void store_sum(bf16* p, float v) { *p = __float2bfloat16_rn(v); }
template <typename OUT>
__global__ void __launch_bounds__(1024) colsum_k(const float* __restrict__ partial, OUT* __restrict__ out, int nblocks, int dim) {
  after_previous_kernel(partial);
  __shared__ float red[32][33];
  const int cx = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (c < dim) {
#pragma unroll 5
    for (int b = slice; b < nblocks; b += 32) s += partial[(int64_t)b * dim + c];
  }
  red[slice][cx] = s;
  __syncthreads();
  // warp `slice` adds up column `slice` of the block
  const float t = warp_sum(red[cx][slice]);
  const int co = blockIdx.x * 32 + slice;
  if (cx == 0 && co < dim) store_sum(out + co, t);
}

// ------------------------------------------------------------------------------------------- RoPE

__global__ void rope_tables_k(const int64_t* __restrict__ pos, float* __restrict__ cos_o, float* __restrict__ sin_o,
                              int64_t T, int half, float theta) {
  after_previous_kernel(pos);
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * half) return;
  const int k = (int)(i % half);
  const int64_t t = i / half;
  const float inv_freq = 1.0f / powf(theta, (float)(2 * k) / (float)(2 * half));
  const float ang = (float)pos[t] * inv_freq;
  float s, c;
  sincosf(ang, &s, &c);
  cos_o[i] = c;
  sin_o[i] = s;
}

// Rotary embedding over a [T, heads, head_dim] tensor whose heads come in groups of `period`: the first `n_rot` heads of
// every group are rotated, the rest are not.  In place (COPY false: only the rotated heads are touched) or from `src`
// to `dst` (COPY true: the other heads are copied as they are, so a rotation that follows a copy costs one pass, not two).
template <bool COPY>
__global__ void rope_k(const bf16* __restrict__ src, bf16* __restrict__ dst, const float* __restrict__ cos_t,
                       const float* __restrict__ sin_t, int64_t T, int groups, int period, int n_rot, int head_dim,
                       int64_t src_stride, int64_t dst_stride, int inverse) {
  after_previous_kernel(src, cos_t, sin_t);
  const int half = head_dim >> 1;
  const int vec_per_head = half >> 3;
  const int per_group = COPY ? period : n_rot;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t total = T * groups * per_group * vec_per_head;
  if (i >= total) return;
  const int kv = (int)(i % vec_per_head);
  const int hh = (int)((i / vec_per_head) % ((int64_t)groups * per_group));
  const int64_t t = i / ((int64_t)vec_per_head * groups * per_group);
  const int g = hh / per_group, hg = hh - g * per_group;
  const int64_t col = ((int64_t)g * period + hg) * head_dim + kv * 8;
  const bf16* s1 = src + t * src_stride + col;
  bf16* d1 = dst + t * dst_stride + col;
  if (COPY && hg >= n_rot) {
    st8(d1, ld8(s1));
    st8(d1 + half, ld8(s1 + half));
    return;
  }
  float a[8], b[8], o1[8], o2[8];
  unpack8(ld8(s1), a);
  unpack8(ld8(s1 + half), b);
  const float* cp = cos_t + t * half + kv * 8;
  const float* sp = sin_t + t * half + kv * 8;
  const float4 c0 = *reinterpret_cast<const float4*>(cp), c1 = *reinterpret_cast<const float4*>(cp + 4);
  const float4 s0 = *reinterpret_cast<const float4*>(sp), s1v = *reinterpret_cast<const float4*>(sp + 4);
  const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
  const float s[8] = {s0.x, s0.y, s0.z, s0.w, s1v.x, s1v.y, s1v.z, s1v.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float sj = inverse ? -s[j] : s[j];
    o1[j] = a[j] * c[j] - b[j] * sj;
    o2[j] = b[j] * c[j] + a[j] * sj;
  }
  st8(d1, pack8(o1));
  st8(d1 + half, pack8(o2));
}

// ------------------------------------------------------------------------------------------- SwiGLU

__global__ void swiglu_fwd_k(const bf16* __restrict__ gu, bf16* __restrict__ h, int64_t T, int64_t I) {
  after_previous_kernel(gu);
  const int64_t vpr = I >> 3;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * vpr) return;
  const int64_t t = i / vpr, c = (i % vpr) * 8;
  float g[8], u[8], o[8];
  unpack8(ld8(gu + t * 2 * I + c), g);
  unpack8(ld8(gu + t * 2 * I + I + c), u);
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
  st8(h + t * I + c, pack8(o));
}

__global__ void swiglu_bwd_k(const bf16* __restrict__ dh, const bf16* __restrict__ gu, bf16* __restrict__ dgu,
                             int64_t T, int64_t I) {
  after_previous_kernel(dh, gu);
  const int64_t vpr = I >> 3;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * vpr) return;
  const int64_t t = i / vpr, c = (i % vpr) * 8;
  float g[8], u[8], d[8], dg[8], du[8];
  unpack8(ld8(gu + t * 2 * I + c), g);
  unpack8(ld8(gu + t * 2 * I + I + c), u);
  unpack8(ld8(dh + t * I + c), d);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float sig = 1.f / (1.f + __expf(-g[j]));
    dg[j] = d[j] * u[j] * sig * (1.f + g[j] * (1.f - sig));
    du[j] = d[j] * g[j] * sig;
  }
  st8(dgu + t * 2 * I + c, pack8(dg));
  st8(dgu + t * 2 * I + I + c, pack8(du));
}

// ------------------------------------------------------------------------------------------- cross-entropy

constexpr int CE_THREADS = 512, CE_VECS = 8;

// Two columns of a packed vector
__device__ __forceinline__ void unpack2(uint32_t p, float& a, float& b) {
  a = __uint_as_float(p << 16);
  b = __uint_as_float(p & 0xffff0000u);
}

// log-sum-exp of one row by a block of CE_THREADS.  A thread has eight vectors of the row in flight and keeps them packed (32768
// columns a round): with one load at a time, each followed by its update of the running maximum and sum, the loads' latency
// bound the pass.  Arithmetic on two columns at once.  Rows in the L2, us: forward of 1531 rows x 32000 columns 43 -> 37, 8192 x
// 32000 141 -> 123, 4096 x 128256 (beyond it) 233 to 312 -> 210.
__device__ __forceinline__ float row_lse(const bf16* lr, int64_t V, float* red) {
  float m = -INFINITY, s = 0.f;
  for (int64_t base = 0; base < V; base += CE_THREADS * 8 * CE_VECS) {
    uint4 p[CE_VECS];
#pragma unroll
    for (int i = 0; i < CE_VECS; ++i) {
      const int64_t c = base + (int64_t)(i * CE_THREADS + (int)threadIdx.x) * 8;
      p[i] = c < V ? *reinterpret_cast<const uint4*>(lr + c) : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // -inf
    }
    __nv_bfloat162 mx2 = *reinterpret_cast<__nv_bfloat162*>(&p[0].x);
#pragma unroll
    for (int i = 0; i < CE_VECS; ++i) {
      const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(&p[i]);
      mx2 = __hmax2(mx2, __hmax2(__hmax2(v[0], v[1]), __hmax2(v[2], v[3])));
    }
    // finite also when all logits so far are -inf: their exponentials are 0 then, not those of a difference of infinities
    const float mn = fmaxf(fmaxf(m, fmaxf(__low2float(mx2), __high2float(mx2))), -FLT_MAX);
    const uint64_t nmn = pk2(-mn, -mn), log2e = pk2(1.4426950408889634f, 1.4426950408889634f);
    uint64_t acc[2] = {pk2(0.f, 0.f), pk2(0.f, 0.f)};
#pragma unroll
    for (int i = 0; i < CE_VECS; ++i) {
      const uint32_t w[4] = {p[i].x, p[i].y, p[i].z, p[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float a, b;
        unpack2(w[j], a, b);
        upk2(mul2(add2(pk2(a, b), nmn), log2e), a, b);
        acc[j & 1] = add2(acc[j & 1], pk2(exp2_mufu(a), exp2_mufu(b)));
      }
    }
    float a, b;
    upk2(add2(acc[0], acc[1]), a, b);
    s = s * __expf(m - mn) + (a + b);
    m = mn;
  }
  const float M = block_max(m, red);
  const float S = block_sum(s * __expf(m - M), red);
  return M + logf(S);
}

// (softmax - onehot) * sc of 8 columns p, from c of a row with log-sum-exp l and target column tg, to dst = row + c
__device__ __forceinline__ void ce_grad8(const uint4& p, float l, int64_t c, int64_t tg, float sc, bf16* dst) {
  const uint64_t nl = pk2(-l, -l), log2e = pk2(1.4426950408889634f, 1.4426950408889634f), sc2 = pk2(sc, sc);
  const uint32_t w[4] = {p.x, p.y, p.z, p.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a, b;
    unpack2(w[j], a, b);
    upk2(mul2(add2(pk2(a, b), nl), log2e), a, b);
    upk2(mul2(pk2(exp2_mufu(a), exp2_mufu(b)), sc2), a, b);
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    o[j] = *reinterpret_cast<const uint32_t*>(&t);
  }
  *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
  const uint64_t at = (uint64_t)(tg - c);
  if (at < 8) {                              // one vector of the row: its target column once more
    const uint32_t pair = at < 4 ? (at < 2 ? p.x : p.y) : (at < 6 ? p.z : p.w);
    float a, b;
    unpack2(pair, a, b);
    dst[at] = __float2bfloat16_rn((exp2_mufu((((at & 1) ? b : a) - l) * 1.4426950408889634f) - 1.f) * sc);
  }
}

__global__ void __launch_bounds__(CE_THREADS, 2) ce_fwd_k(const bf16* __restrict__ logits, const int64_t* __restrict__ targets,
                                                          float* __restrict__ loss, float* __restrict__ lse, int64_t V,
                                                          int64_t ignore_index) {
  after_previous_kernel(logits, targets);
  __shared__ float red[33];
  const int64_t row = blockIdx.x;
  const bf16* lr = logits + row * V;
  const float l = row_lse(lr, V, red);
  if (threadIdx.x == 0) {
    lse[row] = l;
    const int64_t tg = targets[row];
    loss[row] = (tg == ignore_index) ? 0.f : l - __bfloat162float(lr[tg]);
  }
}

// Loss and gradient of a row in one kernel, for callers that know the scale before they see the loss (the chunked lm_head +
// loss): the second pass over the row reads it from the L2 (two blocks per SM, so at most 296 rows are open, 76 MB at 128256
// words) and writes the gradient over it, four vectors of a thread in flight.  1531 rows x 32000 97 -> 60 us, 8192 x 32000 400 ->
// 268, 4096 x 128256 610 -> 450, in two kernels (ce_fwd_k, ce_bwd_k) 79, 313 and 575.
__global__ void __launch_bounds__(CE_THREADS, 2) ce_grad_k(bf16* logits, const int64_t* __restrict__ targets,
                                                           float* __restrict__ loss, const float* __restrict__ scale, int64_t V,
                                                           int64_t ignore_index) {
  after_previous_kernel(logits, targets, scale);
  __shared__ float red[33];
  const int64_t row = blockIdx.x;
  bf16* lr = logits + row * V;
  const float l = row_lse(lr, V, red);
  const int64_t tg = targets[row];
  if (threadIdx.x == 0) loss[row] = (tg == ignore_index) ? 0.f : l - __bfloat162float(lr[tg]);
  __syncthreads();                                   // the target's logit has been read
  const float sc = (tg == ignore_index) ? 0.f : scale[0];
  for (int64_t base = (int64_t)threadIdx.x * 8; base < V; base += CE_THREADS * 8 * 4) {
    uint4 p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (base + i * CE_THREADS * 8 < V) p[i] = *reinterpret_cast<const uint4*>(lr + base + i * CE_THREADS * 8);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t c = base + i * CE_THREADS * 8;
      if (c < V) ce_grad8(p[i], l, c, tg, sc, lr + c);
    }
  }
}

__global__ void __launch_bounds__(256) ce_bwd_k(bf16* __restrict__ logits, const int64_t* __restrict__ targets, const float* __restrict__ lse,
                                                const float* __restrict__ scale, int64_t V, int64_t ignore_index) {
  after_previous_kernel(logits, targets, lse, scale);
  const int64_t row = blockIdx.y;
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= V) return;
  bf16* at = logits + row * V + c;
  const uint4 p = *reinterpret_cast<const uint4*>(at);
  const int64_t tg = targets[row];
  const float sc = (tg == ignore_index) ? 0.f : scale[0];
  ce_grad8(p, lse[row], c, tg, sc, at);
}

// ------------------------------------------------------------------------------------------- scaling by a device scalar

// dst = src * scale[0], eight values per thread (dst may be src); bound by memory.  [128256, 4096]: 338 us, where a broadcast
// multiplication by a 0-d tensor and a copy of its result took 1449.
__global__ void __launch_bounds__(256) scale_k(bf16* dst, const bf16* src, const float* __restrict__ scale, int64_t n) {
  after_previous_kernel(src, scale);
  const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 8;
  if (i >= n) return;
  const float sc = scale[0];
  float f[8];
  unpack8(ld8(src + i), f);
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] *= sc;
  st8(dst + i, pack8(f));
}

// ------------------------------------------------------------------------------------------- embedding gradient

// dw[ids[t]] += dy[t] in bf16: one thread per 8 columns of a token, one 16-byte vector reduction each.  Tokens that share a
// row add in no fixed order, as with index_add.  An id outside the table is skipped and reported.  Reads dy once; bound by
// memory.  With the zero fill of dw: 75 us at 8192 tokens of 32000 x 4096, where the fill and index_add with its scalar
// reductions took 353; 204 and 693 at 12288 of 128256.
__global__ void __launch_bounds__(256) embedding_grad_k(const bf16* __restrict__ dy, const int64_t* __restrict__ ids,
                                                        bf16* __restrict__ dw, int64_t total, int vpr, int64_t vocab,
                                                        int* __restrict__ err) {
  after_previous_kernel(dy, ids);
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= total) return;
  const int64_t t = i / vpr;
  const int c = (int)(i - t * vpr) * 8;
  const int64_t id = ids[t];
  if (id < 0 || id >= vocab) {
    if (err != nullptr) atomicCAS(err, 0, ODY_ERR_BAD_INDEX);
    return;
  }
  const uint4 v = *reinterpret_cast<const uint4*>(dy + i * 8);
  bf16* dst = dw + id * ((int64_t)vpr * 8) + c;
  asm volatile("red.relaxed.gpu.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

// ------------------------------------------------------------------------------------------- AdamW

__global__ void adamw_k(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                        const bf16* __restrict__ grad, bf16* __restrict__ param, int64_t n, float decay, float beta1,
                        float beta2, float step_size, float inv_sqrt_bc2, float eps, float grad_scale,
                        const float* __restrict__ guard) {
  after_previous_kernel(master, m, v, grad, guard);
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  // a non-zero guard word (the step's kernel status, summed over ranks) means some gradient is incomplete:
  // leave master, moments and parameters untouched so the host can stop or restart from here
  if (guard != nullptr && *guard != 0.f) return;
  float g[8];
  unpack8(ld8(grad + i), g);
  float4 w0 = *reinterpret_cast<float4*>(master + i), w1 = *reinterpret_cast<float4*>(master + i + 4);
  float4 m0 = *reinterpret_cast<float4*>(m + i), m1 = *reinterpret_cast<float4*>(m + i + 4);
  float4 v0 = *reinterpret_cast<float4*>(v + i), v1 = *reinterpret_cast<float4*>(v + i + 4);
  float W[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
  float M[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
  float Vv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float gj = g[j] * grad_scale;
    M[j] = beta1 * M[j] + (1.f - beta1) * gj;
    Vv[j] = beta2 * Vv[j] + (1.f - beta2) * gj * gj;
    const float denom = sqrtf(Vv[j]) * inv_sqrt_bc2 + eps;
    W[j] = W[j] * decay - step_size * M[j] / denom;
  }
  *reinterpret_cast<float4*>(master + i) = make_float4(W[0], W[1], W[2], W[3]);
  *reinterpret_cast<float4*>(master + i + 4) = make_float4(W[4], W[5], W[6], W[7]);
  *reinterpret_cast<float4*>(m + i) = make_float4(M[0], M[1], M[2], M[3]);
  *reinterpret_cast<float4*>(m + i + 4) = make_float4(M[4], M[5], M[6], M[7]);
  *reinterpret_cast<float4*>(v + i) = make_float4(Vv[0], Vv[1], Vv[2], Vv[3]);
  *reinterpret_cast<float4*>(v + i + 4) = make_float4(Vv[4], Vv[5], Vv[6], Vv[7]);
  st8(param + i, pack8(W));
}

// ------------------------------------------------------------------------------------------- attention merge

// out [T_total, H, hd] fp32 and lse [H, T_total] fp32 are the running result; (o [T, H, hd] bf16,
// l [H, T] fp32) is a partial over a disjoint key set for rows [row0, row0 + T).
__global__ void attn_merge_k(float* __restrict__ out, float* __restrict__ lse, const bf16* __restrict__ o,
                             const float* __restrict__ l, int64_t T, int H, int hd, int64_t row0, int64_t T_total) {
  const int vph = hd >> 3;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = i < T * H * vph;
  float la = 0.f, lb = 0.f;
  int64_t t = 0;
  int h = 0, kv = 0;
  if (live) {
    kv = (int)(i % vph);
    h = (int)((i / vph) % H);
    t = i / ((int64_t)vph * H);
    la = lse[(int64_t)h * T_total + row0 + t];
    lb = l[(int64_t)h * T + t];
  }
  __syncwarp();  // every lane of a (t, h) group has read the old lse before its leader overwrites it
  if (!live) return;
  const float mx = fmaxf(la, lb);
  const float ln = mx + logf(__expf(la - mx) + __expf(lb - mx));
  const float wa = __expf(la - ln), wb = __expf(lb - ln);
  float* po = out + ((row0 + t) * H + h) * hd + kv * 8;
  float b[8];
  unpack8(ld8(o + (t * H + h) * hd + kv * 8), b);
  float4 a0 = *reinterpret_cast<float4*>(po), a1 = *reinterpret_cast<float4*>(po + 4);
  a0 = make_float4(a0.x * wa + b[0] * wb, a0.y * wa + b[1] * wb, a0.z * wa + b[2] * wb, a0.w * wa + b[3] * wb);
  a1 = make_float4(a1.x * wa + b[4] * wb, a1.y * wa + b[5] * wb, a1.z * wa + b[6] * wb, a1.w * wa + b[7] * wb);
  *reinterpret_cast<float4*>(po) = a0;
  *reinterpret_cast<float4*>(po + 4) = a1;
  if (kv == 0) lse[(int64_t)h * T_total + row0 + t] = ln;
}

// dst rows [begin_i, begin_i + rows_i) += src_i, summed in fp32 over all sources; dst [T, C] with row pitch dst_ld.
struct SumRowsArgs {
  const bf16* src[8];
  int64_t src_ld[8], begin[8], rows[8];
  int n;
};
__global__ void sum_rows_k(bf16* __restrict__ dst, int64_t dst_ld, int64_t T, int64_t C, const __grid_constant__ SumRowsArgs a) {
  const int64_t vpr = C >> 3;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * vpr) return;
  const int64_t t = i / vpr, c = (i % vpr) * 8;
  bf16x8 part[8];
  bool on[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    on[k] = k < a.n && t >= a.begin[k] && t < a.begin[k] + a.rows[k];
    if (on[k]) part[k] = ld8(a.src[k] + (t - a.begin[k]) * a.src_ld[k] + c);
  }
  float acc[8];
  unpack8(ld8(dst + t * dst_ld + c), acc);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (on[k]) {
      float b[8];
      unpack8(part[k], b);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += b[e];
    }
  }
  st8(dst + t * dst_ld + c, pack8(acc));
}

// One-pass merge of up to 8 attention partials over disjoint key sets: partial i covers rows
// [begin_i, begin_i + rows_i) with o_i [rows_i, H, hd] bf16 and lse_i [H, rows_i].  out [T, H, hd] bf16, lse [H, T].
struct MergeArgs {
  const bf16* o[8];
  const float* lse[8];
  int64_t begin[8], rows[8];
  int n;
};
__global__ void attn_merge_parts_k(bf16* __restrict__ out, float* __restrict__ lse, int64_t T, int H, int hd,
                                   const __grid_constant__ MergeArgs a) {
  const int vph = hd >> 3;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * H * vph) return;
  const int kv = (int)(i % vph);
  const int h = (int)((i / vph) % H);
  const int64_t t = i / ((int64_t)vph * H);
  float l[8], mx = -INFINITY;
  bf16x8 part[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const bool on = k < a.n && t >= a.begin[k] && t < a.begin[k] + a.rows[k];
    l[k] = -INFINITY;
    if (on) {
      const int64_t tt = t - a.begin[k];
      l[k] = a.lse[k][(int64_t)h * a.rows[k] + tt];
      part[k] = ld8(a.o[k] + (tt * H + h) * hd + kv * 8);
      mx = fmaxf(mx, l[k]);
    }
  }
  float den = 0.f, acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (l[k] != -INFINITY) {
      const float w = __expf(l[k] - mx);
      den += w;
      float b[8];
      unpack8(part[k], b);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += w * b[e];
    }
  }
  const float inv = den > 0.f ? 1.f / den : 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] *= inv;
  st8(out + (t * H + h) * hd + kv * 8, pack8(acc));
  if (kv == 0) lse[(int64_t)h * T + t] = den > 0.f ? mx + logf(den) : -INFINITY;
}

}  // namespace ody

// =========================================================================================== launchers

using namespace ody;

static inline int last_err() { return (int)cudaGetLastError(); }
static inline unsigned blocks_for(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }

extern "C" int ody_rmsnorm_fwd(const void* x, const void* delta, const void* w, void* sum_out, void* y, float* rstd,
                               int64_t rows, int dim, float eps, cudaStream_t st) {
  if (dim % 8 != 0 || dim > 256 * 8 * 8) return (int)cudaErrorInvalidValue;
  if (rows == 0) return 0;
  const int nv = (dim + 2047) / 2048;
#define L(NV)                                                                                               \
  launch_kernel(rmsnorm_fwd_k<NV>, (unsigned)rows, 256, 0, st, 1, (const bf16*)x, (const bf16*)delta, (const bf16*)w,    \
                                                    (bf16*)sum_out, (bf16*)y, rstd, dim, eps)
  if (nv <= 1) L(1); else if (nv <= 2) L(2); else if (nv <= 4) L(4); else L(8);
#undef L
  return last_err();
}

extern "C" int ody_rmsnorm_bwd_blocks(int64_t rows, int dim) {
  const int64_t b = dim > 4096 && dim <= 8192 ? 148 : 148 * 2;       // resident blocks: registers, and the ring's shared memory
  return (int)(rows < b ? (rows > 0 ? rows : 1) : b);
}

template <int NV, bool DS>
static int launch_norm_ring(const void* dy, const void* x, const void* w, const float* rstd, const void* ds, void* dx,
                            float* dw_partial, int64_t rows, int dim, int nb, cudaStream_t st) {
  constexpr int SMEM = NORM_STAGES * (DS ? 3 : 2) * NV * 256 * 16;
  static std::atomic<uint64_t> configured{0};      // one bit per device: the attribute belongs to the device's copy of the kernel
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev > 63 || !(configured.load(std::memory_order_relaxed) >> dev & 1)) {
    const cudaError_t e = cudaFuncSetAttribute(rmsnorm_bwd_ring_k<NV, DS>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    if (dev <= 63) configured.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  launch_kernel(rmsnorm_bwd_ring_k<NV, DS>, nb, 256, SMEM, st, 1, (const bf16*)dy, (const bf16*)x, (const bf16*)w, rstd, (const bf16*)ds,
                                                    (bf16*)dx, dw_partial, rows, dim);
  return last_err();
}

extern "C" int ody_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* ds,
                               void* dx, float* dw, float* dw_partial, int64_t rows, int dim, cudaStream_t st) {
  return ody_rmsnorm_bwd_to(dy, x, w, rstd, ds, dx, dw, 0, dw_partial, rows, dim, st);
}

extern "C" int ody_rmsnorm_bwd_to(const void* dy, const void* x, const void* w, const float* rstd, const void* ds, void* dx,
                                  void* dw, int dw_bf16, float* dw_partial, int64_t rows, int dim, cudaStream_t st) {
  if (dim % 8 != 0 || dim > 256 * 8 * 8) return (int)cudaErrorInvalidValue;
  const int nb = ody_rmsnorm_bwd_blocks(rows, dim);
  int e = 0;
#define R(NV)                                                                                         \
  e = ds != nullptr ? launch_norm_ring<NV, true>(dy, x, w, rstd, ds, dx, dw_partial, rows, dim, nb, st) \
                    : launch_norm_ring<NV, false>(dy, x, w, rstd, ds, dx, dw_partial, rows, dim, nb, st)
  if (dim <= 2048) R(1); else if (dim <= 4096) R(2); else if (dim <= 8192) R(4);
#undef R
  else   // a ring of such rows does not fit the shared memory
    launch_kernel(rmsnorm_bwd_k<8>, nb, 256, 0, st, 1, (const bf16*)dy, (const bf16*)x, (const bf16*)w, rstd, (const bf16*)ds,
                                         (bf16*)dx, dw_partial, rows, dim);
  if (e) return e;
  if (dw_bf16)
    launch_kernel(colsum_k<bf16>, blocks_for(dim, 32), 1024, 0, st, 1, dw_partial, (bf16*)dw, nb, dim);
  else
    launch_kernel(colsum_k<float>, blocks_for(dim, 32), 1024, 0, st, 1, dw_partial, (float*)dw, nb, dim);
  return last_err();
}

extern "C" int ody_rope_tables(const int64_t* positions, float* cos_out, float* sin_out, int64_t T, int head_dim,
                               float theta, cudaStream_t st) {
  const int half = head_dim / 2;
  if (T == 0) return 0;
  launch_kernel(rope_tables_k, blocks_for(T * half, 256), 256, 0, st, 1, positions, cos_out, sin_out, T, half, theta);
  return last_err();
}

extern "C" int ody_rope(const void* src, void* dst, const float* cos_t, const float* sin_t, int64_t T, int heads,
                        int period, int n_rot, int head_dim, int64_t src_stride, int64_t dst_stride, int inverse,
                        cudaStream_t st) {
  if (head_dim % 16 != 0 || src_stride % 8 != 0 || dst_stride % 8 != 0 || period <= 0 || heads % period != 0 ||
      n_rot < 0 || n_rot > period)
    return (int)cudaErrorInvalidValue;
  const int groups = heads / period;
  const bool copy = src != (const void*)dst;
  const int64_t total = T * groups * (copy ? period : n_rot) * (head_dim / 16);
  if (total == 0) return 0;
  if (copy)
    launch_kernel(rope_k<true>, blocks_for(total, 256), 256, 0, st, 1, (const bf16*)src, (bf16*)dst, cos_t, sin_t, T, groups, period,
                                                         n_rot, head_dim, src_stride, dst_stride, inverse);
  else
    launch_kernel(rope_k<false>, blocks_for(total, 256), 256, 0, st, 1, (const bf16*)src, (bf16*)dst, cos_t, sin_t, T, groups, period,
                                                          n_rot, head_dim, src_stride, dst_stride, inverse);
  return last_err();
}

extern "C" int ody_rope_inplace(void* x, const float* cos_t, const float* sin_t, int64_t T, int n_rot, int head_dim,
                                int64_t row_stride, int inverse, cudaStream_t st) {
  if (n_rot == 0 || T == 0) return 0;
  return ody_rope(x, x, cos_t, sin_t, T, n_rot, n_rot, n_rot, head_dim, row_stride, row_stride, inverse, st);
}

extern "C" int ody_swiglu_fwd(const void* gu, void* h, int64_t T, int64_t I, cudaStream_t st) {
  if (I % 8 != 0) return (int)cudaErrorInvalidValue;
  if (T * I == 0) return 0;
  launch_kernel(swiglu_fwd_k, blocks_for(T * (I / 8), 256), 256, 0, st, 1, (const bf16*)gu, (bf16*)h, T, I);
  return last_err();
}

extern "C" int ody_swiglu_bwd(const void* dh, const void* gu, void* dgu, int64_t T, int64_t I, cudaStream_t st) {
  if (I % 8 != 0) return (int)cudaErrorInvalidValue;
  if (T * I == 0) return 0;
  launch_kernel(swiglu_bwd_k, blocks_for(T * (I / 8), 256), 256, 0, st, 1, (const bf16*)dh, (const bf16*)gu, (bf16*)dgu, T, I);
  return last_err();
}

extern "C" int ody_ce_fwd(const void* logits, const int64_t* targets, float* loss, float* lse, int64_t T, int64_t V,
                          int64_t ignore_index, cudaStream_t st) {
  if (V % 8 != 0) return (int)cudaErrorInvalidValue;
  if (T == 0) return 0;
  launch_kernel(ce_fwd_k, (unsigned)T, CE_THREADS, 0, st, 1, (const bf16*)logits, targets, loss, lse, V, ignore_index);
  return last_err();
}

extern "C" int ody_ce_grad(void* logits, const int64_t* targets, float* loss, const float* scale, int64_t T, int64_t V,
                           int64_t ignore_index, cudaStream_t st) {
  if (V % 8 != 0) return (int)cudaErrorInvalidValue;
  if (T == 0) return 0;
  launch_kernel(ce_grad_k, (unsigned)T, CE_THREADS, 0, st, 1, (bf16*)logits, targets, loss, scale, V, ignore_index);
  return last_err();
}

extern "C" int ody_ce_bwd(void* logits, const int64_t* targets, const float* lse, const float* scale, int64_t T,
                          int64_t V, int64_t ignore_index, cudaStream_t st) {
  if (V % 8 != 0 || T > 65535) return (int)cudaErrorInvalidValue;
  if (T == 0) return 0;
  dim3 grid(blocks_for(V / 8, 256), (unsigned)T);
  launch_kernel(ce_bwd_k, grid, 256, 0, st, 1, (bf16*)logits, targets, lse, scale, V, ignore_index);
  return last_err();
}

extern "C" int ody_scale(void* dst, const void* src, const float* scale, int64_t n, cudaStream_t st) {
  if (n % 8 != 0 || (((uintptr_t)dst | (uintptr_t)src) & 15)) return (int)cudaErrorInvalidValue;
  if (n == 0) return 0;
  launch_kernel(scale_k, blocks_for(n / 8, 256), 256, 0, st, 1, (bf16*)dst, (const bf16*)src, scale, n);
  return last_err();
}

extern "C" int ody_embedding_grad(const void* dy, const int64_t* ids, void* dw, int64_t T, int dim, int64_t vocab, int* err,
                                  cudaStream_t st) {
  if (dim % 8 != 0 || vocab <= 0 || (((uintptr_t)dy | (uintptr_t)dw) & 15)) return (int)cudaErrorInvalidValue;
  const cudaError_t e = cudaMemsetAsync(dw, 0, (size_t)vocab * dim * 2, st);
  if (e != cudaSuccess) return (int)e;
  const int64_t total = T * (dim / 8);
  if (total == 0) return 0;
  launch_kernel(embedding_grad_k, blocks_for(total, 256), 256, 0, st, 1, (const bf16*)dy, ids, (bf16*)dw, total, dim / 8, vocab, err);
  return last_err();
}

extern "C" int ody_adamw(float* master, float* m, float* v, const void* grad, void* param, int64_t n, float lr,
                         float beta1, float beta2, float eps, float weight_decay, int step, float grad_scale,
                         const float* guard, cudaStream_t st) {
  if (n % 8 != 0) return (int)cudaErrorInvalidValue;
  if (n == 0) return 0;
  const double bc1 = 1.0 - pow((double)beta1, (double)step);
  const double bc2 = 1.0 - pow((double)beta2, (double)step);
  launch_kernel(adamw_k, blocks_for(n / 8, 256), 256, 0, st, 1, master, m, v, (const bf16*)grad, (bf16*)param, n,
                                                  1.f - lr * weight_decay, beta1, beta2, (float)(lr / bc1),
                                                  (float)(1.0 / sqrt(bc2)), eps, grad_scale, guard);
  return last_err();
}

extern "C" int ody_attn_merge(float* out, float* lse, const void* o, const float* l, int64_t T, int H, int hd,
                              int64_t row0, int64_t T_total, cudaStream_t st) {
  if (hd % 8 != 0 || 32 % (hd / 8) != 0) return (int)cudaErrorInvalidValue;
  const int64_t total = T * H * (hd / 8);
  if (total == 0) return 0;
  attn_merge_k<<<blocks_for(total, 256), 256, 0, st>>>(out, lse, (const bf16*)o, l, T, H, hd, row0, T_total);
  return last_err();
}

extern "C" int ody_sum_rows(void* dst, int64_t dst_ld, int64_t T, int64_t C, const void* const* src, const int64_t* src_ld,
                            const int64_t* begin, const int64_t* rows, int n, cudaStream_t st) {
  if (n < 0 || n > 8 || (C % 8) || (dst_ld % 8) || ((uintptr_t)dst & 15)) return (int)cudaErrorInvalidValue;
  if (n == 0 || T * C == 0) return 0;
  SumRowsArgs a;
  memset(&a, 0, sizeof(a));
  a.n = n;
  for (int k = 0; k < n; ++k) {
    if ((src_ld[k] % 8) || ((uintptr_t)src[k] & 15) || begin[k] < 0 || begin[k] + rows[k] > T) return (int)cudaErrorInvalidValue;
    a.src[k] = (const bf16*)src[k]; a.src_ld[k] = src_ld[k]; a.begin[k] = begin[k]; a.rows[k] = rows[k];
  }
  sum_rows_k<<<blocks_for(T * (C / 8), 256), 256, 0, st>>>((bf16*)dst, dst_ld, T, C, a);
  return last_err();
}

extern "C" int ody_attn_merge_parts(void* out, float* lse, int64_t T, int H, int hd, const void* const* o,
                                    const float* const* l, const int64_t* begin, const int64_t* rows, int n, cudaStream_t st) {
  if (n < 1 || n > 8 || hd % 8 != 0) return (int)cudaErrorInvalidValue;
  if (T * H == 0) return 0;
  MergeArgs a;
  memset(&a, 0, sizeof(a));
  a.n = n;
  for (int k = 0; k < n; ++k) {
    if (begin[k] < 0 || begin[k] + rows[k] > T || ((uintptr_t)o[k] & 15)) return (int)cudaErrorInvalidValue;
    a.o[k] = (const bf16*)o[k]; a.lse[k] = l[k]; a.begin[k] = begin[k]; a.rows[k] = rows[k];
  }
  attn_merge_parts_k<<<blocks_for(T * H * (hd / 8), 256), 256, 0, st>>>((bf16*)out, lse, T, H, hd, a);
  return last_err();
}
