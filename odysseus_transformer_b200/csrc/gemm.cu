// bf16 GEMM for sm_100a: TMA -> shared memory -> tcgen05.mma -> TMEM -> epilogue -> TMA store.
//
// This is the GEMM core behind every linear layer of the model (the reference reaches cuBLAS through
// torch.matmul / F.linear: reference utils/linear_tpsp.py:173,217,291,588; utils/linear_zero3.py:44,68,74).
//
//   layout 0 (NT): C[M,N] = A[M,K] * B[N,K]^T      forward   y  = x  W^T     (A, B K-major)
//   layout 1 (NN): C[M,N] = A[M,K] * B[K,N]        dgrad     dx = dy W       (B MN-major)
//   layout 2 (TN): C[M,N] = A[K,M]^T * B[K,N]      wgrad     dW = dy^T x     (A, B MN-major)
//
// One persistent CTA per SM, 192 threads: warp 0 = TMA producer, warp 1 = MMA issuer (one elected
// thread) and TMEM owner, warps 2-5 = epilogue.  Tile 128 x 256 x 64, 4-stage smem ring (48 KB / stage),
// two 256-column fp32 accumulators in TMEM (all 512 columns) so the epilogue of tile i overlaps the
// main loop of tile i+1.  The epilogue converts to bf16, stages 128 x 64 blocks in swizzled smem and
// writes them with TMA stores (edges are clipped by the tensor map).  No cluster multicast anywhere.
// gemm_2cta.cu holds the same GEMM on CTA pairs (cta_group::2), gemm_cluster.cu on small tiles with K shared by a cluster; the
// functions at the end of this file choose.
#include "ody_kernels.h"
#include "sm100.cuh"
#include "launch.cuh"

namespace ody {

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4;
constexpr int UMMA_K = 16;
constexpr int A_BYTES = BM * BK * 2;             // 16 KB
constexpr int B_BYTES = BN * BK * 2;             // 32 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;   // 48 KB
constexpr int EPI_COLS = 64;
constexpr int EPI_BYTES = BM * EPI_COLS * 2;     // 16 KB
constexpr int SMEM_TILES = STAGES * STAGE_BYTES + 2 * EPI_BYTES;
constexpr int SMEM_TOTAL = SMEM_TILES + 256 + 1024;   // + barriers + alignment slack
constexpr int NUM_THREADS = 192;
constexpr int GROUP_M = 16;

struct GemmBars {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint64_t drain;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int tiles_n, int& tm, int& tn) {
  const int per_group = GROUP_M * tiles_n;
  const int g = tile / per_group;
  const int first_m = g * GROUP_M;
  const int gsize = min(GROUP_M, tiles_m - first_m);
  const int local = tile - g * per_group;
  tm = first_m + local % gsize;
  tn = local / gsize;
}

__device__ __forceinline__ bool epi_all_ok(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.and.pred p, 2, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)ok)
      : "memory");
  return r != 0;
}

// ROPE: the epilogue rotates the q / k heads of a packed projection (RopeEpi, sm100.cuh); a separate instance, so that
// the plain one keeps its register allocation
//
// SPLIT: `splits` CTAs share a tile's k-blocks; each writes its fp32 accumulator to part [splits][M][N] and
// splitk_sum_kernel does what the epilogue would have done.
template <int LAYOUT, bool ROPE, bool SPLIT = false>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const __nv_bfloat16* __restrict__ c_in, int M, int N, int K,
                 int64_t ldc, int accumulate, int mn3d, RopeEpi rp, int* __restrict__ err,
                 float* __restrict__ part = nullptr, int splits = 1) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  GemmBars* bars = (GemmBars*)(smem + SMEM_TILES);
  uint8_t* epi = smem + STAGES * STAGE_BYTES;
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  const int num_items = tiles_m * tiles_n * (SPLIT ? splits : 1);      // item = tile * splits + which share of its k-blocks
  const int kblocks = (K + BK - 1) / BK;
  auto kb_begin = [&](int item) { return SPLIT ? (int)((int64_t)kblocks * (item % splits) / splits) : 0; };
  auto kb_end = [&](int item) { return SPLIT ? (int)((int64_t)kblocks * (item % splits + 1) / splits) : kblocks; };
  constexpr bool A_MN = (LAYOUT == 2), B_MN = (LAYOUT != 0);
  constexpr uint32_t IDESC = make_idesc_bf16(BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars->tmem_full[b], 1);
      mbar_init(&bars->tmem_empty[b], 128);
    }
    mbar_init(&bars->drain, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
    prefetch_tmap(&tmC);
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  if constexpr (ROPE) after_previous_kernel(c_in, rp.cos, rp.sin); else after_previous_kernel(c_in);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
        int tm, tn;
        tile_coords(SPLIT ? item / splits : item, tiles_m, tiles_n, tm, tn);
        const int m0 = tm * BM, n0 = tn * BN;
        const int kb1 = kb_end(item);
        for (int kb = kb_begin(item); kb < kb1; ++kb) {
          if (!mbar_wait(&bars->empty[stage], phase ^ 1, abort_flag, err, ODY_ERR_TIMEOUT_EMPTY)) { ok = false; break; }
          uint8_t* sA = smem + stage * STAGE_BYTES;
          uint8_t* sB = sA + A_BYTES;
          mbar_expect_tx(&bars->full[stage], STAGE_BYTES);
          const int k0 = kb * BK;
          if (!A_MN) {
            tma_load_2d(sA, &tmA, k0, m0, &bars->full[stage]);
          } else if (mn3d & 1) {
            tma_load_3d(sA, &tmA, 0, k0, m0 / 64, &bars->full[stage]);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d(sA + j * 8192, &tmA, m0 + 64 * j, k0, &bars->full[stage]);
          }
          if (!B_MN) {
            tma_load_2d(sB, &tmB, k0, n0, &bars->full[stage]);
          } else if (mn3d & 2) {
            tma_load_3d(sB, &tmB, 0, k0, n0 / 64, &bars->full[stage]);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_2d(sB + j * 8192, &tmB, n0 + 64 * j, k0, &bars->full[stage]);
          }
          ++issued;
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok || *abort_flag) {
        // give copies still in flight a bounded chance to land before the CTA retires
        int n = issued < STAGES ? issued : STAGES;
        for (int i = 0; i < n; ++i) {
          if (--stage < 0) { stage = STAGES - 1; phase ^= 1; }
          const long long t0 = clock64();
          while (!mbar_try_wait(&bars->full[stage], phase) && clock64() - t0 < ODY_SPIN_LIMIT_CYCLES / 8) {}
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    {
      // every lane runs the control flow, so the compiler keeps descriptors and loop state in uniform registers and an MMA
      // costs a few instructions; one elected lane issues the tcgen05 instructions (benchmarks/mma_issue_rate.cu)
      const bool leader = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      int local_tile = 0;
      bool ok = true;
      const uint32_t s0 = smem_u32(smem);
      const uint64_t adesc0 = A_MN ? make_smem_desc(s0, 8192, 1024) : make_smem_desc(s0, 16, 1024);
      const uint64_t bdesc0 = B_MN ? make_smem_desc(s0 + A_BYTES, 8192, 1024) : make_smem_desc(s0 + A_BYTES, 16, 1024);
      for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x, ++local_tile) {
        const int kb0 = kb_begin(item), kb1 = kb_end(item);
        const int buf = local_tile & 1;
        const uint32_t acc_phase = (local_tile >> 1) & 1;
        if (!mbar_wait(&bars->tmem_empty[buf], acc_phase ^ 1, abort_flag, err, ODY_ERR_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&bars->full[stage], phase, abort_flag, err, ODY_ERR_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a0 = desc_advance(adesc0, stage * STAGE_BYTES), b0 = desc_advance(bdesc0, stage * STAGE_BYTES);
          if (leader) umma_ss(d_tmem, a0, b0, IDESC, kb > kb0 ? 1u : 0u);
#pragma unroll
          for (int kk = 1; kk < BK / UMMA_K; ++kk)
            if (leader) umma_ss(d_tmem, desc_advance(a0, kk * (A_MN ? 2048 : 32)), desc_advance(b0, kk * (B_MN ? 2048 : 32)), IDESC, 1u);
          if (leader) umma_commit(&bars->empty[stage]);        // frees the smem stage once these MMAs have read it
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok && leader) umma_commit(&bars->tmem_full[buf]);  // accumulator complete
      }
      if (!ok || *abort_flag) {
        if (leader) umma_commit(&bars->drain);
        const long long t0 = clock64();
        while (!mbar_try_wait(&bars->drain, 0) && clock64() - t0 < ODY_SPIN_LIMIT_CYCLES / 8) {}
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;                      // TMEM lane quarter this warp may read
    const int r = q * 32 + lane;                 // row inside the tile
    const bool store_thread = (warp == 2 && lane == 0);
    int local_tile = 0;
    for (int item = blockIdx.x; item < num_items; item += gridDim.x, ++local_tile) {
      int tm, tn;
      tile_coords(SPLIT ? item / splits : item, tiles_m, tiles_n, tm, tn);
      const int m0 = tm * BM, n0 = tn * BN;
      const int buf = local_tile & 1;
      const uint32_t acc_phase = (local_tile >> 1) & 1;
      bool ok = mbar_wait(&bars->tmem_full[buf], acc_phase, abort_flag, err, ODY_ERR_TIMEOUT_TMEM_FULL);
      if (!epi_all_ok(ok)) break;
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < BN / EPI_COLS; ++c) {
        if (ROPE && rope_epi_wants(rp, n0 + c * EPI_COLS)) {
          // both halves of a head at once; its high half is the next chunk
          const int row = m0 + r, col0 = n0 + c * EPI_COLS;
          if (store_thread) tma_store_wait_read<0>();
          named_barrier(1, 128);
          rope_epi_head(rp, row, row < M, tmem_base + buf * BN + c * EPI_COLS + ((uint32_t)(q * 32) << 16), epi, epi + EPI_BYTES, r,
                        accumulate && row < M && col0 < N ? c_in + (int64_t)row * ldc + col0 : nullptr);
          if (c == BN / EPI_COLS - 2) {
            tc_fence_before();
            mbar_arrive(&bars->tmem_empty[buf]);
          }
          fence_proxy_async_smem();
          named_barrier(1, 128);
          if (store_thread && col0 < N) {
            tma_store_2d(&tmC, epi, col0, m0);
            tma_store_2d(&tmC, epi + EPI_BYTES, col0 + EPI_COLS, m0);
            tma_store_commit();
          }
          ++c;
          continue;
        }
        uint8_t* sbuf = epi + (c & 1) * EPI_BYTES;
        if (!SPLIT) {
          if (store_thread) tma_store_wait_read<ROPE ? 0 : 1>();     // a rotated head leaves both tiles in one group
          named_barrier(1, 128);
        }
        const uint32_t taddr = tmem_base + buf * BN + c * EPI_COLS + ((uint32_t)(q * 32) << 16);
        uint32_t v[64];
        tmem_ld_32x32(taddr, v);
        tmem_ld_32x32(taddr + 32, v + 32);
        tmem_ld_wait();
        const int row = m0 + r, col0 = n0 + c * EPI_COLS;
        if (c == BN / EPI_COLS - 1) {
          tc_fence_before();
          mbar_arrive(&bars->tmem_empty[buf]);
        }
        if constexpr (SPLIT) {
          if (row < M) {
            float* dst = part + ((int64_t)(item % splits) * M + row) * N + col0;
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (col0 + j * 4 < N)
                *reinterpret_cast<uint4*>(dst + j * 4) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
          continue;
        }
        if (accumulate && row < M) {
          const __nv_bfloat16* cp = c_in + (int64_t)row * ldc + col0;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (col0 + j * 8 < N) {   // N is a multiple of 8
              const uint4 old = *reinterpret_cast<const uint4*>(cp + j * 8);
              const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                const float2 f = __bfloat1622float2(o2[t]);
                v[j * 8 + 2 * t] = __float_as_uint(__uint_as_float(v[j * 8 + 2 * t]) + f.x);
                v[j * 8 + 2 * t + 1] = __float_as_uint(__uint_as_float(v[j * 8 + 2 * t + 1]) + f.y);
              }
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint4 pk;
          __nv_bfloat162* p2 = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
          for (int t = 0; t < 4; ++t)
            p2[t] = __floats2bfloat162_rn(__uint_as_float(v[j * 8 + 2 * t]), __uint_as_float(v[j * 8 + 2 * t + 1]));
          *reinterpret_cast<uint4*>(sbuf + r * 128 + ((j ^ (r & 7)) << 4)) = pk;
        }
        fence_proxy_async_smem();
        named_barrier(1, 128);
        if (store_thread && col0 < N) {
          tma_store_2d(&tmC, sbuf, col0, m0);
          tma_store_commit();
        }
      }
    }
    if (store_thread) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// C = sum over the shares of a split product, in order, then what the GEMM epilogue does: rotary embedding of the q / k heads,
// plus what C accumulates onto or the residual, one rounding.  Eight columns per thread; bound by the partials' reads (L2).
__global__ void __launch_bounds__(256) splitk_sum_kernel(const float* __restrict__ part, int splits, int M, int N,
                                                         const __nv_bfloat16* c_in, int64_t ld_in, int accumulate, RopeEpi rp,
                                                         __nv_bfloat16* C, int64_t ldc) {
  after_previous_kernel(part, c_in, rp.cos, rp.sin);
  const int vpr = N / 8;
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (int64_t)M * vpr) return;
  const int row = (int)(i / vpr), col = (int)(i % vpr) * 8;
  auto sum8 = [&](int c, float* a) {
    const float* p = part + (int64_t)row * N + c;
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = 0.f;
#pragma unroll 4
    for (int z = 0; z < splits; ++z) {
      const float4 x = *reinterpret_cast<const float4*>(p + (int64_t)z * M * N), y = *reinterpret_cast<const float4*>(p + (int64_t)z * M * N + 4);
      a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w;
      a[4] += y.x; a[5] += y.y; a[6] += y.z; a[7] += y.w;
    }
  };
  float a[8];
  sum8(col, a);
  if (rope_epi_wants(rp, col & ~63)) {
    // the other half of this head, 64 columns away
    const bool hi = (col & 64) != 0;
    float w[8];
    sum8(hi ? col - 64 : col + 64, w);
    const float* cs = rp.cos + (int64_t)row * 64 + (col & 63);
    const float* sn = rp.sin + (int64_t)row * 64 + (col & 63);
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = a[e] * cs[e] + (hi ? 1.f : -1.f) * w[e] * sn[e];
  }
  if (accumulate) {
    const uint4 old = *reinterpret_cast<const uint4*>(c_in + (int64_t)row * ld_in + col);
    const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float2 f = __bfloat1622float2(o2[t]);
      a[2 * t] += f.x;
      a[2 * t + 1] += f.y;
    }
  }
  uint4 o;
  __nv_bfloat162* p2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int t = 0; t < 4; ++t) p2[t] = __floats2bfloat162_rn(a[2 * t], a[2 * t + 1]);
  *reinterpret_cast<uint4*>(C + (int64_t)row * ldc + col) = o;
}

static int g_num_sms = 0;

template <int LAYOUT, bool ROPE, bool SPLIT = false>
static int launch_gemm(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                       int64_t ldc, int accumulate, const void* c_in, int64_t ld_in, const RopeEpi& rp, int* err,
                       cudaStream_t st, float* part = nullptr, int splits = 1) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_bf16_kernel<LAYOUT, ROPE, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  CUtensorMap tA, tB, tC;
  int r;
  int mn3d = 0;   // bit 0: A tile is one blocked 3-D TMA load, bit 1: B tile is
  if (LAYOUT == 2 && (M % 64) == 0) { r = make_tmap_mn_blocked_bf16(&tA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, BK, BM / 64); mn3d |= 1; }
  else if (LAYOUT == 2) r = make_tmap_2d_bf16(&tA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, 64, 64);
  else r = make_tmap_2d_bf16(&tA, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, 64, BM);
  if (r) return 700000 + r;
  if (LAYOUT == 0) r = make_tmap_2d_bf16(&tB, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, 64, BN);
  else if ((N % 64) == 0) { r = make_tmap_mn_blocked_bf16(&tB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, BK, BN / 64); mn3d |= 2; }
  else r = make_tmap_2d_bf16(&tB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, 64);
  if (r) return 710000 + r;
  r = make_tmap_2d_bf16(&tC, C, (uint64_t)N, (uint64_t)M, (uint64_t)ldc * 2, EPI_COLS, BM);
  if (r) return 720000 + r;
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN) * splits;
  const int grid = tiles < g_num_sms ? tiles : g_num_sms;
  launch_kernel(gemm_bf16_kernel<LAYOUT, ROPE, SPLIT>, grid, NUM_THREADS, SMEM_TOTAL, st, 1, tA, tB, tC, (const __nv_bfloat16*)c_in,
                M, N, K, ld_in, accumulate, mn3d, rp, err, part, splits);
  if (SPLIT)
    launch_kernel(splitk_sum_kernel, (unsigned)(((int64_t)M * (N / 8) + 255) / 256), 256, 0, st, 1, part, splits, M, N,
                  (const __nv_bfloat16*)c_in, ld_in, accumulate, rp, (__nv_bfloat16*)C, ldc);
  return (int)cudaGetLastError();
}

}  // namespace ody

static int g_gemm_variant = 0;
// 0: choose per problem (the pair kernel of gemm_2cta.cu once there are two row blocks to pair up), 1: always the
// one-CTA kernel of this file, 2: always the pair kernel
extern "C" int ody_gemm_set_variant(int v) {
  if (v < 0 || v > 2) return (int)cudaErrorInvalidValue;
  g_gemm_variant = v;
  return 0;
}

// Checks an epilogue description against the problem and turns it into what the kernels take: where the values added
// to the product come from (C itself when accumulating, the residual otherwise) and the rotary description.
extern "C" int ody_gemm_resolve_epilogue(const OdyEpilogue* epi, const void* C, int M, int N, int64_t ldc, int* accumulate,
                                         const void** c_in, int64_t* ld_in, ody::RopeEpi* rp) {
  *c_in = C;
  *ld_in = ldc;
  rp->cos = nullptr;
  rp->sin = nullptr;
  rp->period_cols = rp->rot_cols = 0;
  if (epi == nullptr) return 0;
  if (epi->residual != nullptr) {
    if (*accumulate || (epi->residual_ld % 8) || ((uintptr_t)epi->residual & 15)) return (int)cudaErrorInvalidValue;
    *c_in = epi->residual;
    *ld_in = epi->residual_ld;
    *accumulate = 1;
  }
  if (epi->rope_cos != nullptr) {
    if (epi->rope_sin == nullptr || epi->rope_period_cols <= 0 || (epi->rope_period_cols % 128) || (epi->rope_rot_cols % 128) ||
        epi->rope_rot_cols < 0 || epi->rope_rot_cols > epi->rope_period_cols || (N % 128) ||
        ((uintptr_t)epi->rope_cos & 15) || ((uintptr_t)epi->rope_sin & 15))
      return (int)cudaErrorInvalidValue;
    rp->cos = epi->rope_cos;
    rp->sin = epi->rope_sin;
    rp->period_cols = epi->rope_period_cols;
    rp->rot_cols = epi->rope_rot_cols;
  }
  (void)M;
  return 0;
}

// CTAs that share a tile's k-blocks (1: none).  A product with few output tiles and a long K leaves most SMs idle and the
// others in a long chain (512 x 1024 from K = 32000, the gradient of a small model's last hidden state: 16 tiles of 500
// k-blocks).  Estimates in us: 0.3 per 64-deep k-block of a 128 x 256 tile, operands at 6 TB/s, and for a split one
// more launch and its partials written and read in the L2; a split has to promise a sixth.  That product
// 158 -> 52 us with its sum.  The estimate lacks the operands that every tile fetches again: it puts that product at 26 us (31.6
// with the constants of ody_gemm_cluster_plan), so that for such a K it says which forms are near each other and no more.
// Products that fit one wave of the cluster kernel with a shorter K go there (ody_gemm_cluster_plan).
static int gemm_splits(int M, int N, int K) {
  const int sms = 148;
  if (g_gemm_variant != 0 || (N % 8)) return 1;
  const int64_t tiles = (int64_t)((M + 127) / 128) * ((N + 255) / 256), kblocks = (K + 63) / 64;
  if (tiles > sms / 2 || kblocks < 8) return 1;
  const double mem = ((double)M * K + (double)N * K) * 2.0 / 6.0e6;
  double best = 0.3 * kblocks > mem ? 0.3 * kblocks : mem;
  best *= 0.85;
  int splits = 1;
  for (int s = 2; s <= sms / tiles && s <= 32 && s * 4 <= kblocks; ++s) {
    double t = 0.3 * ((kblocks + s - 1) / s);
    t = (t > mem ? t : mem) + 3.0 + (double)s * M * N * 8.0 / 6.0e6;
    if (t < best) { best = t; splits = s; }
  }
  return splits;
}

// Whether a product goes to the pair kernel.  Both kernels are persistent; what differs per problem is how full their last wave is.
// The pair kernel is the faster one per tile (measured ~6 %), so it is chosen unless its tail costs more than that.
static bool takes_pairs(int M, int N) {
  if (g_gemm_variant != 0 || M <= 128) return g_gemm_variant == 2;
  const int sms = ody::g_num_sms > 0 ? ody::g_num_sms : 148;
  const int64_t t1 = (int64_t)((M + 127) / 128) * ((N + 255) / 256), t2 = (int64_t)((M + 255) / 256) * ((N + 255) / 256);
  const int64_t s1 = sms, s2 = sms / 2;
  const double e1 = (double)t1 / (double)(((t1 + s1 - 1) / s1) * s1), e2 = (double)t2 / (double)(((t2 + s2 - 1) / s2) * s2);
  return e2 * 1.06 >= e1;
}

// Tiles and shares of K for gemm_cluster.cu, or 0 where the kernels above are expected to be as fast.  Estimates in us from
// back-to-back launches of 90 products: a fixed part, so much per 64-deep k-block of a CTA, and what sharing costs at the end.
//   128 x 64 tiles 3.9 + 0.185 (two shares 1.0, four 1.4, eight 1.8 more), 128 x 128 5.4 + 0.196 (1.0, 2.5, 4.0)
//   one-CTA kernel 4.5 + 0.27 a wave, pairs 6.8 + 0.24 a wave, split K 8.5 + 0.3 and its partials written and read (too little for
//   512 x 1024 from K = 32000: 31.6 us against 52, see gemm_splits)
// At most one wave of CTAs (clusters leave SMs of a GPC unused: 128 CTAs in clusters of eight take two rounds), and at most 192
// k-blocks to a CTA: beyond that the wide tiles' smaller operand traffic wins (1024 x 1024 from K = 32000: 60 us, here 63).
// Measured, before -> cluster: 128 x 3072 from K = 1024 9.7 -> 6.6, 128 x 1024 from 2816 13.1 -> 7.4, 512 x 1024 from 1024 10.3 -> 6.6,
// from 5632 17.3 -> 12.7, 1531 x 1024 from 1536 12.7 -> 10.5, 1024 x 1024 from 2816 18.4 -> 11.4, 128 x 4096 from 11008 30.7 -> 22.0.
// Products that the split kernel shares among more CTAs than a cluster has are the faster ones here too: 128 x 256 from K = 4096 12.6
// -> 6.6, from 12288 15.8 -> 9.6, 1 x 256 from 4096 7.7 -> 4.2, 512 x 64 from 12288 12.0 -> 9.6, 218 x 72 from 10728 13.0 -> 10.9.
extern "C" int ody_gemm_cluster_plan(int M, int N, int K, int rope, int* bn, int* splits) {
  if (g_gemm_variant != 0 || M <= 0 || N <= 0 || K <= 0 || (N % 8)) return 0;
  const int64_t kblocks = (K + 63) / 64, tiles = (int64_t)((M + 127) / 128) * ((N + 255) / 256);
  const int s_old = gemm_splits(M, N, K);
  double limit;
  if (s_old > 1) {
    limit = 8.5 + 0.3 * ((kblocks + s_old - 1) / s_old) + (double)s_old * M * N * 8.0 / 6.0e6;
  } else if (takes_pairs(M, N)) {
    limit = 6.8 + 0.24 * kblocks * (((int64_t)((M + 255) / 256) * ((N + 255) / 256) + 73) / 74);
  } else {
    limit = 4.5 + 0.27 * kblocks * ((tiles + 147) / 148);
  }
  double best = 0.95 * limit;
  int found = 0;
  for (int b = rope ? 128 : 64; b <= 128; b += 64) {
    const int64_t t = (int64_t)((M + 127) / 128) * ((N + b - 1) / b);
    for (int i = 0, s = 1; i < 4 && s <= kblocks; ++i, s *= 2) {
      static const int max_ctas[4] = {148, 144, 128, 64};
      static const double sharing[2][4] = {{0.0, 1.0, 1.4, 1.8}, {0.0, 1.0, 2.5, 4.0}};
      const int64_t kb = (kblocks + s - 1) / s;
      if (t * s > max_ctas[i] || kb > 192) continue;
      const double e = (b == 64 ? 3.9 + 0.185 * kb : 5.4 + 0.196 * kb) + sharing[b / 128][i];
      if (e < best) { best = e; *bn = b; *splits = s; found = 1; }
    }
  }
  return found;
}

// Scratch ody_gemm_bf16_ws can use for this product; 0: it is not split.
extern "C" int64_t ody_gemm_split_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const int s = gemm_splits(M, N, K);
  return s > 1 ? (int64_t)s * M * N * 4 : 0;
}

// ody_gemm_bf16_ex with scratch (16-byte aligned, ody_gemm_split_bytes of the sizes; none is needed where ody_gemm_cluster_plan
// answers): products with few tiles share K.
extern "C" int ody_gemm_bf16_ws(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                                int64_t ldc, int layout, int accumulate, const OdyEpilogue* epi, void* ws, int64_t ws_bytes,
                                int* err, cudaStream_t st) {
  int bn, shares;
  if (ody_gemm_cluster_plan(M, N, K, epi != nullptr && epi->rope_cos != nullptr, &bn, &shares))
    return ody_gemm_bf16_cluster(A, B, C, M, N, K, lda, ldb, ldc, layout, accumulate, epi, bn, shares, err, st);
  const int64_t need = ody_gemm_split_bytes(M, N, K);
  if (need == 0 || ws == nullptr || ws_bytes < need || ((uintptr_t)ws & 15))
    return ody_gemm_bf16_ex(A, B, C, M, N, K, lda, ldb, ldc, layout, accumulate, epi, err, st);
  if ((lda % 8) || (ldb % 8) || (ldc % 8) || (N % 8) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15) || ((uintptr_t)C & 15))
    return (int)cudaErrorInvalidValue;
  const void* c_in;
  int64_t ld_in;
  ody::RopeEpi rp;
  if (int r = ody_gemm_resolve_epilogue(epi, C, M, N, ldc, &accumulate, &c_in, &ld_in, &rp)) return r;
  if (rp.cos != nullptr && layout != 0) return (int)cudaErrorInvalidValue;
  const int splits = gemm_splits(M, N, K);
  switch (layout) {
    case 0: return ody::launch_gemm<0, false, true>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, err, st, (float*)ws, splits);
    case 1: return ody::launch_gemm<1, false, true>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, err, st, (float*)ws, splits);
    case 2: return ody::launch_gemm<2, false, true>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, err, st, (float*)ws, splits);
  }
  return (int)cudaErrorInvalidValue;
}

extern "C" int ody_gemm_bf16_ex(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                                int64_t ldc, int layout, int accumulate, const OdyEpilogue* epi, int* err, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return (int)cudaErrorInvalidValue;
  if (takes_pairs(M, N)) return ody_gemm_bf16_2cta_ex(A, B, C, M, N, K, lda, ldb, ldc, layout, accumulate, epi, err, st);
  if ((lda % 8) || (ldb % 8) || (ldc % 8) || (N % 8) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15) || ((uintptr_t)C & 15))
    return (int)cudaErrorInvalidValue;
  const void* c_in;
  int64_t ld_in;
  ody::RopeEpi rp;
  if (int r = ody_gemm_resolve_epilogue(epi, C, M, N, ldc, &accumulate, &c_in, &ld_in, &rp)) return r;
  if (rp.cos != nullptr)   // a forward projection: layout 0 only
    return layout == 0 ? ody::launch_gemm<0, true>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, err, st)
                       : (int)cudaErrorInvalidValue;
  switch (layout) {
    case 0: return ody::launch_gemm<0, false>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, err, st);
    case 1: return ody::launch_gemm<1, false>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, err, st);
    case 2: return ody::launch_gemm<2, false>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, err, st);
  }
  return (int)cudaErrorInvalidValue;
}

extern "C" int ody_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                             int64_t ldc, int layout, int accumulate, int* err, cudaStream_t st) {
  return ody_gemm_bf16_ex(A, B, C, M, N, K, lda, ldb, ldc, layout, accumulate, nullptr, err, st);
}
