// bf16 GEMM for products with few output tiles: small tiles, the K dimension shared by the CTAs of a cluster.
//
// Same contract as gemm.cu (layouts 0 NT, 1 NN, 2 TN; rotary embedding, residual and accumulation in the epilogue).  The
// kernels of gemm.cu and gemm_2cta.cu work on 128 x 256 and 256 x 256 tiles: a linear layer of a narrow model or of a short
// sequence has 4 - 48 of those, each a serial chain over all of K on one SM while the others idle.  Here a tile is 128 x 64 or
// 128 x 128 and the S CTAs of a cluster take a share of its k-blocks each.  The fp32 shares meet in distributed shared
// memory: every CTA leaves its accumulator in its own shared memory, and after a cluster barrier CTA z adds rows [128 z / S,
// 128 (z + 1) / S) of all of them, in order, applies the epilogue and writes them - no scratch, no second kernel, no atomics.
//
// 192 threads: warp 0 = TMA producer, warp 1 = MMA issuer and TMEM owner, warps 2-5 move the accumulator to shared memory;
// all six add.  Loads are plain TMA loads of each CTA's own operands (no multicast).  Every wait on an mbarrier is bounded; the
// two cluster barriers are reached by every thread on every path.
#include <limits.h>

#include "ody_kernels.h"
#include "sm100.cuh"
#include "launch.cuh"

extern "C" int ody_gemm_resolve_epilogue(const OdyEpilogue* epi, const void* C, int M, int N, int64_t ldc, int* accumulate,
                                         const void** c_in, int64_t* ld_in, ody::RopeEpi* rp);

namespace ody {
namespace gs {

constexpr int BM = 128, BK = 64, UMMA_K = 16;
constexpr int A_BYTES = BM * BK * 2;
constexpr int NUM_THREADS = 192;
// 128 x 64 tiles: 8 stages of 24 KB; 128 x 128 tiles: 6 stages of 32 KB.  These products are bound by the latency of their loads, so
// the ring takes what an SM has (four stages of 128 x 64, two CTAs to an SM: 128 x 1024 from K = 2816 8.1 us, this 7.4; three
// stages of 128 x 128: 1024 x 1024 from 2816 13.3, this 11.4).
template <int BN> constexpr int stages() { return BN == 64 ? 8 : 6; }
template <int BN> constexpr int stage_bytes() { return A_BYTES + BN * BK * 2; }
template <int BN> constexpr int ring_bytes() { return stages<BN>() * stage_bytes<BN>(); }
template <int BN> constexpr int smem_total() { return ring_bytes<BN>() + 256 + 1024; }
template <int BN> constexpr int row_bytes() { return BN * 4 + 16; }      // fp32 row of the tile; the pad keeps 16-byte pieces of 8 rows apart
static_assert(BM * row_bytes<64>() <= ring_bytes<64>() && BM * row_bytes<128>() <= ring_bytes<128>(), "the accumulator fits the ring");

struct Bars {
  uint64_t full[8], empty[8], acc_full, drain;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// 8 columns of one row: bf16 of a (plus what C accumulates onto or the residual)
__device__ __forceinline__ void finish8(float* a, const __nv_bfloat16* add, __nv_bfloat16* dst) {
  if (add != nullptr) {
    const uint4 old = *reinterpret_cast<const uint4*>(add);
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
  *reinterpret_cast<uint4*>(dst) = o;
}

template <int LAYOUT, int BN, bool ROPE>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __nv_bfloat16* c_in,
                    int64_t ld_in, __nv_bfloat16* C, int64_t ldc, int M, int N, int K, int splits, int accumulate, int mn3d,
                    RopeEpi rp, int* __restrict__ err) {
  static_assert(!ROPE || BN == 128, "a rotated head needs both of its halves");
  constexpr int ST = stages<BN>(), STAGE = stage_bytes<BN>(), ROW = row_bytes<BN>();
  constexpr bool A_MN = (LAYOUT == 2), B_MN = (LAYOUT != 0);
  constexpr uint32_t IDESC = make_idesc_bf16(BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Bars* bars = (Bars*)(smem + ring_bytes<BN>());
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int z = (int)cluster_rank();                         // clusters are `splits` CTAs along x
  const int tile = blockIdx.x / splits;
  const int tiles_m = (M + BM - 1) / BM;
  const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * BN;
  const int kblocks = (K + BK - 1) / BK;
  const int kb0 = (int)((int64_t)kblocks * z / splits), kb1 = (int)((int64_t)kblocks * (z + 1) / splits);   // not empty: splits <= kblocks

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) { mbar_init(&bars->full[s], 1); mbar_init(&bars->empty[s], 1); }
    mbar_init(&bars->acc_full, 1);
    mbar_init(&bars->drain, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) { tmem_alloc(&bars->tmem_base, BN); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  if constexpr (ROPE) after_previous_kernel(c_in, rp.cos, rp.sin); else after_previous_kernel(c_in);

  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&bars->empty[stage], phase ^ 1, abort_flag, err, ODY_ERR_TIMEOUT_EMPTY)) { ok = false; break; }
        uint8_t* sA = smem + stage * STAGE;
        uint8_t* sB = sA + A_BYTES;
        uint64_t* full = &bars->full[stage];
        mbar_expect_tx(full, STAGE);
        const int k0 = kb * BK;
        if (!A_MN) {
          tma_load_2d(sA, &tmA, k0, m0, full);
        } else if (mn3d & 1) {
          tma_load_3d(sA, &tmA, 0, k0, m0 / 64, full);
        } else {
#pragma unroll
          for (int j = 0; j < BM / 64; ++j) tma_load_2d(sA + j * 8192, &tmA, m0 + 64 * j, k0, full);
        }
        if (!B_MN) {
          tma_load_2d(sB, &tmB, k0, n0, full);
        } else if (mn3d & 2) {
          tma_load_3d(sB, &tmB, 0, k0, n0 / 64, full);
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(sB + j * 8192, &tmB, n0 + 64 * j, k0, full);
        }
        ++issued;
        if (++stage == ST) { stage = 0; phase ^= 1; }
      }
      if (!ok || *abort_flag) {
        // give copies still in flight a bounded chance to land before this shared memory is used for anything else
        const int n = issued < ST ? issued : ST;
        for (int i = 0; i < n; ++i) {
          if (--stage < 0) { stage = ST - 1; phase ^= 1; }
          const long long t0 = clock64();
          while (!mbar_try_wait(&bars->full[stage], phase) && clock64() - t0 < ODY_SPIN_LIMIT_CYCLES / 8) {}
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const bool leader = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    const uint32_t s0 = smem_u32(smem);
    const uint64_t adesc0 = A_MN ? make_smem_desc(s0, 8192, 1024) : make_smem_desc(s0, 16, 1024);
    const uint64_t bdesc0 = B_MN ? make_smem_desc(s0 + A_BYTES, 8192, 1024) : make_smem_desc(s0 + A_BYTES, 16, 1024);
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait(&bars->full[stage], phase, abort_flag, err, ODY_ERR_TIMEOUT_FULL)) { ok = false; break; }
      tc_fence_after();
      const uint64_t a0 = desc_advance(adesc0, stage * STAGE), b0 = desc_advance(bdesc0, stage * STAGE);
#pragma unroll
      for (int kk = 0; kk < BK / UMMA_K; ++kk)
        if (leader) umma_ss(tmem, desc_advance(a0, kk * (A_MN ? 2048 : 32)), desc_advance(b0, kk * (B_MN ? 2048 : 32)), IDESC, kk > 0 || kb > kb0 ? 1u : 0u);
      if (leader) umma_commit(&bars->empty[stage]);
      if (++stage == ST) { stage = 0; phase ^= 1; }
    }
    if (ok) {
      if (leader) umma_commit(&bars->acc_full);
    } else {
      if (leader) umma_commit(&bars->drain);
      const long long t0 = clock64();
      while (!mbar_try_wait(&bars->drain, 0) && clock64() - t0 < ODY_SPIN_LIMIT_CYCLES / 8) {}
    }
    __syncwarp();
  } else {
    const int q = warp & 3, r = q * 32 + lane;               // TMEM lane quarter of this warp, row of the tile
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_full, 0, abort_flag, err, ODY_ERR_TIMEOUT_TMEM_FULL));
    if (ok) {
      // all loads of this CTA have been consumed: the ring takes the fp32 tile
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < BN; c += 64) {
        uint32_t v[64];
        tmem_ld_32x32(tmem + ((uint32_t)(q * 32) << 16) + c, v);
        tmem_ld_32x32(tmem + ((uint32_t)(q * 32) << 16) + c + 32, v + 32);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j)
          *reinterpret_cast<uint4*>(smem + r * ROW + c * 4 + j * 16) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
    }
    tc_fence_before();
  }
  cluster_sync();            // every share lies in its CTA's shared memory
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, BN); }

  if (!*abort_flag) {
    const int r0 = BM * z / splits, r1 = min(BM * (z + 1) / splits, M - m0);
    const uint32_t s0 = smem_u32(smem);
    constexpr int PER_ROW = ROPE ? 8 : BN / 8;               // work items of a row: 8 columns, or 8 columns of both halves of a head
    for (int i = threadIdx.x; i < (r1 - r0) * PER_ROW; i += NUM_THREADS) {
      const int r = r0 + i / PER_ROW, c = (i % PER_ROW) * 8;
      if (n0 + c >= N) continue;                             // N is a multiple of 8, with ROPE of 128
      constexpr int P = ROPE ? 2 : 1;
      float a[P][8];
#pragma unroll
      for (int p = 0; p < P; ++p)
#pragma unroll
        for (int e = 0; e < 8; ++e) a[p][e] = 0.f;
#pragma unroll 4
      for (int s = 0; s < splits; ++s) {
        const uint32_t src = map_to_cta(s0 + r * ROW + c * 4, s);
#pragma unroll
        for (int p = 0; p < P; ++p) {
          const float4 x = ld_cluster(src + p * 256), y = ld_cluster(src + p * 256 + 16);
          a[p][0] += x.x; a[p][1] += x.y; a[p][2] += x.z; a[p][3] += x.w;
          a[p][4] += y.x; a[p][5] += y.y; a[p][6] += y.z; a[p][7] += y.w;
        }
      }
      const int64_t row = m0 + r;
      if constexpr (ROPE) {
        if (rope_epi_wants(rp, n0)) {
          const float* cs = rp.cos + row * 64 + c;
          const float* sn = rp.sin + row * 64 + c;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float co = __ldg(cs + e), si = __ldg(sn + e), lo = a[0][e], hi = a[1][e];
            a[0][e] = lo * co - hi * si;
            a[1][e] = hi * co + lo * si;
          }
        }
      }
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const int col = n0 + c + p * 64;
        finish8(a[p], accumulate ? c_in + row * ld_in + col : nullptr, C + row * ldc + col);
      }
    }
  }
  cluster_sync();            // nobody leaves while its shared memory is being read
}

template <int LAYOUT, int BN, bool ROPE>
static int launch(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc, int accumulate,
                  const void* c_in, int64_t ld_in, const RopeEpi& rp, int splits, int* err, cudaStream_t st) {
  static std::atomic<uint64_t> done{0};
  if (int r = allow_smem(gemm_cluster_kernel<LAYOUT, BN, ROPE>, smem_total<BN>(), done)) return r;
  CUtensorMap tA, tB;
  int r, mn3d = 0;   // bit 0: the A tile is one blocked 3-D load, bit 1: the B tile is
  if (LAYOUT != 2) r = make_tmap_2d_bf16(&tA, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, 64, BM);
  else if (M % 64 == 0) { r = make_tmap_mn_blocked_bf16(&tA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, BK, BM / 64); mn3d |= 1; }
  else r = make_tmap_2d_bf16(&tA, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, 64, 64);
  if (r) return 700000 + r;
  if (LAYOUT == 0) r = make_tmap_2d_bf16(&tB, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, 64, BN);
  else if (N % 64 == 0) { r = make_tmap_mn_blocked_bf16(&tB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, BK, BN / 64); mn3d |= 2; }
  else r = make_tmap_2d_bf16(&tB, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, 64);
  if (r) return 710000 + r;
  const int64_t ctas = (int64_t)((M + BM - 1) / BM) * ((N + BN - 1) / BN) * splits;
  if (ctas > INT_MAX) return (int)cudaErrorInvalidValue;
  return launch_kernel(gemm_cluster_kernel<LAYOUT, BN, ROPE>, (unsigned)ctas, NUM_THREADS, smem_total<BN>(), st, splits, tA, tB,
                       (const __nv_bfloat16*)c_in, ld_in, (__nv_bfloat16*)C, ldc, M, N, K, splits, accumulate, mn3d, rp, err);
}

}  // namespace gs
}  // namespace ody

extern "C" int ody_gemm_bf16_cluster(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc,
                                     int layout, int accumulate, const OdyEpilogue* epi, int bn, int splits, int* err, cudaStream_t st) {
  using namespace ody::gs;
  if (M <= 0 || N <= 0 || K <= 0 || layout < 0 || layout > 2 || (bn != 64 && bn != 128)) return (int)cudaErrorInvalidValue;
  if (splits < 1 || splits > 8 || splits > (K + BK - 1) / BK) return (int)cudaErrorInvalidValue;
  if ((lda % 8) || (ldb % 8) || (ldc % 8) || (N % 8) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15) || ((uintptr_t)C & 15))
    return (int)cudaErrorInvalidValue;
  const void* c_in;
  int64_t ld_in;
  ody::RopeEpi rp;
  if (int r = ody_gemm_resolve_epilogue(epi, C, M, N, ldc, &accumulate, &c_in, &ld_in, &rp)) return r;
  if (rp.cos != nullptr)
    return layout == 0 && bn == 128 ? launch<0, 128, true>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, splits, err, st)
                                    : (int)cudaErrorInvalidValue;
#define ODY_GS(L)                                                                                                              \
  return bn == 64 ? launch<L, 64, false>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, splits, err, st)         \
                  : launch<L, 128, false>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, c_in, ld_in, rp, splits, err, st)
  if (layout == 0) ODY_GS(0);
  if (layout == 1) ODY_GS(1);
  ODY_GS(2);
#undef ODY_GS
}
