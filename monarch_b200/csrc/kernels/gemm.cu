// Host launchers for the tcgen05 GEMM (see gemm_tcgen05.cuh).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdio.h>

#include "gemm2_tcgen05.cuh"
#include "gemm_tcgen05.cuh"
#include "mb200.h"

namespace mb200 {

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                              const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn get_encode() {
  static EncodeFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeFn>(p);
  }
  return fn;
}

// 2-D bf16 tensor map: inner extent `inner` (contiguous), outer extent `outer` with
// leading dimension `ld` elements; box = {box_inner, box_outer}; 128-byte swizzle.
int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                      uint64_t ld, uint32_t box_inner, uint32_t box_outer) {
  EncodeFn enc = get_encode();
  if (!enc) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld & 7)) return -2;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

static int sm_count(int dev) {
  static PerDevice<int> known;
  int* n = known.at(dev);
  int now = n ? *n : 0;
  if (!now) {
    cudaDeviceGetAttribute(&now, cudaDevAttrMultiProcessorCount, dev < 0 ? 0 : dev);
    if (n) *n = now;
  }
  return now;
}
int sm_count() {
  return sm_count(current_device());
}

template <bool A_MN, bool B_MN, int BN, int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA,
                     const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  gemm_cta_body<A_MN, B_MN, BN, EPI>(&tmA, &tmB, p, blockIdx.x, gridDim.x, smem_raw);
}

template <bool A_MN, bool B_MN, int BN, int EPI = kEpiStore>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int grid,
                  cudaStream_t st, int dev) {
  static PerDevice<int> smem_ok;
  if (const cudaError_t e =
          allow_smem(gemm_bf16_kernel<A_MN, B_MN, BN, EPI>, GemmTile<BN>::kSmemBytes, smem_ok, dev))
    return (int)e;
  return (int)launch_dep(gemm_bf16_kernel<A_MN, B_MN, BN, EPI>, grid, GEMM_THREADS,
                         GemmTile<BN>::kSmemBytes, st, ta, tb, p);
}

static int make_gemm_tmaps_bn(CUtensorMap* ta, CUtensorMap* tb, const void* A, const void* B,
                              int M, int N, int K, int lda, int ldb, int a_mn, int b_mn, int bn) {
  int r;
  if (a_mn)
    r = make_tmap_bf16_2d(ta, A, M, K, lda, 64, 64);
  else
    r = make_tmap_bf16_2d(ta, A, K, M, lda, 64, GEMM_BM);
  if (r) return r;
  if (b_mn)
    r = make_tmap_bf16_2d(tb, B, N, K, ldb, 64, 64);
  else
    r = make_tmap_bf16_2d(tb, B, K, N, ldb, 64, bn);
  return r;
}
int make_gemm_tmaps(CUtensorMap* ta, CUtensorMap* tb, const void* A, const void* B, int M, int N,
                    int K, int lda, int ldb, int a_mn, int b_mn) {
  return make_gemm_tmaps_bn(ta, tb, A, B, M, N, K, lda, ldb, a_mn, b_mn, GEMM_BN);
}

template <int BN>
static int launch_gemm_bn(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                          int a_mn, int b_mn, int grid, cudaStream_t st, int dev) {
  if (a_mn && b_mn) return launch<true, true, BN>(ta, tb, p, grid, st, dev);
  if (a_mn) return launch<true, false, BN>(ta, tb, p, grid, st, dev);
  if (b_mn) return launch<false, true, BN>(ta, tb, p, grid, st, dev);
  return launch<false, false, BN>(ta, tb, p, grid, st, dev);
}
int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int a_mn,
                int b_mn, int grid, cudaStream_t st) {
  return launch_gemm_bn<GEMM_BN>(ta, tb, p, a_mn, b_mn, grid, st, current_device());
}

// ------------------------------------------------------------------- split over K
// A product with fewer tiles than SMs is bound by what one SM can fetch (64 to 76 B/clk by
// TMA, measured), not by the tensor cores.  Here a cluster of SPLIT CTAs shares one 128 x BN
// tile: each multiplies its part of K, leaves the fp32 partial tile in its own shared memory
// (the stage buffers are free by then), and after a cluster barrier each CTA adds up
// 128 / SPLIT rows of all parts over distributed shared memory, in rank order, and stores
// them.  No workspace, no second launch, the same bits on every run.
// 64x4096x14336: 69.8 us as 256x256 pair tiles -> 25.7 us (4.5 TB/s); 64x4096x4096: 24.3 -> 10.1 us.
template <int BN, int SPLIT>
struct SplitTile {
  static constexpr int kLd = BN + 4;   // floats per row of the partial tile: no bank conflicts
  static_assert(GEMM_BM * kLd * 4 <= GemmTile<BN>::kStages * GemmTile<BN>::kStageBytes, "");
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(cluster_addr)
               : "memory");
  return v;
}

template <bool A_MN, bool B_MN, int BN, int SPLIT>
__global__ void __cluster_dims__(SPLIT, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
    gemm_split_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  constexpr int STAGES = GemmTile<BN>::kStages;
  constexpr int STAGE_BYTES = GemmTile<BN>::kStageBytes;
  constexpr int LD = SplitTile<BN, SPLIT>::kLd;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  auto* sh = reinterpret_cast<GemmShared<STAGES>*>(smem + STAGES * STAGE_BYTES);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int part = (int)cluster_ctarank();
  const int tile = (int)blockIdx.x / SPLIT;
  const int m_blocks = (p.M + GEMM_BM - 1) / GEMM_BM;
  const int m0 = (tile % m_blocks) * GEMM_BM, n0 = (tile / m_blocks) * BN;
  const int all_iters = (p.K + GEMM_BK - 1) / GEMM_BK;   // >= SPLIT (launcher)
  const int k_begin = (int)((long long)all_iters * part / SPLIT);
  const int k_end = (int)((long long)all_iters * (part + 1) / SPLIT);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    mbar_init(&sh->tmem_full[0], 1);
    sh->abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&sh->tmem_base, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  volatile int* abort_word = &sh->abort_word;
  dep_wait();

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      int stage = 0;
      uint32_t phase = 0;
      for (int k = k_begin; k < k_end; ++k) {
        if (!mbar_wait(&sh->empty[stage], phase ^ 1, abort_word, p.status)) break;
        uint8_t* sa = smem + stage * STAGE_BYTES;
        uint8_t* sb = sa + GEMM_A_BYTES;
        mbar_expect_tx(&sh->full[stage], STAGE_BYTES);
        const int k0 = k * GEMM_BK;
        if (A_MN) {
#pragma unroll
          for (int j = 0; j < GEMM_BM / 64; ++j)
            tma_load_2d(sa + j * 8192, &tmA, &sh->full[stage], m0 + j * 64, k0);
        } else {
          tma_load_2d(sa, &tmA, &sh->full[stage], k0, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)
            tma_load_2d(sb + j * 8192, &tmB, &sh->full[stage], n0 + j * 64, k0);
        } else {
          tma_load_2d(sb, &tmB, &sh->full[stage], k0, n0);
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(GEMM_BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int k = k_begin; k < k_end; ++k) {
        ok = mbar_wait(&sh->full[stage], phase, abort_word, p.status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
        const uint32_t sb = sa + GEMM_A_BYTES;
#pragma unroll
        for (int kk = 0; kk < GEMM_BK / 16; ++kk) {
          const uint64_t da = A_MN ? umma_smem_desc_sw128(sa + kk * 2048, 8192, 1024)
                                   : umma_smem_desc_sw128(sa + kk * 32, 16, 1024);
          const uint64_t db = B_MN ? umma_smem_desc_sw128(sb + kk * 2048, 8192, 1024)
                                   : umma_smem_desc_sw128(sb + kk * 32, 16, 1024);
          umma_f16(tmem_base, da, db, idesc, (k > k_begin || kk > 0) ? 1u : 0u);
        }
        umma_commit(&sh->empty[stage]);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok) umma_commit(&sh->tmem_full[0]);
    }
  } else {
    // every load of this CTA has landed and every MMA has read its stage once tmem_full is
    // signalled, so the stage buffers can take the partial tile
    const int quad = warp & 3;
    if (mbar_wait(&sh->tmem_full[0], 0, abort_word, p.status)) {
      tc_fence_after();
      float* row = reinterpret_cast<float*>(smem) + (quad * 32 + lane) * LD;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(tmem_base + c * 32 + ((uint32_t)(quad * 32) << 16), v);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<uint4*>(row + c * 32 + q * 4) =
              make_uint4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
      }
    }
  }
  tc_fence_before();
  cluster_sync_all();   // all parts are in shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
  {
    constexpr int ROWS = GEMM_BM / SPLIT;
    const bool vec_ok = ((p.ldc & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0) &&
                        (!p.R || (((p.ldr & 7) == 0) &&
                                  ((reinterpret_cast<uintptr_t>(p.R) & 15) == 0)));
    const uint32_t base = smem_u32(smem);
    for (int it = threadIdx.x; it < ROWS * (BN / 8); it += GEMM_THREADS) {
      const int r = part * ROWS + it / (BN / 8), c = (it % (BN / 8)) * 8;
      const int row = m0 + r, col = n0 + c;
      if (row >= p.M || col >= p.N) continue;
      float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < SPLIT; ++s) {
        const uint32_t src = mapa_u32(base + (uint32_t)(r * LD + c) * 4, s);
        const float4 x = ld_cluster_f4(src), y = ld_cluster_f4(src + 16);
        f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
        f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
      }
      gemm_store8(p, f, row, col, vec_ok);
    }
  }
  cluster_sync_all();   // keep the parts until every CTA of the cluster has read them
}

// Number of clusters of SPLIT CTAs that can be resident at once; 0 when there is no answer.
template <bool A_MN, bool B_MN, int BN, int SPLIT>
static int split_capacity(int dev) {
  static PerDevice<int> known;   // capacity + 1
  int* cap = known.at(dev);
  if (cap && *cap) return *cap - 1;
  static PerDevice<int> smem_ok;
  if (allow_smem(gemm_split_kernel<A_MN, B_MN, BN, SPLIT>, GemmTile<BN>::kSmemBytes, smem_ok,
                 dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(SPLIT * (sm_count(dev) / SPLIT));
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = GemmTile<BN>::kSmemBytes;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = SPLIT;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_split_kernel<A_MN, B_MN, BN, SPLIT>, &cfg) !=
      cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  if (cap) *cap = n + 1;
  return n;
}

template <bool A_MN, bool B_MN, int BN, int SPLIT>
static int launch_split(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                        int tiles, cudaStream_t st, int dev) {
  if (split_capacity<A_MN, B_MN, BN, SPLIT>(dev) <= 0) return 1002;
  return (int)launch_dep(gemm_split_kernel<A_MN, B_MN, BN, SPLIT>, tiles * SPLIT, GEMM_THREADS,
                         GemmTile<BN>::kSmemBytes, st, ta, tb, p);
}
template <int BN, int SPLIT>
static int launch_split_ab(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                           int a_mn, int b_mn, int tiles, cudaStream_t st, int dev) {
  if (a_mn && b_mn) return launch_split<true, true, BN, SPLIT>(ta, tb, p, tiles, st, dev);
  if (a_mn) return launch_split<true, false, BN, SPLIT>(ta, tb, p, tiles, st, dev);
  if (b_mn) return launch_split<false, true, BN, SPLIT>(ta, tb, p, tiles, st, dev);
  return launch_split<false, false, BN, SPLIT>(ta, tb, p, tiles, st, dev);
}
template <int BN>
static int launch_split_n(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                          int a_mn, int b_mn, int split, int tiles, cudaStream_t st, int dev) {
  if (split == 8) return launch_split_ab<BN, 8>(ta, tb, p, a_mn, b_mn, tiles, st, dev);
  if (split == 4) return launch_split_ab<BN, 4>(ta, tb, p, a_mn, b_mn, tiles, st, dev);
  return launch_split_ab<BN, 2>(ta, tb, p, a_mn, b_mn, tiles, st, dev);
}

// ------------------------------------------------------------------ CTA-pair variant
template <bool A_MN, bool B_MN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(gemm2_threads(EPI), 1)
    gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  gemm2_cta_body<A_MN, B_MN, EPI>(&tmA, &tmB, p, blockIdx.x >> 1, gridDim.x >> 1, smem_raw);
}

// Number of CTA pairs that can be resident at once (<= SMs / 2; fewer when a GPC has an
// odd number of usable SMs).  Queried once per operand-layout variant.
template <bool A_MN, bool B_MN, int EPI>
static int pair_capacity() {
  static PerDevice<int> known, smem_ok;
  const int dev = current_device();
  int* cap = known.at(dev);
  if (cap && *cap) return *cap;
  if (allow_smem(gemm2_bf16_kernel<A_MN, B_MN, EPI>, G2_SMEM_BYTES, smem_ok, dev) != cudaSuccess)
    return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (sm_count() / 2));
  cfg.blockDim = dim3(gemm2_threads(EPI));
  cfg.dynamicSmemBytes = G2_SMEM_BYTES;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemm2_bf16_kernel<A_MN, B_MN, EPI>, &cfg) != cudaSuccess ||
      n <= 0) {
    cudaGetLastError();
    n = sm_count() / 2;
  }
  if (n > sm_count() / 2) n = sm_count() / 2;
  if (cap) *cap = n;
  return n;
}

template <bool A_MN, bool B_MN, int EPI = kEpiStore>
static int launch2(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                   cudaStream_t st) {
  const int cap = pair_capacity<A_MN, B_MN, EPI>();
  if (cap <= 0) return 1002;
  const int tiles = ((p.M + G2_BM - 1) / G2_BM) * ((p.N + G2_BN - 1) / G2_BN);
  const int pairs = tiles < cap ? tiles : cap;
  return (int)launch_dep(gemm2_bf16_kernel<A_MN, B_MN, EPI>, 2 * pairs, gemm2_threads(EPI),
                         G2_SMEM_BYTES, st, ta, tb, p);
}

int make_gemm2_tmaps(CUtensorMap* ta, CUtensorMap* tb, const void* A, const void* B, int M, int N,
                     int K, int lda, int ldb, int a_mn, int b_mn) {
  int r;
  if (a_mn)
    r = make_tmap_bf16_2d(ta, A, M, K, lda, 64, 64);
  else
    r = make_tmap_bf16_2d(ta, A, K, M, lda, 64, G2_HALF);
  if (r) return r;
  if (b_mn)
    r = make_tmap_bf16_2d(tb, B, N, K, ldb, 64, 64);
  else
    r = make_tmap_bf16_2d(tb, B, K, N, ldb, 64, G2_HALF);
  return r;
}

int launch_gemm2(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int a_mn,
                 int b_mn, cudaStream_t st) {
  if (a_mn && b_mn) return launch2<true, true>(ta, tb, p, st);
  if (a_mn) return launch2<true, false>(ta, tb, p, st);
  if (b_mn) return launch2<false, true>(ta, tb, p, st);
  return launch2<false, false>(ta, tb, p, st);
}

// 1: single-CTA 128x256 tiles; 2: CTA-pair 256x256 tiles, or smaller ones where gemm_plan
// finds them faster.
static int g_gemm_impl = 2;

// Tile and K split of the plain product under implementation 2: the smallest estimate of
//   t0 + (waves - 1) * max(steps * c, e) + steps * c,   steps: 64-deep steps of one CTA or pair
// with the microseconds measured on this chip.  c is what limits a step: 32 KB per SM and the
// tensor pipe for the pair, the 24 to 48 KB that one SM fetches for the others.  e is a tile's
// epilogue, which a further wave hides behind its products or waits for; t0 is launch, first
// load, last epilogue; a split adds its cluster barriers and the exchange.  Estimate ->
// measured, us: 8192x1024x1024 pair 18.0 -> 18.1; 2048x4096x4096 pair 51.2 -> 50.2, 128x256
// 54.5 -> 55.1, 128x128 67.0 -> 68.7; 2048^3 128x256 17.5 -> 15.2, pair 18.0 -> 16.6;
// 1000x2048x3072 128x128 16.1 -> 14.4, pair 23.6 -> 21.2; 200x768x256 128x64 4.4 -> 4.7, pair
// 8.4 -> 9.0; 64x4096x4096 128x128 in 4 parts 10.3 -> 10.1, 128x64 in 2 parts 10.8 -> 11.1;
// 3928x10808x38 pair 41.5 -> 47.8, 128x256 29.1 -> 35.7, 128x64 35.6 -> 43.2.
//
// Rows of A, B or C that do not start on 128-byte lines make a step of the single CTAs longer by
// `unaligned`, for 128x256 always, for the narrower ones once there is more than one wave (the
// pair's tiles share fewer lines with their neighbours): 2944x408x5432 128x256 53.4 us, pair 41.3;
// 352x13448x1352 128x128 31.7 and 28.8; 6968x984x912 27.1 and 24.6; but 3072x2048x1000 with both
// operands along 3072 and 2048 128x128 15.8 and 17.8.
//
// Over 243 products without a split (K from 1 to 15768, four layouts; e and `unaligned` are
// fitted to them, t0 and c are from aligned ones) the choice takes 0.6 % more than the best tile
// and 3 are slower than the pair by over 1 %, by at most 5 %; without e and `unaligned` 3.5 % more,
// 34 slower than the pair, by up to 17 %.
struct GemmPlan {
  int bn;      // 0: the CTA pair's 256x256 tile, else the columns of a single CTA's 128-row tile
  int split;   // CTAs of a cluster that share a tile along K
};
// Clusters of `split` CTAs that run at once (they have to share a GPC: fewer than SMs / split).
static int split_clusters(int bn, int split, int dev) {
  if (bn == 64)
    return split == 2   ? split_capacity<false, false, 64, 2>(dev)
           : split == 4 ? split_capacity<false, false, 64, 4>(dev)
                        : split_capacity<false, false, 64, 8>(dev);
  return split == 2   ? split_capacity<false, false, 128, 2>(dev)
         : split == 4 ? split_capacity<false, false, 128, 4>(dev)
                      : split_capacity<false, false, 128, 8>(dev);
}
// aligned: the leading dimensions of A, B and C are multiples of 64 elements
static GemmPlan gemm_plan(int M, int N, int K, bool aligned, int dev) {
  const int iters = (K + GEMM_BK - 1) / GEMM_BK;
  const auto div = [](long long a, long long b) { return (a + b - 1) / b; };
  const int sms = sm_count(dev);
  GemmPlan best = {0, 1};
  const auto estimate = [&](float t0, float c, float e, long long waves) {
    const float steps = c * iters;
    return t0 + (waves - 1) * (steps > e ? steps : e) + steps;
  };
  // an estimate within 2 % of the pair's goes to the pair (6136x5992x656 66.9, 128x256 83.4 us)
  float t = 0.98f * estimate(7.0f, 0.345f, 3.8f, div(div(M, G2_BM) * div(N, G2_BN), sms / 2));
  struct { int bn; float t0, c, e, unaligned, t_split[3]; } const kinds[] = {
      {256, 5.2f, 0.385f, 2.6f, 1.4f, {0.f, 0.f, 0.f}},
      {128, 4.3f, 0.245f, 1.75f, 1.55f, {1.05f, 2.1f, 3.2f}},   // splits of 2, 4, 8
      {64, 3.6f, 0.200f, 0.9f, 1.55f, {0.8f, 1.5f, 2.3f}},
  };
  for (const auto& k : kinds) {
    const long long tiles = div(M, GEMM_BM) * div(N, k.bn);
    const bool slow = !aligned && (k.bn == 256 || tiles > sms);
    const float u = estimate(k.t0, k.c * (slow ? k.unaligned : 1.f), k.e, div(tiles, sms));
    if (u < t) t = u, best = {k.bn, 1};
    if (k.bn == 256) continue;
    for (int i = 0; i < 3; ++i) {
      const int split = 2 << i;
      // one wave only
      if (tiles * split > sms || iters < 2 * split || tiles > split_clusters(k.bn, split, dev)) break;
      const float v = k.t0 + k.t_split[i] + k.c * div(iters, split);
      if (v < t) t = v, best = {k.bn, split};
    }
  }
  return best;
}

}  // namespace mb200

using namespace mb200;

extern "C" int mb200_gemm_bf16(const void* A, const void* B, void* C, const void* R, int M, int N,
                               int K, int lda, int ldb, int ldc, int ldr, int a_mn, int b_mn,
                               int accumulate, int* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  GemmParams p{};
  p.C = reinterpret_cast<__nv_bfloat16*>(C);
  p.R = reinterpret_cast<const __nv_bfloat16*>(R);
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc; p.ldr = ldr;
  p.accumulate = accumulate;
  p.status = status;
  p.b_ready = nullptr;
  p.b_ready_target = 0;
  p.flag_chunk_elems = 1;
  p.b_flag_elem0 = 0;
  p.ldb = ldb;
  p.n_blk_rot = 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap ta, tb;
  const int dev = current_device();
  const GemmPlan plan = g_gemm_impl == 2 ? gemm_plan(M, N, K, ((lda | ldb | ldc) & 63) == 0, dev)
                                         : GemmPlan{GEMM_BN, 1};
  const int bn = plan.bn;
  if (bn == 0) {
    const int r = make_gemm2_tmaps(&ta, &tb, A, B, M, N, K, lda, ldb, a_mn, b_mn);
    return r ? 1000 - r : launch_gemm2(ta, tb, p, a_mn, b_mn, st);
  }
  const int r = make_gemm_tmaps_bn(&ta, &tb, A, B, M, N, K, lda, ldb, a_mn, b_mn, bn);
  if (r) return 1000 - r;
  const int tiles = ((M + GEMM_BM - 1) / GEMM_BM) * ((N + bn - 1) / bn);
  if (plan.split > 1)
    return bn == 64 ? launch_split_n<64>(ta, tb, p, a_mn, b_mn, plan.split, tiles, st, dev)
                    : launch_split_n<128>(ta, tb, p, a_mn, b_mn, plan.split, tiles, st, dev);
  const int sms = sm_count(dev), grid = tiles < sms ? tiles : sms;
  if (bn == 64) return launch_gemm_bn<64>(ta, tb, p, a_mn, b_mn, grid, st, dev);
  if (bn == 128) return launch_gemm_bn<128>(ta, tb, p, a_mn, b_mn, grid, st, dev);
  return launch_gemm_bn<GEMM_BN>(ta, tb, p, a_mn, b_mn, grid, st, dev);
}

// ------------------------------------------------------- gated activation in the epilogue
// C[M, F] = silu(A Wg^T) * (A Wu^T) with W = [Wg; Wu] of 2F rows; gu ([M, 2F], or null) gets the
// two products.  The gate and up columns of an output column meet in one tile because its B rows
// come from both halves of W.
//
// What it saves is the pass over memory and a launch; what it costs is a longer epilogue, which
// the next tile's products hide if there is a next one and K is long enough.  Device time of the
// two kernels -> of one, us (T rows, both in turn, w of 0.02):
//   pair tiles, forward without gu: faster wherever the pair is the product's own tile: T 8192
//     F 14336 K 4096 1348 -> 1186, K 512 428 -> 321, T 2048 F 2048 K 3072 42 -> 40.  Where the
//     product alone would take 128x256 tiles the pair's loss comes first: T 1024 F 2048 K 2048
//     18.9 -> 19.5, T 2048 F 8192 K 256 (7 waves of pairs) 50.2 -> 50.4, T 4096 F 8192 K 256
//     (14 waves) 110 -> 100.
//   pair tiles, forward with gu: T 8192 F 14336 K 4096 1348 -> 1271, F 2048 K 2560 129 -> 123,
//     K 2048 108 -> 107; T 4096 F 2048 K 2560 70 -> 68, F 1024 37.0 -> 38.3, F 4096 K 2048
//     109 -> 113; T 2048 F 8192 K 3072 151 -> 154.
//   pair tiles, backward: T 8192 F 14336 K 4096 988 -> 888, F 2048 K 4096 121 -> 115, K 3072
//     97.2 -> 97.6, K 2560 93 -> 98; T 2048 F 4096 K 4096 61.4 -> 61.0, F 2048 (one wave)
//     34.2 -> 36.9.
//   small tiles: always slower on the device (256x512x256 6.2 -> 8.4 forward and 6.4 -> 8.4
//     backward; 8192x2048x256 backward 53 -> 97), but with one wave by no more than the second
//     launch costs the host, which is what calls as short as that wait for.  128x128 tiles lose
//     4.4 us in the backward.
constexpr int kGluKeepMinK = 2560, kGluKeepMinM = 4096, kGluKeepMinTiles = 256;
constexpr int kGluBwdMinK = 4096;
constexpr int kGluSmallMaxK = 1024;   // longer products outlast the host's second launch

enum GluKind { kGluFwd, kGluFwdKeep, kGluBwd };
// 1: CTA-pair tile, 0: small single-CTA tile, -1: two kernels.
static int glu_tile(GluKind kind, int M, int N, int F, int K, bool aligned, int dev,
                    GemmPlan* plan) {
  *plan = g_gemm_impl == 2 ? gemm_plan(M, N, K, aligned, dev) : GemmPlan{128, 1};
  if (plan->split > 1) return -1;
  const auto div = [](int a, int b) { return (long long)(a + b - 1) / b; };
  if (plan->bn == 64 || plan->bn == 128) {
    if (kind == kGluBwd && plan->bn != 64) return -1;
    return div(M, GEMM_BM) * div(F, 64) <= sm_count(dev) && K <= kGluSmallMaxK ? 0 : -1;
  }
  if (F % 128) return -1;
  const long long tiles = div(M, G2_BM) * div(N, G2_BN), pairs = sm_count(dev) / 2;
  bool fuse;
  if (kind == kGluFwd)
    fuse = plan->bn == 0 || tiles > 8 * pairs;
  else if (kind == kGluFwdKeep)
    fuse = plan->bn == 0 && K >= kGluKeepMinK && M >= kGluKeepMinM && tiles >= kGluKeepMinTiles;
  else
    fuse = plan->bn == 0 && K >= kGluBwdMinK && tiles > pairs;
  return fuse ? 1 : -1;
}

extern "C" int mb200_gemm_swiglu_fwd(const void* A, const void* W, void* H, void* gu, int M, int F,
                                     int K, int lda, int ldw, int ldh, int ld_gu, int keep_gu,
                                     int* status, void* stream) {
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if (F % 64 || (ldh & 7) || (ld_gu & 7) || (keep_gu && !gu) ||
      ((reinterpret_cast<uintptr_t>(H) | reinterpret_cast<uintptr_t>(gu)) & 15))
    return 1001;
  GemmPlan plan;
  const int dev = current_device();
  const int tile = glu_tile(keep_gu ? kGluFwdKeep : kGluFwd, M, 2 * F, F, K,
                            ((lda | ldw | ldh | ld_gu) & 63) == 0, dev, &plan);
  if (tile < 0) {
    if (!gu) return MB200_NOT_FUSED;
    const int rc = ld_gu == 2 * F && ldh == F
                       ? mb200_gemm_bf16(A, W, gu, nullptr, M, 2 * F, K, lda, ldw, ld_gu, 0, 0, 0, 0,
                                         status, stream)
                       : 1001;
    if (rc) return rc;
    const int rc2 = mb200_swiglu_fwd(gu, H, M, F, stream);
    return rc2 ? rc2 : MB200_TWO_KERNELS;
  }
  if (!keep_gu) gu = nullptr;
  GemmParams p{};
  p.C = reinterpret_cast<__nv_bfloat16*>(H);
  p.M = M; p.N = 2 * F; p.K = K;
  p.ldc = ldh;
  p.status = status;
  p.flag_chunk_elems = 1;
  p.gu_out = reinterpret_cast<__nv_bfloat16*>(gu);
  p.ld_gu = ld_gu;
  p.glu_f = F;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap ta, tb;
  if (tile == 1) {
    const int r = make_gemm2_tmaps(&ta, &tb, A, W, M, 2 * F, K, lda, ldw, 0, 0);
    if (r) return 1000 - r;
    return gu ? launch2<false, false, kEpiSwigluFwdKeep>(ta, tb, p, st)
              : launch2<false, false, kEpiSwigluFwd>(ta, tb, p, st);
  }
  const int r = make_gemm_tmaps_bn(&ta, &tb, A, W, M, 2 * F, K, lda, ldw, 0, 0, 64);
  if (r) return 1000 - r;
  const int tiles = ((M + GEMM_BM - 1) / GEMM_BM) * (F / 64);
  const int sms = sm_count(dev), grid = tiles < sms ? tiles : sms;
  return gu ? launch<false, false, 128, kEpiSwigluFwdKeep>(ta, tb, p, grid, st, dev)
            : launch<false, false, 128, kEpiSwigluFwd>(ta, tb, p, grid, st, dev);
}

// dgu[M, 2F] = gradient of silu(gate) * up at gu for dh = A W (W [K, F] row-major), without
// storing dh.
extern "C" int mb200_gemm_swiglu_bwd(const void* A, const void* W, const void* gu, void* dgu,
                                     void* dh, int M, int F, int K, int lda, int ldw, int ld_gu,
                                     int* status, void* stream) {
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if (F % 32 || (ld_gu & 7) || ((reinterpret_cast<uintptr_t>(gu) |
                                 reinterpret_cast<uintptr_t>(dgu)) & 15))
    return 1001;
  GemmPlan plan;
  const int dev = current_device();
  const int tile = glu_tile(kGluBwd, M, F, F, K, ((lda | ldw | ld_gu) & 63) == 0, dev, &plan);
  if (tile < 0) {
    if (!dh) return MB200_NOT_FUSED;
    const int rc = ld_gu == 2 * F ? mb200_gemm_bf16(A, W, dh, nullptr, M, F, K, lda, ldw, F, 0, 0, 1, 0,
                                                    status, stream)
                                  : 1001;
    if (rc) return rc;
    const int rc2 = mb200_swiglu_bwd(gu, dh, dgu, M, F, stream);
    return rc2 ? rc2 : MB200_TWO_KERNELS;
  }
  GemmParams p{};
  p.M = M; p.N = F; p.K = K;
  p.status = status;
  p.flag_chunk_elems = 1;
  p.gu_in = reinterpret_cast<const __nv_bfloat16*>(gu);
  p.gu_out = reinterpret_cast<__nv_bfloat16*>(dgu);
  p.ld_gu = ld_gu;
  p.glu_f = F;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap ta, tb;
  if (tile == 1) {
    const int r = make_gemm2_tmaps(&ta, &tb, A, W, M, F, K, lda, ldw, 0, 1);
    return r ? 1000 - r : launch2<false, true, kEpiSwigluBwd>(ta, tb, p, st);
  }
  const int r = make_gemm_tmaps_bn(&ta, &tb, A, W, M, F, K, lda, ldw, 0, 1, 64);
  if (r) return 1000 - r;
  const int tiles = ((M + GEMM_BM - 1) / GEMM_BM) * ((F + 63) / 64);
  const int sms = sm_count(dev), grid = tiles < sms ? tiles : sms;
  return launch<false, true, 64, kEpiSwigluBwd>(ta, tb, p, grid, st, dev);
}

// The tile (columns; 0: the CTA pair's) and K split that a product takes.
extern "C" int mb200_gemm_plan(int M, int N, int K, int lda, int ldb, int ldc, int* bn, int* split) {
  if (M <= 0 || N <= 0 || K <= 0) return 1001;
  const GemmPlan plan = gemm_plan(M, N, K, ((lda | ldb | ldc) & 63) == 0, current_device());
  *bn = plan.bn;
  *split = plan.split;
  return 0;
}

extern "C" int mb200_gemm_set_impl(int impl) {
  if (impl != 1 && impl != 2) return 1001;
  g_gemm_impl = impl;
  return 0;
}
extern "C" int mb200_gemm_get_impl() { return g_gemm_impl; }
