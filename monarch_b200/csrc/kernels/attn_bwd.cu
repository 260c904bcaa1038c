// Causal grouped-query flash attention, backward, for sm_100a (tcgen05 + TMEM + TMA).
//
// Three launches:
//   1. delta[b,h,s] = sum_d dO * O
//   2. dK, dV: one CTA per (kv block of 128 rows, kv head, batch); it keeps K and V in
//      shared memory, walks over every query block at or below the diagonal of every
//      query head of the group, and accumulates dV += P^T dO and dK += dS^T Q in TMEM:
//        S^T = K Q^T, dP^T = V dO^T      (tcgen05.mma, operands in shared memory)
//        P^T = exp2(S^T c - lse), dS^T = P^T (dP^T - delta)   (16 warps, a quarter of a
//                                         kv row per thread, written back as bf16)
//        dV += P^T dO, dK += dS^T Q      (A operand from TMEM, dO / Q MN-major from smem)
//   3. dQ: one CTA per (query block, query head, batch), walks over the kv blocks up to
//      the diagonal:  S = Q K^T, dP = dO V^T, dS = P (dP - delta), dQ += dS K.
// Splitting dQ off costs two extra MMAs per block pair but needs no atomics, no fp32 dQ
// buffer and no transposed copy of dS in shared memory: every operand is either a TMA tile
// or lives in TMEM.  Accumulators never leave TMEM until the epilogue.
//
// Both kernels step through their inner dimension 128 rows at a time.  A 128x128x128 MMA with
// both operands in shared memory reads 64 KB in the 512 cycles the tensor pipe needs for it
// (measured: 514 cycles); a 128x64x128 one still reads 48 KB in 256 cycles of math and takes
// 386, so 64-row steps made the scores a third more expensive.  With 128-row steps TMEM is full
// (dK, dV, S, dP: 4 x 128 columns at hd 128), and the overlap of math and exponentials comes
// from the order in which the MMA warp issues, not from a second set of accumulators:
//   dK/dV:  dV(t)  S(t+1)  dK(t)  dP(t+1) ...    P(t+1) is computed under dK(t) and dP(t+1),
//                                                dS(t+1) under dV(t+1) and S(t+2)
//   dQ:     S(t+1) dP(t+1) dQ(t) ...             (dP has two buffers here, S is free again as
//                                                soon as the warps hold it in registers)
// dK/dV is bound by the chain P(t) -> dV(t) -> S(t+1) -> P(t+1), as P lies over S: P is handed
// over in halves, so that dV starts under the second half of the exponentials; at hd 64 TMEM
// has room for P beside S and S(t+1) is issued as soon as S(t) is in registers.
// B1 S8192 32q/8kv hd128, dK/dV + dQ + delta: 2638 us with 64-row steps, 1564 with 128-row steps,
// 1518 with the halves: 7 MMAs per block pair at 1.35 PFLOP/s, which is what the chip sustains
// under its power cap (exponentials on the FMA pipe took 6 % off the cycles and as much off the
// clock).  B2 S4096 32q/8kv hd64: 1120, 703, 641 us.
//
// Warp roles (576 threads): 0 TMA producer, 1 MMA issuer, 2-17 compute/epilogue; warps w,
// w+4, w+8, w+12 share a TMEM lane quadrant and split the 128 columns of a tile in quarters
// (four warps per scheduler hide the TMEM load latency of each other).  The bf16 operand of
// quarter c is written at columns [32c, 32c+16) of the fp32 columns it replaces, so no warp
// overwrites columns another warp still has to read.
#include <cuda.h>
#include <cuda_runtime.h>
#include <math.h>

#include "launch.cuh"
#include "mb200.h"
#include "ptx.cuh"

namespace mb200 {

int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                      uint64_t ld, uint32_t box_inner, uint32_t box_outer);

constexpr int AB_T = 128;        // tile rows (queries and keys)
constexpr int AB_THREADS = 576;   // TMA warp, MMA warp, 16 compute warps
constexpr float kLog2e = 1.4426950408889634f;

struct AttBwdParams {
  const float* lse;    // [B, Hq, S]
  const float* delta;  // [B, Hq, S]
  __nv_bfloat16* dq;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  int ld_d;            // row stride of dq/dk/dv
  int B, S, Hq, Hkv;
  float scale, scale_log2;
  int* status;
};

// ------------------------------------------------------------------------- delta
// HD / 8 lanes per row (16-byte loads), four rows per lane with all their loads in flight, and
// a block's rows belong to one head, so that it writes 64 or 128 consecutive results.  Bound by
// HBM: B1 S8192 32 heads hd128 (134 MB) 53 -> 24 us against one warp per row with 4-byte loads
// and one scattered 4-byte store.
// VEC false: operands that are only 4-byte aligned.
constexpr int AB_DELTA_U = 4;
template <bool VEC>
__device__ __forceinline__ uint4 load_8bf16(const __nv_bfloat16* p) {
  if (VEC) return *reinterpret_cast<const uint4*>(p);
  const uint32_t* q = reinterpret_cast<const uint32_t*>(p);
  return make_uint4(q[0], q[1], q[2], q[3]);
}
template <int HD, bool VEC>
__global__ void __launch_bounds__(256)
    attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                      float* __restrict__ delta, int S, int Hq, int ld_o, int ld_do) {
  constexpr int LANES = HD / 8, ROWS = 256 / LANES;   // rows of a block: ROWS * AB_DELTA_U
  dep_launch();
  dep_wait();
  const int h = (int)(blockIdx.x % Hq);
  const int lane = (int)threadIdx.x % LANES;
  const long long row0 =
      (long long)(blockIdx.x / Hq) * (ROWS * AB_DELTA_U) + threadIdx.x / LANES;
  uint4 a[AB_DELTA_U], g[AB_DELTA_U];
#pragma unroll
  for (int u = 0; u < AB_DELTA_U; ++u) {
    const long long t = row0 + u * ROWS;
    a[u] = load_8bf16<VEC>(o + t * ld_o + h * HD + lane * 8);
    g[u] = load_8bf16<VEC>(dout + t * ld_do + h * HD + lane * 8);
  }
#pragma unroll
  for (int u = 0; u < AB_DELTA_U; ++u) {
    const uint32_t x[4] = {a[u].x, a[u].y, a[u].z, a[u].w};
    const uint32_t y[4] = {g[u].x, g[u].y, g[u].z, g[u].w};
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 p = unpack_bf16x2(x[i]), q = unpack_bf16x2(y[i]);
      acc += p.x * q.x + p.y * q.y;
    }
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) {
      const long long t = row0 + u * ROWS;
      const long long b = t / S;
      delta[(b * Hq + h) * S + (t - b * S)] = acc;
    }
  }
}

// ------------------------------------------------------------------------ dK, dV
// The operand that the last MMA of a step still reads has three stages (its buffer comes free
// only two MMAs before the next tile in it is needed), the other one two.
constexpr int AB_ST3 = 3;
constexpr int AB_ST2 = 2;

// Both kernels: two resident tiles, a ring of three and a ring of two tiles.  With hd 128 that
// is 224 KB, which leaves no room to align the base by hand: the dynamic shared memory itself
// is declared 1024-byte aligned (no static shared memory in these kernels).
template <int HD>
struct AbSmem {
  static constexpr int kTile = AB_T * HD * 2;
  static constexpr int kRowBytes = AB_T * 4;       // lse or delta of 128 query rows
  static constexpr int kData = (2 + AB_ST3 + AB_ST2) * kTile;
  static constexpr int kTotal = kData + AB_ST2 * 2 * kRowBytes + 256;
  static_assert(kTotal <= 232448, "more than 227 KB of shared memory");
};

struct DkvBars {
  uint64_t kv_full;
  uint64_t q_full[AB_ST3], q_empty[AB_ST3];
  uint64_t do_full[AB_ST2], do_empty[AB_ST2];
  uint64_t ld_full[AB_ST2], ld_empty[AB_ST2];
  // P of step t signals p_half/p_ready[t & 1]: at hd 64 S(t+1) is issued ahead of the waits for
  // P(t), so the warps may have handed over P(t+1) too before the issuing warp looks
  uint64_t s_full, s_free, dp_full, p_half[2], p_ready[2], ds_ready, acc_done;
  uint32_t tmem_base;
  volatile int abort_word;
};
static_assert(sizeof(DkvBars) <= 256, "barriers outgrew their space");

// A 128-row tile of `HD` columns as 64-column slices
template <int HD>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* m, uint64_t* bar,
                                          int col, int row) {
#pragma unroll
  for (int c = 0; c < HD / 64; ++c)
    tma_load_2d(dst + c * (AB_T * 128), m, bar, col + c * 64, row);
}
// D[128, 128] = A B^T over HD, both tiles K-major in shared memory
template <int HD>
__device__ __forceinline__ void mma_scores(uint32_t d_tmem, uint32_t sa, uint32_t sb) {
  constexpr uint32_t idesc = umma_idesc_bf16(AB_T, AB_T, 0, 0);
#pragma unroll
  for (int kk = 0; kk < HD / 16; ++kk) {
    const uint32_t off = (kk / 4) * (AB_T * 128) + (kk % 4) * 32;
    umma_f16(d_tmem, umma_smem_desc_sw128(sa + off, 16, 1024),
             umma_smem_desc_sw128(sb + off, 16, 1024), idesc, kk > 0 ? 1u : 0u);
  }
}
// D[128, HD] (+)= A B over 128 rows: A bf16 in TMEM (quarters of 16 columns), B MN-major
template <int HD, int QUARTER = 32>
__device__ __forceinline__ void mma_grad_half(uint32_t d_tmem, uint32_t a_tmem, uint32_t sb,
                                              int half, bool accumulate) {
  // one half of every quarter
  constexpr uint32_t idesc = umma_idesc_bf16(AB_T, HD, 0, 1);
#pragma unroll
  for (int c = 0; c < 4; ++c)
    umma_f16_ts(d_tmem, a_tmem + c * QUARTER + half * 8,
                umma_smem_desc_sw128(sb + (2 * c + half) * 2048, AB_T * 128, 1024), idesc,
                (accumulate || c > 0) ? 1u : 0u);
}
template <int HD>
__device__ __forceinline__ void mma_grad(uint32_t d_tmem, uint32_t a_tmem, uint32_t sb,
                                         bool accumulate) {
  mma_grad_half<HD>(d_tmem, a_tmem, sb, 0, accumulate);
  mma_grad_half<HD>(d_tmem, a_tmem, sb, 1, true);
}

__device__ __forceinline__ float2 exp2_pair(uint64_t x) {
  const float2 e = unpack_f32x2(x);
  return make_float2(ex2_approx(e.x), ex2_approx(e.y));
}

template <int HD>
__global__ void __launch_bounds__(AB_THREADS, 1)
    attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ,
                        const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV,
                        const __grid_constant__ CUtensorMap tmDO, const AttBwdParams p) {
  using SM = AbSmem<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sK = smem;
  uint8_t* sV = sK + SM::kTile;
  uint8_t* sQ = sV + SM::kTile;                 // [AB_ST3]
  uint8_t* sDO = sQ + AB_ST3 * SM::kTile;       // [AB_ST2]
  float* sLD = reinterpret_cast<float*>(smem + SM::kData);  // [AB_ST2] x {lse[128], delta[128]}
  DkvBars* bars = reinterpret_cast<DkvBars*>(smem + SM::kData + AB_ST2 * 2 * SM::kRowBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_blk = p.S / AB_T;
  // linear block id: all (head, batch) pairs of kv block 0 first, then block 1, ...: low j
  // = most work, so the heaviest CTAs of every head start first
  const int heads_x_batch = p.Hkv * p.B;
  const int j = (int)blockIdx.x / heads_x_batch;
  const int hb = (int)blockIdx.x % heads_x_batch;
  const int kv_head = hb % p.Hkv;
  const int b = hb / p.Hkv;
  const int group = p.Hq / p.Hkv;
  const int nq = n_blk - j;          // query blocks at or below the diagonal
  const int nsteps = group * nq;
  const int row_base = b * p.S;

  if (threadIdx.x == 0) {
    mbar_init(&bars->kv_full, 1);
    for (int s = 0; s < AB_ST3; ++s) {
      mbar_init(&bars->q_full[s], 1);
      mbar_init(&bars->q_empty[s], 1);
    }
    for (int s = 0; s < AB_ST2; ++s) {
      mbar_init(&bars->do_full[s], 1);
      mbar_init(&bars->do_empty[s], 1);
      mbar_init(&bars->ld_full[s], 1);
      mbar_init(&bars->ld_empty[s], 1);
    }
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->s_free, 16);
    mbar_init(&bars->dp_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->p_half[s], 16);
      mbar_init(&bars->p_ready[s], 16);
    }
    mbar_init(&bars->ds_ready, 16);
    mbar_init(&bars->acc_done, 1);
    bars->abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  volatile int* abort_word = &bars->abort_word;
  dep_wait();
  // TMEM columns: S^T at 0, dP^T/dS^T at 128, dV at 256, dK at 256 + HD; P^T over S^T at hd 128.
  // At hd 64 P^T(t) has 64 columns of its own at 384 + (t & 1) * 64: S(t) was issued behind
  // dV(t-2), so a warp that has S(t) may overwrite P(t-2).
  constexpr bool kOwnP = HD == 64;
  constexpr uint32_t kColDP = 128, kColDV = 256, kColDK = 256 + HD, kColP = kOwnP ? 384 : 0;
  constexpr int kQuarterP = kOwnP ? 16 : 32;   // columns from one quarter of P to the next

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      tma_prefetch_desc(&tmDO);
      mbar_expect_tx(&bars->kv_full, 2 * SM::kTile);
      load_tile<HD>(sK, &tmK, &bars->kv_full, kv_head * HD, row_base + j * AB_T);
      int h = kv_head * group, qb = j;   // head and query block of step t
      for (int t = 0; t < nsteps; ++t) {
        const int s3 = t % AB_ST3, s2 = t % AB_ST2;
        const uint32_t ph3 = ((uint32_t)(t / AB_ST3) & 1) ^ 1;
        const uint32_t ph2 = ((uint32_t)(t / AB_ST2) & 1) ^ 1;
        if (!mbar_wait(&bars->q_empty[s3], ph3, abort_word, p.status)) break;
        mbar_expect_tx(&bars->q_full[s3], SM::kTile);
        load_tile<HD>(sQ + s3 * SM::kTile, &tmQ, &bars->q_full[s3], h * HD, row_base + qb * AB_T);
        if (t == 0) load_tile<HD>(sV, &tmV, &bars->kv_full, kv_head * HD, row_base + j * AB_T);
        if (!mbar_wait(&bars->do_empty[s2], ph2, abort_word, p.status)) break;
        mbar_expect_tx(&bars->do_full[s2], SM::kTile);
        load_tile<HD>(sDO + s2 * SM::kTile, &tmDO, &bars->do_full[s2], h * HD,
                      row_base + qb * AB_T);
        if (!mbar_wait(&bars->ld_empty[s2], ph2, abort_word, p.status)) break;
        mbar_expect_tx(&bars->ld_full[s2], 2 * SM::kRowBytes);
        const size_t lrow = ((size_t)b * p.Hq + h) * p.S + (size_t)qb * AB_T;
        bulk_load_1d(sLD + s2 * 2 * AB_T, p.lse + lrow, SM::kRowBytes, &bars->ld_full[s2]);
        bulk_load_1d(sLD + s2 * 2 * AB_T + AB_T, p.delta + lrow, SM::kRowBytes,
                     &bars->ld_full[s2]);
        if (++qb == n_blk) {
          qb = j;
          ++h;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t sk = smem_u32(sK), sv = smem_u32(sV);
      const uint32_t sq = smem_u32(sQ), sdo = smem_u32(sDO);
      bool ok = mbar_wait(&bars->kv_full, 0, abort_word, p.status) &&
                mbar_wait(&bars->q_full[0], 0, abort_word, p.status);
      if (ok) {
        tc_fence_after();
        mma_scores<HD>(tmem_base, sk, sq);
        umma_commit(&bars->s_full);
        ok = mbar_wait(&bars->do_full[0], 0, abort_word, p.status);
      }
      if (ok) {
        tc_fence_after();
        mma_scores<HD>(tmem_base + kColDP, sv, sdo);
        umma_commit(&bars->dp_full);
      }
      const auto next_s = [&](int t) -> bool {   // S(t + 1)
        const int n3 = (t + 1) % AB_ST3;
        if (!mbar_wait(&bars->q_full[n3], (uint32_t)((t + 1) / AB_ST3) & 1, abort_word, p.status))
          return false;
        tc_fence_after();
        mma_scores<HD>(tmem_base, sk, sq + n3 * SM::kTile);
        umma_commit(&bars->s_full);
        return true;
      };
      for (int t = 0; ok && t < nsteps; ++t) {
        const int q3 = t % AB_ST3, d2 = t % AB_ST2, nd2 = (t + 1) % AB_ST2;
        const uint32_t par = (uint32_t)t & 1;
        const bool more = t + 1 < nsteps;
        if (kOwnP && more) {
          ok = mbar_wait(&bars->s_free, par, abort_word, p.status) && next_s(t);
          if (!ok) break;
        }
        const uint32_t p_par = (uint32_t)(t >> 1) & 1;
        ok = mbar_wait(&bars->p_half[t & 1], p_par, abort_word, p.status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tp = tmem_base + kColP + (kOwnP ? (t & 1) * 64 : 0);
        mma_grad_half<HD, kQuarterP>(tmem_base + kColDV, tp, sdo + d2 * SM::kTile, 0, t > 0);
        ok = mbar_wait(&bars->p_ready[t & 1], p_par, abort_word, p.status);
        if (!ok) break;
        tc_fence_after();
        mma_grad_half<HD, kQuarterP>(tmem_base + kColDV, tp, sdo + d2 * SM::kTile, 1, true);
        umma_commit(&bars->do_empty[d2]);
        if (!kOwnP && more) {   // overwrites P(t): ordered behind dV(t) on the tensor pipe
          ok = next_s(t);
          if (!ok) break;
        }
        ok = mbar_wait(&bars->ds_ready, par, abort_word, p.status);
        if (!ok) break;
        tc_fence_after();
        mma_grad<HD>(tmem_base + kColDK, tmem_base + kColDP, sq + q3 * SM::kTile, t > 0);
        umma_commit(&bars->q_empty[q3]);
        umma_commit(&bars->ld_empty[d2]);   // lse and delta of step t were read before dS(t)
        if (more) {
          ok = mbar_wait(&bars->do_full[nd2], (uint32_t)((t + 1) / AB_ST2) & 1, abort_word,
                         p.status);
          if (!ok) break;
          tc_fence_after();
          mma_scores<HD>(tmem_base + kColDP, sv, sdo + nd2 * SM::kTile);
          umma_commit(&bars->dp_full);
        }
      }
      if (ok) umma_commit(&bars->acc_done);
    }
  } else {
    const int quad = warp & 3;
    const int part = (warp - 2) >> 2;  // quarter of the 128 columns this warp converts
    const int r = quad * 32 + lane;    // kv row inside the block
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t t_st = tmem_base + lane_off + part * 32;
    const uint32_t t_dp = t_st + kColDP;
    const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2);
    const uint64_t nlog2e = pack_f32x2(-kLog2e, -kLog2e);
    const uint64_t neg1 = pack_f32x2(-1.f, -1.f);
    bool ok = true;
    int sub = 0;                       // query block of this step relative to the diagonal
    for (int t = 0; t < nsteps; ++t) {
      const int s2 = t % AB_ST2;
      const uint32_t par = (uint32_t)t & 1;
      ok = mbar_wait(&bars->ld_full[s2], (uint32_t)(t / AB_ST2) & 1, abort_word, p.status);
      if (!ok) break;
      const float* sl = sLD + s2 * 2 * AB_T + part * 32;
      ok = mbar_wait(&bars->s_full, par, abort_word, p.status);
      if (!ok) break;
      tc_fence_after();
      uint32_t sv[32];
      tmem_ld_32x32b_x32(t_st, sv);
      tmem_ld_wait();
      if (kOwnP) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->s_free);
      }
      uint32_t pk[16];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int i = half * 4; i < half * 4 + 4; ++i) {
          const float4 l4 = *reinterpret_cast<const float4*>(sl + 4 * i);
          const float2 e0 = exp2_pair(
              fma_f32x2(pack_f32x2(__uint_as_float(sv[4 * i]), __uint_as_float(sv[4 * i + 1])),
                        c2, mul_f32x2(pack_f32x2(l4.x, l4.y), nlog2e)));
          const float2 e1 = exp2_pair(
              fma_f32x2(pack_f32x2(__uint_as_float(sv[4 * i + 2]), __uint_as_float(sv[4 * i + 3])),
                        c2, mul_f32x2(pack_f32x2(l4.z, l4.w), nlog2e)));
          float pv[4] = {e0.x, e0.y, e1.x, e1.y};
          if (sub == 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (part * 32 + 4 * i + e < r) pv[e] = 0.f;  // query before the key position
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) sv[4 * i + e] = __float_as_uint(pv[e]);
          pk[2 * i] = pack_bf16x2(pv[0], pv[1]);
          pk[2 * i + 1] = pack_bf16x2(pv[2], pv[3]);
        }
        const uint32_t t_p = tmem_base + lane_off + kColP + part * kQuarterP +
                             (kOwnP ? (t & 1) * 64 : 0);
        tmem_st_32x32b_x8(t_p + half * 8,
                          *reinterpret_cast<const uint32_t(*)[8]>(&pk[half * 8]));
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(half == 0 ? &bars->p_half[t & 1] : &bars->p_ready[t & 1]);
      }
      ok = mbar_wait(&bars->dp_full, par, abort_word, p.status);
      if (!ok) break;
      tc_fence_after();
      uint32_t dv[32];
      tmem_ld_32x32b_x32(t_dp, dv);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 d4 = *reinterpret_cast<const float4*>(sl + AB_T + 4 * i);
        // dP - delta as fma(delta, -1, dP): one rounding, like the subtraction
        const uint64_t a0 = fma_f32x2(
            pack_f32x2(d4.x, d4.y), neg1,
            pack_f32x2(__uint_as_float(dv[4 * i]), __uint_as_float(dv[4 * i + 1])));
        const uint64_t a1 = fma_f32x2(
            pack_f32x2(d4.z, d4.w), neg1,
            pack_f32x2(__uint_as_float(dv[4 * i + 2]), __uint_as_float(dv[4 * i + 3])));
        const float2 x0 = unpack_f32x2(mul_f32x2(
            a0, pack_f32x2(__uint_as_float(sv[4 * i]), __uint_as_float(sv[4 * i + 1]))));
        const float2 x1 = unpack_f32x2(mul_f32x2(
            a1, pack_f32x2(__uint_as_float(sv[4 * i + 2]), __uint_as_float(sv[4 * i + 3]))));
        pk[2 * i] = pack_bf16x2(x0.x, x0.y);
        pk[2 * i + 1] = pack_bf16x2(x1.x, x1.y);
      }
      tmem_st_32x32b_x16(t_dp, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->ds_ready);
      if (++sub == nq) sub = 0;
    }
    if (ok) ok = mbar_wait(&bars->acc_done, 0, abort_word, p.status);
    if (ok) {
      tc_fence_after();
      const size_t grow = (size_t)(row_base + j * AB_T + r);
      constexpr int kCols = HD / 4;   // columns of dV and dK this warp writes (32 or 16)
      __nv_bfloat16* dvrow = p.dv + grow * p.ld_d + kv_head * HD + part * kCols;
      __nv_bfloat16* dkrow = p.dk + grow * p.ld_d + kv_head * HD + part * kCols;
      uint32_t a[kCols], bq[kCols];
      if constexpr (kCols == 32) {
        tmem_ld_32x32b_x32(tmem_base + kColDV + lane_off + part * kCols, a);
        tmem_ld_32x32b_x32(tmem_base + kColDK + lane_off + part * kCols, bq);
      } else {
        tmem_ld_32x32b_x16(tmem_base + kColDV + lane_off + part * kCols, a);
        tmem_ld_32x32b_x16(tmem_base + kColDK + lane_off + part * kCols, bq);
      }
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < kCols / 8; ++q) {
        uint4 x, y;
        x.x = pack_bf16x2(__uint_as_float(a[q * 8 + 0]), __uint_as_float(a[q * 8 + 1]));
        x.y = pack_bf16x2(__uint_as_float(a[q * 8 + 2]), __uint_as_float(a[q * 8 + 3]));
        x.z = pack_bf16x2(__uint_as_float(a[q * 8 + 4]), __uint_as_float(a[q * 8 + 5]));
        x.w = pack_bf16x2(__uint_as_float(a[q * 8 + 6]), __uint_as_float(a[q * 8 + 7]));
        y.x = pack_bf16x2(__uint_as_float(bq[q * 8 + 0]) * p.scale,
                          __uint_as_float(bq[q * 8 + 1]) * p.scale);
        y.y = pack_bf16x2(__uint_as_float(bq[q * 8 + 2]) * p.scale,
                          __uint_as_float(bq[q * 8 + 3]) * p.scale);
        y.z = pack_bf16x2(__uint_as_float(bq[q * 8 + 4]) * p.scale,
                          __uint_as_float(bq[q * 8 + 5]) * p.scale);
        y.w = pack_bf16x2(__uint_as_float(bq[q * 8 + 6]) * p.scale,
                          __uint_as_float(bq[q * 8 + 7]) * p.scale);
        *reinterpret_cast<uint4*>(dvrow + q * 8) = x;
        *reinterpret_cast<uint4*>(dkrow + q * 8) = y;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ----------------------------------------------------------------------------- dQ
struct DqBars {
  uint64_t qdo_full;
  uint64_t k_full[AB_ST3], k_empty[AB_ST3];
  uint64_t v_full[AB_ST2], v_empty[AB_ST2];
  uint64_t s_full, s_free, dp_full[2], ds_ready[2], acc_done;
  uint32_t tmem_base;
  volatile int abort_word;
};
static_assert(sizeof(DqBars) <= 256, "barriers outgrew their space");

template <int HD>
__global__ void __launch_bounds__(AB_THREADS, 1)
    attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ,
                       const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV,
                       const __grid_constant__ CUtensorMap tmDO, const AttBwdParams p) {
  using SM = AbSmem<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sDO = sQ + SM::kTile;
  uint8_t* sK = sDO + SM::kTile;             // [AB_ST3]
  uint8_t* sV = sK + AB_ST3 * SM::kTile;     // [AB_ST2]
  DqBars* bars = reinterpret_cast<DqBars*>(smem + SM::kData);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_blk = p.S / AB_T;
  const int i = n_blk - 1 - (int)blockIdx.x;  // query block; heavy blocks first
  const int h = blockIdx.y;
  const int b = blockIdx.z;
  const int kv_head = h / (p.Hq / p.Hkv);
  const int row_base = b * p.S;
  const int nsteps = i + 1;                   // kv blocks up to the diagonal

  if (threadIdx.x == 0) {
    mbar_init(&bars->qdo_full, 1);
    for (int s = 0; s < AB_ST3; ++s) {
      mbar_init(&bars->k_full[s], 1);
      mbar_init(&bars->k_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->v_full[s], 1);
      mbar_init(&bars->v_empty[s], 1);
      mbar_init(&bars->dp_full[s], 1);
      mbar_init(&bars->ds_ready[s], 16);
    }
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->s_free, 16);
    mbar_init(&bars->acc_done, 1);
    bars->abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  volatile int* abort_word = &bars->abort_word;
  dep_wait();
  // TMEM columns: S at 0, dP/dS of step t at 128 + (t&1)*128, dQ at 384
  constexpr uint32_t kColDP = 128, kColDQ = 384;

  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      tma_prefetch_desc(&tmDO);
      mbar_expect_tx(&bars->qdo_full, 2 * SM::kTile);
      load_tile<HD>(sQ, &tmQ, &bars->qdo_full, h * HD, row_base + i * AB_T);
      for (int t = 0; t < nsteps; ++t) {
        const int s3 = t % AB_ST3, s2 = t % AB_ST2;
        if (!mbar_wait(&bars->k_empty[s3], ((uint32_t)(t / AB_ST3) & 1) ^ 1, abort_word,
                       p.status))
          break;
        mbar_expect_tx(&bars->k_full[s3], SM::kTile);
        load_tile<HD>(sK + s3 * SM::kTile, &tmK, &bars->k_full[s3], kv_head * HD,
                      row_base + t * AB_T);
        if (t == 0) load_tile<HD>(sDO, &tmDO, &bars->qdo_full, h * HD, row_base + i * AB_T);
        if (!mbar_wait(&bars->v_empty[s2], ((uint32_t)(t / AB_ST2) & 1) ^ 1, abort_word,
                       p.status))
          break;
        mbar_expect_tx(&bars->v_full[s2], SM::kTile);
        load_tile<HD>(sV + s2 * SM::kTile, &tmV, &bars->v_full[s2], kv_head * HD,
                      row_base + t * AB_T);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t sq = smem_u32(sQ), sdo = smem_u32(sDO);
      const uint32_t sk = smem_u32(sK), sv = smem_u32(sV);
      bool ok = mbar_wait(&bars->qdo_full, 0, abort_word, p.status);
      // S and dP of step t; S(t-1) must have been read, dP's buffer was last read by dQ(t-2)
      auto issue_sdp = [&](int t) -> bool {
        const int s3 = t % AB_ST3, s2 = t % AB_ST2;
        if (!mbar_wait(&bars->k_full[s3], (uint32_t)(t / AB_ST3) & 1, abort_word, p.status) ||
            !mbar_wait(&bars->s_free, ((uint32_t)t & 1) ^ 1, abort_word, p.status))
          return false;
        tc_fence_after();
        mma_scores<HD>(tmem_base, sq, sk + s3 * SM::kTile);
        umma_commit(&bars->s_full);
        if (!mbar_wait(&bars->v_full[s2], (uint32_t)(t / AB_ST2) & 1, abort_word, p.status))
          return false;
        tc_fence_after();
        mma_scores<HD>(tmem_base + kColDP + (t & 1) * 128, sdo, sv + s2 * SM::kTile);
        umma_commit(&bars->dp_full[t & 1]);
        umma_commit(&bars->v_empty[s2]);
        return true;
      };
      if (ok) ok = issue_sdp(0);
      for (int t = 0; ok && t < nsteps; ++t) {
        if (t + 1 < nsteps) {
          ok = issue_sdp(t + 1);
          if (!ok) break;
        }
        ok = mbar_wait(&bars->ds_ready[t & 1], (uint32_t)(t >> 1) & 1, abort_word, p.status);
        if (!ok) break;
        tc_fence_after();
        const int s3 = t % AB_ST3;
        mma_grad<HD>(tmem_base + kColDQ, tmem_base + kColDP + (t & 1) * 128,
                     sk + s3 * SM::kTile, t > 0);
        umma_commit(&bars->k_empty[s3]);
      }
      if (ok) umma_commit(&bars->acc_done);
    }
  } else {
    const int quad = warp & 3;
    const int part = (warp - 2) >> 2;  // quarter of the 128 columns this warp converts
    const int r = quad * 32 + lane;    // query row inside the block
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t t_s = tmem_base + lane_off + part * 32;
    const size_t lrow = ((size_t)b * p.Hq + h) * p.S + (size_t)i * AB_T + r;
    const float neg_lse2 = -p.lse[lrow] * kLog2e;
    const float neg_dl = -p.delta[lrow];
    const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2);
    const uint64_t nl2 = pack_f32x2(neg_lse2, neg_lse2);
    const uint64_t nd2 = pack_f32x2(neg_dl, neg_dl);
    bool ok = true;
    for (int t = 0; t < nsteps; ++t) {
      ok = mbar_wait(&bars->s_full, (uint32_t)t & 1, abort_word, p.status);
      if (!ok) break;
      tc_fence_after();
      uint32_t sv[32];
      tmem_ld_32x32b_x32(t_s, sv);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->s_free);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float2 x = exp2_pair(
            fma_f32x2(pack_f32x2(__uint_as_float(sv[2 * e]), __uint_as_float(sv[2 * e + 1])), c2,
                      nl2));
        sv[2 * e] = __float_as_uint(x.x);
        sv[2 * e + 1] = __float_as_uint(x.y);
      }
      if (t == i) {   // the diagonal block
#pragma unroll
        for (int e = 0; e < 32; ++e)
          if (part * 32 + e > r) sv[e] = 0u;
      }
      const uint32_t t_dp = t_s + kColDP + (t & 1) * 128;
      ok = mbar_wait(&bars->dp_full[t & 1], (uint32_t)(t >> 1) & 1, abort_word, p.status);
      if (!ok) break;
      tc_fence_after();
      uint32_t dv[32];
      tmem_ld_32x32b_x32(t_dp, dv);
      tmem_ld_wait();
      uint32_t ds[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float2 x = unpack_f32x2(mul_f32x2(
            add_f32x2(pack_f32x2(__uint_as_float(dv[2 * e]), __uint_as_float(dv[2 * e + 1])),
                      nd2),
            pack_f32x2(__uint_as_float(sv[2 * e]), __uint_as_float(sv[2 * e + 1]))));
        ds[e] = pack_bf16x2(x.x, x.y);
      }
      tmem_st_32x32b_x16(t_dp, ds);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->ds_ready[t & 1]);
    }
    if (ok) ok = mbar_wait(&bars->acc_done, 0, abort_word, p.status);
    if (ok) {
      tc_fence_after();
      constexpr int kCols = HD / 4;
      const size_t grow = (size_t)(row_base + i * AB_T + r);
      __nv_bfloat16* dqrow = p.dq + grow * p.ld_d + h * HD + part * kCols;
      uint32_t a[kCols];
      if constexpr (kCols == 32)
        tmem_ld_32x32b_x32(tmem_base + kColDQ + lane_off + part * kCols, a);
      else
        tmem_ld_32x32b_x16(tmem_base + kColDQ + lane_off + part * kCols, a);
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < kCols / 8; ++q) {
        uint4 x;
        x.x = pack_bf16x2(__uint_as_float(a[q * 8 + 0]) * p.scale,
                          __uint_as_float(a[q * 8 + 1]) * p.scale);
        x.y = pack_bf16x2(__uint_as_float(a[q * 8 + 2]) * p.scale,
                          __uint_as_float(a[q * 8 + 3]) * p.scale);
        x.z = pack_bf16x2(__uint_as_float(a[q * 8 + 4]) * p.scale,
                          __uint_as_float(a[q * 8 + 5]) * p.scale);
        x.w = pack_bf16x2(__uint_as_float(a[q * 8 + 6]) * p.scale,
                          __uint_as_float(a[q * 8 + 7]) * p.scale);
        *reinterpret_cast<uint4*>(dqrow + q * 8) = x;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int HD>
static int launch_attn_bwd(const void* q, const void* k, const void* v, const void* dout,
                           int ld_qkv, int ld_do, const AttBwdParams& p, cudaStream_t st) {
  static PerDevice<int> dkv_smem_ok, dq_smem_ok;
  if (const cudaError_t e = allow_smem(attn_bwd_dkv_kernel<HD>, AbSmem<HD>::kTotal, dkv_smem_ok))
    return (int)e;
  if (const cudaError_t e = allow_smem(attn_bwd_dq_kernel<HD>, AbSmem<HD>::kTotal, dq_smem_ok))
    return (int)e;
  const uint64_t T = (uint64_t)p.B * p.S;
  CUtensorMap tq, tk, tv, tdo;   // boxes of 64 columns x 128 rows
  int r = make_tmap_bf16_2d(&tq, q, (uint64_t)p.Hq * HD, T, ld_qkv, 64, AB_T);
  if (!r) r = make_tmap_bf16_2d(&tk, k, (uint64_t)p.Hkv * HD, T, ld_qkv, 64, AB_T);
  if (!r) r = make_tmap_bf16_2d(&tv, v, (uint64_t)p.Hkv * HD, T, ld_qkv, 64, AB_T);
  if (!r) r = make_tmap_bf16_2d(&tdo, dout, (uint64_t)p.Hq * HD, T, ld_do, 64, AB_T);
  if (r) return 1000 - r;
  const int n_blk = p.S / AB_T;
  const cudaError_t e = launch_dep(attn_bwd_dkv_kernel<HD>, n_blk * p.Hkv * p.B, AB_THREADS,
                                   AbSmem<HD>::kTotal, st, tq, tk, tv, tdo, p);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_dep(attn_bwd_dq_kernel<HD>, dim3(n_blk, p.Hq, p.B), AB_THREADS,
                         AbSmem<HD>::kTotal, st, tq, tk, tv, tdo, p);
}

}  // namespace mb200

using namespace mb200;

// dout must have the layout of o ([B*S, Hq*hd], row stride ld_o).
extern "C" int mb200_attn_bwd(const void* q, const void* k, const void* v, const void* o,
                              const void* dout, const float* lse, float* delta, void* dq, void* dk,
                              void* dv, int B, int S, int Hq, int Hkv, int hd, int ld_qkv,
                              int ld_o, int ld_dqkv, float scale, int* status, void* stream) {
  if (B <= 0 || S <= 0) return 0;
  if ((S % AB_T) || (hd != 64 && hd != 128) || Hkv <= 0 || (Hq % Hkv) || (ld_dqkv & 7) ||
      (ld_o & 7) || (reinterpret_cast<uintptr_t>(dq) & 15) ||
      (reinterpret_cast<uintptr_t>(dk) & 15) || (reinterpret_cast<uintptr_t>(dv) & 15) ||
      (reinterpret_cast<uintptr_t>(lse) & 15) || (reinterpret_cast<uintptr_t>(delta) & 15))
    return 1001;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // S is a multiple of 128, so a block's 64 (hd 128) or 128 rows are whole and of one batch
  const auto* ob = reinterpret_cast<const __nv_bfloat16*>(o);
  const auto* db = reinterpret_cast<const __nv_bfloat16*>(dout);
  const bool vec = !((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dout)) & 15);
  const auto delta_kernel =
      hd == 128 ? (vec ? attn_delta_kernel<128, true> : attn_delta_kernel<128, false>)
                : (vec ? attn_delta_kernel<64, true> : attn_delta_kernel<64, false>);
  const long long rows = (long long)B * S;
  const cudaError_t e =
      launch_dep(delta_kernel, (unsigned)(rows / (hd == 128 ? 64 : 128) * Hq), 256, 0, st, ob, db,
                 delta, S, Hq, ld_o, ld_o);
  if (e != cudaSuccess) return (int)e;
  AttBwdParams p{};
  p.lse = lse;
  p.delta = delta;
  p.dq = reinterpret_cast<__nv_bfloat16*>(dq);
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk);
  p.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  p.ld_d = ld_dqkv;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv;
  p.scale = scale;
  p.scale_log2 = scale * kLog2e;
  p.status = status;
  if (hd == 128) return launch_attn_bwd<128>(q, k, v, dout, ld_qkv, ld_o, p, st);
  return launch_attn_bwd<64>(q, k, v, dout, ld_qkv, ld_o, p, st);
}
