// Memory-bound kernels of the transformer step: RMSNorm, RoPE, SwiGLU, cross-entropy,
// AdamW, embedding. All are 16-byte vectorised, one pass over HBM where possible.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "launch.cuh"
#include "mb200.h"
#include "ptx.cuh"

namespace mb200 {

int sm_count();

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z),
         d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  unpack8(*reinterpret_cast<const uint4*>(p), f);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]);
  u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]);
  u.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Sum across the block; result valid in every thread. `red` holds >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < nw ? red[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// ------------------------------------------------------------------ RMSNorm --
// A row is held in registers by WPR warps (16-byte loads, NV per lane, all in flight at once)
// and read from memory once; with one warp per row there is no block barrier at all.  Bound by
// HBM for many rows, by the chain of a row's loads, reduction and stores for few: then more warps
// with fewer loads each are faster (rmsnorm_fwd below has both sides).
constexpr int rms_fwd_threads(int wpr) { return wpr > 4 ? 32 * wpr : 128; }
template <int NV, int WPR>
__global__ void __launch_bounds__(rms_fwd_threads(WPR))
    rmsnorm_fwd_row_kernel(const __nv_bfloat16* __restrict__ x,
                           const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                           float* __restrict__ rstd, int rows, int d, float eps) {
  dep_wait();
  constexpr int kRows = rms_fwd_threads(WPR) / 32 / WPR;   // of a block
  __shared__ float red[kRows * WPR];
  const int warp = threadIdx.x >> 5;
  const int t = (int)threadIdx.x % (32 * WPR);   // place in the row's group of warps
  const int row = (int)blockIdx.x * kRows + warp / WPR;
  const bool on = row < rows;
  const __nv_bfloat16* xr = x + (size_t)row * d;
  uint4 v[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (i * 32 * WPR + t) * 8;
    v[i] = on && c < d ? *reinterpret_cast<const uint4*>(xr + c) : make_uint4(0, 0, 0, 0);
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    float f[8];
    unpack8(v[i], f);
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
  }
  ss = warp_sum(ss);
  if (WPR > 1) {
    if ((threadIdx.x & 31) == 0) red[warp] = ss;
    __syncthreads();
    ss = 0.f;
#pragma unroll
    for (int k = 0; k < WPR; ++k) ss += red[warp / WPR * WPR + k];
  }
  if (!on) return;
  const float rs = rsqrtf(ss / d + eps);
  if (t == 0 && rstd) rstd[row] = rs;
  __nv_bfloat16* yr = y + (size_t)row * d;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (i * 32 * WPR + t) * 8;
    if (c < d) {
      float f[8], g[8];
      unpack8(v[i], f);
      load8(w + c, g);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = f[e] * rs * g[e];
      store8(yr + c, f);
    }
  }
}

// Rows too long for registers: one block per row, two passes.
__global__ void __launch_bounds__(256)
    rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                       __nv_bfloat16* __restrict__ y, float* __restrict__ rstd, int d, float eps) {
  dep_wait();
  __shared__ float red[33];
  const size_t row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * d;
  float ss = 0.f;
  for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
    float f[8];
    load8(xr + c, f);
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  }
  ss = block_sum(ss, red);
  const float rs = rsqrtf(ss / d + eps);
  if (threadIdx.x == 0 && rstd) rstd[row] = rs;
  __nv_bfloat16* yr = y + row * d;
  for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
    float f[8], g[8];
    load8(xr + c, f);
    load8(w + c, g);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = f[i] * rs * g[i];
    store8(yr + c, f);
  }
}

constexpr int RMS_BWD_MAX_D = 8192;
constexpr int RMS_BWD_MAX_STAGES = 8;

// One block walks rows blockIdx.x, blockIdx.x + gridDim.x, ...; a thread owns NCH chunks of 8
// columns and keeps their weight-gradient sums in registers.  The rows of x, dy and dres come
// through a ring of `stages` rows in shared memory, filled by bulk copies several rows ahead:
// the reduction in the middle of every row then no longer stops the loads, which is what held
// the register-staged version at half the HBM rate (and at d > 4096, where only one block of it
// fitted, at a fifth).  The barrier of row i+1 also tells that every thread is done with row i,
// whose stage is refilled right after it.
// A copy that does not land within the wait's limit is reported through the status word, and the
// block's rows from there on and the weight gradient become NaN (the entry point without a status
// word has only that).  Every thread still walks through all rows: none is missing at a barrier.
// 8192x4096 with dres: 82.8 -> 48.2 us, 8192x5120: 239 -> 66 us, 8192x2048: 49.9 -> 34.8 us.
template <int NT, int NCH, bool RES>
__global__ void __launch_bounds__(NT, 1024 / (NT * NCH))
    rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                       const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                       const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                       float* __restrict__ dw_partial, int rows, int d, int stages,
                       int* __restrict__ status) {
  constexpr int NW = NT / 32;
  constexpr int NIN = RES ? 3 : 2;
  extern __shared__ __align__(128) uint8_t ring[];   // [stages][NIN][d] bf16
  __shared__ uint64_t full[RMS_BWD_MAX_STAGES];
  __shared__ float red[2][NW];
  __shared__ volatile int abort_word;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t row_bytes = (uint32_t)d * 2;
  const int n = rows > (int)blockIdx.x ? (rows - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const auto fill = [&](int it) {   // one thread
    const int st = it % stages;
    const size_t off = ((size_t)blockIdx.x + (size_t)it * gridDim.x) * d;
    uint8_t* dst = ring + (size_t)st * NIN * row_bytes;
    mbar_expect_tx(&full[st], NIN * row_bytes);
    bulk_load_1d(dst, x + off, row_bytes, &full[st]);
    bulk_load_1d(dst + row_bytes, dy + off, row_bytes, &full[st]);
    if (RES) bulk_load_1d(dst + 2 * row_bytes, dres + off, row_bytes, &full[st]);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) mbar_init(&full[s], 1);
    abort_word = 0;
    mbar_fence_init();
  }
  dep_wait();
  if (threadIdx.x == 0) {
    for (int it = 0; it < stages && it < n; ++it) fill(it);
  }
  float acc[NCH][8];
  uint4 wv[NCH];
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) {
    const int c = (threadIdx.x + ch * NT) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[ch][i] = 0.f;
    wv[ch] = c < d ? *reinterpret_cast<const uint4*>(w + c) : make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  float rs_next = n > 0 ? rstd[blockIdx.x] : 0.f;
  int lost = n;   // the first row that did not land
  for (int it = 0; it < n; ++it) {
    const int row = (int)blockIdx.x + it * (int)gridDim.x;
    const int st = it % stages;
    const float rs = rs_next;
    if (it + 1 < n) rs_next = rstd[row + gridDim.x];
    // (without the status word: polling it in the wait cost up to 8 %)
    if (lost == n && !mbar_wait(&full[st], (uint32_t)(it / stages) & 1, &abort_word, nullptr))
      lost = it;
    const __nv_bfloat16* sx = reinterpret_cast<const __nv_bfloat16*>(
        ring + (size_t)st * NIN * row_bytes);
    float xh[NCH][8], g[NCH][8];
    float dot = 0.f;
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const int c = (threadIdx.x + ch * NT) * 8;
      if (c < d) {
        float wf[8];
        load8(sx + c, xh[ch]);
        load8(sx + d + c, g[ch]);
        unpack8(wv[ch], wf);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          xh[ch][i] *= rs;
          acc[ch][i] += g[ch][i] * xh[ch][i];
          g[ch][i] *= wf[i];
          dot += g[ch][i] * xh[ch][i];
        }
      }
    }
    dot = warp_sum(lost <= it ? __int_as_float(0x7fffffff) : dot);
    if (lane == 0) red[it & 1][warp] = dot;
    __syncthreads();
    if (threadIdx.x == 0 && it > 0 && it - 1 + stages < n && lost > it) fill(it - 1 + stages);
    dot = 0.f;
#pragma unroll
    for (int k = 0; k < NW; ++k) dot += red[it & 1][k];
    dot /= d;
    __nv_bfloat16* dxr = dx + (size_t)row * d;
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const int c = (threadIdx.x + ch * NT) * 8;
      if (c < d) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = rs * (g[ch][i] - xh[ch][i] * dot);
        if (RES) {
          float r[8];
          load8(sx + 2 * d + c, r);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += r[i];
        }
        store8(dxr + c, o);
      }
    }
  }
  if (lost < n) {
    if (status) atomicCAS(status, kStatusOk, kStatusMbarTimeout);
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[ch][i] = __int_as_float(0x7fffffff);
    if (threadIdx.x == 0) {   // copies in flight still write to this block's memory
      const long long t0 = clock64();
      for (int k = lost; k < n && k < stages + (lost > 0 ? lost - 1 : 0); ++k)
        while (!mbar_try_wait(&full[k % stages], (uint32_t)(k / stages) & 1) &&
               clock64() - t0 < MB200_WAIT_CYCLES) {
        }
    }
  }
  float* out = dw_partial + (size_t)blockIdx.x * d;
#pragma unroll
  for (int ch = 0; ch < NCH; ++ch) {
    const int c = (threadIdx.x + ch * NT) * 8;
    if (c < d) {
      *reinterpret_cast<float4*>(out + c) = make_float4(acc[ch][0], acc[ch][1], acc[ch][2], acc[ch][3]);
      *reinterpret_cast<float4*>(out + c + 4) =
          make_float4(acc[ch][4], acc[ch][5], acc[ch][6], acc[ch][7]);
    }
  }
}

// Column sums of the [nblocks, d] partials.  A block covers 32 columns: its 32 thread rows
// stride over the partial rows (each warp reads 128 contiguous bytes per row) and are
// combined through shared memory.  Bound by the latency of a thread's chain of loads, hence
// many thread rows: 296 x 4096 in 3.4 us (8 thread rows: 6.0).
__global__ void __launch_bounds__(1024)
    rmsnorm_dw_reduce_kernel(const float* __restrict__ partial, int nblocks, int d,
                             __nv_bfloat16* __restrict__ dw, int accumulate) {
  dep_wait();
  __shared__ float sh[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < d) {
#pragma unroll 4
    for (int b = ty; b < nblocks; b += 32) s += partial[(size_t)b * d + c];
  }
  sh[ty][tx] = s;
  __syncthreads();
  s = warp_sum(sh[tx][ty]);   // warp ty sums column ty of the block
  const int oc = blockIdx.x * 32 + ty;
  if (tx == 0 && oc < d) {
    if (accumulate) s += __bfloat162float(dw[oc]);
    dw[oc] = __float2bfloat16(s);
  }
}

template <int NT, int NCH, bool RES>
static int launch_rmsnorm_bwd_t(int nb, const __nv_bfloat16* dy, const __nv_bfloat16* x,
                                const __nv_bfloat16* w, const float* rstd,
                                const __nv_bfloat16* dres, __nv_bfloat16* dx, float* dw_partial,
                                int rows, int d, int* status, cudaStream_t st) {
  // four blocks of 48 KB, two of 96 or one of 192 per SM
  constexpr int kRing = NT * NCH * 192;
  static PerDevice<int> smem_ok;
  if (const cudaError_t e = allow_smem(rmsnorm_bwd_kernel<NT, NCH, RES>, kRing, smem_ok))
    return (int)e;
  const int stage = (RES ? 3 : 2) * d * 2;
  int stages = kRing / stage;
  if (stages > RMS_BWD_MAX_STAGES) stages = RMS_BWD_MAX_STAGES;
  return (int)launch_dep(rmsnorm_bwd_kernel<NT, NCH, RES>, nb, NT, stages * stage, st, dy, x, w,
                         rstd, dres, dx, dw_partial, rows, d, stages, status);
}

// Launches the backward pair: nb row-striding blocks (fewer where one block fills an SM), then
// the column reduction.
static int launch_rmsnorm_bwd(int nb, const __nv_bfloat16* dy, const __nv_bfloat16* x,
                              const __nv_bfloat16* w, const float* rstd,
                              const __nv_bfloat16* dres, __nv_bfloat16* dx, float* dw_partial,
                              __nv_bfloat16* dw, int dw_accumulate, int rows, int d, int* status,
                              cudaStream_t st) {
  int rc;
  const int resident = sm_count() * (d > 4096 ? 1 : d > 2048 ? 2 : 4);
  if (nb > resident) nb = resident;
#define MB200_RMS_BWD(NT, NCH)                                                                  \
  (dres ? launch_rmsnorm_bwd_t<NT, NCH, true>(nb, dy, x, w, rstd, dres, dx, dw_partial, rows, d, \
                                              status, st)                                       \
        : launch_rmsnorm_bwd_t<NT, NCH, false>(nb, dy, x, w, rstd, dres, dx, dw_partial, rows, d, \
                                               status, st))
  if (d <= 2048)
    rc = MB200_RMS_BWD(256, 1);
  else if (d <= 4096)
    rc = MB200_RMS_BWD(256, 2);
  else
    rc = MB200_RMS_BWD(512, 2);
#undef MB200_RMS_BWD
  if (rc) return rc;
  return (int)launch_dep(rmsnorm_dw_reduce_kernel, (d + 31) / 32, 1024, 0, st, dw_partial, nb, d,
                         dw, dw_accumulate);
}

// --------------------------------------------------------------------- RoPE --
// A thread keeps the 8 cosines and sines of its column pairs and applies them to every step-th
// head of its row, ROPE_U heads at a time so that their loads are in flight together.  (One
// thread per head and 8 pairs spent its time in 64-bit divisions and in reading the tables again
// for every head: 8192 rows of 40 heads of 128 32.1 us, so 27.1.)
constexpr int ROPE_U = 5;
__global__ void __launch_bounds__(256)
    rope_row_kernel(__nv_bfloat16* __restrict__ qkv, const float* __restrict__ cos_t,
                    const float* __restrict__ sin_t, int rows, int seq_len, int n_rot_heads,
                    int log2_hd, int log2_step, int row_stride, int inverse) {
  dep_wait();
  const int hd = 1 << log2_hd, half = hd >> 1, per_head = hd >> 4, step = 1 << log2_step;
  const int log2_row = log2_hd - 4 + log2_step;   // step * per_head threads per row
  const int row = ((int)blockIdx.x << (8 - log2_row)) + ((int)threadIdx.x >> log2_row);
  if (row >= rows) return;
  const int t = (int)threadIdx.x & ((1 << log2_row) - 1);
  const int j = t & (per_head - 1);
  const size_t tab = (size_t)(row % seq_len) * half + j * 8;
  float c[8], s[8];
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    const float4 a = *reinterpret_cast<const float4*>(cos_t + tab + i);
    const float4 b = *reinterpret_cast<const float4*>(sin_t + tab + i);
    c[i] = a.x; c[i + 1] = a.y; c[i + 2] = a.z; c[i + 3] = a.w;
    s[i] = b.x; s[i + 1] = b.y; s[i + 2] = b.z; s[i + 3] = b.w;
  }
  if (inverse) {
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = -s[i];
  }
  __nv_bfloat16* base = qkv + (size_t)row * row_stride + j * 8;
  for (int h0 = t >> (log2_hd - 4); h0 < n_rot_heads; h0 += step * ROPE_U) {
    uint4 lo[ROPE_U], hi[ROPE_U];
#pragma unroll
    for (int u = 0; u < ROPE_U; ++u) {
      const int h = h0 + u * step;
      if (h < n_rot_heads) {
        lo[u] = *reinterpret_cast<const uint4*>(base + (size_t)h * hd);
        hi[u] = *reinterpret_cast<const uint4*>(base + (size_t)h * hd + half);
      }
    }
#pragma unroll
    for (int u = 0; u < ROPE_U; ++u) {
      const int h = h0 + u * step;
      if (h < n_rot_heads) {
        float a[8], b[8], o1[8], o2[8];
        unpack8(lo[u], a);
        unpack8(hi[u], b);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          o1[i] = a[i] * c[i] - b[i] * s[i];
          o2[i] = b[i] * c[i] + a[i] * s[i];
        }
        store8(base + (size_t)h * hd, o1);
        store8(base + (size_t)h * hd + half, o2);
      }
    }
  }
}

// log2 of `step`, the heads that a row's threads work on side by side (at most 256 threads).
// Many rows: up to 8 heads per thread, so that the tables are read by few, and no more than 8 side
// by side.  Few rows: 64 Ki threads if there are that many pairs of columns, since a thread's
// batches follow one another.  us by step, heads of 128:
//   8192 rows,  1 head 1: 2.2, 8: 8.7;   8 heads 1: 4.6, 2: 4.9, 8: 9.6;   20 heads 2: 15.0,
//               4: 14.7, 8: 18.1;   40 heads 4: 27.7, 8: 27.1, 16: 34.2;   80 heads 4: 54.0,
//               8: 52.2, 16: 54.3
//   2048 rows, 20 heads 2: 3.5, 4: 3.3, 8: 4.1;   512 rows, 20 heads 4: 2.4, 8: 2.1, 32: 3.2
//     64 rows, 40 heads 8: 2.3, 32: 1.9;   heads of 64: 80 heads 8: 3.9, 64: 1.8
static inline int rope_log2_step(int rows, int heads, int log2_hd) {
  const int most = 12 - log2_hd;
  int s = 0;
  while (s < most && s < 3 && (8 << s) < heads) ++s;
  while (s < most && (1 << s) < heads && ((long long)rows << (s + log2_hd - 3)) <= 64 * 1024) ++s;
  return s;
}

// Head sizes that are no power of two up to 512.
__global__ void rope_kernel(__nv_bfloat16* __restrict__ qkv, const float* __restrict__ cos_t,
                            const float* __restrict__ sin_t, long long total, int seq_len,
                            int n_rot_heads, int hd, int row_stride, int inverse) {
  dep_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int half = hd >> 1;
  const int per_head = half >> 3;  // threads per head (8 pairs each)
  const int j = (int)(idx % per_head);
  const long long hh = idx / per_head;
  const int h = (int)(hh % n_rot_heads);
  const long long row = hh / n_rot_heads;
  const int pos = (int)(row % seq_len);
  __nv_bfloat16* base = qkv + row * row_stride + (size_t)h * hd + j * 8;
  float a[8], b[8], c[8], s[8];
  load8(base, a);
  load8(base + half, b);
  const float* cp = cos_t + (size_t)pos * half + j * 8;
  const float* sp = sin_t + (size_t)pos * half + j * 8;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    c[i] = cp[i];
    s[i] = inverse ? -sp[i] : sp[i];
  }
  float o1[8], o2[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    o1[i] = a[i] * c[i] - b[i] * s[i];
    o2[i] = b[i] * c[i] + a[i] * s[i];
  }
  store8(base, o1);
  store8(base + half, o2);
}

// ------------------------------------------------------------------- SwiGLU --
// Rows on grid.x, 8-column chunks on grid.y: no division per thread (a 64-bit one by F/8 cost
// the forward a fifth of its time: 8192x14336 133.6 -> 113 us, backward 181 -> 178 us).  A block
// takes several rows of fewer than 256 chunks.
template <bool SHORT>   // several rows per block (their index costs the long ones 1 %)
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu,
                                  __nv_bfloat16* __restrict__ h, int rows, int F) {
  dep_wait();
  const size_t row = SHORT ? (size_t)blockIdx.x * blockDim.y + threadIdx.y : blockIdx.x;
  const int c = (int)(blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= F || (SHORT && row >= (size_t)rows)) return;
  float g[8], u[8], o[8];
  load8(gu + row * 2 * F + c, g);
  load8(gu + row * 2 * F + F + c, u);
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = g[i] / (1.f + __expf(-g[i])) * u[i];
  store8(h + row * F + c, o);
}

template <bool SHORT>
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu,
                                  const __nv_bfloat16* __restrict__ dh,
                                  __nv_bfloat16* __restrict__ dgu, int rows, int F) {
  dep_wait();
  const size_t row = SHORT ? (size_t)blockIdx.x * blockDim.y + threadIdx.y : blockIdx.x;
  const int c = (int)(blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= F || (SHORT && row >= (size_t)rows)) return;
  float g[8], u[8], d[8], dg[8], du[8];
  load8(gu + row * 2 * F + c, g);
  load8(gu + row * 2 * F + F + c, u);
  load8(dh + row * F + c, d);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float sg = 1.f / (1.f + __expf(-g[i]));
    const float silu = g[i] * sg;
    du[i] = d[i] * silu;
    dg[i] = d[i] * u[i] * sg * (1.f + g[i] * (1.f - sg));
  }
  store8(dgu + row * 2 * F + c, dg);
  store8(dgu + row * 2 * F + F + c, du);
}
// Block for rows of n 8-column chunks (x: chunks, y: rows), and the grid that covers them.  One
// row per block, whatever its length, took 8192 rows of 64 columns 5.74 us, as long as rows of 512.
static inline dim3 row_block(int n) { return n >= 256 ? dim3(256) : dim3(n, 256 / n); }
static inline dim3 row_grid(int rows, int n, dim3 b) {
  return dim3((rows + b.y - 1) / b.y, (n + b.x - 1) / b.x);
}

// ------------------------------------------------------------ cross-entropy --
// One block per row; the row is read twice (maximum and sum, then the gradient) and written
// once.  Bound by HBM and, close behind, by instructions (two exponentials per logit), hence the
// two-wide arithmetic.  Long rows get blocks of 1024 threads: with two of them per SM most of
// the rows being worked on (296 x 256 KB at a vocabulary of 128256) are still in L2 at their
// second read, with four blocks of 512 they were not: 4096x128256 492 -> 390 us.  Short rows get
// small blocks, whose reductions and start-up are shorter.  us by threads of a block, 4096 rows:
//   V  4096  128: 13.8  256: 17.6  512: 22.7      V 16384  128: 52.9  256: 46.9  512: 49.5
//   V  6144  128: 21.5  256: 24.9  512: 30.9      V 32000  256: 101.7  512: 91.4  1024: 110.8
//   V  8192  128: 26.7  256: 25.4  512: 35.9      V 50264  256: 188.9  512: 147.3  1024: 160.9
//                                                 V 65536  256: 243.3  512: 206.0  1024: 182.8
// Below 512 rows the chip is not full and a row's own time counts: 64 rows, V 4096 128: 2.9
// 512: 2.7; V 6144 128: 3.6 512: 3.2; V 16384 256: 4.2 512: 3.8; V 65536 512: 8.0 1024: 7.8.
template <int CE_THREADS>
__global__ void __launch_bounds__(CE_THREADS, 2048 / CE_THREADS)
    cross_entropy_kernel(__nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ targets,
                         float* __restrict__ loss_rows, int V, int ld, float grad_scale) {
  dep_wait();
  __shared__ float red_m[CE_THREADS / 32];
  __shared__ float red_s[CE_THREADS / 32];
  __shared__ float bc[2];
  const size_t row = blockIdx.x;
  __nv_bfloat16* lr = logits + row * ld;
  const int tgt = (int)targets[row];
  float m = -INFINITY, s = 0.f;
  const int vec_end = V & ~7;
  const uint64_t log2e = pack_f32x2(kLog2e, kLog2e);
  for (int c = threadIdx.x * 8; c < vec_end; c += CE_THREADS * 8) {
    float f[8];
    load8(lr + c, f);
    float nm = m;
#pragma unroll
    for (int i = 0; i < 8; i += 2) asm("max.f32 %0, %0, %1, %2;" : "+f"(nm) : "f"(f[i]), "f"(f[i + 1]));
    const uint64_t neg = pack_f32x2(-nm, -nm);
    uint64_t acc = 0;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const float2 e = unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(f[i], f[i + 1]), neg), log2e));
      acc = add_f32x2(acc, pack_f32x2(ex2_approx(e.x), ex2_approx(e.y)));
    }
    const float2 a = unpack_f32x2(acc);
    s = s * __expf(m - nm) + (a.x + a.y);
    m = nm;
  }
  for (int c = vec_end + threadIdx.x; c < V; c += CE_THREADS) {
    const float f = __bfloat162float(lr[c]);
    const float nm = fmaxf(m, f);
    s = s * __expf(m - nm) + __expf(f - nm);
    m = nm;
  }
  // combine (m, s) across the block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float wm = warp_max(m);
  float ws = warp_sum(m == -INFINITY ? 0.f : s * __expf(m - wm));
  if (lane == 0) {
    red_m[warp] = wm;
    red_s[warp] = ws;
  }
  __syncthreads();
  if (warp == 0) {
    float mm = lane < CE_THREADS / 32 ? red_m[lane] : -INFINITY;
    float ss = lane < CE_THREADS / 32 ? red_s[lane] : 0.f;
    const float gm = warp_max(mm);
    ss = warp_sum(mm == -INFINITY ? 0.f : ss * __expf(mm - gm));
    if (lane == 0) {
      bc[0] = gm;
      bc[1] = ss;
    }
  }
  __syncthreads();
  const float gm = bc[0];
  const float inv = 1.f / bc[1];
  if (threadIdx.x == 0) {
    const float lt = __bfloat162float(lr[tgt]);
    loss_rows[row] = logf(bc[1]) + gm - lt;
  }
  __syncthreads();  // the target logit is read before anyone overwrites it
  const uint64_t neg = pack_f32x2(-gm, -gm), inv2 = pack_f32x2(inv, inv);
  const uint64_t gs2 = pack_f32x2(grad_scale, grad_scale);
  for (int c = threadIdx.x * 8; c < vec_end; c += CE_THREADS * 8) {
    float f[8];
    load8(lr + c, f);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      float2 e = unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(f[i], f[i + 1]), neg), log2e));
      e.x = ex2_approx(e.x);
      e.y = ex2_approx(e.y);
      e = unpack_f32x2(mul_f32x2(pack_f32x2(e.x, e.y), inv2));
      f[i] = e.x;
      f[i + 1] = e.y;
    }
    if ((tgt & ~7) == c) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c + i == tgt) f[i] -= 1.f;
    }
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const float2 e = unpack_f32x2(mul_f32x2(pack_f32x2(f[i], f[i + 1]), gs2));
      f[i] = e.x;
      f[i + 1] = e.y;
    }
    store8(lr + c, f);
  }
  for (int c = vec_end + threadIdx.x; c < V; c += CE_THREADS) {
    float p = __expf(__bfloat162float(lr[c]) - gm) * inv;
    if (c == tgt) p -= 1.f;
    lr[c] = __float2bfloat16(p * grad_scale);
  }
}

// -------------------------------------------------------------------- AdamW --
__global__ void adamw_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                             const void* __restrict__ g, __nv_bfloat16* __restrict__ pb, int64_t n,
                             int g_bf16, float lr, float beta1, float beta2, float eps, float wd,
                             float inv_bc1, float inv_sqrt_bc2, float grad_scale) {
  dep_wait();
  const int64_t i4 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i4 >= n) return;
  float pv[4], mv[4], vv[4], gv[4];
  const bool full = i4 + 4 <= n;
  if (full) {
    float4 a = *reinterpret_cast<const float4*>(p + i4);
    float4 b = *reinterpret_cast<const float4*>(m + i4);
    float4 c = *reinterpret_cast<const float4*>(v + i4);
    pv[0] = a.x; pv[1] = a.y; pv[2] = a.z; pv[3] = a.w;
    mv[0] = b.x; mv[1] = b.y; mv[2] = b.z; mv[3] = b.w;
    vv[0] = c.x; vv[1] = c.y; vv[2] = c.z; vv[3] = c.w;
    if (g_bf16) {
      uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(g) + i4);
      float2 x = unpack_bf16x2(u.x), y = unpack_bf16x2(u.y);
      gv[0] = x.x; gv[1] = x.y; gv[2] = y.x; gv[3] = y.y;
    } else {
      float4 d = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(g) + i4);
      gv[0] = d.x; gv[1] = d.y; gv[2] = d.z; gv[3] = d.w;
    }
  } else {
    for (int k = 0; k < 4; ++k) {
      const bool ok = i4 + k < n;
      pv[k] = ok ? p[i4 + k] : 0.f;
      mv[k] = ok ? m[i4 + k] : 0.f;
      vv[k] = ok ? v[i4 + k] : 0.f;
      gv[k] = !ok ? 0.f
                  : (g_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(g)[i4 + k])
                            : reinterpret_cast<const float*>(g)[i4 + k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float gg = gv[k] * grad_scale;
    pv[k] *= (1.f - lr * wd);
    mv[k] = beta1 * mv[k] + (1.f - beta1) * gg;
    vv[k] = beta2 * vv[k] + (1.f - beta2) * gg * gg;
    const float denom = sqrtf(vv[k]) * inv_sqrt_bc2 + eps;
    pv[k] -= lr * inv_bc1 * mv[k] / denom;
  }
  if (full) {
    *reinterpret_cast<float4*>(p + i4) = make_float4(pv[0], pv[1], pv[2], pv[3]);
    *reinterpret_cast<float4*>(m + i4) = make_float4(mv[0], mv[1], mv[2], mv[3]);
    *reinterpret_cast<float4*>(v + i4) = make_float4(vv[0], vv[1], vv[2], vv[3]);
    if (pb) {
      uint2 o;
      o.x = pack_bf16x2(pv[0], pv[1]);
      o.y = pack_bf16x2(pv[2], pv[3]);
      *reinterpret_cast<uint2*>(pb + i4) = o;
    }
  } else {
    for (int k = 0; k < 4 && i4 + k < n; ++k) {
      p[i4 + k] = pv[k];
      m[i4 + k] = mv[k];
      v[i4 + k] = vv[k];
      if (pb) pb[i4 + k] = __float2bfloat16(pv[k]);
    }
  }
}

// ---------------------------------------------------------------- embedding --
__global__ void embedding_fwd_kernel(const __nv_bfloat16* __restrict__ table,
                                     const int64_t* __restrict__ ids,
                                     __nv_bfloat16* __restrict__ out, long long total, int d) {
  dep_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int per_row = d >> 3;
  const long long row = idx / per_row;
  const int c = (int)(idx % per_row) * 8;
  const int64_t id = ids[row];
  *reinterpret_cast<uint4*>(out + row * d + c) =
      *reinterpret_cast<const uint4*>(table + id * d + c);
}
// 16 bytes per reduction (four bf16 pairs, each element rounded as a single addition would
// be): 8192x2048 34.8 -> 10.4 us against one pair per reduction.
template <bool SHORT>
__global__ void embedding_bwd_vec_kernel(const __nv_bfloat16* __restrict__ dout,
                                         const int64_t* __restrict__ ids,
                                         __nv_bfloat16* __restrict__ dtable, int rows, int d) {
  dep_wait();
  const size_t row = SHORT ? (size_t)blockIdx.x * blockDim.y + threadIdx.y : blockIdx.x;
  const int c = (int)(blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= d || (SHORT && row >= (size_t)rows)) return;
  const int64_t id = ids[row];
  const uint4 g = *reinterpret_cast<const uint4*>(dout + row * d + c);
  asm volatile("red.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(dtable + id * d + c),
               "r"(g.x), "r"(g.y), "r"(g.z), "r"(g.w)
               : "memory");
}
__global__ void embedding_bwd_kernel(const __nv_bfloat16* __restrict__ dout,
                                     const int64_t* __restrict__ ids,
                                     __nv_bfloat16* __restrict__ dtable, long long total, int d) {
  dep_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int per_row = d >> 1;
  const long long row = idx / per_row;
  const int c = (int)(idx % per_row) * 2;
  const int64_t id = ids[row];
  const __nv_bfloat162 g = *reinterpret_cast<const __nv_bfloat162*>(dout + row * d + c);
  atomicAdd(reinterpret_cast<__nv_bfloat162*>(dtable + id * d + c), g);
}

__global__ void sumsq_kernel(const void* __restrict__ x, int64_t n, int is_bf16,
                             float* __restrict__ out) {
  dep_wait();
  __shared__ float red[33];
  float s = 0.f;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float f = is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[i])
                            : reinterpret_cast<const float*>(x)[i];
    s += f * f;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static inline unsigned blocks_for(long long total, int threads) {
  return (unsigned)((total + threads - 1) / threads);
}

}  // namespace mb200

using namespace mb200;
#define ST(s) reinterpret_cast<cudaStream_t>(s)
#define BF(p) reinterpret_cast<__nv_bfloat16*>(p)
#define CBF(p) reinterpret_cast<const __nv_bfloat16*>(p)

extern "C" int mb200_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int rows,
                                 int d, float eps, void* stream) {
  if (rows <= 0) return 0;
  if (d % 8) return 1001;
#define MB200_RMS_FWD(NV, WPR)                                                           \
  return (int)launch_dep(rmsnorm_fwd_row_kernel<NV, WPR>,                                 \
                         blocks_for(rows, rms_fwd_threads(WPR) / 32 / WPR),               \
                         rms_fwd_threads(WPR), 0, ST(stream), CBF(x), CBF(w), BF(y), rstd, rows, \
                         d, eps)
  // us on (loads per lane, warps per row); the limits lie between the measured row counts
  //   d  512: 1000 rows (2,1) 1.85 (2,2) 1.70;   4000 rows 2.29 and 2.69
  //   d 1024: 1000 rows (4,1) 2.48 (2,4) 1.96;   4000 rows 2.96 and 3.84
  //   d 1032: 1000 rows (4,2) 2.48 (2,4) 2.29;   4000 rows (8,1) 5.03 (4,2) 4.17 (2,4) 4.18;
  //           8192 rows 7.8, 8.0, 8.9
  //   d 2048:   16 rows (8,1) 3.14 (2,4) 1.71;   8192 rows 13.25, (4,2) 12.30, 12.25
  //   d 4096:   16 rows (8,2) 3.17 (4,4) 2.29 (2,8) 1.76;  1000 rows 4.02, 3.21, 3.56;
  //           8192 rows 24.7, 23.0 (5.8 TB/s), 23.9
  //   d 5120:   16 rows (8,4) 2.52 (4,8) 2.13;   8192 rows 29.9 and 30.9
  //   d 8192:   16 rows (8,4) 3.15 (4,8) 2.39;   8192 rows 44.1 and 42.5
  const bool few = rows <= 2048;
  if (d <= 512 && few) MB200_RMS_FWD(2, 2);
  if (d <= 512) MB200_RMS_FWD(2, 1);
  if (d <= 1024 && !few) MB200_RMS_FWD(4, 1);
  if (d <= 2048 && !few) MB200_RMS_FWD(4, 2);
  if (d <= 2048) MB200_RMS_FWD(2, 4);
  if (d <= 4096 && rows <= 768) MB200_RMS_FWD(2, 8);
  if (d <= 4096) MB200_RMS_FWD(4, 4);
  if (d <= 6144 && !few) MB200_RMS_FWD(8, 4);
  if (d <= 8192) MB200_RMS_FWD(4, 8);
#undef MB200_RMS_FWD
  return (int)launch_dep(rmsnorm_fwd_kernel, rows, 256, 0, ST(stream), CBF(x), CBF(w), BF(y), rstd,
                         d, eps);
}

extern "C" int mb200_rmsnorm_bwd_blocks(int rows) {
  const int cap = sm_count() * 4;   // one resident wave: four blocks per SM at d <= 2048
  return rows < cap ? rows : cap;
}

extern "C" int mb200_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd,
                                 const void* dres, void* dx, float* dw_partial, void* dw,
                                 int dw_accumulate, int rows, int d, int* status,
                                 void* stream) {
  if (rows <= 0) return 0;
  if (d % 8 || d > RMS_BWD_MAX_D) return 1001;
  const int nb = mb200_rmsnorm_bwd_blocks(rows);
  return launch_rmsnorm_bwd(nb, CBF(dy), CBF(x), CBF(w), rstd, CBF(dres), BF(dx), dw_partial,
                            BF(dw), dw_accumulate, rows, d, status, ST(stream));
}

extern "C" int mb200_rope_inplace(void* qkv, const float* cos_t, const float* sin_t, int rows,
                                  int seq_len, int n_rot_heads, int hd, int row_stride,
                                  int inverse, void* stream) {
  if (rows <= 0) return 0;
  if (hd % 16 || row_stride % 8 || hd <= 0 || n_rot_heads <= 0) return 1001;
  if (hd <= 512 && (hd & (hd - 1)) == 0 && aligned16(cos_t) && aligned16(sin_t)) {
    const int log2_hd = __builtin_ctz(hd);
    const int log2_step = rope_log2_step(rows, n_rot_heads, log2_hd);
    return (int)launch_dep(rope_row_kernel, blocks_for(rows, 256 >> (log2_hd - 4 + log2_step)), 256,
                           0, ST(stream), BF(qkv), cos_t, sin_t, rows, seq_len, n_rot_heads, log2_hd,
                           log2_step, row_stride, inverse);
  }
  const long long total = (long long)rows * n_rot_heads * (hd / 16);
  return (int)launch_dep(rope_kernel, blocks_for(total, 256), 256, 0, ST(stream), BF(qkv), cos_t,
                         sin_t, total, seq_len, n_rot_heads, hd, row_stride, inverse);
}

extern "C" int mb200_swiglu_fwd(const void* gu, void* h, int rows, int F, void* stream) {
  if (rows <= 0) return 0;
  if (F % 8 || F <= 0) return 1001;
  const dim3 b = row_block(F / 8);
  return (int)launch_dep(b.y > 1 ? swiglu_fwd_kernel<true> : swiglu_fwd_kernel<false>,
                         row_grid(rows, F / 8, b), b, 0, ST(stream), CBF(gu), BF(h), rows, F);
}
extern "C" int mb200_swiglu_bwd(const void* gu, const void* dh, void* dgu, int rows, int F,
                                void* stream) {
  if (rows <= 0) return 0;
  if (F % 8 || F <= 0) return 1001;
  const dim3 b = row_block(F / 8);
  return (int)launch_dep(b.y > 1 ? swiglu_bwd_kernel<true> : swiglu_bwd_kernel<false>,
                         row_grid(rows, F / 8, b), b, 0, ST(stream), CBF(gu), CBF(dh), BF(dgu), rows,
                         F);
}

extern "C" int mb200_cross_entropy_fwd_bwd(void* logits, const int64_t* targets, float* loss_rows,
                                           int rows, int V, int ld, float grad_scale,
                                           void* stream) {
  if (rows <= 0) return 0;
  if (ld % 8) return 1001;
#define MB200_CE(NT)                                                                      \
  return (int)launch_dep(cross_entropy_kernel<NT>, rows, NT, 0, ST(stream), BF(logits), targets, \
                         loss_rows, V, ld, grad_scale)
  const bool many = rows >= 512;
  if (V <= (many ? 6144 : 4096)) MB200_CE(128);
  if (many && V <= 16384) MB200_CE(256);
  if (V < 65536) MB200_CE(512);
  MB200_CE(1024);
#undef MB200_CE
}

extern "C" int mb200_adamw(float* p, float* m, float* v, const void* g, void* p_bf16, int64_t n,
                           int g_bf16, float lr, float beta1, float beta2, float eps, float wd,
                           int step, float grad_scale, void* stream) {
  if (n <= 0) return 0;
  const double bc1 = 1.0 - pow((double)beta1, (double)step);
  const double bc2 = 1.0 - pow((double)beta2, (double)step);
  const long long nthreads = (n + 3) / 4;
  return (int)launch_dep(adamw_kernel, blocks_for(nthreads, 256), 256, 0, ST(stream), p, m, v, g,
                         BF(p_bf16), n, g_bf16, lr, beta1, beta2, eps, wd, (float)(1.0 / bc1),
                         (float)(1.0 / sqrt(bc2)), grad_scale);
}

extern "C" int mb200_embedding_fwd(const void* table, const int64_t* ids, void* out, int rows,
                                   int d, void* stream) {
  if (rows <= 0) return 0;
  if (d % 8) return 1001;
  const long long total = (long long)rows * (d / 8);
  return (int)launch_dep(embedding_fwd_kernel, blocks_for(total, 256), 256, 0, ST(stream),
                         CBF(table), ids, BF(out), total, d);
}
extern "C" int mb200_embedding_bwd(const void* dout, const int64_t* ids, void* dtable, int rows,
                                   int d, void* stream) {
  if (rows <= 0) return 0;
  if (d % 2 || d <= 0) return 1001;
  if (d % 8 == 0 && aligned16(dout) && aligned16(dtable)) {
    const dim3 b = row_block(d / 8);
    return (int)launch_dep(b.y > 1 ? embedding_bwd_vec_kernel<true>
                                   : embedding_bwd_vec_kernel<false>,
                           row_grid(rows, d / 8, b), b, 0, ST(stream), CBF(dout), ids, BF(dtable),
                           rows, d);
  }
  const long long total = (long long)rows * (d / 2);
  return (int)launch_dep(embedding_bwd_kernel, blocks_for(total, 256), 256, 0, ST(stream),
                         CBF(dout), ids, BF(dtable), total, d);
}

extern "C" int mb200_sumsq(const void* x, int64_t n, int is_bf16, float* out, void* stream) {
  if (n <= 0) return 0;
  return (int)launch_dep(sumsq_kernel, 592, 256, 0, ST(stream), x, n, is_bf16, out);
}

// ------------------------------------------------- allocation-free RMSNorm backward ----
// See mb200_noalloc.h.  The partial weight-gradient sums live in this file-scope device
// array instead of a caller-provided buffer.  In host code `g_noalloc_scratch` is only a
// handle for the runtime, not a device address: the address the kernels receive comes
// from cudaGetSymbolAddress, resolved once per device.
#include <stdio.h>

#include <mutex>

#include "mb200_noalloc.h"

static __device__ __align__(256) float g_noalloc_scratch[MB200_NOALLOC_SCRATCH_FLOATS];

namespace {
constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mu;
float* g_noalloc_ptr[kNoallocMaxDevices] = {nullptr};

// Device address of the scratch on the current device (resolved on first use).
int noalloc_scratch(float** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kNoallocMaxDevices) return MB200_NOALLOC_ERR_SYMBOL;
  std::lock_guard<std::mutex> g(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      fprintf(stderr, "mb200_rmsnorm_bwd_noalloc: cudaGetSymbolAddress failed on device %d: %s\n",
              dev, cudaGetErrorString(e));
      return e != cudaSuccess ? (int)e : MB200_NOALLOC_ERR_SYMBOL;
    }
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}
}  // namespace

extern "C" int mb200_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w,
                                         const float* rstd, const void* dres, void* dx, void* dw,
                                         int dw_accumulate, int rows, int d, void* stream) {
  if (rows < 0) {
    fprintf(stderr, "mb200_rmsnorm_bwd_noalloc: rows = %d is negative\n", rows);
    return MB200_NOALLOC_ERR_BAD_ROWS;
  }
  if (d <= 0 || d % 8 || d > MB200_NOALLOC_MAX_D) {
    fprintf(stderr,
            "mb200_rmsnorm_bwd_noalloc: d = %d is not supported (multiple of 8, at most %d: the "
            "built-in scratch holds %d floats)\n",
            d, MB200_NOALLOC_MAX_D, MB200_NOALLOC_SCRATCH_FLOATS);
    return MB200_NOALLOC_ERR_BAD_D;
  }
  if (rows == 0) return 0;
  float* scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  // As many row-striding blocks as the scratch has room for ([blocks, d] floats).
  int nb = mb200_rmsnorm_bwd_blocks(rows);
  const int cap = MB200_NOALLOC_SCRATCH_FLOATS / d;
  if (nb > cap) nb = cap;
  return launch_rmsnorm_bwd(nb, CBF(dy), CBF(x), CBF(w), rstd, CBF(dres), BF(dx), scratch, BF(dw),
                            dw_accumulate, rows, d, /*status=*/nullptr, ST(stream));
}
