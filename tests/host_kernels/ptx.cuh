// Stands in for csrc/kernels/ptx.cuh when a kernel's source is compiled for the CPU: the warps of
// a block are coroutines (lane 0 of each), the barriers count as mbarriers do, and the TMA unit and
// the tensor pipe are two more actors that finish what was issued whenever the schedule lets
// them.  What is checked is that no schedule lets a wait miss its phase or pass on another one,
// that every warp ends, and that none ends while others wait at a block barrier or copies are in
// flight.  The tensor pipe computes nothing.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <ucontext.h>

#include <deque>
#include <map>
#include <random>
#include <string>
#include <utility>
#include <vector>

#undef __launch_bounds__
#define __launch_bounds__(...)
#undef __grid_constant__
#define __grid_constant__

struct HostDim {
  unsigned x = 0, y = 0, z = 0;
};
static HostDim threadIdx, blockIdx, blockDim, gridDim;

namespace hostsim {

struct Barrier {
  int count = 0, pending = 0;
  long long tx = 0;
  int done = 0;   // completed phases
};
struct Warp {
  ucontext_t ctx;
  std::vector<char> stack;
  bool ended = false, at_block_barrier = false, polls = false;
  uint64_t* waits_on = nullptr;
  volatile int* abort_word = nullptr;
  int* status = nullptr;
  uint32_t parity = 0;
  int phase = 0;                          // the phase that this wait is for
  std::map<uint64_t*, int> next_phase;    // of this warp's next wait on a barrier
};

struct Load {
  uint64_t* bar;
  long long bytes;
  void* dst;
  const void* src;
};
struct Sim {
  std::map<uint64_t*, Barrier> bars;
  std::vector<Warp> warps;
  std::deque<uint64_t*> commits;                                 // tensor pipe, in order
  std::vector<Load> loads;                                       // TMA, in any order
  int issued = 0, drop = -1;                                     // this one never lands
  ucontext_t main;
  int cur = -1, at_barrier = 0;
  std::string error;
  std::mt19937 rng;
  int starved = -1;   // this actor runs only when no other can
};
static Sim* S = nullptr;

static void settle(Barrier& b) {
  if (b.pending == 0 && b.tx == 0) {
    ++b.done;
    b.pending = b.count;
  }
}
static void yield() { swapcontext(&S->warps[S->cur].ctx, &S->main); }
static void arrive(uint64_t* bar) {
  Barrier& b = S->bars[bar];
  if (--b.pending < 0) S->error = "more arrivals than the barrier's count";
  settle(b);
}
static bool passes(uint64_t* bar, uint32_t parity) {
  return (uint32_t)(S->bars[bar].done & 1) != parity;
}
static bool gives_up(const Warp& w) { return *w.abort_word || (w.status && *w.status); }
static void load(uint64_t* bar, long long bytes, void* dst = nullptr, const void* src = nullptr) {
  if (S->issued++ != S->drop) S->loads.push_back({bar, bytes, dst, src});
}

// Runs one block; `body` is the kernel with its arguments bound.
template <typename F>
static std::string run_block(int n_warps, unsigned seed, int starved, int drop, F&& body) {
  Sim sim;
  S = &sim;
  sim.rng.seed(seed);
  sim.starved = starved;
  sim.drop = drop;
  sim.warps.resize(n_warps);
  static F* entry;
  entry = &body;
  for (int i = 0; i < n_warps; ++i) {
    Warp& w = sim.warps[i];
    w.stack.resize(256 << 10);
    getcontext(&w.ctx);
    w.ctx.uc_stack.ss_sp = w.stack.data();
    w.ctx.uc_stack.ss_size = w.stack.size();
    w.ctx.uc_link = &sim.main;
    makecontext(&w.ctx, (void (*)())+[] {
      (*entry)();
      S->warps[S->cur].ended = true;
    }, 0);
  }
  const int kTensor = n_warps, kTma = n_warps + 1;
  while (sim.error.empty()) {
    std::vector<int> can;
    bool all_ended = true;
    for (int i = 0; i < n_warps; ++i) {
      Warp& w = sim.warps[i];
      if (w.ended) continue;
      all_ended = false;
      if (w.at_block_barrier || w.polls) continue;
      if (w.waits_on) {
        const int done = sim.bars[w.waits_on].done;
        if (done >= w.phase + 2)
          sim.error = "warp " + std::to_string(i) + ": phase " + std::to_string(w.phase) +
                      " of a barrier came and went before the wait for it";
        else if (passes(w.waits_on, w.parity) && done != w.phase + 1)
          sim.error = "warp " + std::to_string(i) + ": a wait passes before its phase";
        if (!passes(w.waits_on, w.parity) && !gives_up(w)) continue;
      }
      can.push_back(i);
    }
    if (all_ended && !sim.loads.empty()) sim.error = "copies in flight at the block's end";
    if (all_ended || !sim.error.empty()) break;
    if (!sim.commits.empty()) can.push_back(kTensor);
    if (!sim.loads.empty()) can.push_back(kTma);
    for (int i = 0; i < n_warps && can.empty(); ++i)   // a bounded loop, slower than all else
      if (!sim.warps[i].ended && sim.warps[i].polls) can.push_back(i);
    for (int i = 0; i < n_warps && can.empty() && drop >= 0; ++i) {
      Warp& w = sim.warps[i];   // a wait's limit is reached
      if (w.ended || !w.waits_on) continue;
      *w.abort_word = 1;
      if (w.status && !*w.status) *w.status = 1;
      can.push_back(i);
    }
    if (can.empty()) {
      sim.error = "no warp can go on";
      break;
    }
    std::vector<int> pick;
    for (int i : can)
      if (i != sim.starved) pick.push_back(i);
    if (pick.empty()) pick = can;
    const int a = pick[sim.rng() % pick.size()];
    if (a == kTensor) {
      uint64_t* bar = sim.commits.front();
      sim.commits.pop_front();
      arrive(bar);
    } else if (a == kTma) {
      const size_t k = sim.rng() % sim.loads.size();
      const Load& l = sim.loads[k];
      Barrier& b = sim.bars[l.bar];
      b.tx -= l.bytes;
      if (l.dst) memcpy(l.dst, l.src, (size_t)l.bytes);
      sim.loads.erase(sim.loads.begin() + k);
      settle(b);
    } else {
      sim.cur = a;
      threadIdx.x = a * 32;
      swapcontext(&sim.main, &sim.warps[a].ctx);
    }
  }
  return sim.error;
}
}  // namespace hostsim

static inline void __syncthreads() {
  using namespace hostsim;
  if (++S->at_barrier == (int)S->warps.size()) {
    S->at_barrier = 0;
    for (auto& w : S->warps) w.at_block_barrier = false;   // (a warp that has ended never arrives)
  } else {
    S->warps[S->cur].at_block_barrier = true;
  }
  yield();
}
static inline void __syncwarp() {}
static inline int __any_sync(unsigned, int p) { return p; }
static inline float __shfl_xor_sync(unsigned, float v, int) { return v; }
static inline float __uint_as_float(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static inline uint32_t __float_as_uint(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static inline float __int_as_float(int i) { return __uint_as_float((uint32_t)i); }
static inline float rsqrtf(float x) { return 1.f / sqrtf(x); }
static inline long long clock64() {
  static long long t = 0;
  return t += 100;
}
#define MB200_WAIT_CYCLES 100000
// Two devices: what a kernel may use on one says nothing about the other.
namespace hostsim {
static int g_device = 0;
static std::map<std::pair<const void*, int>, int> g_allowed;
}  // namespace hostsim
extern "C" cudaError_t cudaGetDevice(int* dev) {
  *dev = hostsim::g_device;
  return cudaSuccess;
}
template <typename F>
static cudaError_t cudaFuncSetAttribute(F* kernel, cudaFuncAttribute, int bytes) {
  hostsim::g_allowed[{(const void*)kernel, hostsim::g_device}] = bytes;
  return cudaSuccess;
}

static inline int atomicCAS(int* p, int want, int now) {
  const int was = *p;
  if (was == want) *p = now;
  return was;
}

namespace mb200 {
enum : int { kStatusOk = 0, kStatusMbarTimeout = 1 };
inline int sm_count() { return 148; }
inline uint8_t smem[232448] __attribute__((aligned(1024)));       // dynamic shared memory, by the
inline uint8_t smem_raw[232448] __attribute__((aligned(1024)));   // names the kernels give it
inline uint8_t ring[232448] __attribute__((aligned(1024)));

static inline uint32_t smem_u32(const void* p) { return (uint32_t)(uintptr_t)p; }
static inline uint32_t elect_one() { return 1; }
static inline void mbar_init(uint64_t* b, uint32_t n) {
  hostsim::S->bars[b] = hostsim::Barrier{(int)n, (int)n, 0, 0};
}
static inline void mbar_fence_init() {}
static inline void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  hostsim::S->bars[b].tx += bytes;
  hostsim::arrive(b);
  hostsim::yield();
}
static inline void mbar_arrive(uint64_t* b) {
  hostsim::arrive(b);
  hostsim::yield();
}
static inline bool mbar_try_wait(uint64_t* b, uint32_t parity) {
  auto& w = hostsim::S->warps[hostsim::S->cur];
  w.polls = true;
  hostsim::yield();
  w.polls = false;
  return hostsim::passes(b, parity);
}
static inline bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort_word, int* status) {
  auto& w = hostsim::S->warps[hostsim::S->cur];
  // parity 1 at the first wait asks for the phase before the first
  auto it = w.next_phase.emplace(b, parity ? -1 : 0).first;
  w.waits_on = b;
  w.parity = parity;
  w.phase = it->second++;
  w.abort_word = abort_word;
  w.status = status;
  hostsim::yield();
  w.waits_on = nullptr;
  if (hostsim::passes(b, parity)) return true;
  *abort_word = 1;
  return false;
}
static inline void tma_prefetch_desc(const CUtensorMap*) {}
static inline void tma_load_2d(void*, const CUtensorMap*, uint64_t* bar, int, int) {
  hostsim::load(bar, 64 * 128 * 2);   // a box of 128 rows of 64 bf16
}
static inline void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  hostsim::load(bar, bytes, dst, src);
}
static inline void tmem_alloc(uint32_t* dst, int) { *dst = 0; }
static inline void tmem_relinquish() {}
static inline void tmem_dealloc(uint32_t, int) {}
static inline void tc_fence_before() {}
static inline void tc_fence_after() {}
static inline void umma_commit(uint64_t* bar) {
  hostsim::S->commits.push_back(bar);
  hostsim::yield();
}
template <typename... A> static inline void umma_f16(A...) {}
template <typename... A> static inline void umma_f16_ts(A...) {}
template <typename... A> static inline uint64_t umma_smem_desc_sw128(A...) { return 0; }
constexpr uint32_t umma_idesc_bf16(int, int, int, int) { return 0; }
template <size_t N> static inline void tmem_ld_32x32b_x32(uint32_t, uint32_t (&v)[N]) { memset(v, 0, sizeof v); }
template <size_t N> static inline void tmem_ld_32x32b_x16(uint32_t, uint32_t (&v)[N]) { memset(v, 0, sizeof v); }
template <typename T> static inline void tmem_st_32x32b_x32(uint32_t, const T&) {}
template <typename T> static inline void tmem_st_32x32b_x16(uint32_t, const T&) {}
template <typename T> static inline void tmem_st_32x32b_x8(uint32_t, const T&) {}
static inline void tmem_ld_wait() {}
static inline void tmem_st_wait() {}
static inline float ex2_approx(float x) { return exp2f(x); }
static inline uint32_t pack_bf16x2(float a, float b) {
  const __nv_bfloat16 v[2] = {__float2bfloat16(a), __float2bfloat16(b)};
  uint32_t u;
  memcpy(&u, v, 4);
  return u;
}
static inline float2 unpack_bf16x2(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
static inline uint64_t pack_f32x2(float, float) { return 0; }
static inline float2 unpack_f32x2(uint64_t) { return make_float2(0.f, 0.f); }
static inline uint64_t fma_f32x2(uint64_t, uint64_t, uint64_t) { return 0; }
static inline uint64_t add_f32x2(uint64_t, uint64_t) { return 0; }
static inline uint64_t mul_f32x2(uint64_t, uint64_t) { return 0; }
}  // namespace mb200
