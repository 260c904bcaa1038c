// Runs an attention kernel's source under many schedules (tests/test_kernel_waits.py).
// Arguments: head size, warps of a block, seeds per actor that is held back.
#include KERNEL_SOURCE

#include <stdlib.h>

namespace mb200 {
int make_tmap_bf16_2d(CUtensorMap*, const void*, uint64_t, uint64_t, uint64_t, uint32_t, uint32_t) {
  return 0;
}
}  // namespace mb200

int main(int, char** argv) {
  const int hd = atoi(argv[1]);
  const int B = 1, S = 3 * 128, Hq = 2, Hkv = 1, ld = (Hq + 2 * Hkv) * hd;
  std::vector<__nv_bfloat16> qkv((size_t)B * S * ld), o((size_t)B * S * Hq * hd + 16);
  std::vector<float> lse((size_t)B * Hq * S + 16), delta((size_t)B * Hq * S + 16);
  const auto up16 = [](void* p) { return (float*)(((uintptr_t)p + 15) & ~(uintptr_t)15); };
  std::vector<__nv_bfloat16> d(qkv.size() + 16);
  auto* dq = (__nv_bfloat16*)up16(d.data());
  auto* ob = (__nv_bfloat16*)up16(o.data());
  const int n_warps = atoi(argv[2]), n_seeds = atoi(argv[3]);
  // random schedules, and for every warp, the tensor pipe and the TMA unit some that hold it back
  for (int starved = -1; starved < n_warps + 2; ++starved)
    for (int seed = 0; seed < n_seeds; ++seed) {
      hostsim::g_seed = (unsigned)seed;
      hostsim::g_starved = starved;
      hostsim::g_device = seed & 1;
#ifdef BACKWARD
      const int rc = mb200_attn_bwd(qkv.data(), qkv.data(), qkv.data(), ob, ob, up16(lse.data()),
                                    up16(delta.data()), dq, dq + Hq * hd, dq + (Hq + Hkv) * hd, B, S,
                                    Hq, Hkv, hd, ld, Hq * hd, ld, 1.f, nullptr, nullptr);
#else
      const int rc = mb200_attn_fwd(qkv.data(), qkv.data(), qkv.data(), ob, up16(lse.data()), B, S, Hq,
                                    Hkv, hd, ld, Hq * hd, 1.f, nullptr, nullptr);
#endif
      if (rc) {
        printf("held back %d, seed %d: %d %s\n", starved, seed, rc, hostsim::g_error.c_str());
        return 1;
      }
    }
  return 0;
}
