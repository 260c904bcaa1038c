// The RMSNorm backward's source with a copy that never lands (tests/test_kernel_waits.py).
// Arguments: row width, the copy that is left out (-1: none), seeds per actor that is held back.
#include KERNEL_SOURCE

#include <stdlib.h>

using namespace mb200;

int main(int, char** argv) {
  const int d = atoi(argv[1]), drop = atoi(argv[2]), n_seeds = atoi(argv[3]);
  const int rows = 23, nb = 2;
  const auto one = __float2bfloat16(1.f);
  std::vector<__nv_bfloat16> x((size_t)rows * d, one), w(d, one), dx(x.size()), dw(d);
  std::vector<float> rstd(rows, 1.f), part((size_t)nb * d);
  const int n_warps = d > 4096 ? 16 : 8;
  for (int starved = -1; starved < n_warps + 2; ++starved)
    for (int seed = 0; seed < n_seeds; ++seed)
      for (int res = 0; res < 2; ++res) {
        hostsim::g_seed = (unsigned)seed;
        hostsim::g_starved = starved;
        hostsim::g_device = seed & 1;
        hostsim::g_drop = drop;
        int status = 0;
        const auto untouched = __float2bfloat16(7.f);
        for (auto& v : dx) v = untouched;
        const int rc = launch_rmsnorm_bwd(nb, x.data(), x.data(), w.data(), rstd.data(),
                                          res ? x.data() : nullptr, dx.data(), part.data(),
                                          dw.data(), 0, rows, d, &status, nullptr);
        if (rc) {
          printf("held back %d, seed %d: %d %s\n", starved, seed, rc, hostsim::g_error.c_str());
          return 1;
        }
        // the copies of a row are issued together, in the order of a block's rows
        const int lost = drop < 0 ? rows : drop / (2 + res) * nb;
        if (status != (drop >= 0)) return printf("status %d\n", status), 1;
        for (int row = 0; row < rows; ++row)
          for (int c = 0; c < d; c += 256) {   // the columns of lane 0
            const float v = __bfloat162float(dx[(size_t)row * d + c]);
            // (the status is sticky: a later block may give up on its first row already)
            if (row < lost && (row % nb == 0 || drop < 0) ? !isfinite(v) || v == 7.f
                : row < lost                              ? v == 7.f
                                                          : !isnan(v))
              return printf("held back %d, seed %d, residual %d: row %d of %d, lost from %d: dx %g\n", starved, seed, res, row, rows, lost, v), 1;
          }
        for (int b = 0; b < nb; ++b)
          if (isnan(part[(size_t)b * d]) != (drop >= 0)) return printf("weight gradient\n"), 1;
      }
  return 0;
}
