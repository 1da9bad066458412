// Host build of the float32 numerators that count draws
// (pg_gpu_gb300/csrc/pgld_epilogue.cuh, pgld_multi.cuh) for tests/test_draws_cpu.py.
#include <utility>

#define __host__
#define __device__
#include "../../pg_gpu_gb300/csrc/pgld_multi.cuh"

using namespace pgld;

// counts [N][3][4] -> out [N][6]: pi2, triple (times 2), ijij (times 16) of the
// first two populations, shared of the three, DD and the rest of DD
extern "C" void pgld_check_hap_draws(const int* c, int N, float* out) {
  for (int k = 0; k < N; ++k, c += 12, out += 6) {
    multi::Hap h[3];
    for (int p = 0; p < 3; ++p)
      h[p] = multi::make_hap((float)c[4 * p], (float)c[4 * p + 1], (float)c[4 * p + 2], (float)c[4 * p + 3]);
    const multi::Den one = {1.0f, 0.0f};
    out[0] = h[0].pi;
    out[1] = multi::triple(h[0], h[1], one, true);
    out[2] = multi::ijij(h[0], h[1]);
    out[3] = multi::shared(h[0], h[1], h[2]);
    out[4] = h[0].dd;
    out[5] = h[0].ddr;
  }
}

// counts [N][3][9] -> out [N][2]: ijij and shared (both a quarter)
extern "C" void pgld_check_geno_draws(const int* c, int N, float* out) {
  for (int k = 0; k < N; ++k, c += 27, out += 2) {
    multi::Geno g[3];
    for (int p = 0; p < 3; ++p) g[p] = multi::make_geno(gmom::from_counts(c + 9 * p));
    out[0] = multi::ijij(g[0], g[1]);
    out[1] = multi::shared(g[0], g[1], g[2]);
  }
}
