// Host build of the unrolled multi-population statistics
// (pg_gpu_gb300/csrc/pgld_multi.cuh) for tests/test_multi_cpu.py.
#include <utility>

#define __host__
#define __device__
#include "../../pg_gpu_gb300/csrc/pgld_multi.cuh"

using namespace pgld;

template <int P, class F>
static void run(const F (&f)[P], float* out) {
  const std::vector<multi::Place> o = multi::order(P, F::geno);
  multi::eval<P, true, true>(f, [&](int k, float v) { out[o[k].stat] = v * o[k].factor; });
}

template <int P>
static void rows(const int* c, int N, bool geno, float* out, int S) {
  for (int k = 0; k < N; ++k, out += S) {
    if (geno) {
      multi::Geno f[P];
      for (int p = 0; p < P; ++p) f[p] = multi::make_geno(gmom::from_counts(c + (k * P + p) * 9));
      run<P>(f, out);
    } else {
      multi::Hap f[P];
      for (int p = 0; p < P; ++p) {
        const int* x = c + (k * P + p) * 4;
        f[p] = multi::make_hap((float)x[0], (float)x[1], (float)x[2], (float)x[3]);
      }
      run<P>(f, out);
    }
  }
}

// counts [N][P][4 or 9] -> out [N][S], every statistic in moments' order
extern "C" void pgld_check_multi(const int* counts, int N, int P, int geno, float* out, int S) {
  if (P == 2) rows<2>(counts, N, geno != 0, out, S);
  if (P == 3) rows<3>(counts, N, geno != 0, out, S);
  if (P == 4) rows<4>(counts, N, geno != 0, out, S);
}

// float32 denominators M a b / M (M = 1, 2, 4) and the two conversions' of M a b
extern "C" void pgld_check_den(const float* a, const float* b, int N, float* out) {
  for (int k = 0; k < N; ++k, out += 6) {
    out[0] = multi::round_den<1>(a[k], b[k]);
    out[1] = multi::round_den<2>(a[k], b[k]);
    out[2] = multi::round_den<4>(a[k], b[k]);
    for (int m = 0; m < 3; ++m) {
      const long long x = ((long long)a[k] * (long long)b[k]) << m;
      out[3 + m] = fmaf((float)(int)(x >> 31), 2147483648.0f, (float)(int)(x & 0x7fffffff)) / (1 << m);
    }
  }
}
