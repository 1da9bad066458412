// Host build of the integer quotient (pg_gpu_gb300/csrc/pgld_quot.cuh) for
// tests/test_quot_cpu.py.
#include "../../pg_gpu_gb300/csrc/pgld_quot.cuh"

extern "C" void pgld_check_quot(const long long* num, const long long* den, int n, double* out) {
  for (int k = 0; k < n; ++k) out[k] = pgld::quotient(num[k], den[k]);
}
// the digit estimates with the reciprocal off by `ulps` of 2^-23 (the device's
// approximate reciprocal): the remainder's bound after each digit, in units of B
extern "C" double pgld_check_remainder(const long long* num, const long long* den, int n, double off) {
  double worst = 0.0;
  for (int k = 0; k < n; ++k) {
    using namespace pgld::quot_detail;
    const int la = lead0(num[k]), lb = lead0(den[k]);
    const pgld::u64 A = (pgld::u64)num[k] << (la - 4), B = (pgld::u64)den[k] << (lb - 4);
    const float r = (float)((1.0 / (double)(float)(uint32_t)(B >> 28)) * (1.0 + off));
    const uint32_t V = (uint32_t)(r * (36028797018963968.0f * (1.0f - 2.0f / 4194304.0f)));
    unsigned __int128 R = A >= B ? A - B : A;
    for (int s = 0; s < 3; ++s) {
      const uint32_t d = mulhi((uint32_t)(R >> 32), V);
      const unsigned __int128 up = R << 19, take = (unsigned __int128)d * B;
      if (take > up) return -1.0;
      R = up - take;
      const double ratio = (double)R / (double)B;
      worst = ratio > worst ? ratio : worst;
    }
  }
  return worst;
}
