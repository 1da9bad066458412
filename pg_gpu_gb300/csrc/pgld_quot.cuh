// The correctly rounded float64 quotient of two 64-bit integers on the integer
// pipes.  GB300 issues about two float64 operations per SM and clock, so a
// statistic's two conversions and division keep that pipe busy for five clocks
// per value; long division by three 19-bit digits takes about ninety 32-bit
// integer instructions, 64 lanes a clock.
//
// With A and B the operands shifted to 60 bits, A / B lies in (1/2, 2) and
// Q = floor(2^57 A / B) is built from the integer bit and three digits.  A
// digit is estimated from the top bits of the remainder R with V, a slightly
// low 2^55 / floor(B / 2^28) from the float32 reciprocal: the estimate never
// exceeds R 2^19 / B and falls short of it by less than 2, so R stays below
// 2 B from digit to digit (the next digit takes the excess up), and the low 64
// bits of R 2^19 - digit B are exact.  One comparison completes Q; its 57 or 58
// bits and whether a remainder is left round to 53 bits (nearest, ties to
// even) like the division instruction.
#pragma once
#include <stdint.h>

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define PGLD_Q_HD __host__ __device__ __forceinline__
#else
#define PGLD_Q_HD inline
#endif

namespace pgld {

typedef unsigned long long u64;

namespace quot_detail {
PGLD_Q_HD int lead0(u64 x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}
PGLD_Q_HD uint32_t mulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((u64)a * b) >> 32);
#endif
}
// below 2^55 / bh by a relative 2^-22 to 2^-20 (bh in [2^31, 2^32)): the
// conversion, the reciprocal and the product are each off by at most 2^-23
PGLD_Q_HD uint32_t low_reciprocal(uint32_t bh) {
  constexpr float scale = 36028797018963968.0f * (1.0f - 2.0f / 4194304.0f);  // 2^55 (1 - 2^-21)
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint2float_rn(bh)));
  return __float2uint_rz(r * scale);
#else
  return (uint32_t)((1.0f / (float)bh) * scale);
#endif
}
}  // namespace quot_detail

// num / den rounded to float64, 0 < den < 2^53, |num| < 2^53
PGLD_Q_HD double quotient53(long long num, long long den) {
  using namespace quot_detail;
  const u64 a = num < 0 ? (u64)-num : (u64)num;
  if (a == 0) return 0.0;
  const int la = lead0(a), lb = lead0((u64)den);
  const u64 A = a << (la - 4), B = (u64)den << (lb - 4);
  const uint32_t V = low_reciprocal((uint32_t)(B >> 28));
  u64 Q = A >= B ? 1 : 0;
  u64 R = A - (Q ? B : 0);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int k = 0; k < 3; ++k) {
    const uint32_t d = mulhi((uint32_t)(R >> 32), V);
    R = (R << 19) - (u64)d * B;
    Q = (Q << 19) + d;
  }
  if (R >= B) {
    R -= B;
    ++Q;
  }
  int e = lb - la;
  if (!(Q >> 57)) {
    Q <<= 1;
    --e;
  }
  Q |= R != 0 ? 1 : 0;
  const u64 m = (Q + 0xf + ((Q >> 5) & 1)) >> 5;  // 2^52 .. 2^53: the hidden bit adds to the exponent
  const u64 bits = ((u64)(e + 1022) << 52) + m + (num < 0 ? 1ull << 63 : 0ull);
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)bits);
#else
  double v;
  std::memcpy(&v, &bits, 8);
  return v;
#endif
}

// (double)num / (double)den for den > 0: operands of more than 53 bits are
// rounded first, by the float64 unit
PGLD_Q_HD double quotient(long long num, long long den) {
  const u64 a = num < 0 ? (u64)-num : (u64)num;
  if (((a | (u64)den) >> 53) != 0) return (double)num / (double)den;
  return quotient53(num, den);
}

}  // namespace pgld
