// Float32 finalisation of the moments statistics of two to four populations
// (haplotypes: three and four; genotypes: two to four), unrolled at compile
// time.
//
// The statistic table of P populations falls into classes by the denominator
// its statistics share -- products of falling factorials of the populations'
// valid sample sizes:
//   d4(i)        n(n-1)(n-2)(n-3)          DD_ii, Dz_iii, pi2_iiii
//   d22(i,j)     n_i(n_i-1) n_j(n_j-1)     DD_ij, Dz_ijj, Dz_jii, pi2_iijj, pi2_ijij
//   d31(i,j)     n_i(n_i-1)(n_i-2) n_j     Dz_iij, pi2_iiij
//   d211(s,a,b)  n_s(n_s-1) n_a n_b        Dz_sab, pi2_ssab, pi2_sasb
//   d1111        n_0 n_1 n_2 n_3           the three pi2 of four populations
// so a pair takes one reciprocal per class, two where haplotype denominators of
// one class round apart (21 for three populations, 53 for four) instead of one
// division per term (63 and 315 terms).
//
// Features per population are exact float32 integers for sample sizes up to
// kMaxN.  The numerators of mixed pi2 statistics are counts of draws: the product
// of two exact features, one per SNP, less the choices that take a haplotype (an
// individual) twice, a sum of non-negative products that is smaller by a factor
// n.  They are exact where they are small or 0 and otherwise round once in
// effect, like the 64-bit integers of the term table on their way to float32;
// pi2_ijij is a two-product sum by Kahan's algorithm, and DD of one population
// keeps its rounding error.  Against 64 bits the values of every statistic are no
// further off than the table's: root mean square 0.51 - 0.83 units of 2^-24 of the
// statistic where the table has 0.59 - 0.87 (three and four haplotype populations of
// 30 - 400), 0.46 - 0.81 and 0.55 - 0.86 (two to four genotype populations of 30 -
// 500), the largest ones 4.2 and 4.6 units of the terms' absolute sum.
//
// A quotient is num * (r + rl): r the approximate reciprocal of the
// denominator den (the exact integer in float32: a product of two exact
// factors below 2^24, rounded as round_den says), rl = r (1 - den r) its correction, added
// before the product rounds.  So a quotient carries no bias that repeats over
// the pairs of equal sample size, as a rounded reciprocal would: sums over
// 10^8 pairs keep an error near 1e-9.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "pgld_epilogue.cuh"
#include "pgld_geno_mom.cuh"

namespace pgld {
namespace multi {

constexpr int kMaxN = 2048;  // largest sample size whose features are exact

// statistics of group 0 (d4, d22, d31) and group 1 (d211, d1111)
__host__ __device__ constexpr int group_size(int P, int g) {
  return g == 0 ? 3 * P + 5 * P * (P - 1) / 2 + 2 * P * (P - 1)
                : 3 * P * (P - 1) * (P - 2) / 2 + (P == 4 ? 3 : 0);
}

struct Den {
  float r, rl;
};
// a b, exact factors below 2^23 (haplotype denominators): the float32 of M a b
// over M, as the two 32-bit conversions of the 64-bit product round it -- its
// bits from 2^31 on, plus the rounded rest.  M is the factor that the term
// table's denominator carries (1, 2 or 4).  From n = 152 on this is not always
// the nearest float32 of a b; where one sample size is frequent (n = 390, 4%
// missing) the difference would shift a bin's sum by 1e-8 of a statistic.
template <int M>
PGLD_HD float round_den(float a, float b) {
  constexpr float G = 1.5f * 18014398509481984.0f / M;  // ulp 2^31 / M
#ifdef __CUDA_ARCH__
  const float s = __fmaf_rd(a, b, G);
#else
  constexpr double U = 2147483648.0 / M;
  const double fl = (double)(long long)((double)a * b / U) * U;
  const float s = (float)(G + fl);
#endif
  const float low = fmaf(a, b, G - s);
  return (s - G) + low;
}
// den: the rounded denominator.  Where it is 0 (fewer samples than draws) the
// numerators count no draws and are exactly 0, so any other value will do
PGLD_HD Den make_den(float den) {
  Den d;
  den = fmaxf(den, 1.0f);
#ifdef __CUDA_ARCH__
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(d.r) : "f"(den));
#else
  d.r = 1.0f / den;
#endif
  d.rl = d.r * fmaf(-den, d.r, 1.0f);
  return d;
}
PGLD_HD float quot(float num, Den d) { return fmaf(num, d.r, fast::fmul(num, d.rl)); }
// of a numerator and the rest that its rounding dropped
PGLD_HD float quot(float num, float rest, Den d) {
  return fmaf(num, d.r, fmaf(rest, d.r, fast::fmul(num, d.rl)));
}

struct Size {
  float n, m, m2, k, m2b;  // n, n - 1, n (n - 1), n - 2, (n - 2)(n - 3)
};
PGLD_HD Size make_size(float n) {
  Size s;
  s.n = n;
  s.m = n - 1.0f;
  s.m2 = n * (n - 1.0f);
  s.k = n - 2.0f;
  s.m2b = s.k * (n - 3.0f);
  return s;
}

// A statistic that averages quotients of two kinds adds them term by term, in
// the table's order (a, a, b, b or a, a, a, a, b, b, b, b; the factor of the
// first is left out here: two_two is (a + a + b + b) / 2, four_four a
// quarter).  At small sample sizes every numerator is an exact float32, the
// same few quotients recur in all pairs, and their roundings do not average
// out: the sum of the terms and the quotient of the summed numerators differ
// by up to 2e-9 of a bin of 10^8 pairs.
PGLD_HD float two_two(float a, float b) { return fmaf(b, 0.5f, fmaf(b, 0.5f, a)); }
PGLD_HD float four_four(float a, float b) {
  return fmaf(b, 0.25f, fmaf(b, 0.25f, fmaf(b, 0.25f, fmaf(b, 0.25f, a))));
}

// ---- haplotypes ------------------------------------------------------------
struct Hap {
  Size z;
  float c1, c2, c3, c4;
  float x, w, dA, dB;         // c1c4 - c2c3, dA dB + e, qA - pA, qB - pB
  float pA, qA, pB, qB, hA, hB;  // hA = pA qA, hB = pB qB
  float yb, yB;               // pA c4 + c2 qA, pA c3 + c1 qA: draws (A, a), one of them also b / B
  float dd, ddr, dz, pi;      // numerators over d4, ddr the rest of dd
  static constexpr bool geno = false;
};

PGLD_HD Hap make_hap(float c1, float c2, float c3, float c4) {
  const fast::Pop p = fast::make(c1, c2, c3, c4);
  Hap h;
  h.z = make_size(p.ns);
  h.c1 = c1; h.c2 = c2; h.c3 = c3; h.c4 = c4;
  h.x = p.x;
  h.dA = p.dA;
  h.dB = p.dB;
  h.w = p.dA * p.dB + p.e;
  h.pA = p.pA; h.qA = p.qA; h.pB = p.pB; h.qB = p.qB;
  h.hA = p.pA * p.qA;
  h.hB = p.pB * p.qB;
  h.yb = p.pA * c4 + c2 * p.qA;
  h.yB = p.pA * c3 + c1 * p.qA;
  const fast::X2 d = fast::dd_split(p);
  h.dd = d.s;
  h.ddr = d.e;
  h.dz = fast::dz_num(p);
  h.pi = fast::pi2_pairs(p, h.hA, h.hB);
  return h;
}

PGLD_HD float dz31(const Hap& t, const Hap& s) { return t.x * (t.dA * s.dB + t.dB * s.dA); }
// heterozygosity of one draw each from a and b at the first / second SNP
PGLD_HD float mixA(const Hap& a, const Hap& b) { return a.pA * b.qA + a.qA * b.pA; }
PGLD_HD float mixB(const Hap& a, const Hap& b) { return a.pB * b.qB + a.qB * b.pB; }
// twice mixB, from what ijij needs of the pair
PGLD_HD float mix2(const Hap& a, const Hap& b) { return a.z.n * b.z.n - a.dB * b.dB; }
// sixteen times the draws: Y Y' + m m' (n n' - dA dA' - dB dB')
PGLD_HD float ijij(const Hap& i, const Hap& j) {
  return fast::dot2(i.z.m * j.z.m, mix2(i, j) - i.dA * j.dA, i.w, j.w);
}
// the four terms of pi2_ttts are equal
PGLD_HD float triple(const Hap& t, const Hap& s, Den d, bool) {
  return quot(fmaf(t.hA, 0.5f * mix2(t, s), -fmaf(t.yb, s.pB, fast::fmul(t.yB, s.qB))), d);
}
PGLD_HD float dz211(const Hap& s, const Hap& a, const Hap& b) {
  return s.x * (a.dA * b.dB + b.dA * a.dB);
}
// s and a at the first SNP, s and b at the second
PGLD_HD float shared(const Hap& s, const Hap& a, const Hap& b) {
  const float y1 = s.c1 * b.qB + s.c2 * b.pB, y2 = s.c3 * b.qB + s.c4 * b.pB;
  return fmaf(mixA(s, a), mixB(s, b), -fmaf(a.qA, y1, fast::fmul(a.pA, y2)));
}

// ---- genotypes -------------------------------------------------------------
// over the centred moments m[3 x + y] = sum c_I^x c_J^y (pgld_geno_mom.cuh);
// P2 = n + m3 = 2 pA and so on
struct Geno {
  Size z;
  float m1, m3;
  float y, w;               // n m4 - m1 m3 = D16 / 4, m1 m3 - m4
  float P2, R2, Q2, S2, hA, hB;
  float J1, J2, J3, J4;     // a quarter of sum (1 +- c_I)(1 +- c_J): ++, +-, -+, --
  float EA1, EA2, EB1, EB2; // half the draws hA one of which has also 1 +- c_J; exchanged
  float u, v;               // n m7 - m1 m6, n m5 - m3 m2: a third draw's corrections
  float dd, dz, pi;         // numerators over 4, 2 and 16 d4
  static constexpr bool geno = true;
};

// integer of magnitude below 2^22 to float32 without the conversion pipe
PGLD_HD float small_f(int v) {
#ifdef __CUDA_ARCH__
  return __int_as_float(0x4B400000 + v) - 12582912.0f;
#else
  return (float)v;
#endif
}
PGLD_HD float num_f(long long v) {
#ifdef __CUDA_ARCH__
  return pgld::ll2f(v);
#else
  return (float)v;
#endif
}

PGLD_HD Geno make_geno(const gmom::Mom& o) {
  Geno g;
  const float n = small_f(o.m[0]), m1 = small_f(o.m[1]), m2 = small_f(o.m[2]),
              m3 = small_f(o.m[3]), m4 = small_f(o.m[4]), m5 = small_f(o.m[5]),
              m6 = small_f(o.m[6]), m7 = small_f(o.m[7]);
  g.z = make_size(n);
  g.m1 = m1;
  g.m3 = m3;
  const float m13 = m1 * m3;
  g.y = n * m4 - m13;
  g.w = m13 - m4;
  g.P2 = n + m3; g.R2 = n - m3; g.Q2 = n + m1; g.S2 = n - m1;
  g.hA = g.P2 * g.R2 - (n - m6);
  g.hB = g.Q2 * g.S2 - (n - m2);
  const float s1 = 0.25f * (n + m4), s2 = 0.25f * (n - m4), t1 = 0.25f * (m3 + m1), t2 = 0.25f * (m3 - m1);
  g.J1 = s1 + t1; g.J2 = s2 + t2; g.J3 = s2 - t2; g.J4 = s1 - t1;
  const float eA = g.z.m * m1 - m3 * m4 + m7, eB = g.z.m * m3 - m1 * m4 + m5;
  g.EA1 = g.hA + eA;
  g.EA2 = g.hA - eA;
  g.EB1 = g.hB + eB;
  g.EB2 = g.hB - eB;
  g.u = n * m7 - m1 * m6;
  g.v = n * m5 - m3 * m2;
  // one population: the polynomials cancel heavily, so in 64-bit integers
  const gmom::Terms t = gmom::terms(o);
  g.dd = num_f(gmom::dd_num(o, t));
  g.dz = num_f(gmom::dz_num(o, t));
  g.pi = num_f(gmom::pi2_num(o, t));
  return g;
}

PGLD_HD float mixA(const Geno& a, const Geno& b) { return a.z.n * b.z.n - a.m3 * b.m3; }
PGLD_HD float mixB(const Geno& a, const Geno& b) { return a.z.n * b.z.n - a.m1 * b.m1; }
// a quarter of the draws: w w' + m m' (n n' - m3 m3' - m1 m1')
PGLD_HD float ijij(const Geno& i, const Geno& j) {
  const float g = i.z.n * j.z.n - i.m3 * j.m3 - i.m1 * j.m1;
  return fast::dot2(i.z.m * j.z.m, g, i.w, j.w);
}
// y (m3 m1' + m1 m3') - (u m1' + v m3'): the two corrections are summed exactly
// (TwoProduct, TwoSum; Ogita, Rump and Oishi, "Accurate sum and dot product",
// SIAM J. Sci. Comput. 26, 2005), since all three may cancel where D is small
PGLD_HD float dz31(const Geno& t, const Geno& s) {
  const float p = fast::fmul(t.u, s.m1), pe = fmaf(t.u, s.m1, -p);
  const float q = fast::fmul(t.v, s.m3), qe = fmaf(t.v, s.m3, -q);
  const float h = fast::fadd(p, q), b = fast::fsub(h, p);
  const float l = fast::fadd(fast::fadd(fast::fsub(p, fast::fsub(h, b)), fast::fsub(q, b)),
                             fast::fadd(pe, qe));
  return fast::fsub(fmaf(t.y, t.m3 * s.m1 + t.m1 * s.m3, -h), l);
}
// half the draws with t twice at the first SNP, and twice at the second
PGLD_HD float triple(const Geno& t, const Geno& s, Den d, bool first) {
  const float a = quot(fmaf(t.hA, mixB(t, s), -fmaf(t.EA1, s.S2, fast::fmul(t.EA2, s.Q2))), d);
  const float b = quot(fmaf(t.hB, mixA(t, s), -fmaf(t.EB1, s.R2, fast::fmul(t.EB2, s.P2))), d);
  return first ? two_two(a, b) : two_two(b, a);
}
PGLD_HD float dz211(const Geno& s, const Geno& a, const Geno& b) {
  return s.y * (a.m3 * b.m1 + b.m3 * a.m1);
}
// a quarter of the draws
PGLD_HD float shared(const Geno& s, const Geno& a, const Geno& b) {
  return fmaf(mixA(s, a), mixB(s, b),
              -fmaf(a.R2, fmaf(s.J1, b.S2, fast::fmul(s.J2, b.Q2)),
                    fast::fmul(a.P2, fmaf(s.J3, b.S2, fast::fmul(s.J4, b.Q2)))));
}

// denominator M a b of a class
template <class F, int M>
PGLD_HD Den class_den(float a, float b) {
  return make_den(F::geno ? a * b : round_den<M>(a, b));
}

PGLD_HD float dd_quot(const Hap& h, Den d) { return quot(h.dd, h.ddr, d); }
PGLD_HD float dd_quot(const Geno& g, Den d) { return quot(g.dd, d); }
// D of one population (x of the haplotype, y of the genotype features)
PGLD_HD float dval(const Hap& h) { return h.x; }
PGLD_HD float dval(const Geno& g) { return g.y; }

// ---- the statistics in class order -----------------------------------------
// sink(k, value) for k = 0 .. group_size(P, 0) - 1 (G0), then on (G1); the
// values still lack the power-of-two factors of order()
template <int P, bool G0, bool G1, class F, class Sink>
PGLD_HD void eval(const F (&f)[P], Sink&& sink) {
  int k = 0;
  if (G0) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const Den d = class_den<F, 1>(f[i].z.m2, f[i].z.m2b);
      sink(k++, dd_quot(f[i], d));
      sink(k++, quot(f[i].dz, d));
      sink(k++, quot(f[i].pi, d));
    }
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int j = i + 1; j < P; ++j) {
        const Den d = class_den<F, 1>(f[i].z.m2, f[j].z.m2);
        const Den d4 = class_den<F, 4>(f[i].z.m2, f[j].z.m2);
        sink(k++, quot(dval(f[i]) * dval(f[j]), d));
        sink(k++, quot(dval(f[i]) * f[j].w, d));
        sink(k++, quot(dval(f[j]) * f[i].w, d));
        sink(k++, quot(fast::fmul(f[i].hA, f[j].hB), d) + quot(fast::fmul(f[j].hA, f[i].hB), d));
        sink(k++, quot(ijij(f[i], f[j]), d4));
      }
#pragma unroll
    for (int i = 0; i < P; ++i)
#pragma unroll
      for (int j = 0; j < P; ++j)
        if (j != i) {
          const Den d = class_den<F, 2>(f[i].z.m2, f[i].z.k * f[j].z.n);
          sink(k++, quot(dz31(f[i], f[j]), d));
          sink(k++, triple(f[i], f[j], d, i < j));
        }
  }
  if (G1) {
#pragma unroll
    for (int s = 0; s < P; ++s)
#pragma unroll
      for (int a = 0; a < P; ++a)
#pragma unroll
        for (int b = a + 1; b < P; ++b)
          if (a != s && b != s) {
            const Den d = class_den<F, 2>(f[s].z.m2, f[a].z.n * f[b].z.n);
            const Den d4 = class_den<F, 4>(f[s].z.m2, f[a].z.n * f[b].z.n);
            sink(k++, quot(dz211(f[s], f[a], f[b]), d));
            // the table lists the pair with the smaller population first
            const float sA = quot(fast::fmul(f[s].hA, mixB(f[a], f[b])), d);
            const float sB = quot(fast::fmul(f[s].hB, mixA(f[a], f[b])), d);
            sink(k++, s < a ? two_two(sA, sB) : two_two(sB, sA));
            sink(k++, four_four(quot(shared(f[s], f[a], f[b]), d4), quot(shared(f[s], f[b], f[a]), d4)));
          }
    if (P == 4) {
      const Den d = class_den<F, 4>(f[0].z.n * f[1].z.n, f[P - 2].z.n * f[P - 1].z.n);
#pragma unroll
      for (int b = 1; b < 4; ++b) {
        const int c = b == 1 ? 2 : 1, e = b == 3 ? 2 : 3;  // the other two
        const F &f0 = f[0], &f1 = f[b % P], &f2 = f[c % P], &f3 = f[e % P];
        sink(k++, four_four(quot(fast::fmul(mixA(f0, f1), mixB(f2, f3)), d),
                            quot(fast::fmul(mixA(f2, f3), mixB(f0, f1)), d)));
      }
    }
  }
}

// where eval()'s k-th value belongs: statistic in moments' order (names DD_i_j,
// Dz_i_j_k, pi2_i_j_k_l, ld_pipeline.py:357-376) and its power-of-two factor
struct Place {
  int stat;
  float factor;
};

inline std::vector<Place> order(int P, bool geno) {
  auto dd = [&](int i, int j) {
    int s = 0;
    for (int a = 0; a < P; ++a)
      for (int b = a; b < P; ++b, ++s)
        if (a == i && b == j) return s;
    return -1;
  };
  auto dz = [&](int i, int j, int k) {
    if (j > k) std::swap(j, k);
    int s = P * (P + 1) / 2;
    for (int a = 0; a < P; ++a)
      for (int b = 0; b < P; ++b)
        for (int c = b; c < P; ++c, ++s)
          if (a == i && b == j && c == k) return s;
    return -1;
  };
  // pi2 of the locus pairs {i, j} and {k, l}, in whichever order the table has
  auto pi2 = [&](int i, int j, int k, int l) {
    if (i > j) std::swap(i, j);
    if (k > l) std::swap(k, l);
    int s = P * (P + 1) / 2 + P * P * (P + 1) / 2;
    for (int a = 0; a < P; ++a)
      for (int b = a; b < P; ++b)
        for (int c = a; c < P; ++c)
          for (int d = c; d < P; ++d) {
            if (c == a && a == d && b != a) continue;
            if (a == c && d < b) continue;
            if ((a == i && b == j && c == k && d == l) || (a == k && b == l && c == i && d == j))
              return s;
            ++s;
          }
    return -1;
  };
  std::vector<Place> o;
  for (int i = 0; i < P; ++i) {
    o.push_back({dd(i, i), geno ? 0.25f : 1.0f});
    o.push_back({dz(i, i, i), geno ? 0.5f : 1.0f});
    o.push_back({pi2(i, i, i, i), geno ? 0.0625f : 1.0f});
  }
  for (int i = 0; i < P; ++i)
    for (int j = i + 1; j < P; ++j) {
      o.push_back({dd(i, j), geno ? 0.25f : 1.0f});
      o.push_back({dz(i, j, j), geno ? 0.5f : 1.0f});
      o.push_back({dz(j, i, i), geno ? 0.5f : 1.0f});
      o.push_back({pi2(i, i, j, j), geno ? 1.0f / 32 : 0.5f});
      o.push_back({pi2(i, j, i, j), 1.0f / 16});
    }
  for (int i = 0; i < P; ++i)
    for (int j = 0; j < P; ++j)
      if (j != i) {
        o.push_back({dz(i, i, j), geno ? 0.25f : 0.5f});
        o.push_back({pi2(i, i, i, j), geno ? 1.0f / 32 : 0.5f});
      }
  for (int s = 0; s < P; ++s)
    for (int a = 0; a < P; ++a)
      for (int b = a + 1; b < P; ++b)
        if (a != s && b != s) {
          o.push_back({dz(s, a, b), geno ? 0.25f : 0.5f});
          o.push_back({pi2(s, s, a, b), geno ? 1.0f / 32 : 0.25f});
          o.push_back({pi2(s, a, s, b), geno ? 1.0f / 32 : 0.125f});
        }
  if (P == 4)
    for (int b = 1; b < 4; ++b) {
      const int c = b == 1 ? 2 : 1, e = b == 3 ? 2 : 3;
      o.push_back({pi2(0, b, c, e), geno ? 1.0f / 32 : 0.125f});
    }
  return o;
}

}  // namespace multi
}  // namespace pgld
