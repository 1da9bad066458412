// Device side of the multi-population binned sums shared by the haplotype and
// genotype kernels: the tile's pairs ordered by distance bin, and the warp
// totals of many statistics.
#pragma once
#include "pgld_band.cuh"
#include "pgld_multi.cuh"

namespace pgld {
namespace multi {

// moments' statistic and power-of-two factor of eval()'s values, by kernel argument
struct Places {
  unsigned char stat[105];
  float factor[105];
};
inline Places places(int P, bool geno) {
  Places p{};
  const std::vector<Place> o = order(P, geno);
  for (size_t k = 0; k < o.size(); ++k) {
    p.stat[k] = (unsigned char)o[k].stat;
    p.factor[k] = o[k].factor;
  }
  return p;
}

// Warp totals of N values by recursive halving: a step exchanges half of the
// values that a lane still holds with its partner, so N values take about N
// shuffles (5 N for N butterflies).  Lane l ends with values halved(N, l, k),
// each v[k] + e[k]: every step keeps its rounding errors (TwoSum), so that a
// total carries those of a lane's own run only and a short distance bin with
// few pairs is summed as closely as a long one (10,000 SNPs, 14 bins: 3e-10 of
// the bin closer than with the last three steps' errors alone, for 3% of the
// time of three populations).
template <int N, int O = 16>
__device__ __forceinline__ void halve(float* v, float* e) {
  constexpr int H = (N + 1) / 2;
  const bool up = (threadIdx.x & O) != 0;
#pragma unroll
  for (int k = 0; k < H; ++k) {
    const float hi = k + H < N ? v[k + H] : 0.f;
    const float give = up ? v[k] : hi, keep = up ? hi : v[k];
    const float got = __shfl_xor_sync(0xffffffffu, give, O);
    const float sum = __fadd_rn(keep, got);
    const float b = __fsub_rn(sum, keep);
    float err = __fadd_rn(__fsub_rn(keep, __fsub_rn(sum, b)), __fsub_rn(got, b));
    if constexpr (O < 16) {
      const float ehi = k + H < N ? e[k + H] : 0.f;
      err += (up ? ehi : e[k]) + __shfl_xor_sync(0xffffffffu, up ? e[k] : ehi, O);
    }
    e[k] = err;
    v[k] = sum;
  }
  if constexpr (O > 1) halve<H, O / 2>(v, e);
}
// the same without the errors: each total is the butterfly's
template <int N, int O = 16>
__device__ __forceinline__ void halve_plain(float* v) {
  constexpr int H = (N + 1) / 2;
  const bool up = (threadIdx.x & O) != 0;
#pragma unroll
  for (int k = 0; k < H; ++k) {
    const float hi = k + H < N ? v[k + H] : 0.f;
    v[k] = __fadd_rn(up ? hi : v[k], __shfl_xor_sync(0xffffffffu, up ? v[k] : hi, O));
  }
  if constexpr (O > 1) halve_plain<H, O / 2>(v);
}
template <int N, int O = 16>
__device__ __forceinline__ constexpr int halved_len() {
  if constexpr (O == 0)
    return N;
  else
    return halved_len<(N + 1) / 2, O / 2>();
}
// index of the k-th value that this lane ends with, -1 for padding
template <int N, int O = 16>
__device__ __forceinline__ int halved(int k) {
  if constexpr (O == 0) {
    return k;
  } else {
    constexpr int H = (N + 1) / 2;
    const int sub = halved<H, O / 2>(k);
    const int at = sub + ((threadIdx.x & O) ? H : 0);
    return sub < 0 || at >= N ? -1 : at;
  }
}

// adds the warp's totals of values K0 .. K0 + N - 1 to the bin's float64 slots
template <int N, int K0>
__device__ __forceinline__ void flush(float* acc, double* slots, const Places& pl) {
  float err[(N + 1) / 2];
  halve<N>(acc, err);
#pragma unroll
  for (int k = 0; k < halved_len<N>(); ++k) {
    const int at = halved<N>(k);
    if (at >= 0)
      atomicAdd(slots + pl.stat[K0 + at],
                (double)(acc[k] * pl.factor[K0 + at]) + (double)(err[k] * pl.factor[K0 + at]));
  }
}

// The pairs of a tile (32 to a row) grouped by bin, in steps of 32 pairs of one bin
// (the last of a bin padded): a step's totals then go to one bin however the
// tile's distances fall, so short distances with several bins across a row
// cost no more than long ones.  The order is fixed (bin, then warp, then row,
// then column): equal inputs give equal sums.
constexpr int kGroupPairs = 1024;
template <int WARPS, int PAIRS = kGroupPairs>
struct Groups {
  unsigned short list[PAIRS + 31 * kMaxBins];  // pair = 32 row + column; 0xffff: none
  unsigned char step_bin[PAIRS / 32 + kMaxBins];
  unsigned short warp_cnt[WARPS][kMaxBins];
  int n_steps;
};

// bin[q]: bin (or -1) of the thread's pair (row0 + q, lane).  All WARPS warps
// call it together (sync() meets them); fills g and adds the pairs per bin to bcnt.
template <int WARPS, int ROWS, int PAIRS, class Sync>
__device__ __forceinline__ void group_pairs(Groups<WARPS, PAIRS>& g, const int (&bin)[ROWS], int row0,
                                            int warp, int n_bins, unsigned long long* bcnt,
                                            Sync&& sync) {
  const int lane = threadIdx.x & 31;
  for (int b = lane; b < n_bins; b += 32) g.warp_cnt[warp][b] = 0;
  __syncwarp();
  int rank[ROWS];
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
    const unsigned same = __match_any_sync(0xffffffffu, bin[q]);
    rank[q] = __popc(same & ((1u << lane) - 1u));
    if (bin[q] >= 0) rank[q] += g.warp_cnt[warp][bin[q]];
    __syncwarp();
    if (bin[q] >= 0 && lane == __ffs(same) - 1)
      g.warp_cnt[warp][bin[q]] += (unsigned short)__popc(same);
    __syncwarp();
  }
  sync();
  // one warp: padded starts of the bins, and each warp's start within its bin
  if (warp == 0) {
    int carry = 0;
    for (int b0 = 0; b0 < n_bins; b0 += 32) {
      const int b = b0 + lane;
      int tot = 0;
      if (b < n_bins)
#pragma unroll
        for (int w = 0; w < WARPS; ++w) tot += g.warp_cnt[w][b];
      const int steps = (tot + 31) >> 5;
      int incl = steps;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const int first = carry + incl - steps;
      if (tot) {
        atomicAdd(bcnt + b, (unsigned long long)tot);
        int at = 32 * first;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
          const int c = g.warp_cnt[w][b];
          g.warp_cnt[w][b] = (unsigned short)at;
          at += c;
        }
        for (; at < 32 * (first + steps); ++at) g.list[at] = 0xffff;
        for (int s = 0; s < steps; ++s) g.step_bin[first + s] = (unsigned char)b;
      }
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) g.n_steps = carry;
  }
  sync();
#pragma unroll
  for (int q = 0; q < ROWS; ++q)
    if (bin[q] >= 0)
      g.list[g.warp_cnt[warp][bin[q]] + rank[q]] = (unsigned short)((row0 + q) * 32 + lane);
  sync();
}

// The steps [s0, s1) of a grouped tile: each run of steps of one bin summed in
// registers, its totals added to the bin's slots.  load(pair, b, f) sets the
// features of the lane's pair of bin b (pair 0xffff: of nobody, whose quotients
// are 0).  Up to three populations take one pass (G = 0); four take two, G = 0
// with 66 statistics and G = 1 with 39, so that the sums stay in registers.
template <int P, int G, class F, int WARPS, int PAIRS, class Load>
__device__ __forceinline__ void sum_steps(const Groups<WARPS, PAIRS>& g, int s0, int s1, double* slots,
                                          int n_stats, const Places& pl, Load&& load) {
  constexpr bool G0 = P < 4 || G == 0, G1 = P < 4 || G == 1;
  constexpr int N = (G0 ? group_size(P, 0) : 0) + (G1 ? group_size(P, 1) : 0);
  constexpr int K0 = G0 ? 0 : group_size(P, 0);
  const int lane = threadIdx.x & 31;
  // a lane's haplotype sums of pi2_iiii keep their rounding errors (TwoSum): with
  // few haplotypes those sums add a few recurring values, whose roundings do not
  // average out (30 haplotypes: 2e-9 of the statistic after eight steps)
  constexpr bool kKeep = G0 && !F::geno;
  constexpr int E = kKeep ? P : 1;
  float acc[N], err[E];
  for (int s = s0; s < s1;) {
    const int b = g.step_bin[s];
#pragma unroll
    for (int k = 0; k < N; ++k) acc[k] = 0.f;
#pragma unroll
    for (int k = 0; k < E; ++k) err[k] = 0.f;
    for (; s < s1 && g.step_bin[s] == b; ++s) {
      F f[P];
      load((int)g.list[32 * s + lane], b, f);
      eval<P, G0, G1>(f, [&](int k, float v) {
        if (kKeep && k < 3 * P && k % 3 == 2) {
          const float t = __fadd_rn(acc[k], v), z = __fsub_rn(t, acc[k]);
          err[k / 3] += __fadd_rn(__fsub_rn(acc[k], __fsub_rn(t, z)), __fsub_rn(v, z));
          acc[k] = t;
        } else {
          acc[k] += v;
        }
      });
    }
    if (kKeep) {
#pragma unroll
      for (int k = 0; k < E; ++k) acc[3 * k + 2] += err[k];
    }
    flush<N, K0>(acc, slots + b * n_stats, pl);
  }
}

}  // namespace multi
}  // namespace pgld
