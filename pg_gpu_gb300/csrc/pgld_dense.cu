// Dense all-pairs LD of one population (the M x M outputs of
// HaplotypeMatrix.pairwise_LD_v / pairwise_r2, haplotype_matrix.py:1092-1170)
// and the distance-binned r^2 percentiles of windowed_r_squared
// (haplotype_matrix.py:1235-1317) without moving the pair values to the host:
// the valid pairs' r^2 are grouped by distance bin on the device and the
// requested order statistics are found by radix selection.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "pgld_band.cuh"
#include "pgld_internal.cuh"

using pgld::i64;

int pgld_tc_int_positions(pgld_context* h, const double* pos, long long n, int* ipos, int* bad,
                          cudaStream_t st);

namespace pgld {
namespace dense {

constexpr int kT = 32;         // SNPs per tile side
constexpr int kThreads = 256;  // warp w: rows w + 8 q of the tile, lane: column
constexpr int kKW = 32;        // words of a plane staged per chunk
constexpr int kPad = 33;
constexpr int kPadRows = 36;   // 16-byte aligned rows

struct __align__(16) Smem {
  uint32_t ci[kKW][kPadRows], vi[kKW][kPadRows], cj[kKW][kPad], vj[kKW][kPad];
  double tr[kT][kT + 1];   // mirrored tile
  double bins[kMaxBins + 1];
  int thr[kMaxBins + 1];
  int bin_cnt[kMaxBins];
  long long bin_base[kMaxBins];
};

// upper-triangle tile t -> (bi, bj), bj >= bi, of nb blocks (row bi owns
// tiles bi .. nb - 1, starting at bi nb - bi (bi - 1) / 2)
__device__ __forceinline__ void tri_decode(i64 t, i64 nb, i64& bi, i64& bj) {
  // largest bi with start(bi) <= t, from the quadratic, then corrected (in
  // float32: a float64 root by every thread of a block takes 5,000 cycles)
  const i64 b = 2 * nb + 1;
  const float disc = (float)(b * b - 8 * t);
  i64 r = (i64)(0.5f * ((float)b - sqrtf(disc > 0.f ? disc : 0.f)));
  r = max((i64)0, min(r, nb - 1));
  auto start = [&](i64 x) { return x * nb - x * (x - 1) / 2; };
  while (r > 0 && start(r) > t) --r;
  while (r + 1 < nb && start(r + 1) <= t) ++r;
  bi = r;
  bj = r + (t - start(r));
}

// carrier and valid (carrier | reference) words [w0, w0 + 32) of the tile's rows
// and columns, transposed; L = 1 << lsh lanes (at least the words there are) to a
// SNP.  Row r is kept at 4 (r % 8) + r / 8: the four rows of a warp are one 16-byte
// load
__device__ __forceinline__ void stage(Smem& sm, const uint32_t* __restrict__ planes, int W, i64 i0,
                                      i64 j0, i64 n, int w0, int lsh) {
  const int w = threadIdx.x & ((1 << lsh) - 1);
  for (int x = threadIdx.x; x < (2 * kT) << lsh; x += kThreads) {
    const int row = x >> lsh, r = row & (kT - 1);
    const bool col = row >= kT;
    const i64 s = (col ? j0 : i0) + r;
    uint32_t cc = 0, zz = 0;
    if (s < n && w0 + w < W) {
      const uint32_t* p = planes + s * 2 * W + w0 + w;
      cc = __ldg(p);
      zz = __ldg(p + W);
    }
    if (col) {
      sm.cj[w][r] = cc;
      sm.vj[w][r] = cc | zz;
    } else {
      const int k = 4 * (r & 7) + (r >> 3);
      sm.ci[w][k] = cc;
      sm.vi[w][k] = cc | zz;
    }
  }
}

// joint counts of the tile's pairs (i0 + wid + 8 q, j0 + lane): C_i.C_j
// (n11), C_i.V_j (pA), V_i.C_j (pB) and V_i.V_j (the pairwise-valid n)
__device__ __forceinline__ void tile_counts(Smem& sm, const uint32_t* planes, int W, i64 n, i64 i0,
                                            i64 j0, int (&cc)[4], int (&cv)[4], int (&vc)[4],
                                            int (&vv)[4]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) cc[q] = cv[q] = vc[q] = vv[q] = 0;
  for (int w0 = 0; w0 < W; w0 += kKW) {
    __syncthreads();
    stage(sm, planes, W, i0, j0, n, w0, W <= 8 ? 3 : W <= 16 ? 4 : 5);
    __syncthreads();
    const int nw = min(kKW, W - w0);
    for (int w = 0; w < nw; ++w) {
      const uint32_t cj = sm.cj[w][lane], vj = sm.vj[w][lane];
      const uint4 c4 = *reinterpret_cast<const uint4*>(&sm.ci[w][4 * wid]);
      const uint4 v4 = *reinterpret_cast<const uint4*>(&sm.vi[w][4 * wid]);
      const uint32_t ci[4] = {c4.x, c4.y, c4.z, c4.w}, vi[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        cc[q] += __popc(ci[q] & cj);
        cv[q] += __popc(ci[q] & vj);
        vc[q] += __popc(vi[q] & cj);
        vv[q] += __popc(vi[q] & vj);
      }
    }
  }
}

__global__ void site_freq_kernel(const uint32_t* __restrict__ planes, int W, i64 n,
                                 double* __restrict__ p) {
  for (i64 s = (i64)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (i64)gridDim.x * blockDim.x) {
    int car = 0, val = 0;
    for (int w = 0; w < W; ++w) {
      const uint32_t c = planes[s * 2 * W + w], z = planes[s * 2 * W + W + w];
      car += __popc(c);
      val += __popc(c | z);
    }
    // p = sum / n_valid where n_valid > 0 (haplotype_matrix.py:1122)
    p[s] = val > 0 ? __ddiv_rn((double)car, (double)val) : 0.0;
  }
}

// D = pAB - p_i p_j and r^2 = D^2 / (p_i (1 - p_i) p_j (1 - p_j)) of every
// pair, rounded operation by operation as the reference's float64 matrix
// expressions (haplotype_matrix.py:1125-1128, 1165-1169), zero diagonal
__global__ void __launch_bounds__(kThreads) pairwise_ld_kernel(const uint32_t* __restrict__ planes,
                                                               int W, i64 n,
                                                               const double* __restrict__ p,
                                                               double* __restrict__ D_out,
                                                               double* __restrict__ r2_out, i64 ld) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const i64 nb = (n + kT - 1) / kT;
  const i64 n_tiles = nb * (nb + 1) / 2;
  for (i64 t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    i64 bi, bj;
    tri_decode(t, nb, bi, bj);
    const i64 i0 = bi * kT, j0 = bj * kT;
    int n11[4], cv[4], vc[4], nv[4];
    tile_counts(sm, planes, W, n, i0, j0, n11, cv, vc, nv);
    for (int out = 0; out < 2; ++out) {
      double* M = out == 0 ? D_out : r2_out;
      if (!M) continue;
      double val[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const i64 i = i0 + wid + 8 * q, j = j0 + lane;
        double v = 0.0;
        if (i < n && j < n && i != j) {
          const double pi = p[i], pj = p[j];
          const double pab = nv[q] > 0 ? __ddiv_rn((double)n11[q], (double)nv[q]) : 0.0;
          const double d = __dsub_rn(pab, __dmul_rn(pi, pj));
          if (out == 0) {
            v = d;
          } else {
            const double den = __dmul_rn(__dmul_rn(pi, __dsub_rn(1.0, pi)),
                                         __dmul_rn(pj, __dsub_rn(1.0, pj)));
            v = den > 0.0 ? __ddiv_rn(__dmul_rn(d, d), den) : 0.0;
          }
        }
        val[q] = v;
        if (i < n && j < n) M[i * ld + j] = v;
      }
      if (bj != bi) {
        // the mirrored block (j, i), written row by row through shared memory
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) sm.tr[lane][wid + 8 * q] = val[q];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const i64 j = j0 + wid + 8 * q, i = i0 + lane;
          if (i < n && j < n) M[j * ld + i] = sm.tr[wid + 8 * q][lane];
        }
      }
    }
  }
}

__device__ __forceinline__ int bin_index(const double* sb, int n_bins, double d) {
  // digitize(d, bins) - 1 with right-open bins; -1 outside [bins[0], bins[n_bins])
  if (!(d >= sb[0]) || !(d < sb[n_bins])) return -1;
  int lo = 0, hi = n_bins;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (sb[mid] <= d) lo = mid; else hi = mid;
  }
  return lo;
}

// smallest integer distance of each bin edge
__device__ __forceinline__ int int_edge(double b) {
  const double c = ceil(b);
  return c > 2147483647.0 ? 2147483647 : (c < -2147483647.0 ? -2147483647 : (int)c);
}
__device__ __forceinline__ int bin_index(const int* thr, int n_bins, int d) {
  if (d < thr[0] || d >= thr[n_bins]) return -1;
  int lo = 0, hi = n_bins;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (thr[mid] <= d) lo = mid; else hi = mid;
  }
  return lo;
}

// every pair i < j: its value (r^2 from the joint counts, or values[k] of the
// condensed upper triangle), NaN skipped, binned by pos[j] - pos[i].
// counts mode (out == NULL): bin_counts[b] += pairs; fill mode: the values
// are written grouped by bin at cursor[b] (advanced atomically per tile).
// The float64 pipe (two operations per SM and clock) would bound it: integer
// positions are compared as integers, counting asks only whether the
// denominator is positive, the quotient is an integer division, and a warp's pairs
// of a bin take their places with one shared-memory addition.  300 haplotypes x
// 5,001 SNPs, both passes: 1.0 ms when they divided and searched the bins in
// float64, 0.62 with a float64 root per thread to find a tile, an addition per
// pair and 32 lanes to a staged SNP, 0.42 now.
__global__ void __launch_bounds__(kThreads) pairs_by_bin_kernel(
    const uint32_t* __restrict__ planes, int W, const double* __restrict__ values, i64 n,
    const double* __restrict__ pos, const int* __restrict__ ipos, const int* __restrict__ ipos_bad,
    const double* __restrict__ bins, int n_bins,
    unsigned long long* __restrict__ bin_counts, unsigned long long* __restrict__ cursor,
    const unsigned long long* __restrict__ bin_end, double* __restrict__ out,
    int32_t* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int x = threadIdx.x; x <= n_bins; x += kThreads) {
    sm.bins[x] = bins[x];
    sm.thr[x] = int_edge(bins[x]);
  }
  const bool use_int = *ipos_bad == 0;
  const i64 nb = (n + kT - 1) / kT;
  const i64 n_tiles = nb * (nb + 1) / 2;
  for (i64 t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    i64 bi, bj;
    tri_decode(t, nb, bi, bj);
    const i64 i0 = bi * kT, j0 = bj * kT;
    int n11[4] = {0, 0, 0, 0}, cv[4] = {0, 0, 0, 0}, vc[4] = {0, 0, 0, 0}, nv[4] = {0, 0, 0, 0};
    if (!values) {
      tile_counts(sm, planes, W, n, i0, j0, n11, cv, vc, nv);
    } else {
      __syncthreads();
    }
    for (int x = threadIdx.x; x < n_bins; x += kThreads) sm.bin_cnt[x] = 0;
    __syncthreads();
    int bin[4], slot[4];
    double val[4];
    const i64 j = j0 + lane;
    const int pj = use_int && j < n ? ipos[j] : 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const i64 i = i0 + wid + 8 * q;
      bin[q] = -1;
      val[q] = 0.0;
      if (i < j && j < n) {
        double v = 0.0;
        bool defined;
        if (values) {
          v = values[i * (2 * n - i - 1) / 2 + (j - i - 1)];
          defined = v == v;
        } else {
          // r^2 of ld_statistics.r_squared (haplotype_kernels.py:32-42):
          // (n11 n00 - n10 n01)^2 over pA (n - pA) pB (n - pB) of the pair's
          // valid haplotypes as exact integers, divided once; NaN where the
          // denominator is 0
          const int a = n11[q], pa = cv[q], pb = vc[q], nn = nv[q];
          defined = pa > 0 && pa < nn && pb > 0 && pb < nn;
          if (out && defined) {
            const int b = pa - a, c = pb - a, d = nn - pa - pb + a;
            const long long x = (long long)a * d - (long long)b * c;
            v = quotient(x * x, ((long long)pa * (nn - pa)) * ((long long)pb * (nn - pb)));
          }
        }
        val[q] = v;
        if (defined)
          bin[q] = use_int ? bin_index(sm.thr, n_bins, pj - ipos[i])
                           : bin_index(sm.bins, n_bins, pos[j] - pos[i]);
      }
      // the warp's pairs of a bin take their places with one addition
      const unsigned same = __match_any_sync(0xffffffffu, bin[q]);
      const int first = __ffs(same) - 1;
      int at = 0;
      if (lane == first && bin[q] >= 0) at = atomicAdd(&sm.bin_cnt[bin[q]], __popc(same));
      slot[q] = __shfl_sync(0xffffffffu, at, first) + __popc(same & ((1u << lane) - 1u));
    }
    __syncthreads();
    for (int x = threadIdx.x; x < n_bins; x += kThreads) {
      const int c = sm.bin_cnt[x];
      if (!out) {
        if (c) atomicAdd(bin_counts + x, (unsigned long long)c);
      } else {
        sm.bin_base[x] = c ? (long long)atomicAdd(cursor + x, (unsigned long long)c) : 0;
      }
    }
    __syncthreads();
    if (out) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (bin[q] < 0) continue;
        const unsigned long long k = (unsigned long long)sm.bin_base[bin[q]] + (unsigned)slot[q];
        // the bin's range comes from a counting pass over the same inputs;
        // a pair beyond it (inputs changed in between) is dropped and flagged
        if (k < bin_end[bin[q]]) out[k] = val[q];
        else if (status) atomicCAS(status, 0, 4001);
      }
    }
    __syncthreads();
  }
}

// Order statistics of segments by radix selection: values are non-negative
// doubles, whose bit patterns order like the values, so six passes over the
// values fix 11, 11, 11, 11, 10 and 10 bits of every target.  A pass is one
// launch over all segments (a block: one chunk of one segment, histograms of
// the next digit in shared memory, one per distinct prefix among the segment's
// targets) and one small launch that picks the targets' digits.  60 targets in
// 12.5 million values (15 bins): 4.2 ms with one CTA per target and eight
// passes of its own, 0.17 ms here.
constexpr int kDigits = 6, kDigitBins = 2048;
constexpr int kKthChunk = 1 << 15;
constexpr int kKthGroup = 4;  // histograms per block at a time

__host__ __device__ constexpr int digit_bits(int pass) { return pass < 4 ? 11 : 10; }
__host__ __device__ constexpr int digit_shift(int pass) {
  return pass < 4 ? 53 - 11 * pass : (pass == 4 ? 10 : 0);
}

struct KthArgs {
  const double* values;
  const long long* seg_off;    // [n_seg + 1]
  const long long* chunk_off;  // [n_seg + 1] chunks of the segments before each
  const int* tgt_off;          // [n_seg + 1] targets of the segments before each
  long long* rank;             // [n_targets], rank among the values that share the prefix
  unsigned long long* prefix;  // [n_targets], the bits fixed so far
  int* rep;                    // [n_targets], first target with the same segment and prefix
  unsigned* hist;              // [n_targets][kDigitBins]
  int n_seg, n_targets;
};

__global__ void __launch_bounds__(256) kth_count_kernel(KthArgs a, int pass) {
  __shared__ unsigned hist[kKthGroup][kDigitBins];
  __shared__ int reps[kKthGroup];
  int lo = 0, hi = a.n_seg;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (a.chunk_off[mid] <= (long long)blockIdx.x) lo = mid; else hi = mid;
  }
  const long long v0 = a.seg_off[lo] + ((long long)blockIdx.x - a.chunk_off[lo]) * kKthChunk;
  const long long v1 = min(a.seg_off[lo + 1], v0 + kKthChunk);
  const int shift = digit_shift(pass), above = shift + digit_bits(pass);
  const unsigned mask = (1u << digit_bits(pass)) - 1u;
  for (int t = a.tgt_off[lo]; t < a.tgt_off[lo + 1];) {
    // the next distinct prefixes
    int n = 0;
    __syncthreads();
    for (; t < a.tgt_off[lo + 1] && n < kKthGroup; ++t)
      if (a.rep[t] == t) {
        if (threadIdx.x == 0) reps[n] = t;
        ++n;
      }
    for (int x = threadIdx.x; x < n * kDigitBins; x += 256) (&hist[0][0])[x] = 0u;
    __syncthreads();
    unsigned long long want[kKthGroup];
#pragma unroll
    for (int g = 0; g < kKthGroup; ++g)
      want[g] = g < n && pass > 0 ? a.prefix[reps[g]] >> above : 0ull;
#pragma unroll 4
    for (long long k = v0 + threadIdx.x; k < v1; k += 256) {
      const unsigned long long key = (unsigned long long)__double_as_longlong(a.values[k]);
      const unsigned d = (unsigned)(key >> shift) & mask;
      const unsigned long long top = pass > 0 ? key >> above : 0ull;
#pragma unroll
      for (int g = 0; g < kKthGroup; ++g)
        if (g < n && top == want[g]) atomicAdd(&hist[g][d], 1u);
    }
    __syncthreads();
    for (int x = threadIdx.x; x < n * kDigitBins; x += 256) {
      const unsigned c = (&hist[0][0])[x];
      if (c) atomicAdd(a.hist + (size_t)reps[x / kDigitBins] * kDigitBins + x % kDigitBins, c);
    }
  }
}

// inclusive sum over the block of one count per thread; total: the block's sum
template <int THREADS>
__device__ __forceinline__ unsigned block_scan(unsigned v, unsigned* warp_sums, unsigned& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  unsigned before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < THREADS / 32; ++w) {
    const unsigned x = warp_sums[w];
    if (w < warp) before += x;
    total += x;
  }
  __syncthreads();
  return incl + before;
}

// a block per target: the digit whose cumulative count passes the rank, eight
// digits to a thread
__global__ void __launch_bounds__(256) kth_pick_kernel(KthArgs a, int pass) {
  __shared__ unsigned warp_sums[8];
  const int t = blockIdx.x;
  const uint4* h = reinterpret_cast<const uint4*>(a.hist + (size_t)a.rep[t] * kDigitBins);
  const uint4 x = h[2 * threadIdx.x], y = h[2 * threadIdx.x + 1];
  const unsigned c[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  unsigned sum = 0, total;
#pragma unroll
  for (int k = 0; k < 8; ++k) sum += c[k];
  long long r = a.rank[t];
  r -= (long long)(block_scan<256>(sum, warp_sums, total) - sum);
  if (r >= 0 && r < (long long)sum) {  // one thread: the rank is below the total
    int k = 0;
    while (r >= (long long)c[k]) r -= (long long)c[k++];
    a.rank[t] = r;
    a.prefix[t] |= (unsigned long long)(8 * threadIdx.x + k) << digit_shift(pass);
  }
}

// Short segments: a block per target does all passes by itself, one launch
// instead of 23.  34 targets in 17 segments of 15,000 values: 104 us of the device
// and 170 us of the call in passes over the grid, 18 us and none here; 16 in 8 of
// 140,000: 164 and 140 us; 30 in 15 of 830,000: 171 and 825 us.
constexpr int kSmallSeg = 1 << 17;
constexpr int kSmallCopies = 4;
__global__ void __launch_bounds__(1024) kth_small_kernel(KthArgs a, const int* __restrict__ tseg) {
  __shared__ unsigned hist[kSmallCopies][kDigitBins];
  __shared__ unsigned warp_sums[32];
  __shared__ unsigned long long s_prefix;
  __shared__ long long s_rank;
  const int t = blockIdx.x;
  const long long v0 = a.seg_off[tseg[t]], v1 = a.seg_off[tseg[t] + 1];
  unsigned long long prefix = 0;
  long long rank = a.rank[t];
  unsigned* mine = hist[(threadIdx.x >> 5) & (kSmallCopies - 1)];
  for (int pass = 0; pass < kDigits; ++pass) {
    const int shift = digit_shift(pass), above = shift + digit_bits(pass);
    const unsigned mask = (1u << digit_bits(pass)) - 1u;
    for (int x = threadIdx.x; x < kSmallCopies * kDigitBins; x += 1024) (&hist[0][0])[x] = 0u;
    __syncthreads();
    const unsigned long long want = pass > 0 ? prefix >> above : 0ull;
#pragma unroll 8
    for (long long k = v0 + threadIdx.x; k < v1; k += 1024) {
      const unsigned long long key = (unsigned long long)__double_as_longlong(a.values[k]);
      if (pass == 0 || key >> above == want) atomicAdd(mine + ((unsigned)(key >> shift) & mask), 1u);
    }
    __syncthreads();
    unsigned c0 = 0, c1 = 0, total;
#pragma unroll
    for (int w = 0; w < kSmallCopies; ++w) {
      c0 += hist[w][2 * threadIdx.x];
      c1 += hist[w][2 * threadIdx.x + 1];
    }
    long long r = rank - (long long)(block_scan<1024>(c0 + c1, warp_sums, total) - (c0 + c1));
    if (r >= 0 && r < (long long)(c0 + c1)) {  // one thread
      const bool second = r >= (long long)c0;
      s_rank = second ? r - (long long)c0 : r;
      s_prefix = prefix | (unsigned long long)(2 * threadIdx.x + second) << shift;
    }
    __syncthreads();
    rank = s_rank;
    prefix = s_prefix;
  }
  if (threadIdx.x == 0) a.prefix[t] = prefix;
}

// the first target of the same segment with the same prefix
__global__ void kth_rep_kernel(KthArgs a, const int* __restrict__ tseg) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n_targets) return;
  int r = a.tgt_off[tseg[t]];
  while (a.prefix[r] != a.prefix[t]) ++r;
  a.rep[t] = r;
}

// ---------------------------------------------------------------------------
// all pairs of one population in upper-triangle order, 32 x 32 SNP tiles
// ---------------------------------------------------------------------------
// a chunk of 32 words of one plane of 32 SNPs, as [word][SNP]; rows of 36 words
// so that a warp's four SNPs load as one 16-byte word
constexpr int kRow = 36;
__device__ __forceinline__ void stage_words(uint32_t (*dst)[kRow], const uint32_t* __restrict__ src,
                                            i64 stride, i64 s0, i64 n, int w0, int W) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int sl = wid * 4 + q;
    const i64 s = s0 + sl;
    dst[lane][sl] = s < n && w0 + lane < W ? __ldg(src + s * stride + w0 + lane) : 0u;
  }
}
// first pair of row i of the condensed upper triangle
__device__ __forceinline__ i64 tri_row(i64 i, i64 n) { return i * (2 * n - i - 1) / 2; }

// joint counts of every pair (HaplotypeMatrix.tally_gpu_haplotypes): a warp's
// stores are 32 consecutive pairs of a row.  2,000 SNPs x 200 haplotypes (2.0
// million pairs, 32 MB): 279 us with a lane group per pair that searched the
// triangle for its SNPs, 22 us here.
template <bool VALID>
__global__ void __launch_bounds__(kThreads) tally_kernel(const uint32_t* __restrict__ planes,
                                                         const uint32_t* __restrict__ valid, int W,
                                                         i64 n, int32_t* __restrict__ counts,
                                                         bool aligned, int32_t* __restrict__ n_valid) {
  __shared__ __align__(16) uint32_t ci[kKW][kRow], zi[kKW][kRow], cj[kKW][kRow], zj[kKW][kRow];
  __shared__ __align__(16) uint32_t vi[VALID ? kKW : 1][kRow], vj[VALID ? kKW : 1][kRow];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const i64 nb = (n + kT - 1) / kT, n_tiles = nb * (nb + 1) / 2;
  for (i64 t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    i64 bi, bj;
    tri_decode(t, nb, bi, bj);
    const i64 i0 = bi * kT, j0 = bj * kT;
    int c[4][4] = {}, nv[4] = {};
    for (int w0 = 0; w0 < W; w0 += kKW) {
      __syncthreads();
      stage_words(ci, planes, 2 * W, i0, n, w0, W);
      stage_words(zi, planes + W, 2 * W, i0, n, w0, W);
      stage_words(cj, planes, 2 * W, j0, n, w0, W);
      stage_words(zj, planes + W, 2 * W, j0, n, w0, W);
      if constexpr (VALID) {
        stage_words(vi, valid, W, i0, n, w0, W);
        stage_words(vj, valid, W, j0, n, w0, W);
      }
      __syncthreads();
      const int nw = min(kKW, W - w0);
#pragma unroll 4
      for (int w = 0; w < nw; ++w) {
        const uint32_t b1 = cj[w][lane], b0 = zj[w][lane];
        const uint4 a1 = *reinterpret_cast<const uint4*>(&ci[w][wid * 4]);
        const uint4 a0 = *reinterpret_cast<const uint4*>(&zi[w][wid * 4]);
        const uint32_t x1[4] = {a1.x, a1.y, a1.z, a1.w}, x0[4] = {a0.x, a0.y, a0.z, a0.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          c[q][0] += __popc(x1[q] & b1);
          c[q][1] += __popc(x1[q] & b0);
          c[q][2] += __popc(x0[q] & b1);
          c[q][3] += __popc(x0[q] & b0);
        }
        if constexpr (VALID) {
#pragma unroll
          for (int q = 0; q < 4; ++q) nv[q] += __popc(vi[w][wid * 4 + q] & vj[w][lane]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const i64 i = i0 + wid * 4 + q, j = j0 + lane;
      if (i < j && j < n) {
        const i64 k = tri_row(i, n) + (j - i - 1);
        if (aligned) {
          reinterpret_cast<int4*>(counts)[k] = make_int4(c[q][0], c[q][1], c[q][2], c[q][3]);
        } else {
#pragma unroll
          for (int x = 0; x < 4; ++x) counts[4 * k + x] = c[q][x];
        }
        if (n_valid) n_valid[k] = VALID ? nv[q] : c[q][0] + c[q][1] + c[q][2] + c[q][3];
      }
    }
  }
}

// per-SNP dosage sum and n sum g^2 - (sum g)^2
__global__ void dosage_site_kernel(const uint32_t* __restrict__ planes, int W, i64 m, int n,
                                   int2* __restrict__ site) {
  for (i64 s = (i64)blockIdx.x * blockDim.x + threadIdx.x; s < m; s += (i64)gridDim.x * blockDim.x) {
    int one = 0, two = 0;
    for (int w = 0; w < W; ++w) {
      one += __popc(planes[s * 3 * W + W + w]);
      two += __popc(planes[s * 3 * W + 2 * W + w]);
    }
    const int g = one + 2 * two;
    site[s] = make_int2(g, n * (one + 4 * two) - g * g);
  }
}

// Rogers-Huff r of every SNP pair of n individuals without missing dosages
// (ld_statistics.py:410-443): cov = n sum g_i g_j - sum g_i sum g_j over
// sqrt(var_i var_j), the exact integers of the general form (pgld_geno.cuh),
// of which only sum g_i g_j depends on the pair: three popcounts a word, since
// the individuals with dosages (1, 2) and (2, 1) are disjoint.  The float64
// square root and division bound it (about 20 operations a pair on a pipe of
// two a clock).  1,000 individuals x 3,000 SNPs: 2.30 ms with 36-byte counts
// per pair, an index list and a kernel for the quotients, 0.21 ms here.
__global__ void __launch_bounds__(kThreads) rogers_huff_kernel(const uint32_t* __restrict__ planes,
                                                               int W, i64 m, int n,
                                                               const int2* __restrict__ site,
                                                               double* __restrict__ out) {
  __shared__ __align__(16) uint32_t i1[kKW][kRow], i2[kKW][kRow], j1[kKW][kRow], j2[kKW][kRow];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const i64 nb = (m + kT - 1) / kT, n_tiles = nb * (nb + 1) / 2;
  for (i64 t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    i64 bi, bj;
    tri_decode(t, nb, bi, bj);
    const i64 i0 = bi * kT, j0 = bj * kT;
    int s[4] = {0, 0, 0, 0};
    for (int w0 = 0; w0 < W; w0 += kKW) {
      __syncthreads();
      stage_words(i1, planes + W, 3 * W, i0, m, w0, W);
      stage_words(i2, planes + 2 * W, 3 * W, i0, m, w0, W);
      stage_words(j1, planes + W, 3 * W, j0, m, w0, W);
      stage_words(j2, planes + 2 * W, 3 * W, j0, m, w0, W);
      __syncthreads();
      const int nw = min(kKW, W - w0);
#pragma unroll 4
      for (int w = 0; w < nw; ++w) {
        const uint32_t b1 = j1[w][lane], b2 = j2[w][lane];
        const uint4 a1 = *reinterpret_cast<const uint4*>(&i1[w][wid * 4]);
        const uint4 a2 = *reinterpret_cast<const uint4*>(&i2[w][wid * 4]);
        const uint32_t x1[4] = {a1.x, a1.y, a1.z, a1.w}, x2[4] = {a2.x, a2.y, a2.z, a2.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
          s[q] += __popc(x1[q] & b1) + 2 * __popc((x1[q] & b2) | (x2[q] & b1)) +
                  4 * __popc(x2[q] & b2);
      }
    }
    const i64 j = j0 + lane;
    const int2 sj = j < m ? site[j] : make_int2(0, 0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const i64 i = i0 + wid * 4 + q;
      if (i < j && j < m) {
        const int2 si = site[i];
        const int cov = n * s[q] - si.x * sj.x;
        const i64 den = (i64)si.y * sj.y;
        out[tri_row(i, m) + (j - i - 1)] = den > 0 ? (double)cov / sqrt(__ll2double_rn(den))
                                                   : __longlong_as_double(0x7ff8000000000000LL);
      }
    }
  }
}

}  // namespace dense
}  // namespace pgld

// ---------------------------------------------------------------------------
// entry points
// ---------------------------------------------------------------------------
static int dense_grid(pgld_context* h, const void* kern, size_t smem, i64 n_tiles) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, pgld::dense::kThreads, smem);
  per_sm = std::max(1, per_sm);
  return (int)std::max<i64>(1, std::min<i64>(n_tiles, (i64)h->n_sm * per_sm));
}

int pgld_tally_tiles(pgld_context* h, const uint32_t* planes, const uint32_t* valid, int W, i64 n,
                     int32_t* counts, int32_t* n_valid, cudaStream_t st) {
  using namespace pgld::dense;
  const bool aligned = ((uintptr_t)counts & 15) == 0;
  const i64 nb = (n + kT - 1) / kT;
  const bool v = valid && n_valid;
  const void* kern = v ? (const void*)tally_kernel<true> : (const void*)tally_kernel<false>;
  const int grid = dense_grid(h, kern, 0, nb * (nb + 1) / 2);
  pgld_time_begin(h, st);
  if (v)
    tally_kernel<true><<<grid, kThreads, 0, st>>>(planes, valid, W, n, counts, aligned, n_valid);
  else
    tally_kernel<false><<<grid, kThreads, 0, st>>>(planes, nullptr, W, n, counts, aligned, n_valid);
  pgld_time_end(h, st);
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  return PGLD_OK;
}

extern "C" int pgld_geno_rogers_huff_sites(pgld_handle h, const uint32_t* planes, int32_t n_words,
                                           int32_t n_rows, int64_t n_snp, int32_t* sites, double* out,
                                           void* stream) {
  using namespace pgld::dense;
  PGLD_REQUIRE(h, h != nullptr, "pgld_geno_rogers_huff: NULL handle");
  PGLD_REQUIRE(h, n_words >= 1 && n_rows >= 0 && n_rows <= 8192 && n_rows <= 32 * (int64_t)n_words && n_snp >= 0,
               "pgld_geno_rogers_huff: sizes");
  if (n_snp < 2) return PGLD_OK;
  PGLD_REQUIRE(h, planes && sites && out, "pgld_geno_rogers_huff: NULL buffer");
  PGLD_REQUIRE(h, ((uintptr_t)sites & 7) == 0, "pgld_geno_rogers_huff: sites must be 8-byte aligned");
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  int2* site = reinterpret_cast<int2*>(sites);
  const unsigned sb = (unsigned)std::max<i64>(1, std::min<i64>((n_snp + 255) / 256, h->n_sm * 8LL));
  dosage_site_kernel<<<sb, 256, 0, st>>>(planes, n_words, n_snp, n_rows, site);
  const i64 nb = (n_snp + kT - 1) / kT;
  const int grid = dense_grid(h, (const void*)rogers_huff_kernel, 0, nb * (nb + 1) / 2);
  pgld_time_begin(h, st);
  rogers_huff_kernel<<<grid, kThreads, 0, st>>>(planes, n_words, n_snp, n_rows, site, out);
  pgld_time_end(h, st);
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  return PGLD_OK;
}

extern "C" int pgld_geno_rogers_huff(pgld_handle h, const uint32_t* planes, int32_t n_words,
                                     int32_t n_rows, int64_t n_snp, double* out, void* stream) {
  PGLD_REQUIRE(h, h != nullptr && n_snp >= 0, "pgld_geno_rogers_huff: sizes");
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  void* ws = nullptr;
  int rc = pgld_workspace(h, (size_t)n_snp * 8, &ws);
  if (rc) return rc;
  rc = pgld_geno_rogers_huff_sites(h, planes, n_words, n_rows, n_snp, (int32_t*)ws, out, stream);
  if (rc) return rc;
  // the handle's workspace holds the sites: a call on another stream may take it next
  PGLD_CHECK_CUDA(h, cudaStreamSynchronize((cudaStream_t)stream));
  return PGLD_OK;
}

extern "C" int pgld_hap_pairwise_ld(pgld_handle h, const uint32_t* planes, int32_t n_words,
                                    int64_t n_snp, double* D_out, double* r2_out, int64_t ld,
                                    void* stream) {
  using namespace pgld::dense;
  PGLD_REQUIRE(h, h != nullptr, "pgld_hap_pairwise_ld: NULL handle");
  PGLD_REQUIRE(h, n_words >= 1 && n_snp >= 0 && ld >= n_snp, "pgld_hap_pairwise_ld: sizes");
  PGLD_REQUIRE(h, D_out || r2_out, "pgld_hap_pairwise_ld: no output");
  if (n_snp == 0) return PGLD_OK;
  PGLD_REQUIRE(h, planes != nullptr, "pgld_hap_pairwise_ld: NULL planes");
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  void* ws = nullptr;
  int rc = pgld_workspace(h, (size_t)n_snp * 8, &ws);
  if (rc) return rc;
  double* p = (double*)ws;
  const unsigned sb = (unsigned)std::max<i64>(1, std::min<i64>((n_snp + 255) / 256, h->n_sm * 8LL));
  site_freq_kernel<<<sb, 256, 0, st>>>(planes, n_words, n_snp, p);
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  const i64 nb = (n_snp + kT - 1) / kT;
  const size_t smem = sizeof(Smem);
  auto kern = pairwise_ld_kernel;
  PGLD_CHECK_CUDA(h, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = dense_grid(h, (const void*)kern, smem, nb * (nb + 1) / 2);
  pgld_time_begin(h, st);
  kern<<<grid, kThreads, smem, st>>>(planes, n_words, n_snp, p, D_out, r2_out, ld);
  pgld_time_end(h, st);
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  return PGLD_OK;
}

extern "C" int pgld_pairs_by_bin(pgld_handle h, const uint32_t* planes, int32_t n_words,
                                 const double* pair_values, int64_t n_snp, const double* pos,
                                 const double* bins, int32_t n_bins, int64_t* bin_counts,
                                 double* values_out, void* stream) {
  using namespace pgld::dense;
  PGLD_REQUIRE(h, h != nullptr, "pgld_pairs_by_bin: NULL handle");
  PGLD_REQUIRE(h, n_bins >= 1 && n_bins <= pgld::kMaxBins, "pgld_pairs_by_bin: n_bins %d", n_bins);
  PGLD_REQUIRE(h, bins && bin_counts && n_snp >= 0, "pgld_pairs_by_bin: arguments");
  PGLD_REQUIRE(h, pair_values || (planes && n_words >= 1) || n_snp < 2,
               "pgld_pairs_by_bin: needs planes or pair values");
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  if (!values_out)
    for (int b = 0; b < n_bins; ++b) bin_counts[b] = 0;
  if (n_snp < 2) return PGLD_OK;
  PGLD_REQUIRE(h, pos != nullptr, "pgld_pairs_by_bin: NULL pos");
  // workspace: counters [n_bins], cursors [n_bins], bin ends [n_bins], integer
  // positions and their flag
  void* ws = nullptr;
  int rc = pgld_workspace(h, (size_t)3 * n_bins * 8 + 16 + (size_t)n_snp * 4, &ws);
  if (rc) return rc;
  unsigned long long* cnt = (unsigned long long*)ws;
  unsigned long long* cur = cnt + n_bins;
  unsigned long long* end = cur + n_bins;
  int* ipos_bad = (int*)(end + n_bins);
  int* ipos = ipos_bad + 4;
  rc = pgld_tc_int_positions(h, pos, n_snp, ipos, ipos_bad, st);
  if (rc) return rc;
  std::vector<unsigned long long> host(2 * n_bins);
  if (values_out) {
    unsigned long long acc = 0;
    for (int b = 0; b < n_bins; ++b) {
      PGLD_REQUIRE(h, bin_counts[b] >= 0, "pgld_pairs_by_bin: negative count");
      host[b] = acc;
      acc += (unsigned long long)bin_counts[b];
      host[n_bins + b] = acc;
    }
    PGLD_CHECK_CUDA(h, cudaMemcpyAsync(cur, host.data(), (size_t)2 * n_bins * 8,
                                       cudaMemcpyHostToDevice, st));
    PGLD_CHECK_CUDA(h, cudaStreamSynchronize(st));  // host staging buffer is freed below
  } else {
    PGLD_CHECK_CUDA(h, cudaMemsetAsync(cnt, 0, (size_t)n_bins * 8, st));
  }
  const i64 nb = (n_snp + kT - 1) / kT;
  const size_t smem = sizeof(Smem);
  auto kern = pairs_by_bin_kernel;
  PGLD_CHECK_CUDA(h, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = dense_grid(h, (const void*)kern, smem, nb * (nb + 1) / 2);
  pgld_time_begin(h, st);
  kern<<<grid, kThreads, smem, st>>>(planes, n_words, pair_values, n_snp, pos, ipos, ipos_bad, bins,
                                     n_bins, cnt, cur, end, values_out, h->dev_status);
  pgld_time_end(h, st);
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  if (!values_out) {
    PGLD_CHECK_CUDA(h, cudaMemcpyAsync(host.data(), cnt, (size_t)n_bins * 8, cudaMemcpyDeviceToHost, st));
    PGLD_CHECK_CUDA(h, cudaStreamSynchronize(st));
    for (int b = 0; b < n_bins; ++b) bin_counts[b] = (int64_t)host[b];
  }
  return PGLD_OK;
}

extern "C" int pgld_segment_kth(pgld_handle h, const double* values, const int64_t* seg_offsets,
                                int32_t n_seg, const int64_t* targets, int32_t n_targets,
                                double* out, void* stream) {
  using namespace pgld::dense;
  PGLD_REQUIRE(h, h != nullptr, "pgld_segment_kth: NULL handle");
  PGLD_REQUIRE(h, n_seg >= 1 && n_targets >= 0 && seg_offsets && (n_targets == 0 || (targets && out)),
               "pgld_segment_kth: arguments");
  if (n_targets == 0) return PGLD_OK;
  PGLD_REQUIRE(h, values != nullptr, "pgld_segment_kth: NULL values");
  for (int s = 0; s < n_seg; ++s)
    PGLD_REQUIRE(h, seg_offsets[s] >= 0 && seg_offsets[s + 1] >= seg_offsets[s] &&
                        seg_offsets[s + 1] - seg_offsets[s] < (1ll << 32),
                 "pgld_segment_kth: segment %d offsets", s);
  for (int t = 0; t < n_targets; ++t) {
    const int64_t sg = targets[2 * t], rk = targets[2 * t + 1];
    PGLD_REQUIRE(h, sg >= 0 && sg < n_seg && rk >= 0 && rk < seg_offsets[sg + 1] - seg_offsets[sg],
                 "pgld_segment_kth: target %d (segment %lld, rank %lld) out of range", t,
                 (long long)sg, (long long)rk);
  }
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  // targets in segment order; chunks and targets of the segments before each
  std::vector<int> by(n_targets), tseg(n_targets), tgt_off(n_seg + 1, 0);
  for (int t = 0; t < n_targets; ++t) by[t] = t;
  std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return targets[2 * x] < targets[2 * y]; });
  std::vector<long long> chunk_off(n_seg + 1, 0), rank(n_targets);
  for (int t = 0; t < n_targets; ++t) {
    tseg[t] = (int)targets[2 * by[t]];
    rank[t] = targets[2 * by[t] + 1];
    ++tgt_off[tseg[t] + 1];
  }
  for (int s = 0; s < n_seg; ++s) {
    // only the segments that have targets are read
    const long long len = tgt_off[s + 1] ? seg_offsets[s + 1] - seg_offsets[s] : 0;
    chunk_off[s + 1] = chunk_off[s] + (len + kKthChunk - 1) / kKthChunk;
    tgt_off[s + 1] += tgt_off[s];
  }
  std::vector<int> rep(n_targets);
  for (int t = 0; t < n_targets; ++t) rep[t] = tgt_off[tseg[t]];
  PGLD_REQUIRE(h, chunk_off[n_seg] < (1ll << 31), "pgld_segment_kth: too many values");
  // one upload: offsets, chunk offsets, ranks, prefixes (0), then the int tables
  const size_t nl = 2 * (size_t)(n_seg + 1) + 2 * (size_t)n_targets;
  std::vector<long long> up(nl + ((size_t)(n_seg + 1) + 2 * (size_t)n_targets + 1) / 2, 0);
  long long* u = up.data();
  std::copy(seg_offsets, seg_offsets + n_seg + 1, u);
  std::copy(chunk_off.begin(), chunk_off.end(), u + n_seg + 1);
  std::copy(rank.begin(), rank.end(), u + 2 * (n_seg + 1));
  int* ui = (int*)(u + nl);
  std::copy(tgt_off.begin(), tgt_off.end(), ui);
  std::copy(rep.begin(), rep.end(), ui + n_seg + 1);
  std::copy(tseg.begin(), tseg.end(), ui + n_seg + 1 + n_targets);
  const size_t up_b = (up.size() * 8 + 255) & ~size_t(255);
  long long longest = 0;
  for (int t = 0; t < n_targets; ++t)
    longest = std::max<long long>(longest, seg_offsets[tseg[t] + 1] - seg_offsets[tseg[t]]);
  const bool small = longest <= kSmallSeg;
  const size_t hist_b = small ? 0 : (size_t)n_targets * kDigitBins * 4;
  void* ws = nullptr;
  int rc = pgld_workspace(h, up_b + hist_b, &ws);
  if (rc) return rc;
  KthArgs a{};
  a.values = values;
  a.seg_off = (long long*)ws;
  a.chunk_off = a.seg_off + (n_seg + 1);
  a.rank = (long long*)ws + 2 * (n_seg + 1);
  a.prefix = (unsigned long long*)(a.rank + n_targets);
  a.tgt_off = (int*)((long long*)ws + nl);
  a.rep = (int*)((long long*)ws + nl) + (n_seg + 1);
  a.hist = (unsigned*)((char*)ws + up_b);
  a.n_seg = n_seg;
  a.n_targets = n_targets;
  const int* d_tseg = a.rep + n_targets;
  PGLD_CHECK_CUDA(h, cudaMemcpyAsync(ws, u, up.size() * 8, cudaMemcpyHostToDevice, st));
  if (small) {
    kth_small_kernel<<<(unsigned)n_targets, 1024, 0, st>>>(a, d_tseg);
    PGLD_CHECK_CUDA(h, cudaGetLastError());
  }
  for (int pass = 0; pass < kDigits && !small; ++pass) {
    PGLD_CHECK_CUDA(h, cudaMemsetAsync(a.hist, 0, hist_b, st));
    kth_count_kernel<<<(unsigned)chunk_off[n_seg], 256, 0, st>>>(a, pass);
    kth_pick_kernel<<<(unsigned)n_targets, 256, 0, st>>>(a, pass);
    if (pass + 1 < kDigits) kth_rep_kernel<<<(unsigned)((n_targets + 255) / 256), 256, 0, st>>>(a, d_tseg);
    PGLD_CHECK_CUDA(h, cudaGetLastError());
  }
  std::vector<double> got(n_targets);
  PGLD_CHECK_CUDA(h, cudaMemcpyAsync(got.data(), a.prefix, (size_t)n_targets * 8, cudaMemcpyDeviceToHost, st));
  PGLD_CHECK_CUDA(h, cudaStreamSynchronize(st));
  for (int t = 0; t < n_targets; ++t) out[by[t]] = got[t];
  return PGLD_OK;
}
