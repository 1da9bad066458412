// Binned moments sums of three and four haplotype populations.
//
// A CTA takes 32 x 64 SNP tiles of the band work list.  The carrier and
// reference words of all populations are staged together (a chunk holds 32
// words of the concatenated populations, so small populations share one
// staging pass and its latency), each thread counts eight pairs with AND + POPC
// and leaves the counts in shared memory as 16-bit integers; then the warps
// take the tile's pairs in steps of 32 pairs of one distance bin and finalise
// them in float32 (pgld_multi.cuh), summing over a run of steps of one bin in
// registers (tiles of 32 x 32 halve the runs, whose totals take as long as two
// steps).  Four populations make two passes over the steps (66 + 39
// statistics), so that the sums stay in registers.
//
// Bound by issue: per pair of three populations of 200 about 700 instructions
// for features and statistics, 250 for the counts and 100 for the totals.  Three
// populations of 200 haplotypes, 50,000 SNPs, 12 bins to 100 kb (5.0e7 pairs):
// 103 ms per launch with the exact 64-bit term table evaluated per pair
// (band_plain_kernel), 3.0 ms in tiles of 32 x 32, 2.8 ms here.
#include <cuda_runtime.h>

#include <algorithm>

#include "pgld_band.cuh"
#include "pgld_internal.cuh"
#include "pgld_multi_sum.cuh"

namespace pgld {
namespace multi {
namespace {

constexpr int kWords = 32;   // words of the concatenated populations per staged chunk
constexpr int kPitch = 36;   // row pitch in words: 16-byte aligned rows for 4-SNP loads
constexpr int kCols = 64;    // SNPs j of a tile
constexpr int kPitchJ = kCols + 1;
constexpr int kPairs = kTile * kCols;
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;

struct __align__(16) Smem {
  union {  // the staged words until the counts are done, then the steps
    struct {
      uint32_t ci[kWords][kPitch], zi[kWords][kPitch], cj[kWords][kPitchJ], zj[kWords][kPitchJ];
    };
    Groups<kWarps, kPairs> g;
  };
  double bins[kMaxBins + 1];
  int thr[kMaxBins + 1];  // ceil(bins[k]) for integer distances
  int reli[kTile], relj[kCols];
};

template <class T>
__device__ __forceinline__ int bin_at(const T* edge, int n_bins, T d) {
  if (!(d >= edge[0]) || !(d < edge[n_bins])) return -1;
  int lo = 0, hi = n_bins;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (edge[mid] <= d) lo = mid; else hi = mid;
  }
  return lo;
}

template <int P>
__global__ void __launch_bounds__(kThreads, P == 3 ? 2 : 1) band_multi_kernel(BandArgs a, Places pl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  // counts n11 | n10 << 16, n01 | n00 << 16 of every population and pair
  uint2* cnt = reinterpret_cast<uint2*>(smem_raw + sizeof(Smem));
  double* acc = reinterpret_cast<double*>(cnt + P * kPairs);
  unsigned long long* bcnt = reinterpret_cast<unsigned long long*>(acc + a.n_bins * a.n_stats);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int x = threadIdx.x; x < a.n_bins * a.n_stats; x += kThreads) acc[x] = 0.0;
  for (int x = threadIdx.x; x < a.n_bins; x += kThreads) bcnt[x] = 0ull;
  for (int x = threadIdx.x; x <= a.n_bins; x += kThreads) {
    const double b = a.bins[x], cb = ceil(b);
    sm.bins[x] = b;
    sm.thr[x] = cb > 2147483647.0 ? 2147483647 : (cb < -2147483647.0 ? -2147483647 : (int)cb);
  }
  long long n_items = a.item_off[a.n_blocks];
  if (n_items < 0 || n_items > a.n_blocks * (a.n_blocks + 1) / 2) {
    if (threadIdx.x == 0 && a.status) atomicCAS(a.status, 0, 2001);
    n_items = 0;
  }
  const long long n_anchor = anchors_of(a);
  if (n_items > 0 && n_anchor < a.n_snp) n_items = a.item_off[(n_anchor + kTile - 1) / kTile];
  const int maxd_int = a.max_dist >= 2147483647.0 ? 2147483647 : (int)floor(a.max_dist);
  int first[P + 1];  // first word of each population among the concatenated ones
  first[0] = 0;
#pragma unroll
  for (int p = 0; p < P; ++p) first[p + 1] = first[p] + a.W[p];

  for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
    long long lo = 0, hi = a.n_blocks;
    while (hi - lo > 1) {
      const long long mid = (lo + hi) >> 1;
      if (a.item_off[mid] <= item) lo = mid; else hi = mid;
    }
    const long long i0 = lo * kTile, j0 = (lo * kTile / kCols + (item - a.item_off[lo])) * kCols;
    __syncthreads();  // the previous tile's steps are done with the shared memory

    bool is_int = true;
    if (threadIdx.x < kTile + kCols) {
      const bool row = threadIdx.x < kTile;
      const int t = row ? threadIdx.x : threadIdx.x - kTile;
      const long long s = (row ? i0 : j0) + t;
      int r = 0;
      if (s < a.n_snp) {
        const double rel = a.pos[s] - a.pos[i0];
        is_int = (rel == rint(rel)) && fabs(rel) < 1073741824.0;
        r = is_int ? (int)rel : 0;
      }
      if (row) sm.reli[t] = r; else sm.relj[t] = r;
    }
    const bool all_int = __syncthreads_and(is_int ? 1 : 0) && a.bcoord == nullptr;

    // ---- counts: warp w counts the rows 4 w .. 4 w + 3, lane = column ----
    for (int c0 = 0; c0 < first[P]; c0 += kWords) {
      if (c0) __syncthreads();
      {
        const int g = c0 + lane;
        int p = 0;
#pragma unroll
        for (int q = 1; q < P; ++q) p += g >= first[q];
        const bool live = g < first[P];
        int W = 0, f0 = 0;
        const uint32_t* pl_p = nullptr;
#pragma unroll
        for (int q = 0; q < P; ++q)
          if (p == q) {
            W = a.W[q];
            f0 = first[q];
            pl_p = a.planes[q];
          }
        const uint32_t* src = pl_p + (g - f0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int sl = wid * 4 + q;
          const long long si = i0 + sl;
          const bool oi = live && si < a.n_snp;
          sm.ci[lane][sl] = oi ? __ldg(src + si * 2 * W) : 0u;
          sm.zi[lane][sl] = oi ? __ldg(src + si * 2 * W + W) : 0u;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int sl = wid * 8 + q;
          const long long sj = j0 + sl;
          const bool oj = live && sj < a.n_snp;
          sm.cj[lane][sl] = oj ? __ldg(src + sj * 2 * W) : 0u;
          sm.zj[lane][sl] = oj ? __ldg(src + sj * 2 * W + W) : 0u;
        }
      }
      __syncthreads();
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const int w0 = max(first[p], c0) - c0, w1 = min(first[p + 1], c0 + kWords) - c0;
        if (w0 >= w1) continue;
        int c[8][4];  // pair 2 q + h: row 4 wid + q, column 32 h + lane
#pragma unroll
        for (int q = 0; q < 8; ++q) c[q][0] = c[q][1] = c[q][2] = c[q][3] = 0;
#pragma unroll 2
        for (int w = w0; w < w1; ++w) {
          const uint32_t cj[2] = {sm.cj[w][lane], sm.cj[w][32 + lane]};
          const uint32_t zj[2] = {sm.zj[w][lane], sm.zj[w][32 + lane]};
          const uint4 ci4 = *reinterpret_cast<const uint4*>(&sm.ci[w][wid * 4]);
          const uint4 zi4 = *reinterpret_cast<const uint4*>(&sm.zi[w][wid * 4]);
          const uint32_t ci[4] = {ci4.x, ci4.y, ci4.z, ci4.w};
          const uint32_t zi[4] = {zi4.x, zi4.y, zi4.z, zi4.w};
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            c[q][0] += __popc(ci[q >> 1] & cj[q & 1]);
            c[q][1] += __popc(ci[q >> 1] & zj[q & 1]);
            c[q][2] += __popc(zi[q >> 1] & cj[q & 1]);
            c[q][3] += __popc(zi[q >> 1] & zj[q & 1]);
          }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          // at most 2,048 per count: the halves of a word never carry
          uint2* o = cnt + p * kPairs + (wid * 8 + q) * 32 + lane;
          uint2 v = make_uint2((uint32_t)c[q][0] | (uint32_t)c[q][1] << 16,
                               (uint32_t)c[q][2] | (uint32_t)c[q][3] << 16);
          if (c0 + w0 > first[p]) {
            v.x += o->x;
            v.y += o->y;
          }
          *o = v;
        }
      }
    }

    // ---- bins of the thread's pairs ----
    int bin[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int il = wid * 4 + (q >> 1), jl = 32 * (q & 1) + lane;
      const long long i = i0 + il, j = j0 + jl;
      bool ok = i < j && j < a.n_snp && i < n_anchor;
      bin[q] = -1;
      if (all_int) {
        const int d = sm.relj[jl] - sm.reli[il];
        if (ok && d <= maxd_int) bin[q] = bin_at(sm.thr, a.n_bins, d);
      } else if (ok) {
        const double dp = a.pos[j] - a.pos[i];
        if (dp <= a.max_dist)
          bin[q] = bin_at(sm.bins, a.n_bins, a.bcoord ? fabs(a.bcoord[j] - a.bcoord[i]) : dp);
      }
    }
    __syncthreads();  // the staged words are counted
    group_pairs<kWarps, 8>(sm.g, bin, wid * 8, wid, a.n_bins, bcnt, [] { __syncthreads(); });

    const int s0 = sm.g.n_steps * wid / kWarps, s1 = sm.g.n_steps * (wid + 1) / kWarps;
    auto load = [&](int pair, int, Hap(&f)[P]) {
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const uint2 c = pair < kPairs ? cnt[p * kPairs + pair] : make_uint2(0u, 0u);
        f[p] = make_hap(small_f(c.x & 0xffff), small_f(c.x >> 16), small_f(c.y & 0xffff),
                        small_f(c.y >> 16));
      }
    };
    sum_steps<P, 0, Hap>(sm.g, s0, s1, acc, a.n_stats, pl, load);
    if constexpr (P == 4) sum_steps<P, 1, Hap>(sm.g, s0, s1, acc, a.n_stats, pl, load);
  }

  __syncthreads();
  for (int x = threadIdx.x; x < a.n_bins * a.n_stats; x += kThreads)
    if (acc[x] != 0.0) atomicAdd(a.sums + x, acc[x]);
  if (a.pair_counts)
    for (int x = threadIdx.x; x < a.n_bins; x += kThreads)
      if (bcnt[x]) atomicAdd(reinterpret_cast<unsigned long long*>(a.pair_counts) + x, bcnt[x]);
}

template <int P>
int launch(pgld_context* h, const BandArgs& a, cudaStream_t st) {
  const size_t smem = sizeof(Smem) + (size_t)P * kPairs * sizeof(uint2) +
                      (size_t)a.n_bins * (a.n_stats + 1) * 8;
  auto kern = band_multi_kernel<P>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "band_multi smem attribute");
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem);
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "band_multi occupancy");
  const Places pl = places(P, false);
  pgld_time_begin(h, st);
  kern<<<(unsigned)(h->n_sm * std::max(1, per_sm)), kThreads, smem, st>>>(a, pl);
  pgld_time_end(h, st);
  e = cudaGetLastError();
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "band_multi_kernel");
  return PGLD_OK;
}

}  // namespace
}  // namespace multi

// three and four populations of 0/1/-1 data whose features are exact in
// float32 (at most 2,048 haplotypes each); others keep the 64-bit term table
bool band_multi_applies(const BandArgs& a, int mode) {
  if (mode != kModeBinned || a.n_pops < 3) return false;
  for (int p = 0; p < a.n_pops; ++p)
    if (a.valid[p] != nullptr || 32 * a.W[p] > multi::kMaxN) return false;
  return true;
}

int band_multi_cols() { return multi::kCols; }

int launch_band_multi(pgld_context* h, const BandArgs& a, cudaStream_t st) {
  return a.n_pops == 3 ? multi::launch<3>(h, a, st) : multi::launch<4>(h, a, st);
}

}  // namespace pgld
