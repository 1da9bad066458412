// Per-site work on int8 matrices (rows = haplotypes or individuals, columns =
// sites): bit-plane packing, allele counts and presence flags, the lists of
// kept sites, and the heterozygosity sums.
//
// All of it is one pass over the matrix, four sites of a row per 32-bit load
// and four values per instruction: a comparison with a small constant leaves
// 0x80 in the bytes that match.  Rows start at any byte (the row stride is the
// number of sites), so a lane whose four bytes straddle two aligned words
// loads both and shifts; each such word holds at least one byte of the row.
// The kernels move the matrix once; packing writes three (haplotypes) or four
// (genotypes) bits per value.
#include <cuda_runtime.h>

#include <algorithm>

#include "pgld_geno.cuh"
#include "pgld_internal.cuh"

using pgld::i64;

namespace pgld {
namespace sites {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kWarpSites = 128;       // four per lane
constexpr uint32_t kTop = 0x80808080u, kLow = 0x7f7f7f7fu;

// the n < 4 bytes at p (the others read as 0)
__device__ __forceinline__ uint32_t load_tail(const int8_t* p, i64 n) {
  uint32_t v = 0;
  for (int k = 0; k < (int)n; ++k) v |= (uint32_t)(uint8_t)__ldg(p + k) << (8 * k);
  return v;
}
// eight rows' four bytes at column s0: ALIGNED, one aligned word each, else the
// two that the bytes lie in; all loads are issued before the first is used
template <bool ALIGNED, class Row>
__device__ __forceinline__ void load_rows(const int8_t* x, i64 ld, i64 s0, Row&& row,
                                          uint32_t (&v)[8]) {
  if constexpr (ALIGNED) {
#pragma unroll
    for (int r = 0; r < 8; ++r)
      v[r] = __ldg(reinterpret_cast<const uint32_t*>(x + row(r) * ld + s0));
  } else {
    uint32_t hi[8], sh[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int8_t* p = x + row(r) * ld + s0;
      const int a = (int)((uintptr_t)p & 3);
      const uint32_t* w = reinterpret_cast<const uint32_t*>(p - a);
      sh[r] = 8 * a;
      v[r] = __ldg(w);
      hi[r] = __ldg(w + (a != 0));  // an aligned row's own word again
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = __funnelshift_r(v[r], hi[r], sh[r]);
  }
}

// 0x80 in every byte equal to c (0 <= c < 0x80): adding 0x7f to the low seven
// bits of v ^ c sets the top bit unless they are all zero
__device__ __forceinline__ uint32_t equal4(uint32_t v, uint32_t c) {
  return ~((((v ^ (c * 0x01010101u)) & kLow) + kLow) | v) & kTop;
}

// The planes of a value.  split() leaves 0x80 in the bytes that belong to a
// plane; neg1 / neg2 collect (in their top bits) the bytes equal to -1 and the
// other negative ones: adding 1 to the low seven bits carries for -1 only.
// over(): of one site's words, those above the values of the planes.
struct HapPlanes {
  static constexpr int N = 3, kValid = 2, kMain = 2, kExt = 0;
  __device__ static void split(uint32_t v, uint32_t (&m)[N], uint32_t& neg1, uint32_t& neg2) {
    m[0] = equal4(v, 1);
    m[1] = equal4(v, 0);
    m[2] = ~v & kTop;
    const uint32_t up = (v & kLow) + 0x01010101u;
    neg1 |= v & up;
    neg2 |= v & ~up;
  }
  static constexpr bool kAnyNegativeIsMissing = false;
};
// genotypes: dosages 0, 1, 2, valid, and (EXT) the values 3 .. 8
template <bool EXT>
struct GenoPlanes {
  static constexpr int N = EXT ? 10 : 4, kValid = 3, kMain = 3, kExt = EXT ? 6 : 0;
  __device__ static void split(uint32_t v, uint32_t (&m)[N], uint32_t& neg1, uint32_t&) {
    m[0] = equal4(v, 0);
    m[1] = equal4(v, 1);
    m[2] = equal4(v, 2);
    m[3] = ~v & kTop;
    neg1 |= v;
#pragma unroll
    for (int e = 0; e < kExt; ++e) m[4 + e] = equal4(v, 3 + e);
  }
  static constexpr bool kAnyNegativeIsMissing = true;
};

struct PackArgs {
  const int8_t* x;
  i64 ld, n_snp;
  const int32_t* rows;    // row of each haplotype / individual (NULL: 0 .. n_rows - 1)
  int n_rows, W;
  const int32_t* before;  // kept sites before each site, [n_snp + 1] (NULL: all kept)
  uint32_t *planes, *valid, *ext;
  int32_t* flags;
  int words_log2;         // words per block (at most kWarps)
};

// A warp turns 32 rows x 128 sites into one word per site and plane: a row's
// comparison bytes move to the row's bit (a high multiply, beside the
// comparisons on the other pipe) in a register per plane and eight rows, byte
// transposes then give the words.  The block's words of a site are
// stored together (32-byte segments at eight words), through shared memory.
// Values above the planes' show in the words themselves: valid, but in no plane.
template <class S, bool ALIGNED>
__global__ void __launch_bounds__(kThreads) pack_kernel(PackArgs a) {
  constexpr int kPitch = kWarps + 1;
  __shared__ uint32_t out[S::N][kWarpSites * kPitch];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int words = 1 << a.words_log2, chunks = kWarps >> a.words_log2;  // 128-site chunks per block
  const int word = blockIdx.y * words + (warp & (words - 1));
  const i64 s0 = ((i64)blockIdx.x * chunks + (warp >> a.words_log2)) * kWarpSites + 4 * lane;
  const int live = min(32, a.n_rows - 32 * word);  // rows of the word (none for a padding word)
  uint32_t acc[S::N][4];
#pragma unroll
  for (int p = 0; p < S::N; ++p) acc[p][0] = acc[p][1] = acc[p][2] = acc[p][3] = 0;
  uint32_t neg1 = 0, neg2 = 0;
  const i64 left = a.n_snp - s0;
  // (rows past the last are loaded as the last one, and not used)
  int mine = min(32 * word + lane, a.n_rows - 1);
  if (a.rows) mine = __ldg(a.rows + mine);
  const bool whole = s0 - 4 * lane + kWarpSites <= a.n_snp;  // a warp-uniform choice
#pragma unroll
  for (int o = 0; o < 4; ++o) {
    uint32_t v[8];
    auto row = [&](int r) { return (i64)__shfl_sync(0xffffffffu, mine, 8 * o + r); };
    if (whole) {
      load_rows<ALIGNED>(a.x, a.ld, s0, row, v);
    } else {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const i64 at = row(r);
        v[r] = 8 * o + r < live && left > 0 ? load_tail(a.x + at * a.ld + s0, min(left, (i64)4)) : 0u;
      }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (8 * o + r < live) {
        uint32_t m[S::N];
        S::split(v[r], m, neg1, neg2);
#pragma unroll
        for (int p = 0; p < S::N; ++p)  // m >> (7 - r), and add: the bits are apart
          acc[p][o] = r == 7 ? acc[p][o] + m[p] : __umulhi(m[p], 1u << (25 + r)) + acc[p][o];
      }
    }
  }
  // the lane's sites that exist and are kept
  uint32_t kept = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < left && (!a.before || a.before[s0 + k + 1] > a.before[s0 + k])) kept |= 0x80u << (8 * k);
  uint32_t above[4];  // rows in a site's valid word and in no plane
#pragma unroll
  for (int p = 0; p < S::N; ++p) {
    const uint32_t l0 = __byte_perm(acc[p][0], acc[p][1], 0x5140), l1 = __byte_perm(acc[p][0], acc[p][1], 0x7362);
    const uint32_t h0 = __byte_perm(acc[p][2], acc[p][3], 0x5140), h1 = __byte_perm(acc[p][2], acc[p][3], 0x7362);
    uint32_t* o = out[p] + lane * kPitch + warp;  // site 4 lane + k at 32 k + lane
    const uint32_t w[4] = {__byte_perm(l0, h0, 0x5410), __byte_perm(l0, h0, 0x7632),
                           __byte_perm(l1, h1, 0x5410), __byte_perm(l1, h1, 0x7632)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      o[32 * k * kPitch] = w[k];
      if (p == 0) above[k] = ~w[k];
      else if (p < S::kMain) above[k] &= ~w[k];
      else if (p == S::kValid) above[k] &= w[k];
    }
  }
  uint32_t over = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (kept & (0x80u << (8 * k))) over |= above[k];
  const bool any_miss = __any_sync(0xffffffffu, (neg1 & kept) != 0);
  const bool any_other = __any_sync(0xffffffffu, over != 0 || (!S::kAnyNegativeIsMissing && (neg2 & kept) != 0));
  if (lane == 0) {
    if (any_miss) atomicOr(a.flags, 1);
    if (any_other) atomicOr(a.flags + 1, 1);
  }
  __syncthreads();
  // consecutive threads: the words of a site, then the next site of the block
  const i64 b0 = (i64)blockIdx.x * chunks * kWarpSites;
  for (int t = threadIdx.x; t < (chunks * kWarpSites) << a.words_log2; t += kThreads) {
    const int w = t & (words - 1), at = t >> a.words_log2;
    const int W0 = blockIdx.y * words + w;
    const i64 s = b0 + at;
    if (W0 >= a.W || s >= a.n_snp) continue;
    i64 d = s;
    if (a.before) {
      d = a.before[s];
      if (a.before[s + 1] == d) continue;
    }
    const int site = at & (kWarpSites - 1);
    const int from = (32 * (site & 3) + (site >> 2)) * kPitch + ((at / kWarpSites) << a.words_log2) + w;
#pragma unroll
    for (int p = 0; p < S::kMain; ++p) a.planes[d * S::kMain * a.W + p * a.W + W0] = out[p][from];
    if (a.valid) a.valid[d * a.W + W0] = out[S::kValid][from];
#pragma unroll
    for (int e = 0; e < S::kExt; ++e) a.ext[d * S::kExt * a.W + e * a.W + W0] = out[S::kValid + 1 + e][from];
  }
}

template <class S>
int launch_pack(pgld_context* h, PackArgs a, cudaStream_t st) {
  int words = 1;
  while (words < a.W && words < kWarps) {
    words <<= 1;
    ++a.words_log2;
  }
  const i64 per_block = (i64)(kWarps / words) * kWarpSites;
  const dim3 grid((unsigned)((a.n_snp + per_block - 1) / per_block),
                  (unsigned)((a.W + words - 1) / words));
  if ((((uintptr_t)a.x | (uintptr_t)a.ld) & 3) == 0)
    pack_kernel<S, true><<<grid, kThreads, 0, st>>>(a);
  else
    pack_kernel<S, false><<<grid, kThreads, 0, st>>>(a);
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  return PGLD_OK;
}

// ---------------------------------------------------------------------------
// per-site sums of the non-negative values, valid counts, presence flags
// ---------------------------------------------------------------------------
// block: 128 sites x a share of the rows, one row in eight per warp; at most
// 255 rows per warp, so byte counters and 16-bit sums (127 each) never carry.
// SUMS: sum and valid; FLAGS: the presence bits.
template <bool ALIGNED, bool SUMS, bool FLAGS>
__global__ void __launch_bounds__(kThreads) site_counts_kernel(
    const int8_t* __restrict__ x, i64 ld, i64 n_snp, const int32_t* __restrict__ rows, int n_rows,
    int share, int32_t* __restrict__ sum, int32_t* __restrict__ valid,
    uint32_t* __restrict__ flags) {
  __shared__ int s_sum[kWarpSites], s_valid[kWarpSites], s_flag[kWarpSites];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < kWarpSites) s_sum[threadIdx.x] = s_valid[threadIdx.x] = s_flag[threadIdx.x] = 0;
  __syncthreads();
  const i64 s0 = (i64)blockIdx.x * kWarpSites + 4 * lane, left = n_snp - s0;
  const bool whole = s0 - 4 * lane + kWarpSites <= n_snp;
  const int r_end = min(n_rows, (int)(blockIdx.y + 1) * share);
  uint32_t even = 0, odd = 0, nv = 0, zero = 0, one = 0, bits = 0;
  auto add = [&](uint32_t v) {
    uint32_t neg;  // 0xff for each negative byte (prmt's sign mode)
    asm("prmt.b32 %0, %1, %1, 0xba98;" : "=r"(neg) : "r"(v));
    const uint32_t pos = v & ~neg;
    if (SUMS) {
      even += pos & 0x00ff00ffu;
      odd += __byte_perm(pos, 0u, 0x4341u);
      nv += ~neg & 0x01010101u;
    }
    if (FLAGS) {
      zero |= equal4(v, 0);
      one |= equal4(v, 1);
      bits |= pos;
    }
  };
  auto at = [&](int r) { return rows ? (i64)__ldg(rows + r) : (i64)r; };
  int r = (int)blockIdx.y * share + warp;
  if (whole)
    for (; r + 7 * kWarps < r_end; r += 8 * kWarps) {
      uint32_t v[8];
      load_rows<ALIGNED>(x, ld, s0, [&](int k) { return at(r + k * kWarps); }, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) add(v[k]);
    }
  if (left > 0) {
    for (; r < r_end; r += kWarps) {
      const int8_t* p = x + at(r) * ld + s0;
      add(ALIGNED && left >= 4 ? __ldg(reinterpret_cast<const uint32_t*>(p))
                               : load_tail(p, min(left, (i64)4)));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= left) break;
      if (SUMS) {
        atomicAdd(&s_sum[4 * lane + k], (int)((((k & 1) ? odd : even) >> (k & 2 ? 16 : 0)) & 0xffffu));
        atomicAdd(&s_valid[4 * lane + k], (int)((nv >> (8 * k)) & 0xffu));
      }
      if (FLAGS) {
        const int f = (int)((zero >> (8 * k + 7)) & 1u) | (int)((one >> (8 * k + 7)) & 1u) << 1 |
                      (((bits >> (8 * k)) & 0x7eu) ? 4 : 0);
        if (f) atomicOr(&s_flag[4 * lane + k], f);
      }
    }
  }
  __syncthreads();
  const i64 s = (i64)blockIdx.x * kWarpSites + threadIdx.x;
  if (threadIdx.x < kWarpSites && s < n_snp) {
    // several blocks share a site when the rows are split (outputs zeroed before)
    if (sum) atomicAdd(sum + s, s_sum[threadIdx.x]);
    if (valid) atomicAdd(valid + s, s_valid[threadIdx.x]);
    if (flags && s_flag[threadIdx.x]) atomicOr(flags + s, (uint32_t)s_flag[threadIdx.x]);
  }
}

// ---------------------------------------------------------------------------
// kept sites: rule, counts before each site and the list, in two launches (a
// block of the second adds up the totals of the tiles before its own)
// ---------------------------------------------------------------------------
constexpr int kKeepThreads = 256;
constexpr int kKeepTile = kKeepThreads * 16;

__device__ __forceinline__ bool keeps(int rule, const int32_t* sum, const int32_t* valid,
                                      const uint32_t* flags, i64 s) {
  if (rule == PGLD_KEEP_BIALLELIC) return (flags[s] & 7u) == 3u;
  const int a = sum[s], n = valid[s];
  if (rule == PGLD_KEEP_SEGREGATING) return a > 0 && a < n;
  return a > 0 && a < 2 * n && n >= 2;
}

// exclusive prefix of v over the block's threads; *total the block's sum
__device__ __forceinline__ int block_scan(int v, int* sh, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kKeepThreads / 32; ++w) {
    if (w < warp) before += sh[w];
    all += sh[w];
  }
  __syncthreads();
  *total = all;
  return before + x - v;
}

__global__ void __launch_bounds__(kKeepThreads) keep_totals_kernel(
    int rule, const int32_t* sum, const int32_t* valid, const uint32_t* flags, i64 n,
    int32_t* __restrict__ part) {
  const i64 base = (i64)blockIdx.x * kKeepTile;
  int c = 0;
  for (int k = threadIdx.x; k < kKeepTile; k += kKeepThreads)
    if (base + k < n) c += keeps(rule, sum, valid, flags, base + k);
  __shared__ int sh[kKeepThreads / 32];
  int tot;
  block_scan(c, sh, &tot);
  if (threadIdx.x == 0) part[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kKeepThreads) keep_apply_kernel(
    int rule, const int32_t* sum, const int32_t* valid, const uint32_t* flags, i64 n,
    const int32_t* __restrict__ part, int32_t* __restrict__ before, int32_t* __restrict__ index) {
  __shared__ int sh[kKeepThreads / 32];
  const i64 base = (i64)blockIdx.x * kKeepTile;
  int c = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += kKeepThreads) c += part[k];
  int at;
  block_scan(c, sh, &at);
  for (int k0 = 0; k0 < kKeepTile; k0 += kKeepThreads) {
    const i64 s = base + k0 + threadIdx.x;
    const bool keep = s < n && keeps(rule, sum, valid, flags, s);
    int tot;
    const int off = at + block_scan(keep, sh, &tot);
    at += tot;
    if (s <= n) before[s] = off;  // s == n: the total
    if (keep) index[off] = (int32_t)s;
  }
  // n a multiple of the tile: no thread stood at s == n
  if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1 && base + kKeepTile == n) before[n] = at;
}

// ---------------------------------------------------------------------------
// heterozygosity sums of moments (moments_ld.py:346-388): H_ij for i <= j, the
// same float64 expressions per site as the reference's arrays
// ---------------------------------------------------------------------------
struct HetArgs {
  const int32_t* sum[PGLD_MAX_POPS];
  const int32_t* valid[PGLD_MAX_POPS];  // NULL: n_rows everywhere
  double n_rows[PGLD_MAX_POPS];
  int n_pops;
  double per;  // allele copies per row
};

// PARTS: block b's sums to out[b][], for the caller to add in a fixed order (equal
// inputs then give equal bits); else added to out[] in whatever order the blocks end
template <bool PARTS>
__global__ void __launch_bounds__(256) het_kernel(HetArgs a, i64 n, double* __restrict__ out) {
  __shared__ double sh[8];
  double tot[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (i64 s = (i64)blockIdx.x * 256 + threadIdx.x; s < n; s += (i64)gridDim.x * 256) {
    double alt[PGLD_MAX_POPS], ref[PGLD_MAX_POPS], m[PGLD_MAX_POPS];
#pragma unroll
    for (int p = 0; p < PGLD_MAX_POPS; ++p)
      if (p < a.n_pops) {
        alt[p] = (double)a.sum[p][s];
        m[p] = a.per * (a.valid[p] ? (double)a.valid[p][s] : a.n_rows[p]);
        ref[p] = m[p] - alt[p];
      }
    int k = 0;
#pragma unroll
    for (int i = 0; i < PGLD_MAX_POPS; ++i)
#pragma unroll
      for (int j = i; j < PGLD_MAX_POPS; ++j, ++k)
        if (j < a.n_pops)
          tot[k] += i == j ? 2.0 * ref[i] * alt[i] / (m[i] * (m[i] - 1.0))
                           : (ref[i] * alt[j] + alt[i] * ref[j]) / (m[i] * m[j]);
  }
  int k = 0, o = 0;
#pragma unroll
  for (int i = 0; i < PGLD_MAX_POPS; ++i)
#pragma unroll
    for (int j = i; j < PGLD_MAX_POPS; ++j, ++k) {
      if (j >= a.n_pops) continue;
      double v = tot[k];
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
      __syncthreads();
      if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) v += sh[w];
        if (PARTS) out[(size_t)blockIdx.x * (a.n_pops * (a.n_pops + 1) / 2) + o] = v;
        else atomicAdd(out + o, v);
      }
      ++o;
    }
}

}  // namespace sites
}  // namespace pgld

// ---------------------------------------------------------------------------
// entry points
// ---------------------------------------------------------------------------
extern "C" int pgld_pack_haplotypes_kept(pgld_handle h, const int8_t* hap, int64_t ld, int64_t n_snp,
                                         const int32_t* rows, int32_t n_rows, const int32_t* before,
                                         uint32_t* planes, uint32_t* valid, int32_t* flags,
                                         void* stream) {
  PGLD_REQUIRE(h, h != nullptr, "pgld_pack_haplotypes: NULL handle");
  PGLD_REQUIRE(h, n_snp >= 0 && n_rows >= 0, "pgld_pack_haplotypes: negative size");
  PGLD_REQUIRE(h, planes && flags && (hap || n_snp == 0 || n_rows == 0),
               "pgld_pack_haplotypes: NULL buffer");
  PGLD_REQUIRE(h, ld >= n_snp, "pgld_pack_haplotypes: row stride %lld < n_snp %lld",
               (long long)ld, (long long)n_snp);
  const int W = (n_rows + 31) / 32;
  if (n_snp == 0 || W == 0) return PGLD_OK;
  PGLD_REQUIRE(h, W <= 65535, "pgld_pack_haplotypes: too many rows");
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  return pgld::sites::launch_pack<pgld::sites::HapPlanes>(
      h, {hap, ld, n_snp, rows, n_rows, W, before, planes, valid, nullptr, flags, 0},
      (cudaStream_t)stream);
}

extern "C" int pgld_pack_haplotypes(pgld_handle h, const int8_t* hap, int64_t ld, int64_t n_snp,
                                    const int32_t* rows, int32_t n_rows, uint32_t* planes,
                                    uint32_t* valid, int32_t* flags, void* stream) {
  return pgld_pack_haplotypes_kept(h, hap, ld, n_snp, rows, n_rows, nullptr, planes, valid, flags,
                                   stream);
}

extern "C" int pgld_pack_genotypes_kept(pgld_handle h, const int8_t* geno, int64_t ld, int64_t n_snp,
                                        const int32_t* rows, int32_t n_rows, const int32_t* before,
                                        uint32_t* planes, uint32_t* valid, uint32_t* ext,
                                        int32_t* flags, void* stream) {
  PGLD_REQUIRE(h, h != nullptr, "pgld_pack_genotypes: NULL handle");
  PGLD_REQUIRE(h, n_snp >= 0 && n_rows >= 0, "pgld_pack_genotypes: negative size");
  PGLD_REQUIRE(h, planes && flags && (geno || n_snp == 0 || n_rows == 0),
               "pgld_pack_genotypes: NULL buffer");
  PGLD_REQUIRE(h, ld >= n_snp, "pgld_pack_genotypes: row stride %lld < n_snp %lld",
               (long long)ld, (long long)n_snp);
  PGLD_REQUIRE(h, n_rows <= pgld::geno::kMaxGenoN,
               "pgld_pack_genotypes: %d individuals exceed %d per population", n_rows,
               pgld::geno::kMaxGenoN);
  const int W = (n_rows + 31) / 32;
  if (n_snp == 0 || W == 0) return PGLD_OK;
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  const pgld::sites::PackArgs a{geno, ld, n_snp, rows, n_rows, W, before, planes, valid, ext, flags, 0};
  if (ext) return pgld::sites::launch_pack<pgld::sites::GenoPlanes<true>>(h, a, (cudaStream_t)stream);
  return pgld::sites::launch_pack<pgld::sites::GenoPlanes<false>>(h, a, (cudaStream_t)stream);
}

extern "C" int pgld_pack_genotypes(pgld_handle h, const int8_t* geno, int64_t ld, int64_t n_snp,
                                   const int32_t* rows, int32_t n_rows, uint32_t* planes,
                                   uint32_t* valid, uint32_t* ext, int32_t* flags, void* stream) {
  return pgld_pack_genotypes_kept(h, geno, ld, n_snp, rows, n_rows, nullptr, planes, valid, ext, flags,
                                  stream);
}

extern "C" int pgld_site_counts(pgld_handle h, const int8_t* x, int64_t ld, int64_t n_snp,
                                const int32_t* rows, int32_t n_rows, int32_t* sum, int32_t* valid,
                                uint32_t* flags, void* stream) {
  using namespace pgld::sites;
  PGLD_REQUIRE(h, h != nullptr, "pgld_site_counts: NULL handle");
  PGLD_REQUIRE(h, n_snp >= 0 && n_rows >= 0 && ld >= n_snp, "pgld_site_counts: sizes");
  PGLD_REQUIRE(h, x || n_snp == 0 || n_rows == 0, "pgld_site_counts: NULL matrix");
  if (n_snp == 0) return PGLD_OK;
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  if (sum) PGLD_CHECK_CUDA(h, cudaMemsetAsync(sum, 0, (size_t)n_snp * 4, st));
  if (valid) PGLD_CHECK_CUDA(h, cudaMemsetAsync(valid, 0, (size_t)n_snp * 4, st));
  if (flags) PGLD_CHECK_CUDA(h, cudaMemsetAsync(flags, 0, (size_t)n_snp * 4, st));
  if (n_rows == 0) return PGLD_OK;
  // rows are split until every SM has a few blocks (at least one row per warp,
  // at most 255)
  const i64 gx = (n_snp + kWarpSites - 1) / kWarpSites;
  i64 gy = std::max<i64>(1, std::min<i64>((4 * h->n_sm + gx - 1) / gx, (n_rows + 4 * kWarps - 1) / (4 * kWarps)));
  i64 share = (n_rows + gy - 1) / gy;
  share = std::min<i64>((share + kWarps - 1) / kWarps, 255) * kWarps;
  gy = (n_rows + share - 1) / share;
  PGLD_REQUIRE(h, gy <= 65535, "pgld_site_counts: too many rows");
  const bool aligned = (((uintptr_t)x | (uintptr_t)ld) & 3) == 0;
  const bool sums = sum || valid;
  auto kern = !flags ? (aligned ? site_counts_kernel<true, true, false> : site_counts_kernel<false, true, false>)
              : !sums ? (aligned ? site_counts_kernel<true, false, true> : site_counts_kernel<false, false, true>)
                      : (aligned ? site_counts_kernel<true, true, true> : site_counts_kernel<false, true, true>);
  kern<<<dim3((unsigned)gx, (unsigned)gy), kThreads, 0, st>>>(x, ld, n_snp, rows, n_rows, (int)share, sum,
                                                              valid, flags);
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  return PGLD_OK;
}

extern "C" int pgld_keep_sites(pgld_handle h, int32_t rule, const int32_t* sum, const int32_t* valid,
                               const uint32_t* flags, int64_t n_snp, int32_t* before, int32_t* index,
                               int64_t* n_kept, void* stream) {
  using namespace pgld::sites;
  PGLD_REQUIRE(h, h != nullptr, "pgld_keep_sites: NULL handle");
  PGLD_REQUIRE(h, rule >= PGLD_KEEP_BIALLELIC && rule <= PGLD_KEEP_DIPLOID, "pgld_keep_sites: rule %d", rule);
  PGLD_REQUIRE(h, n_snp >= 0 && n_snp < (int64_t(1) << 31) - 1, "pgld_keep_sites: n_snp");
  PGLD_REQUIRE(h, before && n_kept && (index || n_snp == 0), "pgld_keep_sites: NULL output");
  PGLD_REQUIRE(h, n_snp == 0 || (rule == PGLD_KEEP_BIALLELIC ? flags != nullptr : sum && valid),
               "pgld_keep_sites: the rule's counts are missing");
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  *n_kept = 0;
  if (n_snp == 0) {
    PGLD_CHECK_CUDA(h, cudaMemsetAsync(before, 0, 4, st));
    return PGLD_OK;
  }
  const i64 tiles = (n_snp + kKeepTile - 1) / kKeepTile;
  void* ws = nullptr;
  int rc = pgld_workspace(h, (size_t)tiles * 4, &ws);
  if (rc) return rc;
  keep_totals_kernel<<<(unsigned)tiles, kKeepThreads, 0, st>>>(rule, sum, valid, flags, n_snp, (int32_t*)ws);
  keep_apply_kernel<<<(unsigned)tiles, kKeepThreads, 0, st>>>(rule, sum, valid, flags, n_snp,
                                                              (const int32_t*)ws, before, index);
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  int32_t n = 0;
  PGLD_CHECK_CUDA(h, cudaMemcpyAsync(&n, before + n_snp, 4, cudaMemcpyDeviceToHost, st));
  PGLD_CHECK_CUDA(h, cudaStreamSynchronize(st));
  *n_kept = n;
  return PGLD_OK;
}

// parts > 0: the sums of that many blocks; 0: their total
static int heterozygosity(pgld_handle h, int32_t n_pops, const int32_t* const* sum,
                          const int32_t* const* valid, const int32_t* n_rows, int32_t ploidy,
                          int64_t n_snp, int32_t parts, double* out, void* stream) {
  using namespace pgld::sites;
  PGLD_REQUIRE(h, h != nullptr, "pgld_heterozygosity: NULL handle");
  PGLD_REQUIRE(h, n_pops >= 1 && n_pops <= PGLD_MAX_POPS && n_snp >= 0 && ploidy >= 1,
               "pgld_heterozygosity: sizes");
  PGLD_REQUIRE(h, sum && n_rows && out, "pgld_heterozygosity: NULL argument");
  HetArgs a{};
  a.n_pops = n_pops;
  a.per = ploidy;
  for (int p = 0; p < n_pops; ++p) {
    PGLD_REQUIRE(h, sum[p] != nullptr || n_snp == 0, "pgld_heterozygosity: counts of population %d", p);
    a.sum[p] = sum[p];
    a.valid[p] = valid ? valid[p] : nullptr;
    a.n_rows[p] = n_rows[p];
  }
  PGLD_CHECK_CUDA(h, cudaSetDevice(h->device));
  cudaStream_t st = (cudaStream_t)stream;
  if (parts > 0) {
    het_kernel<true><<<(unsigned)parts, 256, 0, st>>>(a, n_snp, out);
  } else {
    PGLD_CHECK_CUDA(h, cudaMemsetAsync(out, 0, (size_t)n_pops * (n_pops + 1) / 2 * 8, st));
    if (n_snp == 0) return PGLD_OK;
    const unsigned blocks = (unsigned)std::min<i64>((n_snp + 255) / 256, (i64)h->n_sm * 4);
    het_kernel<false><<<blocks, 256, 0, st>>>(a, n_snp, out);
  }
  PGLD_CHECK_CUDA(h, cudaGetLastError());
  return PGLD_OK;
}

extern "C" int pgld_heterozygosity(pgld_handle h, int32_t n_pops, const int32_t* const* sum,
                                   const int32_t* const* valid, const int32_t* n_rows,
                                   int32_t ploidy, int64_t n_snp, double* out, void* stream) {
  return heterozygosity(h, n_pops, sum, valid, n_rows, ploidy, n_snp, 0, out, stream);
}

extern "C" int pgld_heterozygosity_parts(pgld_handle h, int32_t n_pops, const int32_t* const* sum,
                                         const int32_t* const* valid, const int32_t* n_rows,
                                         int32_t ploidy, int64_t n_snp, int32_t n_parts, double* out,
                                         void* stream) {
  PGLD_REQUIRE(h, n_parts >= 1 && n_parts <= 1 << 20, "pgld_heterozygosity_parts: n_parts");
  return heterozygosity(h, n_pops, sum, valid, n_rows, ploidy, n_snp, n_parts, out, stream);
}
