// Per-window sums of panels whose listed SNPs all have the same valid
// haplotypes (no missing data among them), on the tensor cores (sm_103a).
//
// With n, p_A and p_B fixed by the SNPs, a pair's statistics follow from n11
// alone, so the operand has one row per SNP (its carriers) instead of two, a
// 128 x 256 MMA tile holds 32,768 pairs instead of 8,192, and a pair costs one
// accumulator element instead of four.  With a = n11 n00, t = n11 + n00 and
// x = n n11 - p_A p_B the numerators are
//   DD   = x (x + n - t) - a n + 2 a - x
//   Dz   = x ((q_A - p_A)(q_B - p_B) + n - 2 t) + 4 a - 2 x
//   pi2  = a (n^2 - 4 n + 2) + x ((2 - n) t + x + n - 1)
// those of pgld_epilogue2.cuh with the other counts eliminated, rounded alike;
// the pairs are also added up in the general kernel's order (blocks of 16 x 32
// from the window's start rounded down to 8), so that the two kernels' sums are
// the same to the last bits.
//
// Whether a list is complete is found on the device: the packing kernel compares
// every SNP's valid haplotypes with the first one's and stops at a difference,
// after which the general kernel (pgld_tc_wide.cu) does the windows and this
// one has no tile; otherwise the other way round.  No answer comes back to the
// host.
//
// One CTA per SM: warp 0 TMA producer (A 128 rows, B 256 rows of 128 bytes),
// warp 1 MMA issuer (M = 128, N = 256, two accumulators), warps 4-19 epilogue:
// the four warps of a TMEM lane quarter take 32 x 64 pieces of the tiles in
// 16 x 32 blocks, one load each; the rows' and columns' p come from global and
// shared memory.  Every mbarrier wait is bounded.
//
// Bound by the float32 pipe: sigma_D^2 takes 21 float32 operations and a division
// per pair.  400 haplotypes, 512 windows of 500-20,000 SNPs (1.37e10 pairs): 20.6 ms
// in the general kernel, 9.4 ms here, 83% of the pipe's rate; the whole call 23.7
// and 11.9 ms.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "pgld_epilogue2.cuh"
#include "pgld_internal.cuh"
#include "pgld_tcgen05.cuh"
#include "pgld_window.cuh"
#include "pgld_window_complete.cuh"

namespace pgld {
namespace wcomp {

using namespace pgld::tc;
using fast2::V;
using fast2::vadd;
using fast2::vfma;
using fast2::vmul;
using fast2::vs;

constexpr int kEpiWarps = 16;  // 96 registers; 12 warps of 128: 9.74 ms where these take 9.36
constexpr int kThreads = (4 + kEpiWarps) * 32;
constexpr int kBoxA = 128 * kKChunk, kBoxB = 256 * kKChunk, kStage = kBoxA + kBoxB;  // 48 KB
constexpr int kUnits = 16;  // a tile's 32 x 64 pieces
constexpr uint32_t kTmemCols = 512;
// D f32, A/B E4M3, both K-major, N = 256, M = 128
constexpr uint32_t kIdesc256 = (1u << 4) | ((256u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_256(uint32_t d, uint64_t a, uint64_t b, uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(kIdesc256), "r"(accum)
      : "memory");
}

struct Params {
  int W;                       // words per plane: K = 32 W haplotypes
  const State* state;
  const float2* site;          // per list position: p_A, 1 / (p_A q_A) (0 where monomorphic)
  long long n_idx;
  const long long* win_begin;
  const long long* win_end;
  int n_win;
  const long long* tile_off;
  double* wsums;               // [n_win][6]
  unsigned long long* wcnt;    // [n_win][3]
  int32_t* status;
  int stages;
  long long wait_cycles;
  int no_copies;               // test hook: the TMA producer issues nothing
};

// ---- the list's valid haplotypes, its operand and its sites -------------------
// the first SNP's valid haplotypes, compared with those of 256 SNPs spread over
// the list: a list with missing data is nearly always known here, and the packing
// kernel's warps then leave at once (50 windows of 200 haplotypes, 1% missing: 37 us
// there when its warps found out by themselves)
__global__ void __launch_bounds__(1024) first_mask_kernel(const uint32_t* __restrict__ planes, int W,
                                                          long long n_snp, long long n_idx,
                                                          const int32_t* __restrict__ idx, State* st) {
  __shared__ uint32_t mask[64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long s = idx ? (long long)idx[0] : 0;
  bool same = s >= 0 && s < n_snp;  // a bad index is the general path's to report
  if (warp == 0) {
    int n = 0;
    for (int w = lane; w < W; w += 32) {
      const uint32_t m = same ? planes[s * 2 * W + w] | planes[s * 2 * W + W + w] : 0u;
      mask[w] = st->mask[w] = m;
      n += __popc(m);
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) st->n = n;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const long long r = n_idx * (8 * warp + k) / 256, x = idx ? (long long)idx[r] : r;
    const bool ok = x >= 0 && x < n_snp;
    same = same && ok;
    for (int w = lane; ok && w < W; w += 32)
      same = same && (__ldg(planes + x * 2 * W + w) | __ldg(planes + x * 2 * W + W + w)) == mask[w];
  }
  same = __syncthreads_and(same ? 1 : 0) != 0;
  if (threadIdx.x == 0) st->complete = same ? 1 : 0;
}

// a warp per list position: lane = word.  Stops at the first SNP whose valid
// haplotypes differ.  out: 32 W bytes per position, E4M3 1.0 per carrier
template <int WL>  // words per lane (W <= 32 WL)
__global__ void __launch_bounds__(256) pack_complete_kernel(
    const uint32_t* __restrict__ planes, int W, long long n_snp, long long n_idx,
    const int32_t* __restrict__ idx, State* st, uint4* __restrict__ out,
    float2* __restrict__ site) {
  const int lane = threadIdx.x & 31;
  uint32_t mask[WL];
#pragma unroll
  for (int q = 0; q < WL; ++q) mask[q] = lane + 32 * q < W ? st->mask[lane + 32 * q] : 0u;
  const int n = st->n;
  volatile int* complete = &st->complete;
  const long long step = (long long)gridDim.x * 8;
  constexpr int kRows = 4;  // list positions in flight per warp
  for (long long r0 = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); r0 < n_idx; r0 += kRows * step) {
    // one decision for the warp: another warp may clear the flag while this one reads it
    if (!__any_sync(0xffffffffu, *complete)) return;
    long long s[kRows];
    uint32_t c[kRows][WL], z[kRows][WL];
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const long long r = r0 + k * step;
      s[k] = r < n_idx ? (idx ? (long long)idx[r] : r) : -2;
    }
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const bool ok = s[k] >= 0 && s[k] < n_snp;
#pragma unroll
      for (int q = 0; q < WL; ++q) {
        const int w = lane + 32 * q;
        c[k][q] = ok && w < W ? __ldg(planes + s[k] * 2 * W + w) : 0u;
        z[k][q] = ok && w < W ? __ldg(planes + s[k] * 2 * W + W + w) : 0u;
      }
    }
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const long long r = r0 + k * step;
      if (r >= n_idx) break;
      bool same = s[k] >= 0 && s[k] < n_snp;
      int d = 0;
#pragma unroll
      for (int q = 0; q < WL; ++q) {
        same = same && (c[k][q] | z[k][q]) == mask[q];
        d += __popc(c[k][q]);
      }
      if (!__all_sync(0xffffffffu, same)) {
        if (lane == 0) *complete = 0;
        return;
      }
      d = __reduce_add_sync(0xffffffffu, d);
      if (lane == 0) {
        const float4 f = win::site_freq(d, n);
        site[r] = make_float2(f.x, f.w);
      }
      uint4* dst = out + r * 2 * W;
#pragma unroll
      for (int q = 0; q < 2 * WL; ++q) {
        const int ch = lane + 32 * q;  // 16 haplotypes: a half word
        const uint32_t word = __shfl_sync(0xffffffffu, c[k][q >> 1], (16 * q + (lane >> 1)) & 31);
        const uint32_t bits = (lane & 1) ? word >> 16 : word & 0xffffu;
        uint32_t v[4];
#pragma unroll
        for (int y = 0; y < 4; ++y) v[y] = nibble_bytes(bits >> (4 * y)) * kOne;
        if (ch < 2 * W) dst[ch] = make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
  }
}

// ---- the tiles ----------------------------------------------------------------
struct Tile {
  long long i0, j0, begin, end;
  int w;
};
// the tile of an item; the window is found stepping forward from hint
__device__ __forceinline__ Tile tile_of(const Params& a, long long item, int& hint) {
  int lo = hint, steps = 0;
  while (lo + 1 < a.n_win && a.tile_off[lo + 1] <= item && steps < 4) {
    ++lo;
    ++steps;
  }
  if (steps == 4) {
    int hi = a.n_win;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (a.tile_off[mid] <= item) lo = mid; else hi = mid;
    }
  }
  hint = lo;
  const long long base = a.win_begin[lo] & ~7ll, m = a.win_end[lo] - base;
  const long long C = (m + 255) >> 8;
  long long b, first;
  row_block(item - a.tile_off[lo], (m + 127) >> 7, C, b, first);
  Tile r;
  r.i0 = base + b * 128;
  r.j0 = base + ((b >> 1) + (item - a.tile_off[lo] - first)) * 256;
  r.begin = a.win_begin[lo];
  r.end = a.win_end[lo];
  r.w = lo;
  return r;
}

// constants of the list's sample size
struct Consts {
  float n, m1, tw, pn, r4;  // n, n - 1, 2 - n, n^2 - 4 n + 2
};

// two pairs of one row (p_A, q_A = n - p_A, u_i) with the columns pB, uj: their
// statistics added to acc, each rounded as pgld_epilogue2.cuh and
// window_pair2_same round it.  live0 / live1 matter where FULL is false
template <int COLS, bool FULL>
__device__ __forceinline__ void two_pairs(const Consts& k, float pA, float qA, float ui, V c1, V pB,
                                          V uj, bool live0, bool live1, V (&acc)[6], int& nr2) {
  const V x = vfma(vs(k.n), c1, vmul(vs(-pA), pB));
  if constexpr ((COLS & 33) != 0) {
    V uu = vmul(vs(ui), uj);
    if (!FULL) uu = make_float2(live0 ? uu.x : 0.f, live1 ? uu.y : 0.f);
    if constexpr ((COLS & 1) != 0) nr2 += (uu.x > 0.f ? 1 : 0) + (uu.y > 0.f ? 1 : 0);
    const V r2 = vmul(vmul(x, x), uu);
    if constexpr ((COLS & 1) != 0) acc[0] = vadd(acc[0], r2);
    if constexpr ((COLS & 32) != 0) acc[5] = vadd(acc[5], r2);
  }
  if constexpr ((COLS & 30) != 0) {
    const V c4 = vadd(c1, fast2::vsub(vs(qA), pB));
    const V a = vmul(c1, c4), t = vadd(c1, c4);
    const V ab = vfma(a, vs(2.0f), fast2::vneg(x));  // n11 n00 + n10 n01
    // DD: the residual e of a n is exact
    const V an = vmul(a, vs(k.n)), e = vfma(a, vs(k.n), fast2::vneg(an));
    const V xs = fast2::vsub(vadd(x, vs(k.n)), t);
    const V dd = vadd(vfma(x, xs, fast2::vneg(an)), fast2::vsub(ab, e));
    // pi2 by Kahan's two-product algorithm: 0 only where it is 0
    const V pi = fast2::dot2(a, vs(k.pn), x, vfma(vs(k.tw), t, vadd(x, vs(k.m1))));
    if constexpr ((COLS & 2) != 0) {
      // pi2 = 0 (no two draws differ at either SNP) leaves DD = 0 as well
      V q = make_float2(__fdividef(dd.x, fmaxf(pi.x, 1.0f)), __fdividef(dd.y, fmaxf(pi.y, 1.0f)));
      if (!FULL) q = make_float2(live0 ? q.x : 0.f, live1 ? q.y : 0.f);
      acc[1] = vadd(acc[1], q);
    }
    if constexpr ((COLS & 28) != 0) {
      const V dB = vfma(pB, vs(-2.0f), vs(k.n));
      const V w = vfma(vs(qA - pA), dB, vfma(t, vs(-2.0f), vs(k.n)));
      const V dz = vfma(x, w, vadd(ab, ab));
      const V r4 = FULL ? vs(k.r4) : make_float2(live0 ? k.r4 : 0.f, live1 ? k.r4 : 0.f);
      acc[2] = vfma(dd, r4, acc[2]);
      acc[3] = vfma(dz, r4, acc[3]);
      acc[4] = vfma(pi, r4, acc[4]);
    }
  }
}

template <int COLS>
__global__ void __launch_bounds__(kThreads, 1)
    window_complete_kernel(const __grid_constant__ CUtensorMap map_a,
                           const __grid_constant__ CUtensorMap map_b, Params a) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* ring = smem_dyn + ((1024 - (smem_u32(smem_dyn) & 1023)) & 1023);
  const int stages = a.stages;
  float* cols = reinterpret_cast<float*>(ring + (size_t)stages * kStage);  // [warps][2][64]
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(cols + kEpiWarps * 128);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &ctrl->abort_flag;
  const long long n_items = a.state->complete ? a.tile_off[a.n_win] : 0;
  if (n_items <= 0) return;  // the general kernel has the windows

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ctrl->full[s], 1);
      mbar_init(&ctrl->empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&ctrl->tfull[s], 1);
      mbar_init(&ctrl->tempty[s], kUnits);
    }
    mbar_init(&ctrl->drain, 1);
    ctrl->abort_flag = 0;
    ctrl->consumed = 0;
    for (int q = 0; q < 4; ++q) ctrl->unit_next[q] = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ctrl->tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctrl->tmem_base;
  const int kchunks = (a.W + 3) / 4;

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- TMA producer ----------------
      int stage = 0, issued = 0, hint = 0;
      uint32_t phase = 0;
      const long long n_copy = a.no_copies ? 0 : n_items;
      for (long long item = blockIdx.x; item < n_copy && !*abort_flag; item += gridDim.x) {
        const Tile t = tile_of(a, item, hint);
        for (int kc = 0; kc < kchunks; ++kc) {
          if (!mbar_wait_role(&ctrl->empty[stage], phase ^ 1, abort_flag, a.wait_cycles)) {
            set_abort(ctrl, a.status, 3002);
            break;
          }
          // a box past the last row or haplotype is filled with zeros
          mbar_expect_tx(&ctrl->full[stage], kStage);
          unsigned char* sa = ring + (size_t)stage * kStage;
          tma_load_2d(sa, &map_a, &ctrl->full[stage], kc * kKChunk, (int)t.i0);
          tma_load_2d(sa + kBoxA, &map_b, &ctrl->full[stage], kc * kKChunk, (int)t.j0);
          ++issued;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (*abort_flag) {
        // drain: every issued copy lands before the CTA may exit
        const int consumed = *(volatile int*)&ctrl->consumed;
        int st2 = consumed % stages;
        uint32_t ph2 = (uint32_t)((consumed / stages) & 1);
        for (int k = consumed; k < issued; ++k) {
          mbar_wait_drain(&ctrl->full[st2], ph2);
          if (++st2 == stages) {
            st2 = 0;
            ph2 ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- MMA issuer ----------------
      int stage = 0, t = 0, consumed = 0;
      uint32_t phase = 0;
      bool any = false;
      for (long long item = blockIdx.x; item < n_items && !*abort_flag; item += gridDim.x, ++t) {
        const int acc = t & 1;
        if (!mbar_wait_role(&ctrl->tempty[acc], (uint32_t)((t >> 1) & 1) ^ 1, abort_flag,
                            a.wait_cycles)) {
          set_abort(ctrl, a.status, 3003);
          break;
        }
        tc_fence_after();
        bool ok = true;
        const uint32_t d = tmem_base + (uint32_t)(acc * 256);
        for (int kc = 0; kc < kchunks; ++kc) {
          if (!mbar_wait_role(&ctrl->full[stage], phase, abort_flag, a.wait_cycles)) {
            set_abort(ctrl, a.status, 3004);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(ring + (size_t)stage * kStage);
          const uint64_t da = smem_desc(sa), db = smem_desc(sa + kBoxA);
          const int steps = min(4, a.W - 4 * kc);  // 32 haplotypes each
          for (int k = 0; k < steps; ++k)
            mma_256(d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), (kc | k) != 0);
          mma_commit(&ctrl->empty[stage]);
          any = true;
          *(volatile int*)&ctrl->consumed = ++consumed;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        mma_commit(&ctrl->tfull[acc]);
      }
      if (*abort_flag && any) {
        // drain: every issued MMA completes before TMEM is freed
        mma_commit(&ctrl->drain);
        mbar_wait_drain(&ctrl->drain, 0);
      }
    }
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    const int quarter = warp & 3;
    float* cp = cols + (warp - 4) * 128;
    float* cu = cp + 64;
    Consts kc;
    {
      const int n = a.state->n;
      float4 e4;
      fast2::recip_entry4(n, &e4);
      kc.n = (float)n;
      kc.m1 = (float)(n - 1);
      kc.tw = (float)(2 - n);
      kc.pn = (float)(n * (n - 4) + 2);
      kc.r4 = n >= 4 ? e4.w : 0.f;
    }
    constexpr bool kU = (COLS & 33) != 0;
    int cur_w = -1, nr2 = 0, units = 0, hint = 0;
    float run[6], comp[6];  // compensated sums of the warp's current window
#pragma unroll
    for (int c = 0; c < 6; ++c) run[c] = comp[c] = 0.f;
    auto emit = [&]() {
      if (cur_w >= 0) {
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          if (!((COLS >> c) & 1)) continue;
          double v = (double)run[c] + (double)comp[c];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane == 0 && v != 0.0) atomicAdd(a.wsums + (long long)cur_w * 6 + c, v);
        }
        if constexpr ((COLS & 1) != 0) {
          const int k = __reduce_add_sync(0xffffffffu, nr2);
          if (lane == 0 && k) atomicAdd(a.wcnt + (long long)cur_w * 3 + 1, (unsigned long long)k);
        }
      }
#pragma unroll
      for (int c = 0; c < 6; ++c) run[c] = comp[c] = 0.f;
      nr2 = units = 0;
    };
#pragma unroll 1
    for (;;) {
      // the quarter's next piece, whichever of its warps is free first
      uint32_t U = 0;
      if (lane == 0) U = atomicAdd(&ctrl->unit_next[quarter], 1u);
      U = __shfl_sync(0xffffffffu, U, 0);
      const int t = (int)(U >> 2), u = (int)(U & 3);
      const long long item = blockIdx.x + (long long)t * gridDim.x;
      if (item >= n_items) break;
      const int acc = t & 1;
      const Tile tl = tile_of(a, item, hint);
      const long long si = tl.i0 + 32 * quarter, sj = tl.j0 + 64 * u;
      const bool none = si >= tl.end || sj >= tl.end || sj + 63 <= si || si + 31 < tl.begin;
      const bool full = si >= tl.begin && si + 31 < sj && sj + 63 < tl.end;
      // the rows' and the columns' sites, loaded before the wait: the lane's
      // rows si + 8 k + lane / 4
      const float2 zero = make_float2(0.f, 0.f);
      float2 fi[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const long long i = si + 8 * k + (lane >> 2);
        fi[k] = !none && i < tl.end ? a.site[i] : zero;
      }
      if (!none) {
        const float2 f0 = sj + lane < tl.end ? a.site[sj + lane] : zero;
        const float2 f1 = sj + 32 + lane < tl.end ? a.site[sj + 32 + lane] : zero;
        __syncwarp();  // the previous piece's columns are read
        cp[lane] = f0.x;
        cp[32 + lane] = f1.x;
        if (kU) {
          cu[lane] = f0.y;
          cu[32 + lane] = f1.y;
        }
        __syncwarp();
      }
      const bool ready = __all_sync(
          0xffffffffu, mbar_wait(&ctrl->tfull[acc], (uint32_t)((t >> 1) & 1), abort_flag, a.wait_cycles));
      if (!ready) {
        if (lane == 0) set_abort(ctrl, a.status, 3005);
        break;
      }
      tc_fence_after();
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctrl->tempty[acc]);
      };
      if (none) {
        release();
        continue;
      }
      if (tl.w != cur_w) {
        emit();
        cur_w = tl.w;
      }
      const uint32_t ta = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * 256 + 64 * u);
      // the window's rows from ib, columns before je, column j being row j + dj
      const int ib = (int)max(tl.begin - si, 0ll), je = (int)min(tl.end - sj, 64ll), dj = (int)(sj - si);
      // a 16x256b load gives a lane the pairs of its rows hh = 0, 1 (8 apart)
      // with the columns 8 g + 2 (lane % 4) + 0, 1 of a 16 x 32 block
      auto body = [&](auto full_c) {
        constexpr bool F = decltype(full_c)::value;
        uint32_t r[2][16];
        tmem_ld16x256_x4(ta, r[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {  // block: rows 16 (c / 2), columns 32 (c % 2)
          tmem_wait_ld();
          if (c < 3)
            tmem_ld16x256_x4(ta + ((uint32_t)(16 * ((c + 1) >> 1)) << 16) + 32 * ((c + 1) & 1),
                             r[(c + 1) & 1]);
          else
            release();
          V ws2[6];
#pragma unroll
          for (int k = 0; k < 6; ++k) ws2[k] = vs(0.f);
          const int cb = 32 * (c & 1) + 2 * (lane & 3);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int hh = (q >> 1) & 1, g = 2 * (q >> 2) + (q & 1);
            const float2 f = fi[2 * (c >> 1) + hh];
            const int i = 8 * (2 * (c >> 1) + hh) + (lane >> 2), j = cb + 8 * g;
            const bool l0 = F || (i >= ib && i < j + dj && j < je);
            const bool l1 = F || (i >= ib && i <= j + dj && j + 1 < je);
            const float2 pB = *reinterpret_cast<const float2*>(cp + cb + 8 * g);
            const float2 uj = kU ? *reinterpret_cast<const float2*>(cu + cb + 8 * g) : zero;
            const uint32_t* rr = &r[c & 1][4 * g + 2 * hh];
            two_pairs<COLS, F>(kc, f.x, kc.n - f.x, f.y,
                               make_float2(__uint_as_float(rr[0]), __uint_as_float(rr[1])), pB, uj, l0,
                               l1, ws2, nr2);
          }
          // TwoSum of the block's totals into the running sums
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            if (!((COLS >> k) & 1)) continue;
            const float v = __fadd_rn(ws2[k].x, ws2[k].y);
            const float sum = __fadd_rn(run[k], v);
            const float b = __fsub_rn(sum, run[k]);
            const float e = __fadd_rn(__fsub_rn(run[k], __fsub_rn(sum, b)), __fsub_rn(v, b));
            comp[k] = __fadd_rn(comp[k], e);
            run[k] = sum;
          }
        }
      };
      if (full) body(std::true_type{});
      else body(std::false_type{});
      // bounded lane counts and compensated sums
      if (++units == 4096) emit();
    }
    if (!*abort_flag) emit();
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(kTmemCols)
                 : "memory");
  }
}

template <int COLS>
static int prepare(pgld_context* h, const Params& prm, const CUtensorMap& map_a,
                  const CUtensorMap& map_b, size_t smem, cudaStream_t st, std::function<int()>* out) {
  auto kern = window_complete_kernel<COLS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "window_complete smem attribute");
  *out = [=]() -> int {
    kern<<<(unsigned)h->n_sm, kThreads, smem, st>>>(map_a, map_b, prm);
    const cudaError_t l = cudaGetLastError();
    return l != cudaSuccess ? pgld_cuda_fail(h, l, "window_complete_kernel") : PGLD_OK;
  };
  return PGLD_OK;
}

}  // namespace wcomp
}  // namespace pgld

using namespace pgld::wcomp;

// The list's operand (32 W bytes per position) and sites, and in state whether
// it is complete.
int pgld_window_complete_pack(pgld_context* h, const uint32_t* planes, int W, long long n_snp,
                              long long n_idx, const int32_t* idx, State* state,
                              unsigned char* op, float2* site, cudaStream_t st) {
  first_mask_kernel<<<1, 1024, 0, st>>>(planes, W, n_snp, n_idx, idx, state);
  const unsigned blocks =
      (unsigned)std::max<long long>(1, std::min<long long>((n_idx + 31) / 32, h->n_sm * 8LL));
  if (W <= 32)
    pack_complete_kernel<1><<<blocks, 256, 0, st>>>(planes, W, n_snp, n_idx, idx, state, (uint4*)op, site);
  else
    pack_complete_kernel<2><<<blocks, 256, 0, st>>>(planes, W, n_snp, n_idx, idx, state, (uint4*)op, site);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "pack_complete_kernel");
  return PGLD_OK;
}

// The windows' sums where state says the list is complete (columns: 2, 32 or all).
// Makes the launch ready: the caller issues it just before the general kernel, in
// one timed interval.
int pgld_window_complete_sums(pgld_context* h, const State* state, int W, long long n_idx,
                              const unsigned char* op, const float2* site, const long long* wb,
                              const long long* we, int n_win, const long long* tile_off, double* sums,
                              unsigned long long* counts, int columns, cudaStream_t st,
                              std::function<int()>* launch) {
  CUtensorMap map_a, map_b;
  int rc = pgld::tchost::make_map(h, &map_a, op, n_idx, 32 * W, 128);
  if (rc) return rc;
  rc = pgld::tchost::make_map(h, &map_b, op, n_idx, 32 * W, 256);
  if (rc) return rc;
  Params prm{};
  prm.W = W;
  prm.state = state;
  prm.site = site;
  prm.n_idx = n_idx;
  prm.win_begin = wb;
  prm.win_end = we;
  prm.n_win = n_win;
  prm.tile_off = tile_off;
  prm.wsums = sums;
  prm.wcnt = counts;
  prm.status = h->dev_status;
  prm.wait_cycles = pgld::tc::kWaitCycles;
  if (h->test_fault == PGLD_TEST_FAULT_NO_COPIES) {
    prm.no_copies = 1;  // the general kernel's launch takes the hook's flag back
    prm.wait_cycles = 20000000ll;
  }
  const size_t fixed = sizeof(pgld::tc::Ctrl) + kEpiWarps * 128 * 4 + 1024;
  int max_smem = 0;
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
  int stages = (int)std::min<long long>(8, ((long long)max_smem - (long long)fixed) / kStage);
  if (h->tc_stages_cap > 0) stages = std::min(stages, h->tc_stages_cap);
  if (stages < 2) return pgld_fail(h, PGLD_ERR_TOO_LARGE, "complete windows: shared memory");
  prm.stages = stages;
  const size_t smem = (size_t)stages * kStage + fixed;
  if (columns == 2) return prepare<2>(h, prm, map_a, map_b, smem, st, launch);
  if (columns == 32) return prepare<32>(h, prm, map_a, map_b, smem, st, launch);
  return prepare<pgld::win::kAllColumns>(h, prm, map_a, map_b, smem, st, launch);
}
