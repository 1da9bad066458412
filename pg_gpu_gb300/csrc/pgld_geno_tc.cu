// tcgen05 tensor-core form of the genotype distance-band pairs (sm_103a).
//
// Everything a single-population pair needs -- the 9-way counts, the
// pairwise-valid n, Rogers-Huff r^2 and the moments DD, Dz, pi2 -- follows
// from the nine centred moments m[3 x + y] = sum c_i^x c_j^y over the
// individuals valid at both SNPs, c = dosage - 1 in {-1, 0, 1}
// (pgld_geno_mom.cuh).  Those are dot products over the individuals: with A =
// the planes (valid, c, c^2) of 32 SNPs j and B the same for 32 SNPs i,
// D = A B^T holds m[3 x + y] for all 1,024 pairs of the tile.  The operand
// rows are plane-major within a 32-SNP block (row = 96 * block + 32 * plane
// + SNP), so D[32 y + j][32 x + i] = m[3 x + y](i, j); the A tile's rows
// 96..127 (M = 128) are zero rows kept in shared memory.
// Operands are E4M3 bytes (0x38 = 1.0, 0xB8 = -1.0) in K-major rows padded to
// 128 bytes; the float32 accumulators hold integers of magnitude below 2^24,
// so the moments are exact.
//
// One CTA per SM:
//   warp 0      TMA producer (96-row x 128-byte boxes, SWIZZLE_128B)
//   warp 1      allocates the TMEM columns; one lane issues M=128 N=96 K=32
//               kind::f8f6f4 MMAs (the B rows of planes 0-2) into the tile's
//               accumulator stage
//   warps 4-    epilogue: two to four groups of four warps take the tiles in
//               turn; in a group the warps of TMEM lane quarters 0-2 (planes
//               0-2) copy the moments to shared memory, then all four turn the
//               pairs into outputs or sums
// Every mbarrier wait is bounded; the warps of an epilogue group meet at
// their named barrier and agree on aborting at the first meeting of a tile.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "pgld_band.cuh"
#include "pgld_epilogue.cuh"
#include "pgld_geno_mom.cuh"
#include "pgld_internal.cuh"
#include "pgld_geno.cuh"
#include "pgld_multi_sum.cuh"
#include "pgld_scan.cuh"
#include "pgld_tc_common.cuh"
#include "pgld_tcgen05.cuh"

namespace pgld {
namespace gtc {

using namespace pgld::tc;

constexpr int kTileSnp = 32;          // SNPs per tile side (4 planes = 128 rows)
constexpr uint32_t kTmemCols = 256;   // two accumulator stages of 128 columns
constexpr int kBlkRows = 96;          // operand rows of a 32-SNP block (3 planes)
constexpr int kABytes = kBoxBytes;     // A: 96 loaded rows + 32 zero rows (M = 128)
constexpr int kBBytes = kBlkRows * kKChunk;  // B: 96 rows (N = 96)
constexpr int kGStageBytes = kABytes + kBBytes;  // 28 KB
constexpr int kCntPitch = 98;         // int16 pitch of the 96 x 96 moment block (49 words: odd)
// instruction descriptor: D f32, A/B E4M3, both K-major, N = 96, M = 128
constexpr uint32_t kIdescN96 = (1u << 4) | ((96u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_f8_n96(uint32_t dtmem, uint64_t a, uint64_t b,
                                           uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(dtmem),
      "l"(a), "l"(b), "r"(kIdescN96), "r"(accum)
      : "memory");
}

struct Params {
  int kchunks;
  long long n_snp;
  const long long* item_off;
  long long n_blocks;
  const long long* pair_off;
  int32_t* counts;   // [n_pairs][9] or NULL
  int32_t* nvalid;   // [n_pairs] or NULL
  float* stats;      // [n_pairs][4] or NULL
  int stat_mask;
  int32_t* status;
  int stages;
  int groups;  // epilogue groups of four warps (2-4)
};

constexpr int kMaxGroups = 4;
constexpr int kPairThreads = (4 + 4 * kMaxGroups) * 32;
constexpr int kMomWords = 25;                // pitch of a half tile's 24 moment words (odd)
constexpr int kMomBytes = 96 * kMomWords * 4;
constexpr int kCtrlBytes = 512;             // the control block, 16-byte aligned end
constexpr int kCountStage = (9 * 32 + 4) * 4;  // bytes of a warp's staged counts, any alignment

constexpr int kChunkItems = 16;  // consecutive tiles a CTA takes per turn (resident form)

// control block: the stage / accumulator barriers, plus the resident form's
// B barriers and the per-stage tile flags the producer hands the MMA issuer
struct GCtrl : Ctrl {
  uint64_t bfull, bempty;
  uint64_t gfull[kMaxGroups];   // an epilogue group's next tile is accumulated
  uint64_t gempty[kMaxGroups];  // an accumulator stage is copied
  int meta[8];  // first stage of a tile: bit 0 = first tile of a strip, bit 1 = last
};

static_assert(sizeof(GCtrl) <= kCtrlBytes, "control block");

// the t-th tile of this CTA: turns of `chunk` consecutive items, round robin
// over the CTAs (chunk 1: item blockIdx.x + t * gridDim.x)
__device__ __forceinline__ long long tile_item(int t, int chunk) {
  return ((long long)blockIdx.x + (long long)(t / chunk) * gridDim.x) * chunk + t % chunk;
}

// row block of an item, moving forward from lo (the items a thread visits
// ascend): a few steps, then a binary search
__device__ __forceinline__ long long advance_block(const long long* item_off, long long n_blocks,
                                                   long long lo, long long item) {
#pragma unroll 1
  for (int s = 0; s < 4; ++s) {
    if (lo + 1 >= n_blocks || item_off[lo + 1] > item) return lo;
    ++lo;
  }
  long long hi = n_blocks;
  while (hi - lo > 1) {
    const long long mid = (lo + hi) >> 1;
    if (item_off[mid] <= item) lo = mid; else hi = mid;
  }
  return lo;
}

// The nine counts of the warp's pairs first + lane (lanes lo <= lane < hi) to
// counts[][9].  The lanes' values lie 36 bytes apart: stored one by one, each of
// nine stores would touch every sector of the row.  They pass through the
// warp's staging words, placed as the row lies to a 16-byte boundary, and leave
// as 16-byte stores, the ends of the row word by word.
__device__ __forceinline__ void store_counts(int32_t* counts, long long first, int lo, int hi,
                                             int lane, uint32_t* stage, const int (&c)[9]) {
  int32_t* row = counts + first * 9;
  const int a0 = (int)((reinterpret_cast<uintptr_t>(row) >> 2) & 3);
  __syncwarp();  // the previous row has left the staging words
#pragma unroll
  for (int x = 0; x < 9; ++x) stage[a0 + 9 * lane + x] = (uint32_t)c[x];
  __syncwarp();
  if (lo >= hi) return;
  const int w0 = a0 + 9 * lo, w1 = a0 + 9 * hi;  // the row's words of the stage
  row -= a0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int s = 4 * (lane + 32 * q);
    if (s >= w0 && s + 4 <= w1)
      __stcs(reinterpret_cast<int4*>(row + s), *reinterpret_cast<const int4*>(stage + s));
  }
  // the words of the first and last quarters that are not whole
  const int f = w0 & ~3, l = w1 & ~3;
  const int s = lane < 4 ? f + lane : l + lane - 4;
  const bool part = lane < 4 ? f < w0 || f + 4 > w1 : lane < 8 && l < w1 && l != f;
  if (part && s >= w0 && s < w1) __stcs(row + s, (int)stage[s]);
}

// MASK: the statistic columns when fixed at compile time (-1: a.stat_mask).
// A (M = 128 with 32 zero rows) is the column block j, B (N = 96) the row block
// i: accumulator lanes are planes of the SNPs j, columns planes of the SNPs i.
// RES: the resident form -- the row block's 96 operand rows (every K chunk)
// stay in shared memory for a strip of consecutive tiles of that row block, and
// only the column block streams.  Otherwise both blocks stream per K chunk.
template <int MASK, bool RES>
__global__ void __launch_bounds__(kPairThreads, 1)
    gtc_pairs_kernel(const __grid_constant__ CUtensorMap map, Params a) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* base = smem_dyn + ((1024 - (smem_u32(smem_dyn) & 1023)) & 1023);
  const int stages = a.stages;
  constexpr int kStage = RES ? kABytes : kGStageBytes;
  const int chunk = RES ? kChunkItems : 1;
  unsigned char* ring = base;
  unsigned char* bres = ring + (size_t)stages * kStage;  // resident B (RES only)
  GCtrl* ctrl = reinterpret_cast<GCtrl*>(bres + (RES ? (size_t)a.kchunks * kBBytes : 0));
  unsigned char* moms = reinterpret_cast<unsigned char*>(ctrl) + kCtrlBytes;  // [groups][96][kMomWords]
  const int groups = a.groups;
  unsigned char* stage_c = moms + (size_t)groups * kMomBytes;  // [4 * groups][kCountStage]
  const uint32_t tmem_cols = groups > 2 ? 512u : kTmemCols;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &ctrl->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ctrl->full[s], 1);
      mbar_init(&ctrl->empty[s], 1);
    }
    for (int s = 0; s < groups; ++s) {
      mbar_init(&ctrl->gfull[s], 1);
      mbar_init(&ctrl->gempty[s], 4);  // the four warps of epilogue group s
    }
    mbar_init(&ctrl->drain, 1);
    mbar_init(&ctrl->bfull, 1);
    mbar_init(&ctrl->bempty, 1);
    ctrl->abort_flag = 0;
    ctrl->consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ctrl->tmem_base)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // rows 96..127 of every A stage (the last 4 KB: whole 1 KB swizzle atoms)
  // stay zero: TMA writes only the 96 operand rows
  for (int s = 0; s < stages; ++s) {
    uint4* z = reinterpret_cast<uint4*>(ring + (size_t)s * kStage + kBlkRows * kKChunk);
    for (int k = threadIdx.x; k < (kABytes - kBlkRows * kKChunk) / 16; k += blockDim.x)
      z[k] = make_uint4(0u, 0u, 0u, 0u);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctrl->tmem_base;

  long long n_items = a.item_off[a.n_blocks];
  if (n_items < 0 || n_items > a.n_blocks * (a.n_blocks + 1) / 2) {
    if (threadIdx.x == 0) set_abort(ctrl, a.status, 4001);
    n_items = 0;
  }

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0, strips = 0;
      long long item = tile_item(0, chunk);
      long long lo = item < n_items ? advance_block(a.item_off, a.n_blocks, 0, item) : 0;
      long long lo_prev = -1;
      for (int t = 0; item < n_items && !*abort_flag; ++t) {
        const long long jb = lo + (item - a.item_off[lo]);
        const long long next = tile_item(t + 1, chunk);
        const long long lo_next =
            next < n_items ? advance_block(a.item_off, a.n_blocks, lo, next) : -1;
        const bool first = lo != lo_prev, last = lo_next != lo;
        bool ok = true;
        if (RES && first) {
          // a new strip: its row block replaces the resident B once the MMAs
          // of the previous strip are done with it
          if (strips > 0 && !mbar_wait_role(&ctrl->bempty, (uint32_t)((strips - 1) & 1),
                                            abort_flag)) {
            set_abort(ctrl, a.status, 4006);
            break;
          }
          mbar_expect_tx(&ctrl->bfull, (uint32_t)(a.kchunks * kBBytes));
          for (int kc = 0; kc < a.kchunks; ++kc)
            tma_load_2d(bres + (size_t)kc * kBBytes, &map, &ctrl->bfull, kc * kKChunk,
                        (int)(lo * kBlkRows));
          ++strips;
        }
        for (int kc = 0; kc < a.kchunks; ++kc) {
          if (!mbar_wait_role(&ctrl->empty[stage], phase ^ 1, abort_flag)) {
            set_abort(ctrl, a.status, 4002);
            ok = false;
            break;
          }
          if (kc == 0) ctrl->meta[stage] = (first ? 1 : 0) | (last ? 2 : 0);
          unsigned char* sa = ring + (size_t)stage * kStage;
          if (RES) {
            mbar_expect_tx(&ctrl->full[stage], kBBytes);
            tma_load_2d(sa, &map, &ctrl->full[stage], kc * kKChunk, (int)(jb * kBlkRows));
          } else {
            mbar_expect_tx(&ctrl->full[stage], 2 * kBBytes);
            tma_load_2d(sa, &map, &ctrl->full[stage], kc * kKChunk, (int)(jb * kBlkRows));
            tma_load_2d(sa + kABytes, &map, &ctrl->full[stage], kc * kKChunk,
                        (int)(lo * kBlkRows));
          }
          ++issued;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        lo_prev = lo;
        lo = lo_next;
        item = next;
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
        if (RES && strips > 0) mbar_wait_drain(&ctrl->bfull, (uint32_t)((strips - 1) & 1));
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int consumed = 0, strips = 0;
      bool any = false;
      int acc = -1;
      uint32_t aph = 1;
      for (int t = 0; !*abort_flag; ++t) {
        if (tile_item(t, chunk) >= n_items) break;
        if (++acc == groups || t == 0) {
          acc = 0;
          aph ^= 1;
        }
        if (!mbar_wait_role(&ctrl->gempty[acc], aph ^ 1, abort_flag)) {
          set_abort(ctrl, a.status, 4003);
          break;
        }
        tc_fence_after();
        bool ok = true, last = false;
        const uint32_t d = tmem_base + (uint32_t)(acc * 128);
        for (int kc = 0; kc < a.kchunks; ++kc) {
          if (!mbar_wait_role(&ctrl->full[stage], phase, abort_flag)) {
            set_abort(ctrl, a.status, 4004);
            ok = false;
            break;
          }
          if (kc == 0) {
            const int m = ctrl->meta[stage];
            last = (m & 2) != 0;
            if (RES && (m & 1)) {
              if (!mbar_wait_role(&ctrl->bfull, (uint32_t)(strips & 1), abort_flag)) {
                set_abort(ctrl, a.status, 4007);
                ok = false;
                break;
              }
              ++strips;
            }
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(ring + (size_t)stage * kStage);
          const uint64_t da = smem_desc(sa);
          const uint64_t db =
              smem_desc(RES ? smem_u32(bres + (size_t)kc * kBBytes) : sa + kABytes);
#pragma unroll
          for (int k = 0; k < kKChunk / 32; ++k)
            mma_f8_n96(d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), (kc | k) != 0);
          mma_commit(&ctrl->empty[stage]);
          any = true;
          *(volatile int*)&ctrl->consumed = ++consumed;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        mma_commit(&ctrl->gfull[acc]);
        if (RES && last) mma_commit(&ctrl->bempty);  // the strip's MMAs are all issued
      }
      if (*abort_flag && any) {
        mma_commit(&ctrl->drain);
        mbar_wait_drain(&ctrl->drain, 0);
      }
    }
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    // Groups of four warps take the tiles in turn (group g: tiles g, g + groups,
    // ... of this CTA, accumulator stage g, moment buffer g), so one group's
    // copy and the others' statistics overlap.  A group takes its tile in two
    // halves of 16 rows i: the warp of TMEM lane quarter q < 3 copies plane q's
    // 48 moment columns of the half, two int16 moments (rows i, i + 1) to a
    // word, and all four warps turn its 512 pairs into outputs (4 per thread).
    // Whole tiles would take 28 KB more of shared memory, two of the stages
    // that keep the column block streaming.
    const int e = warp - 4;
    const int grp = e >> 2;
    const int wq = warp & 3;  // TMEM lanes 32q..32q+31: plane q of the SNPs j
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    const uint32_t bar_id = 1u + (uint32_t)grp;
    uint32_t* buf = reinterpret_cast<uint32_t*>(moms + (size_t)grp * kMomBytes);
    uint32_t* cstage = reinterpret_cast<uint32_t*>(stage_c + (size_t)e * kCountStage);
    int t = grp;
    long long item = tile_item(t, chunk);

    // tile location: items ascend, so the row block lo only moves forward;
    // nv holds item_off[lo + 1 + lane], loaded one tile ahead
    long long lo = 0;
    long long nv = 1 + lane <= a.n_blocks ? a.item_off[1 + lane] : LLONG_MAX;
    long long i0 = 0, j0 = 0, off_lo = 0;
    int off_n = 0;
    auto locate = [&](long long it) {
      unsigned bal = __ballot_sync(0xffffffffu, nv <= it);
      lo += __popc(bal);
      if (bal == 0xffffffffu) {
        const long long idx = lo + 1 + lane;
        bal = __ballot_sync(0xffffffffu, idx <= a.n_blocks && a.item_off[idx] <= it);
        lo += __popc(bal);
        if (bal == 0xffffffffu) {
          long long l2 = lo, h2 = a.n_blocks;
          while (h2 - l2 > 1) {
            const long long mid = (l2 + h2) >> 1;
            if (a.item_off[mid] <= it) l2 = mid; else h2 = mid;
          }
          lo = l2;
        }
      }
      i0 = lo * kTileSnp;
      j0 = (lo + (it - a.item_off[lo])) * kTileSnp;
      // band offsets of the tile's 32 rows: lane l holds row i0 + l
      const long long ri = i0 + lane < a.n_snp ? i0 + lane : a.n_snp;
      off_lo = a.pair_off[ri];
      off_n = (int)((ri < a.n_snp ? a.pair_off[ri + 1] : off_lo) - off_lo);
    };
    if (item < n_items) locate(item);

    for (int u = 0; item < n_items; ++u) {
      bool ready = true;
      if (lane == 0) ready = mbar_wait(&ctrl->gfull[grp], (uint32_t)(u & 1), abort_flag);
      ready = __shfl_sync(0xffffffffu, ready ? 1 : 0, 0) != 0;
      if (!ready && lane == 0) set_abort(ctrl, a.status, 4005);
      // the group meets before overwriting its buffer (every warp is done
      // reading the previous tile) and takes one decision on aborting: the
      // barrier ORs every thread's view (its own wait failed, or the control
      // block's flag is set), so no warp is left waiting
      uint32_t any_abort = 0;
      const uint32_t mine = (ready ? 0u : 1u) | (uint32_t)(*abort_flag != 0);
      asm volatile(
          "{\n .reg .pred pin, pout;\n setp.ne.u32 pin, %1, 0;\n"
          " bar.red.or.pred pout, %2, 128, pin;\n selp.u32 %0, 1, 0, pout;\n}"
          : "=r"(any_abort)
          : "r"(mine), "r"(bar_id)
          : "memory");
      if (any_abort) break;
      tc_fence_after();
      const bool want_nv = a.nvalid != nullptr;
      // this tile's location; the next tile's offsets load during the pairs
      const long long ti0 = i0, tj0 = j0, toff = off_lo;
      const int tn = off_n;
      t += groups;
      const long long next = tile_item(t, chunk);
      if (next < n_items) nv = lo + 1 + lane <= a.n_blocks ? a.item_off[lo + 1 + lane] : LLONG_MAX;

#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        if (wq < 3) {
          uint32_t* row = buf + (wq * 32 + lane) * kMomWords;
          uint32_t r[3][16];
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tmem_ld16(tmem_base + lane_base + (uint32_t)(grp * 128 + 32 * x + 16 * h), r[x]);
          tmem_wait_ld();
          if (h) asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");  // half 0 is read
#pragma unroll
          for (int x = 0; x < 3; ++x)
#pragma unroll
            for (int v = 0; v < 8; ++v)
              row[8 * x + v] =
                  fast::f2i_pair(__uint_as_float(r[x][2 * v]), __uint_as_float(r[x][2 * v + 1]));
        } else if (h) {
          asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");
        }
        if (h) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctrl->gempty[grp]);
        }
        asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");

        // four pairs per thread, two rows at a time; every value is computed
        // and only the stores depend on the pair lying in the band.  The
        // outputs go out as streaming global stores (st.global.cs): they are
        // not re-read, and being global-space they cannot alias the
        // shared-memory moments.
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
          const uint32_t* w0 = buf + lane * kMomWords + wq + 4 * k;
          uint32_t w[9];
#pragma unroll
          for (int x = 0; x < 3; ++x)
#pragma unroll
            for (int y = 0; y < 3; ++y) w[3 * x + y] = w0[y * 32 * kMomWords + x * 8];
#pragma unroll
          for (int z = 0; z < 2; ++z) {
            const int il = 16 * h + 2 * (wq + 4 * k) + z;
            const long long row_off = __shfl_sync(0xffffffffu, toff, il);
            const int row_n = __shfl_sync(0xffffffffu, tn, il);
            const int d0 = (int)(tj0 - ti0) - il - 1;  // j - i - 1 of lane 0
            const int d = d0 + lane;
            // d < row_n keeps j inside the band and below n_snp
            const bool ok = d >= 0 && d < row_n;
            gmom::Mom mo;
#pragma unroll
            for (int x = 0; x < 9; ++x)
              mo.m[x] = z ? (int)w[x] >> 16 : (int)(short)(w[x] & 0xffff);
            const long long kk = row_off + d;
            if (a.counts) {
              int c9[9];
              gmom::to_counts(mo, c9);
              store_counts(a.counts, row_off + d0, max(0, -d0), min(32, row_n - d0), lane, cstage,
                           c9);
            }
            st_cs_if(ok && want_nv, a.nvalid + kk, mo.m[0]);
            if (a.stats) {
              const float4 o = gmom::stats_f32<MASK>(mo, a.stat_mask);
              st_cs_if(ok, reinterpret_cast<float4*>(a.stats) + kk, o);
            }
          }
        }
      }
      item = next;
      if (item < n_items) locate(item);
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(tmem_cols)
                 : "memory");
  }
}

// operand rows: row 96 * (s / 32) + 32 * plane + s % 32 holds, per
// individual, plane 0: 1 if the dosage at SNP s is known, plane 1: c = dosage
// - 1 (+1, 0, -1; 0 if missing), plane 2: c^2.  A warp
// writes the three rows of its SNPs in 16-byte chunks (16 individuals), the
// bit planes read once (1,000 individuals, 100,000 SNPs, 307 MB written: 104 us
// with a warp per row, 53 us).
constexpr int kPackSnps = 2;  // SNPs in flight per warp
__global__ void __launch_bounds__(256) pack_gtc_kernel(const uint32_t* __restrict__ planes, int W,
                                                       long long n_snp, long long n_blocks,
                                                       int k_pad, uint32_t* __restrict__ out) {
  const int lane = threadIdx.x & 31, chunks = k_pad / 16;
  uint4* rows = reinterpret_cast<uint4*>(out);
  const long long n_out = n_blocks * kTileSnp, step = (long long)gridDim.x * 8 * kPackSnps;
  for (long long s0 = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * kPackSnps; s0 < n_out;
       s0 += step) {
    for (int c = lane; c < chunks; c += 32) {
      const int w = c >> 1, sh = 16 * (c & 1);
      uint32_t g[kPackSnps][3];
#pragma unroll
      for (int k = 0; k < kPackSnps; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d)
          g[k][d] = s0 + k < n_snp && w < W ? __ldg(planes + (s0 + k) * 3 * W + d * W + w) >> sh : 0u;
#pragma unroll
      for (int k = 0; k < kPackSnps; ++k) {
        const long long s = s0 + k;
        uint4* dst = rows + ((s / kTileSnp) * kBlkRows + (s % kTileSnp)) * chunks + c;
        const uint32_t hom = g[k][0] | g[k][2], known = hom | g[k][1];
        uint32_t v[3][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          v[0][q] = nibble_bytes(known >> (4 * q)) * kOne;
          v[2][q] = nibble_bytes(hom >> (4 * q)) * kOne;
          v[1][q] = v[2][q] | nibble_bytes(g[k][0] >> (4 * q)) * 0x80u;  // the sign bit
        }
#pragma unroll
        for (int d = 0; d < 3; ++d)
          dst[(long long)d * kTileSnp * chunks] = make_uint4(v[d][0], v[d][1], v[d][2], v[d][3]);
      }
    }
  }
}
static unsigned pack_gtc_blocks(const pgld_context* h, long long n_blocks) {
  return (unsigned)std::max<long long>(
      1, std::min<long long>((n_blocks * kTileSnp + 8 * kPackSnps - 1) / (8 * kPackSnps), h->n_sm * 16LL));
}

// ---------------------------------------------------------------------------
// Distance-binned sums of the genotype statistics of 1-4 populations.  The
// tile of 32 x 32 SNPs takes one M = 128, N = 96 MMA chain per population
// (the operand rows of population p start at row p * n_blocks * 96), each
// into its own 96 TMEM columns of the tile's accumulator stage.  One
// population: DD, Dz and pi2 in float32 straight from the moments
// (gmom::stats_f32).  Several: the group orders the tile's pairs by distance
// bin and its warps take them in steps of 32 pairs of one bin, the statistics
// unrolled in float32 from the moments (pgld_multi.cuh); the rare pair with
// fewer than four valid individuals in a population, where the reference's
// thresholds and zero denominators differ from statistic to statistic, goes
// through the exact term table by itself.  Sums per distance bin in float64
// slots of the CTA.  G epilogue groups take the tiles in turn, each with a
// moment buffer of its own; the accumulator stages (four of one population, two
// of two, one of three or four) are freed once copied.  Bound by the
// statistics' instructions, about 600 a pair of two populations: 500
// individuals, 100,000 SNPs, 12 bins to 100 kb (1.0e8 pairs) 4.1 ms with two
// groups, 3.6 with three (sixteen warps in two groups: 5.1, registers and totals
// of four steps); three populations of 200, 20,000 SNPs 1.78 and 1.41 ms with one
// group of eight warps and two of four; one population of 200, 60,000 SNPs: 1.5 ms
// with distances and bins in 64 bits, a butterfly per total and an addition to the
// slots each, 0.83 here.
// ---------------------------------------------------------------------------
struct BParams {
  int kchunks;
  long long n_snp;
  const long long* item_off;
  long long n_blocks;
  int n_pops;
  int pop_rows;             // operand rows per population (n_blocks * 96)
  const double* pos;
  const double* bcoord;     // distances for binning (NULL: positions)
  const int* ipos;          // integer positions (valid when *ipos_bad == 0)
  const int* ipos_bad;
  double max_dist;
  const double* bins;
  int n_bins;
  int exact;                // every pair through the term table (samples above multi::kMaxN)
  const pgld_term* terms;
  int n_terms, n_stats;
  double* sums;             // [n_bins][n_stats]
  unsigned long long* pair_counts;
  int32_t* status;
  int stages;
};

// the statistics of one pair through the exact term table, added to slots
template <int P>
__device__ __noinline__ void term_table_pair(const gmom::Mom* mo, const BParams& a, double* slots) {
  int cc[P][9];
  geno::GPop gp[P];
  const int* cp[P];
  for (int p = 0; p < P; ++p) {
    gmom::to_counts(mo[p], cc[p]);
    gp[p] = geno::make_gpop(cc[p], -1);
    cp[p] = cc[p];
  }
  int t = 0;
  for (int s = 0; s < a.n_stats; ++s) {
    float v = 0.f;
    for (; t < a.n_terms && a.terms[t].stat == s; ++t) {
      const pgld_term tm = a.terms[t];
      v += (float)tm.weight * geno::term_value<float>(tm, gp, cp);
    }
    atomicAdd(slots + s, (double)v);
  }
}

// G groups of kGW epilogue warps take the tiles in turn, A accumulator stages
// (four populations leave room for one group's moments only)
template <int P>
struct Binned {
  static constexpr int G = P == 1 ? 4 : P == 2 ? 3 : P == 3 ? 2 : 1;
  static constexpr int kGW = P <= 2 ? 4 : 8 / G;
  static constexpr int A = P == 1 ? 4 : P == 2 ? 2 : 1;
  static constexpr int kThreads = (4 + G * kGW) * 32;
};
template <int P>
__global__ void __launch_bounds__(Binned<P>::kThreads, 1)
    gtc_binned_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ BParams a,
                      const __grid_constant__ multi::Places pl) {
  constexpr int G = Binned<P>::G, A = Binned<P>::A, kGW = Binned<P>::kGW;
  constexpr int kRows = 32 / kGW;      // rows of a tile per warp
  constexpr uint32_t kStageCols = 512u / A;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* base = smem_dyn + ((1024 - (smem_u32(smem_dyn) & 1023)) & 1023);
  const int stages = a.stages;
  unsigned char* ring = base;
  GCtrl* ctrl = reinterpret_cast<GCtrl*>(ring + (size_t)stages * kGStageBytes);
  int16_t* cnt = reinterpret_cast<int16_t*>(ctrl + 1);  // [G][P][96][kCntPitch]
  double* sbins = reinterpret_cast<double*>(cnt + (size_t)G * P * 96 * kCntPitch);
  double* acc = sbins + (kMaxBins + 1);                 // [n_bins][n_stats]
  unsigned long long* bcnt =
      reinterpret_cast<unsigned long long*>(acc + (size_t)a.n_bins * a.n_stats);
  int* thr = reinterpret_cast<int*>(bcnt + a.n_bins);   // ceil(bins[k]), integer distances
  multi::Groups<kGW>* groups = reinterpret_cast<multi::Groups<kGW>*>(thr + kMaxBins + 2);  // [G]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &ctrl->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ctrl->full[s], 1);
      mbar_init(&ctrl->empty[s], 1);
    }
    for (int s = 0; s < G; ++s) mbar_init(&ctrl->gfull[s], 1);
    for (int s = 0; s < A; ++s) mbar_init(&ctrl->gempty[s], kGW);
    mbar_init(&ctrl->drain, 1);
    ctrl->abort_flag = 0;
    ctrl->consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ctrl->tmem_base)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int s = 0; s < stages; ++s) {
    uint4* z = reinterpret_cast<uint4*>(ring + (size_t)s * kGStageBytes + kBlkRows * kKChunk);
    for (int k = threadIdx.x; k < (kABytes - kBlkRows * kKChunk) / 16; k += blockDim.x)
      z[k] = make_uint4(0u, 0u, 0u, 0u);
  }
  for (int x = threadIdx.x; x < a.n_bins * a.n_stats; x += blockDim.x) acc[x] = 0.0;
  for (int x = threadIdx.x; x < a.n_bins; x += blockDim.x) bcnt[x] = 0ull;
  for (int x = threadIdx.x; x <= a.n_bins; x += blockDim.x) {
    const double b = a.bins[x], cb = ceil(b);
    sbins[x] = b;
    thr[x] = cb > 2147483647.0 ? 2147483647 : (cb < -2147483647.0 ? -2147483647 : (int)cb);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctrl->tmem_base;

  long long n_items = a.item_off[a.n_blocks];
  if (n_items < 0 || n_items > a.n_blocks * (a.n_blocks + 1) / 2) {
    if (threadIdx.x == 0) set_abort(ctrl, a.status, 4101);
    n_items = 0;
  }

  if (warp == 0) {
    // ---------------- TMA producer: per tile, every population's K chunks ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int issued = 0;
      long long lo = 0;
      bool ok = true;
      for (long long item = blockIdx.x; item < n_items && ok && !*abort_flag; item += gridDim.x) {
        lo = advance_block(a.item_off, a.n_blocks, lo, item);
        const long long jb = lo + (item - a.item_off[lo]);
        for (int p = 0; p < P && ok; ++p)
          for (int kc = 0; kc < a.kchunks; ++kc) {
            if (!mbar_wait_role(&ctrl->empty[stage], phase ^ 1, abort_flag)) {
              set_abort(ctrl, a.status, 4102);
              ok = false;
              break;
            }
            unsigned char* sa = ring + (size_t)stage * kGStageBytes;
            mbar_expect_tx(&ctrl->full[stage], 2 * kBBytes);
            tma_load_2d(sa, &map, &ctrl->full[stage], kc * kKChunk,
                        p * a.pop_rows + (int)(jb * kBlkRows));
            tma_load_2d(sa + kABytes, &map, &ctrl->full[stage], kc * kKChunk,
                        p * a.pop_rows + (int)(lo * kBlkRows));
            ++issued;
            if (++stage == stages) {
              stage = 0;
              phase ^= 1;
            }
          }
      }
      if (*abort_flag) {
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
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int consumed = 0;
      bool any = false, ok = true;
      for (int t = 0; ok && !*abort_flag; ++t) {
        if ((long long)blockIdx.x + (long long)t * gridDim.x >= n_items) break;
        const int sg = t % A;
        const uint32_t tph = (uint32_t)((t / A) & 1);
        if (!mbar_wait_role(&ctrl->gempty[sg], tph ^ 1, abort_flag)) {
          set_abort(ctrl, a.status, 4103);
          break;
        }
        tc_fence_after();
        for (int p = 0; p < P && ok; ++p) {
          const uint32_t d = tmem_base + (uint32_t)sg * kStageCols + (uint32_t)(p * 96);
          for (int kc = 0; kc < a.kchunks; ++kc) {
            if (!mbar_wait_role(&ctrl->full[stage], phase, abort_flag)) {
              set_abort(ctrl, a.status, 4104);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_u32(ring + (size_t)stage * kGStageBytes);
            const uint64_t da = smem_desc(sa), db = smem_desc(sa + kABytes);
#pragma unroll
            for (int k = 0; k < kKChunk / 32; ++k)
              mma_f8_n96(d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), (kc | k) != 0);
            mma_commit(&ctrl->empty[stage]);
            any = true;
            *(volatile int*)&ctrl->consumed = ++consumed;
            if (++stage == stages) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
        if (!ok) break;
        mma_commit(&ctrl->gfull[t % G]);
      }
      if (*abort_flag && any) {
        mma_commit(&ctrl->drain);
        mbar_wait_drain(&ctrl->drain, 0);
      }
    }
  } else if (warp >= 4) {
    // ---------------- epilogue ----------------
    const int e = warp - 4;
    const int grp = e / kGW;
    const int gi = e % kGW;                // warp within the group
    const int wq = warp & 3;               // TMEM lane quarter: plane wq of the SNPs j
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    const uint32_t bar_id = 1u + (uint32_t)grp;
    int16_t* gbuf = cnt + (size_t)grp * P * 96 * kCntPitch;
    const bool use_int = a.bcoord == nullptr && *a.ipos_bad == 0;
    const int maxd_int = a.max_dist >= 2147483647.0 ? 2147483647 : (int)floor(a.max_dist);
    long long lo = 0;
    // one population: a lane's running total (its row and statistic of eight) and,
    // in lanes 0-7, its row's pairs, added to the slots when the bin changes: the
    // rows of a tile mostly share a bin, and eight float64 additions to one slot
    // retry one another
    double v_run = 0.0;
    int v_bin = -1, n_bin = -1, n_run = 0;
    // the tile is ready on the group's own barrier, whose phases the group alone
    // follows (a stage's would pass through other groups' tiles)
    for (int t = grp, u = 0;; t += G, ++u) {
      const int sg = t % A;  // accumulator stage
      const long long item = (long long)blockIdx.x + (long long)t * gridDim.x;
      if (item >= n_items) break;
      bool ready = true;
      if (lane == 0) ready = mbar_wait(&ctrl->gfull[grp], (uint32_t)(u & 1), abort_flag);
      ready = __shfl_sync(0xffffffffu, ready ? 1 : 0, 0) != 0;
      if (!ready && lane == 0) set_abort(ctrl, a.status, 4105);
      // the group meets before overwriting its moment buffers and takes one
      // decision on aborting (bar.red.or over every thread's view)
      uint32_t any_abort = 0;
      const uint32_t mine = (ready ? 0u : 1u) | (uint32_t)(*abort_flag != 0);
      asm volatile(
          "{\n .reg .pred pin, pout;\n setp.ne.u32 pin, %1, 0;\n"
          " bar.red.or.pred pout, %2, %3, pin;\n selp.u32 %0, 1, 0, pout;\n}"
          : "=r"(any_abort)
          : "r"(mine), "r"(bar_id), "r"(kGW * 32)
          : "memory");
      if (any_abort) break;
      tc_fence_after();
      // copy: the warps of lane quarters 0-2 copy plane wq's moments of the
      // populations they own (with two warps per quarter, alternate ones)
      if (wq < 3) {
        const int half = gi >> 2;   // 0 with four warps per group
        for (int p = half; p < P; p += kGW / 4) {
          uint32_t* row = reinterpret_cast<uint32_t*>(gbuf + ((size_t)p * 96 + wq * 32 + lane) * kCntPitch);
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            uint32_t r[3][16];
#pragma unroll
            for (int c = 0; c < 3; ++c)
              tmem_ld16(tmem_base + lane_base +
                            ((uint32_t)sg * kStageCols + (uint32_t)(p * 96 + 48 * h + 16 * c)),
                        r[c]);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
              for (int v = 0; v < 8; ++v)
                row[24 * h + 8 * c + v] =
                    fast::f2i_pair(__uint_as_float(r[c][2 * v]), __uint_as_float(r[c][2 * v + 1]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctrl->gempty[sg]);
      asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(kGW * 32) : "memory");

      lo = advance_block(a.item_off, a.n_blocks, lo, item);
      const long long i0 = lo * kTileSnp, j0 = (lo + (item - a.item_off[lo])) * kTileSnp;
      const long long j = j0 + lane;
      const bool j_ok = j < a.n_snp;
      if constexpr (P > 1) {
        // bins of the warp's rows, then the tile's pairs grouped by bin
        int bin[kRows];
        if (use_int) {
          const int pj = j_ok ? a.ipos[j] : 0;
          const int pi = i0 + lane < a.n_snp ? a.ipos[i0 + lane] : 0;
#pragma unroll
          for (int q = 0; q < kRows; ++q) {
            const int il = gi * kRows + q;
            const int d = pj - __shfl_sync(0xffffffffu, pi, il);
            bin[q] = i0 + il < j && j_ok && d <= maxd_int ? bin_of_int(thr, a.n_bins, d) : -1;
          }
        } else {
          const double pj = j_ok ? a.pos[j] : 0.0;
          const double cj = (j_ok && a.bcoord) ? a.bcoord[j] : 0.0;
#pragma unroll
          for (int q = 0; q < kRows; ++q) {
            const long long i = i0 + gi * kRows + q;
            bin[q] = -1;
            if (i < j && j_ok) {
              const double dpos = pj - a.pos[i];
              if (dpos <= a.max_dist)
                bin[q] = bin_of_f64(sbins, a.n_bins, a.bcoord ? fabs(cj - a.bcoord[i]) : dpos);
            }
          }
        }
        multi::Groups<kGW>& g = groups[grp];
        multi::group_pairs<kGW, kRows>(g, bin, gi * kRows, gi, a.n_bins, bcnt, [&] {
          asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(kGW * 32) : "memory");
        });
        // with two passes over the steps the first takes the term-table pairs
        auto load = [&](int pair, int b, multi::Geno(&f)[P], bool first) {
          gmom::Mom mo[P];
          const int il = (pair >> 5) & 31, jl = pair & 31;
          int n_least = 1 << 20;
#pragma unroll
          for (int p = 0; p < P; ++p) {
            const int16_t* bp = gbuf + (size_t)p * 96 * kCntPitch;
#pragma unroll
            for (int x = 0; x < 3; ++x)
#pragma unroll
              for (int y = 0; y < 3; ++y)
                mo[p].m[3 * x + y] = bp[(y * 32 + jl) * kCntPitch + x * 32 + il];
            n_least = min(n_least, mo[p].m[0]);
          }
          const bool live = pair < multi::kGroupPairs;
          const bool table = live && (n_least < 4 || a.exact);
          if (table && first) term_table_pair<P>(mo, a, acc + b * a.n_stats);
          if (!live || table) {
#pragma unroll
            for (int p = 0; p < P; ++p)
#pragma unroll
              for (int x = 0; x < 9; ++x) mo[p].m[x] = 0;
          }
#pragma unroll
          for (int p = 0; p < P; ++p) f[p] = multi::make_geno(mo[p]);
        };
        const int s0 = g.n_steps * gi / kGW, s1 = g.n_steps * (gi + 1) / kGW;
        multi::sum_steps<P, 0, multi::Geno>(
            g, s0, s1, acc, a.n_stats, pl,
            [&](int pair, int b, multi::Geno(&f)[P]) { load(pair, b, f, true); });
        if constexpr (P == 4)
          multi::sum_steps<P, 1, multi::Geno>(
              g, s0, s1, acc, a.n_stats, pl,
              [&](int pair, int b, multi::Geno(&f)[P]) { load(pair, b, f, false); });
        continue;
      }
      // one population: DD, Dz, pi2 in float32 from the moments
      // (gmom::stats_f32, within 1e-6 relative of each exact value), summed over
      // each row's pairs of a bin; eight rows at a time, whose totals take 24
      // exchanges together instead of 15 each (the sums are the same: every step
      // adds the same two halves)
      const int pj = use_int && j_ok ? a.ipos[j] : 0;
      const int pi = use_int && i0 + lane < a.n_snp ? a.ipos[i0 + lane] : 0;
      const double pj64 = !use_int && j_ok ? a.pos[j] : 0.0;
      const double cj = j_ok && a.bcoord ? a.bcoord[j] : 0.0;
#pragma unroll 1
      for (int k0 = 0; k0 < kRows; k0 += 8) {
        float v[24];
        int bins[8];  // bin of the lane's pair of each row
        unsigned more = 0;  // rows with pairs of another bin than the first
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int il = gi + kGW * (k0 + k);
          const long long i = i0 + il;
          int b = -1;
          if (use_int) {
            const int d = pj - __shfl_sync(0xffffffffu, pi, il);
            if (i < j && j_ok && d <= maxd_int) b = bin_of_int(thr, a.n_bins, d);
          } else if (i < j && j_ok) {
            const double dpos = pj64 - a.pos[i];
            if (dpos <= a.max_dist)
              b = bin_of_f64(sbins, a.n_bins, a.bcoord ? fabs(cj - a.bcoord[i]) : dpos);
          }
          bins[k] = b;
        }
        float4 o4[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int il = gi + kGW * (k0 + k);
          gmom::Mom mo;
#pragma unroll
          for (int x = 0; x < 3; ++x)
#pragma unroll
            for (int y = 0; y < 3; ++y)
              mo.m[3 * x + y] = gbuf[(y * 32 + lane) * kCntPitch + x * 32 + il];
          o4[k] = gmom::stats_f32<14>(mo, 14);
        }
        unsigned pending[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) pending[k] = __ballot_sync(0xffffffffu, bins[k] >= 0);
        do {
          int slot = -1;  // lane k: the bin of row k in this turn
          more = 0;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            v[3 * k] = v[3 * k + 1] = v[3 * k + 2] = 0.f;
            if (!pending[k]) continue;
            const int bb = __shfl_sync(0xffffffffu, bins[k], __ffs(pending[k]) - 1);
            const bool mine = bins[k] == bb;
            const unsigned same = __ballot_sync(0xffffffffu, mine);
            if (mine) {
              v[3 * k] = o4[k].y;
              v[3 * k + 1] = o4[k].z;
              v[3 * k + 2] = o4[k].w;
            }
            if (lane == k) {
              slot = bb;
              if (bb != n_bin) {
                if (n_bin >= 0) atomicAdd(&bcnt[n_bin], (unsigned long long)n_run);
                n_bin = bb;
                n_run = 0;
              }
              n_run += __popc(same);
            }
            pending[k] &= ~same;
            more |= pending[k];
          }
          // lane l: the totals of value multi::halved<24>(0)
          multi::halve_plain<24>(v);
          const int at = multi::halved<24>(0);
          const int bb = __shfl_sync(0xffffffffu, slot, at < 0 ? 0 : at / 3);
          if (at >= 0 && bb >= 0) {
            if (bb != v_bin) {
              if (v_bin >= 0) atomicAdd(&acc[v_bin * 3 + at % 3], v_run);
              v_bin = bb;
              v_run = 0.0;
            }
            v_run += (double)v[0];
          }
        } while (more);
      }
      if (n_run >= 1 << 30) {
        atomicAdd(&bcnt[n_bin], (unsigned long long)n_run);
        n_run = 0;
      }
    }
    if (P == 1) {
      if (v_bin >= 0) atomicAdd(&acc[v_bin * 3 + multi::halved<24>(0) % 3], v_run);
      if (n_bin >= 0 && n_run) atomicAdd(&bcnt[n_bin], (unsigned long long)n_run);
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (!*abort_flag) {
    for (int x = threadIdx.x; x < a.n_bins * a.n_stats; x += blockDim.x)
      if (acc[x] != 0.0) atomicAdd(a.sums + x, acc[x]);
    if (a.pair_counts)
      for (int x = threadIdx.x; x < a.n_bins; x += blockDim.x)
        if (bcnt[x]) atomicAdd(a.pair_counts + x, bcnt[x]);
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(512)
                 : "memory");
  }
}

}  // namespace gtc
}  // namespace pgld

// Genotype band pairs on the tensor cores: one population, dosages 0/1/2
// (missing allowed), no values above 2.  a carries the band and outputs.
int pgld_geno_tc_pairs(pgld_context* h, const pgld_geno_panel* panel, const double* pos,
                       double max_dist, const long long* offsets, int32_t* counts, int32_t* n_valid,
                       float* stats, int32_t stat_mask, cudaStream_t st) {
  using namespace pgld::gtc;
  int rc = pgld::tchost::get_encode(h);
  if (rc) return rc;
  const long long n = panel->n_snp;
  const int W = panel->n_words[0];
  const long long nb = (n + kTileSnp - 1) / kTileSnp;
  if (nb * kBlkRows > 2147483647LL)
    return pgld_fail(h, PGLD_ERR_TOO_LARGE, "genotype tensor-core form: too many SNPs");
  const int k_pad = ((W * 32 + kKChunk - 1) / kKChunk) * kKChunk;
  const size_t op_bytes = (size_t)nb * kBlkRows * k_pad;
  const size_t sb = pgld::scan_scratch_bytes(std::max<long long>(nb, n));
  auto al = [](size_t x) { return (x + 1023) & ~size_t(1023); };
  const size_t off_items = 0, off_scan = al((nb + 1) * 8), off_op = off_scan + al(sb),
               off_poff = off_op + al(op_bytes),
               total = off_poff + (offsets ? 0 : al((size_t)(n + 1) * 8));
  void* ws = nullptr;
  rc = pgld_workspace(h, total, &ws);
  if (rc) return rc;
  char* w = (char*)ws;
  long long* items = (long long*)(w + off_items);
  unsigned char* op = (unsigned char*)(w + off_op);
  const long long* poff = offsets;
  if (!poff) {
    poff = (long long*)(w + off_poff);
    rc = pgld_band_offsets(h, pos, n, max_dist, (long long*)(w + off_poff), w + off_scan, sb, st);
    if (rc) return rc;
  }
  {
    pack_gtc_kernel<<<pack_gtc_blocks(h, nb), 256, 0, st>>>(panel->planes[0], W, n, nb, k_pad, (uint32_t*)op);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return pgld_cuda_fail(h, e, "pack_gtc_kernel");
  }
  rc = pgld::band_schedule(h, pos, n, max_dist, items, w + off_scan, sb, st, kTileSnp);
  if (rc) return rc;
  CUtensorMap map;
  rc = pgld::tchost::make_map(h, &map, op, nb * kBlkRows, k_pad, kBlkRows);
  if (rc) return rc;
  Params prm{};
  prm.kchunks = k_pad / kKChunk;
  prm.n_snp = n;
  prm.item_off = items;
  prm.n_blocks = nb;
  prm.pair_off = poff;
  prm.counts = counts;
  prm.nvalid = n_valid;
  prm.stats = stats;
  prm.stat_mask = stat_mask;
  prm.status = h->dev_status;
  int max_smem = 0;
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
  // the resident form when the row block (every K chunk) fits beside at least
  // four 16 KB A stages, with as many epilogue groups as leave six: a copy
  // takes about 1.6 us under load, so the stages in flight set the pace of long
  // rows (1,000 individuals, 1.0e8 pairs: two groups and six stages 2.17 ms, three
  // and five 2.24, four and four 2.31; short rows are bound by the statistics,
  // which four groups do in 1.39 ms at 250 individuals)
  const long long res_bytes = (long long)prm.kchunks * kBBytes;
  auto fixed = [](int g) { return (long long)kCtrlBytes + 1024 + g * (kMomBytes + 4ll * kCountStage); };
  auto ring = [&](int g, long long resident, int stage) {
    return (int)std::min<long long>(8, (max_smem - fixed(g) - resident) / stage);
  };
  int g = kMaxGroups;
  while (g > 2 && ring(g, res_bytes, kABytes) < 6) --g;
  const bool res = ring(g, res_bytes, kABytes) >= 4;
  if (!res) g = 3;
  const int stages = res ? ring(g, res_bytes, kABytes) : ring(g, 0, kGStageBytes);
  if (stages < 2) return pgld_fail(h, PGLD_ERR_TOO_LARGE, "genotype tensor-core form: shared memory");
  prm.stages = stages;
  prm.groups = g;
  const size_t smem =
      (size_t)fixed(g) + (res ? (size_t)stages * kABytes + (size_t)res_bytes : (size_t)stages * kGStageBytes);
  // the two column sets of the band workloads get their own instantiation
  void (*kern)(CUtensorMap, Params);
  if (res)
    kern = !stats ? gtc_pairs_kernel<0, true>
           : stat_mask == 3 ? gtc_pairs_kernel<3, true>
           : stat_mask == 15 ? gtc_pairs_kernel<15, true>
                             : gtc_pairs_kernel<-1, true>;
  else
    kern = !stats ? gtc_pairs_kernel<0, false>
           : stat_mask == 3 ? gtc_pairs_kernel<3, false>
           : stat_mask == 15 ? gtc_pairs_kernel<15, false>
                             : gtc_pairs_kernel<-1, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "gtc smem attribute");
  pgld_time_begin(h, st);
  kern<<<(unsigned)h->n_sm, (4 + 4 * g) * 32, smem, st>>>(map, prm);
  pgld_time_end(h, st);
  e = cudaGetLastError();
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "gtc_pairs_kernel");
  return PGLD_OK;
}

int pgld_tc_int_positions(pgld_context* h, const double* pos, long long n, int* ipos, int* bad,
                          cudaStream_t st);

// Genotype distance-binned sums on the tensor cores: 1-4 populations of
// dosages 0/1/2 (missing allowed, no values above 2), at most kMaxGenoN
// individuals each; ba carries the bins, term table and outputs (sums and
// pair counts already zeroed).
int pgld_geno_tc_binned(pgld_context* h, const pgld_geno_panel* panel, const pgld::BandArgs& ba,
                        cudaStream_t st) {
  using namespace pgld::gtc;
  int rc = pgld::tchost::get_encode(h);
  if (rc) return rc;
  const int P = panel->n_pops;
  const long long n = panel->n_snp;
  const long long nb = (n + kTileSnp - 1) / kTileSnp;
  int W = 0;
  for (int p = 0; p < P; ++p) W = std::max(W, panel->n_words[p]);
  if ((long long)P * nb * kBlkRows > 2147483647LL)
    return pgld_fail(h, PGLD_ERR_TOO_LARGE, "genotype tensor-core binned form: too many SNPs");
  const int k_pad = ((W * 32 + kKChunk - 1) / kKChunk) * kKChunk;
  const size_t op_pop = (size_t)nb * kBlkRows * k_pad;
  const size_t sb = pgld::scan_scratch_bytes(nb);
  auto al = [](size_t x) { return (x + 1023) & ~size_t(1023); };
  const size_t off_items = 0, off_scan = al((nb + 1) * 8), off_op = off_scan + al(sb),
               off_ipos = off_op + al(op_pop * P), off_bad = off_ipos + al((size_t)n * 4),
               total = off_bad + 1024;
  void* ws = nullptr;
  rc = pgld_workspace(h, total, &ws);
  if (rc) return rc;
  char* w = (char*)ws;
  long long* items = (long long*)(w + off_items);
  unsigned char* op = (unsigned char*)(w + off_op);
  for (int p = 0; p < P; ++p) {
    pack_gtc_kernel<<<pack_gtc_blocks(h, nb), 256, 0, st>>>(panel->planes[p], panel->n_words[p], n, nb, k_pad,
                                            (uint32_t*)(op + op_pop * p));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return pgld_cuda_fail(h, e, "pack_gtc_kernel");
  }
  rc = pgld::band_schedule(h, ba.pos, n, ba.max_dist, items, w + off_scan, sb, st, kTileSnp);
  if (rc) return rc;
  int* ipos = (int*)(w + off_ipos);
  int* ipos_bad = (int*)(w + off_bad);
  rc = pgld_tc_int_positions(h, ba.pos, n, ipos, ipos_bad, st);
  if (rc) return rc;
  CUtensorMap map;
  rc = pgld::tchost::make_map(h, &map, op, (long long)P * nb * kBlkRows, k_pad, kBlkRows);
  if (rc) return rc;
  BParams prm{};
  prm.kchunks = k_pad / kKChunk;
  prm.n_snp = n;
  prm.item_off = items;
  prm.n_blocks = nb;
  prm.n_pops = P;
  prm.pop_rows = (int)(nb * kBlkRows);
  prm.pos = ba.pos;
  prm.bcoord = ba.bcoord;
  prm.ipos = ipos;
  prm.ipos_bad = ipos_bad;
  prm.max_dist = ba.max_dist;
  prm.bins = ba.bins;
  prm.n_bins = ba.n_bins;
  prm.exact = 32 * W > pgld::multi::kMaxN;
  prm.terms = ba.terms;
  prm.n_terms = ba.n_terms;
  prm.n_stats = ba.n_stats;
  prm.sums = ba.sums;
  prm.pair_counts = reinterpret_cast<unsigned long long*>(ba.pair_counts);
  prm.status = h->dev_status;
  const int G = P == 1 ? Binned<1>::G : P == 2 ? Binned<2>::G : P == 3 ? Binned<3>::G : Binned<4>::G;
  const int threads = P == 1   ? Binned<1>::kThreads
                      : P == 2 ? Binned<2>::kThreads
                      : P == 3 ? Binned<3>::kThreads : Binned<4>::kThreads;
  const size_t group_bytes = P == 1 ? 0 : G * sizeof(pgld::multi::Groups<8>);
  const size_t fixed = sizeof(GCtrl) + (size_t)G * P * 96 * kCntPitch * 2 +
                       (size_t)(pgld::kMaxBins + 1) * 8 + (size_t)ba.n_bins * ba.n_stats * 8 +
                       (size_t)ba.n_bins * 8 + (size_t)(pgld::kMaxBins + 2) * 4 + group_bytes + 1024;
  int max_smem = 0;
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
  const int stages =
      (int)std::min<long long>(8, ((long long)max_smem - (long long)fixed) / kGStageBytes);
  if (stages < 2)
    return pgld_fail(h, PGLD_ERR_TOO_LARGE, "genotype tensor-core binned form: shared memory");
  prm.stages = stages;
  const size_t smem = (size_t)stages * kGStageBytes + fixed;
  void (*kern)(CUtensorMap, BParams, pgld::multi::Places) =
      P == 1 ? gtc_binned_kernel<1> : P == 2 ? gtc_binned_kernel<2>
      : P == 3 ? gtc_binned_kernel<3> : gtc_binned_kernel<4>;
  const pgld::multi::Places pl = P > 1 ? pgld::multi::places(P, true) : pgld::multi::Places{};
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "gtc binned smem attribute");
  pgld_time_begin(h, st);
  kern<<<(unsigned)h->n_sm, threads, smem, st>>>(map, prm, pl);
  pgld_time_end(h, st);
  e = cudaGetLastError();
  if (e != cudaSuccess) return pgld_cuda_fail(h, e, "gtc_binned_kernel");
  return PGLD_OK;
}
