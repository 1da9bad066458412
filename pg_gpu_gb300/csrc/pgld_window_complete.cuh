// State and tile order shared by the window kernels of complete lists
// (pgld_window_complete.cu) and of others (pgld_tc_wide.cu).
#pragma once
#include <stdint.h>

#include <functional>

namespace pgld {
namespace wcomp {

struct State {
  int complete;       // every listed SNP has the first one's valid haplotypes
  int n;              // how many those are
  uint32_t mask[64];
};

// upper-triangle tiles of a window, the columns of a tile twice its rows: row
// block b of a window of C column blocks holds the column blocks b / 2 .. C - 1;
// the tiles before row block b
__host__ __device__ __forceinline__ long long tiles_before(long long b, long long C) {
  const long long k = b >> 1;
  return b * C - ((b & 1) ? k * k : k * (k - 1));
}

// the row block b < R of the window's tile t and the tiles before it: for even
// b, tiles_before = b C - b^2 / 4 + b / 2, whose root in b, (2C + 1) -
// sqrt((2C + 1)^2 - 4 t), starts the search; the steps make it exact
// (tiles_before rises by C - floor(b / 2) >= 1 per row block)
__device__ __forceinline__ void row_block(long long t, long long R, long long C, long long& b,
                                          long long& first) {
  const long long c2 = 2 * C + 1;
  const float disc = (float)(c2 * c2 - 4 * t);
  b = (long long)((float)c2 - sqrtf(disc > 0.f ? disc : 0.f));
  b = b < 0 ? 0 : (b > R - 1 ? R - 1 : b);
  while (b > 0 && tiles_before(b, C) > t) --b;
  while (b + 1 < R && tiles_before(b + 1, C) <= t) ++b;
  first = tiles_before(b, C);
}

}  // namespace wcomp
}  // namespace pgld

struct pgld_context;
int pgld_window_complete_pack(pgld_context* h, const uint32_t* planes, int W, long long n_snp,
                              long long n_idx, const int32_t* idx, pgld::wcomp::State* state,
                              unsigned char* op, float2* site, cudaStream_t st);
int pgld_window_complete_sums(pgld_context* h, const pgld::wcomp::State* state, int W,
                              long long n_idx, const unsigned char* op, const float2* site,
                              const long long* wb, const long long* we, int n_win,
                              const long long* tile_off, double* sums, unsigned long long* counts,
                              int columns, cudaStream_t st, std::function<int()>* launch);
