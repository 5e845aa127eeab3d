// rank.cuh -- shared by the ranks' kernels (rank.cu, rank_local.cu).
#pragma once
#include "gcvl.cuh"

namespace gcvl {

// Keys as unsigned integers in rank order (nesl/cvl/serial/rank.c:94-99, 258-280).
__device__ __forceinline__ unsigned long long rk_key(unsigned long long b, int up) {
  unsigned long long k = (b >> 63) ? ~b : (b ^ (1ULL << 63));
  return up ? k : ~k;
}
__device__ __forceinline__ unsigned rk_key(unsigned x, int up) { return x ^ (up ? 0x80000000u : 0x7FFFFFFFu); }

// The tile of a local rank's CTA: the segments that start in LR_T elements,
// each of at most LR_MAX, so at most LR_CAP elements.
constexpr int LR_BLOCK = 512, LR_T = 2048, LR_MAX = 2048, LR_CAP = LR_T + LR_MAX;
inline int lr_tiles(long n) { return (int)((n + LR_T - 1) / LR_T); }

// Segments too long for one CTA, numbered in the order they were met and
// laid one after another in a compacted vector.
struct LongSegs {
  unsigned long long *total;  // how many << 32 | their elements
  int *first;                 // by number: first element
  int *base;                  // by number: first place in the compacted vector
  int *of_tile;               // by tile: number of the long segment that starts there, or -1 (at most one: LR_MAX >= LR_T)
};
static_assert(LR_MAX >= LR_T, "at most one long segment starts in a tile");

// Ranks of the segments of at most LR_MAX elements; the longer ones are
// registered in ls (ls.total starts at zero).  whole: all n <= LR_CAP
// elements in one CTA, no long segments, ls unused (n or the number of
// segments at most LR_T).
template <class K>
void rank_local(const void *src, int *rank, const SegView &sv, int n, int up, bool whole, const LongSegs &ls);

}  // namespace gcvl
