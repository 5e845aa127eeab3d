// rank_warp.cuh -- the ranks of a warp's elements among those with their
// digit, in element order (the digit passes of rank.cu).
//
// Only warp intrinsics and shared-memory atomics are used, and no include, so
// that the step also runs on the host with lanes that take turns in any order.
#pragma once

// What orders the lanes: every access of one lane that another lane relies on
// has a __syncwarp() (or a shuffle, vote or ballot) between the two.  Lanes of
// a warp need not run in step, even after a branch that they left together.
//
// Item c of lane l is element 32 c + l of the warp.  wr[c] becomes
// rank << 8 | digit, the rank among the warp's elements of that digit, in
// element order.  cnt: the warp's [256] counts, zero before, the digits'
// totals afterwards.  mask: the warp's lane masks, one word a digit, those of
// item u of a group `stride` words on; zero before and afterwards.
//
// An item's peers (the lanes with its digit) come from a lane mask per digit
// in shared memory: every lane sets its bit, reads the mask back, and the
// first peer counts for all and clears it; G items at a time with masks of
// their own, so that their accesses are in flight together.  Eight ballots an
// item (four ALU instructions a bit) kept the ALU busy and the shared-memory
// pipe idle: a pass over 2^26 keys 406 us, now 370 us with the shared-memory
// pipe 77 % busy.  Ballots for one, two or three of every five items changed
// nothing or lost; counting without masks and ordering the lanes that share a
// digit afterwards took 4 % more.  An item whose lanes all hold one digit
// skips the masks: 32 adds to one word take turns (2^25 keys of two values
// 1217 -> 961 us, 1183 with the ballots; random keys pay 1.5 %).
template <int ITEMS, int G, class K>
__device__ __forceinline__ void warp_digit_ranks(unsigned (&wr)[ITEMS], const K (&key)[ITEMS], int shift,
                                                 unsigned *cnt, unsigned *mask, int stride, int lane) {
  static_assert(ITEMS % G == 0, "whole groups");
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int c0 = 0; c0 < ITEMS; c0 += G) {
    unsigned m[G];
    bool one[G];  // all lanes hold the same digit
#pragma unroll
    for (int u = 0; u < G; u++) {
      const unsigned d = (unsigned)(key[c0 + u] >> shift) & 255u;
      one[u] = __all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0));
      if (!one[u]) atomicOr(mask + u * stride + d, 1u << lane);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < G; u++) {
      m[u] = 0xffffffffu;
      if (!one[u]) m[u] = mask[u * stride + ((unsigned)(key[c0 + u] >> shift) & 255u)];
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < G; u++) {
      const unsigned d = (unsigned)(key[c0 + u] >> shift) & 255u;
      unsigned r = 0;
      if ((m[u] & lt) == 0) {
        r = atomicAdd(cnt + d, (unsigned)__popc(m[u]));
        mask[u * stride + d] = 0;
      }
      wr[c0 + u] = r;
      __syncwarp();  // the next item's first peer of this digit is another lane
    }
#pragma unroll
    for (int u = 0; u < G; u++) {
      const unsigned d = (unsigned)(key[c0 + u] >> shift) & 255u;
      wr[c0 + u] = ((__shfl_sync(0xffffffffu, wr[c0 + u], __ffs(m[u]) - 1) + (unsigned)__popc(m[u] & lt)) << 8) | d;
    }
  }
}
