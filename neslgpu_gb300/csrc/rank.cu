// rank.cu -- stable radix rank, up and down, int and double, segmented and
// unsegmented (nesl/cvl/serial/rank.c:49-362), and the partitioned scatter
// that large permutes share with it.
//
// d[j] is the position of element j in the stable sorted order of its
// segment.  Keys are made order-preserving unsigned integers exactly as the
// serial CVL does: int keys flip the sign bit (up) or every other bit
// (down), rank.c:94-99; double keys flip all bits of negatives and the sign
// bit of the rest, and down ranks complement that, rank.c:258-280.  The
// digit passes rank long segments as a stable sort by (segment, key): the
// key passes carry each element's segment number, then further passes sort
// by it.
//
// GPU design.  Segments of at most LR_MAX elements, and whole vectors of at
// most LR_CAP, are ranked by one CTA each (rank_local.cu).  Longer vectors,
// and the compacted long segments of a segmented rank, are sorted onesweep
// style.  One prepare pass builds every pass's 256-bin digit histogram at
// once with shared-memory atomics (and compacts the long segments' keys,
// indices and segment numbers).  Then one pass per 8-bit digit: each warp of
// a CTA loads its 32 x ITEMS consecutive keys and values into registers,
// ranks them stably by lane masks, the CTA learns how many earlier tiles'
// elements fall in each digit by a per-digit decoupled look-back, reorders
// the tile in shared memory and writes coalesced runs.  The first pass of an
// unsegmented rank reads the caller's keys and transforms them itself.
//
// The result is the inverse of the sort permutation: rank[index] = position,
// a scatter to random places.  Below RK_DIRECT_MAX elements the last pass
// writes it directly (the rank vector fits in L2, which absorbs the random
// writes).  Above it the last pass writes each (index, position) pair
// grouped by the top 8 bits of the index -- 256 windows of the output, each
// element's slot from a second per-window look-back in the same pass -- and
// a streaming kernel writes each window's ranks while the window sits in
// L2, so DRAM sees whole sectors instead of a read-modify-write per 4-byte
// element.  Large permutes and gathers (smp_pu*, bck_pu*, the default and
// flag permutes) split their pairs by window with passes of their own (the
// window split below) and share the window scatter.
#include "gcvl.cuh"
#include "rank.cuh"
#include "rank_warp.cuh"

#include <algorithm>
#include <type_traits>
#include <utility>

namespace gcvl {

// Keys per thread of a digit pass (tile = 256 x RK_ITEMS), and the CTAs per
// SM of the 32-bit unsegmented passes, measured at 2^28 (int / double /
// segmented int rank, every pass over all elements): 16 items at 4 CTAs 9.09 /
// 21.4 / 18.0 ms; 20 at 3 9.06 / 19.8 / 17.2; 24 at 3 9.43 / 18.7 / 17.0; 32 at
// 2 10.1 / 25.9 / 21.9.  Now 8.39 / 19.5 ms; segmented, int / double, by log-normal
// lengths 14.9 / 25.0 (17.8 / 29.0 then), in segments of 20000, all of them
// long, 17.0 / 30.0 (16.2 / 27.4: there the compaction comes on top).
#ifndef GCVL_RK_ITEMS
#define GCVL_RK_ITEMS 20
#endif
constexpr int RK_BLOCK = 256, RK_ITEMS_LARGE = GCVL_RK_ITEMS;
constexpr int RK_WARPS = RK_BLOCK / 32;
constexpr int RK_MAXPASS = 12;
#ifndef GCVL_RK_LB
#define GCVL_RK_LB 4
#endif
// Resident CTAs per SM the register allocation must allow: 32-bit keys
// without segment numbers fit 64 registers (the pass holds its keys and
// values in registers); 64-bit keys and segmented passes would spill there.
#ifndef GCVL_RK_MINB
#define GCVL_RK_MINB 2
#endif
#ifndef GCVL_RK_MINB_NARROW
#define GCVL_RK_MINB_NARROW 3
#endif
// Shorter vectors take smaller tiles, so that more CTAs work.  Int / double
// ranks in tiles of 20, 16 and 8 items a thread, us: 2^21 keys 108 / 244, 121 /
// 232; 2^20 95 / 176, 79 / 150, 88 / 173; 2^18 67 / 117, 59 / 102, 55 / 100;
// 2^13 50 / 91, 41 / 78, 33 / 60.
constexpr int RK_ITEMS_SMALL = 16, RK_SMALL_MAX = 1 << 20, RK_ITEMS_TINY = 8, RK_TINY_MAX = 1 << 18;
constexpr int RK_LB = GCVL_RK_LB;  // predecessors read per look-back round trip
constexpr int RK_DIRECT_MAX = 1 << 23;
// 8 measured best at 2^28 (bck_puz / smp_puz): 4 items 2.87 / 2.94 ms,
// 8 items 2.63 / 2.78, 16 items 3.01 / 2.78
#ifndef GCVL_SC_ITEMS
#define GCVL_SC_ITEMS 8
#endif
constexpr int SC_ITEMS = GCVL_SC_ITEMS;  // elements per thread in the window and streaming passes
constexpr unsigned RK_INC = 0x80000000u;

// where a pass gets its tile from, and where it puts it
enum { IN_ARRAYS = 0, IN_SRC = 1 };                    // IN_SRC: caller's keys, value = position
// OUT_RANK: rank[v] = pos; OUT_WIN: (v, pos) grouped by the output window of
// v (the partition of the inverse scatter)
enum { OUT_ARRAYS = 0, OUT_RANK = 1, OUT_WIN = 3 };

__host__ __device__ inline int bit_length(unsigned x) {
  int b = 0;
  while (x) { b++; x >>= 1; }
  return b;
}

__device__ __forceinline__ int key_digit(unsigned long long k, int q) { return (int)((k >> (8 * q)) & 255); }

// Every key pass's 256-bin digit histogram of the caller's keys, in one read
// of them, and the cleared look-back words of all passes.
template <class K>
__global__ void __launch_bounds__(RK_BLOCK) k_rank_prep(const K *__restrict__ src, int n, int up,
                                                        unsigned *__restrict__ hist, uint4 *__restrict__ state,
                                                        long state_vecs) {
  constexpr int P = sizeof(K);
  __shared__ unsigned s_hist[P * 256];
  for (int i = threadIdx.x; i < P * 256; i += RK_BLOCK) s_hist[i] = 0;
  const long stride = (long)gridDim.x * RK_BLOCK;
  long i = (long)blockIdx.x * RK_BLOCK + threadIdx.x;
  for (long w = i; w < state_vecs; w += stride) state[w] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  // four independent loads in flight per thread
  for (; i < n; i += 4 * stride) {
    K r[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i + u * stride < n) r[u] = rk_key(__ldcs(src + i + u * stride), up);
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i + u * stride < n)
#pragma unroll
        for (int q = 0; q < P; q++) atomicAdd(&s_hist[q * 256 + key_digit(r[u], q)], 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < P * 256; b += RK_BLOCK)
    if (s_hist[b]) atomicAdd(&hist[b], s_hist[b]);
}

// The long segments of a segmented rank: their keys, indices and segment
// numbers into the compacted vector, the digit histograms of the key and the
// segment-number passes, and the cleared look-back words of the compacted
// vector's tiles.  A tile of LR_T elements holds at most two pieces of long
// segments: the rest of one that started earlier and the start of another.
// Returns at once when there are none.
template <class K>
__global__ void __launch_bounds__(RK_BLOCK) k_rank_prep_long(const K *__restrict__ src, int n, int up, SegView sv,
                                                             LongSegs ls, int seg_passes, K *__restrict__ key,
                                                             unsigned *__restrict__ idx, unsigned *__restrict__ aux,
                                                             unsigned *__restrict__ hist, unsigned *__restrict__ state,
                                                             long state_words, int tile_elems) {
  constexpr int P = sizeof(K);
  __shared__ unsigned s_hist[RK_MAXPASS * 256];
  __shared__ int s_num[2], s_from[2], s_to[2];
  const long total = (long)(unsigned)*(volatile const unsigned long long *)ls.total;
  if (total == 0) return;
  const int tid = threadIdx.x, bins = (P + seg_passes) * 256;
  for (int i = tid; i < bins; i += RK_BLOCK) s_hist[i] = 0;
  const long words = (total + tile_elems - 1) / tile_elems * 256;
  for (long w = (long)blockIdx.x * RK_BLOCK + tid; w < 3 * words; w += (long)gridDim.x * RK_BLOCK)
    state[w / words * state_words + w % words] = 0;
  const int tiles = (int)(((long)n + LR_T - 1) / LR_T);
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    __syncthreads();
    const int lo = t * LR_T, hi = (int)min((long)lo + LR_T, (long)n);
    if (tid < 2) {
      int num = -1, a = 0, b = 0;
      if (tid == 0) {  // the segment that covers the tile's first element, if it started earlier
        const int s = seg_of(sv, lo), o = __ldg(sv.off + s), e = __ldg(sv.off + s + 1);
        if (o < lo && e - o > LR_MAX) { num = ls.of_tile[o / LR_T]; a = lo; b = min(e, hi); }
      } else if ((num = ls.of_tile[t]) >= 0) {
        a = ls.first[num];
        b = hi;  // longer than a tile: at least up to the next tile
      }
      s_num[tid] = num; s_from[tid] = a; s_to[tid] = b;
    }
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < 2; p++) {
      const int num = s_num[p];
      if (num < 0) continue;
      const int first = ls.first[num], base = ls.base[num];
      for (int i = s_from[p] + tid; i < s_to[p]; i += RK_BLOCK) {
        const K k = rk_key(__ldcs(src + i), up);
        const int c = base + (i - first);
        key[c] = k;
        idx[c] = (unsigned)i;
        aux[c] = (unsigned)num;
#pragma unroll
        for (int q = 0; q < P; q++) atomicAdd(&s_hist[q * 256 + key_digit(k, q)], 1u);
      }
      if (tid == 0)
        for (int q = 0; q < seg_passes; q++)
          atomicAdd(&s_hist[(P + q) * 256 + ((num >> (8 * q)) & 255)], (unsigned)(s_to[p] - s_from[p]));
    }
  }
  __syncthreads();
  for (int i = tid; i < bins; i += RK_BLOCK)
    if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// d[idx[i]] = s[i] when the indices ascend (gate word zero): the stores of a
// warp then fall on few lines, and no partition is needed
template <class V>
__global__ void __launch_bounds__(RK_BLOCK) k_sorted_scatter(V *__restrict__ d, const V *__restrict__ s,
                                                             const int *__restrict__ idx, long n,
                                                             const unsigned *__restrict__ gate) {
  if (*(const volatile unsigned *)gate) return;
  for (long i0 = (long)blockIdx.x * (RK_BLOCK * SC_ITEMS) + threadIdx.x; i0 < n;
       i0 += (long)gridDim.x * (RK_BLOCK * SC_ITEMS)) {
    int k[SC_ITEMS];
    V v[SC_ITEMS];
#pragma unroll
    for (int u = 0; u < SC_ITEMS; u++) {
      const long i = i0 + (long)u * RK_BLOCK;
      if (i < n) { k[u] = __ldcs(idx + i); v[u] = __ldcs(s + i); }
    }
#pragma unroll
    for (int u = 0; u < SC_ITEMS; u++) {
      const long i = i0 + (long)u * RK_BLOCK;
      if (i < n) d[k[u]] = v[u];
    }
  }
}

template <class K, class V> struct PassArgs {
  const K *kin; const V *vin; const unsigned *ain;
  K *kout; V *vout; unsigned *aout;
  const void *src; int up;            // IN_SRC: the caller's keys
  int *rank; const int *segbase;      // OUT_RANK / OUT_WIN (segment passes: the segments' first places)
  unsigned *pidx, *ppos;              // OUT_WIN
  const unsigned *hist;               // this pass's digit counts
  unsigned *state;                    // [tiles][256] look-back words
  unsigned *clear;                    // another pass's look-back words, cleared for a later one
  unsigned *wstate;                   // OUT_WIN: [tiles][256] look-back words of the window counts
  int wshift;                         // OUT_WIN: window of v = v >> wshift
  unsigned *counter;
  int n, shift;
  unsigned *status, *gave_up;         // gave_up: marked RK_STOP when a wait of this pass runs out
  int spin_limit;
};

template <class K, class V, bool AUX, int ITEMS> constexpr size_t pass_smem() {
  return (size_t)RK_BLOCK * ITEMS * (sizeof(K) + sizeof(V) + (AUX ? 4 : 0)) + RK_WARPS * 256 * 4 + 256 * 4 + 256 * 8;
}

// A wait of this call gave up: noted for the host, and in a word of the call's
// own.  What a pass writes after that stays inside its outputs (a prefix only
// comes out too small), but places are left unwritten, so no later pass of the
// call may take its output for indices.  The word is cleared with the call's
// tickets; the status word stays set until the host reads it, and the calls
// that come before then are carried out.
constexpr unsigned RK_STOP = 0x80000000u;
__device__ __forceinline__ void rk_give_up(unsigned *status, unsigned *gave_up) {
  atomicOr(status, DEV_TIMEOUT);
  atomicOr(gave_up, RK_STOP);
}

// Publish this tile's count of one bin (digit or window), then look back for
// the earlier tiles' total.  One 32-bit word per (tile, bin): 0 = not yet,
// 1 + count = this tile's count (aggregate), RK_INC | prefix = the bin's
// count in this and all earlier tiles (inclusive; < 2^31 because n is an
// int).  RK_LB predecessors per round trip, nearest first, until an
// inclusive count is found (bounded waits).  Each word is self-contained, so
// relaxed loads suffice and all RK_LB are in flight together; a warp's loads
// of one predecessor are one 128-byte line.
__device__ __forceinline__ unsigned bin_lookback(unsigned *state, int tile, int bin, unsigned tot,
                                                 unsigned *status, unsigned *gave_up, int spin_limit) {
  unsigned *stw = state + (long)tile * 256 + bin;
  if (tile == 0) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(stw), "r"(RK_INC | tot) : "memory");
    return 0;
  }
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(stw), "r"(1u + tot) : "memory");
  unsigned prefix = 0;
  long t0 = tile - 1;
  bool done = false;
  while (!done && t0 >= 0) {
    unsigned w[RK_LB];
#pragma unroll
    for (int j = 0; j < RK_LB; j++) {
      w[j] = RK_INC;  // beyond tile 0: an inclusive zero
      if (t0 - j >= 0)
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(w[j]) : "l"(state + (t0 - j) * 256 + bin) : "memory");
    }
#pragma unroll
    for (int j = 0; j < RK_LB; j++) {
      if (done) break;
      int it = 0;
      while (w[j] == 0) {
        if (++it >= spin_limit) { rk_give_up(status, gave_up); w[j] = RK_INC; break; }
        __nanosleep(32);
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(w[j]) : "l"(state + (t0 - j) * 256 + bin) : "memory");
      }
      if (w[j] & RK_INC) { prefix += w[j] & ~RK_INC; done = true; }
      else prefix += w[j] - 1u;
    }
    t0 -= RK_LB;
  }
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(stw), "r"(RK_INC | (prefix + tot)) : "memory");
  return prefix;
}

// Equal digits keep their order (each warp ranks its elements in element order).
template <class K, bool AUX> constexpr int rk_minb() { return sizeof(K) == 4 && !AUX ? GCVL_RK_MINB_NARROW : GCVL_RK_MINB; }
template <class K, class V, bool AUX, int IN, int OUT, int ITEMS>
__device__ __forceinline__ void radix_tile(const PassArgs<K, V> &a, const int n, const int tile) {
  constexpr int RK_ITEMS = ITEMS, RK_TILE = RK_BLOCK * ITEMS;
  // 32-bit keys and values leave the reorder as one 8-byte pair
  constexpr bool PAIR = sizeof(K) == 4 && sizeof(V) == 4 && OUT == OUT_ARRAYS;
  extern __shared__ __align__(16) unsigned char rk_smem[];
  // the reordered tile (the input stays in registers)
  long long *s_gb = (long long *)rk_smem;                  // [256] global base per digit
  K *s_kout = (K *)(s_gb + 256);
  V *s_vout = (V *)(s_kout + RK_TILE);
  uint2 *s_pair = (uint2 *)s_kout;                         // PAIR: [RK_TILE] (key, value)
  unsigned *s_aout = (unsigned *)(s_vout + RK_TILE);
  unsigned *s_loc = s_aout + (AUX ? RK_TILE : 0);          // [256] tile offset per digit
  unsigned *s_cnt = s_loc + 256;                           // [RK_WARPS][256]
  __shared__ unsigned s_ws[RK_WARPS], s_hs[RK_WARPS];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < RK_WARPS * 256; i += RK_BLOCK) s_cnt[i] = 0;
  for (int i = tid; i < RK_ITEMS / 4 * RK_WARPS * 256 / 4; i += RK_BLOCK)
    ((uint4 *)s_kout)[i] = make_uint4(0, 0, 0, 0);  // the lane masks
  __syncthreads();
  const long base = (long)tile * RK_TILE;
  const int valid = (int)min((long)RK_TILE, (long)n - base);

  // each warp's 32 * RK_ITEMS consecutive elements straight into registers
  // (element wbase + 32c + lane in item c: coalesced, every load in flight)
  const int wbase = warp * 32 * RK_ITEMS;
  K kr[RK_ITEMS];
  V vr[RK_ITEMS];
  unsigned ar[AUX ? RK_ITEMS : 1];
#pragma unroll
  for (int c = 0; c < RK_ITEMS; c++) {
    const int e = wbase + c * 32 + lane;
    // past the vector's end: the largest digit, ranked behind the tile's own
    kr[c] = ~(K)0;
    vr[c] = 0;
    if (AUX) ar[c] = 0;
    if (e < valid) {
      if constexpr (IN == IN_SRC) {
        kr[c] = rk_key(__ldcs((const K *)a.src + base + e), a.up);
        vr[c] = (V)(base + e);
      } else {
        kr[c] = __ldcs(a.kin + base + e);
        vr[c] = __ldcs(a.vin + base + e);
        if (AUX) ar[c] = __ldcs(a.ain + base + e);
      }
    }
  }

  // the ranks within each warp's elements, by lane masks where the tile is reordered later
  constexpr int G = RK_ITEMS / 4;  // [G][RK_WARPS][256] masks
  static_assert((size_t)G * RK_WARPS * 256 * 4 <= (size_t)RK_TILE * (sizeof(K) + sizeof(V)),
                "the masks fit where the tile is reordered");
  unsigned wr[RK_ITEMS];
  warp_digit_ranks<RK_ITEMS, G>(wr, kr, a.shift, s_cnt + warp * 256, (unsigned *)s_kout + warp * 256, RK_WARPS * 256,
                                lane);
  __syncthreads();

  // per digit: tile count, per-warp exclusive offsets
  const int dd = tid;  // RK_BLOCK == 256 digits
  if (OUT == OUT_ARRAYS && a.clear) a.clear[(long)tile * 256 + dd] = 0;
  unsigned tot = 0;
#pragma unroll
  for (int w = 0; w < RK_WARPS; w++) {
    unsigned c = s_cnt[w * 256 + dd];
    s_cnt[w * 256 + dd] = tot;
    tot += c;
  }
  const unsigned prefix = bin_lookback(a.state, tile, dd, tot, a.status, a.gave_up, a.spin_limit);
  // exclusive scans over the digits of the tile's counts -> tile offsets,
  // and of the vector's counts -> digit starts
  {
    const unsigned all = __ldg(a.hist + dd);
    unsigned incl = tot, hincl = all;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned x = shfl_up(incl, o), y = shfl_up(hincl, o);
      if (lane >= o) { incl += x; hincl += y; }
    }
    if (lane == 31) { s_ws[warp] = incl; s_hs[warp] = hincl; }
    __syncthreads();
    unsigned wp = 0, hp = 0;
#pragma unroll
    for (int w = 0; w < RK_WARPS; w++)
      if (w < warp) { wp += s_ws[w]; hp += s_hs[w]; }
    const unsigned loc = wp + incl - tot;
    s_loc[dd] = loc;
    s_gb[dd] = (long long)(hp + hincl - all) + (long long)prefix - (long long)loc;
    // each warp's counter of this digit becomes the digit's slot in the
    // reordered tile for that warp (one shared-memory lookup per element
    // below instead of two)
#pragma unroll
    for (int w = 0; w < RK_WARPS; w++) s_cnt[w * 256 + dd] += loc;
  }
  __syncthreads();
  if constexpr (OUT == OUT_WIN) {
    // (v, pos) straight into the output windows of v: each element's sorted
    // position from the digit offsets (no reorder by digit), then an
    // unstable slot in its window, the windows' counts looked back over the
    // earlier tiles like the digits', and a reorder by window so that each
    // window's run leaves as one coalesced run
    unsigned pos[RK_ITEMS];
#pragma unroll
    for (int c = 0; c < RK_ITEMS; c++) {
      const unsigned x = wr[c], d = x & 255u;
      pos[c] = 0;
      if (wbase + c * 32 + lane < valid) {
        long long g = s_gb[d] + s_cnt[warp * 256 + d] + (x >> 8);
        if (a.segbase) g -= __ldg(a.segbase + (int)kr[c]);
        pos[c] = (unsigned)g;
      }
    }
    __syncthreads();  // s_cnt, s_loc and s_gb are free
    unsigned *s_wc = s_cnt;  // [256] window counts
    s_wc[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < RK_ITEMS; c++) {
      if (wbase + c * 32 + lane < valid) {
        const unsigned w = (unsigned)vr[c] >> a.wshift;
        wr[c] = (atomicAdd(s_wc + w, 1u) << 8) | w;
      }
    }
    __syncthreads();
    const unsigned wtot = s_wc[tid];
    const unsigned wprefix = bin_lookback(a.wstate, tile, tid, wtot, a.status, a.gave_up, a.spin_limit);
    {
      unsigned incl = wtot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        unsigned xx = shfl_up(incl, o);
        if (lane >= o) incl += xx;
      }
      if (lane == 31) s_ws[warp] = incl;
      __syncthreads();
      unsigned wp = 0;
#pragma unroll
      for (int w = 0; w < RK_WARPS; w++) if (w < warp) wp += s_ws[w];
      const unsigned wloc = wp + incl - wtot;
      s_loc[tid] = wloc;
      // distinct indices: window w's pairs have room from its first index on
      s_gb[tid] = ((long long)tid << a.wshift) + (long long)wprefix - (long long)wloc;
    }
    __syncthreads();
    uint2 *s_vp = (uint2 *)s_kout;  // (v, position) by window slot: one 8-byte store
#pragma unroll
    for (int c = 0; c < RK_ITEMS; c++) {
      const unsigned x = wr[c];
      if (wbase + c * 32 + lane < valid) s_vp[s_loc[x & 255u] + (x >> 8)] = make_uint2((unsigned)vr[c], pos[c]);
    }
    __syncthreads();
#pragma unroll 4
    for (int e = tid; e < valid; e += RK_BLOCK) {
      const uint2 vp = s_vp[e];
      const long g = s_gb[vp.x >> a.wshift] + e;
      a.pidx[g] = vp.x;
      a.ppos[g] = vp.y;
    }
    return;
  }
  // reorder the tile in shared memory (what lies past the vector's end lands
  // past the tile's own elements)
#pragma unroll
  for (int c = 0; c < RK_ITEMS; c++) {
    const unsigned lp = s_cnt[warp * 256 + (wr[c] & 255u)] + (wr[c] >> 8);
    if constexpr (PAIR) {
      s_pair[lp] = make_uint2((unsigned)kr[c], (unsigned)vr[c]);
    } else {
      s_kout[lp] = kr[c];
      s_vout[lp] = vr[c];
    }
    if (AUX) s_aout[lp] = ar[c];
  }
  __syncthreads();
  // coalesced runs out
#pragma unroll 4
  for (int e = tid; e < valid; e += RK_BLOCK) {
    K k;
    V vv;
    if constexpr (PAIR) {
      const uint2 kv = s_pair[e];
      k = (K)kv.x;
      vv = (V)kv.y;
    } else {
      k = s_kout[e];
      vv = s_vout[e];
    }
    const int d = (int)((k >> a.shift) & 255);
    const long g = s_gb[d] + e;
    if (OUT == OUT_ARRAYS) {
      a.kout[g] = k;
      a.vout[g] = vv;
      if (AUX) a.aout[g] = s_aout[e];
    } else {  // OUT_RANK
      int r = (int)g;
      if (a.segbase) r -= __ldg(a.segbase + (int)k);
      a.rank[(unsigned)vv] = r;
    }
  }
}

// One tile per CTA, taken in ticket order.  The word that a pass's waits mark
// when they give up is the next pass's ticket counter: that pass's tickets
// then are no tiles, and it marks the one after it and writes nothing.  (A
// word apart, read by every CTA, took 1.4 % of a rank of 2^26 keys.)
template <class K, class V, bool AUX, int IN, int OUT, int ITEMS>
__global__ void __launch_bounds__(RK_BLOCK, rk_minb<K, AUX>()) k_radix_pass(PassArgs<K, V> a) {
  __shared__ unsigned s_tile;
  if (threadIdx.x == 0) {
    s_tile = atomicAdd(a.counter, 1u);
    if (s_tile & RK_STOP) atomicOr(a.gave_up, RK_STOP);
  }
  __syncthreads();
  if (s_tile & RK_STOP) return;
  radix_tile<K, V, AUX, IN, OUT, ITEMS>(a, a.n, (int)s_tile);
}

// Waits until all CTAs of a resident grid have arrived as often as this one:
// what any of them stored before, all may load afterwards.  Returns the
// CTA's number, read from memory after the wait, so that loads whose address
// comes from it cannot be moved ahead; negative when the bounded wait, or any
// wait of the call before it, gave up (the next pass would follow indices nobody wrote).
__device__ __forceinline__ int rk_meet(unsigned *count, unsigned arrivals, unsigned *status, unsigned *gave_up,
                                       int limit) {
  __shared__ volatile int s_cta;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1, it = 0;
    __threadfence();
    atomicAdd(count, 1u);
    while (*(volatile unsigned *)count < arrivals) {
      if (++it >= limit) { ok = 0; rk_give_up(status, gave_up); break; }
      if (it > 64) __nanosleep(32);
    }
    __threadfence();
    s_cta = ok && !*(volatile unsigned *)gave_up ? (int)blockIdx.x : -1;
  }
  __syncthreads();
  return s_cta;
}

// The digit passes over the long segments, whose number and elements only
// the device knows: by the key, then by the segment number.
template <class K> struct LongArgs {
  K *key[2];                // pass q reads [q & 1] and writes the other
  unsigned *idx[2], *aux[2];
  int *rank; const int *segbase;
  const unsigned *hist;
  unsigned *state[3], *meet;
  const unsigned long long *total;
  int seg_passes, direct, wshift;
  unsigned *status, *gave_up;
  int spin_limit;
};
// One cooperative launch that meets between passes.  There are usually no
// long segments, and then a launch for every pass was much of a call: in
// segments of 64, a launch a pass / this, us: 2^16 int keys 37 / 22, 2^24 202 /
// 181; 2^20 float64 71 / 34.  With long segments: 2^19 int bimodal 80 / 71,
// 2^24 611 / 598; float64 log-normal 2^20 161 / 144, 2^23 651 / 623.
// All CTAs are resident and take their tiles in increasing order, so a tile's
// look-back waits only for tiles that are being ranked: no tickets, whose two
// round trips a pass the meeting would not make up for.  None of a pass's
// loads of an earlier one's output is a read-only load.
template <class K, int ITEMS>
__global__ void __launch_bounds__(RK_BLOCK, GCVL_RK_MINB) k_rank_long(const __grid_constant__ LongArgs<K> l) {
  const int n = (int)(unsigned)*(volatile const unsigned long long *)l.total;
  if (n == 0) return;  // every CTA alike
  const int tiles = (int)(((long)n + RK_BLOCK * ITEMS - 1) / (RK_BLOCK * ITEMS));
  const int ctas = min(tiles, (int)gridDim.x);
  if ((int)blockIdx.x >= ctas) return;
  constexpr int P = sizeof(K);
  const int passes = P + l.seg_passes;
  auto common = [&](auto &a, int q) {
    a.vin = l.idx[q & 1]; a.vout = l.idx[~q & 1];
    a.hist = l.hist + q * 256;
    a.state = l.state[q % 3];
    a.clear = q > 0 && q < passes - 1 ? l.state[(q + 2) % 3] : nullptr;
    a.status = l.status; a.gave_up = l.gave_up; a.spin_limit = l.spin_limit;
  };
  int first = blockIdx.x;
#pragma unroll 1
  for (int q = 0; q < passes; q++) {
    if (q > 0 && (first = rk_meet(l.meet, (unsigned)(q * ctas), l.status, l.gave_up, l.spin_limit)) < 0) return;
#pragma unroll 1
    for (int tile = first; tile < tiles; tile += ctas) {
      if (q < P) {
        PassArgs<K, unsigned> a{};
        common(a, q);
        a.kin = l.key[q & 1]; a.kout = l.key[~q & 1];
        a.ain = l.aux[q & 1]; a.aout = l.aux[~q & 1];
        a.shift = 8 * q;
        radix_tile<K, unsigned, true, IN_ARRAYS, OUT_ARRAYS, ITEMS>(a, n, tile);
      } else {  // the segment number is the key, indices ride along
        PassArgs<unsigned, unsigned> a{};
        common(a, q);
        a.kin = q == P ? l.aux[0] : (const unsigned *)l.key[q & 1];
        a.kout = (unsigned *)l.key[~q & 1];
        a.rank = l.rank; a.segbase = l.segbase; a.shift = 8 * (q - P);
        if (q < passes - 1) radix_tile<unsigned, unsigned, false, IN_ARRAYS, OUT_ARRAYS, ITEMS>(a, n, tile);
        else if (ITEMS != RK_ITEMS_LARGE || l.direct)
          radix_tile<unsigned, unsigned, false, IN_ARRAYS, OUT_RANK, ITEMS>(a, n, tile);
        else if constexpr (ITEMS == RK_ITEMS_LARGE) {  // the pairs by window take the buffers this pass does not read
          a.pidx = a.vout; a.ppos = a.kout;
          a.wstate = l.state[(q + 1) % 3]; a.wshift = l.wshift;
          radix_tile<unsigned, unsigned, false, IN_ARRAYS, OUT_WIN, ITEMS>(a, n, tile);
        }
      }
      __syncthreads();
    }
  }
}

// d[key[i]] = val[i], streaming over pairs that a partition pass grouped by
// output window.  A key past n_d is followed nowhere: after a wait that gave
// up some pairs are unwritten.
template <class V>
__global__ void __launch_bounds__(RK_BLOCK) k_window_scatter(V *__restrict__ d, const unsigned *__restrict__ key,
                                                             const V *__restrict__ val, long n, unsigned n_d,
                                                             const unsigned *__restrict__ gate) {
  // one CTA per 2048 pairs, not a grid-stride loop: CTAs dispatched in
  // order keep the writes within a few windows of the output at a time
  // (a grid-stride form let the CTAs drift apart: rank 11.6 -> 17.1 ms)
  if (gate && *(const volatile unsigned *)gate == 0) return;
  const long i0 = (long)blockIdx.x * (RK_BLOCK * SC_ITEMS) + threadIdx.x;
  unsigned k[SC_ITEMS];
  V v[SC_ITEMS];
#pragma unroll
  for (int u = 0; u < SC_ITEMS; u++) {
    const long i = i0 + (long)u * RK_BLOCK;
    if (i < n) { k[u] = __ldcs(key + i); v[u] = __ldcs(val + i); }
  }
#pragma unroll
  for (int u = 0; u < SC_ITEMS; u++) {
    const long i = i0 + (long)u * RK_BLOCK;
    if (i < n && k[u] < n_d) d[k[u]] = v[u];
  }
}

// ------------------------------------------------------ window split ---
// Groups keys by window (key >> shift, clamped below nw: the same function in
// every pass) without any tile waiting on another: a histogram pass writes
// each tile's per-window counts (window-major), their exclusive scan (the
// library's int +-scan, in place) is every (window, tile)'s first slot --
// the windows before w, then the tiles before t -- and the split pass
// places each tile's keys there.  Slots within a window and tile come from shared-memory atomics (no
// particular order); the tile is staged in shared memory by window and each
// window's run leaves as one coalesced run; with POS, pos[k] = the slot key
// k went to, written in the input order.  The partitioned gather uses it.
constexpr int WS_ITEMS = 16, WS_TILE = RK_BLOCK * WS_ITEMS, WS_MAXW = 256;
__device__ __forceinline__ unsigned ws_window(unsigned k, int shift, int nw) { return min(k >> shift, (unsigned)(nw - 1)); }
// this key's slot among the keys of window w counted in cnt[w] so far (w <
// 0: none).  One shared-memory atomic per key: a per-warp form (lanes of
// one window found by a ballot per window bit, one atomic per window) made
// the partitioned gather and scatter 1.4-1.6x slower.
__device__ __forceinline__ unsigned ws_slot(unsigned *cnt, int w) { return w >= 0 ? atomicAdd(cnt + w, 1u) : 0u; }

// counts[w * tiles + t] = keys of tile t in window w; *unsorted != 0 when
// some key exceeds its successor.  VEC: key is 16-byte aligned, and each
// thread reads four keys at a time.
template <bool VEC>
__global__ void __launch_bounds__(RK_BLOCK) k_ws_hist(const unsigned *__restrict__ key, long n, int shift, int wbits,
                                                      unsigned *__restrict__ counts, unsigned *unsorted) {
  __shared__ unsigned s_cnt[WS_MAXW];
  __shared__ int s_uns;
  const int tid = threadIdx.x, nw = 1 << wbits;
  const int tiles = gridDim.x, t = blockIdx.x;
  s_cnt[tid] = 0;
  if (tid == 0) s_uns = 0;
  __syncthreads();
  const long base = (long)t * WS_TILE;
  int uns = 0;
  if constexpr (VEC) {
    uint4 q[WS_ITEMS / 4];
    unsigned nx[WS_ITEMS / 4];
#pragma unroll
    for (int c = 0; c < WS_ITEMS / 4; c++) {
      const long e = base + 4L * (c * RK_BLOCK + tid);
      q[c] = make_uint4(0, 0, 0, 0);
      nx[c] = 0xFFFFFFFFu;
      if (e + 3 < n) {
        q[c] = __ldcs(reinterpret_cast<const uint4 *>(key + e));
        // the successor of the fourth key: the next lane's line, just read
        if (e + 4 < n) nx[c] = __ldg(key + e + 4);
      }
    }
#pragma unroll
    for (int c = 0; c < WS_ITEMS / 4; c++) {
      const long e = base + 4L * (c * RK_BLOCK + tid);
      const unsigned k4[4] = {q[c].x, q[c].y, q[c].z, q[c].w};
      if (e + 3 < n) {
        if (k4[0] > k4[1] || k4[1] > k4[2] || k4[2] > k4[3] || k4[3] > nx[c]) uns = 1;
      } else {
        for (int u = 0; u < 4; u++)  // the vector's ragged end
          if (e + u + 1 < n && __ldg(key + e + u) > __ldg(key + e + u + 1)) uns = 1;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        int w = -1;
        if (e + u < n) w = (int)ws_window(e + 3 < n ? k4[u] : __ldg(key + e + u), shift, nw);
        ws_slot(s_cnt, w);
      }
    }
  } else {
    unsigned k[WS_ITEMS];
#pragma unroll
    for (int c = 0; c < WS_ITEMS; c++) {
      const long e = base + c * RK_BLOCK + tid;
      k[c] = e < n ? __ldcs(key + e) : 0u;
    }
#pragma unroll
    for (int c = 0; c < WS_ITEMS; c++) {
      const long e = base + c * RK_BLOCK + tid;
      // the successor's load usually hits the line just read by the next lane
      if (e + 1 < n && k[c] > __ldg(key + e + 1)) uns = 1;
      ws_slot(s_cnt, e < n ? (int)ws_window(k[c], shift, nw) : -1);
    }
  }
  if (__any_sync(0xffffffffu, uns) && (tid & 31) == 0) s_uns = 1;
  __syncthreads();
  if (tid < nw) counts[(long)tid * tiles + t] = s_cnt[tid];
  if (tid == 0 && s_uns) atomicOr(unsorted, 1u);
}

// VAL: each key's value (val[k]) moves with it to vout.  Dynamic shared
// memory: ws_split_smem<V, VAL>() bytes.
template <class V, bool VAL> constexpr size_t ws_split_smem() { return (size_t)WS_TILE * (4 + (VAL ? sizeof(V) : 0)); }
template <bool POS, class V = unsigned, bool VAL = false>
__global__ void __launch_bounds__(RK_BLOCK) k_window_split(const unsigned *__restrict__ key, long n, int shift,
                                                           int wbits, const unsigned *__restrict__ first,
                                                           const unsigned *gate, unsigned *__restrict__ kout,
                                                           unsigned *__restrict__ pos, const V *__restrict__ val = nullptr,
                                                           V *__restrict__ vout = nullptr) {
  __shared__ unsigned s_cnt[WS_MAXW];   // the tile's count per window, then its first slot there in the tile
  __shared__ unsigned s_base[WS_MAXW];  // global slot of the window's first key of this tile
  extern __shared__ __align__(16) unsigned char rk_smem[];
  unsigned *s_key = (unsigned *)rk_smem;                  // [WS_TILE] keys by window
  V *s_val = (V *)(rk_smem + (size_t)WS_TILE * 4);        // [WS_TILE] their values (VAL)
  __shared__ unsigned s_ws[RK_WARPS];
  if (!*(const volatile unsigned *)gate) return;  // the same answer for every CTA
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = 1 << wbits;
  const int tiles = gridDim.x, t = blockIdx.x;
  s_cnt[tid] = 0;
  if (tid < nw) s_base[tid] = __ldg(first + (long)tid * tiles + t);
  __syncthreads();
  const long base = (long)t * WS_TILE;
  const int valid = (int)min((long)WS_TILE, n - base);
  unsigned k[WS_ITEMS], r[WS_ITEMS];
  V v[VAL ? WS_ITEMS : 1];
#pragma unroll
  for (int c = 0; c < WS_ITEMS; c++) {
    const int e = c * RK_BLOCK + tid;
    if (e < valid) {
      k[c] = __ldcs(key + base + e);
      if constexpr (VAL) v[c] = __ldcs(val + base + e);
    }
  }
#pragma unroll
  for (int c = 0; c < WS_ITEMS; c++)
    r[c] = ws_slot(s_cnt, c * RK_BLOCK + tid < valid ? (int)ws_window(k[c], shift, nw) : -1);
  __syncthreads();
  // the windows' first slots within the tile: exclusive scan over the bins
  const unsigned tot = s_cnt[tid];
  // a scan whose wait gave up can leave any slot here: the tile's keys stay inside the n
  if (tid < nw) s_base[tid] = min(s_base[tid], (unsigned)n - tot);
  unsigned incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = shfl_up(incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) s_ws[warp] = incl;
  __syncthreads();
  unsigned wp = 0;
#pragma unroll
  for (int q = 0; q < RK_WARPS; q++) if (q < warp) wp += s_ws[q];
  s_cnt[tid] = wp + incl - tot;
  __syncthreads();
#pragma unroll
  for (int c = 0; c < WS_ITEMS; c++) {
    const int e = c * RK_BLOCK + tid;
    if (e < valid) {
      const unsigned w = ws_window(k[c], shift, nw);
      s_key[s_cnt[w] + r[c]] = k[c];
      if constexpr (VAL) s_val[s_cnt[w] + r[c]] = v[c];
      if (POS) pos[base + e] = s_base[w] + r[c];
    }
  }
  __syncthreads();
  // coalesced runs: slot e of the tile holds window w's key e - s_cnt[w]
#pragma unroll 4
  for (int e = tid; e < valid; e += RK_BLOCK) {
    const unsigned kk = s_key[e];
    const unsigned w = ws_window(kk, shift, nw);
    const unsigned g = s_base[w] + (unsigned)e - s_cnt[w];
    kout[g] = kk;
    if constexpr (VAL) vout[g] = s_val[e];
  }
}

// p[j] = s[key[j]] over keys that a window split grouped by source window:
// CTAs dispatched in order keep the reads within a few windows of s, which
// sit in L2 while they are read.  An index outside [0, n_src) reads nothing
// (its value is 0) and sets DEV_RANGE.  p may be key itself (4-byte values).
template <class V>
__global__ void __launch_bounds__(RK_BLOCK) k_window_gather(V *p, const V *__restrict__ s, const unsigned *key,
                                                            long n, unsigned n_src, const unsigned *gate,
                                                            unsigned *status) {
  if (gate && *(const volatile unsigned *)gate == 0) return;
  const long i0 = (long)blockIdx.x * (RK_BLOCK * SC_ITEMS) + threadIdx.x;
  unsigned k[SC_ITEMS];
  V v[SC_ITEMS];
#pragma unroll
  for (int u = 0; u < SC_ITEMS; u++) {
    const long i = i0 + (long)u * RK_BLOCK;
    k[u] = i < n ? __ldcs(key + i) : 0u;
  }
  bool bad = false;
#pragma unroll
  for (int u = 0; u < SC_ITEMS; u++) {
    v[u] = (V)0;
    if (i0 + (long)u * RK_BLOCK < n) {
      if (k[u] < n_src) v[u] = __ldg(s + k[u]);
      else bad = true;
    }
  }
  if (bad) atomicOr(status, DEV_RANGE);
#pragma unroll
  for (int u = 0; u < SC_ITEMS; u++) {
    const long i = i0 + (long)u * RK_BLOCK;
    if (i < n) p[i] = v[u];
  }
}

// d[i] = s[idx[i]], run only when (*gate != 0) == when_set
template <class V>
__global__ void __launch_bounds__(RK_BLOCK) k_gather_gated(V *__restrict__ d, const V *__restrict__ s,
                                                           const unsigned *__restrict__ idx, long n,
                                                           const unsigned *gate, int when_set) {
  if ((*(const volatile unsigned *)gate != 0) != (when_set != 0)) return;
  // grid-stride: launched with one CTA per 2048 elements it makes one pass;
  // launched with few CTAs it costs little when the gate turns it away
  for (long i0 = (long)blockIdx.x * (RK_BLOCK * SC_ITEMS) + threadIdx.x; i0 < n;
       i0 += (long)gridDim.x * (RK_BLOCK * SC_ITEMS)) {
    unsigned k[SC_ITEMS];
    V v[SC_ITEMS];
#pragma unroll
    for (int u = 0; u < SC_ITEMS; u++) {
      const long i = i0 + (long)u * RK_BLOCK;
      k[u] = i < n ? __ldcs(idx + i) : 0u;
    }
#pragma unroll
    for (int u = 0; u < SC_ITEMS; u++)
      if (i0 + (long)u * RK_BLOCK < n) v[u] = __ldg(s + k[u]);
#pragma unroll
    for (int u = 0; u < SC_ITEMS; u++) {
      const long i = i0 + (long)u * RK_BLOCK;
      if (i < n) __stcs(d + i, v[u]);
    }
  }
}

template <class K, class V, bool AUX, int IN, int OUT, int ITEMS>
void launch_pass_items(const PassArgs<K, V> &a) {
  constexpr size_t sm = pass_smem<K, V, AUX, ITEMS>();
  static bool attr = false;
  if (!attr) {
    GCVL_CK(cudaFuncSetAttribute(k_radix_pass<K, V, AUX, IN, OUT, ITEMS>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    attr = true;
  }
  k_radix_pass<K, V, AUX, IN, OUT, ITEMS><<<ceil_div(a.n, RK_BLOCK * ITEMS), RK_BLOCK, sm, stream()>>>(a);
  launch_check("k_radix_pass");
}
inline int rk_tile(long n) {
  return RK_BLOCK * (n <= RK_TINY_MAX ? RK_ITEMS_TINY : n <= RK_SMALL_MAX ? RK_ITEMS_SMALL : RK_ITEMS_LARGE);
}
template <class K, class V, bool AUX, int IN, int OUT> void launch_pass(const PassArgs<K, V> &a) {
  if (a.n > RK_SMALL_MAX) launch_pass_items<K, V, AUX, IN, OUT, RK_ITEMS_LARGE>(a);
  else if constexpr (OUT != OUT_WIN) {
    if (a.n > RK_TINY_MAX) launch_pass_items<K, V, AUX, IN, OUT, RK_ITEMS_SMALL>(a);
    else launch_pass_items<K, V, AUX, IN, OUT, RK_ITEMS_TINY>(a);
  }
}
template <class K, int ITEMS> void launch_long_items(LongArgs<K> l, int n) {
  constexpr size_t sm =
      std::max(pass_smem<K, unsigned, true, ITEMS>(), pass_smem<unsigned, unsigned, false, ITEMS>());
  static int per_sm = 0;  // of a cooperative launch, whose CTAs are all resident
  if (per_sm < 1) {
    GCVL_CK(cudaFuncSetAttribute(k_rank_long<K, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    int nb = 0;
    if (!GCVL_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_rank_long<K, ITEMS>, RK_BLOCK, sm))) return;
    per_sm = std::max(nb, 1);
  }
  const int grid = std::min(ceil_div(n, RK_BLOCK * ITEMS), per_sm * st().sm_count);
  void *args[] = {&l};
  GCVL_CK(cudaLaunchCooperativeKernel((const void *)k_rank_long<K, ITEMS>, dim3(grid), dim3(RK_BLOCK), args, sm,
                                      stream()));
  launch_check("k_rank_long");
}
template <class K> void launch_long(const LongArgs<K> &l, int n) {
  if (n > RK_SMALL_MAX) launch_long_items<K, RK_ITEMS_LARGE>(l, n);
  else if (n > RK_TINY_MAX) launch_long_items<K, RK_ITEMS_SMALL>(l, n);
  else launch_long_items<K, RK_ITEMS_TINY>(l, n);
}
static_assert(RK_SMALL_MAX <= RK_DIRECT_MAX, "windows only for large tiles");

inline int sc_blocks(long n) { return (int)((n + RK_BLOCK * SC_ITEMS - 1) / (RK_BLOCK * SC_ITEMS)); }
// grid of the sorted-index scatter: grid-stride over at most 16 CTAs per
// SM, so that when its gate says "not this time" it costs a few
// microseconds instead of a launch of one CTA per 2048 elements
inline int sc_grid(long n) {
  const long need = (n + RK_BLOCK * SC_ITEMS - 1) / (RK_BLOCK * SC_ITEMS);
  const long cap = (long)st().sm_count * 16;
  return (int)(need < cap ? (need < 1 ? 1 : need) : cap);
}
inline size_t rk_state_bytes(long n) { return (size_t)ceil_div(n, rk_tile(n)) * 256 * 4; }
// of any vector of at most n elements (a shorter one in smaller tiles may have
// more of them), so that scratch of a call covers every shorter call
inline size_t rk_state_room(long n) {
  size_t b = rk_state_bytes(n);
  for (const long line : {(long)RK_TINY_MAX, (long)RK_SMALL_MAX})
    if (n > line) b = std::max(b, rk_state_bytes(line));
  return b;
}
inline int ws_tiles(long n) { return (int)((n + WS_TILE - 1) / WS_TILE); }  // tiles of the window split
// top-8-bit windows of [0, n)
inline int window_shift(int n) { int b = bit_length((unsigned)(n > 1 ? n - 1 : 1)); return b > 8 ? b - 8 : 0; }

// the window counts of every tile of idx[0, n) and the gate word
inline void ws_hist(const int *idx, long n, int shift, int wbits, int tiles, unsigned *counts, unsigned *unsorted) {
  if (((uintptr_t)idx & 15) == 0)
    k_ws_hist<true><<<tiles, RK_BLOCK, 0, stream()>>>((const unsigned *)idx, n, shift, wbits, counts, unsorted);
  else
    k_ws_hist<false><<<tiles, RK_BLOCK, 0, stream()>>>((const unsigned *)idx, n, shift, wbits, counts, unsorted);
  launch_check("k_ws_hist");
}

// ------------------------------------------------ partitioned scatter ---
// d[idx[k]] = s[k] for k < n (idx in [0, n_d)) when d is larger than L2 can
// absorb random writes to (each would cost a DRAM read-modify-write of a
// sector): the (index, value) pairs are split by destination window (windows
// of at most 8 MB, at most 256 of them, with the same histogram, scan and
// split passes as the partitioned gather), then written window by window
// while each window sits in L2.  Ascending indices take one streaming scatter instead; the
// device decides (the kernels of the branch not taken return at once).
struct ScatterLayout { size_t kout, vout, counts, scan, flags, total; };
inline ScatterLayout scatter_layout(long n, size_t vsize) {
  ScatterLayout L;
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o += align_up(bytes, 256); return at; };
  L.kout = take((size_t)n * 4);
  L.vout = take((size_t)n * vsize);
  L.counts = take((size_t)ws_tiles(n) * WS_MAXW * 4);
  L.scan = take((size_t)add_suz_scratch(ws_tiles(n) * WS_MAXW) * 8);
  L.flags = take(256);
  L.total = o + 256;  // room to align the base
  return L;
}
bool scatter_partitioned_wanted(long n_d, size_t vsize) { return (size_t)n_d * vsize > (size_t)RK_DIRECT_MAX * 4; }
size_t scatter_partitioned_bytes(long n, size_t vsize) { return scatter_layout(n, vsize).total; }
// Window sizes, measured on int32 permutations: the gather runs fastest
// with at least 8 windows of at most 64 MB (2.81 -> 2.69 ms at 2^28 against
// 32 MB windows), the scatter with windows of at most 8 MB (2^28: 3.28 ms
// with 32 MB windows, 3.06 with 16, 2.78 with 8; 2^25: 0.45, 0.40, 0.36).
#ifndef GCVL_WS_GATHER_MB
#define GCVL_WS_GATHER_MB 64
#endif
#ifndef GCVL_WS_GATHER_MINBITS
#define GCVL_WS_GATHER_MINBITS 3
#endif
#ifndef GCVL_WS_SCATTER_MB
#define GCVL_WS_SCATTER_MB 8
#endif
// windows of at most `mb` MB of `bytes`, a power of two from 2^min_bits to
// 256: (log2 of the count, shift of an index of [0, len) to its window)
inline void ws_windows(size_t bytes, long len, int mb, int min_bits, int *wbits, int *shift) {
  int wb = min_bits;
  while (wb < 8 && (bytes >> wb) > ((size_t)mb << 20)) ++wb;
  const int nb = bit_length((unsigned)(len > 1 ? len - 1 : 1));
  *wbits = wb;
  *shift = nb > wb ? nb - wb : 0;
}

template <class V>
void scatter_partitioned(V *d, const V *s, const int *idx, int n, int n_d, vec_p scratch) {
  State &S = st();
  if (n <= 0) return;
  ScatterLayout L = scatter_layout(n, sizeof(V));
  char *raw = (char *)scratch_or_work(scratch, L.total);
  if (!raw) return;
  char *mem = (char *)align_up((size_t)raw, 256);
  unsigned *kout = (unsigned *)(mem + L.kout);
  V *vout = (V *)(mem + L.vout);
  unsigned *counts = (unsigned *)(mem + L.counts);
  void *scan_scratch = mem + L.scan;
  unsigned *unsorted = (unsigned *)(mem + L.flags);  // the gate: non-zero when some index exceeds its successor
  int wbits, shift;
  ws_windows((size_t)n_d * sizeof(V), n_d, GCVL_WS_SCATTER_MB, 1, &wbits, &shift);
  const int nw = 1 << wbits;
  const int tiles = ws_tiles(n);
  constexpr size_t smem = ws_split_smem<V, true>();
  static bool attr = false;
  if (!attr) {
    GCVL_CK(cudaFuncSetAttribute(k_window_split<false, V, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    attr = true;
  }
  if (!GCVL_CK(cudaMemsetAsync(unsorted, 0, 4, S.stream))) return;
  ws_hist(idx, n, shift, wbits, tiles, counts, unsorted);
  k_sorted_scatter<V><<<sc_grid(n), RK_BLOCK, 0, S.stream>>>(d, s, idx, n, unsorted);
  launch_check("k_sorted_scatter");
  add_suz(counts, counts, nw * tiles, scan_scratch);  // first slot of every (window, tile)
  k_window_split<false, V, true><<<tiles, RK_BLOCK, smem, S.stream>>>((const unsigned *)idx, n, shift, wbits, counts,
                                                                      unsorted, kout, nullptr, s, vout);
  launch_check("k_window_split");
  k_window_scatter<V><<<sc_blocks(n), RK_BLOCK, 0, S.stream>>>(d, kout, vout, n, (unsigned)n_d, unsorted);
  launch_check("k_window_scatter");
}

// ------------------------------------------------- partitioned gather ---
// d[k] = s[idx[k]] for k < n (idx in [0, n_src)) when s is larger than L2 can
// serve random reads from: each random 4- or 8-byte read from DRAM costs a
// whole sector, and most miss.  Instead the indices are split by source
// window (at least 8 windows of at most 64 MB, at most 256), with pos[k] = where
// index k went; a gather in window order reads each window of s while it
// sits in L2, into p; and d[k] = p[pos[k]] reads p through as many sequential
// runs as there are windows, few enough that L1 and L2 keep each run's
// current lines.  The passes stream: 4 (histogram) + 12 (split) + 12 + 12
// bytes per 4-byte element.  Ascending indices take one plain gather
// instead; the device decides, as for the scatter.
struct GatherLayout { size_t kout, pos, p, counts, scan, flags, total; };
inline GatherLayout gather_layout(long n, size_t vsize) {
  GatherLayout L;
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o += align_up(bytes, 256); return at; };
  L.kout = take((size_t)n * 4);
  L.pos = take((size_t)n * 4);
  L.p = vsize == 4 ? L.kout : take((size_t)n * vsize);  // 4-byte values overwrite their keys in place
  L.counts = take((size_t)ws_tiles(n) * WS_MAXW * 4);
  L.scan = take((size_t)add_suz_scratch(ws_tiles(n) * WS_MAXW) * 8);
  L.flags = take(256);
  L.total = o + 256;  // room to align the base
  return L;
}
bool gather_partitioned_wanted(long n_src, long n, size_t vsize) {
  return (size_t)n_src * vsize > ((size_t)64 << 20) && n >= (1L << 20);
}
size_t gather_partitioned_bytes(long n, size_t vsize) { return gather_layout(n, vsize).total; }

template <class V>
void gather_partitioned(V *d, const V *s, const int *idx, int n, int n_src, vec_p scratch) {
  State &S = st();
  if (n <= 0) return;
  GatherLayout L = gather_layout(n, sizeof(V));
  char *raw = (char *)scratch_or_work(scratch, L.total);
  if (!raw) return;
  char *mem = (char *)align_up((size_t)raw, 256);
  unsigned *kout = (unsigned *)(mem + L.kout);
  unsigned *pos = (unsigned *)(mem + L.pos);
  V *p = (V *)(mem + L.p);
  unsigned *counts = (unsigned *)(mem + L.counts);
  void *scan_scratch = mem + L.scan;
  unsigned *unsorted = (unsigned *)(mem + L.flags);  // the gate: non-zero when some index exceeds its successor
  int wbits, shift;
  ws_windows((size_t)n_src * sizeof(V), n_src, GCVL_WS_GATHER_MB, GCVL_WS_GATHER_MINBITS, &wbits, &shift);
  const int nw = 1 << wbits;
  const int tiles = ws_tiles(n);
  GCVL_CK(cudaMemsetAsync(unsorted, 0, 4, S.stream));
  ws_hist(idx, n, shift, wbits, tiles, counts, unsorted);
  k_gather_gated<V><<<sc_grid(n), RK_BLOCK, 0, S.stream>>>(d, s, (const unsigned *)idx, n, unsorted, 0);
  launch_check("k_gather_gated");
  add_suz(counts, counts, nw * tiles, scan_scratch);  // first slot of every (window, tile)
  k_window_split<true><<<tiles, RK_BLOCK, ws_split_smem<unsigned, false>(), S.stream>>>(
      (const unsigned *)idx, n, shift, wbits, counts, unsorted, kout, pos);
  launch_check("k_window_split");
  k_window_gather<V><<<sc_blocks(n), RK_BLOCK, 0, S.stream>>>(p, s, kout, n, (unsigned)n_src, unsorted,
                                                              S.d_status);
  launch_check("k_window_gather");
  k_gather_gated<V><<<sc_blocks(n), RK_BLOCK, 0, S.stream>>>(d, p, pos, n, unsorted, 1);
  launch_check("k_gather_gated");
}
template void gather_partitioned<unsigned>(unsigned *, const unsigned *, const int *, int, int, vec_p);
template void gather_partitioned<unsigned long long>(unsigned long long *, const unsigned long long *,
                                                     const int *, int, int, vec_p);
template void scatter_partitioned<unsigned>(unsigned *, const unsigned *, const int *, int, int, vec_p);
template void scatter_partitioned<unsigned long long>(unsigned long long *, const unsigned long long *,
                                                      const int *, int, int, vec_p);

// ------------------------------------------------------------- rank ---
// rank[index] = position from the (index, position) pairs of the last pass,
// grouped by window of the index: window w's pairs lie from slot w << wshift
// on, as many as the last pass counted (all the window's indices when the
// vector was ranked whole).  One CTA per 2048 slots, as k_window_scatter;
// DYN (long segments, usually none): a resident grid, which takes the slots in
// ticket order (each CTA striding through them, the CTAs drift apart over the
// windows: 2^28 ints, all in long segments, 18.2 ms, now 17.0).  After a wait of the
// passes gave up the pairs may be anything: DYN, whose counts may be missing
// too, writes nothing, and otherwise an index is looked at before it is
// followed (10 us of 340 at 2^26 keys; asking the word in every CTA took 20).
template <bool DYN>
__global__ void __launch_bounds__(RK_BLOCK) k_rank_scatter(int *__restrict__ rank, const unsigned *__restrict__ pidx,
                                                           const unsigned *__restrict__ ppos, int n, int wshift,
                                                           const unsigned long long *total,
                                                           const unsigned *__restrict__ wstate, int tile_elems,
                                                           const unsigned *gave_up, unsigned *ticket) {
  __shared__ unsigned s_block;
  const unsigned *counts = nullptr;  // the last tile's inclusive window counts
  if constexpr (DYN) {
    const long t = (long)(unsigned)*(volatile const unsigned long long *)total;
    if (t == 0) return;
    if (*(const volatile unsigned *)gave_up) return;
    counts = wstate + (t - 1) / tile_elems * 256;
  }
  for (;;) {
    long b = blockIdx.x;
    if constexpr (DYN) {
      if (threadIdx.x == 0) s_block = atomicAdd(ticket, 1u);
      __syncthreads();
      b = s_block;
      __syncthreads();
    }
    if (b * (RK_BLOCK * SC_ITEMS) >= n) return;
    const long i0 = b * (RK_BLOCK * SC_ITEMS) + threadIdx.x;
    unsigned k[SC_ITEMS], v[SC_ITEMS];
    bool ok[SC_ITEMS];
#pragma unroll
    for (int u = 0; u < SC_ITEMS; u++) {
      const long i = i0 + (long)u * RK_BLOCK;
      ok[u] = i < n;
      if (DYN && ok[u]) ok[u] = (i & ((1L << wshift) - 1)) < (long)(__ldg(counts + (i >> wshift)) & ~RK_INC);
      if (ok[u]) { k[u] = __ldcs(pidx + i); v[u] = __ldcs(ppos + i); }
    }
#pragma unroll
    for (int u = 0; u < SC_ITEMS; u++)
      if (ok[u] && k[u] < (unsigned)n) rank[k[u]] = (int)v[u];
    if (!DYN) return;
  }
}

// Scratch of the digit passes.  Whole vectors: pairs twice, digit counts,
// look-back words three times over (a pass's own, those it clears for the
// one after the next, and those in between; the last pass takes two).
// Segmented: the same for the long segments, with their numbers and tables.
struct RankLayout {
  size_t hist, counter, lsum, state, key_a, key_b, idx_a, idx_b, aux_a, aux_b, first, base, of_tile, total;
};
inline RankLayout rank_layout(int n, int is_double, int seg) {
  RankLayout L;
  size_t ks = is_double ? 8 : 4;
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o += align_up(bytes, 256); return at; };
  L.hist = take(RK_MAXPASS * 256 * 4);  // these three are cleared together
  L.counter = take((RK_MAXPASS + 3) * 4);  // tickets, the long segments' meetings, whether a wait gave up, the scatter's
  L.lsum = take(8);
  L.state = take(rk_state_room(n) * 3);
  L.key_a = take((size_t)n * ks);
  L.key_b = take((size_t)n * ks);
  L.idx_a = take((size_t)n * 4);
  L.idx_b = take((size_t)n * 4);
  L.aux_a = take(seg ? (size_t)n * 4 : 0);
  L.aux_b = take(seg ? (size_t)n * 4 : 0);
  L.first = take(seg ? ((size_t)n / LR_MAX + 1) * 4 : 0);
  L.base = take(seg ? ((size_t)n / LR_MAX + 1) * 4 : 0);
  L.of_tile = take(seg ? (size_t)lr_tiles(n) * 4 : 0);
  L.total = o + 256;  // room to align the base
  return L;
}
// one CTA ranks the whole vector: at most LR_CAP elements in at most LR_T segments
inline bool rank_whole(int n, int m) { return n <= LR_CAP && (m <= LR_T || n <= LR_T); }
int rank_units(int n, int is_double, int seg) {
  if (n <= 0) return 0;
  return (int)((rank_layout(n, is_double, seg).total + 7) / 8);
}

template <class K>
void rank_impl(vec_p d, vec_p s, vec_p sd, int n, int m, vec_p scratch, int is_double, int up) {
  ensure_init();
  State &S = st();
  if (n <= 0) return;
  const bool seg = sd != nullptr && m > 1;
  const SegView sv = seg ? seg_view(sd, n, m) : SegView{nullptr, nullptr, nullptr, nullptr, n, 1};
  if (rank_whole(n, m)) {
    rank_local<K>(s, (int *)d, sv, n, up, true, LongSegs{});
    return;
  }
  const RankLayout L = rank_layout(n, is_double, seg);
  char *raw = (char *)scratch_or_work(scratch, L.total);
  if (!raw) return;
  char *mem = (char *)align_up((size_t)raw, 256);
  unsigned *hist = (unsigned *)(mem + L.hist), *counters = (unsigned *)(mem + L.counter);
  const size_t state_bytes = rk_state_bytes(n);
  unsigned *state[3];
  for (int b = 0; b < 3; b++) state[b] = (unsigned *)(mem + L.state + b * state_bytes);
  if (!GCVL_CK(cudaMemsetAsync(mem + L.hist, 0, L.state - L.hist, S.stream))) return;

  char *kA = mem + L.key_a, *kB = mem + L.key_b;
  unsigned *iA = (unsigned *)(mem + L.idx_a), *iB = (unsigned *)(mem + L.idx_b);
  unsigned *aA = (unsigned *)(mem + L.aux_a), *aB = (unsigned *)(mem + L.aux_b);
  const int key_passes = (int)sizeof(K);
  const bool direct = n <= RK_DIRECT_MAX;
  const int wshift = window_shift(n);
  unsigned *pidx = nullptr, *ppos = nullptr, *wstate = nullptr, *gave_up = nullptr;
  const unsigned long long *total = nullptr;
  if (seg) {
    LongSegs ls;
    ls.total = (unsigned long long *)(mem + L.lsum);
    ls.first = (int *)(mem + L.first);
    ls.base = (int *)(mem + L.base);
    ls.of_tile = (int *)(mem + L.of_tile);
    rank_local<K>(s, (int *)d, sv, n, up, false, ls);
    // the long segments, if there are any: the kernels below return at once otherwise
    total = ls.total;
    // the numbers of as many long segments as there can be
    const int seg_passes = std::max(1, (bit_length((unsigned)(std::min(m, n / (LR_MAX + 1)) - 1)) + 7) / 8);
    const int pg = std::min(S.sm_count * 8, lr_tiles(n));
    k_rank_prep_long<K><<<pg, RK_BLOCK, 0, S.stream>>>((const K *)s, n, up, sv, ls, seg_passes, (K *)kA, iA, aA, hist,
                                                       state[0], (long)(state_bytes / 4), rk_tile(n));
    launch_check("k_rank_prep_long");
    LongArgs<K> l{};
    l.key[0] = (K *)kA; l.key[1] = (K *)kB;
    l.idx[0] = iA; l.idx[1] = iB;
    l.aux[0] = aA; l.aux[1] = aB;
    l.rank = (int *)d; l.segbase = ls.base; l.hist = hist;
    for (int b = 0; b < 3; b++) l.state[b] = state[b];
    l.meet = counters + RK_MAXPASS;
    l.total = total; l.seg_passes = seg_passes; l.direct = direct; l.wshift = wshift;
    l.status = S.d_status; l.gave_up = gave_up = counters + RK_MAXPASS + 1; l.spin_limit = S.spin_limit;
    launch_long<K>(l, n);
    const int last = key_passes + seg_passes - 1;
    pidx = l.idx[~last & 1];
    ppos = (unsigned *)l.key[~last & 1];
    wstate = state[(last + 1) % 3];
  } else {
    // at least 16 keys a thread: every CTA adds its histograms to the vector's
    // with an atomic per bin (2^20 keys by 1216 CTAs 14.6 us, by 256 5)
    const int pg = std::min(S.sm_count * 8, ceil_div(n, (long)RK_BLOCK * 16));
    k_rank_prep<K><<<pg, RK_BLOCK, 0, S.stream>>>((const K *)s, n, up, hist, (uint4 *)state[0],
                                                  (long)(3 * state_bytes / 16));
    launch_check("k_rank_prep");
    for (int q = 0; q < key_passes; q++) {
      const bool final = (q == key_passes - 1);
      PassArgs<K, unsigned> a{};
      a.kin = (const K *)kA; a.kout = (K *)kB;
      a.vin = iA; a.vout = iB;
      a.src = s; a.up = up; a.shift = 8 * q;
      a.hist = hist + q * 256; a.counter = counters + q;
      a.state = state[q % 3]; a.clear = q > 0 && !final ? state[(q + 2) % 3] : nullptr;
      a.n = n; a.status = S.d_status; a.gave_up = counters + q + 1; a.spin_limit = S.spin_limit;
      if (final) {  // the pairs by window take the buffers the last pass does not read
        a.rank = (int *)d;
        a.pidx = pidx = iB;
        a.ppos = ppos = (unsigned *)kB;
        a.wstate = state[(q + 1) % 3]; a.wshift = wshift;
      }
      if (q == 0) launch_pass<K, unsigned, false, IN_SRC, OUT_ARRAYS>(a);
      else if (!final) launch_pass<K, unsigned, false, IN_ARRAYS, OUT_ARRAYS>(a);
      else if (direct) launch_pass<K, unsigned, false, IN_ARRAYS, OUT_RANK>(a);
      else launch_pass<K, unsigned, false, IN_ARRAYS, OUT_WIN>(a);
      std::swap(kA, kB);
      std::swap(iA, iB);
    }
  }

  if (!direct) {
    if (seg)
      k_rank_scatter<true><<<sc_grid(n), RK_BLOCK, 0, S.stream>>>((int *)d, pidx, ppos, n, wshift, total, wstate,
                                                                  rk_tile(n), gave_up, counters + RK_MAXPASS + 2);
    else
      k_rank_scatter<false><<<sc_blocks(n), RK_BLOCK, 0, S.stream>>>((int *)d, pidx, ppos, n, wshift, nullptr, nullptr,
                                                                     rk_tile(n), nullptr, nullptr);
    launch_check("k_rank_scatter");
  }
}

}  // namespace gcvl

using namespace gcvl;

GCVL_EXPORT void rku_luz(vec_p d, vec_p s, int len, vec_p scratch) { rank_impl<unsigned>(d, s, nullptr, len, 1, scratch, 0, 1); }
GCVL_EXPORT int rku_luz_scratch(int len) { return rank_units(len, 0, 0); }
GCVL_EXPORT unsigned rku_luz_inplace(void) { return INPLACE_NONE; }
GCVL_EXPORT void rkd_luz(vec_p d, vec_p s, int len, vec_p scratch) { rank_impl<unsigned>(d, s, nullptr, len, 1, scratch, 0, 0); }
GCVL_EXPORT int rkd_luz_scratch(int len) { return rank_units(len, 0, 0); }
GCVL_EXPORT unsigned rkd_luz_inplace(void) { return INPLACE_NONE; }
GCVL_EXPORT void rku_lez(vec_p d, vec_p s, vec_p sd, int n, int m, vec_p scratch) { rank_impl<unsigned>(d, s, sd, n, m, scratch, 0, 1); }
GCVL_EXPORT int rku_lez_scratch(int n, int m) { return rank_units(n, 0, m > 1); }
GCVL_EXPORT unsigned rku_lez_inplace(void) { return INPLACE_NONE; }
GCVL_EXPORT void rkd_lez(vec_p d, vec_p s, vec_p sd, int n, int m, vec_p scratch) { rank_impl<unsigned>(d, s, sd, n, m, scratch, 0, 0); }
GCVL_EXPORT int rkd_lez_scratch(int n, int m) { return rank_units(n, 0, m > 1); }
GCVL_EXPORT unsigned rkd_lez_inplace(void) { return INPLACE_NONE; }
GCVL_EXPORT void rku_lud(vec_p d, vec_p s, int len, vec_p scratch) { rank_impl<unsigned long long>(d, s, nullptr, len, 1, scratch, 1, 1); }
GCVL_EXPORT int rku_lud_scratch(int len) { return rank_units(len, 1, 0); }
GCVL_EXPORT unsigned rku_lud_inplace(void) { return INPLACE_NONE; }
GCVL_EXPORT void rkd_lud(vec_p d, vec_p s, int len, vec_p scratch) { rank_impl<unsigned long long>(d, s, nullptr, len, 1, scratch, 1, 0); }
GCVL_EXPORT int rkd_lud_scratch(int len) { return rank_units(len, 1, 0); }
GCVL_EXPORT unsigned rkd_lud_inplace(void) { return INPLACE_NONE; }
GCVL_EXPORT void rku_led(vec_p d, vec_p s, vec_p sd, int n, int m, vec_p scratch) { rank_impl<unsigned long long>(d, s, sd, n, m, scratch, 1, 1); }
GCVL_EXPORT int rku_led_scratch(int n, int m) { return rank_units(n, 1, m > 1); }
GCVL_EXPORT unsigned rku_led_inplace(void) { return INPLACE_NONE; }
GCVL_EXPORT void rkd_led(vec_p d, vec_p s, vec_p sd, int n, int m, vec_p scratch) { rank_impl<unsigned long long>(d, s, sd, n, m, scratch, 1, 0); }
GCVL_EXPORT int rkd_led_scratch(int n, int m) { return rank_units(n, 1, m > 1); }
GCVL_EXPORT unsigned rkd_led_inplace(void) { return INPLACE_NONE; }
