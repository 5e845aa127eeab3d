// rank_local.cu -- ranks that one CTA can finish: segmented ranks of segments
// of at most LR_MAX elements, and whole vectors of at most LR_CAP.
//
// A CTA takes the segments that start in its LR_T elements, so it holds whole
// segments and needs no other CTA: one read of the keys, one write of the
// ranks.  Inside, every segment is cut into as many buckets as it has
// elements by where a key lies between the segment's smallest and largest
// (a non-decreasing map, so buckets are in key order); the elements are
// placed bucket by bucket in shared memory, and an element's rank is its
// bucket's start plus the keys before its own inside the bucket, ties by
// index (the stable order of nesl/cvl/serial/rank.c:49-362).  With keys
// spread over their range a bucket holds one or two elements whatever the
// segment's length.  A CTA whose buckets came out crowded (few distinct keys,
// clustered keys) sorts its keys instead with stable 8-bit digit passes in
// shared memory, skipping the digits on which all its keys agree.
//
// Segments longer than LR_MAX are numbered and given room in a compacted
// vector, which the digit passes of rank.cu then sort.
#include "gcvl.cuh"
#include "rank.cuh"

namespace gcvl {

constexpr int LR_WARPS = LR_BLOCK / 32;
constexpr int LR_STEPS = LR_CAP / LR_BLOCK;  // elements of a thread in a full CTA
constexpr int LR_WORDS = LR_CAP / 32 + 1;    // head-bit words: a full CTA's, and the one that may end it
constexpr size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }
// CTAs an SM is asked to hold: all its threads with 4-byte keys (rku_sez at
// 2^24 with segments of 64 by 2 CTAs 227.6 us, by 3 207.2, by 4 203.1); two
// with 8-byte keys, whose tile takes twice the shared memory.
template <class K> constexpr int lr_minb() { return sizeof(K) == 4 ? 4 : 2; }
// Buckets are compared element by element while that costs less than the
// digit passes: about 10 instructions per comparison against 45 per element
// and digit.
constexpr unsigned LR_CROWD_MEAN = 24, LR_CROWD_MAX = 256;
static_assert(LR_CAP == LR_T + LR_MAX && LR_CAP % LR_BLOCK == 0 && LR_T % LR_BLOCK == 0, "whole steps");
static_assert(LR_CAP <= 4096, "local positions and bucket counts are packed into 16 bits each");

// Order key of the float that lies nearest a key towards zero: a
// non-decreasing 32-bit image of the key, in which differences follow the
// values (the bits of a double are logarithmic).  Infinities and NaNs take
// the ends of the range.
__device__ __forceinline__ unsigned lr_image(unsigned k, int) { return k; }
__device__ __forceinline__ unsigned lr_image(unsigned long long k, int up) {
  const unsigned long long ku = up ? k : ~k;
  const bool neg = !(ku >> 63);
  const unsigned long long raw = neg ? ~ku : ku ^ (1ULL << 63);
  const unsigned hi = (unsigned)(raw >> 32) & 0x7FFFFFFFu;
  const int e = (int)(hi >> 20) - 896;
  unsigned f = ((unsigned)e << 23) | ((hi & 0xFFFFFu) << 3) | ((unsigned)raw >> 29);
  if (e <= 0) f = 0;
  if (e >= 255) f = 0x7F7FFFFFu;
  const unsigned o = neg ? ~(f | 0x80000000u) : f | 0x80000000u;
  return up ? o : ~o;
}
__device__ __forceinline__ float lr_image_value(unsigned o) {
  return __uint_as_float((o & 0x80000000u) ? o & 0x7FFFFFFFu : ~o);
}
// distance of an image above the segment's smallest, as a float
template <class K> __device__ __forceinline__ float lr_above(unsigned o, unsigned omin) {
  if constexpr (sizeof(K) == 4) return __uint2float_rn(o - omin);
  else return __fsub_rn(lr_image_value(o), lr_image_value(omin));
}
// buckets per unit of distance; 0: one bucket (equal keys, or a range too wide for a float)
template <class K> __device__ __forceinline__ float lr_scale(unsigned omin, unsigned omax, int len) {
  const float r = lr_above<K>(omax, omin);
  return r > 0.0f ? __fdividef((float)len, sizeof(K) == 4 ? r + 1.0f : r) : 0.0f;
}

// Where the elements are placed by bucket.  A 32-bit key shares an 8-byte word
// with its element (relative to the tile) and its place in the bucket, so one
// load and one comparison order two elements by key, then by element.
template <class K> struct LrPut;
template <> struct LrPut<unsigned> {
  unsigned long long *w;  // key << 24 | element << 12 | place
  static constexpr size_t bytes = (size_t)(LR_CAP + 1) * 8;
  __device__ explicit LrPut(unsigned char *mem) : w((unsigned long long *)mem) {}
  struct Item { unsigned long long v; };
  __device__ Item item(unsigned k, int l, int pos) const { return {(unsigned long long)k << 24 | (unsigned)(l << 12 | pos)}; }
  __device__ void set(int at, const Item &x) const { w[at] = x.v; }
  __device__ Item get(int at) const { return {w[at]}; }
  __device__ void sentinel(int at) const { w[at] = ~0ULL; }
  static __device__ int place(const Item &x) { return (int)(x.v & 0xFFFu); }
  static __device__ int element(const Item &x) { return (int)((x.v >> 12) & 0xFFFu); }
  static __device__ int before(const Item &x, const Item &y) { return x.v < y.v ? 1 : 0; }
};
template <> struct LrPut<unsigned long long> {
  unsigned long long *w;  // keys
  unsigned *id;           // element << 12 | place
  static constexpr size_t bytes = (size_t)(LR_CAP + 2) * 12;
  __device__ explicit LrPut(unsigned char *mem) : w((unsigned long long *)mem), id((unsigned *)(w + LR_CAP + 2)) {}
  struct Item { unsigned long long v; unsigned i; };
  __device__ Item item(unsigned long long k, int l, int pos) const { return {k, (unsigned)(l << 12 | pos)}; }
  __device__ void set(int at, const Item &x) const { w[at] = x.v; id[at] = x.i; }
  __device__ Item get(int at) const { return {w[at], id[at]}; }
  __device__ void sentinel(int at) const { id[at] = ~0u; }
  static __device__ int place(const Item &x) { return (int)(x.i & 0xFFFu); }
  static __device__ int element(const Item &x) { return (int)(x.i >> 12); }
  static __device__ int before(const Item &x, const Item &y) {
    return (int)(x.v < y.v) | ((int)(x.v == y.v) & (int)(x.i < y.i));
  }
};
// the placed elements (in the digit passes: keys and the first numbers), the
// second half-words, and the digit passes' counts per warp
template <class K> constexpr size_t lr_smem() {
  return align16(LrPut<K>::bytes) + LR_CAP * 2 + (LR_T + 8) * 2 + LR_WARPS * 256 * 2;
}

// Bound by issue: about 300 instructions per element and lane (79 % of issue
// slots), 2^24 int keys in geometric(64) segments 160 us where the bytes take
// 20; the whole call 1284 -> 181 us against sorting by (segment, key)
// globally (7 digit passes).  The shape: 512 threads and four CTAs per SM;
// with 256 threads each holding rows of eight consecutive keys in shared
// memory 280 us, with bucket ends found in a bit map of bucket starts instead
// of from the places 219 us.
//
// Positions are relative to the tile's first element.  Element l is handled
// by lane l % 32 of the warp and step that hold its 32-element word, its key
// in a register from the load on.
template <class K>
__global__ void __launch_bounds__(LR_BLOCK, lr_minb<K>()) k_rank_local(const K *__restrict__ src,
                                                                       int *__restrict__ rank, SegView sv, int n,
                                                                       int up, int whole, LongSegs ls) {
  extern __shared__ __align__(16) unsigned char lr_mem[];
  const LrPut<K> put(lr_mem);
  unsigned short *s_cnt = (unsigned short *)(lr_mem + align16(LrPut<K>::bytes));  // [LR_CAP] bucket counts, starts; then ranks
  unsigned short *s_start = s_cnt + LR_CAP;                        // [LR_T + 8] segment starts
  unsigned short *s_wc = s_start + LR_T + 8;                       // [LR_WARPS][256] digit passes: a warp's counts
  // the segments' smallest and largest images, then smallest and scale, where the elements are placed later
  uint2 *s_mm = (uint2 *)lr_mem;
  static_assert(LR_T * 8 <= LrPut<K>::bytes, "they fit there");
  __shared__ unsigned s_hw[LR_WORDS];              // head bits
  __shared__ unsigned short s_hp[LR_WORDS];        // heads before the word
  __shared__ unsigned s_red[3][LR_WARPS];
  __shared__ unsigned long long s_red64[LR_WARPS];
  __shared__ int s_from, s_last, s_end, s_nseg;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lo = whole ? 0 : blockIdx.x * LR_T;
  const int left = min(n - lo, LR_CAP);  // elements there are from lo on, up to a full CTA

  // ---- the tile's keys and head bits; the bits of the longest segment that can start in it
  K k[LR_STEPS];
#pragma unroll
  for (int c = 0; c < LR_STEPS; c++) {
    const int l = c * LR_BLOCK + tid;
    if ((whole || c < LR_T / LR_BLOCK) && l < left) k[c] = __ldcs(src + lo + l);
  }
  for (int i = tid; i < LR_WORDS; i += LR_BLOCK) {
    unsigned w = 0;
    if (32 * i < n - lo) w = sv.bits ? __ldg(sv.bits + (lo >> 5) + i) : (i == 0 ? 1u : 0u);
    s_hw[i] = w;
  }
  for (int i = tid; i < LR_CAP / 8; i += LR_BLOCK) ((uint4 *)s_cnt)[i] = make_uint4(0, 0, 0, 0);
  for (int i = tid; i < LR_T / 2; i += LR_BLOCK) ((uint4 *)s_mm)[i] = make_uint4(0xFFFFFFFFu, 0, 0xFFFFFFFFu, 0);
  __syncthreads();
  if (warp == 0) {
    const int tile = whole ? LR_CAP : LR_T;  // heads before it are this CTA's
    int from = LR_CAP, last = -1, end = whole ? left : (left < LR_CAP ? left : LR_CAP + 1);
    unsigned run = 0;
    for (int i0 = 0; i0 < LR_WORDS; i0 += 32) {
      const unsigned w = i0 + lane < LR_WORDS ? s_hw[i0 + lane] : 0u;
      const int at = 32 * (i0 + lane);
      if (w && at < tile) {
        from = min(from, at + __ffs(w) - 1);
        last = max(last, at + 31 - __clz(w));
      } else if (w) {
        end = min(end, at + __ffs(w) - 1);
      }
      const int h = at < tile ? __popc(w) : 0;
      int incl = h;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int x = shfl_up(incl, d);
        if (lane >= d) incl += x;
      }
      if (i0 + lane < LR_WORDS) s_hp[i0 + lane] = (unsigned short)(run + incl - h);
      run += shfl_idx(incl, 31);
    }
    from = __reduce_min_sync(0xffffffffu, from);
    last = __reduce_max_sync(0xffffffffu, last);
    end = __reduce_min_sync(0xffffffffu, end);
    if (lane == 0) {
      int num = -1;
      if (last >= 0 && !whole && end - last > LR_MAX) {
        // a long last segment: left to the digit passes
        const int s = seg_of(sv, lo + last), a = __ldg(sv.off + s), b = __ldg(sv.off + s + 1);
        const unsigned long long at = atomicAdd(ls.total, (1ULL << 32) | (unsigned)(b - a));
        num = (int)(at >> 32);
        ls.first[num] = a;
        ls.base[num] = (int)(unsigned)at;
        end = last;
        --run;
      }
      if (!whole) ls.of_tile[blockIdx.x] = num;
      s_from = from;
      s_last = last;
      s_end = end;
      s_nseg = (int)run;
      if (last >= 0) s_start[run] = (unsigned short)end;
    }
  }
  __syncthreads();
  const int from = s_from, end = s_end, nseg = s_nseg;
  if (s_last < 0 || end <= from) return;  // no segment starts here, or only a long one
#pragma unroll
  for (int c = 0; c < LR_STEPS; c++) {
    const int l = c * LR_BLOCK + tid;
    if (!whole && c >= LR_T / LR_BLOCK && l < end) k[c] = __ldcs(src + lo + l);
  }

  // ---- segment starts, smallest and largest images
#pragma unroll
  for (int c = 0; c < LR_STEPS; c++) {
    const int l0 = c * LR_BLOCK + warp * 32, l = l0 + lane;
    if (l0 >= end) break;
    if (l0 + 31 >= from) {
      k[c] = rk_key(k[c], up);
      const unsigned hb = l0 < LR_T || whole ? s_hw[l0 >> 5] : 0u;
      const int num = (int)s_hp[l0 >> 5] + __popc(hb & (0xFFFFFFFFu >> (31 - lane))) - 1;
      const bool mine = l >= from && l < end;
      if (mine && ((hb >> lane) & 1u)) s_start[num] = (unsigned short)l;
      const unsigned o = mine ? lr_image(k[c], up) : 0u;
      unsigned mn = mine ? o : 0xFFFFFFFFu, mx = o;
      if ((hb & ~1u) == 0) {  // one segment
        mn = __reduce_min_sync(0xffffffffu, mn);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0 && num >= 0) { atomicMin(&s_mm[num].x, mn); atomicMax(&s_mm[num].y, mx); }
      } else {
        const unsigned hl = hb & (0xFFFFFFFFu >> (31 - lane));
        const int reach = hl ? lane - (31 - __clz(hl)) : lane;  // lanes of my segment before me
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const unsigned a = shfl_up(mn, d), b = shfl_up(mx, d);
          if (reach >= d) { mn = min(mn, a); mx = max(mx, b); }
        }
        const bool tail = lane == 31 || ((hb >> (lane + 1)) & 1u);
        if (tail && num >= 0 && num < nseg) { atomicMin(&s_mm[num].x, mn); atomicMax(&s_mm[num].y, mx); }
      }
    }
  }
  __syncthreads();
  for (int s = tid; s < nseg; s += LR_BLOCK)
    s_mm[s].y = __float_as_uint(lr_scale<K>(s_mm[s].x, s_mm[s].y, (int)s_start[s + 1] - (int)s_start[s]));
  __syncthreads();
  // ---- every element's bucket and its place among the bucket's elements
  unsigned bp[LR_STEPS];                 // bucket | place << 16
  unsigned short first[LR_STEPS];        // its segment's start
#pragma unroll
  for (int c = 0; c < LR_STEPS; c++) {
    const int l0 = c * LR_BLOCK + warp * 32, l = l0 + lane;
    if (l0 >= end) break;
    if (l >= from && l < end) {
      const unsigned hb = l0 < LR_T || whole ? s_hw[l0 >> 5] : 0u;
      const int num = (int)s_hp[l0 >> 5] + __popc(hb & (0xFFFFFFFFu >> (31 - lane))) - 1;
      const int start = s_start[num], last = (int)s_start[num + 1] - start - 1;
      const uint2 mm = s_mm[num];
      const float x = __fmul_rn(lr_above<K>(lr_image(k[c], up), mm.x), __uint_as_float(mm.y));
      const int b = start + min(__float2int_rd(x), last);
      const int sh = (b & 1) * 16;
      first[c] = (unsigned short)start;
      bp[c] = (unsigned)b | (((atomicAdd((unsigned *)s_cnt + (b >> 1), 1u << sh) >> sh) & 0xFFFFu) << 16);
    }
  }
  __syncthreads();
  // ---- bucket starts (eight consecutive buckets of a thread), and how crowded they are
  {
    constexpr int PER = LR_CAP / LR_BLOCK;
    static_assert(PER == 8, "one 16-byte access of 16-bit counts");
    unsigned v[PER], sum = 0, sq = 0, top = 0, incl = 0;
    const bool used = warp * 32 * PER < end;  // the whole warp alike
    if (used) {
      const uint4 w = ((const uint4 *)s_cnt)[tid];
      v[0] = w.x & 0xFFFFu; v[1] = w.x >> 16; v[2] = w.y & 0xFFFFu; v[3] = w.y >> 16;
      v[4] = w.z & 0xFFFFu; v[5] = w.z >> 16; v[6] = w.w & 0xFFFFu; v[7] = w.w >> 16;
#pragma unroll
      for (int q = 0; q < PER; q++) {
        sum += v[q];
        sq += v[q] * v[q];
        top = max(top, v[q]);
      }
      incl = sum;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned x = shfl_up(incl, d);
        if (lane >= d) incl += x;
      }
      sq = __reduce_add_sync(0xffffffffu, sq);
      top = __reduce_max_sync(0xffffffffu, top);
    }
    if (lane == 31) { s_red[0][warp] = incl; s_red[1][warp] = sq; s_red[2][warp] = top; }
    __syncthreads();
    if (used) {
      unsigned at = (unsigned)from + incl - sum;
#pragma unroll
      for (int q = 0; q < LR_WARPS; q++)
        if (q < warp) at += s_red[0][q];
#pragma unroll
      for (int q = 0; q < PER; q++) {
        const unsigned x = v[q];
        v[q] = at;
        at += x;
      }
      ((uint4 *)s_cnt)[tid] = make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
    }
  }
  unsigned sq = lane < LR_WARPS ? s_red[1][lane] : 0u, top = lane < LR_WARPS ? s_red[2][lane] : 0u;
  sq = __reduce_add_sync(0xffffffffu, sq);
  top = __reduce_max_sync(0xffffffffu, top);
  __syncthreads();

  if (top <= LR_CROWD_MAX && sq <= LR_CROWD_MEAN * (unsigned)(end - from)) {
#pragma unroll
    for (int c = 0; c < LR_STEPS; c++) {
      const int l = c * LR_BLOCK + tid;
      if (l - lane >= end) break;
      if (l >= from && l < end) put.set(s_cnt[bp[c] & 0xFFFFu] + (bp[c] >> 16), put.item(k[c], l, bp[c] >> 16));
    }
    if (tid == 0) put.sentinel(end);
    __syncthreads();
    // an element's rank: its bucket's start, and the bucket's elements before
    // it (a bucket ends where the places start again)
#pragma unroll
    for (int c = 0; c < LR_STEPS; c++) {
      const int j = c * LR_BLOCK + tid;
      if (j - lane >= end) break;
      if (j >= from && j < end) {
        const auto me = put.get(j);
        const int b0 = j - LrPut<K>::place(me);
        int r = b0;
        for (int i = b0;; i++) {
          const auto x = put.get(i);
          if (LrPut<K>::place(x) != i - b0) break;
          r += LrPut<K>::before(x, me);
        }
        s_cnt[LrPut<K>::element(me)] = (unsigned short)r;  // the bucket starts are no longer read
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < LR_STEPS; c++) {
      const int l = c * LR_BLOCK + tid;
      if (l - lane >= end) break;
      if (l >= from && l < end) __stcs(rank + lo + l, (int)s_cnt[l] - (int)first[c]);
    }
    return;
  }

  // ---- crowded buckets: stable digit passes over the elements' numbers,
  // by key and then by segment
  K *s_key = (K *)lr_mem;
  unsigned short *s_id = (unsigned short *)(s_key + LR_CAP);
  static_assert(LR_CAP * (sizeof(K) + 2) <= LrPut<K>::bytes, "keys and numbers fit where the elements were placed");
  unsigned short *idin = s_id, *idout = s_cnt;
  const int cnt = end - from;
#pragma unroll
  for (int c = 0; c < LR_STEPS; c++) {
    const int l = c * LR_BLOCK + tid;
    if (l >= from && l < end) {
      s_key[l] = k[c];
      s_id[l - from] = (unsigned short)l;
    }
  }
  __syncthreads();
  unsigned long long diff = 0;
#pragma unroll
  for (int c = 0; c < LR_STEPS; c++) {
    const int l = c * LR_BLOCK + tid;
    if (l >= from && l < end) diff |= (unsigned long long)(k[c] ^ s_key[from]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) diff |= __shfl_xor_sync(0xffffffffu, diff, d);
  if (lane == 0) s_red64[warp] = diff;
  __syncthreads();
  diff = 0;
#pragma unroll
  for (int w = 0; w < LR_WARPS; w++) diff |= s_red64[w];
  auto seg_num = [&](int l) {
    const unsigned hb = l < LR_T || whole ? s_hw[l >> 5] : 0u;
    return (int)s_hp[l >> 5] + __popc(hb & (0xFFFFFFFFu >> (31 - (l & 31)))) - 1;
  };
  const int span = (((cnt + LR_WARPS - 1) / LR_WARPS) + 31) & ~31;  // consecutive places of a warp
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll 1
  for (int q = 0; q < (int)sizeof(K) + 2; q++) {
    const bool by_key = q < (int)sizeof(K);
    const int shift = 8 * (by_key ? q : q - (int)sizeof(K));
    if (by_key ? ((diff >> shift) & 255) == 0 : ((nseg - 1) >> shift) == 0) continue;  // all agree
    for (int i = tid; i < LR_WARPS * 256; i += LR_BLOCK) s_wc[i] = 0;
    __syncthreads();
    unsigned short *wc = s_wc + warp * 256;
    unsigned wr[LR_STEPS];
#pragma unroll
    for (int c = 0; c < LR_STEPS; c++) {
      wr[c] = 0xFFFFFFFFu;
      if (c * 32 < span) {
        const int e = warp * span + c * 32 + lane;
        int d = -1, id = 0;
        if (e < cnt) {
          id = idin[e];
          d = by_key ? (int)((s_key[id] >> shift) & 255) : (seg_num(id) >> shift) & 255;
        }
        const unsigned peers = warp_match8(d);
        unsigned r = 0;
        if (d >= 0) r = wc[d] + __popc(peers & lt);
        __syncwarp();
        if (d >= 0 && (peers & lt) == 0) wc[d] = (unsigned short)(wc[d] + __popc(peers));
        __syncwarp();
        if (d >= 0) wr[c] = (r << 20) | ((unsigned)id << 8) | (unsigned)d;
      }
    }
    __syncthreads();
    unsigned tot = 0, incl = 0;  // digit tid: the warps before, then the digits before
    if (tid < 256) {
#pragma unroll
      for (int w = 0; w < LR_WARPS; w++) {
        const unsigned x = s_wc[w * 256 + tid];
        s_wc[w * 256 + tid] = (unsigned short)tot;
        tot += x;
      }
      incl = tot;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned x = shfl_up(incl, d);
        if (lane >= d) incl += x;
      }
      if (lane == 31) s_red[0][warp] = incl;
    }
    __syncthreads();
    if (tid < 256) {
      unsigned loc = incl - tot;
#pragma unroll
      for (int w = 0; w < 8; w++)
        if (w < warp) loc += s_red[0][w];
#pragma unroll
      for (int w = 0; w < LR_WARPS; w++) s_wc[w * 256 + tid] = (unsigned short)(s_wc[w * 256 + tid] + loc);
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < LR_STEPS; c++)
      if (wr[c] != 0xFFFFFFFFu) idout[wc[wr[c] & 255u] + (wr[c] >> 20)] = (unsigned short)((wr[c] >> 8) & 0xFFFu);
    __syncthreads();
    unsigned short *sorted = idout;
    idout = idin;
    idin = sorted;
  }
  for (int p = tid; p < cnt; p += LR_BLOCK) {
    const int id = idin[p];
    rank[lo + id] = from + p - (int)s_start[seg_num(id)];
  }
}

template <class K>
void rank_local(const void *src, int *rank, const SegView &sv, int n, int up, bool whole, const LongSegs &ls) {
  static bool attr = false;
  if (!attr) {
    GCVL_CK(cudaFuncSetAttribute(k_rank_local<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lr_smem<K>()));
    attr = true;
  }
  k_rank_local<K><<<whole ? 1 : lr_tiles(n), LR_BLOCK, lr_smem<K>(), stream()>>>((const K *)src, rank, sv, n, up,
                                                                               whole ? 1 : 0, ls);
  launch_check("k_rank_local");
}
template void rank_local<unsigned>(const void *, int *, const SegView &, int, int, bool, const LongSegs &);
template void rank_local<unsigned long long>(const void *, int *, const SegView &, int, int, bool, const LongSegs &);

}  // namespace gcvl
