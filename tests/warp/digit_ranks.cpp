// The digit ranks of a warp (neslgpu_gb300/csrc/rank_warp.cuh) with its 32
// lanes as fibres that take turns at every atomic, vote, shuffle and
// __syncwarp(), in an order drawn from a seed: what CUDA promises of a warp,
// and no more.  Prints the number of elements whose rank is wrong.
#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

namespace {
constexpr int LANES = 32;
struct Fibre {
  ucontext_t ctx;
  std::vector<char> stack = std::vector<char>(64 << 10);
  bool done = false, waits = false;  // waits: at a barrier
};
Fibre fibres[LANES];
ucontext_t scheduler;
int me, arrived;
uint32_t slot[LANES];
std::mt19937 rng;
void (*body)(int);
int lowest_last;  // lanes in descending order instead of a drawn one

void yield() { swapcontext(&fibres[me].ctx, &scheduler); }
void barrier() {
  if (++arrived == LANES) {
    arrived = 0;
    for (Fibre &f : fibres) f.waits = false;
  } else {
    fibres[me].waits = true;
  }
  yield();
}
void enter() {
  body(me);
  fibres[me].done = true;
  yield();
}
void run_warp(void (*f)(int)) {
  body = f;
  arrived = 0;
  for (int l = 0; l < LANES; l++) {
    Fibre &x = fibres[l];
    x.done = x.waits = false;
    getcontext(&x.ctx);
    x.ctx.uc_stack.ss_sp = x.stack.data();
    x.ctx.uc_stack.ss_size = x.stack.size();
    x.ctx.uc_link = &scheduler;
    makecontext(&x.ctx, enter, 0);
  }
  for (;;) {
    int ready[LANES], n = 0;
    for (int l = 0; l < LANES; l++)
      if (!fibres[l].done && !fibres[l].waits) ready[n++] = l;
    if (n == 0) break;
    me = lowest_last ? ready[n - 1] : ready[rng() % n];
    swapcontext(&scheduler, &fibres[me].ctx);
  }
}
}  // namespace

#define __device__
#define __forceinline__ inline
static void __syncwarp() { barrier(); }
static unsigned __shfl_sync(unsigned, unsigned v, int lane) {
  slot[me] = v;
  barrier();
  const unsigned r = slot[lane & 31];
  barrier();
  return r;
}
static bool __all_sync(unsigned, bool v) {
  slot[me] = v;
  barrier();
  bool r = true;
  for (uint32_t x : slot) r = r && x;
  barrier();
  return r;
}
static unsigned atomicOr(unsigned *p, unsigned v) { const unsigned o = *p; *p |= v; yield(); return o; }
static unsigned atomicAdd(unsigned *p, unsigned v) { const unsigned o = *p; *p += v; yield(); return o; }
static int __popc(unsigned x) { return __builtin_popcount(x); }
static int __ffs(unsigned x) { return __builtin_ffs((int)x); }
#include "rank_warp.cuh"

namespace {
constexpr int MAXI = 20;
uint32_t keys[MAXI][LANES], ranks[MAXI][LANES], cnt[256], masks[5 * 256];

template <int ITEMS, int G> void lane_body(int lane) {
  uint32_t k[ITEMS], wr[ITEMS];
  for (int c = 0; c < ITEMS; c++) k[c] = keys[c][lane];
  warp_digit_ranks<ITEMS, G>(wr, k, 8, cnt, masks, 256, lane);
  for (int c = 0; c < ITEMS; c++) ranks[c][lane] = wr[c];
}

template <int ITEMS, int G> int wrong(int digits) {
  for (int c = 0; c < ITEMS; c++)
    for (int l = 0; l < LANES; l++) keys[c][l] = (uint32_t)(rng() % digits * 37 % 256) << 8 | (rng() & 255u) | 0xABu << 24;
  if (digits > 1) {  // an item of one digit among them
    for (int l = 0; l < LANES; l++) keys[1][l] = keys[0][3];
  }
  memset(cnt, 0, sizeof cnt);
  memset(masks, 0, sizeof masks);
  run_warp(lane_body<ITEMS, G>);
  uint32_t seen[256] = {};
  int bad = 0;
  for (int c = 0; c < ITEMS; c++)
    for (int l = 0; l < LANES; l++) {
      const uint32_t d = keys[c][l] >> 8 & 255u;
      bad += ranks[c][l] != (seen[d]++ << 8 | d);
    }
  bad += memcmp(seen, cnt, sizeof cnt) != 0;
  for (uint32_t m : masks) bad += m != 0;
  return bad;
}
}  // namespace

int main(int argc, char **argv) {
  const int digits = atoi(argv[1]);
  lowest_last = argc > 2 && !strcmp(argv[2], "descending");
  long bad = 0;
  for (unsigned seed = 0; seed < (lowest_last ? 1u : 20u); seed++) {
    rng.seed(seed * 977 + digits);
    bad += wrong<20, 5>(digits) + wrong<16, 4>(digits) + wrong<8, 2>(digits);
  }
  printf("%ld\n", bad);
}
