// The walk kernel's own text (walk_extract.h, cut out of pk_compact.cu by the test) run on the
// host, one coroutine per lane: a lane runs until it reaches a warp-wide operation, and no
// lane passes one before all have reached it -- all that the hardware promises.  Prints what
// the walk leaves, once with lane 0 always ahead of the others and once with it behind.
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <ucontext.h>

#include <algorithm>
#include <functional>
#include <vector>

#define __device__
#define __global__
#define __forceinline__ inline
#define __restrict__
#define __launch_bounds__(...)
using std::min;
struct uint2 { uint32_t x, y; };
struct int2 { int32_t x, y; };
struct int3 { int32_t x, y, z; };
struct alignas(16) uint4 { uint32_t x, y, z, w; };
static uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return uint4{x, y, z, w}; }
static struct { unsigned x; } threadIdx, blockIdx, blockDim;
static uint4 __ldg(const uint4* p) { return *p; }
static unsigned long long atomicAdd(unsigned long long* p, unsigned long long v) { return (*p += v) - v; }
static void atomicOr(uint32_t* p, uint32_t v) { *p |= v; }

static ucontext_t g_main, g_lane[32];
static int g_now, g_at[32];  // the running lane; where each lane stands (-1: returned)
static uint64_t g_slot[32];
static void sync_at(int line) {
  g_at[g_now] = line;
  swapcontext(&g_lane[g_now], &g_main);
}
template <typename T>
static T shfl_at(int line, T v, int from) {
  g_slot[g_now] = (uint64_t)v;
  sync_at(line);
  const T r = (T)g_slot[from];
  sync_at(-2 - line);
  return r;
}
#define __syncwarp() sync_at(__LINE__)
#define __shfl_sync(mask, v, from) shfl_at(__LINE__, v, from)

#include "walk_extract.h"

static std::function<void()> g_kernel;
static void lane_main() {
  g_kernel();
  g_at[g_now] = -1;
}

static void run_warp(bool lane0_first) {
  static std::vector<char> stacks(32 * (64 << 10));
  for (int l = 0; l < 32; l++) {
    getcontext(&g_lane[l]);
    g_lane[l].uc_stack.ss_sp = &stacks[l * (64 << 10)];
    g_lane[l].uc_stack.ss_size = 64 << 10;
    g_lane[l].uc_link = &g_main;
    g_at[l] = 0;
    makecontext(&g_lane[l], lane_main, 0);
  }
  while (g_at[0] != -1) {
    for (int i = 0; i < 32; i++) {
      g_now = lane0_first ? i : 31 - i;
      threadIdx.x = (unsigned)g_now;
      swapcontext(&g_main, &g_lane[g_now]);
    }
    for (int l = 1; l < 32; l++)
      if (g_at[l] != g_at[0]) {
        printf("lanes 0 and %d part\n", l);
        exit(0);
      }
  }
}

int main(int argc, char** argv) {
  const bool lane0_first = argc > 1 && !strcmp(argv[1], "first");
  const int L = 7;
  // one begin; a prefix of four wires, each to a prefix of two, each to one, each to a terminal
  std::vector<WStep> step(28);
  for (int i = 0; i < 28; i++) {
    step[i] = WStep{};
    step[i].xoff = 100 * (i + 1);
    step[i].xlen = 1 + i % 5;
    step[i].cnt = i < 4 ? 2 : 1;
    step[i].next = i < 4 ? 4 + 2 * i : i < 12 ? 12 + (i - 4) : 20 + (i - 12);
    step[i].n_next = i < 4 ? 2 : 1;
    if (i >= 20) step[i].xlen |= kTerm;
  }
  uint64_t key = 0x1b1b;
  uint32_t eoff[2] = {0, 2}, xlen[2] = {3u | kTerm, 0}, err = 0;
  uint64_t xoff[2] = {7, 0};
  int32_t vis[2] = {8, 0};
  int2 beg[2] = {{0, 4}, {0, 0}};
  Side<uint64_t> s{};
  s.key = &key;
  s.eoff = eoff;
  s.xlen = xlen;
  s.xoff = xoff;
  s.vis = vis;
  s.beg = beg;
  const uint2 begins[1] = {{0, 0}};
  const uint32_t cap = 64;
  std::vector<WResume> resume(cap);
  std::vector<WPath> path(cap);
  std::vector<WPiece> pieces(256);
  std::vector<WContig> contigs(64);
  unsigned long long recorded[2] = {0, 0};
  uint4 col[1] = {}, off[1] = {};
  uint64_t ct_off[64] = {};
  std::vector<uint8_t> out(4096);
  blockDim.x = 128;
  g_kernel = [&] {
    k_walk<uint64_t, 0>(s, L, begins, 1, step.data(), resume.data(), path.data(), cap, col, nullptr, nullptr,
                        pieces.data(), nullptr, contigs.data(), 64, 256, recorded, &err);
  };
  run_warp(lane0_first);
  auto dump = [&](const char* what, size_t np) {
    printf("%s err %u contigs %u bases %u pieces %u\n", what, err, col[0].x, col[0].y, col[0].z);
    for (size_t i = 0; i < np; i++)
      printf("%llu %llu %u\n", (unsigned long long)pieces[i].src, (unsigned long long)pieces[i].dst, pieces[i].len);
  };
  dump("recorded", recorded[1]);
  for (size_t i = 0; i < recorded[0]; i++)
    printf("contig %llu %u\n", (unsigned long long)contigs[i].dst, contigs[i].index);
  std::fill(pieces.begin(), pieces.end(), WPiece{});
  g_kernel = [&] {
    k_walk<uint64_t, 1>(s, L, begins, 1, step.data(), resume.data(), path.data(), cap, nullptr, off, ct_off,
                        pieces.data(), out.data(), nullptr, 0, 0, nullptr, &err);
  };
  run_warp(lane0_first);
  dump("written", col[0].z);
  for (uint32_t i = 0; i < col[0].x; i++) printf("contig %llu\n", (unsigned long long)ct_off[i]);
  for (uint32_t i = 0; i < col[0].y; i++) printf("%d", out[i]);
  printf("\n");
}
