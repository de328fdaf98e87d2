// Test-only: several thread blocks of the emulated kernels (one thread each),
// for the host build of the refiner's sources.  Included before every source.
//
// The blocks of a launch are host threads of which one runs at a time.  A block
// runs until it waits at a barrier of its team and another one goes on, so that
// every order of the blocks' phases can be had: the schedule says which of the
// blocks that can go on is taken (0: the lowest, which lets the first block run
// ahead of all others; 1: the highest; beyond: drawn with that seed).  When no
// block can go on, the waits are given up, as a barrier's limit does on the GPU.
#pragma once
#include <condition_variable>
#include <mutex>
#include <random>
#include <thread>
#include <vector>

#include "cuda_fake/cuda_runtime.h"

inline thread_local dim3_emu gqm_emu_block = {0, 0, 0}, gqm_emu_grid = {1, 1, 1};
#define blockIdx gqm_emu_block
#define gridDim gqm_emu_grid

struct GqmEmuGrid {
  std::mutex m;
  std::condition_variable cv;
  int running = -1;
  bool stuck = false;
  struct Block {
    bool done = false;
    const unsigned long long *word = nullptr;
    unsigned long long target = 0;
  };
  std::vector<Block> blocks;
  std::mt19937 rng;
};
inline int gqm_emu_order = 0;           // the schedule
inline int gqm_emu_stuck = 0;           // launches whose blocks could not go on
inline long long gqm_emu_break = -1;    // waits until a launch's waits are given up (-1: never)
inline thread_local GqmEmuGrid *gqm_emu_cur = nullptr;
extern "C" __attribute__((weak)) void gqm_emu_schedule(int order) {
  gqm_emu_order = order;
  gqm_emu_stuck = 0;
}
extern "C" __attribute__((weak)) void gqm_emu_break_at(long long wait) { gqm_emu_break = wait; }
extern "C" __attribute__((weak)) int gqm_emu_stuck_count(void) { return gqm_emu_stuck; }

inline void gqm_emu_next(GqmEmuGrid &g) {
  std::vector<int> ready;
  bool left = false;
  for (int b = 0; b < (int)g.blocks.size(); ++b) {
    const GqmEmuGrid::Block &x = g.blocks[b];
    if (x.done) continue;
    left = true;
    if (g.stuck || !x.word || *x.word >= x.target) ready.push_back(b);
  }
  if (ready.empty() && left) {
    g.stuck = true;
    ++gqm_emu_stuck;
    gqm_emu_next(g);
    return;
  }
  g.running = ready.empty() ? -1
              : gqm_emu_order == 0 ? ready.front()
              : gqm_emu_order == 1 ? ready.back() : ready[g.rng() % ready.size()];
  g.cv.notify_all();
}
inline bool gqm_emu_wait(const unsigned long long *word, unsigned long long target) {
  GqmEmuGrid &g = *gqm_emu_cur;
  const int me = (int)gqm_emu_block.x;
  std::unique_lock<std::mutex> lock(g.m);
  if (gqm_emu_break >= 0 && gqm_emu_break-- == 0) g.stuck = true;
  g.blocks[me].word = word;
  g.blocks[me].target = target;
  gqm_emu_next(g);
  g.cv.wait(lock, [&] { return g.running == me; });
  g.blocks[me].word = nullptr;
  return !g.stuck && *word >= target;
}
inline int gqm_emu_largest = 0;  // most blocks of a launch since that was last asked
extern "C" __attribute__((weak)) int gqm_emu_largest_launch(void) {
  const int n = gqm_emu_largest;
  gqm_emu_largest = 0;
  return n;
}
template <class F>
void gqm_emu_launch(int n, F f) {
  gqm_emu_largest = std::max(gqm_emu_largest, n);
  GqmEmuGrid g;
  g.blocks.resize(n);
  g.rng.seed((unsigned)gqm_emu_order);
  std::vector<std::thread> pool;
  for (int b = 0; b < n; ++b)
    pool.emplace_back([&, b] {
      gqm_emu_cur = &g;
      gqm_emu_block.x = (unsigned)b;
      gqm_emu_grid.x = (unsigned)n;
      {
        std::unique_lock<std::mutex> lock(g.m);
        g.cv.wait(lock, [&] { return g.running == b; });
      }
      f();
      std::unique_lock<std::mutex> lock(g.m);
      g.blocks[b].done = true;
      gqm_emu_next(g);
    });
  {
    std::unique_lock<std::mutex> lock(g.m);
    gqm_emu_next(g);
  }
  for (auto &t : pool) t.join();
}
inline int gqm_emu_blocks = 4;  // most blocks of a launch
extern "C" __attribute__((weak)) void gqm_emu_set_blocks(int n) { gqm_emu_blocks = n; }
#define GQM_EMU_BLOCKS gqm_emu_blocks
#define GQM_EMU_GRID(blocks, call) gqm_emu_launch(blocks, [&] { call; })
#define GQM_EMU_WAIT(word, target) gqm_emu_wait(word, target)
