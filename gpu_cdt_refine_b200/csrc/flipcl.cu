// The flip-flop loop of the single-domain engine in one launch.
//
// flipFlop (GPU_Refine/refine.cu:2328-2490) runs a step after another until no
// triangle is flagged.  Here the whole loop is one cooperative launch whose
// blocks separate the phases of a step (flip_step in kernels.cuh) with a
// barrier in global memory, and no launch, condition node or host read stands
// between two phases or two steps.
//
// Most steps are small: of the ~1,030 steps of a 2,000,000-point refinement,
// ~680 have at most 1,024 active triangles, and all blocks' barriers would
// cost more than such a step's work.  Those steps are run by one team of the
// first blocks while the others wait at one barrier: by default block 0 alone,
// whose barrier is __syncthreads() and which keeps the list lengths, the queues
// and the decisions in shared memory; gqm_tuning.small_cluster asks for 8 or 16
// blocks instead.
//
// Threads: 512 per SM at up to 128 registers.  640, 768 and 1,024 threads (96,
// 80 and 64 registers) gave 72.5, 72.7 and 75.2 ms for the refinement of
// 2,000,000 points against 71.2 ms: more warps do not shorten the chains.
//
// Every wait is bounded; one that runs out records GQM_ERR_TOPOLOGY and every
// block leaves the loop.
#define GQM_CLUSTER_MODE 1
#define gqm gqm_cl
#include <cuda_runtime.h>

#include <chrono>
#include <cstring>

#include "../../include/gqm_refine.h"
#include "kernels.cuh"

namespace gqm {

// One thread block.
struct BlockTeam {
  __device__ __forceinline__ int tid() const { return (int)threadIdx.x; }
  __device__ __forceinline__ int size() const { return (int)blockDim.x; }
  __device__ __forceinline__ bool lead() const { return threadIdx.x == 0; }
  __device__ __forceinline__ bool sync() {
    __syncthreads();
    return true;
  }
};

// The first `nb` blocks of the launch.  A barrier adds one arrival per block to
// a word that only grows (it starts at zero with every refinement); a block
// waits until all arrivals of its own barrier have been counted.  The arrival
// is a reduction with no answer to wait for, and the wait polls one word.
struct GridBar {
  unsigned long long arrived;  // arrivals of all barriers
  unsigned long long base;     // arrivals when the current launch began
  int broken;
};
constexpr unsigned kBarrierPolls = 1u << 25;  // tens of seconds
struct GridTeam {
  GridBar *bar;
  int nb;
  unsigned long long target;
  int *err;
  __device__ __forceinline__ int tid() const { return (int)(blockIdx.x * blockDim.x + threadIdx.x); }
  __device__ __forceinline__ int size() const { return nb * (int)blockDim.x; }
  __device__ __forceinline__ bool lead() const { return blockIdx.x == 0 && threadIdx.x == 0; }
  __device__ __forceinline__ bool sync() {
#ifdef GQM_HOST_EMU
    return true;
#else
    target += (unsigned long long)nb;
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(&bar->arrived), "l"(1ull) : "memory");
      unsigned polls = 0;
      unsigned long long v;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&bar->arrived) : "memory");
        if (v >= target) break;
        if (++polls > 64u) __nanosleep(64);
        if (polls >= kBarrierPolls || ((polls & 1023u) == 0 && *(volatile int *)&bar->broken)) {
          *(volatile int *)&bar->broken = 1;
          atomicCAS(err, 0, GQM_ERR_TOPOLOGY);
          ok = 0;
          break;
        }
      }
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
    }
    return __syncthreads_and(threadIdx.x == 0 ? ok : 1) != 0;
#endif
  }
};

// shared-memory copies of the small steps' lists
constexpr int kSmallCap = 1024;
struct SmallLists {
  FlipCnt cnt;
  int4 rec[kSmallCap];
};

template <int PRED, int NT>
__global__ void __launch_bounds__(NT, 1)
    k_flip_loop(Mesh mesh, FlipLists lists, GridBar *bars, const int *team, int small_limit, int small_team,
                KTimer *ktm, KTimer *stm) {
  const int nb = min(*team, (int)gridDim.x);  // blocks this refinement uses; the rest leave at once
  if ((int)blockIdx.x >= nb) return;
  __shared__ SmallLists sh;
  __shared__ Mesh M;  // the phases are calls: they read the pointers from shared memory
  __shared__ FlipLists L;
  if (threadIdx.x == 0) {
    M = mesh;
    L = lists;
  }
  __syncthreads();
  FlipCtl *c = lists.c;
  FlipRegs R{c->gen, c->epoch, c->steps};
  const int entry = R.steps;
  const int st_blocks = min(small_team, nb);
  GridTeam G{bars, nb, bars[0].base, c->errp};
  GridTeam S{bars + 1, st_blocks, bars[1].base, c->errp};
  const int timed = ktm->on;
  const unsigned long long t0 = G.lead() ? global_ns() : 0;
  int status = FLIP_GO;
  // Every block takes the same way through the loop: what it decides on (list
  // lengths, the control block) was written before the last barrier of all
  // blocks and is not written again before the next.
  while (status == FLIP_GO) {
    const int n = vload(&c->cnt.qn[R.gen & 1]);
    if (n == 0) break;
    if (n > small_limit) {
      status = flip_step<PRED>(M, L, &c->cnt, R, entry, G, (R.gen & 1) ? L.q1 : L.q0, n, L.rec, timed ? ktm : nullptr,
                               nullptr);
      continue;
    }
    // small steps
    const int steps0 = R.steps;
    if ((int)blockIdx.x < st_blocks) {
      const unsigned long long s0 = timed && G.lead() ? global_ns() : 0;
      int items = 0, wins = 0, m = n;
      if (st_blocks == 1) {
        BlockTeam B;
        if (B.lead()) sh.cnt = c->cnt;
        B.sync();
        while (status == FLIP_GO && m > 0 && m <= small_limit) {
          items += m;
          status = flip_step<PRED>(M, L, &sh.cnt, R, entry, B, (R.gen & 1) ? L.q1 : L.q0, m,
                                   m <= kSmallCap ? sh.rec : L.rec, nullptr, timed ? &wins : nullptr);
          m = vload(&sh.cnt.qn[R.gen & 1]);
        }
        B.sync();
        if (B.lead()) c->cnt = sh.cnt;
      } else {
        while (status == FLIP_GO && m > 0 && m <= small_limit) {
          items += m;
          status = flip_step<PRED>(M, L, &c->cnt, R, entry, S, (R.gen & 1) ? L.q1 : L.q0, m, L.rec, nullptr,
                                   timed ? &wins : nullptr);
          m = vload(&c->cnt.qn[R.gen & 1]);
        }
      }
      if (G.lead()) {
        c->gen = R.gen;
        c->epoch = R.epoch;
        c->steps = R.steps;
        c->small_steps += R.steps - steps0;
        L.c->small_status = status;
        if (timed) ktimer_add(stm, s0, items, wins);
      }
    }
    if (!G.sync()) {
      status = FLIP_BROKEN;
      break;
    }
    R.gen = vload(&c->gen);
    R.epoch = (unsigned)vload((const int *)&c->epoch);
    R.steps = vload(&c->steps);
    status = vload(&c->small_status);
  }
  if (status != FLIP_BROKEN && !G.sync()) status = FLIP_BROKEN;  // nobody reads the control block any more
  if (G.lead()) {
    flip_close(c, R);
    c->ran++;
    c->loop_ns += global_ns() - t0;
    c->loops++;
    if (status != FLIP_BROKEN) {
      bars[0].base = G.target;
      bars[1].base = bars[1].arrived;
    }
  }
}

constexpr int kLoopThreads[2] = {256, 512};  // one block per SM at up to 255 / 128 registers
typedef void (*LoopFn)(Mesh, FlipLists, GridBar *, const int *, int, int, KTimer *, KTimer *);
static LoopFn loop_fn(int pred, int budget) {
  if (budget == 1) return pred ? k_flip_loop<1, 256> : k_flip_loop<0, 256>;
  return pred ? k_flip_loop<1, 512> : k_flip_loop<0, 512>;
}

}  // namespace gqm

// Bytes of the barrier words that gqm_flip_loop_launch needs (zeroed before
// every refinement).
size_t gqm_flip_bar_bytes() { return 2 * sizeof(gqm::GridBar); }

// Most blocks of a launch that can be resident together, one per SM.
int gqm_flip_max_blocks(int budget) {
#ifdef GQM_HOST_EMU
  (void)budget;
  return 1;
#else
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  for (int pred = 0; pred < 2; ++pred) {
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void *)gqm::loop_fn(pred, budget),
                                                      gqm::kLoopThreads[budget == 1 ? 0 : 1], 0) != cudaSuccess ||
        per < 1)
      return 0;
  }
  return sms;
#endif
}

// Launch of k_flip_loop on the single-domain engine's buffers (refine.cu).
// mesh and lists point at the caller's Mesh and FlipLists (the same layouts in
// every compilation); *team is the number of blocks the refinement uses.
int gqm_flip_loop_launch(const void *mesh, size_t mesh_bytes, const void *lists, size_t lists_bytes, void *bars,
                         const int *team, int pred, int blocks, int budget, int small_limit, int small_team,
                         void *ktimer, void *stimer, cudaStream_t st) {
  if (mesh_bytes != sizeof(gqm::Mesh) || lists_bytes != sizeof(gqm::FlipLists)) return GQM_ERR_ARGUMENT;
  gqm::Mesh M;
  gqm::FlipLists L;
  memcpy(&M, mesh, sizeof(M));
  memcpy(&L, lists, sizeof(L));
  gqm::GridBar *b = static_cast<gqm::GridBar *>(bars);
  gqm::KTimer *kt = static_cast<gqm::KTimer *>(ktimer), *stm = static_cast<gqm::KTimer *>(stimer);
#ifdef GQM_HOST_EMU
  (void)blocks;
  (void)st;
  gqm::loop_fn(pred, budget)(M, L, b, team, small_limit, small_team, kt, stm);
  return GQM_OK;
#else
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)gqm::kLoopThreads[budget == 1 ? 0 : 1]);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, gqm::loop_fn(pred, budget), M, L, b, team, small_limit, small_team, kt, stm) ==
                 cudaSuccess
             ? GQM_OK
             : GQM_ERR_CUDA;
#endif
}

// The incircle expansion-fallback counter of this translation unit's kernels
// (a device variable exists once per translation unit): added to *sum, then
// zeroed when `reset` is set.  Called by the single-domain driver, which
// reports the counters of all its kernels together.
int gqm_fallbacks_cluster(unsigned long long *sum, int reset, cudaStream_t st) {
  unsigned long long v = 0;
#ifdef GQM_HOST_EMU
  (void)st;
  v = gqm::g_incircle_fallbacks;
  if (reset) gqm::g_incircle_fallbacks = 0;
#else
  if (sum && (cudaMemcpyFromSymbolAsync(&v, gqm::g_incircle_fallbacks, sizeof(v), 0, cudaMemcpyDeviceToHost, st) !=
                  cudaSuccess ||
              cudaStreamSynchronize(st) != cudaSuccess))
    return GQM_ERR_CUDA;
  if (reset) {
    const unsigned long long zero = 0;
    if (cudaMemcpyToSymbolAsync(gqm::g_incircle_fallbacks, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, st) !=
        cudaSuccess)
      return GQM_ERR_CUDA;
  }
#endif
  if (sum) *sum += v;
  return GQM_OK;
}
