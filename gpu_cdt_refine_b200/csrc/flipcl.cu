// The flip-flop loop of the single-domain engine in one launch.
//
// flipFlop (GPU_Refine/refine.cu:2328-2490) runs a step after another until no
// triangle is flagged.  Here the whole loop is one cooperative launch whose
// blocks separate the phases of a step (flip_step in kernels.cuh) with a
// barrier in global memory, and no launch, condition node or host read stands
// between two phases or two steps.
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

template <int PRED, int NT>
__global__ void __launch_bounds__(NT, 1)
    k_flip_loop(Mesh mesh, FlipLists lists, GridBar *bars, const int *team, int small_limit, int small_team,
                KTimer *ktm, KTimer *stm) {
  const int nb = min(*team, (int)gridDim.x);  // blocks this refinement uses; the rest leave at once
  // a barrier broke in an earlier loop of the run: its counts order nothing any more
  if ((int)blockIdx.x >= nb || bars[0].broken || bars[1].broken) return;
  __shared__ SmallLists sh;
  __shared__ Mesh M;  // the phases are calls: they read the pointers from shared memory
  __shared__ FlipLists L;
  if (threadIdx.x == 0) {
    M = mesh;
    L = lists;
  }
  __syncthreads();
  int *err = lists.c->errp;
  GridTeam G{bars, nb, (int)blockIdx.x, bars[0].base, err};
  GridTeam S{bars + 1, min(small_team, nb), (int)blockIdx.x, bars[1].base, err};
  if (!flip_loop<PRED>(M, L, sh, G, small_limit, small_team > 1 ? &S : nullptr, ktm, stm)) return;
  if (G.lead()) {  // behind the loop's last barrier: every block has read the bases and made its arrivals
    bars[0].base = G.target;
    bars[1].base = bars[1].arrived;
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
  return GQM_EMU_BLOCKS;
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
  GQM_EMU_GRID(blocks, gqm::loop_fn(pred, budget)(M, L, b, team, small_limit, small_team, kt, stm));
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
