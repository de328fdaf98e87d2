// Teams of thread blocks that run an algorithm's phases together, separated by
// barriers instead of launches.  Every wait is bounded.
#pragma once
#include <cuda_runtime.h>

#include "../../include/gqm_refine.h"

// A host build of the kernels runs one block of one thread, unless it defines
// these: the blocks of a launch, the launch of so many, and a block's wait for
// a word to reach a value (false: it never will).
#if defined(GQM_HOST_EMU) && !defined(GQM_EMU_BLOCKS)
#define GQM_EMU_BLOCKS 1
#define GQM_EMU_GRID(blocks, call) call
#define GQM_EMU_WAIT(word, target) true
#endif

namespace gqm {

__device__ __forceinline__ int vload(const int *p) { return *(const volatile int *)p; }

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

// `nb` blocks, all of them resident (a cooperative launch).  A barrier adds one
// arrival per block to a word that only grows; a block waits until all arrivals
// of its own barrier have been counted.  The arrival is a reduction with no
// answer to wait for, and the wait polls one word.
struct GridBar {
  unsigned long long arrived;  // arrivals of all barriers
  unsigned long long base;     // arrivals when the current launch began
  int broken;
};
constexpr unsigned kBarrierPolls = 1u << 25;  // tens of seconds
struct GridTeam {
  GridBar *bar;
  int nb, rank;  // blocks of the team, this block's place among them
  unsigned long long target;
  int *err;
  int code = GQM_ERR_TOPOLOGY;  // recorded in *err when a wait runs out
  __device__ __forceinline__ int tid() const { return rank * (int)blockDim.x + (int)threadIdx.x; }
  __device__ __forceinline__ int size() const { return nb * (int)blockDim.x; }
  __device__ __forceinline__ bool lead() const { return rank == 0 && threadIdx.x == 0; }
  __device__ __forceinline__ bool sync() {
#ifdef GQM_HOST_EMU
    if (nb == 1) return true;
    target += (unsigned long long)nb;
    ++bar->arrived;
    if (GQM_EMU_WAIT(&bar->arrived, target)) return true;
    bar->broken = 1;
    if (*err == 0) *err = code;
    return false;
#else
    if (nb == 1) {
      __syncthreads();
      return true;
    }
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
          atomicCAS(err, 0, code);
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

}  // namespace gqm
