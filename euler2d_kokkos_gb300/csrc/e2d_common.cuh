// e2d_common.cuh -- device helpers shared by the FP64 and FP32 kernels.
#pragma once

#include "e2d_internal.h"

namespace e2d {

// Source cell of a ghost along one axis: the composition of the X-face pass
// (all rows) and the Y-face pass (all columns) of MakeBoundariesFunctor
// (src/HydroRunFunctors.h:1855-2024).  Reflect mirrors (2g-1-i) and flips
// the normal momentum, absorb copies the first interior cell, periodic
// wraps.  With n >= 2 the result is always an interior cell, so a ghost never
// reads another ghost and corners follow the X-then-Y fill order.
__device__ __forceinline__ int ghost_source(int i, int n, int bc_lo, int bc_hi, bool &flip) {
  flip = false;
  if (i < 2) {
    if (bc_lo == E2D_BC_REFLECT) {
      flip = true;
      return 3 - i;
    }
    if (bc_lo == E2D_BC_ABSORB) return 2;
    return n + i;
  }
  if (i >= n + 2) {
    if (bc_hi == E2D_BC_REFLECT) {
      flip = true;
      return 2 * n + 3 - i;
    }
    if (bc_hi == E2D_BC_ABSORB) return n + 1;
    return i - n;
  }
  return i;
}

__device__ __forceinline__ bool nonfinite64(double x) {
  return ((__double_as_longlong(x) >> 52) & 0x7ff) == 0x7ff;
}

__device__ __forceinline__ unsigned long long timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Barrier over the blocks of a cooperative launch: `arrived` counts blocks
// over all barriers so far, `target` is what it reaches at this one.  Every
// thread calls it; what any block wrote before is visible to every thread
// after (ordinary and L2 loads, not ld.global.nc).  The wait gives up after a
// second and returns false for the whole block.
__device__ __forceinline__ bool grid_barrier(unsigned int *arrived, const unsigned int target) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
    unsigned int n;
    bool ok = true;
    unsigned long long t0 = 0ull;
    for (int k = 0;; ++k) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(arrived) : "memory");
      if ((int)(n - target) >= 0) break;
      if ((k & 255) == 255) {
        const unsigned long long t = timer_ns();
        if (t0 == 0ull) t0 = t;
        if (t - t0 > 1000000000ull) {
          ok = false;
          break;
        }
      }
    }
    s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  return s_ok != 0;
}

// The state of a multi-step launch as each block follows it: every block
// forms the same t, nstep and dt.
struct LoopClock {
  double t, t_end;
  int ns;
};
__device__ __forceinline__ LoopClock loop_begin(const DevClock *clk) {
  LoopClock c;
  c.t = __ldcg(&clk->t);
  c.t_end = __ldcg(&clk->t_end);
  c.ns = __ldcg(&clk->nstep);
  return c;
}
// The CFL maximum step s of the launch reads.
__device__ __forceinline__ unsigned long long loop_cfl(const DevClock *clk, const LoopClock &c, int s) {
  return s == 0 ? __ldcg(&clk->acc[c.ns & 1]) : __ldcg(&clk->acc3[s % 3]);
}
// Step s took dt: one thread of block 0 records it and clears the maximum
// that step s + 2 will read (no block has read or folded into it since the
// barrier before last).
__device__ __forceinline__ void loop_record(DevClock *clk, const LoopClock &c, int s, double dt, double *trace) {
  clk->acc3[(s + 2) % 3] = 0ull;
  const int slot = c.ns - clk->trace_base;
  if (trace && slot >= 0 && slot < clk->trace_cap) trace[slot] = dt;
  clk->dt = dt;
  if (!(dt > 0.0) || nonfinite64(dt)) atomicOr(&clk->status, (unsigned)E2D_FLAG_BAD_DT);
}
// After the last barrier, one thread of block 0: what a launch per step
// leaves behind (src/main.cpp:139-143).
__device__ __forceinline__ void loop_end(DevClock *clk, const LoopClock &c, int s) {
  clk->t = c.t;
  clk->nstep = c.ns;
  if (s > 0) clk->acc[c.ns & 1] = __ldcg(&clk->acc3[s % 3]);
}

}  // namespace e2d
