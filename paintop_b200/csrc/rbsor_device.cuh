// rbsor_device.cuh -- device helpers shared by the red-black SOR kernels
// (rbsor_kernels.cu, rbsor_cluster.cu): plane indexing, fixed-order block sums
// and the per-system state machine.
#pragma once

#include <cmath>

#include "rbsor.cuh"

namespace ptk {

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// The call's clock: its start, and whether its wall budget is spent. (Another
// multiprocessor's clock may lag behind the one that stored the start.)
__device__ __forceinline__ unsigned long long *call_start(const KParams &P) {
  return reinterpret_cast<unsigned long long *>(P.bar + kBarStart);
}
__device__ __forceinline__ bool over_budget(const KParams &P, unsigned long long t_start) {
  const unsigned long long now = gtimer();
  return now > t_start && now - t_start > P.budget_ns;
}

__device__ __forceinline__ int ld_vol(const int *p) { return *reinterpret_cast<const volatile int *>(p); }

// Deterministic block sum: fixed xor-butterfly inside each warp, then warps in
// index order. The total is valid in thread 0. Uses sred[0 .. blockDim.x/32).
__device__ __forceinline__ double block_sum(double v, double *sred) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sred[warp] = v;
  __syncthreads();
  double tot = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += sred[w];
  __syncthreads();
  return tot;
}

__device__ __forceinline__ long long plane_index(const SysDesc &d, int c, int y, int i) {
  return d.off + (long long)c * d.plane + (long long)y * d.pw + i;
}

__device__ __forceinline__ void apply_stall(SysState &s, double rel, int &done) {
  // poisson.rs:219-228 (window 16 for a given omega; see k_init for automatic omega)
  if (rel < s.best * (1.0 - kStallImprovement)) {
    s.best = rel;
    s.since = 0;
  } else {
    s.since += 1;
    if (s.since >= s.stall_window) done = 1;
  }
}

__device__ inline SysState load_sys_state(const SysState *p) {
  SysState s;
  const int *pi = reinterpret_cast<const int *>(p);
  int *si = reinterpret_cast<int *>(&s);
  for (int k = 0; k < (int)(sizeof(SysState) / sizeof(int)); ++k) si[k] = __ldcg(pi + k);
  return s;
}

// One step of a system's state machine, by one thread, after a step in `mode`.
// nrms[j] = the residual norm after sweep j of the step (M_SWEEP), or of the
// iterate (M_RESID), rels[j] = its ratio to r0 (poisson.rs:206). `hist` receives the history entries (null: they
// are another thread's to write). cap: sweeps per step. True when the system
// is done.
__device__ inline bool step_state(const SysDesc &d, SysState &s, int mode, const double *nrms, const double *rels,
                                  double *hist, int cap) {
  bool done = false;
  switch (mode) {
    case M_SWEEP: {
      int kind = P_NONE, stop_j = -1;
      bool refine = false;
      for (int j = 0; j < s.s; ++j) {
        const double nrm = nrms[j], rel = rels[j];
        s.iterations += 1;
        if (hist) hist[s.iterations - 1] = rel;
        s.last = rel;
        if (rel <= d.tol) { kind = P_CONV; stop_j = j; break; }  // poisson.rs:210-214
        int stalled = 0;
        apply_stall(s, rel, stalled);
        if (stalled) { kind = P_STALL; stop_j = j; break; }
        if (s.iterations >= d.max_it) { kind = P_MAX; stop_j = j; break; }
        // residual-correction trigger (does not change the iterate, only when
        // the FP64 fold happens, so it waits for the end of the block)
        if (nrm <= kRefineFactor * s.ibase) refine = true;
        if (nrm < s.ibest * kInnerGain) { s.ibest = nrm; s.isince = 0; }
        else if (++s.isince >= kInnerWindow) refine = true;
      }
      if (kind == P_NONE) {
        s.cur ^= 1;
        if (refine) { s.pending = P_REFINE; s.mode = M_FOLD; }
        else { s.mode = M_SWEEP; s.s = min(cap, d.max_it - s.iterations); }
      } else if (stop_j == s.s - 1) {
        s.cur ^= 1; s.pending = kind; s.mode = M_FOLD;
      } else {
        // stop inside the block: re-run the block from the same start with
        // exactly stop_j+1 sweeps (identical arithmetic), so the iterate kept is
        // the one after the reported sweep.
        s.pending = kind; s.mode = M_REDO; s.s = stop_j + 1;
      }
    } break;
    case M_REDO:
      s.cur ^= 1;
      s.mode = M_FOLD;
      break;
    case M_FOLD:
      s.mode = M_RESID;
      break;
    case M_RESID: {
      const double nrm = nrms[0], rel = rels[0];
      s.outer = nrm;
      s.ibase = nrm;
      s.ibest = INFINITY;
      s.isince = 0;
      s.refinements += 1;
      if (s.iterations > 0) {
        if (hist) hist[s.iterations - 1] = rel;
        s.last = rel;
      }
      int stop = -1;
      if (rel <= d.tol) stop = STOP_CONVERGED;
      else if (s.pending == P_STALL) stop = STOP_STALLED;
      else if (s.pending == P_MAX || s.iterations >= d.max_it) stop = STOP_MAX;
      else if (s.pending == P_CONV) {
        // the per-sweep estimate met the tolerance but the FP64 residual does
        // not: apply the stall rule the estimate skipped, then keep sweeping
        int stalled = 0;
        apply_stall(s, rel, stalled);
        if (stalled) stop = STOP_STALLED;
      }
      s.pending = P_NONE;
      if (stop >= 0) {
        s.mode = M_DONE;
        s.status = stop;
        done = true;
      } else {
        s.mode = M_SWEEP;
        s.s = min(cap, d.max_it - s.iterations);
      }
    } break;
    default:
      break;
  }
  s.steps += 1;
  return done;
}

}  // namespace ptk
