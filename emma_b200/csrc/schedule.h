// schedule.h -- device state of the level schedule (see schedule.cu).
#pragma once
#include "plan_types.h"

namespace emma {

struct SchedState {
  double tsim, dt_param, time_max, cfl;
  double adt[kMaxLevels];               // the reference's adt array, index level-1
  double dx[kMaxLevels];                // cell size per level
  unsigned long long smax[kMaxLevels];  // max signal speed per level from the CFL reduction kernel
                                        // (bits of a non-negative double)
  unsigned long long smax_next[kMaxLevels];  // the same, accumulated by the level kernel over the
                                             // state it writes
  int fresh[kMaxLevels];                // smax_next holds the max of the level's current state
  int stale[kMaxLevels];                // !fresh: the state was set from the host (smax is then
                                        // zeroed with it, for the reduction kernel)
  int cfl_gate[kMaxLevels];             // subcycled iteration: active and stale
  int azall[kMaxLevels];                // the level was updated since its state was set: every
                                        // split cell holds the averaged state (sound speed 0)
  double dtacc[kMaxLevels];             // dt accumulated by the current Advance_level(L) call
  double tloc[kMaxLevels];              // its local time
  int is[kMaxLevels];                   // its iteration count
  int active[kMaxLevels];               // gate of the current iteration of level L
  long long updates;                    // cell-updates performed (leaf cells x substeps)
  int lcoarse, lmax, nsub;
  int gate_all;
  unsigned ticket[2];                   // work queue of the level kernel: next item, CTAs done
                                        // (the last CTA of a launch puts both back to 0)
};

// Control block of the fused coarse step (step_kernel.cuh), zeroed before each
// launch: the grid-wide job barrier, the job in progress and the schedule's
// position in Advance_level's recursion.
struct StepCtl {
  unsigned epoch;    // jobs published so far
  unsigned arrived;  // CTAs done with the current job
  unsigned ticket;   // next work item of the current job
  int kind, L, n, shape;  // the current job: kind, level, work items, brick shape
  int pc, pcL;       // schedule position (pc 0: start of the coarse step) and its level
  int pad[7];
};
enum : int { kJobNone = 0, kJobLevel = 1, kJobCfl = 2, kJobDone = 3 };

// Arguments of a fused coarse step.
struct StepArgs {
  LevelArgs *lv;
  SchedState *S;
  StepCtl *ctl;
  unsigned *done;       // scratch for the tiles' completion counts
  unsigned *status;
  long long wait_limit;  // bounded spin of a CTA waiting for the next job
  int lfine;             // finest level with octs
  unsigned shapes;       // brick shapes of the tree's levels (bit i: kShapes[i])
  struct StepJobRecord *jobt;  // optional: kStepJobLog records of the jobs' releases
};
// One released job of a fused coarse step: the device times (ns, %globaltimer) at
// which every CTA had reached the barrier before it and at its release (the
// schedule ran in between), its kind and level.
struct StepJobRecord {
  unsigned long long t_all, t;
  int kind, L;
};
constexpr unsigned kStepJobLog = 256;

// The CFL reduction of a level (src/advanceamr.c:122-128) by a grid of 256-thread blocks:
// this block's share of the cells, the maximum added to *out (bits of a non-negative
// double, which order like the numbers).  For units built with -fmad=false.
static __device__ __forceinline__ void cfl_block(const double *__restrict__ W, long long n8, unsigned long long *out) {
  double m = 0.;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    const double d = W[i], u = W[n8 + i], v = W[2 * n8 + i], w = W[3 * n8 + i], p = W[4 * n8 + i];
    const double va = sqrt(u * u + v * v + w * w);
    const double aa = sqrt((5. / 3.) * p / d);
    const double s = va + aa;
    m = fmax(m, s);  // fmax drops NaN like the reference's FMAX
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ double sm[32];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = (threadIdx.x < (blockDim.x >> 5)) ? sm[threadIdx.x] : 0.;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
  }
}

// The end of a step that advanced every level once: buffers swapped, counters, time.
static __device__ __forceinline__ void batch_end(SchedState *S, LevelArgs *lv) {
  const int lc = S->lcoarse, lm = S->lmax;
  for (int L = lc; L <= lm; L++) {
    if (lv[L].noct == 0) break;
    double *t = lv[L].W;
    lv[L].W = lv[L].Wn;
    lv[L].Wn = t;
    lv[L].wait_slot = -1;
    S->updates += lv[L].leaf;
    S->fresh[L] = 1;
    S->stale[L] = 0;
    S->azall[L] = 1;
  }
  S->tsim += S->adt[lc - 1];
}

// ... run by the last block of a launch to finish (one thread of each block calls this,
// after the block's last access to the level slots); S->ticket[1] counts the blocks.
static __device__ __forceinline__ void batch_end_by_last(SchedState *S, LevelArgs *lv) {
  __threadfence();
  if (atomicAdd(&S->ticket[1], 1u) == gridDim.x - 1) {
    S->ticket[1] = 0u;
    batch_end(S, lv);
  }
}

__global__ void k_set_args(LevelArgs *lv, int slot, LevelArgs a);
__global__ void k_bind_level(LevelArgs *lv, int L, int lcoarse, int lmax, double dt);
__global__ void k_swap_level(LevelArgs *lv, int L, const int *gate);
__global__ void k_clear(double *p, long long n, const int *gate);
__global__ void k_batch_begin(SchedState *S, LevelArgs *lv, unsigned *done);
__global__ void k_cfl_begin(SchedState *S, LevelArgs *lv, unsigned *done, int L);
__global__ void k_batch_end(SchedState *S, LevelArgs *lv);
__global__ void k_sub_begin(SchedState *S, int L, int it);
__global__ void k_sub_dt(SchedState *S, int L);
__global__ void k_sub_prelaunch(SchedState *S, LevelArgs *lv, int L, int has_fine);
__global__ void k_sub_end(SchedState *S, LevelArgs *lv, int L);
__global__ void k_sub_final(SchedState *S);

}  // namespace emma
