// apt_batch.cuh — one launch advances every active simulation of a server by
// one step (continuous batching).
//
// Each simulation keeps its own pair buffers, tensor maps, parameters, step
// counter and ping-pong index in device memory (BatchSim), so a captured CUDA
// graph of K (step, finish) launch pairs can be replayed without host updates.
// The step kernel is persistent: CTAs pull (simulation, column tile, z chunk)
// work items from an atomic counter until the list is exhausted, and run the
// same per-item code as the single-simulation kernel (step_item), so a
// simulation's arithmetic and results do not depend on what else is batched
// with it.
#pragma once

#include "apt_step.cuh"

namespace cupf {

struct BatchSim {
  StepArgs a;          // in / out / t are filled per step from the fields below
  void* buf[2];
  uint8_t* quiet[2];   // quiet-item flags of each buffer (StepArgs::quiet_in/out)
  uint8_t* redo[2];    // change marks of each buffer (StepArgs::redo_in/out)
  long long steps;     // explicit steps done
  long long target;    // steps requested
  int cur;             // buffer holding the current state
  int active;          // 1 while steps < target
  int use_iuc;
  int pad;
};

// The batched kernel's shared memory: a step's, then the current item's StepArgs
// (read from there: a copy per thread spills at these kernels' register budget).
template <int NP, class S, int TY>
constexpr int batch_args_off() {
  return (StepSmem<NP, S, TY>::kBytes + 15) & ~15;
}
template <int NP, class S, int TY>
constexpr int batch_smem_bytes() {
  return batch_args_off<NP, S, TY>() + (int)sizeof(StepArgs);
}

// TY: the column-tile height of every simulation in the launch (the server
// launches one kernel per tile height present in a round).
template <int NP, class S, int TY>
__global__ void __launch_bounds__(tile_threads<TY>(), step_min_blocks<NP, S, TY>())
    apt_batch_step_kernel(BatchSim* sims, const CUtensorMap* tmaps, const int4* items, int nitems,
                          int* work, const int* err) {
  extern __shared__ __align__(128) unsigned char smem[];
  CtaSmem<NP, S, TY> sm(smem);
  sm.init();
  StepArgs& a = *reinterpret_cast<StepArgs*>(smem + batch_args_off<NP, S, TY>());
  int qbase = 0, held = -1;  // simulation whose arguments are in a
  WorkItems todo(work, nitems, sm.s_item, err);
  for (;;) {
    const int it = todo.next();
    if (it < 0) break;
    const int4 w = items[it];  // simulation, txi, tyi, zci
    const BatchSim* sd = sims + w.x;
    if (!sd->active) continue;
    const int cur = sd->cur;
    if (sd->quiet[0] && item_quiet<TY>(sd->a, sd->quiet[cur], sd->quiet[cur ^ 1], w.y, w.z, w.w))
      continue;
    // the simulation's arguments in shared memory, its per-step fields filled in, when
    // the CTA comes to another simulation (every thread has left the previous item at
    // the barriers of todo.next())
    if (w.x != held) {
      held = w.x;
      static_assert(sizeof(StepArgs) % 4 == 0, "copied by words");
      for (int e = threadIdx.x; e < (int)(sizeof(StepArgs) / 4); e += tile_threads<TY>())
        reinterpret_cast<uint32_t*>(&a)[e] = reinterpret_cast<const uint32_t*>(&sd->a)[e];
      __syncthreads();
      if (threadIdx.x == 0) {
        a.in = sd->buf[cur];
        a.out = sd->buf[cur ^ 1];
        a.quiet_in = sd->quiet[cur];
        a.quiet_out = sd->quiet[cur ^ 1];
        a.redo_in = sd->redo[cur];
        a.redo_out = sd->redo[cur ^ 1];
        a.use_iuc = sd->use_iuc;
        // t of step n (1-based) = (float)n * dt * tau0, as the single-simulation path
        a.t = __fmul_rn(__fmul_rn((float)(sd->steps + 1), a.dt), a.tau0);
        a.t64 = __dmul_rn(__dmul_rn((double)(sd->steps + 1), (double)a.dt), (double)a.tau0);
        a.sr_key = (uint32_t)(sd->steps + 1);
      }
      __syncthreads();
    }
    step_item<NP, S, TY>(tmaps + 2 * w.x + cur, a, w.y, w.z, w.w, sm, qbase);
  }
  sm.drain();
}

// After every simulation's step: flip its buffers, count the step and retire
// it at its target.
static __global__ void batch_finish_kernel(BatchSim* sims, int nsims) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nsims && sims[i].active) {
    sims[i].cur ^= 1;
    sims[i].steps += 1;
    if (sims[i].steps >= sims[i].target) sims[i].active = 0;
  }
}

}  // namespace cupf
