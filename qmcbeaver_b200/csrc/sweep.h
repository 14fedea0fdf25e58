// sweep.h -- launch of the small-spin sweep kernel (sweep.cu).
#pragma once

#include "rows64.h"

namespace qmcb {

constexpr int kSweepMax = 16;  // largest spin of the kernel: one lane per electron of a spin

struct SweepArgs {
  int step0, nsteps;       // Metropolis: steps step0 .. step0 + nsteps - 1 (electron = step % N)
  int reweight_start;      // steps below keep dW = 1
  int e;                   // evaluate: the moved electron
  double *dump;            // configuration records of every step (dump_configs), or null
  int rin_moved;           // evaluate: R_in holds only the moved electron's position
};

// Shared memory of one CTA (nmax = the larger spin), and the kernels' limit.
int sweep_smem_bytes(int nmax, const Layout &L, const Rows64 &T);
cudaError_t sweep_limits(int max_bytes);

// Metropolis / DMC steps of list entries [0, num) (d_num: device count, grid
// sized for `cap`) with no branching or refresh between them, or one
// evaluate call with the caller's positions.
cudaError_t sweep_launch(bool metropolis, const DevSys &S, const Layout &L, const RunCfg &cfg, const Rows64 &T,
                         double *state, int cap, cudaStream_t st, const int *slots, int num, const int *d_num,
                         const double *R_in, const SweepArgs &a, const EnergyCtl *ectl, double *stats,
                         const EvalOut &out);

}  // namespace qmcb
