// group.h -- member tables of the group kernels (group.cu).
#pragma once

#include "kernels.cuh"

namespace qmcb {

constexpr int kGroupMax = 512;  // members of one group

struct GroupMember {
  DevSys S;
  Layout L;
  RunCfg cfg;
  double *state;
  int *live, *live_tmp, *free_stack, *ctl;
  int2 *copies;
  EnergyCtl *ectl;
  double *stats;
  int step0;           // the member's step number at step offset 0
  int reweight_start;  // reweight_start_step
  int dmc;
  int limit_branching;
  double thr_split, thr_fuse;
  const double *rows;  // tensor-core rows modes: the step's orbital rows (null: FP64 basis and contraction)
};

// Members the constant-memory table holds.
constexpr int kConstMembers = 84;

}  // namespace qmcb
