// launches.h -- the kernels that are compiled in files of their own, as the
// addresses cudaLaunchKernel and cudaFuncSetAttribute take.
#pragma once

#include <cuda_runtime.h>

// Mixed precision: FP32 basis values, orbital rows and contraction; the
// inverse and its Sherman-Morrison update in MIXED_TI.
#ifndef MIXED_TI
#define MIXED_TI double
#endif

namespace qmcb {

struct GroupMember;

// k_move<metropolis, float or double, ..., extras, ginv> (move.cu)
const void *move_fn(bool metropolis, bool mixed, bool extras, bool ginv);
const void *move_dense_fn(bool metropolis);  // FP64, extras, small spins: four blocks per SM
// k_full<float or double, ..., extras, rest> (full.cu)
const void *full_fn(bool mixed, bool extras, bool rest);
const void *rest_dense_fn(bool mixed);  // extras, rest: four blocks per SM
// k_full_md, k_move_md<metropolis> (md.cu)
const void *full_md_fn();
const void *move_md_fn(bool metropolis);
// k_move_group<extras, ginv, table in constant memory, several determinants> (group.cu)
const void *group_move_fn(bool extras, bool ginv, bool cst, bool md);
// Members [first, first + n) of the constant-memory table.
cudaError_t group_upload_const(const GroupMember *members, int n, int first, cudaStream_t st);
// The branching, copy and trial-energy launches of step t for members gm[0..nm).
void group_branch(const GroupMember *gm, int nm, int t, cudaStream_t st);

// Launch of a kernel by its address; the arguments must have the parameters' types.
template <typename... A>
inline cudaError_t launch_kernel(const void *fn, dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A &...args)
{
  void *p[] = {(void *)&args...};
  return cudaLaunchKernel(fn, grid, block, p, smem, st);
}

}  // namespace qmcb
