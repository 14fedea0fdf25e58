// invert.h -- launch of the Slater-matrix inversion (invert.cu).
#pragma once

#include "kernels.cuh"

namespace qmcb {

constexpr int kInvertMax = 128;  // largest spin of the kernel

// The inverses, ln|det| and signs of both spins of list entries [0, num)
// (d_num: device count, grid sized for `cap`) from their stored Slater values
// (mixed: FP32 values); the first copy of an inverse kept in HBM becomes the
// current one.  Singular: sign 0, ln|det| -inf.
cudaError_t invert_launch(bool mixed, const DevSys &S, const Layout &L, double *state, int cap, cudaStream_t st,
                          const int *slots, int num, const int *d_num);

}  // namespace qmcb
