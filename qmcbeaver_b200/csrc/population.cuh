// population.cuh -- the population kernels of one system and the walkers'
// read back; included by qmcb200.cu only.
#pragma once

#include "kernels_population.cuh"

namespace qmcb {

__global__ void __launch_bounds__(1024) k_branch(double *state, Layout L, int *live, int *live_tmp, int *free_stack,
                                                 int *ctl, int2 *copies, double thr_split, double thr_fuse,
                                                 uint64_t seed, int step, double *stats, double e_orig,
                                                 int limit_branching)
{
  branch_block(state, L, live, live_tmp, free_stack, ctl, copies, thr_split, thr_fuse, seed, step, stats, e_orig,
               limit_branching);
}

__global__ void k_copy(double *state, Layout L, const int2 *copies, const int *ctl)
{
  copy_blocks(state, L, copies, ctl, blockIdx.x, gridDim.x);
}

__global__ void k_energy(EnergyCtl *ectl, const double *stats, int min_samples_ok, int dyn_dt, double dt)
{
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  update_energy(ectl, stats, min_samples_ok, dyn_dt, dt);
}

// R [n][3N], then weight, E_L, log|psi|, sign [n] each of the first n live
// walkers into out.
__global__ void k_gather(const double *state, Layout L, int N, const int *live, int n, double *out)
{
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = lane_id();
  if (w >= n) return;
  const double *blk = state + (size_t)live[w] * L.stride;
  double *o = out + (size_t)w * 3 * N, *s = out + (size_t)n * 3 * N + w;
  for (int t = lane; t < 3 * N; t += 32) o[t] = blk[L.R + t];
  if (lane == 0) {
    const double *sc = blk + L.sc;
    s[0] = sc[SC_WEIGHT];
    s[(size_t)n] = sc[SC_EL];
    s[2 * (size_t)n] = sc[SC_LOGDET_A] + sc[SC_LOGDET_B] + sc[SC_U];
    s[3 * (size_t)n] = sc[SC_SIGN_A] * sc[SC_SIGN_B];
  }
}

// Sets the weights of the first n live walkers.
__global__ void k_set_weights(double *state, Layout L, const int *live, int n, const double *w)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    state[(size_t)live[i] * L.stride + L.sc + SC_WEIGHT] = w[i];
}

// Per-walker evaluate outputs moved from the device buffer into mapped
// page-locked host arrays with consecutive threads on consecutive elements,
// so the stores cross the bus as full packets (the evaluate kernels store a
// walker's scalars from one lane, one 8-byte packet each).  Segment
// blockIdx.y: bytes[y] bytes from src[y] to dst[y]; whole 8-byte words when
// both ends and the length allow it, bytes otherwise.
struct PutList {
  const void *src[8];
  void *dst[8];
  size_t bytes[8];
};

__global__ void k_put_outputs(PutList P)
{
  const int y = blockIdx.y;
  const size_t n = P.bytes[y];
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x, di = (size_t)gridDim.x * blockDim.x;
  if (((uintptr_t)P.src[y] | (uintptr_t)P.dst[y] | n) % 8 == 0) {
    const unsigned long long *s = (const unsigned long long *)P.src[y];
    unsigned long long *d = (unsigned long long *)P.dst[y];
    for (size_t i = i0; i < n / 8; i += di) d[i] = s[i];
  } else {
    const unsigned char *s = (const unsigned char *)P.src[y];
    unsigned char *d = (unsigned char *)P.dst[y];
    for (size_t i = i0; i < n; i += di) d[i] = s[i];
  }
}

}  // namespace qmcb
