// kernels_population.cuh -- kernels over the walker population.
//
//   k_branch       nonunit-weight branching of the live list (single CTA)
//   k_copy         state copies for split walkers
//   k_energy       E_est / E_T update after a branching step
//   k_gather       walkers packed for a read back
//   k_set_weights  the caller's weights
//   k_put_outputs  evaluate outputs into mapped host memory
#pragma once

#include "kernels.cuh"

namespace qmcb {

// ------------------------------------------------------------------------
// Nonunit-weight branching (QMCRun::nonunitWeightBranching,
// QMcBeaver/src/QMCRun.cpp:740-814) on the live slot list, one CTA of
// 1024 threads.  Walkers above the branching threshold split in two with
// half the weight each (the copy is appended to the list), walkers below
// 0.01 die, walkers below the fusion threshold are paired in list order and
// one of each pair survives with the sum of the weights (probability
// w1 / (w1 + w2) for the first; the uniform draw of a pair is keyed by
// (seed, position of its first member in the live list, step)).  The split
// test uses the weight before fusion, so a fused survivor does not split in
// the same pass.  Dead slots go on the free stack; copies
// take slots from it and are written to the copy list for k_copy.
// ctl: [0] n_live, [1] n_free, [2] n_copies.
// QMCWalker::branchRecommended (limit_branching): no split for a walker that
// has not moved for more than 4 steps, whose weight grows too fast
// (dW^(age+1) > 5), that is heavy (> 100) and still growing (> 1.5), or whose
// local energy is more than 100x off the input energy.
__device__ __forceinline__ bool branch_recommended(const double *sc, double e_orig, int limit)
{
  if (!limit) return true;
  const double age = sc[SC_AGE], W = sc[SC_WEIGHT], dW = sc[SC_DW];
  const double growth = pow(dW, age + 1.0);
  bool ok = true;
  if (age > 4.0) ok = false;
  if (growth > 5.0)
    ok = false;
  else if (W > 100.0 && growth > 1.5)
    ok = false;
  if (fabs((sc[SC_EL] - e_orig) / e_orig) > 100.0) ok = false;
  return ok;
}

__device__ __forceinline__ void branch_block(double *state, const Layout &L, int *live, int *live_tmp,
                                             int *free_stack, int *ctl, int2 *copies, double thr_split,
                                             double thr_fuse, uint64_t seed, int step, double *stats, double e_orig,
                                             int limit_branching)
{
  __shared__ int s_warp[32];
  __shared__ int s_base[4];
  __shared__ double s_wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n = ctl[0];
  int nfree = ctl[1];
  // pass 1: pair fusion candidates in list order and decide
  int cand_base = 0;
  for (int c0 = 0; c0 < n; c0 += 1024) {
    int i = c0 + tid;
    int slot = i < n ? live[i] : -1;
    double w = slot >= 0 ? state[(size_t)slot * L.stride + L.sc + SC_WEIGHT] : 0.0;
    int is_c = (slot >= 0 && w <= thr_split && w >= 0.01 && w < thr_fuse) ? 1 : 0;
    // block exclusive scan of is_c
    unsigned b = __ballot_sync(QMCB_FULL_MASK, is_c);
    int wpre = __popc(b & ((1u << lane) - 1));
    if (lane == 31) s_warp[wid] = wpre + is_c;
    __syncthreads();
    if (wid == 0) {
      int v = s_warp[lane], x = v;
      for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(QMCB_FULL_MASK, x, o);
        if (lane >= o) x += y;
      }
      s_warp[lane] = x - v;
      if (lane == 31) s_base[0] = x;
    }
    __syncthreads();
    int rank = cand_base + s_warp[wid] + wpre;  // global candidate rank
    int total = s_base[0];
    // candidate ranks are global over the whole list, so pairs (0,1), (2,3)
    // ... may straddle chunk boundaries.
    if (is_c) live_tmp[rank] = i;
    __syncthreads();
    cand_base += total;
  }
  __syncthreads();
  // decide pairs: candidate 2m and 2m+1
  for (int m = tid; 2 * m + 1 < cand_base; m += 1024) {
    int ia = live_tmp[2 * m], ib = live_tmp[2 * m + 1];
    int sa = live[ia], sb = live[ib];
    double *wa = &state[(size_t)sa * L.stride + L.sc + SC_WEIGHT];
    double *wb = &state[(size_t)sb * L.stride + L.sc + SC_WEIGHT];
    double w1 = *wa, w2 = *wb, w3 = w1 + w2;
    double u[4];
    rng_uniform4(seed, (uint32_t)ia, (uint32_t)step, 7u, u);
    if (u[0] < w1 / w3) {
      *wa = w3;
      *wb = -1.0;  // marked dead
      wa[SC_FUSED - SC_WEIGHT] = 1.0;
    } else {
      *wb = w3;
      *wa = -1.0;
      wb[SC_FUSED - SC_WEIGHT] = 1.0;
    }
  }
  __syncthreads();
  // pass 2: survivors keep list order; dead slots to the free stack; splits append copies
  int out_base = 0, split_base = 0;
  // first count survivors + kills to know where split copies go and how many slots free
  for (int c0 = 0; c0 < n; c0 += 1024) {
    int i = c0 + tid;
    int slot = i < n ? live[i] : -1;
    double w = slot >= 0 ? state[(size_t)slot * L.stride + L.sc + SC_WEIGHT] : 0.0;
    int dead = (slot >= 0 && w < 0.01) ? 1 : 0;
    int keep = (slot >= 0 && !dead) ? 1 : 0;
    unsigned bk = __ballot_sync(QMCB_FULL_MASK, keep), bd = __ballot_sync(QMCB_FULL_MASK, dead);
    int pk = __popc(bk & ((1u << lane) - 1)), pd = __popc(bd & ((1u << lane) - 1));
    if (lane == 31) s_warp[wid] = ((pk + keep) << 16) | (pd + dead);
    __syncthreads();
    if (wid == 0) {
      int v = s_warp[lane];
      int vk = v >> 16, vd = v & 0xffff, xk = vk, xd = vd;
      for (int o = 1; o < 32; o <<= 1) {
        int yk = __shfl_up_sync(QMCB_FULL_MASK, xk, o), yd = __shfl_up_sync(QMCB_FULL_MASK, xd, o);
        if (lane >= o) {
          xk += yk;
          xd += yd;
        }
      }
      s_warp[lane] = ((xk - vk) << 16) | (xd - vd);
      if (lane == 31) {
        s_base[1] = xk;
        s_base[2] = xd;
      }
    }
    __syncthreads();
    int ok = s_warp[wid] >> 16, od = s_warp[wid] & 0xffff;
    if (keep) live_tmp[out_base + ok + pk] = slot;
    if (dead) free_stack[nfree + od + pd] = slot;
    int tk = s_base[1], td = s_base[2];
    __syncthreads();
    out_base += tk;
    nfree += td;
  }
  __syncthreads();
  // splits among survivors (in new list order), appended at the end
  int n_keep = out_base;
  double wsum_part = 0.0;
  for (int c0 = 0; c0 < n_keep; c0 += 1024) {
    int i = c0 + tid;
    int slot = i < n_keep ? live_tmp[i] : -1;
    double *wp = slot >= 0 ? &state[(size_t)slot * L.stride + L.sc + SC_WEIGHT] : nullptr;
    double w = wp ? *wp : 0.0;
    // the split test reads the weight before fusion, as the reference's single
    // pass does: the survivor of a fused pair (weight below the fusion
    // threshold before) never splits in the same pass
    const bool fused = wp && wp[SC_FUSED - SC_WEIGHT] != 0.0;
    if (fused) wp[SC_FUSED - SC_WEIGHT] = 0.0;
    int sp = (slot >= 0 && !fused && w > thr_split &&
              branch_recommended(state + (size_t)slot * L.stride + L.sc, e_orig, limit_branching)) ? 1 : 0;
    unsigned bs = __ballot_sync(QMCB_FULL_MASK, sp);
    int ps = __popc(bs & ((1u << lane) - 1));
    if (lane == 31) s_warp[wid] = ps + sp;
    __syncthreads();
    if (wid == 0) {
      int v = s_warp[lane], x = v;
      for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(QMCB_FULL_MASK, x, o);
        if (lane >= o) x += y;
      }
      s_warp[lane] = x - v;
      if (lane == 31) s_base[3] = x;
    }
    __syncthreads();
    int r = split_base + s_warp[wid] + ps;
    if (sp) {
      if (r < nfree) {
        int dst = free_stack[nfree - 1 - r];
        *wp = w * 0.5;
        copies[r] = make_int2(slot, dst);
        live_tmp[n_keep + r] = dst;
        wsum_part += w;  // both halves
      } else {
        wsum_part += w;  // no free slot: keep the walker whole
      }
    } else if (slot >= 0) {
      wsum_part += w;
    }
    int ts = s_base[3];
    __syncthreads();
    split_base += ts;
  }
  int n_split = min(split_base, nfree);
  __syncthreads();
  for (int i = tid; i < n_keep + n_split; i += 1024) live[i] = live_tmp[i];
  double ws = warp_sum(wsum_part);
  if (lane == 0) s_wsum[wid] = ws;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int k = 0; k < 32; k++) t += s_wsum[k];
    stats[ST_FINAL_W] = t;
    ctl[0] = n_keep + n_split;
    ctl[1] = nfree - n_split;
    ctl[2] = n_split;
  }
}

// Copies whole walker blocks for the splits recorded by k_branch; the copy
// keeps the halved weight already written to the source.
__device__ __forceinline__ void copy_blocks(double *state, const Layout &L, const int2 *copies, const int *ctl,
                                            int first, int stride)
{
  const int nc = ctl[2];
  for (int c = first; c < nc; c += stride) {
    int2 p = copies[c];
    const double *src = state + (size_t)p.x * L.stride;
    double *dst = state + (size_t)p.y * L.stride;
    for (int t = threadIdx.x; t < L.stride; t += blockDim.x) dst[t] = src[t];
  }
}

// E_est from the running weighted energy average and
// E_T = E_est - c ln(W / W0) (QMCManager::updateEstimatedEnergy /
// updateTrialEnergy, QMcBeaver/src/QMCManager.cpp:2247-2310).
// dyn_dt: also the effective time step dt <w p dR^2> / <w dR^2>
// (QMCDerivativeProperties::getEffectiveTimeStep, QMcBeaver/src/QMCDerivativeProperties.cpp:25-42).
__device__ __forceinline__ void update_energy(EnergyCtl *ectl, const double *stats, int min_samples_ok, int dyn_dt,
                                              double dt)
{
  if (dyn_dt && stats[ST_RUN_SUM_WD2] > 1e-20) ectl->dt_eff = dt * stats[ST_RUN_SUM_WPD2] / stats[ST_RUN_SUM_WD2];
  double sw = stats[ST_RUN_SUM_W];
  // E_est follows the running average once it holds 100 samples
  // (QMCManager::updateEstimatedEnergy, QMcBeaver/src/QMCManager.cpp:2247-2261)
  if (min_samples_ok && sw > 0.0 && stats[ST_RUN_COUNT] >= 100.0) ectl->e_est = stats[ST_RUN_SUM_WE] / sw;
  double ratio = stats[ST_FINAL_W] / ectl->target_weight;
  double lr = ratio > 1e-250 ? log(ratio) : 0.0;
  ectl->e_trial = ectl->e_est - ectl->pop_control * lr;
}

}  // namespace qmcb
