// md.cu -- the several-determinant kernels (kernels_md.cuh).
#include "kernels_md.cuh"
#include "launches.h"

namespace qmcb {

// ------------------------------------------------------------------------
// Full evaluation (do_basis = true) or refresh from the stored rows.
// Three blocks per SM (168 registers): the refresh of 4,096 / 8,192 walkers of
// 12 and 16 electrons takes 476 and 965 us, 588 and 1,274 at the 241 registers
// the compiler takes uncapped (2 blocks); of 64 walkers 146 both ways.
__global__ void __launch_bounds__(128, 3)
    k_full_md(const __grid_constant__ DevSys S, const __grid_constant__ Layout L, const __grid_constant__ RunCfg cfg,
              double *state, const int *slots, int num, const int *d_num, const double *R_in, int do_basis,
              const __grid_constant__ EvalOut out)
{
  extern __shared__ double smem[];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int nw = d_num ? *d_num : num;
  const int wi = blockIdx.x * (blockDim.x >> 5) + warp;
  if (wi >= nw) return;
  const int N = S.N, K = S.K, nmax = max(S.na, S.nb), amax = max(S.nact[0], S.nact[1]), nd = S.ndet;
  const int slot = slots ? slots[wi] : wi;
  double *blk = state + (size_t)slot * L.stride;
  double *sm = smem + (size_t)warp * full_md_scratch_doubles(N, K, nmax, amax, nd);
  const int ldc = K + 1;
  double *chi = sm;
  double *Dn = chi + even(5 * ldc);
  double *A = Dn + even(5 * amax);
  double *X = A + nmax * nmax;
  double *vv = X + nmax * nmax;
  double *piv = vv + even(nmax);
  double *Rs = piv + even(nmax);
  double *tpr = Rs + even(3 * N);
  double *R = blk + L.R;
  double *sc = blk + L.sc;

  if (R_in) {
    for (int t = lane; t < 3 * N; t += 32) R[t] = R_in[(size_t)wi * 3 * N + t];
    if (lane < 2) sc[SC_MDCUR_A + lane] = 0.0;
  }
  for (int t = lane; t < 3 * N; t += 32) Rs[t] = R[t];
  __syncwarp();

  MdBlock mb[2];
  for (int sp = 0; sp < 2; sp++) mb[sp] = md_block(S, L, blk, sp, sc[SC_MDCUR_A + sp] != 0.0 ? 1 : 0);
  for (int sp = 0; sp < 2; sp++) {
    const int n = sp ? S.nb : S.na, a = S.nact[sp], base = sp ? S.na : 0;
    if (n == 0) continue;
    double *Dv = blk + L.Dv[sp];
    Deriv4<double> *D4 = (Deriv4<double> *)(blk + L.D4[sp]);
    if (do_basis) {
      for (int e = 0; e < n; e++) {
        const double r[3] = {Rs[3 * (base + e)], Rs[3 * (base + e) + 1], Rs[3 * (base + e) + 2]};
        basis_shells_warp(S, r, chi, ldc);
        __syncwarp();
        contract_dmma_warp(chi, ldc, S.ct[sp], a, K, Dn);
        __syncwarp();
        if (S.cusp) {
          cusp_replace_warp(S, sp, r, Dn, a, a);
          __syncwarp();
        }
        for (int o = lane; o < a; o += 32) {
          Dv[e * a + o] = Dn[o];
          D4[o * n + e] = {Dn[a + o], Dn[2 * a + o], Dn[3 * a + o], Dn[4 * a + o]};
        }
        __syncwarp();
      }
    }
    double logdet = 0.0, sign = 1.0;
    bool ok = true;
    for (int c = 0; c < nd; c++) {
      const int *occ = S.docc[sp] + (size_t)c * n;
      // QMCWavefunction::getDataForCI: the columns of determinant c
      for (int t = lane; t < n * n; t += 32) A[t] = Dv[(t / n) * a + occ[t % n]];
      __syncwarp();
      bool lu = c == 0;
      if (c > 0 && ok) {
        // swap in the columns that differ from determinant c-1
        const int *sw = S.dswap[sp] + (size_t)c * n;
        for (int k = 0; k < n && sw[k] >= 0; k++) {
          const double r = inverse_update_col_warp(X, A, vv, n, sw[k]);
          if (!(r != 0.0) || !isfinite(r)) {
            lu = true;
            break;
          }
          logdet += log(fabs(r));
          if (r < 0) sign = -sign;
        }
      } else if (c > 0) {
        lu = true;
      }
      if (lu) {
        for (int t = lane; t < n * n; t += 32) A[t] = Dv[(t / n) * a + occ[t % n]];
        __syncwarp();
        ok = lu_inverse_warp(A, X, vv, piv, n, logdet, sign);
      }
      double *Inv = mb[sp].inv + (size_t)c * n * n;
      for (int t = lane; t < n * n; t += 32) Inv[t] = X[t];
      // ratio sums of determinant c (QMcBeaver/src/QMCSlater.cpp:741-762)
      double lp = 0.0;
      for (int e = lane; e < n; e += 32) {
        double gx = 0, gy = 0, gz = 0;
        for (int o = 0; o < n; o++) {
          const int orb = occ[o];
          const double iv = X[o * n + e];
          const Deriv4<double> v = D4[orb * n + e];
          lp += v.l * iv;
          gx += v.x * iv;
          gy += v.y * iv;
          gz += v.z * iv;
        }
        double *g = mb[sp].g + ((size_t)c * n + e) * 3;
        g[0] = gx;
        g[1] = gy;
        g[2] = gz;
      }
      lp = warp_sum(lp);
      if (lane == 0) {
        double *d = mb[sp].dsc + 4 * c;
        d[0] = ok ? logdet : 0.0;
        d[1] = ok ? sign : 1.0;
        d[2] = ok ? lp : 0.0;
        d[3] = ok ? 0.0 : 1.0;
      }
      __syncwarp();
    }
  }

  double logD, sgnD;
  bool bad;
  md_weights(S, S.na > 0 ? mb[0].dsc : nullptr, S.nb > 0 ? mb[1].dsc : nullptr, tpr, logD, sgnD, bad);
  double *gD = blk + L.gradD, *gr = blk + L.grad, *mg = blk + L.mgrad, *ux = blk + L.Ux;
  const double Dxx = md_combine(S, &mb[0], &mb[1], tpr, gD);
  double U, Uxx, Vee, Ven;
  jastrow_pe_full_warp<true>(S, Rs, ux, U, Uxx, Vee, Ven);
  __syncwarp();
  const double lap = psi_lap_warp(N, gD, ux, gr, Dxx, Uxx);
  __syncwarp();
  const double modratio = qf_modify_warp(S, cfg, Rs, gr, mg, &bad);
  const double PE = S.Pnn + Vee + Ven;
  const double EL = -0.5 * lap + PE;
  if (lane == 0) {
    sc[SC_U] = U;
    sc[SC_UXX] = Uxx;
    sc[SC_VEE] = Vee;
    sc[SC_VEN] = Ven;
    sc[SC_PE] = PE;
    sc[SC_EL] = EL;
    sc[SC_LAP] = lap;
    sc[SC_MODRATIO] = modratio;
    sc[SC_LOGDET_A] = logD;
    sc[SC_LOGDET_B] = 0.0;
    sc[SC_SIGN_A] = sgnD;
    sc[SC_SIGN_B] = 1.0;
    sc[SC_LAPR_A] = Dxx;
    sc[SC_LAPR_B] = 0.0;
    unsigned st = bad ? 1u : 0u;
    if (isnan(EL) || isnan(lap)) st |= 2u;
    sc[SC_STATUS] = (double)st;
    if (R_in) {
      sc[SC_WEIGHT] = 1.0;
      sc[SC_AGE] = 0.0;
      sc[SC_AGE_MOVED] = 0.0;
      sc[SC_DW] = 1.0;
    }
  }
  __syncwarp();
  write_eval_out(out, wi, N, logD + U, sgnD, lap, EL, PE, Ven, Vee, bad, gr, mg);
}

// Four blocks per SM (128 registers, 330 bytes spilled): a move of 4,096 /
// 8,192 walkers of 12 and 16 electrons takes 82 and 205 us, 100 and 212 with
// three; of 64 to 512 walkers 35 both ways.
template <bool kMetropolis>
__global__ void __launch_bounds__(128, 4)
    k_move_md(const __grid_constant__ DevSys S, const __grid_constant__ Layout L, const __grid_constant__ RunCfg cfg,
              double *state, const int *slots, int num, const int *d_num, const double *R_in,
              const __grid_constant__ MoveArgs mv, const EnergyCtl *ectl, double *stats,
              const __grid_constant__ EvalOut out)
{
  extern __shared__ double smem[];
  const int warp = threadIdx.x >> 5;
  const int nw = d_num ? *d_num : num;
  const int wi = blockIdx.x * (blockDim.x >> 5) + warp;
  if (wi >= nw) return;
  const int nmax = max(S.na, S.nb), amax = max(S.nact[0], S.nact[1]);
  const int tail = L.sc + kScalars - L.gradD, tbneed = S.ntb > 0 ? 3 * S.N * S.M : 0;
  double *sm = smem + (size_t)warp * move_md_scratch_doubles(S.N, S.K, nmax, amax, S.ndet, tail, S.nslot, tbneed);
  md_move_walker<kMetropolis>(S, L, cfg, state, slots, wi, sm, R_in, mv, ectl, stats, out);
}

const void *full_md_fn() { return (const void *)k_full_md; }

const void *move_md_fn(bool metropolis)
{
  return metropolis ? (const void *)k_move_md<true> : (const void *)k_move_md<false>;
}

}  // namespace qmcb
