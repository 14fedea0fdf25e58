// sweep.cu -- single-electron steps of small spins, 16 walkers per CTA.
//
// For one determinant whose spins hold at most 16 electrons (no cusp
// replacement, three-body terms or Umrigar93 moves).  A CTA takes 16 walkers
// through all the steps between two branchings or refreshes: a step needs no
// launch of its own, the walkers' positions, gradients, drifts and scalars
// stay in shared memory throughout, and their derivative rows and inverses
// stay in L2 from step to step.  Each step has two phases:
//
//   rows   one walker per half-warp lane: proposals, then the basis shells of
//          the 16 walkers (a shell per half-warp) and their contraction on the FP64 tensor pipe, as
//          rows64.cu, the five orbital rows left in shared memory
//   move   G = 8 or 16 lanes per walker, lane c owning electrons c and
//          G + c, and in registers the moved spin's column of one of them:
//          Jastrow and potential changes, Sherman-Morrison update, ratio
//          sums, psi quantities, drift, acceptance and reweight, write back
//
// One walker per warp spends a third of its instructions on scalars that all
// 32 lanes repeat, on warp reductions and on loops over 15 columns or 6 nuclei
// with idle lanes; with two or four walkers per warp those are shared, and
// the 3 to 8 sums of a stage go through one transposing reduction.
//
// Everything a chain goes on from (rows, inverses, ratio sums, pair sums,
// drifts) rounds as in k_move: the same operations, and sums over lanes in the
// order of its 32 lanes, which a lane here takes two (G = 16) or up to four of.
// A walker next to a node amplifies a rounding by 1e6 and more until the next
// refresh, so sums in any other order showed as 1e-8 of single local energies.
// (The laplacian's sum over the columns and the acceptance's exponents, which
// feed nothing back, add in the lanes' own order, and so does the one sum of
// the drift limited by a common factor, qf_mod 1.)  150 steps of 16,384 walkers
// of 30 electrons take 16.1 ms so, 15.9 with sums in the cheapest order.
//
// Bound by the latency of a step's chain of phases (30 electrons: 40 k cycles
// with one CTA per SM -- proposals 1, basis 7.5, products 6, pair terms 3,
// Sherman-Morrison 2, ratio sums 7, drift 4.5, acceptance and write back 6 --
// at 8 warps), which a second CTA on the SM overlaps (16 walkers a CTA: 98 us
// a step at 16,384 walkers; 32 walkers in one CTA of 16 warps: 129; both with
// the derivative rows as four matrices).  128
// registers a thread; with 223 KB of shared memory the L1 is small, so spilled
// registers cost L2 latencies and the column of the inverse leaves the
// registers for the ratio sums.  30 electrons, 15,710 walkers: 225 us a step
// by the move kernel, 87 here; 10 electrons, 100 walkers: 18 and 9.
#include "rows64_device.cuh"
#include "sweep.h"

namespace qmcb {

// ---- lanes of one walker: groups of G consecutive lanes, mask gm
template <int G>
__device__ __forceinline__ double group_get(double v, int k, unsigned gm)
{
  return __shfl_sync(gm, v, k, G);
}

template <int G>
__device__ __forceinline__ double group_sum(double v, unsigned gm)
{
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(gm, v, o, G);
  return v;
}

// Sums of eight values over the group at once: a lane returns one total
// (group_total).  The widest exchange first, as group_sum and
// warp_sum, so that every total has their bits; each of the first three
// exchanges halves the values a lane keeps.
template <int G>
__device__ __forceinline__ double group_sum8(const double v[8], int c, unsigned gm)
{
  double a[4], b[2];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const bool hi = c & (G / 2);
    const double keep = hi ? v[4 + k] : v[k], give = hi ? v[k] : v[4 + k];
    a[k] = keep + __shfl_xor_sync(gm, give, G / 2, G);
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const bool hi = c & (G / 4);
    const double keep = hi ? a[2 + k] : a[k], give = hi ? a[k] : a[2 + k];
    b[k] = keep + __shfl_xor_sync(gm, give, G / 4, G);
  }
  const bool hi = c & (G / 8);
  const double keep = hi ? b[1] : b[0], give = hi ? b[0] : b[1];
  double s = keep + __shfl_xor_sync(gm, give, G / 8, G);
  if (G == 16) s += __shfl_xor_sync(gm, s, 1, G);
  return s;
}
// The total of v[k] in every lane: it is with the lanes whose three leading
// bits are k's.
template <int G>
__device__ __forceinline__ double group_total(double sums, int k, unsigned gm)
{
  return group_get<G>(sums, k * (G / 8), gm);
}

// The general correlation functions out of line (the closed form stays inline).
static __device__ __noinline__ void pade_general(const DevSys &S, int f, double r, double *u)
{
  pade_eval(S, f, r, u[0], u[1], u[2]);
}

__device__ __forceinline__ void pair_function(const DevSys &S, int f, double r, double &u, double &du, double &d2u)
{
  if (S.pade_simple) {
    const double2 ab = __ldg(&S.pade_ab[f]);
    const double q = 1.0 / fma(ab.y, r, 1.0);
    const double aq = ab.x * q;
    u = aq * r;
    du = aq * q;
    d2u = -2.0 * ab.y * du * q;
  } else {
    double v[3];
    pade_general(S, f, r, v);
    u = v[0];
    du = v[1];
    d2u = v[2];
  }
}

// The pair (moved electron, partner at P): changes of the correlation
// function f (-1: none), weight k of the laplacian terms (2 for electron
// pairs, 1 for nuclei).  v: gradient change on the moved electron; dinv =
// 1 / r_new - 1 / r_old.  Without branches in the closed form, so that a
// lane's pairs overlap; on = false gives zeros.
__device__ __forceinline__ void pair_change(const DevSys &S, int f, double k, bool on, const double ro[3],
                                            const double rn[3], const double P[3], double &dinv, double &dU,
                                            double &dUxx, double v[3])
{
  double xo[3], xn[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    // a lane without a pair computes at distance sqrt(3) and drops the result
    xo[d] = on ? ro[d] - P[d] : 1.0;
    xn[d] = on ? rn[d] - P[d] : 1.0;
  }
  const double r2o = rows64_r2(xo[0], xo[1], xo[2]), r2n = rows64_r2(xn[0], xn[1], xn[2]);
  const double io = rsqrt(r2o), in_ = rsqrt(r2n);
  dinv = on ? in_ - io : 0.0;
  const bool corr = on && f >= 0;
  double uo, duo, d2uo, un, dun, d2un;
  pair_function(S, f < 0 ? 0 : f, r2o * io, uo, duo, d2uo);
  pair_function(S, f < 0 ? 0 : f, r2n * in_, un, dun, d2un);
  const double sn = corr ? dun * in_ : 0.0, so = corr ? duo * io : 0.0;
  dU += corr ? un - uo : 0.0;
  dUxx += corr ? k * ((2.0 * in_ * dun + d2un) - (2.0 * io * duo + d2uo)) : 0.0;
#pragma unroll
  for (int d = 0; d < 3; d++) v[d] = sn * xn[d] - so * xo[d];
}

// The moved electron's change with nucleus A (none from M on), added to the
// sums w: dU, lap, V_ee, V_en, gradient on it.
__device__ __forceinline__ void nuclear_changes(const DevSys &S, int sp, int A, int M, const double ro[3],
                                                const double rn[3], double w[7])
{
  const double4 P = S.nuc[A < M ? A : 0];
  const double p[3] = {P.x, P.y, P.z};
  double v[3], dinv;
  pair_change(S, S.en[sp][A < M ? A : 0], 1.0, A < M, ro, rn, p, dinv, w[0], w[1], v);
  w[3] -= P.w * dinv;
#pragma unroll
  for (int d = 0; d < 3; d++) w[4 + d] += v[d];
}

// The nuclei of more than a walker's lanes hold: those of the move kernel's
// lanes c and G + c (w[0..7), w[7..14), which hold their electrons' sums) and of
// the two lanes 2 G + c, 3 G + c of a group of eight, nuclei l, l + 32, .. each;
// then the sums over these in the order of warp_sum, in w[0..7).
template <int G>
static __device__ __noinline__ void many_nuclei(const DevSys &S, int sp, int c, const double ro[3], const double rn[3],
                                                double w[14])
{
  for (int half = 0; half < 2; half++)
    for (int A = G * half + c; A - c < S.M; A += 32) nuclear_changes(S, sp, A, S.M, ro, rn, w + 7 * half);
  if (G == 8)
    for (int half = 0; half < 2; half++) {
      double x[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      for (int A = 2 * G + G * half + c; A - c < S.M; A += 32) nuclear_changes(S, sp, A, S.M, ro, rn, x);
      for (int k = 0; k < 7; k++) w[7 * half + k] += x[k];
    }
  for (int k = 0; k < 7; k++) w[k] += w[7 + k];
}

// Shared memory of a CTA (offsets in doubles): the chunk of basis values (the
// moved spin's inverses once it is consumed), two coefficient buffers,
// positions [3][TW], displacements [3][TW], acceptance uniforms [TW], rows
// [TW][5][kLdR], sums [9][TW]; then the
// walkers (sweep_walker_doubles each), two record buffers and the chunk table.
constexpr int TW = 16;  // walkers per CTA
template <int G>
struct SweepShared {
  static constexpr int kTiles = G / 8;                 // 8-orbital tiles
  static constexpr int kLdA = rows64_pitch(TW);
  static constexpr int kChunk = rows64_chunk(G);       // functions per chunk of the tables
  static constexpr int kLdB = 8 * kTiles + 4;          // as rows64: 4 mod 8
  static constexpr int kLdR = G + 1;                   // orbitals of a row, zero beyond the spin's
  static constexpr int kSums = 9;
  // (with room for a shell cut by a chunk's end on either side)
  static constexpr int kRowsA = (kChunk + (G == 16 ? 2 * kR64Lead : 0)) * kLdA;
  static constexpr int kChi = ((kRowsA > TW * G * G ? kRowsA : TW * G * G) + 2 * TW - 1) / (2 * TW) * (2 * TW);
  static_assert(kChi % (2 * TW) == 0 && kChi / TW >= G * G, "a walker's inverse in its part of the chunk, 16-byte aligned");
  static constexpr int kC = kChunk * kLdB;
  static constexpr int kPos = kChi + 2 * kC;
  static constexpr int kRows = kPos + 7 * TW;
  static constexpr int kSum = kRows + TW * 5 * kLdR;
  static constexpr int kWalk = (kSum + kSums * TW + 1) & ~1;
};
// a walker's staged arrays: positions, then gradD .. scalars as in its block
__host__ __device__ inline int sweep_walker_doubles(const Layout &L) { return L.mv_r + L.mv_tail; }

// The last orbitals of the slices in which the move kernel's 32 lanes share a
// spin's ratio sums.
__device__ __forceinline__ unsigned slice_ends_of(int n)
{
  unsigned ends = 0;
  if (n > 0) {
    const int slices = 32 / n;
    for (int s = 1; s <= slices; s++) ends |= 1u << n * s / slices >> 1;
  }
  return ends;
}

// One move of the group's walker (list entry wi, tile index gi) from the
// rows in shared memory; lane c of the group.
template <bool kMetropolis, int G>
__device__ __forceinline__ void sweep_move(const DevSys &S, const Layout &L, const RunCfg &cfg, double *blk, int wi,
                                           int gi, int c, unsigned gm, const MoveArgs &mv, const EnergyCtl *ectl,
                                           double *sm, unsigned slice_ends, const EvalOut &out)
{
  using Sh = SweepShared<G>;
  const int N = S.N, e = mv.e, sp = e < S.na ? 0 : 1;
  const int n = sp ? S.nb : S.na, base = sp ? S.na : 0, el = e - base;
  const double *D = sm + Sh::kRows + (size_t)gi * 5 * Sh::kLdR;
  double *sR = sm + Sh::kWalk + (size_t)gi * sweep_walker_doubles(L), *sT = sR + L.mv_r;
  double *sUx = sT + (L.Ux - L.gradD), *smg = sT + (L.mgrad - L.gradD), *sc = sT + (L.sc - L.gradD);
  double *sInv = sm + (size_t)gi * (Sh::kChi / TW);    // the moved spin's inverse, updated in place
  const int idx[2] = {c, G + c};                       // this lane's electrons
  const bool has[2] = {idx[0] < N, idx[1] < N};
  const int col = (c - base) & (G - 1);                // the moved spin's column of one of them,
  const bool mine = col < n;                           // or none
  const int cc = mine ? col : 0;

  // exponent sum of G(R -> R'): the displacement and, as the reference, the
  // drift of the electrons that stay (QMcBeaver/src/QMCWalker.cpp:383-388)
  double gf = 0.0;
  if (kMetropolis && cfg.sampling == 1 && !cfg.exact_gf) {
#pragma unroll
    for (int s = 0; s < 2; s++)
      if (has[s] && idx[s] != e)
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const double dd = cfg.dt * smg[3 * idx[s] + d];
          gf += dd * dd;
        }
  }

  // ---- Jastrow and potential changes (jastrow_pe_move_warp)
  double vx[2][3];  // gradient change of the lane's electrons (subtracted)
  double s8[8];     // dU, lap, V_ee, V_en, gradient on e, drift exponent
  {
    double ro[3], rn[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      ro[d] = sR[3 * e + d];
      rn[d] = sm[Sh::kPos + TW * d + gi];
    }
    // the lanes c and G + c of jastrow_pe_move_warp one after another: lane l's
    // electron l, then nucleus l
    double u[3];
    const auto electron = [&](int s, double &dU, double &dUxx, double &dVee) {
      const double *r = sR + (has[s] ? 3 * idx[s] : 0), P[3] = {r[0], r[1], r[2]};
      dU = dUxx = 0.0;
      pair_change(S, (idx[s] < S.na ? 0 : 1) != sp ? S.ee[0] : sp == 0 ? S.ee[1] : S.ee[2], 2.0,
                  has[s] && idx[s] != e, ro, rn, P, dVee, dU, dUxx, vx[s]);
    };
    electron(0, s8[0], s8[1], s8[2]);
    electron(1, u[0], u[1], u[2]);
    s8[3] = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) s8[4 + d] = vx[0][d];
    if (S.M <= G) {
      nuclear_changes(S, sp, c, S.M, ro, rn, s8);
#pragma unroll
      for (int k = 0; k < 3; k++) s8[k] += u[k];
#pragma unroll
      for (int d = 0; d < 3; d++) s8[4 + d] += vx[1][d];
    } else {
      double w[14];
#pragma unroll
      for (int k = 0; k < 7; k++) w[k] = s8[k];
#pragma unroll
      for (int k = 0; k < 7; k++) w[7 + k] = k < 3 ? u[k] : k == 3 ? 0.0 : vx[1][k - 4];
      many_nuclei<G>(S, sp, c, ro, rn, w);
#pragma unroll
      for (int k = 0; k < 7; k++) s8[k] = w[k];
    }
    s8[7] = gf;
  }
  const double sums1 = group_sum8<G>(s8, c, gm);
  // ---- Sherman-Morrison row replacement (Array2D::inverseUpdateOneRow,
  //      QMcBeaver/include/Array2D.h:1567-1610) on column c in registers
  //      (orbitals beyond the spin's: zero)
  cp_async_wait<0>();
  __syncwarp(gm);
  double inv[G];
#pragma unroll
  for (int o = 0; o < G; o++) inv[o] = o < n ? sInv[o * n + cc] : 0.0;
  const double ratio = group_sum<G>(c < n ? D[c] * sInv[c * n + el] : 0.0, gm);
  double dot = 0.0;
#pragma unroll
  for (int o = 0; o < G; o++) dot = fma(D[o], inv[o], dot);
  bool bad = !(ratio != 0.0) || !isfinite(ratio);
  const double q = 1.0 / ratio;
  {
    // inv - vc * (old column of the moved electron), its own column inv * q
    const double vc = col == el ? 0.0 : dot * q, f = col == el ? q : 1.0;
#pragma unroll
    for (int o = 0; o < G; o++) inv[o] = fma(-vc, o < n ? sInv[o * n + el] : 0.0, f * inv[o]);
  }
  __syncwarp(gm);  // the old column has been read
  // the new column back to shared memory: its registers serve the loads below
  if (mine) {
#pragma unroll
    for (int o = 0; o < G; o++)
      if (o < n) sInv[o * n + col] = inv[o];
  }

  // ---- ratio sums of the moved spin (QMcBeaver/src/QMCSlater.cpp:741-762):
  //      this lane's column of the inverse with its derivative columns (the
  //      moved electron's from the new rows), added up slice by slice as the
  //      move kernel's lanes do.  The rows are read once per move
  //      (from L2), eight orbitals' loads in flight; addresses past the
  //      spin's orbitals are clamped and their terms dropped.
  double lp = 0.0, gn[3] = {0.0, 0.0, 0.0};
  {
    const Deriv4<double> *D4 = (const Deriv4<double> *)(blk + L.D4[sp]) + cc;
    const bool own = col == el;
    constexpr int kB = 8;
    // slice by slice for the larger spins (2 or 3 of up to 8 orbitals), the
    // whole column in one batch for the smaller (4 or more of up to 2)
    const int slices = G == 16 ? __popc(slice_ends) : 1;
    unsigned rest = slice_ends;
    int oa = 0;
#pragma unroll 1
    for (int s = 0; s < slices; s++) {
      const int ob = G == 16 ? __ffs(rest) : n;
      rest &= rest - 1;
      Deriv4<double> g[kB], part = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int u = 0; u < kB; u++) g[u] = ld_deriv<false>(D4 + min(oa + u, ob - 1) * n);
#pragma unroll
      for (int u = 0; u < kB; u++) {
        const int o = min(oa + u, ob - 1);
        const double iv = oa + u < ob ? sInv[o * n + cc] : 0.0;
        const double *Do = D + o;
        part.x = fma(own ? Do[Sh::kLdR] : g[u].x, iv, part.x);
        part.y = fma(own ? Do[2 * Sh::kLdR] : g[u].y, iv, part.y);
        part.z = fma(own ? Do[3 * Sh::kLdR] : g[u].z, iv, part.z);
        part.l = fma(own ? Do[4 * Sh::kLdR] : g[u].l, iv, part.l);
        if (G == 8 ? slice_ends >> u & 1 : u == kB - 1) {  // the same in the whole block
          gn[0] += part.x;
          gn[1] += part.y;
          gn[2] += part.z;
          lp += part.l;
          part = {0.0, 0.0, 0.0, 0.0};
        }
      }
      oa = ob;
    }
    lp = mine ? lp : 0.0;
  }

  // ---- psi quantities (psi_lap_warp) and the modified drift (qf_modify_warp)
  double gr[2][3], mg[2][3], part[2] = {0.0, 0.0}, pu = 0.0, pm = 0.0, pr = 0.0;
  double R[2][3], Ux[2][3], gD[2][3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double ge = group_total<G>(sums1, 4 + d, gm);
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const int i = has[s] ? 3 * idx[s] + d : d;
      const bool me = idx[s] == e;
      const double u = sUx[i] + (me ? ge : -vx[s][d]);
      Ux[s][d] = has[s] ? u : 0.0;
      gD[s][d] = has[s] ? (idx[s] == base + col && mine ? gn[d] : sT[i]) : 0.0;
      R[s][d] = me ? sm[Sh::kPos + TW * d + gi] : sR[i];
    }
  }
#pragma unroll
  for (int s = 0; s < 2; s++)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double x = gD[s][d], u = Ux[s][d];
      gr[s][d] = x + u;
      part[s] += u * x * 2.0;
      part[s] += u * u;
      pu += gr[s][d] * gr[s][d];
    }
  double factor[2] = {1.0, 1.0};
  if (cfg.qf_mod == 1) {
    const double magsq = group_sum<G>(pu, gm), a = cfg.qf_a;
    factor[0] = factor[1] = (-1.0 + sqrt(1.0 + 2 * a * magsq * cfg.dt)) / (a * magsq * cfg.dt);
  } else if (cfg.qf_mod == 2) {
    // closest nucleus: smallest distance, first index on ties
    double cd[2] = {1e300, 1e300};
    int cn[2] = {0, 0};
    for (int A = 0; A < S.M; A++) {
      const double4 P = S.nuc[A];
#pragma unroll
      for (int s = 0; s < 2; s++) {
        const double dx = R[s][0] - P.x, dy = R[s][1] - P.y, dz = R[s][2] - P.z;
        const double d2 = dx * dx + dy * dy + dz * dz;
        if (d2 < cd[s]) {
          cd[s] = d2;
          cn[s] = A;
        }
      }
    }
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const double4 P = S.nuc[cn[s]];
      const double nv[3] = {R[s][0] - P.x, R[s][1] - P.y, R[s][2] - P.z};
      const double il = rsqrt(cd[s]);
      const double ev2 = gr[s][0] * gr[s][0] + gr[s][1] * gr[s][1] + gr[s][2] * gr[s][2];
      const bool tiny = fabs(ev2) < 1e-10;
      const double scl = tiny ? 0.0 : rsqrt(ev2);
      double dotp = 0.0;
#pragma unroll
      for (int d = 0; d < 3; d++) dotp += (nv[d] * il) * (gr[s][d] * scl);
      const double temp = P.w * P.w * cd[s];
      const double a = 0.5 * (1.0 + dotp) + temp / (10.0 * (4.0 + temp));
      factor[s] = tiny ? 1.0 : (-1.0 + sqrt(1.0 + 2.0 * a * ev2 * cfg.dt)) / (a * ev2 * cfg.dt);
    }
  }
#pragma unroll
  for (int s = 0; s < 2; s++)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      mg[s][d] = gr[s][d] * factor[s];
      pm += mg[s][d] * mg[s][d];
    }
  if (kMetropolis && cfg.sampling == 1) {
    // exponent sum of G(R' -> R)
#pragma unroll
    for (int s = 0; s < 2; s++)
      if (has[s] && (idx[s] == e || !cfg.exact_gf))
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const double back = idx[s] == e ? sR[3 * e + d] - R[s][d] : 0.0, tt = back - cfg.dt * mg[s][d];
          pr += tt * tt;
        }
  }
  const double t8[8] = {lp, part[0] + part[1], pm, pu, pr, 0.0, 0.0, 0.0};
  const double sums2 = group_sum8<G>(t8, c, gm);
  const double lapR = group_total<G>(sums2, 0, gm);
  double Dxx = 0.0;
  if (S.na > 0) Dxx += sp == 0 ? lapR : sc[SC_LAPR_A];
  if (S.nb > 0) Dxx += sp == 1 ? lapR : sc[SC_LAPR_B];
  const double dU = group_total<G>(sums1, 0, gm);
  const double U_new = sc[SC_U] + dU, Uxx_new = sc[SC_UXX] + group_total<G>(sums1, 1, gm);
  const double lap = Dxx + Uxx_new + group_total<G>(sums2, 1, gm);
  const double lm = sqrt(group_total<G>(sums2, 2, gm)), lu = sqrt(group_total<G>(sums2, 3, gm));
  const double modratio = lm / lu;
  if (isnan(lm) || isnan(lu) || isnan(modratio) || lu == 0.0) bad = true;
  const double Vee = sc[SC_VEE] + group_total<G>(sums1, 2, gm), Ven = sc[SC_VEN] + group_total<G>(sums1, 3, gm);
  const double PE = S.Pnn + Vee + Ven;
  const double EL = -0.5 * lap + PE;
  if (isnan(EL)) bad = true;
  const double log_abs = log(fabs(ratio));
  const double logdet_new = sc[SC_LOGDET_A + sp] + log_abs;
  const double sign_new = sc[SC_SIGN_A + sp] * (ratio < 0 ? -1.0 : 1.0);

  bool accept = true;
  double p_acc = 1.0;
  if (kMetropolis) {
    double log_g = 0.0;
    if (cfg.sampling == 1) {
      double g_fwd = group_total<G>(sums1, 7, gm);
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const double x = sm[Sh::kPos + (3 + d) * TW + gi];
        g_fwd += x * x;
      }
      log_g = -(group_total<G>(sums2, 4, gm) - g_fwd) / (2.0 * cfg.dt);
    }
    MoveTally ty;
    double ro[3], rn[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      ro[d] = sR[3 * e + d];
      rn[d] = sm[Sh::kPos + TW * d + gi];
    }
    const double age = sc[SC_AGE], w = sc[SC_WEIGHT], mo = sc[SC_MODRATIO], Eo = sc[SC_EL];
    __syncwarp(gm);  // every lane has its old scalars before the leader writes
    accept = accept_and_reweight(cfg, mv, ectl, sc, c == 0, age, w, mo, Eo, ro, rn, sm[Sh::kPos + 6 * TW + gi], log_abs + dU, log_g, ratio < 0, bad,
                                 EL, modratio, ty);
    p_acc = ty.p;
    if (c == 0) {
      double *t = sm + Sh::kSum + gi;
      t[0] += ty.p;
      t[TW] += 1.0;
      if (bad) t[2 * TW] += 1.0;
      if (ty.observed) {
        t[3 * TW] += ty.w;
        t[4 * TW] += ty.w * ty.E;
        t[5 * TW] += ty.w * ty.E * ty.E;
        t[6 * TW] += 1.0;
        t[7 * TW] += ty.w * ty.p * ty.d2;
        t[8 * TW] += ty.w * ty.d2;
      }
    }
  }
  if (kMetropolis && mv.dump) {
    // the step's configuration records (dump_configs)
    const int rec = 6 * N + 4;
    double *tr = mv.dump + (size_t)wi * 2 * rec, *old = tr + rec;
#pragma unroll
    for (int s = 0; s < 2; s++)
      if (has[s])
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const int t = 3 * idx[s] + d;
          tr[t] = R[s][d];
          old[t] = sR[t];
          tr[3 * N + 1 + t] = gD[s][d];
          old[3 * N + 1 + t] = sT[t];
        }
    if (c == 0) {
      tr[3 * N] = Dxx;
      old[3 * N] = (S.na > 0 ? sc[SC_LAPR_A] : 0.0) + (S.nb > 0 ? sc[SC_LAPR_B] : 0.0);
      tr[6 * N + 1] = U_new;
      old[6 * N + 1] = sc[SC_U];
      tr[6 * N + 2] = PE;
      old[6 * N + 2] = sc[SC_PE];
      tr[6 * N + 3] = p_acc;
      old[6 * N + 3] = 1.0 - p_acc;
    }
  }
  __syncwarp(gm);
  if (accept) {
    double *Inv = blk + L.Inv[sp];
    for (int i = c; i < n * n; i += G) Inv[i] = sInv[i];
    if (c < n) {
      // lane c writes orbital c of the moved electron's new rows
      blk[L.Dv[sp] + el * n + c] = D[c];
      ((Deriv4<double> *)(blk + L.D4[sp]))[c * n + el] = {D[Sh::kLdR + c], D[2 * Sh::kLdR + c], D[3 * Sh::kLdR + c],
                                                        D[4 * Sh::kLdR + c]};
    }
#pragma unroll
    for (int s = 0; s < 2; s++)
      if (has[s])
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const int t = 3 * idx[s] + d;
          sT[t] = gD[s][d];  // (the other spin's as they were)
          if (idx[s] == e) sR[t] = R[s][d];
          sUx[t] = Ux[s][d];
          smg[t] = mg[s][d];
        }
    if (c == 0) {
      sc[SC_U] = U_new;
      sc[SC_UXX] = Uxx_new;
      sc[SC_LAPR_A + sp] = lapR;
      sc[SC_LOGDET_A + sp] = logdet_new;
      sc[SC_SIGN_A + sp] = sign_new;
      sc[SC_VEE] = Vee;
      sc[SC_VEN] = Ven;
      sc[SC_PE] = PE;
      sc[SC_EL] = EL;
      sc[SC_LAP] = lap;
      sc[SC_MODRATIO] = modratio;
      sc[SC_STATUS] = bad ? 1.0 : 0.0;
    }
  }
  if (!kMetropolis) {
    if (c == 0) {
      unsigned st = bad ? 1u : 0u;
      if (isnan(EL) || isnan(lap)) st |= 2u;
      // (the scalars hold the new state)
      if (out.log_abs_psi) out.log_abs_psi[wi] = sc[SC_LOGDET_A] + sc[SC_LOGDET_B] + U_new;
      if (out.sign) out.sign[wi] = sc[SC_SIGN_A] * sc[SC_SIGN_B];
      if (out.lap) out.lap[wi] = lap;
      if (out.e_local) out.e_local[wi] = EL;
      if (out.pe) {
        out.pe[3 * wi] = PE;
        out.pe[3 * wi + 1] = Ven;
        out.pe[3 * wi + 2] = Vee;
      }
      if (out.status) out.status[wi] = (unsigned char)st;
    }
    // the per-electron outputs (often stores into host memory) with
    // consecutive lanes on consecutive elements
    __syncwarp(gm);
    for (int t = c; t < 3 * N; t += G) {
      const double x = sT[t] + sUx[t];  // gradPsiRatio, as gr above
      blk[L.grad + t] = x;
      if (out.grad) out.grad[(size_t)wi * 3 * N + t] = x;
      if (out.mgrad) out.mgrad[(size_t)wi * 3 * N + t] = smg[t];
    }
  }
}

template <bool kMetropolis, int G>
__global__ void __launch_bounds__(TW * G, G == 8 ? 4 : 2)
    k_sweep(const __grid_constant__ DevSys S, const __grid_constant__ Layout L, const __grid_constant__ RunCfg cfg,
            const __grid_constant__ Rows64 T, double *state, const int *slots, int num, const int *d_num,
            const double *R_in, const __grid_constant__ SweepArgs a, const EnergyCtl *ectl, double *stats,
            const __grid_constant__ EvalOut out)
{
  using Sh = SweepShared<G>;
  extern __shared__ double sm[];
  constexpr int kWarps = TW * G / 32, kThreads = TW * G, kMT = 5 * TW / 16;
  const int nw = d_num ? *d_num : num;
  const int w0 = blockIdx.x * TW;
  if (w0 >= nw) return;
  const int lane = lane_id(), warp = threadIdx.x >> 5, tid = threadIdx.x;
  double *chi = sm, *Cs = sm + Sh::kChi, *pos = sm + Sh::kPos;
  const int wd = sweep_walker_doubles(L);
  double *walk = sm + Sh::kWalk, *recs = walk + (size_t)TW * wd;
  int4 *chunks = (int4 *)(recs + 2 * T.rec_max);
  // rows phase: lane % TW = walker (those past the list repeat its last walker)
  const int lw = lane % TW, wl = min(w0 + lw, nw - 1);
  const int slot_l = slots ? slots[wl] : wl;
  const double *sR_l = walk + (size_t)(wl - w0) * wd, *smg_l = sR_l + L.mv_r + (L.mgrad - L.gradD);
  // move phase: G lanes per walker
  const int gi = tid / G, c = tid % G, wi = w0 + gi;
  const bool active = wi < nw;
  const unsigned gm = (G == 8 ? 0xffu : 0xffffu) << (lane & ~(G - 1));
  double *blk = state + (size_t)(active ? (slots ? slots[wi] : wi) : 0) * L.stride;

  auto load_chunk = [&](int k, int sp) {
    const int4 ch = chunks[k];
    const int n2 = (chunks[k + 1].y - ch.y) / 2, ldg = T.ldb[sp];
    double *dst = recs + (k & 1) * T.rec_max, *cs = Cs + (k & 1) * Sh::kC;
    for (int i = tid; i < n2; i += kThreads) cp_async16(dst + 2 * i, T.rec + ch.y + 2 * i);
    // coefficient rows in 16-byte pieces, ldg / 2 lanes a row
    const int per = ldg / 2;
    const double *src = T.ct[sp] + (size_t)ch.w * ldg;
    for (int i = tid; i < (ch.z >> 16) * per; i += kThreads) {
      const int k2 = i / per, o = 2 * (i - k2 * per);
      cp_async16(cs + k2 * Sh::kLdB + o, src + (size_t)k2 * ldg + o);
    }
  };

  for (int i = tid; i <= T.nchunk; i += kThreads) chunks[i] = __ldg(&T.chunk[i]);
  if (kMetropolis)
    for (int i = tid; i < Sh::kSums * TW; i += kThreads) sm[Sh::kSum + i] = 0.0;
  // the walkers' arrays
  if (active) {
    double *w = walk + (size_t)gi * wd;
    for (int i = 2 * c; i < L.mv_r; i += 2 * G) cp_async16(w + i, blk + L.R + i);
    for (int i = 2 * c; i < L.mv_tail; i += 2 * G) cp_async16(w + L.mv_r + i, blk + L.gradD + i);
  }
  cp_async_commit();
  __syncthreads();
  const int nsteps = kMetropolis ? a.nsteps : 1;
  const unsigned ends[2] = {slice_ends_of(S.na), slice_ends_of(S.nb)};
  MoveArgs mv{};
  {
    const int e0 = kMetropolis ? a.step0 % S.N : a.e;
    load_chunk(0, e0 < S.na ? 0 : 1);
    cp_async_commit();
  }
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll 1
  for (int s = 0; s < nsteps; s++) {
    mv.step = a.step0 + s;
    mv.e = kMetropolis ? mv.step % S.N : a.e;
    mv.do_reweight = kMetropolis && mv.e == 0;
    mv.reweight_on = mv.step >= a.reweight_start;
    mv.dump = a.dump;
    const int e = mv.e, sp = e < S.na ? 0 : 1, n = sp ? S.nb : S.na;

    // ---- rows: warp d < 3 takes coordinate d of its lane's walker, warp 3 the
    //      acceptance uniform (the draws and formulas of propose_move)
    if (warp < (kMetropolis ? 4 : 3) && lane < TW) {
      if (kMetropolis) {
        const U4 x = philox4x32(U4{(uint32_t)slot_l, (uint32_t)mv.step, (uint32_t)warp, 0x51ED2701u}, cfg.seed);
        if (warp == 3) {
          pos[6 * TW + lane] = u01(x.z, x.w);
        } else {
          const double drift = sqrt(cfg.dt) * (double)gaussian_draw(x);
          double disp = drift;
          if (cfg.sampling == 1) disp += cfg.dt * smg_l[3 * e + warp];
          pos[TW * warp + lane] = sR_l[3 * e + warp] + disp;
          pos[(3 + warp) * TW + lane] = drift;
        }
      } else {
        pos[TW * warp + lane] =
            a.rin_moved ? R_in[(size_t)wl * 3 + warp] : R_in[((size_t)wl * S.N + e) * 3 + warp];
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    // MMA tiles (16 rows x 8 orbitals): tile i = rows i % 5, orbitals i / 5
    const int tiles = kMT * ((n + 7) / 8);
    double acc[2][4];
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[j][q] = 0.0;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll 1
    for (int k = 0; k < T.nchunk; k++) {
      const int4 ch = chunks[k];
      const int padded = ch.z >> 16;
      // the next chunk lands while this one is evaluated and multiplied
      if (k + 1 < T.nchunk) load_chunk(k + 1, sp);
      cp_async_commit();
      {
        const double rx = pos[lw], ry = pos[TW + lw], rz = pos[2 * TW + lw];
        const double *rec = recs + (k & 1) * T.rec_max;
        // a shell per half-warp (a chunk's are sorted by cost: neighbours are alike)
#pragma unroll 1
        for (int i = 2 * warp + lane / TW; i < ch.x; i += 2 * kWarps) {
          const double head = rec[i];
          rows64_shell<TW, true>(rec + __double2hiint(head), __double2loint(head), rx, ry, rz, chi + lw);
        }
        // padding functions: their coefficients are zero, their values must be finite
        for (int i = (ch.z & 0xffff) * 5 * TW + tid; i < padded * 5 * TW; i += kThreads)
          chi[(T.lead + i / (5 * TW)) * Sh::kLdA + i % (5 * TW)] = 0.0;
      }
      __syncthreads();
      // (a warp's two tiles side by side: their chains overlap)
      const double *ap[2], *bp[2];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int i = warp + j * kWarps;
        ap[j] = chi + (T.lead + t) * Sh::kLdA + 16 * (i % kMT) + g;
        bp[j] = Cs + (k & 1) * Sh::kC + t * Sh::kLdB + 8 * (i / kMT) + g;
      }
      for (int kk = 0; kk < padded; kk += 8) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
          if (warp + j * kWarps >= tiles) continue;
          const double av[4] = {ap[j][kk * Sh::kLdA], ap[j][kk * Sh::kLdA + 8], ap[j][(kk + 4) * Sh::kLdA],
                                ap[j][(kk + 4) * Sh::kLdA + 8]};
          dmma_m16n8k8(acc[j], av, bp[j][kk * Sh::kLdB], bp[j][(kk + 4) * Sh::kLdB]);
        }
      }
      cp_async_wait<0>();
      __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int i = warp + j * kWarps;
      if (i >= tiles) continue;
      const int mt = i % kMT, o0 = 8 * (i / kMT) + 2 * t;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        double *row = sm + Sh::kRows + ((size_t)(8 * h + g) * 5 + mt) * Sh::kLdR;
#pragma unroll
        for (int u = 0; u < 2; u++)
          row[o0 + u] = acc[j][2 * h + u];  // zero beyond the spin's orbitals
      }
    }
    if (n <= 8 && G == 16) {  // the second tile of a small spin
      for (int i = tid; i < TW * 5 * 8; i += kThreads) sm[Sh::kRows + (i >> 3) * Sh::kLdR + 8 + (i & 7)] = 0.0;
    }
    // the moved spin's inverses into the consumed chunk, and the next step's
    // first chunk, land during the moves
    if (active) {
      const double *src = blk + L.Inv[sp];
      double *dst = sm + (size_t)gi * (Sh::kChi / TW);
      for (int i = 2 * c; i < n * n; i += 2 * G) cp_async16(dst + i, src + i);
    }
    if (s + 1 < nsteps) load_chunk(0, (mv.step + 1) % S.N < S.na ? 0 : 1);
    cp_async_commit();
    __syncthreads();

    // ---- moves
    if (active) sweep_move<kMetropolis, G>(S, L, cfg, blk, wi, gi, c, gm, mv, ectl, sm, ends[sp], out);
    // the walkers' new state is read by other lanes of this CTA next step
    __syncthreads();
  }
  if (active) {
    const double *w = walk + (size_t)gi * wd;
    for (int i = c; i < 3 * S.N; i += G) {
      blk[L.R + i] = w[i];
      blk[L.gradD + i] = w[L.mv_r + i];
      blk[L.Ux + i] = w[L.mv_r + (L.Ux - L.gradD) + i];
      blk[L.mgrad + i] = w[L.mv_r + (L.mgrad - L.gradD) + i];
    }
    for (int i = c; i < kScalars; i += G) blk[L.sc + i] = w[L.mv_r + (L.sc - L.gradD) + i];
  }
  if (kMetropolis && warp == 0) {
    double v[Sh::kSums];
#pragma unroll
    for (int k = 0; k < Sh::kSums; k++) v[k] = warp_sum(lane < TW ? sm[Sh::kSum + TW * k + lane] : 0.0);
    if (lane == 0) {
      atomicAdd(&stats[ST_SUM_ACC], v[0]);
      atomicAdd(&stats[ST_MOVES], v[1]);
      if (v[2] > 0.0) atomicAdd(&stats[ST_SINGULAR], v[2]);
      if (v[6] > 0.0) {
        atomicAdd(&stats[ST_SUM_W], v[3]);
        atomicAdd(&stats[ST_SUM_WE], v[4]);
        atomicAdd(&stats[ST_SUM_WE2], v[5]);
        atomicAdd(&stats[ST_RUN_SUM_W], v[3]);
        atomicAdd(&stats[ST_RUN_SUM_WE], v[4]);
        atomicAdd(&stats[ST_RUN_COUNT], v[6]);
        if (cfg.dyn_dt) {
          atomicAdd(&stats[ST_RUN_SUM_WPD2], v[7]);
          atomicAdd(&stats[ST_RUN_SUM_WD2], v[8]);
        }
      }
    }
  }
}

int sweep_smem_bytes(int nmax, const Layout &L, const Rows64 &T)
{
  return (int)sizeof(double) * ((nmax > 8 ? SweepShared<16>::kWalk : SweepShared<8>::kWalk) +
                                TW * sweep_walker_doubles(L) + 2 * T.rec_max + 2 * (T.nchunk + 1));
}

static const void *sweep_fn(bool metropolis, int nmax)
{
  if (nmax > 8) return metropolis ? (const void *)k_sweep<true, 16> : (const void *)k_sweep<false, 16>;
  return metropolis ? (const void *)k_sweep<true, 8> : (const void *)k_sweep<false, 8>;
}

cudaError_t sweep_limits(int max_bytes)
{
  cudaError_t e = cudaSuccess;
  for (int nmax : {8, 16})
    for (bool metropolis : {false, true})
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sweep_fn(metropolis, nmax), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 max_bytes);
  return e;
}

cudaError_t sweep_launch(bool metropolis, const DevSys &S, const Layout &L, const RunCfg &cfg, const Rows64 &T,
                         double *state, int cap, cudaStream_t st, const int *slots, int num, const int *d_num,
                         const double *R_in, const SweepArgs &a, const EnergyCtl *ectl, double *stats,
                         const EvalOut &out)
{
  const int nmax = S.na > S.nb ? S.na : S.nb, G = nmax > 8 ? 16 : 8;
  const dim3 g((cap + TW - 1) / TW);
  void *args[] = {(void *)&S, (void *)&L,    (void *)&cfg, (void *)&T,    &state,         &slots, &num,
                  &d_num,     (void *)&R_in, (void *)&a,   (void *)&ectl, (void *)&stats, (void *)&out};
  return cudaLaunchKernel(sweep_fn(metropolis, nmax), g, dim3(TW * G), args, sweep_smem_bytes(nmax, L, T), st);
}

}  // namespace qmcb
