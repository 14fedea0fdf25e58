// invert.cu -- inverses of the walkers' Slater matrices, one thread tile per
// matrix held in registers (refresh and full evaluation).
//
// Gauss-Jordan by exchange steps: y = T x starts as T = D (rows electrons,
// columns orbitals); step j exchanges x_j with the y_b of the largest scaled
// pivot (the rule of the reference's LU, Array2D::ludcmp,
// QMcBeaver/include/Array2D.h:1204-1340) among the rows not yet used, without
// moving rows, so every element keeps its place in one thread's registers;
// at the end x = T y, its rows and columns in the pivots' order.
//
// A step is one pivot column and one pivot row through shared memory (two
// barriers, double-buffered), the pivot search repeated by every warp, and
// RL x CL fused multiply-adds per thread from RL + CL values; bound by its
// instruction issue (350 a warp and step at 50 x 50, 49 of them the update).
// Refresh, one warp per walker with the matrix in shared memory and this way
// (the rest of the refresh with it): 30 electrons, 15,710 walkers 696 and 291
// us; 100 electrons, 7,575 walkers 3,377 and 1,826 (1,124 of it here); 196
// electrons, 512 walkers 3,780 and 1,505.
#include "invert.h"

namespace qmcb {

// TX x TY threads, RL x CL elements each: matrices up to TY RL = TX CL = n.
// kWarp: 32 threads per matrix, four matrices a block.
template <int TX, int TY, int RL, int CL, typename TS>
__global__ void __launch_bounds__(TX *TY == 32 ? 128 : TX * TY)
    k_invert(const __grid_constant__ Layout L, int na, int nb, double *state, const int *slots, int num,
             const int *d_num)
{
  constexpr int kMax = TY * RL;
  static_assert(TX * CL == kMax && TX <= 32 && 32 % TX == 0, "square tiles, a row's threads in one warp");
  constexpr bool kWarp = TX * TY == 32;
  constexpr int kPer = kWarp ? 4 : 1;
  __shared__ double s_col[kPer][2][kMax], s_row[kPer][2][kMax], s_vv[kPer][kMax], s_piv[kPer][kMax];
  __shared__ int s_b[kPer][kMax], s_pos[kPer][kMax];
  const int nw = d_num ? *d_num : num;
  const int m = kWarp ? threadIdx.x >> 5 : 0;
  const int wi = blockIdx.x * kPer + m;
  if (wi >= nw) return;  // a whole block, or a warp that meets no block barrier
  const int sp = blockIdx.y, n = sp ? nb : na;
  if (n == 0) return;
  const int tid = kWarp ? threadIdx.x & 31 : threadIdx.x, lane = threadIdx.x & 31;
  const int tx = tid % TX, ty = tid / TX;
  double *blk = state + (size_t)(slots ? slots[wi] : wi) * L.stride;
  const TS *Dv = (const TS *)(blk + L.Dv[sp]);
  const auto sync = [] {
    if (kWarp)
      __syncwarp();
    else
      __syncthreads();
  };

  double T[RL][CL];
#pragma unroll
  for (int r = 0; r < RL; r++)
#pragma unroll
    for (int c = 0; c < CL; c++) {
      const int i = r * TY + ty, k = c * TX + tx;
      T[r][c] = i < n && k < n ? (double)Dv[i * n + k] : 0.0;
    }
  // scales 1 / max |row| (0 for a zero row: singular)
#pragma unroll
  for (int r = 0; r < RL; r++) {
    double big = 0.0;
#pragma unroll
    for (int c = 0; c < CL; c++) big = fmax(big, fabs(T[r][c]));
#pragma unroll
    for (int o = TX / 2; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(QMCB_FULL_MASK, big, o, TX));
    const int i = r * TY + ty;
    if (tx == 0 && i < n) s_vv[m][i] = big == 0.0 ? 0.0 : 1.0 / big;
  }
  sync();
  bool sing = false;
  for (int i = lane; i < n; i += 32) sing |= s_vv[m][i] == 0.0;
  sing = __any_sync(QMCB_FULL_MASK, sing);  // the same in every warp

#pragma unroll
  for (int jl = 0; jl < CL; jl++) {
    for (int jt = 0; jt < TX; jt++) {
      const int j = jl * TX + jt;
      if (j >= n || sing) break;
      const int par = j & 1;
      // the pivot column, and zero in its place (its new values are products)
      if (tx == jt) {
#pragma unroll
        for (int r = 0; r < RL; r++) {
          s_col[m][par][r * TY + ty] = T[r][jl];  // (zero in the padding)
          T[r][jl] = 0.0;
        }
      }
      sync();
      double best = -1.0;
      int b = -1;
      for (int i = lane; i < n; i += 32) {
        const double s = s_vv[m][i], v = s < 0.0 ? -1.0 : s * fabs(s_col[m][par][i]);
        if (v >= best && s >= 0.0) {
          best = v;
          b = i;
        }
      }
      // the largest candidate: by its leading 32 bits (one warp reduction),
      // and exactly when several lanes share those
      const unsigned key = best < 0.0 ? 0u : 1u + (unsigned)__double2hiint(best);
      const unsigned top = __reduce_max_sync(QMCB_FULL_MASK, key);
      const unsigned who = __ballot_sync(QMCB_FULL_MASK, key == top);
      if (__popc(who) == 1) {
        b = __shfl_sync(QMCB_FULL_MASK, b, __ffs(who) - 1);
      } else {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double ob = __shfl_xor_sync(QMCB_FULL_MASK, best, o);
          const int oi = __shfl_xor_sync(QMCB_FULL_MASK, b, o);
          if (ob > best || (ob == best && oi > b)) {
            best = ob;
            b = oi;
          }
        }
      }
      if (b < 0) {  // every candidate NaN
        sing = true;
        break;
      }
      const double p = s_col[m][par][b];
      if (p == 0.0) {
        sing = true;
        break;
      }
      const int bt = b % TY, bl = b / TY;
      // the pivot row likewise
      if (ty == bt) {
#pragma unroll
        for (int r = 0; r < RL; r++)
          if (r == bl) {
#pragma unroll
            for (int c = 0; c < CL; c++) {
              s_row[m][par][c * TX + tx] = T[r][c];
              T[r][c] = 0.0;
            }
          }
      }
      sync();
      if (tid == 0) {
        s_vv[m][b] = -1.0;  // used (the other warps have searched)
        s_piv[m][j] = p;
        s_b[m][j] = b;
        s_pos[m][b] = j;
      }
      const double pinv = 1.0 / p;
      double rk[CL];
#pragma unroll
      for (int c = 0; c < CL; c++) rk[c] = -s_row[m][par][c * TX + tx] * pinv;
      rk[jl] = tx == jt ? pinv : rk[jl];
#pragma unroll
      for (int r = 0; r < RL; r++) {
        const int i = r * TY + ty;
        const double ci = i == b ? 1.0 : s_col[m][par][i];
#pragma unroll
        for (int c = 0; c < CL; c++) T[r][c] = fma(ci, rk[c], T[r][c]);
      }
    }
  }
  sync();
  double *Inv = blk + L.Inv[sp];
#pragma unroll
  for (int r = 0; r < RL; r++)
#pragma unroll
    for (int c = 0; c < CL; c++) {
      const int i = r * TY + ty, k = c * TX + tx;
      if (i < n && k < n) Inv[sing ? i * n + k : s_pos[m][i] * n + s_b[m][k]] = T[r][c];
    }
  if (tid < 32) {
    double *sc = blk + L.sc;
    double ld = 0.0;
    int flips = 0;  // inversions of the pivots' order, negative pivots
    if (!sing)
      for (int j = lane; j < n; j += 32) {
        ld += log(fabs(s_piv[m][j]));
        flips += s_piv[m][j] < 0.0;
        const int bj = s_b[m][j];
        for (int l = j + 1; l < n; l++) flips += s_b[m][l] < bj;
      }
    ld = warp_sum(ld);
    flips = __reduce_add_sync(QMCB_FULL_MASK, flips);
    if (lane == 0) {
      sc[SC_LOGDET_A + sp] = sing ? -INFINITY : ld;
      sc[SC_SIGN_A + sp] = sing ? 0.0 : flips & 1 ? -1.0 : 1.0;
      sc[SC_INVCUR_A + sp] = 0.0;
    }
  }
}

template <int TX, int TY, int RL, int CL>
static void launch_of(bool mixed, const Layout &L, int na, int nb, double *state, int cap, cudaStream_t st,
                      const int *slots, int num, const int *d_num)
{
  const int per = TX * TY == 32 ? 4 : 1;
  const dim3 g((cap + per - 1) / per, nb > 0 ? 2 : 1), b(TX * TY == 32 ? 128 : TX * TY);
  if (mixed)
    k_invert<TX, TY, RL, CL, float><<<g, b, 0, st>>>(L, na, nb, state, slots, num, d_num);
  else
    k_invert<TX, TY, RL, CL, double><<<g, b, 0, st>>>(L, na, nb, state, slots, num, d_num);
}

cudaError_t invert_launch(bool mixed, const DevSys &S, const Layout &L, double *state, int cap, cudaStream_t st,
                          const int *slots, int num, const int *d_num)
{
  const int n = S.na > S.nb ? S.na : S.nb;
  // one warp up to 32, then blocks of 64 or 256 threads with the smallest
  // square tiles (padding is multiplied like the rest)
  if (n <= 8)
    launch_of<8, 4, 2, 1>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  else if (n <= 16)
    launch_of<8, 4, 4, 2>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  else if (n <= 24)
    launch_of<8, 4, 6, 3>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  else if (n <= 32)
    launch_of<8, 4, 8, 4>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  else if (n <= 40)
    launch_of<8, 8, 5, 5>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  else if (n <= 56)
    launch_of<8, 8, 7, 7>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  else if (n <= 80)
    launch_of<16, 16, 5, 5>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  else if (n <= 112)
    launch_of<16, 16, 7, 7>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  else
    launch_of<16, 16, 8, 8>(mixed, L, S.na, S.nb, state, cap, st, slots, num, d_num);
  return cudaGetLastError();
}

}  // namespace qmcb
