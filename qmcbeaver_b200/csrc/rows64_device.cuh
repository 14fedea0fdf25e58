// rows64_device.cuh -- basis shells one walker per lane, and the FP64 MMA
// (rows64.cu, sweep.cu).
#pragma once

#include "rows64.h"

namespace qmcb {

// D(16x8) += A(16x8) B(8x8), FP64.  Fragments with g = lane / 4, t = lane % 4:
// a0 = A[g][t], a1 = A[g+8][t], a2 = A[g][t+4], a3 = A[g+8][t+4],
// b0 = B[t][g], b1 = B[t+4][g], d0, d1 = D[g][2t, 2t+1], d2, d3 = D[g+8][2t, 2t+1].
__device__ __forceinline__ void dmma_m16n8k8(double d[4], const double a[4], double b0, double b1)
{
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

// The squared distance of the exponentials, and that of the Laplacian's sums:
// the one-walker passes round the latter by itself for a moved electron
// (basis_function_rows: its squares also serve the powers, so its sum is not
// fused) and share the former in a full evaluation (shell_members).  Spelled
// out, so that a walker's rows are the same bits whichever kernel makes them.
__device__ __forceinline__ double rows64_r2(double x, double y, double z)
{
  return fma(z, z, fma(x, x, __dmul_rn(y, y)));
}
template <bool kMoved>
__device__ __forceinline__ double rows64_r2x4(double x, double y, double z, double r2)
{
  return 4.0 * (kMoved ? __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z)) : r2);
}

// A shell of any other shape (kR64Any): rec = centre, (L, primitives) in the
// two words of a double, exponents, then for every function its powers and
// coefficients.  E0 = sum c e, E1 = sum c a e, El = sum c e (4 r^2 a^2 - (4L + 6) a)
// as in basis_function_rows.
template <int TW, bool kMoved>
static __device__ __noinline__ void rows64_shell_any(const double *rec, int nmem, double rx, double ry, double rz,
                                                     double *chi)
{
  const double x = rx - rec[0], y = ry - rec[1], z = rz - rec[2];
  const double r2 = rows64_r2(x, y, z);
  const int L = __double2loint(rec[3]), np = __double2hiint(rec[3]);
  const double Lf = 4.0 * L + 6.0, r2x4 = rows64_r2x4<kMoved>(x, y, z, r2);
  const double *al = rec + 4, *mem = al + np;
  double E0 = 0.0, E1 = 0.0, El = 0.0;
  for (int m = 0; m < nmem; m++, chi += rows64_pitch(TW), mem += np + 1) {
    const int pw = __double2loint(mem[0]);
    if (!(pw >> 24)) {  // else the previous function's coefficients
      E0 = E1 = El = 0.0;
      for (int i = 0; i < np; i++) {
        const double ai = al[i], t = mem[1 + i] * exp(-ai * r2);
        E0 += t;
        E1 = fma(t, ai, E1);
        El = fma(t, ai * fma(r2x4, ai, -Lf), El);
      }
    }
    const int a = pw & 0xff, b = (pw >> 8) & 0xff, c = (pw >> 16) & 0xff;
    const double xa = ipow(x, a), yb = ipow(y, b), zc = ipow(z, c);
    const double P = xa * yb * zc;
    const double Px = a ? a * ipow(x, a - 1) * yb * zc : 0.0;
    const double Py = b ? b * xa * ipow(y, b - 1) * zc : 0.0;
    const double Pz = c ? c * xa * yb * ipow(z, c - 1) : 0.0;
    double Pl = 0.0;
    if (a > 1) Pl += a * (a - 1.0) * ipow(x, a - 2) * yb * zc;
    if (b > 1) Pl += b * (b - 1.0) * xa * ipow(y, b - 2) * zc;
    if (c > 1) Pl += c * (c - 1.0) * xa * yb * ipow(z, c - 2);
    const double w = -2.0 * P * E1;
    chi[0] = E0 * P;
    chi[TW] = fma(E0, Px, x * w);
    chi[2 * TW] = fma(E0, Py, y * w);
    chi[3 * TW] = fma(E0, Pz, z * w);
    chi[4 * TW] = fma(E0, Pl, P * El);
  }
}

// One function of a fast shell: its radial sums from the three primitives'
// exponentials e, exponents a and a (4 r^2 a - (4L + 6)) and its coefficients,
// then its five values from its polynomial P, that polynomial's gradient and
// Laplacian.  Every operation rounds as in basis_function_rows.
struct Rows64Radial {
  double x, y, z, e[3], a[3], l[3];
};
template <int TW>
__device__ __forceinline__ void rows64_function(double *chi, const double *coef, const Rows64Radial &R, double P,
                                                double Px, double Py, double Pz, double Pl)
{
  double E0 = 0.0, E1 = 0.0, El = 0.0;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double t = coef[i] * R.e[i];
    E0 += t;
    E1 = fma(t, R.a[i], E1);
    El = fma(t, R.l[i], El);
  }
  const double w = -2.0 * P * E1;
  chi[0] = E0 * P;
  // (products rounded before the sum also where a constant polynomial
  // derivative would let them be fused)
  chi[TW] = fma(E0, Px, __dmul_rn(R.x, w));
  chi[2 * TW] = fma(E0, Py, __dmul_rn(R.y, w));
  chi[3 * TW] = fma(E0, Pz, __dmul_rn(R.z, w));
  chi[4 * TW] = fma(E0, Pl, __dmul_rn(P, El));
}

// One shell for this lane's position into the chunk (TW walkers a tile: row =
// quantity x TW + walker).  Complete s, p and d
// shells of up to three primitives (padded with zero coefficients) run
// without a branch or a table lookup per function: rec = centre, exponents
// [3], every function's coefficients [3] in the order s; x, y, z; xx, yy, zz,
// xy, xz, yz.
template <int TW, bool kMoved>
__device__ __forceinline__ void rows64_shell(const double *rec, int packed, double rx, double ry, double rz, double *chi)
{
  constexpr int D = rows64_pitch(TW);
  chi += (size_t)(packed & 0xff) * D;
  const int kind = packed >> 16;
  if (kind == kR64Any) {
    rows64_shell_any<TW, kMoved>(rec, (packed >> 8) & 0xff, rx, ry, rz, chi);
    return;
  }
  Rows64Radial R;
  R.x = rx - rec[0];
  R.y = ry - rec[1];
  R.z = rz - rec[2];
  const double r2 = rows64_r2(R.x, R.y, R.z);
  const double Lf = 4.0 * kind + 6.0, r2x4 = rows64_r2x4<kMoved>(R.x, R.y, R.z, r2);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    R.a[i] = rec[3 + i];
    R.e[i] = exp(-R.a[i] * r2);
    R.l[i] = R.a[i] * fma(r2x4, R.a[i], -Lf);
  }
  const double *c = rec + 6;
  if (kind == 0) {
    rows64_function<TW>(chi, c, R, 1.0, 0.0, 0.0, 0.0, 0.0);
  } else if (kind == 1) {
    rows64_function<TW>(chi, c, R, R.x, 1.0, 0.0, 0.0, 0.0);
    rows64_function<TW>(chi + D, c + 3, R, R.y, 0.0, 1.0, 0.0, 0.0);
    rows64_function<TW>(chi + 2 * D, c + 6, R, R.z, 0.0, 0.0, 1.0, 0.0);
  } else {
    rows64_function<TW>(chi, c, R, R.x * R.x, 2.0 * R.x, 0.0, 0.0, 2.0);
    rows64_function<TW>(chi + D, c + 3, R, R.y * R.y, 0.0, 2.0 * R.y, 0.0, 2.0);
    rows64_function<TW>(chi + 2 * D, c + 6, R, R.z * R.z, 0.0, 0.0, 2.0 * R.z, 2.0);
    rows64_function<TW>(chi + 3 * D, c + 9, R, R.x * R.y, R.y, R.x, 0.0, 0.0);
    rows64_function<TW>(chi + 4 * D, c + 12, R, R.x * R.z, R.z, 0.0, R.x, 0.0);
    rows64_function<TW>(chi + 5 * D, c + 15, R, R.y * R.z, 0.0, R.z, R.y, 0.0);
  }
}

}  // namespace qmcb
