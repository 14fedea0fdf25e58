// rows64.cu -- batched FP64 orbital rows on the FP64 tensor pipe.
//
// The orbital contraction of a step (QMCSlater::update_Ds -> Array2D::gemm,
// QMcBeaver/src/QMCSlater.cpp:856-862) for 32 walkers per CTA: the five basis
// quantities of the moved electron of every walker (160 rows) times the
// spin's MO coefficients, basis evaluation and contraction in one kernel.
//
// A warp evaluates one shell of basis functions for 32 walkers, one walker
// per lane: the shell's centre, exponents, coefficients and powers are the
// same for the whole warp, so there are no divergent powers, no per-lane
// table reads and no idle lanes, and the exponentials are formed once per
// shell.  The values go to shared memory as a [functions][160 rows] chunk
// that the warps then multiply with the matching chunk of coefficients
// (mma.sync m16n8k8, one 16-row tile per warp over its orbital tiles).
// One walker per warp reads every coefficient once per walker (160 KB per
// move at 400 functions and 50 orbitals); here a CTA reads them once for 32.
// Measured, a step at 100 electrons / 7,575 walkers: the fused move kernel
// 1,277 us, this kernel and the move kernel on its rows 131 + 472 us; at 30
// electrons / 15,710 walkers 225 us and 39 + 155 us.
#include "rows64_device.cuh"

namespace qmcb {

// The Umrigar93 proposal of electron e, one walker per lane: the draws and
// formulas of umrigar_propose.
static __device__ __noinline__ void rows64_umrigar(const DevSys &S, const RunCfg &cfg, int slot, int step,
                                                   const double *ro, const double *mge, double *pos)
{
  double u[8], rn[3];
  for (int k = 0; k < 4; k++) {
    const U4 c = philox4x32(U4{(uint32_t)slot, (uint32_t)step, (uint32_t)(8 + k), 0x0A7E5A21u}, cfg.seed);
    u[2 * k] = u01(c.x, c.y);
    u[2 * k + 1] = u01(c.z, c.w);
  }
  UmrigarFrame F;
  umrigar_frame(S, cfg, ro, mge, F);
  umrigar_draw(F, cfg, u, rn);
  for (int d = 0; d < 3; d++) pos[32 * d + lane_id()] = rn[d];
}

// rows[list index][5][n] (R64_PROPOSE, R64_GIVEN), or the walkers' stored
// Slater values and derivative rows (R64_ALL).  Grid: R64_ALL: x = tiles of 32
// list entries x electrons of the spin x orbital splits (a tile's electrons
// adjacent, so that their interleaved derivative columns meet in L2; one
// dimension, since the others end at 65,535 tiles); else x = tiles, y = splits.
//
// Per chunk the warps evaluate its shells, meet, multiply, and meet again; the
// next chunk's coefficients and records land meanwhile.  The two
// phases share the FP64 pipe, so running them side by side gains nothing: with
// half the warps multiplying while the others evaluate, every FP64 instruction
// queues behind 64-cycle MMAs (100 electrons, 7,575 walkers: 146 us a step
// against 131).  The products take two thirds of a CTA's cycles at 50 orbitals
// (75% of the pipe's rate while they run) and a third at 15; the floor is the
// FP64 pipe (47 us at 100 electrons, 10 us at 30 electrons and 15,710 walkers,
// measured 39).  One CTA of 20 warps (NH = 2) or two of 10 per SM at 96
// registers: the 237 or 491 tiles of those sizes are two waves.
template <int kMode, int NT, int NH>
__global__ void __launch_bounds__(32 * kR64MTiles *NH, NH == 2 ? 1 : 2)
    k_rows64(const __grid_constant__ DevSys S, const __grid_constant__ Layout L, const __grid_constant__ RunCfg cfg,
             const __grid_constant__ Rows64 T, double *state, const int *slots, int num, const int *d_num,
             const double *R_in, const __grid_constant__ MoveArgs mv, int sp, double *rows)
{
  extern __shared__ double sm64[];
  constexpr int kWarps = kR64MTiles * NH, kThreads = 32 * kWarps;
  constexpr int kLdB = 8 * NT * NH + 4;
  const int nw = d_num ? *d_num : num;
  const int n = sp ? S.nb : S.na, base = sp ? S.na : 0;
  const int splits = rows64_splits(n), per_tile = kMode == R64_ALL ? n * splits : 1;
  const int w0 = blockIdx.x / per_tile * kR64Walkers;
  if (w0 >= nw) return;
  const int lane = lane_id(), warp = threadIdx.x >> 5, tid = threadIdx.x;
  const int split = kMode == R64_ALL ? blockIdx.x % splits : blockIdx.y;
  const int e = kMode == R64_ALL ? base + blockIdx.x % per_tile / splits : mv.e;
  double *chi = sm64;                           // [kR64Lead + kR64Chunk][kR64LdA], the chunk from row T.lead
  double *Cs = chi + (kR64Lead + kR64Chunk) * kR64LdA;  // two buffers [kR64Chunk][kLdB]
  double *pos = Cs + 2 * kR64Chunk * kLdB;      // [3][32]
  double *recs = pos + 3 * kR64Walkers;         // two buffers of a chunk's shell records
  const int wi = min(w0 + lane, nw - 1);        // the lanes past the list repeat its last walker
  const int slot = slots ? slots[wi] : wi;
  const int ldg = T.ldb[sp];
  const double *ct = T.ct[sp] + split * 8 * NT * NH;
  // a chunk's coefficients into its buffer, in the background
  auto load_coefficients = [&](int c) {
    const int4 ch = __ldg(&T.chunk[c]);
    double *dst = Cs + (c & 1) * kR64Chunk * kLdB;
    // 16-byte pieces, a warp per row
    const double *src = ct + (size_t)ch.w * ldg;
    for (int k = warp; k < (ch.z >> 16); k += kWarps)
      if (lane < 4 * NT * NH) cp_async16(dst + k * kLdB + 2 * lane, src + (size_t)k * ldg + 2 * lane);
  };
  auto load_records = [&](int c) {
    const int4 ch = __ldg(&T.chunk[c]);
    const int n2 = (__ldg(&T.chunk[c + 1]).y - ch.y) / 2;
    double *dst = recs + (c & 1) * T.rec_max;
    for (int i = tid; i < n2; i += kThreads) cp_async16(dst + 2 * i, T.rec + ch.y + 2 * i);
  };
  load_records(0);
  load_coefficients(0);
  cp_async_commit();
  // the positions: warp d < 3 takes coordinate d of its lane's walker
  const double *blk = state + (size_t)slot * L.stride;
  if (kMode == R64_PROPOSE && cfg.sampling == 2) {
    if (warp == 0) rows64_umrigar(S, cfg, slot, mv.step, blk + L.R + 3 * e, blk + L.mgrad + 3 * e, pos);
  } else if (warp < 3) {
    double x;
    if (kMode == R64_GIVEN && mv.rin_moved) {
      x = R_in[(size_t)wi * 3 + warp];
    } else if (kMode == R64_GIVEN || (kMode == R64_ALL && R_in)) {
      x = R_in[((size_t)wi * S.N + e) * 3 + warp];
    } else {
      x = blk[L.R + 3 * e + warp];
      if (kMode == R64_PROPOSE) {
        // the draws and formulas of propose_move
        const double m = cfg.sampling == 1 ? blk[L.mgrad + 3 * e + warp] : 0.0;
        const double drift = sqrt(cfg.dt) * (double)gaussian_draw(philox4x32(
                                                U4{(uint32_t)slot, (uint32_t)mv.step, (uint32_t)warp, 0x51ED2701u},
                                                cfg.seed));
        double disp = drift;
        if (cfg.sampling == 1) disp += cfg.dt * m;
        x += disp;
      }
    }
    pos[32 * warp + lane] = x;
  }
  double acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; j++)
#pragma unroll
    for (int q = 0; q < 4; q++) acc[j][q] = 0.0;
  cp_async_wait<0>();
  __syncthreads();
  const int mtile = warp % kR64MTiles, half = warp / kR64MTiles;
  const int g = lane >> 2, t = lane & 3;
  const int cols = n - split * 8 * NT * NH;  // this CTA's orbitals (tiles of padding alone are skipped)
  for (int c = 0; c < T.nchunk; c++) {
    const int4 ch = __ldg(&T.chunk[c]);
    const int padded = ch.z >> 16;
    // the next chunk lands while this one is evaluated and multiplied
    if (c + 1 < T.nchunk) {
      load_records(c + 1);
      load_coefficients(c + 1);
    }
    cp_async_commit();
    {
      const double rx = pos[lane], ry = pos[32 + lane], rz = pos[64 + lane];
      // shells in snake order over the warps (a chunk's are sorted by cost)
      const double *rec = recs + (c & 1) * T.rec_max;
      for (int s0 = 0; s0 < ch.x; s0 += kWarps) {
        const int i = s0 + ((s0 / kWarps) & 1 ? kWarps - 1 - warp : warp);
        if (i >= ch.x) continue;
        const double head = rec[i];
        rows64_shell<kR64Walkers, kMode != R64_ALL>(rec + __double2hiint(head), __double2loint(head), rx, ry, rz, chi + lane);
      }
      // padding functions: their coefficients are zero, their values must be finite
      for (int k = (ch.z & 0xffff) + warp / 5; k < padded; k += kWarps / 5)
        chi[(T.lead + k) * kR64LdA + 32 * (warp % 5) + lane] = 0.0;
    }
    __syncthreads();
    const double *ap = chi + (T.lead + t) * kR64LdA + 16 * mtile + g;
    const double *bp = Cs + (c & 1) * kR64Chunk * kLdB + t * kLdB + 8 * NT * half + g;
    for (int k = 0; k < padded; k += 8) {
      const double a[4] = {ap[k * kR64LdA], ap[k * kR64LdA + 8], ap[(k + 4) * kR64LdA], ap[(k + 4) * kR64LdA + 8]};
#pragma unroll
      for (int j = 0; j < NT; j++)
        if (8 * (half * NT + j) < cols) dmma_m16n8k8(acc[j], a, bp[k * kLdB + 8 * j], bp[(k + 4) * kLdB + 8 * j]);
    }
    cp_async_wait<0>();
    __syncthreads();
  }
  // this warp's 16 rows: quantity mtile / 2 of walkers 16 (mtile % 2) ..
  const int q = mtile >> 1;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int w = 16 * (mtile & 1) + 8 * h + g;
    const int sw = __shfl_sync(QMCB_FULL_MASK, slot, w);
    if (w0 + w >= nw) continue;
#pragma unroll
    for (int j = 0; j < NT; j++) {
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int o = ((split * NH + half) * NT + j) * 8 + 2 * t + u;
        if (o >= n) continue;
        const double v = acc[j][2 * h + u];
        if (kMode == R64_ALL) {
          double *blk = state + (size_t)sw * L.stride;
          const int el = e - base;
          if (q == 0)
            blk[L.Dv[sp] + el * n + o] = v;
          else
            blk[L.D4[sp] + 4 * (o * n + el) + q - 1] = v;
        } else {
          rows[((size_t)(w0 + w) * 5 + q) * n + o] = v;
        }
      }
    }
  }
}

template <int kMode>
static const void *rows64_fn(int nt, int nh)
{
  const void *one[kR64WarpTiles] = {(const void *)k_rows64<kMode, 1, 1>, (const void *)k_rows64<kMode, 2, 1>,
                                    (const void *)k_rows64<kMode, 3, 1>, (const void *)k_rows64<kMode, 4, 1>};
  return nh == 1 ? one[nt - 1] : nt == 3 ? (const void *)k_rows64<kMode, 3, 2> : (const void *)k_rows64<kMode, 4, 2>;
}

cudaError_t rows64_limits()
{
  cudaError_t e = cudaSuccess;
  for (int nh = 1; nh <= 2; nh++)
    for (int nt = nh == 1 ? 1 : 3; nt <= kR64WarpTiles; nt++)
      for (const void *fn : {rows64_fn<R64_PROPOSE>(nt, nh), rows64_fn<R64_GIVEN>(nt, nh), rows64_fn<R64_ALL>(nt, nh)})
        if (e == cudaSuccess)
          e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   rows64_smem_bytes(nt, nh, kR64RecMax));
  return e;
}

cudaError_t rows64_launch(Rows64Mode mode, const DevSys &S, const Layout &L, const RunCfg &cfg, const Rows64 &T,
                          double *state, int cap, cudaStream_t st, const int *slots, int num, const int *d_num,
                          const double *R_in, const MoveArgs &mv, int sp, double *rows)
{
  const int n = sp ? S.nb : S.na;
  if (n == 0) return cudaSuccess;
  const int nt = rows64_tiles(n), nh = rows64_halves(n), splits = rows64_splits(n);
  const int tiles = (cap + kR64Walkers - 1) / kR64Walkers;
  const dim3 g = mode == R64_ALL ? dim3((unsigned)tiles * n * splits) : dim3(tiles, splits);
  const void *fn = mode == R64_ALL       ? rows64_fn<R64_ALL>(nt, nh)
                   : mode == R64_PROPOSE ? rows64_fn<R64_PROPOSE>(nt, nh)
                                         : rows64_fn<R64_GIVEN>(nt, nh);
  void *args[] = {(void *)&S,  (void *)&L,     (void *)&cfg,  (void *)&T,  &state, &slots, &num,
                  &d_num,      (void *)&R_in,  (void *)&mv,   &sp,         &rows};
  return cudaLaunchKernel(fn, g, dim3(32 * kR64MTiles * nh), args, rows64_smem_bytes(nt, nh, T.rec_max), st);
}

}  // namespace qmcb
