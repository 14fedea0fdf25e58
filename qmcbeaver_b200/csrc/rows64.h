// rows64.h -- tables, sizes and launch of the batched FP64 orbital rows (rows64.cu).
#pragma once

#include "kernels.cuh"

namespace qmcb {

constexpr int kR64Walkers = 32;              // walkers per CTA: one per lane
constexpr int kR64Rows = 5 * kR64Walkers;    // row = quantity * 32 + walker
constexpr int kR64MTiles = kR64Rows / 16;    // 16-row MMA tiles
constexpr int kR64Chunk = 48;                // basis functions per shared-memory chunk (multiple of 8)
// Functions per chunk of a handle's tables (nmax: the larger spin).  The
// sweep kernel (spins of up to 16) keeps two CTAs of 16 walkers per SM with 40,
// four with 24 (spins of up to 8).
__host__ __device__ constexpr int rows64_chunk(int nmax) { return nmax <= 8 ? 24 : nmax <= 16 ? 40 : kR64Chunk; }
// row pitches of the two shared arrays, 4 mod 8 doubles: the 16 lanes of a
// half-warp fragment load (4 k x 4 columns) then fall on 16 distinct banks
__host__ __device__ constexpr int rows64_pitch(int walkers) { return 5 * walkers + 4; }
constexpr int kR64LdA = rows64_pitch(kR64Walkers);
constexpr int kR64WarpTiles = 4;             // 8-orbital tiles per warp (accumulators: 4 x 4 doubles per lane)
constexpr int kR64TilesMax = 2 * kR64WarpTiles;  // 8-orbital tiles per CTA

constexpr int kR64RecMax = 1536;             // doubles of a chunk's shell records

// Rows before a chunk's first: the part of a shell that the chunk before it
// holds (a shell cut by a chunk's end is evaluated for both).  The sweep
// kernel's tables (spins of 9 to 16) need room behind a chunk's end too.
constexpr int kR64Lead = 5;

constexpr int kR64Any = 3;                   // shell kind: none of the complete s (0), p (1), d (2) shells

// Tables of the kernel.  A chunk holds at most kR64Chunk functions (padded
// with zero functions to a multiple of 8).  Its shell records: one double per
// shell (low word: first column | functions << 8 | kind << 16, high word:
// offset of its record in doubles), then the records: centre [3]; kinds s, p,
// d: exponents [3], coefficients [functions][3]; kind any: L and number of primitives in the two words of a double, exponents, and for
// every function its powers a | b << 8 | c << 16 | (the previous function's
// coefficients) << 24 in a low word and its coefficients.
struct Rows64 {
  int nchunk;
  int rec_max;          // doubles of the longest chunk's records
  int lead;             // rows before the chunks' first: 0, or kR64Lead where shells are cut
  const int4 *chunk;    // [nchunk + 1] shells, offset in rec, functions | padded functions << 16, first permuted function
  const double *rec;
  const double *ct[2];  // [permuted functions][ldb] coefficients, zero in the padding
  int ldb[2];
};

// An orbital range is cut into CTAs of at most kR64TilesMax 8-orbital tiles
// (each evaluates the basis again), a CTA's tiles over one or two warps per
// 16-row tile.
__host__ __device__ inline int rows64_splits(int n) { return ((n + 7) / 8 + kR64TilesMax - 1) / kR64TilesMax; }
__host__ __device__ inline int rows64_halves(int n) { return n > 8 * kR64WarpTiles ? 2 : 1; }
// 8-orbital tiles per warp
__host__ __device__ inline int rows64_tiles(int n)
{
  const int warps = rows64_splits(n) * rows64_halves(n);
  return n > 0 ? ((n + 7) / 8 + warps - 1) / warps : 1;
}
// coefficient row pitch in global memory: whole warp tiles
__host__ __device__ inline int rows64_ldb(int n) { return n > 0 ? 8 * rows64_splits(n) * rows64_halves(n) * rows64_tiles(n) : 8; }
__host__ __device__ inline int rows64_smem_bytes(int nt, int nh, int rec_max)
{
  return (int)sizeof(double) *
         (kR64Lead * kR64LdA + kR64Chunk * (kR64LdA + 2 * (8 * nt * nh + 4)) + 3 * kR64Walkers + 2 * rec_max);
}

enum Rows64Mode {
  R64_PROPOSE,  // the step's proposed position of electron mv.e
  R64_GIVEN,    // the caller's position of electron mv.e (R_in)
  R64_ALL       // every electron of a spin at its position (R_in, else the stored one)
};

// Raises the kernels' shared-memory limits on the current device.
cudaError_t rows64_limits();

// One launch for spin sp over list entries [0, num) (d_num: device count),
// grid sized for `cap` entries.
cudaError_t rows64_launch(Rows64Mode mode, const DevSys &S, const Layout &L, const RunCfg &cfg, const Rows64 &T,
                          double *state, int cap, cudaStream_t st, const int *slots, int num, const int *d_num,
                          const double *R_in, const MoveArgs &mv, int sp, double *rows);

}  // namespace qmcb
