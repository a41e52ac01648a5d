// The tile kernel of the incompatible-mode Hex8 (sbk_tile.cuh): its launch
// and its device scratch.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "sbk_params.h"

namespace sbk {

// An element's line search (sbk_tile_search.cuh).
struct TileSearch {
  double phi0, reach, s0, f0, s1, f1, step, best, best_step;
  int count, halvings, side, last_is_best;
};

// What the blocks of one launch keep in device memory: the tile counter, the
// list of the elements handed to the single kernel, and per block the
// geometry of its tile's points.
struct TileScratch {
  int32_t* counts;    // [0] the next tile, [1] elements handed on
  int32_t* fallback;  // ne
  double* geo;        // blocks x kTileGeo x points of a tile
  double* cond;       // chunk x tile_record: the elements' records
  int64_t chunk;      // elements of one launch
};

// Where an evaluation reads and writes (launch_elements' arguments).
struct TileArgs {
  int64_t ne;
  const double* coords;
  const int32_t* conn;
  const double* u;
  const double* state;
  const double* alpha_n;
  double* force;
  double* tangent;
  double* energy;
  double* trial;
  double* alpha_out;
  uint8_t* yield;
  int32_t* iterations;
  int32_t* code;
  int32_t* first_failure;
  int want_tangent;
  int batch;
  int elements;      // per tile
  int num_tiles;
  int64_t begin, end;  // the launch's elements
};

constexpr int kTileThreads = 256;
constexpr int kTileBlocksPerSm = 1;
constexpr int kTileMostElements = 32;
constexpr int kTileGeo = 19;  // per point: J^-1 9, det0 / det, U G^T 9

// A converged element's record for the condensation: per point, field-major
// over the element's points, then the element's own values.
constexpr int kCondH = 0;      // displacement gradient 9
constexpr int kCondM = 9;      // material block 36
constexpr int kCondS = 45;     // stress 6
constexpr int kCondW = 51;     // w det J
constexpr int kCondGeo = 52;   // J^-1 9, det0 / det
constexpr int kCondPoint = 62;
constexpr int kCondLu = 0;     // K_aa's factors 81, in pivot order
constexpr int kCondPiv = 81;   // reciprocal pivots 9
constexpr int kCondR = 90;     // r_a 9
constexpr int kCondJ0 = 99;    // J0^-1 9
constexpr int kCondPerm = 108; // 16 row + column of each pivot, 9
constexpr int kCondElement = 118;
__host__ __device__ inline size_t cond_record(int nq) { return (size_t)kCondPoint * nq + kCondElement; }

// A standard Hex8's: per point the fields above, then the mean dilatation's: P^T
// T 6, P^T C m / 3 6, P^T C^T m / 3 6, P^T m 6, m.C m / 9, tr T / 3.
constexpr int kStdSt = 62, kStdU1 = 68, kStdU2 = 74, kStdPv = 80, kStdMcm = 86, kStdTr = 87, kStdPoint = 88;
// Doubles an element of the scratch takes, for either element.
__host__ __device__ inline size_t tile_record(int nq) {
  return cond_record(nq) > (size_t)kStdPoint * nq ? cond_record(nq) : (size_t)kStdPoint * nq;
}

// Elements of a full tile: the points of a block's threads, at most
// kTileMostElements.
inline int tile_most(int nq) {
  const int n = kTileThreads / nq;
  return n < kTileMostElements ? n : kTileMostElements;
}
constexpr int kTileBlocks = 148 * kTileBlocksPerSm;  // resident at once

// Elements of one launch: at most what 1 GiB of records holds (a mesh of more
// takes several launches, so that the scratch does not grow with it), at
// least, where there is no memory for that many, a wave of full tiles.
inline int64_t tile_chunk_most(int nq) { return (int64_t)((size_t(1) << 30) / (tile_record(nq) * sizeof(double))); }
inline int64_t tile_chunk_least(int nq) { return (int64_t)kTileBlocks * tile_most(nq); }

// The condensation of the launch's elements whose code is 0: force and,
// wanted, K*.
int launch_condense(const Params& p, const TileArgs& a, const TileScratch& s, cudaStream_t stream);
// Their shape derivatives (24 an element) into out (sbk_vjp.cu).
int launch_vjp_tile(const Params& p, const TileArgs& a, const TileScratch& s, const double* lambda, double* out,
                    cudaStream_t stream);

// The standard Hex8 over the launch's elements (sbk_standard.cu).
int launch_standard(const Params& p, const TileArgs& a, const TileScratch& s, cudaStream_t stream);

// Bytes of one allocation that tile_scratch_carve splits, for ne elements of
// nq points in launches of chunk.
size_t tile_scratch_bytes(int64_t ne, int nq, int64_t chunk);
void tile_scratch_carve(void* base, int64_t ne, int nq, int64_t chunk, TileScratch& s);

// The tile kernel of the material's kind (one translation unit each).
int launch_tile_j2(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream);
int launch_tile_general0(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream);
int launch_tile_general1(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream);
int launch_tile_general2(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream);
int launch_tile_general4(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream);

}  // namespace sbk
