// K1 as one kernel over tiles of elements: the incompatible-mode Hex8 of any
// rule of up to 32 points.
//
// A block of eight warps, alone on its SM, takes a tile (up to 32 elements,
// 256 points) from start to finish and keeps everything its points and
// elements hand from stage to stage in shared memory (215 KB). Inside a tile
// the local iteration runs in rounds over the elements still iterating, each
// round a few short stages that the whole block walks together:
//
//   points    a thread a point: kinematics at the trial modes, spectral log
//             strain, the trial state; the points that yield are listed;
//   returns   a thread a listed point: the closest-point (or radial) return;
//   map       a thread a point: the logarithmic map of stress and tangent;
//   sums      four lanes a (mode, element): the mode's rows of K_aa, r_a and
//             the scale and floor sums, over the points, then by shuffles;
//   control   16 lanes an element: acceptance of the trial, the pivoted LU
//             of K_aa with a row per lane in registers, Newton's direction,
//             the definiteness test.
//
// Then the states and energies, a thread a point; what the condensation takes
// goes to condense_kernel (sbk_condense.cu). An element whose full Newton step
// is refused goes on in the same rounds, its line search's trial a trial like
// any other (sbk_tile_search.cuh); one whose K_aa is indefinite or whose line
// search fails goes to the single kernel (element_list_kernel).
//
// Why: as one launch per stage over the whole mesh (130 launches) the stages
// handed each other 207 KB per element through DRAM, and a mesh of a few
// thousand elements spent its time on launches. On chip an element moves 17
// KB, its state, K* and the condensation's record among them. What bounds a
// stage is the latency of one warp's chain (a stage takes nearly as long for
// one warp as for eight) and the fetch of its instructions: with two blocks
// of four warps per SM, each at its own place in 250 KB of code, the same
// tiles took 1.7 times as long once the blocks had drifted apart. Hence one
// block, and code that is in the kernel once.
//
// Measured (B200; an evaluation's element kernels before and after, all of
// them): 80 J2 elements 543 -> 88 us, 3,200 626 -> 157 us; Hill48 + two-term
// Chaboche: 2,304 elements of the 2 x 2 x 5 rule 3.39 -> 0.37 ms, 22,350 of
// them 32.4 -> 2.5 ms; 1,000,000 of the 2 x 2 x 2 rule 82.1 -> 45.5 ms.
//
// The algorithm and its constants are element_kernel's (sbk_element.cu),
// which cites the reference.
#pragma once

#include <cuda_runtime.h>

#include "sbk_element_math.cuh"
#include "sbk_smem.h"
#include "sbk_tile.h"
#include "sbk_tile_point.cuh"
#include "sbk_tile_search.cuh"

namespace sbk {

// A point's record in shared memory, field-major over the tile.
constexpr int kRecH = 0;       // displacement gradient 9
constexpr int kRecM = 9;       // material block 36
constexpr int kRecS = 45;      // stress 6
constexpr int kRecHmax = 51;   // largest |H|, then (map) its share of the floor, then the point's energy
constexpr int kRecW = 52;      // w det J
constexpr int kRecL = 53;      // axes 9, mu 3, first 6
constexpr int kRecStrain = 71;
constexpr int kRecWarm = 77;   // closest point 6, dl
constexpr int kRec = 84;

struct TileElement {
  double kc[81];    // K_aa of the last pass; of a converged element its LU
  double r[9], scale[9], flo[9];
  double alpha[9], at[9], jinv0[9], ipiv[9];
  double dir[9], r0[9];  // the direction of the trials, r_a where it starts
  double res;
  int64_t e;
  int fail;         // (stage << 16) | (point << 8) | code of the first failure
  int iterations;
  int stage;        // what the pending trial is (sbk_tile_search.cuh)
  TileSearch search;
  uint8_t rowp[12], colp[12];
};

inline size_t tile_points(int elements, int nq) { return static_cast<size_t>(elements) * nq | 1; }
inline size_t tile_smem(int elements, int nq) {
  const size_t np = tile_points(elements, nq);
  return kRec * np * sizeof(double) + elements * sizeof(TileElement) + (np + 3) / 4 * 4 * (sizeof(int16_t) + 1) + 64;
}

__device__ __forceinline__ double pick9(const double a[9], int k) {
  double v = a[0];
#pragma unroll
  for (int i = 1; i < 9; ++i) v = k == i ? a[i] : v;
  return v;
}
constexpr unsigned kAll = 0xffffffffu;
// Lanes of a (mode, element) in sums. Eight split 20 points into 3 each, and 12
// elements' 288 lanes into two passes of the block; four take 5 each in one:
// 2.09 -> 2.01 ms for 22,350 elements. At 8 points there is no difference.
constexpr int kSumLanes = 4;

template <int NT>
struct Tile {
  const Params& p;
  const TileArgs& a;
  double* rec;       // kRec x np
  TileElement* el;
  int16_t* yields;   // listed points of the round
  uint8_t* flag;     // per point: 0 elastic, 1 plastic, 2 loading window; bit 2: a closest point is kept
  double* geo;       // this block's kTileGeo x np
  int np, nq;

  __device__ __forceinline__ PointRecord point(int pt) const { return PointRecord{rec + pt, np}; }

  // Staging and reference geometry (set_up) of a point: J^-1, w det J,
  // det0 / det, U G^T; point 0 of the element also J0^-1.
  __device__ __forceinline__ void geometry(int k, int q) {
    TileElement& E = el[k];
    const int pt = k * nq + q;
    const double* X = rec + 48 * k;  // staged over the record's first fields
    PointGeometry G;
    if (!point_geometry(p, q, X, X + 24, G)) {
      atomicMin(&E.fail, SBK_EL_MESH_INVERTED);
      return;
    }
    if (q == 0)
#pragma unroll
      for (int i = 0; i < 9; ++i) E.jinv0[i] = G.j0i[i];
    rec[kRecW * np + pt] = G.w;
    double* g = geo + pt;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      g[i * np] = G.ji[i];
      g[(10 + i) * np] = G.du[i];
    }
    g[9 * np] = G.ratio;
  }

  // Kinematics, log strain and trial state of a point at its element's trial
  // modes; true when its return must run.
  __device__ __forceinline__ bool points(int k, int q, bool first) {
    TileElement& E = el[k];
    const int pt = k * nq + q;
    const PointRecord r = point(pt);
    const double* g = geo + pt;
    double h[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) h[i] = g[(10 + i) * np];
    const double ratio = g[9 * np];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const double f = ratio * (-2.0 * p.qp[q][m]);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double gt = f * E.jinv0[m * 3 + j];
#pragma unroll
        for (int i = 0; i < 3; ++i) h[i * 3 + j] += E.at[3 * m + i] * gt;
      }
    }
    double hmax = 0.0;
#pragma unroll
    for (int i = 0; i < 9; ++i) hmax = fmax(hmax, fabs(h[i]));
    double strain[6];
    LogKin L;
#pragma unroll
    for (int i = 0; i < 9; ++i) L.q[i] = first ? (i % 4 == 0 ? 1.0 : 0.0) : r.get(kRecL + i);
    const int code = point_strain(p, h, L, strain);
    if (code) {
      atomicMin(&E.fail, (1 << 16) | (q << 8) | code);
      return false;
    }
    if (p.kinematics == SBK_FINITE_LOGARITHMIC) {
#pragma unroll
      for (int i = 0; i < 9; ++i) r.put(kRecL + i, L.q[i]);
#pragma unroll
      for (int i = 0; i < 3; ++i) r.put(kRecL + 9 + i, L.mu[i]);
#pragma unroll
      for (int i = 0; i < 6; ++i) r.put(kRecL + 12 + i, L.first[i]);
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) r.put(kRecH + i, h[i]);
    r.put(kRecHmax, hmax);
#pragma unroll
    for (int i = 0; i < 6; ++i) r.put(kRecStrain + i, strain[i]);
    PointTrial<NT> T;
    point_trial<NT>(p, strain, a.state + E.e * nq + q, a.ne * nq, T);
    if (!isfinite(T.f)) {
      // The general return fails here, the radial one in its iteration.
      if (NT >= 0) {
        atomicMin(&E.fail, (2 << 16) | (q << 8) | kFailReturn);
        return false;
      }
    }
    if (point_elastic<NT>(p, T) && !point_window<NT>(p, T)) {
#pragma unroll
      for (int i = 0; i < 6; ++i) r.put(kRecS + i, T.s[i] + (i < 3 ? p.K * T.vol : 0.0));
      flag[pt] &= 4;
      return false;
    }
    return true;
  }

  __device__ __forceinline__ void returns(int pt) {
    const int k = pt / nq, q = pt - k * nq;
    TileElement& E = el[k];
    const PointRecord r = point(pt);
    double strain[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) strain[i] = r.get(kRecStrain + i);
    PointTrial<NT> T;
    point_trial<NT>(p, strain, a.state + E.e * nq + q, a.ne * nq, T);
    const int kept = flag[pt] & 4;
    const bool window = point_elastic<NT>(p, T);
    int code = 0;
    if constexpr (NT < 0) {
      if (window) return_window_radial(p, T, r, kRecS, kRecM);
      else code = return_radial(p, T, r, kRecS, kRecM, kRecWarm);
    } else {
      code = return_general<NT>(p, T, window, kept != 0, r, kRecS, kRecM, kRecWarm);
    }
    if (code) atomicMin(&E.fail, (2 << 16) | (q << 8) | code);
    else flag[pt] = window ? kept | 2 : 4 | 1;
  }

  __device__ __forceinline__ void map(int pt) {
    const PointRecord r = point(pt);
    const bool elastic = (flag[pt] & 3) == 0;
    double mmax = 0.0;  // the block's largest entry
    if (p.kinematics == SBK_FINITE_LOGARITHMIC) {
      LogKin L;
#pragma unroll
      for (int i = 0; i < 9; ++i) L.q[i] = r.get(kRecL + i);
#pragma unroll
      for (int i = 0; i < 3; ++i) L.mu[i] = r.get(kRecL + 9 + i);
#pragma unroll
      for (int i = 0; i < 6; ++i) L.first[i] = r.get(kRecL + 12 + i);
      mmax = spectral_map(p, L, elastic, r, kRecS, kRecM);
    } else {
      if (elastic) {
        double C[36];
        elastic_C(p, C);
#pragma unroll
        for (int i = 0; i < 36; ++i) r.put(kRecM + i, C[i]);
      }
#pragma unroll 6
      for (int i = 0; i < 36; ++i) mmax = fmax(mmax, fabs(r.get(kRecM + i)));
    }
    const double hmax = r.get(kRecHmax);
    r.put(kRecHmax, r.get(kRecW) * mmax * hmax * (1.0 + hmax));
  }

  // Rows 3m..3m+2 of K_aa and r_a, and the scale and floor sums of mode m:
  // lane l of kSumLanes sums the points l, l + kSumLanes, ..., the lanes
  // then by a reduce-scatter. V(k, l, n) as in vtensor.
  __device__ __forceinline__ void sums(int k, int m, int lane, bool live) {
    TileElement& E = el[k];
    double acc[36];
#pragma unroll
    for (int i = 0; i < 36; ++i) acc[i] = 0.0;
    const bool small = p.kinematics == SBK_SMALL_STRAIN;
#pragma unroll 1
    for (int q = live ? lane : nq; q < nq; q += kSumLanes) {
      const int pt = k * nq + q;
      const PointRecord r = point(pt);
      const double w = r.get(kRecW), ratio = geo[9 * np + pt];
      double g[3];
      {
        const double f = ratio * (-2.0 * p.qp[q][m]);
#pragma unroll
        for (int i = 0; i < 3; ++i) g[i] = f * E.jinv0[m * 3 + i];
      }
      double F[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) F[i] = (small ? 0.0 : r.get(kRecH + i)) + ((i % 4) == 0 ? 1.0 : 0.0);
      double W[3][6];
#pragma unroll
      for (int c = 0; c < 6; ++c) {
        double col[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) col[i] = r.get(kRecM + i * 6 + c);
        W[0][c] = w * (g[0] * col[0] + g[1] * col[3] + g[2] * col[5]);
        W[1][c] = w * (g[0] * col[3] + g[1] * col[1] + g[2] * col[4]);
        W[2][c] = w * (g[0] * col[5] + g[1] * col[4] + g[2] * col[2]);
      }
      double S[6], sg[3];
#pragma unroll
      for (int i = 0; i < 6; ++i) S[i] = r.get(kRecS + i);
      sg[0] = w * (g[0] * S[0] + g[1] * S[3] + g[2] * S[5]);
      sg[1] = w * (g[0] * S[3] + g[1] * S[1] + g[2] * S[4]);
      sg[2] = w * (g[0] * S[5] + g[1] * S[4] + g[2] * S[2]);
      double gn[3][3];
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        const double f = ratio * (-2.0 * p.qp[q][n]);
#pragma unroll
        for (int i = 0; i < 3; ++i) gn[n][i] = f * E.jinv0[n * 3 + i];
      }
      const double floor_w = r.get(kRecHmax);
#pragma unroll
      for (int kk = 0; kk < 3; ++kk) {
        double Uk[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) Uk[c] = F[kk * 3] * W[0][c] + F[kk * 3 + 1] * W[1][c] + F[kk * 3 + 2] * W[2][c];
#pragma unroll
        for (int l = 0; l < 3; ++l) {
          double v[3];
          v[0] = F[l * 3] * Uk[0] + F[l * 3 + 1] * Uk[3] + F[l * 3 + 2] * Uk[5];
          v[1] = F[l * 3] * Uk[3] + F[l * 3 + 1] * Uk[1] + F[l * 3 + 2] * Uk[4];
          v[2] = F[l * 3] * Uk[5] + F[l * 3 + 1] * Uk[4] + F[l * 3 + 2] * Uk[2];
          if (l == kk && !small)
#pragma unroll
            for (int i = 0; i < 3; ++i) v[i] += sg[i];
#pragma unroll
          for (int n = 0; n < 3; ++n)
            acc[kk * 9 + n * 3 + l] += v[0] * gn[n][0] + v[1] * gn[n][1] + v[2] * gn[n][2];
        }
        acc[27 + kk] += F[kk * 3] * sg[0] + F[kk * 3 + 1] * sg[1] + F[kk * 3 + 2] * sg[2];
        double b[6], s1 = 0.0, s2 = 0.0;
        b[0] = F[kk * 3] * g[0];
        b[1] = F[kk * 3 + 1] * g[1];
        b[2] = F[kk * 3 + 2] * g[2];
        b[3] = F[kk * 3] * g[1] + F[kk * 3 + 1] * g[0];
        b[4] = F[kk * 3 + 1] * g[2] + F[kk * 3 + 2] * g[1];
        b[5] = F[kk * 3 + 2] * g[0] + F[kk * 3] * g[2];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          s1 += fabs(b[i]) * fabs(S[i]);
          s2 += fabs(b[i]);
        }
        acc[30 + kk] += w * s1;
        acc[33 + kk] += floor_w * s2;
      }
    }
#pragma unroll
    for (int c = 0; c < 36 / kSumLanes; ++c) {
      double v[kSumLanes];
#pragma unroll
      for (int i = 0; i < kSumLanes; ++i) v[i] = acc[c * kSumLanes + i];
      const double y = reduce_scatter<kSumLanes>(v, lane, 0xffffffffu);
      const int i = c * kSumLanes + lane;
      if (!live) continue;
      if (i < 27) E.kc[(3 * m) * 9 + i] = y;
      else if (i < 30) E.r[3 * m + i - 27] = y;
      else if (i < 33) E.scale[3 * m + i - 30] = y;
      else if (i < 36) E.flo[3 * m + i - 33] = y;
    }
  }

  // What follows a pass of element k (solve_and_condense's loop,
  // IncompatibleModes.cpp:353-546), by 16 lanes, lane i < 9 the row i of
  // K_aa; both halves of a warp walk it together (a shuffle under a mask
  // known only at run time costs several instructions more). Returns 0: the
  // element goes on with the trial modes `at`; 1: converged; 2: handed to the
  // single kernel; -1: not live; else its failure << 8.
  __device__ __forceinline__ int control(int k, bool live, bool first, int lane) {
    TileElement& E = el[k];
    const int fail = live ? E.fail : 0;
    const bool row = lane < 9;
    const double r = row ? E.r[lane] : 0.0;
    double b = r, full = b * b, largest = fabs(b), scale = row ? fabs(E.scale[lane]) : 0.0,
           floors = row ? fabs(E.flo[lane]) : 0.0;
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) {
      full += __shfl_xor_sync(kAll, full, o, 16);
      largest = fmax(largest, __shfl_xor_sync(kAll, largest, o, 16));
      scale = fmax(scale, __shfl_xor_sync(kAll, scale, o, 16));
      floors = fmax(floors, __shfl_xor_sync(kAll, floors, o, 16));
    }
    full = sqrt(full);
    // fmax drops a NaN, the sum keeps it: a residual that is not a number
    // is no residual of 0 (the lanes beyond the rows), nor an infinite one
    // within an infinite bound.
    if (isnan(full)) largest = full;
    const bool finite = isfinite(largest);
    const double bound = kLocalTolerance * scale + kLocalRoundOff * floors;
    // The full Newton step, accepted when it reduces the residual enough or
    // meets the tolerance; everything else is search_after's.
    const bool evaluated = fail == 0x7fffffff;
    const bool met = finite && largest <= bound;
    const bool reduced = evaluated && finite && (full <= kFullStepReduction * E.res || met);
    int out = -1;
    bool go = live && (first ? evaluated : E.stage == kStageNewton && reduced);
    if (live && first && !evaluated) out = (fail & 0xff) << 8;
    const bool look = live && !first && !go;
    if (__any_sync(kAll, look)) {
      int got = 0;
      if (look && lane == 0)
        got = search_after(E, E.search, evaluated, full, met, full <= kFullStepReduction * E.res);
      got = __shfl_sync(kAll, got, 0, 16);
      __syncwarp();
      if (look) {
        go = got == 1;
        if (!go) out = got;
      }
    }
    if (!__any_sync(kAll, go)) return out;
    // K_aa = L U without exchanges, the right-hand side eliminated beside
    // it, and the symmetric part's L D L^T for the definiteness test (for a
    // symmetric K_aa its own pivots say it), a row per lane.
    const bool symmetric = p.symmetric != 0;
    double A[9], sym[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      A[j] = row ? E.kc[lane * 9 + j] : 0.0;
      sym[j] = row && !symmetric ? 0.5 * (A[j] + E.kc[j * 9 + lane]) : 0.0;
    }
    __syncwarp();
    if (go && row) E.alpha[lane] = E.at[lane];
    double myinv = 0.0, big_pivot = 0.0, small_pivot = 1.0e308;
    bool positive = true, pivots = true;  // a NaN is neither
#pragma unroll
    for (int s = 0; s < 9; ++s) {
      const double d = __shfl_sync(kAll, A[s], s, 16);
      const double inv = 1.0 / d;
      big_pivot = fmax(big_pivot, fabs(d));
      small_pivot = fmin(small_pivot, fabs(d));
      const double l = lane > s ? A[s] * inv : 0.0;
#pragma unroll
      for (int j = s + 1; j < 9; ++j) A[j] -= l * __shfl_sync(kAll, A[j], s, 16);
      b -= l * __shfl_sync(kAll, b, s, 16);
      if (lane > s) A[s] = l;
      if (lane == s) myinv = inv;
      pivots = pivots && d > 0.0;
    }
    if (symmetric) {
      positive = pivots;
    } else {
#pragma unroll
      for (int s = 0; s < 9; ++s) {
        const double d = __shfl_sync(kAll, sym[s], s, 16);
        positive = positive && d > 0.0;
        const double l = lane > s ? sym[s] * (1.0 / d) : 0.0;
#pragma unroll
        for (int j = s + 1; j < 9; ++j) sym[j] -= l * __shfl_sync(kAll, sym[j], s, 16);
      }
    }
    const bool converged = met || largest == 0.0;
    // Definite and far from singular: no pivot search is needed. Anything
    // else takes the complete pivoting and its rank test.
    const bool pivot = go && !(positive && pivots && small_pivot > 1.0e-10 * big_pivot);
    int status = -1;
    if (__any_sync(kAll, pivot)) status = pivoted(E, pivot, r, converged, lane);
    if (go) {
      if (pivot && status) {
        out = SBK_EL_LOCAL_SINGULAR << 8;
      } else if (converged) {
        if (!pivot && row) {
          E.rowp[lane] = E.colp[lane] = (uint8_t)lane;
          E.ipiv[lane] = myinv;
#pragma unroll
          for (int j = 0; j < 9; ++j) E.kc[lane * 9 + j] = A[j];
        }
        out = 1;
      } else {
        out = E.iterations == kMaxLocal || !finite ? SBK_EL_LOCAL_NO_CONVERGE << 8 : (positive ? 0 : 2);
      }
    }
    const bool on = go && out == 0;
    if (!__any_sync(kAll, on)) return out;
    double x = 0.0;
#pragma unroll
    for (int s = 8; s >= 0; --s) {
      const double xs = __shfl_sync(kAll, b * myinv, s, 16);
      if (lane == s) x = xs;
      b -= lane < s ? A[s] * xs : 0.0;
    }
    if (on) {
      if (row) {
        const double d = pivot ? E.dir[lane] : -x;  // pivoted leaves its own
        E.dir[lane] = d;
        E.r0[lane] = r;
        E.at[lane] = E.alpha[lane] + d;
      }
      if (lane == 0) {
        E.iterations += 1;
        E.res = full;
        E.stage = kStageNewton;
      }
    }
    return out;
  }

  // control's step with complete pivoting (Eigen's FullPivLU and its rank
  // test), both halves of the warp together; `need`: this one's outcome
  // counts. No row or column moves: a lane knows its row's step, a mask the
  // columns that are done. Returns 1 for a singular K_aa; else the factors
  // of a converged element are in its record, or minus the solution for r
  // in dir.
  __device__ __noinline__ static int pivoted(TileElement& E, bool need, double r, bool converged, int lane) {
    const bool row = lane < 9;
    double A[9], b = r;
#pragma unroll
    for (int j = 0; j < 9; ++j) A[j] = row ? E.kc[lane * 9 + j] : 0.0;
    __syncwarp();
    unsigned done = 0;
    uint64_t ro = 0, co = 0;
    int mystep = row ? 9 : -1;
    double myinv = 0.0, big_pivot = 0.0, small_pivot = 1.0e308;
    bool singular = false;
#pragma unroll 1
    for (int s = 0; s < 9; ++s) {
      double best = -1.0;
      int bj = 0;
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const double v = fabs(A[j]);
        if (!((done >> j) & 1u) && v > best) {
          best = v;
          bj = j;
        }
      }
      if (mystep != 9) best = -1.0;
      int at = bj * 16 + lane;
#pragma unroll
      for (int o = 8; o >= 1; o >>= 1) {
        const double ob = __shfl_xor_sync(kAll, best, o, 16);
        const int oi = __shfl_xor_sync(kAll, at, o, 16);
        if (ob > best || (ob == best && oi < at)) {
          best = ob;
          at = oi;
        }
      }
      singular = singular || !(best > 0.0);
      const int pr = at & 15, pc = at >> 4;
      big_pivot = fmax(big_pivot, best);
      small_pivot = fmin(small_pivot, best);
      const double l0 = pick9(A, pc);
      const double inv = 1.0 / __shfl_sync(kAll, l0, pr, 16);
      const bool below = mystep == 9 && lane != pr;
      const double l = below ? l0 * inv : 0.0;
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const double u = __shfl_sync(kAll, A[j], pr, 16);
        if (below && !((done >> j) & 1u)) A[j] = j == pc ? l : A[j] - l * u;
      }
      b -= l * __shfl_sync(kAll, b, pr, 16);
      if (lane == pr && mystep == 9) {
        mystep = s;
        myinv = inv;
      }
      done |= 1u << pc;
      ro |= (uint64_t)pr << (4 * s);
      co |= (uint64_t)pc << (4 * s);
    }
    double x = 0.0;
#pragma unroll 1
    for (int s = 8; s >= 0; --s) {
      const int pr = (int)((ro >> (4 * s)) & 15), pc = (int)((co >> (4 * s)) & 15);
      const double xs = __shfl_sync(kAll, b * myinv, pr, 16);
      if (lane == pc) x = xs;
      if (mystep < s) b -= pick9(A, pc) * xs;
    }
    if (singular || !(small_pivot > kEps * 9.0 * big_pivot)) return 1;
    if (!need || !row) return 0;
    if (converged) {
      E.rowp[lane] = (uint8_t)((ro >> (4 * lane)) & 15);
      E.colp[lane] = (uint8_t)((co >> (4 * lane)) & 15);
      E.ipiv[mystep] = myinv;
#pragma unroll 1
      for (int s = 0; s < 9; ++s) E.kc[mystep * 9 + s] = pick9(A, (int)((co >> (4 * s)) & 15));
    } else {
      E.dir[lane] = -x;
    }
    return 0;
  }
};

template <int NT>
__global__ void __launch_bounds__(kTileThreads, kTileBlocksPerSm)
    tile_kernel(const __grid_constant__ Params p, const __grid_constant__ TileArgs a,
                const __grid_constant__ TileScratch scratch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int tile_at, listed, count[2], finished;
  __shared__ int8_t active[2][kTileMostElements + 16], ended[kTileMostElements + 16];
  const int tid = threadIdx.x, lane = tid & 31;
  const int nq = p.nq, elements = a.elements;
  const int np = (elements * nq) | 1;
  Tile<NT> T{p, a, nullptr, nullptr, nullptr, nullptr, nullptr, np, nq};
  T.rec = reinterpret_cast<double*>(smem_raw);
  {
    T.el = reinterpret_cast<TileElement*>(T.rec + kRec * np);
    T.yields = reinterpret_cast<int16_t*>(T.el + elements);
    T.flag = reinterpret_cast<uint8_t*>(T.yields + (np + 3) / 4 * 4);
  }
  T.geo = scratch.geo + (size_t)blockIdx.x * kTileGeo * np;
  for (;;) {
    __syncthreads();
    if (tid == 0) tile_at = atomicAdd(scratch.counts, 1);
    __syncthreads();
    const int tile = tile_at;
    if (tile >= a.num_tiles) return;
    const int64_t e0 = a.begin + (int64_t)tile * elements;
    const int here = (int)(a.end - e0 < elements ? a.end - e0 : elements);
    // Staging: coordinates and displacements (over the record's first
    // fields), the modes, the element's counters.
#pragma unroll 1
    for (int k = tid; k < here; k += kTileThreads) {
      T.el[k].e = e0 + k;
      T.el[k].fail = 0x7fffffff;
      T.el[k].iterations = 0;
      active[0][k] = (int8_t)k;
    }
#pragma unroll 1
    for (int i = tid; i < here * nq; i += kTileThreads) T.flag[i] = 0;
    if (tid == 0) {
      count[0] = here;
      finished = 0;
    }
    __syncthreads();
#pragma unroll 1
    for (int i = tid; i < here * 8; i += kTileThreads) {
      const int k = i >> 3, n = i & 7;
      double* X = T.rec + 48 * k + 3 * n;
      if (a.batch) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          X[c] = a.coords[(e0 + k) * 24 + 3 * n + c];
          X[24 + c] = a.u[(e0 + k) * 24 + 3 * n + c];
        }
      } else {
        const int64_t node = a.conn[(e0 + k) * 8 + n];
        if (p.num_nodes > 0 && (node < 0 || node >= p.num_nodes)) {
          T.el[k].fail = SBK_EL_BAD_NODE;
        } else {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            X[c] = a.coords[node * 3 + c];
            X[24 + c] = a.u[node * 3 + c];
          }
        }
      }
    }
#pragma unroll 1
    for (int i = tid; i < here * 9; i += kTileThreads) {
      const double v = a.alpha_n ? a.alpha_n[e0 * 9 + i] : 0.0;
      T.el[i / 9].alpha[i % 9] = v;
      T.el[i / 9].at[i % 9] = v;
    }
    __syncthreads();
#pragma unroll 1
    for (int i = tid; i < here * nq; i += kTileThreads) {
      const int k = i / nq;
      if (T.el[k].fail != SBK_EL_BAD_NODE) T.geometry(k, i - k * nq);
    }
    __syncthreads();
    int side = 0;
#pragma unroll 1
    for (int round = 0;; ++round) {
      const int n = count[side];
      if (n == 0) break;
      if (tid == 0) {
        listed = 0;
        count[side ^ 1] = 0;
      }
      __syncthreads();
#pragma unroll 1
      for (int i = tid; i < n * nq; i += kTileThreads) {
        const int j = i / nq, k = active[side][j], q = i - j * nq;
        bool yields = false;
        const int fail = T.el[k].fail;
        if (fail != SBK_EL_BAD_NODE && fail != SBK_EL_MESH_INVERTED) yields = T.points(k, q, round == 0);
        if (yields) T.yields[atomicAdd(&listed, 1)] = (int16_t)(k * nq + q);
      }
      __syncthreads();
#pragma unroll 1
      for (int i = tid; i < listed; i += kTileThreads) T.returns(T.yields[i]);
      __syncthreads();
#pragma unroll 1
      for (int i = tid; i < n * nq; i += kTileThreads) {
        const int j = i / nq, k = active[side][j];
        if (T.el[k].fail == 0x7fffffff) T.map(k * nq + i - j * nq);
      }
      __syncthreads();
      // Four lanes a (mode, element).
#pragma unroll 1
      for (int i = tid; i - lane < n * 3 * kSumLanes; i += kTileThreads) {
        const bool task = i < n * 3 * kSumLanes;
        const int j = task ? i / kSumLanes : 0, m = j / n, k = active[side][j - m * n];
        T.sums(k, m, i % kSumLanes, task && T.el[k].fail == 0x7fffffff);
      }
      __syncthreads();
#pragma unroll 1
      for (int i = tid; i - lane < n * 16; i += kTileThreads) {
        const bool live = i < n * 16;
        const int k = active[side][live ? i >> 4 : 0];
        const int out = T.control(k, live, round == 0, i & 15);
        if ((i & 15) == 0 && live) {
          T.el[k].fail = 0x7fffffff;  // a trial's failure is its search's
          if (out == 0) {
            active[side ^ 1][atomicAdd(&count[side ^ 1], 1)] = (int8_t)k;
          } else if (out == 1) {
            ended[atomicAdd(&finished, 1)] = (int8_t)k;
          } else if (out == 2) {
            scratch.fallback[atomicAdd(scratch.counts + 1, 1)] = (int32_t)T.el[k].e;
            a.code[T.el[k].e] = -1;  // not the condensation's
          } else {
            a.code[T.el[k].e] = out >> 8;
            if (a.first_failure) atomicMin(a.first_failure, (int32_t)T.el[k].e);
          }
        }
      }
      side ^= 1;
      __syncthreads();
    }
    // The converged elements: states and energies, and what the condensation
    // takes (condense_kernel).
    const int n = finished;
    const size_t record = cond_record(nq);
#pragma unroll 1
    for (int i = tid; i < n * nq; i += kTileThreads) {
      const int j = i / nq, k = ended[j], q = i - j * nq, pt = k * nq + q;
      const PointRecord r = T.point(pt);
      const int64_t at = T.el[k].e * nq + q;
      double strain[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) strain[c] = r.get(kRecStrain + c);
      const int flag = T.flag[pt] & 3;
      const double energy =
          point_finish<NT>(p, strain, flag, r, kRecWarm, a.state + at, a.trial + at, a.ne * nq);
      a.yield[at] = flag == 1 ? 1 : 0;
      r.put(kRecHmax, r.get(kRecW) * energy);
      double* out = scratch.cond + (size_t)(T.el[k].e - a.begin) * record + q;
#pragma unroll 9
      for (int f = 0; f < 51; ++f) out[f * nq] = r.get(f);
      out[kCondW * nq] = r.get(kRecW);
#pragma unroll
      for (int f = 0; f < 10; ++f) out[(kCondGeo + f) * nq] = T.geo[f * np + pt];
    }
#pragma unroll 1
    for (int i = tid; i < n * kCondElement; i += kTileThreads) {
      const int j = i / kCondElement, f = i - j * kCondElement;
      const TileElement& E = T.el[ended[j]];
      double v = 0.0;
      if (f < kCondPiv) v = E.kc[f];
      else if (f < kCondR) v = E.ipiv[f - kCondPiv];
      else if (f < kCondJ0) v = E.r[f - kCondR];
      else if (f < kCondPerm) v = E.jinv0[f - kCondJ0];
      else if (f < kCondPerm + 9) v = (double)(E.rowp[f - kCondPerm] * 16 + E.colp[f - kCondPerm]);
      scratch.cond[(size_t)(E.e - a.begin) * record + kCondPoint * nq + f] = v;
    }
#pragma unroll 1
    for (int i = tid; i < n * 9; i += kTileThreads) {
      const TileElement& E = T.el[ended[i / 9]];
      a.alpha_out[E.e * 9 + i % 9] = E.alpha[i % 9];
    }
    __syncthreads();
#pragma unroll 1
    for (int j = tid; j < n; j += kTileThreads) {
      const int k = ended[j];
      const int64_t e = T.el[k].e;
      double en = 0.0;
      for (int q = 0; q < nq; ++q) en += T.rec[kRecHmax * np + k * nq + q];
      a.energy[e] = en;
      a.iterations[e] = T.el[k].iterations;
      a.code[e] = 0;
    }
  }
}

template <int NT>
int launch_tile(const Params& p, const TileArgs& a, const TileScratch& s, unsigned grid, cudaStream_t stream) {
  static SmemLimit limit;
  const cudaError_t err = limit.allow(tile_kernel<NT>);
  if (err != cudaSuccess) return (int)err;
  tile_kernel<NT><<<grid, kTileThreads, tile_smem(a.elements, p.nq), stream>>>(p, a, s);
  return (int)cudaGetLastError();
}

}  // namespace sbk
