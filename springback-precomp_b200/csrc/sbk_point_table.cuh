// What the tensor kernels (sbk_condense.cu, sbk_standard.cu) read of a point
// besides its record: the gradients of the nodes and modes and the rows of F,
// five entries (x y z x y) each, so that the cyclic components t, t + 1, t + 2
// of a lane are three consecutive ones; three zeros for a lane without any.
//
// Four lanes a point, eight points at once: two nodes, a mode and a row each,
// straight through. As one loop over the entries, with a division and four
// branches an entry, it was 7,600 to 9,400 of an element's 25,000 to 38,000
// cycles: the condensation of 1,000,000 elements took 11.4 ms, 9.2 so.
#pragma once

#include "sbk_params.h"
#include "sbk_tile.h"

namespace sbk {

__device__ __forceinline__ void put5(double* T, double x, double y, double z) {
  T[0] = T[3] = x;
  T[1] = T[4] = y;
  T[2] = z;
}

// Lane t (0 to 3) of the four of point q, whose record starts at R (stride
// nq): the nodes to T, the modes (MODES; j0 = J0^-1) behind them, F's rows to
// T + rows, the zeros to T + zero.
template <bool MODES>
__device__ __forceinline__ void point_table(const Params& p, int q, int t, bool small, const double* R, int nq,
                                            const double* j0, double* T, int rows, int zero) {
  double ji[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) ji[i] = R[(kCondGeo + i) * nq];
  const double qx = p.qp[q][0], qy = p.qp[q][1], qz = p.qp[q][2];
  const double sx = ((t + 1) >> 1) & 1 ? 1.0 : -1.0, sy = t >> 1 ? 1.0 : -1.0;
  const double fx = 1.0 + qx * sx, fy = 1.0 + qy * sy;
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // nodes t and t + 4
    const double sz = h ? 1.0 : -1.0, fz = 1.0 + qz * sz;
    const double a = sx * fy * fz, b = sy * fx * fz, c = sz * fx * fy;
    double g[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) g[i] = 0.125 * (a * ji[i] + b * ji[3 + i] + c * ji[6 + i]);
    put5(T + 5 * (t + 4 * h), g[0], g[1], g[2]);
  }
  if (t < 3) {
    if (MODES) {
      const double f = R[(kCondGeo + 9) * nq] * (-2.0 * (t == 0 ? qx : t == 1 ? qy : qz));
      put5(T + 5 * (8 + t), f * j0[3 * t], f * j0[3 * t + 1], f * j0[3 * t + 2]);
    }
    double F[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) F[i] = (small ? 0.0 : R[(kCondH + 3 * t + i) * nq]) + (i == t ? 1.0 : 0.0);
    put5(T + rows + 5 * t, F[0], F[1], F[2]);
  } else {
    T[zero] = T[zero + 1] = T[zero + 2] = 0.0;
  }
}

}  // namespace sbk
