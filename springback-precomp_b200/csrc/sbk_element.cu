// K1: the incompatible-mode Hex8 element on the GPU.
//
// One group of G lanes (G = 8 for rules of up to 8 points, 32 for rules of
// 9 to 32 points) evaluates one element; a 32-lane warp holds 32 / G
// elements, and a block of four warps 16 (or 4) elements by default.
// Lane q owns integration point q: its kinematics, its return map and its
// share of K_aa, which a shuffle reduce-scatter sums over the group into
// shared memory. The element-level work of the local Newton iteration - the
// 9x9 factorisations, the line searches and their fallbacks - runs on lane 0
// over shared memory, every decision being read back by the whole group, so
// the group's control flow stays uniform. After convergence the lanes split
// the condensation by element node: lane a forms the rows of node a of K_ua,
// K_uu and K* = K_uu - K_ua K_aa^-1 K_au.
//
// Algorithm: incompatible_elastoplastic_element and solve_and_condense
// (src/fem/IncompatibleModes.cpp:134-600, constants
// src/fem/IncompatibleModes.hpp:98-127). The local iteration, the line
// search on the directional residual, the shifted direction, the
// Levenberg-Marquardt fallback and the condensation follow it step for
// step; the arithmetic is reorganised for the GPU (the strain operator is
// never stored: B^T D B products are formed from F, D and the gradients).
#include <cuda_runtime.h>
#include <stdint.h>

#include "sbk_element.h"
#include "sbk_element_math.cuh"
#include "sbk_material.cuh"
#include "sbk_smem.h"
#include "sbk_tile.h"

namespace sbk {
namespace {

constexpr int kSlot = 54;  // per point: D 36 | S 6 | F 9 | w | energy | floor factor
constexpr int kSlotS = 36, kSlotF = 42, kSlotW = 51, kSlotE = 52, kSlotFl = 53;

__constant__ double kCorner[8][3] = {{-1, -1, -1}, {1, -1, -1}, {1, 1, -1}, {-1, 1, -1},
                                     {-1, -1, 1},  {1, -1, 1},  {1, 1, 1},  {-1, 1, 1}};

template <int G>
struct __align__(16) ElemShared {
  double X[24];
  double U[24];
  double jinv0[9];
  double geo[G][12];  // J^-1 (9), w det J, det0 / det
  double slot[G][kSlot];
  // K_aa (the reduced sums) during the local iteration; the coupling
  // C = K_aa^-1 K_au (9 x 24) in the condensation.
  double kc[216];
  double r[33];
  double scale[9];
  double flo[9];
  double energy;
  double alpha[9];
  double dir[9];
  double dir2[9];
  double r0[9];
  double lu[81];
  // Lane 0's scratch of the local iteration (K_aa at alpha, its symmetric
  // part, the Cholesky test, the shifted and Levenberg-Marquardt systems):
  // in shared memory, where its serial loads stay close.
  double work[243];
  double maxpivot;
  double dval[4];
  int rowp[9], colp[9], perm[9];
  int ival[4];
};

__device__ __forceinline__ void shape_grad(int a, double xi, double eta, double zeta, double dn[3]) {
  const double fx = 1.0 + xi * kCorner[a][0];
  const double fy = 1.0 + eta * kCorner[a][1];
  const double fz = 1.0 + zeta * kCorner[a][2];
  dn[0] = 0.125 * kCorner[a][0] * fy * fz;
  dn[1] = 0.125 * kCorner[a][1] * fx * fz;
  dn[2] = 0.125 * kCorner[a][2] * fx * fy;
}

// Voigt index of the tensor pair (i, j).
__device__ __forceinline__ int voigt(int i, int j) {
  if (i == j) return i;
  const int s = i + j;  // (0,1) -> 3, (1,2) -> 4, (0,2) -> 5
  return s == 1 ? 3 : (s == 3 ? 4 : 5);
}

// Column (3 m + k) of the Green-Lagrange strain variation for an
// augmented node with gradient g (3): b[c] for Voigt c = (i, j).
__device__ __forceinline__ void bcol(const double F[9], const double g[3], int k, double b[6]) {
  b[0] = F[k * 3 + 0] * g[0];
  b[1] = F[k * 3 + 1] * g[1];
  b[2] = F[k * 3 + 2] * g[2];
  b[3] = F[k * 3 + 0] * g[1] + F[k * 3 + 1] * g[0];
  b[4] = F[k * 3 + 1] * g[2] + F[k * 3 + 2] * g[1];
  b[5] = F[k * 3 + 2] * g[0] + F[k * 3 + 0] * g[2];
}

// V(k, l, n) = sum_{j,i,m} g(j) F(k,i) F(l,m) D[v(i,j)][v(m,n)] (D, or D^T
// with `transpose`), times w, plus the geometric w S(j,n) g(j) delta_kl:
// K_ab(k, l) = sum_n V(k, l, n) g_b(n) is the block of B_a^T D B_b + G_a^T S G_b.
__device__ __forceinline__ void vtensor(const double* slot, const double g[3], bool transpose, bool geometric,
                                     double V[27]) {
  const double w = slot[kSlotW];
  const double* D = slot;
  const double* F = slot + kSlotF;
  double W[3][6];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int r = voigt(i, j);
        s += g[j] * (transpose ? D[c * 6 + r] : D[r * 6 + c]);
      }
      W[i][c] = w * s;
    }
  double Uk[3][6];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int c = 0; c < 6; ++c) Uk[k][c] = F[k * 3 + 0] * W[0][c] + F[k * 3 + 1] * W[1][c] + F[k * 3 + 2] * W[2][c];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int l = 0; l < 3; ++l)
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        double s = 0.0;
#pragma unroll
        for (int m = 0; m < 3; ++m) s += F[l * 3 + m] * Uk[k][voigt(m, n)];
        V[(k * 3 + l) * 3 + n] = s;
      }
  if (geometric) {
    const double* S = slot + kSlotS;
    double sg[3];
#pragma unroll
    for (int n = 0; n < 3; ++n)
      sg[n] = w * (g[0] * S[voigt(0, n)] + g[1] * S[voigt(1, n)] + g[2] * S[voigt(2, n)]);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int n = 0; n < 3; ++n) V[(k * 3 + k) * 3 + n] += sg[n];
  }
}

// The per-element context of a group: s is the shared-memory record of its
// element.
template <int G>
struct Ctx {
  const Params* p;
  ElemShared<G>* s;
  int lane;
  unsigned mask;
  int64_t e;
  int64_t npts;  // ne * nq: the state stride
  const double* state;
  double* trial;
  uint8_t* yield;
  double* hu;    // this lane's U G^T (per-lane memory)
  double* warm;  // this lane's last converged closest point (general return)
  __device__ __forceinline__ void sync() const { __syncwarp(mask); }
};

// Mode gradients of point q: g~(i, m) = (det0 / det)(-2 xi_m) J0^-1(m, i).
template <int G>
__device__ __forceinline__ void mode_grads(const Ctx<G>& c, int q, double gt[9]) {
  const double ratio = c.s->geo[q][10];
  const double nat[3] = {c.p->qp[q][0], c.p->qp[q][1], c.p->qp[q][2]};
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const double f = ratio * (-2.0 * nat[m]);
#pragma unroll
    for (int i = 0; i < 3; ++i) gt[i * 3 + m] = f * c.s->jinv0[m * 3 + i];
  }
}
// Gradient of node a at point q: g(i) = sum_c dN_a/dxi_c J^-1(c, i).
template <int G>
__device__ __forceinline__ void node_grad(const Ctx<G>& c, int q, int a, double g[3]) {
  double dn[3];
  shape_grad(a, c.p->qp[q][0], c.p->qp[q][1], c.p->qp[q][2], dn);
  const double* ji = c.s->geo[q];
#pragma unroll
  for (int i = 0; i < 3; ++i) g[i] = dn[0] * ji[i] + dn[1] * ji[3 + i] + dn[2] * ji[6 + i];
}

// Reference geometry (set_up, IncompatibleModes.cpp:134-192). Returns 0 or
// SBK_EL_MESH_INVERTED (group-uniform).
template <int G>
__device__ int set_up(const Ctx<G>& c) {
  ElemShared<G>& s = *c.s;
  const Params& p = *c.p;
  // Centre Jacobian, every lane alike.
  double j0[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    double dn[3];
    shape_grad(a, 0.0, 0.0, 0.0, dn);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int k = 0; k < 3; ++k) j0[i * 3 + k] += s.X[3 * a + i] * dn[k];
  }
  const double det0 = det3(j0);
  int bad = !(det0 > 0.0);
  if (c.lane == 0 && !bad) inv3(j0, s.jinv0);
  const int q = c.lane;
  if (q < p.nq && !bad) {
    double jq[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    double dnq[8][3];
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      shape_grad(a, p.qp[q][0], p.qp[q][1], p.qp[q][2], dnq[a]);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) jq[i * 3 + k] += s.X[3 * a + i] * dnq[a][k];
    }
    const double det = det3(jq);
    if (!(det > 0.0)) {
      bad = 1;
    } else {
      double ji[9];
      inv3(jq, ji);
#pragma unroll
      for (int i = 0; i < 9; ++i) s.geo[q][i] = ji[i];
      s.geo[q][9] = p.qp[q][3] * det;
      s.geo[q][10] = det0 / det;
      // hu = U G^T with G(i, a) = sum_c dN_a/dxi_c J^-1(c, i).
      double hu[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        double g[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) g[i] = dnq[a][0] * ji[i] + dnq[a][1] * ji[3 + i] + dnq[a][2] * ji[6 + i];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) hu[i * 3 + j] += s.U[3 * a + i] * g[j];
      }
#pragma unroll
      for (int i = 0; i < 9; ++i) c.hu[i] = hu[i];
    }
  }
  bad = __any_sync(c.mask, bad);
  c.sync();
  return bad ? SBK_EL_MESH_INVERTED : 0;
}

// The kinematics of point q at the modes `at` (kinematics_at,
// IncompatibleModes.cpp:195-225): its mode gradients gt, F, the largest
// |H| entry, the strain the return takes and, under logarithmic
// kinematics, the spectral data L of the log strain. Returns 0, or a
// point-failure code (an inverted point, a log strain out of range).
template <int G>
__device__ __forceinline__ int point_kinematics(const Ctx<G>& c, int q, const double at[9], double gt[9],
                                                double F[9], double& hmax, double strain[6], LogKin& L) {
  const Params& p = *c.p;
  int code = 0;
  mode_grads(c, q, gt);
  double h[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double v = c.hu[i * 3 + j];
#pragma unroll
      for (int m = 0; m < 3; ++m) v += at[3 * m + i] * gt[j * 3 + m];
      h[i * 3 + j] = v;
    }
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    hmax = fmax(hmax, fabs(h[i]));
    F[i] = h[i] + ((i % 4) == 0 ? 1.0 : 0.0);
  }
  if (p.kinematics == SBK_SMALL_STRAIN) {
    strain[0] = h[0];
    strain[1] = h[4];
    strain[2] = h[8];
    strain[3] = h[1] + h[3];
    strain[4] = h[5] + h[7];
    strain[5] = h[6] + h[2];
#pragma unroll
    for (int i = 0; i < 9; ++i) F[i] = (i % 4) == 0 ? 1.0 : 0.0;
  } else {
    double E[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        E[i * 3 + j] = 0.5 * (h[i * 3 + j] + h[j * 3 + i] + h[0 * 3 + i] * h[0 * 3 + j] +
                              h[1 * 3 + i] * h[1 * 3 + j] + h[2 * 3 + i] * h[2 * 3 + j]);
    double green[6] = {E[0], E[4], E[8], 2.0 * E[1], 2.0 * E[5], 2.0 * E[6]};
    if (p.kinematics == SBK_FINITE) {
#pragma unroll
      for (int i = 0; i < 6; ++i) strain[i] = green[i];
    } else {
      if (!(det3(F) > 0.0)) {
        code = SBK_EL_INVERTED_POINT;
      } else {
        code = log_strain(green, L, strain);
      }
    }
  }
  return code;
}

// After the point's response r: its yield flag, the material block M and
// stress S in the strain measure of the element (the logarithmic map, or
// as they are), and its slot for the group sums.
template <int G>
__device__ __forceinline__ void point_slot(const Ctx<G>& c, int q, const Response& r, const LogKin& L,
                                           const double F[9], double w, double hmax, double M[36], double S[6]) {
  const Params& p = *c.p;
  ElemShared<G>& s = *c.s;
  c.yield[c.e * p.nq + q] = r.yielding ? 1 : 0;
#pragma unroll
  for (int i = 0; i < 36; ++i) M[i] = r.C[i];
  if (p.kinematics == SBK_FINITE_LOGARITHMIC) {
    log_transform(L, r.stress, S, M);
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) S[i] = r.stress[i];
  }
  double mmax = 0.0;
#pragma unroll
  for (int i = 0; i < 36; ++i) {
    s.slot[q][i] = M[i];
    mmax = fmax(mmax, fabs(M[i]));
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) s.slot[q][kSlotS + i] = S[i];
#pragma unroll
  for (int i = 0; i < 9; ++i) s.slot[q][kSlotF + i] = F[i];
  s.slot[q][kSlotW] = w;
  s.slot[q][kSlotE] = r.energy;
  s.slot[q][kSlotFl] = w * mmax * hmax * (1.0 + hmax);
}

// The group's side of a pass after every point has its slot (or failed):
// the first failure in the reference's order (the earliest stage, then the
// lowest point), else K_aa and the force, scale and floor sums. fail =
// (stage << 8) | q of this lane's failure (0: none), code its code.
template <int G>
__device__ __forceinline__ int pass_sums(const Ctx<G>& c, bool active, int fail, int code, const double gt[9],
                                         const double F[9], const double M[36], const double S[6], double w) {
  ElemShared<G>& s = *c.s;
  const Params& p = *c.p;
  const bool geometric = p.kinematics != SBK_SMALL_STRAIN;
  double kbuf[G];
  // The failure of the group: the first point of the earliest stage.
  int key = fail ? fail : 0x7fffffff;
#pragma unroll
  for (int o = G / 2; o >= 1; o >>= 1) key = min(key, __shfl_xor_sync(c.mask, key, o, G));
  if (key != 0x7fffffff) {
    const int owner = key & 0xff;
    const int out = __shfl_sync(c.mask, code, owner, G);
    c.sync();
    return out;
  }
  // K_aa: w ba^T (D ba) + geometric, streamed through the reduce-scatter in
  // chunks of G (row-major 9 x 9).
  const bool live = active;
  double Mba[6][9];
  if (live) {
#pragma unroll
    for (int col = 0; col < 9; ++col) {
      const int m = col / 3, k = col % 3;
      const double g[3] = {gt[0 * 3 + m], gt[1 * 3 + m], gt[2 * 3 + m]};
      double b[6];
      bcol(F, g, k, b);
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        double v = 0.0;
#pragma unroll
        for (int d = 0; d < 6; ++d) v += M[r * 6 + d] * b[d];
        Mba[r][col] = v;
      }
    }
  }
  double geo[9];
  if (live && geometric) {
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        double v = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) v += gt[i * 3 + m] * S[voigt(i, j)] * gt[j * 3 + n];
        geo[m * 3 + n] = w * v;
      }
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    double bi[6];
    if (live) {
      const int m = i / 3, k = i % 3;
      const double g[3] = {gt[0 * 3 + m], gt[1 * 3 + m], gt[2 * 3 + m]};
      bcol(F, g, k, bi);
    }
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      const int idx = i * 9 + j;
      double v = 0.0;
      if (live) {
#pragma unroll
        for (int r = 0; r < 6; ++r) v += bi[r] * Mba[r][j];
        v *= w;
        if (geometric && (i % 3) == (j % 3)) v += geo[(i / 3) * 3 + (j / 3)];
      }
      kbuf[idx % G] = v;
      if (idx % G == G - 1) {
        const double y = reduce_scatter<G>(kbuf, c.lane, c.mask);
        s.kc[(idx / G) * G + c.lane] = y;
      }
    }
  }
  if (81 % G != 0) {
#pragma unroll
    for (int i = 81 % G; i < G; ++i) kbuf[i] = 0.0;
    const double y = reduce_scatter<G>(kbuf, c.lane, c.mask);
    s.kc[(81 / G) * G + c.lane] = y;
  }
  c.sync();
  // The force and the scale sums over the points, in point order: lane a
  // (a < 8) node a, lanes 0-2 also mode a with its scale and floor sums,
  // lane 7 the energy.
  if (c.lane < 8) {
    const int a = c.lane;
    double ra[3] = {0, 0, 0}, rm[3] = {0, 0, 0}, sc[3] = {0, 0, 0}, fl[3] = {0, 0, 0}, en = 0.0;
    for (int qq = 0; qq < p.nq; ++qq) {
      const double* sl = s.slot[qq];
      const double* Fq = sl + kSlotF;
      const double* Sq = sl + kSlotS;
      const double wq = sl[kSlotW];
      double FS[9];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          FS[k * 3 + j] = Fq[k * 3 + 0] * Sq[voigt(0, j)] + Fq[k * 3 + 1] * Sq[voigt(1, j)] + Fq[k * 3 + 2] * Sq[voigt(2, j)];
      double g[3];
      node_grad(c, qq, a, g);
#pragma unroll
      for (int k = 0; k < 3; ++k) ra[k] += wq * (FS[k * 3 + 0] * g[0] + FS[k * 3 + 1] * g[1] + FS[k * 3 + 2] * g[2]);
      if (a < 3) {
        double gtq[9];
        mode_grads(c, qq, gtq);
        const double gm[3] = {gtq[0 * 3 + a], gtq[1 * 3 + a], gtq[2 * 3 + a]};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          rm[k] += wq * (FS[k * 3 + 0] * gm[0] + FS[k * 3 + 1] * gm[1] + FS[k * 3 + 2] * gm[2]);
          double b[6];
          bcol(Fq, gm, k, b);
          double s1 = 0.0, s2 = 0.0;
#pragma unroll
          for (int r = 0; r < 6; ++r) {
            s1 += fabs(b[r]) * fabs(Sq[r]);
            s2 += fabs(b[r]);
          }
          sc[k] += wq * s1;
          fl[k] += sl[kSlotFl] * s2;
        }
      }
      if (a == 7) en += wq * sl[kSlotE];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) s.r[3 * a + k] = ra[k];
    if (a < 3) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        s.r[24 + 3 * a + k] = rm[k];
        s.scale[3 * a + k] = sc[k];
        s.flo[3 * a + k] = fl[k];
      }
    }
    if (a == 7) s.energy = en;
  }
  c.sync();
  return 0;
}

// One pass (IncompatibleModes.cpp:337-342): the kinematics, the returns and
// the sums at `at` (9 values, identical in every lane). Returns 0 or the
// failure code of the first failing point in the reference's order.
template <int G>
__device__ __noinline__ int pass(const Ctx<G>& c, const double at[9]) {
  const Params& p = *c.p;
  const int q = c.lane;
  const bool active = q < p.nq;
  int fail = 0;  // (stage << 8) | q, stage 1 kinematics, 2 return
  int code = 0;
  double gt[9], F[9], hmax = 0.0;
  double M[36], S[6];
  double w = 0.0;
  if (active) {
    w = c.s->geo[q][9];
    double strain[6];
    LogKin L;
    code = point_kinematics(c, q, at, gt, F, hmax, strain, L);
    if (code) fail = (1 << 8) | q;
    if (!fail) {
      PointState st{c.state + c.e * p.nq + q, c.trial + c.e * p.nq + q, c.npts};
      Response r;
      code = p.general ? general_return(p, strain, st, r, c.warm) : radial_return(p, strain, st, r);
      if (code) {
        fail = (2 << 8) | q;
      } else {
        point_slot(c, q, r, L, F, w, hmax, M, S);
      }
    }
  }
  return pass_sums(c, active, fail, code, gt, F, M, S, w);
}

// ---- element-level helpers (lane 0, shared memory) ---------------------------

// FullPivLU of a (9x9 row-major) into lu by the lanes of a group together
// (every lane calls it); true if invertible (Eigen's rank test: every |U_ii|
// above 9 eps of the largest pivot). Step k: lane l scans and eliminates
// rows k + l, k + l + G, ...; the pivot is the group's largest |entry| of
// the remaining block, ties to the first in column-major order as Eigen's
// scan takes it; rows, then columns exchanged; the column below the pivot
// multiplied by its reciprocal, then the rank-one update. rowp / colp hold
// the transpositions.
template <int G>
__device__ __noinline__ bool fullpiv_lu9_rows(const Ctx<G>& c, const double* a, double* lu, int* rowp, int* colp,
                                              double* maxpivot_out) {
  const int lane = c.lane;
  _Pragma("unroll 1") for (int i = lane; i < 81; i += G) lu[i] = a[i];
  c.sync();
  double maxpivot = 0.0;
  int nonzero = 9;
  _Pragma("unroll 1") for (int k = 0; k < 9; ++k) {
    double big = -1.0;
    int bi = k, bj = k;
    _Pragma("unroll 1") for (int j = k; j < 9; ++j)
      _Pragma("unroll 1") for (int i = k + lane; i < 9; i += G) {
        const double v = fabs(lu[i * 9 + j]);
        if (v > big) {
          big = v;
          bi = i;
          bj = j;
        }
      }
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) {
      const double ob = __shfl_xor_sync(c.mask, big, o, G);
      const int oi = __shfl_xor_sync(c.mask, bi, o, G);
      const int oj = __shfl_xor_sync(c.mask, bj, o, G);
      if (ob > big || (ob == big && (oj < bj || (oj == bj && oi < bi)))) {
        big = ob;
        bi = oi;
        bj = oj;
      }
    }
    if (big == 0.0) {
      nonzero = k;
      break;
    }
    if (big > maxpivot) maxpivot = big;
    if (lane == 0) {
      rowp[k] = bi;
      colp[k] = bj;
    }
    if (bi != k)
      _Pragma("unroll 1") for (int j = lane; j < 9; j += G) {
        const double t = lu[k * 9 + j];
        lu[k * 9 + j] = lu[bi * 9 + j];
        lu[bi * 9 + j] = t;
      }
    c.sync();
    if (bj != k)
      _Pragma("unroll 1") for (int i = lane; i < 9; i += G) {
        const double t = lu[i * 9 + k];
        lu[i * 9 + k] = lu[i * 9 + bj];
        lu[i * 9 + bj] = t;
      }
    c.sync();
    const double inv = 1.0 / lu[k * 9 + k];
    _Pragma("unroll 1") for (int i = k + 1 + lane; i < 9; i += G) {
      const double l = lu[i * 9 + k] * inv;
      lu[i * 9 + k] = l;
      _Pragma("unroll 1") for (int j = k + 1; j < 9; ++j) lu[i * 9 + j] -= l * lu[k * 9 + j];
    }
    c.sync();
  }
  if (lane == 0) {
    _Pragma("unroll 1") for (int i = nonzero; i < 9; ++i) rowp[i] = colp[i] = i;
    *maxpivot_out = maxpivot;
  }
  bool mine = true;
  if (nonzero == 9) {
    const double threshold = kEps * 9.0 * maxpivot;
    _Pragma("unroll 1") for (int i = lane; i < 9; i += G) mine = mine && fabs(lu[i * 9 + i]) > threshold;
  }
  const bool ok = __all_sync(c.mask, mine) && nonzero == 9;
  c.sync();
  return ok;
}

// x = A^-1 b with the FullPivLU factors (any lane; b and x may alias).
__device__ __noinline__ void fullpiv_solve9(const double* lu, const int* rowp, const int* colp, const double* b,
                                            double* x) {
  double y[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) y[i] = b[i];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int pk = rowp[k];
#pragma unroll
    for (int i = k + 1; i < 9; ++i) {
      if (i == pk) {
        const double t = y[k];
        y[k] = y[i];
        y[i] = t;
      }
    }
  }
#pragma unroll
  for (int i = 1; i < 9; ++i)
#pragma unroll
    for (int j = 0; j < i; ++j) y[i] -= lu[i * 9 + j] * y[j];
#pragma unroll
  for (int i = 8; i >= 0; --i) {
#pragma unroll
    for (int j = i + 1; j < 9; ++j) y[i] -= lu[i * 9 + j] * y[j];
    y[i] /= lu[i * 9 + i];
  }
#pragma unroll
  for (int k = 8; k >= 0; --k) {
    const int pk = colp[k];
#pragma unroll
    for (int i = k + 1; i < 9; ++i) {
      if (i == pk) {
        const double t = y[k];
        y[k] = y[i];
        y[i] = t;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) x[i] = y[i];
}

// x = A^-T b with the FullPivLU factors of A (P A Q = L U, so
// A^-T = P^T L^-T U^-T Q^T): the column transpositions in order, U^T
// forward, L^T backward (unit diagonal), the row transpositions in reverse.
__device__ __noinline__ void fullpiv_solve9_t(const double* lu, const int* rowp, const int* colp, const double* b,
                                                 double* x) {
  double y[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) y[i] = b[i];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int pk = colp[k];
#pragma unroll
    for (int i = k + 1; i < 9; ++i) {
      if (i == pk) {
        const double t = y[k];
        y[k] = y[i];
        y[i] = t;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) {
#pragma unroll
    for (int j = 0; j < i; ++j) y[i] -= lu[j * 9 + i] * y[j];
    y[i] /= lu[i * 9 + i];
  }
#pragma unroll
  for (int i = 8; i >= 0; --i)
#pragma unroll
    for (int j = i + 1; j < 9; ++j) y[i] -= lu[j * 9 + i] * y[j];
#pragma unroll
  for (int k = 8; k >= 0; --k) {
    const int pk = rowp[k];
#pragma unroll
    for (int i = k + 1; i < 9; ++i) {
      if (i == pk) {
        const double t = y[k];
        y[k] = y[i];
        y[i] = t;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) x[i] = y[i];
}

// llt9 by the lanes of a group together (every lane calls it): step k's
// diagonal by the lane of row k, then the rows below in parallel, each entry
// the same dot product in the same order - the same factor and the same
// answer.
template <int G>
__device__ __noinline__ bool llt9_rows(const Ctx<G>& c, double* a) {
  const int lane = c.lane;
  _Pragma("unroll 1") for (int k = 0; k < 9; ++k) {
    int bad = 0;
    if (lane == k % G) {
      double x = a[k * 9 + k];
      _Pragma("unroll 1") for (int j = 0; j < k; ++j) x -= a[k * 9 + j] * a[k * 9 + j];
      if (x <= 0.0) {
        bad = 1;
      } else {
        a[k * 9 + k] = sqrt(x);
      }
    }
    bad = __shfl_sync(c.mask, bad, k % G, G);
    c.sync();
    if (bad) return false;
    _Pragma("unroll 1") for (int i = k + 1 + ((lane - (k + 1)) % G + G) % G; i < 9; i += G) {
      double v = a[i * 9 + k];
      _Pragma("unroll 1") for (int j = 0; j < k; ++j) v -= a[i * 9 + j] * a[k * 9 + j];
      a[i * 9 + k] = v / a[k * 9 + k];
    }
    c.sync();
  }
  return true;
}

// ---- the local iteration -------------------------------------------------------

template <int G>
struct Local {
  const Ctx<G>& c;
  ElemShared<G>& s;
  double residual;
  int iterations;
  __device__ Local(const Ctx<G>& cc) : c(cc), s(*cc.s), residual(0.0), iterations(0) {}

  __device__ double rnorm() const {
    double v = 0.0;
#pragma unroll
    for (int i = 0; i < 9; ++i) v += s.r[24 + i] * s.r[24 + i];
    return sqrt(v);
  }
  __device__ double rinf() const {
    double v = fabs(s.r[24]);
#pragma unroll
    for (int i = 1; i < 9; ++i) v = fmax(v, fabs(s.r[24 + i]));
    return v;
  }
  __device__ double vmax(const double* v) const {
    double m = fabs(v[0]);
#pragma unroll
    for (int i = 1; i < 9; ++i) m = fmax(m, fabs(v[i]));
    return m;
  }
  __device__ double ddot(const double* a, const double* b) const {
    double v = 0.0;
#pragma unroll
    for (int i = 0; i < 9; ++i) v += a[i] * b[i];
    return v;
  }
  // A pass at alpha + t d; true if every point evaluated.
  __device__ bool try_at(const double* d, double t) {
    double at[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) at[i] = s.alpha[i] + t * d[i];
    return pass<G>(c, at) == 0;
  }
  __device__ void advance(const double* d, double t) {
    c.sync();
    if (c.lane == 0)
#pragma unroll
      for (int i = 0; i < 9; ++i) s.alpha[i] += t * d[i];
    c.sync();
  }

  // search_norm (IncompatibleModes.cpp:359-383).
  __device__ __noinline__ bool search_norm(const double* d, double reach) {
    double best_step = 0.0, best = residual;
    bool last_is_best = false;
    double trial_step = reach;
    for (int search = 0; search < kMaxLineSearch; ++search, trial_step *= 0.5) {
      if (!try_at(d, trial_step)) {
        last_is_best = false;
        continue;
      }
      const double n = rnorm();
      last_is_best = n < best;
      if (last_is_best) {
        best = n;
        best_step = trial_step;
      }
      if (n <= kFullStepReduction * residual) break;
    }
    if (best_step == 0.0) return false;
    if (!last_is_best && !try_at(d, best_step)) return false;
    advance(d, best_step);
    residual = best;
    return true;
  }

  // line_search (IncompatibleModes.cpp:398-456).
  __device__ __noinline__ bool line_search(const double* d) {
    const double phi0 = ddot(d, s.r0);
    double reach = 1.0;
    bool evaluated = try_at(d, 1.0);
    for (int halving = 0; !evaluated && halving < kMaxLineSearch; ++halving) {
      reach *= 0.5;
      evaluated = try_at(d, reach);
    }
    if (!evaluated) return false;
    const double full = rnorm();
    if (full <= kFullStepReduction * residual ||
        rinf() <= kLocalTolerance * vmax(s.scale) + kLocalRoundOff * vmax(s.flo)) {
      advance(d, reach);
      residual = full;
      return true;
    }
    const double phi1 = ddot(d, s.r + 24);
    if (!(phi0 < 0.0) || !(phi1 > 0.0) || !isfinite(phi1)) return search_norm(d, 0.5 * reach);
    double s0 = 0.0, f0 = phi0, s1 = reach, f1 = phi1, step = reach;
    int side = 0;
    for (int search = 0; search < kMaxLineSearch; ++search) {
      const double width = s1 - s0;
      step = fmin(fmax((s0 * f1 - s1 * f0) / (f1 - f0), s0 + 0.1 * width), s1 - 0.1 * width);
      evaluated = try_at(d, step);
      const double f = evaluated ? ddot(d, s.r + 24) : __longlong_as_double(0x7ff0000000000000LL);
      if (evaluated && fabs(f) <= kLineSearchRatio * fabs(phi0)) break;
      if (!evaluated || f > 0.0) {
        s1 = step;
        f1 = evaluated ? f : 0.5 * f1;
        if (side == 1) f0 *= 0.5;
        side = 1;
      } else {
        s0 = step;
        f0 = f;
        if (side == -1) f1 *= 0.5;
        side = -1;
      }
    }
    if (!evaluated) {
      if (s0 == 0.0) return false;
      step = s0;
      if (!try_at(d, step)) return false;
    }
    advance(d, step);
    residual = rnorm();
    return true;
  }

  // solve_and_condense's loop (IncompatibleModes.cpp:353-546). Returns 0 or
  // a failure code; on success the last pass is at s.alpha and s.lu holds
  // the factors of its K_aa.
  __device__ __noinline__ int run() {
    // K_aa at alpha (k0), its symmetric part and scratch: lane 0's alone.
    double* work = s.work;
    {
      double at[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) at[i] = s.alpha[i];
      const int code = pass<G>(c, at);
      if (code) return code;
    }
    residual = rnorm();
    for (;;) {
      const double largest = rinf();
      const double scale = vmax(s.scale);
      const double floor_ = kLocalRoundOff * vmax(s.flo);
      const bool invertible = fullpiv_lu9_rows<G>(c, s.kc, s.lu, s.rowp, s.colp, &s.maxpivot);
      // k0 and r0 copies (the trial passes overwrite the sums).
      for (int i = c.lane; i < 81; i += G) work[i] = s.kc[i];
      for (int i = c.lane; i < 9; i += G) s.r0[i] = s.r[24 + i];
      c.sync();
      if (!invertible) return SBK_EL_LOCAL_SINGULAR;
      if (largest <= kLocalTolerance * scale + floor_ || largest == 0.0) return 0;
      if (iterations == kMaxLocal || !isfinite(largest)) return SBK_EL_LOCAL_NO_CONVERGE;
      ++iterations;
      // Newton's direction and the Cholesky test of the symmetric part.
      for (int idx = c.lane; idx < 81; idx += G) {
        const int i = idx / 9, j = idx % 9;
        const double v = 0.5 * (work[i * 9 + j] + work[j * 9 + i]);
        work[81 + idx] = v;   // sym
        work[162 + idx] = v;  // chol
      }
      c.sync();
      if (c.lane == 0) {
        double nw[9];
        fullpiv_solve9(s.lu, s.rowp, s.colp, s.r0, nw);
        for (int i = 0; i < 9; ++i) s.dir[i] = -nw[i];
      }
      const bool positive = llt9_rows<G>(c, work + 162);
      c.sync();
      if (positive) {
        if (line_search(s.dir)) continue;
      } else {
        if (try_at(s.dir, 1.0)) {
          const double full = rnorm();
          if (full <= kFullStepReduction * residual) {
            advance(s.dir, 1.0);
            residual = full;
            continue;
          }
        }
        if (c.lane == 0) {
          // The shifted direction (K_aa + mu I) d = -r_alpha.
          double* sym = work + 81;
          double* tmp = work + 162;
          for (int i = 0; i < 81; ++i) tmp[i] = sym[i];
          double lo, top;
          sym_eig9(tmp, &lo, &top);
          const double mu = kLocalShift * top - lo;
          for (int i = 0; i < 81; ++i) tmp[i] = work[i];
          for (int i = 0; i < 9; ++i) tmp[i * 9 + i] += mu;
          double x[9];
          plu9_solve(tmp, s.perm, s.r0, x);
          for (int i = 0; i < 9; ++i) s.dir2[i] = -x[i];
        }
        c.sync();
        if (line_search(s.dir2)) continue;
        if (search_norm(s.dir, 0.5)) continue;
      }
      // Levenberg-Marquardt (IncompatibleModes.cpp:522-545).
      double mu = 0.0;
      if (c.lane == 0) {
        double* normal = work + 81;
        for (int i = 0; i < 9; ++i)
          for (int j = 0; j < 9; ++j) {
            double v = 0.0;
            for (int k = 0; k < 9; ++k) v += work[k * 9 + i] * work[k * 9 + j];
            normal[i * 9 + j] = v;
          }
        double dmax = normal[0];
        for (int i = 1; i < 9; ++i) dmax = fmax(dmax, normal[i * 9 + i]);
        s.dval[0] = kLocalMarquardt * dmax;
      }
      c.sync();
      mu = s.dval[0];
      bool moved = false;
      for (int search = 0; search < kMaxLineSearch && !moved; ++search, mu *= 10.0) {
        c.sync();
        if (c.lane == 0) {
          double* normal = work + 81;
          double* a = work + 162;
          for (int i = 0; i < 81; ++i) a[i] = normal[i];
          for (int i = 0; i < 9; ++i) a[i * 9 + i] += mu;
          double grad[9];
          for (int i = 0; i < 9; ++i) {
            double v = 0.0;
            for (int j = 0; j < 9; ++j) v += work[j * 9 + i] * s.r0[j];
            grad[i] = v;
          }
          const bool ok = llt9(a);
          s.ival[2] = ok ? 1 : 0;
          if (ok) {
            double x[9];
            llt9_solve(a, grad, x);
            for (int i = 0; i < 9; ++i) s.dir2[i] = -x[i];
          }
        }
        c.sync();
        if (!s.ival[2]) continue;
        if (!try_at(s.dir2, 1.0)) continue;
        const double n = rnorm();
        if (n < residual) {
          advance(s.dir2, 1.0);
          residual = n;
          moved = true;
        }
      }
      if (!moved) return SBK_EL_LOCAL_NO_DESCENT;
    }
  }
};

// ---- the condensation ---------------------------------------------------------

// The condensation (IncompatibleModes.cpp:549-561) after the local
// iteration converged: lane a (a < 8) forms the rows of node a of K_ua (and
// K_au), the coupling C = K_aa^-1 K_au, f* = f_u - K_ua K_aa^-1 r_a and, with
// the tangent, K* = K_uu - K_ua C, symmetrised for a symmetric tangent. Reads
// the group's shared record: the last pass's slots and sums (slot, r), the
// factors of its K_aa (lu, rowp, colp) and the geometry; kc is overwritten.
template <int G>
__device__ __forceinline__ void condense(const Ctx<G>& c, int want_tangent, double* __restrict__ force,
                                         double* __restrict__ tangent) {
  const Params& p = *c.p;
  ElemShared<G>& s = *c.s;
  const int lane = c.lane;
  const int64_t e = c.e;
  const bool sym = p.symmetric != 0;
  const bool geometric = p.kinematics != SBK_SMALL_STRAIN;
  const int nq = p.nq;
  // K_ua rows of node a (and K_au columns for a non-symmetric tangent).
  double kua[3][9], kau[3][9];
  if (lane < 8) {
    const int a = lane;
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int j = 0; j < 9; ++j) kua[k][j] = kau[k][j] = 0.0;
    for (int q = 0; q < nq; ++q) {
      double g[3], gt[9], V[27];
      node_grad(c, q, a, g);
      mode_grads(c, q, gt);
      vtensor(s.slot[q], g, false, geometric, V);
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int l = 0; l < 3; ++l)
            kua[k][3 * m + l] += V[(k * 3 + l) * 3 + 0] * gt[0 * 3 + m] + V[(k * 3 + l) * 3 + 1] * gt[1 * 3 + m] +
                                 V[(k * 3 + l) * 3 + 2] * gt[2 * 3 + m];
      if (!sym) {
        vtensor(s.slot[q], g, true, geometric, V);
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int l = 0; l < 3; ++l)
              kau[k][3 * m + l] += V[(k * 3 + l) * 3 + 0] * gt[0 * 3 + m] + V[(k * 3 + l) * 3 + 1] * gt[1 * 3 + m] +
                                   V[(k * 3 + l) * 3 + 2] * gt[2 * 3 + m];
      }
    }
    // The coupling C = K_aa^-1 K_au, columns of node a, into shared memory
    // (K_au(3m+l, 3a+k) = kau[k][3m+l], or kua[k][3m+l] when symmetric).
    double* C = s.kc;  // 9 x 24, column-major by DOF: C[col * 9 + i]
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double b[9];
#pragma unroll
      for (int j = 0; j < 9; ++j) b[j] = sym ? kua[k][j] : kau[k][j];
      double x[9];
      fullpiv_solve9(s.lu, s.rowp, s.colp, b, x);
#pragma unroll
      for (int j = 0; j < 9; ++j) C[(3 * a + k) * 9 + j] = x[j];
    }
  }
  c.sync();
  if (lane < 8) {
    const int a = lane;
    // f* = f_u - K_ua K_aa^-1 r_alpha.
    double corr[9];
    fullpiv_solve9(s.lu, s.rowp, s.colp, s.r + 24, corr);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double v = 0.0;
#pragma unroll
      for (int j = 0; j < 9; ++j) v += kua[k][j] * corr[j];
      force[e * 24 + 3 * a + k] = s.r[3 * a + k] - v;
    }
    if (want_tangent) {
      const double* C = s.kc;
#pragma unroll
      for (int chunk = 0; chunk < 2; ++chunk) {
        double acc[4][9];
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
          for (int i = 0; i < 9; ++i) acc[b][i] = 0.0;
        for (int q = 0; q < nq; ++q) {
          double g[3], V[27];
          node_grad(c, q, a, g);
          vtensor(s.slot[q], g, false, geometric, V);
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            double gb[3];
            node_grad(c, q, chunk * 4 + b, gb);
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
              for (int l = 0; l < 3; ++l)
                acc[b][k * 3 + l] += V[(k * 3 + l) * 3 + 0] * gb[0] + V[(k * 3 + l) * 3 + 1] * gb[1] +
                                     V[(k * 3 + l) * 3 + 2] * gb[2];
          }
        }
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int bb = chunk * 4 + b;
          double* out = tangent + e * 576 + (8 * a + bb) * 9;
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int l = 0; l < 3; ++l) {
              double v = acc[b][k * 3 + l];
#pragma unroll
              for (int m = 0; m < 9; ++m) v -= kua[k][m] * C[(3 * bb + l) * 9 + m];
              out[k * 3 + l] = v;
            }
        }
      }
    }
  }
  if (want_tangent && sym) {
    // K* = (K* + K*^T) / 2: the unordered pair {(i, j), (j, i)} by the lane
    // that owns row min(i, j).
    __threadfence_block();
    c.sync();
    if (lane < 8) {
      double* Ke = tangent + e * 576;
      auto at = [&](int i, int j) -> double* { return Ke + (8 * (i / 3) + j / 3) * 9 + 3 * (i % 3) + (j % 3); };
      for (int k = 0; k < 3; ++k) {
        const int i = 3 * lane + k;
        for (int j = i + 1; j < 24; ++j) {
          double* x = at(i, j);
          double* y = at(j, i);
          const double v = 0.5 * (*x + *y);
          *x = v;
          *y = v;
        }
      }
    }
  }
}


// One element of the single kernel, start to finish: staging, set_up, the
// local iteration (Local::run), the condensation and the outputs.
template <int G>
__device__ __forceinline__ void element_body(const Params& p, int64_t ne, bool batch, int64_t e, ElemShared<G>* sh,
                                             int lane, unsigned mask, const double* __restrict__ coords,
                                             const int32_t* __restrict__ conn, const double* __restrict__ u,
                                             const double* __restrict__ state, const double* __restrict__ alpha_n,
                                             int want_tangent, double* __restrict__ force,
                                             double* __restrict__ tangent, double* __restrict__ energy,
                                             double* __restrict__ trial, double* __restrict__ alpha_out,
                                             uint8_t* __restrict__ yield, int32_t* __restrict__ iterations,
                                             int32_t* __restrict__ code, int32_t* __restrict__ first_failure) {
  double hu_lane[9];
  double warm_lane[8];
  warm_lane[7] = 0.0;  // no closest point yet
  Ctx<G> c{&p, sh, lane, mask, e, ne * p.nq, state, trial, yield, hu_lane, warm_lane};
  ElemShared<G>& s = *sh;
  // Stage the element's coordinates and displacements (lane a: node a); a
  // node index out of range fails the element before anything is read.
  int bad_node = 0;
  if (lane < 8) {
    if (batch) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        s.X[3 * lane + k] = coords[e * 24 + 3 * lane + k];
        s.U[3 * lane + k] = u[e * 24 + 3 * lane + k];
      }
    } else {
      const int64_t node = conn[e * 8 + lane];
      if (p.num_nodes > 0 && (node < 0 || node >= p.num_nodes)) {
        bad_node = 1;
      } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          s.X[3 * lane + k] = coords[node * 3 + k];
          s.U[3 * lane + k] = u[node * 3 + k];
        }
      }
    }
  }
  if (__any_sync(mask, bad_node)) {
    if (lane == 0) {
      code[e] = SBK_EL_BAD_NODE;
      if (first_failure) atomicMin(first_failure, (int32_t)e);
    }
    return;
  }
  for (int i = lane; i < 9; i += G) s.alpha[i] = alpha_n ? alpha_n[e * 9 + i] : 0.0;
  c.sync();
  int status = set_up<G>(c);
  Local<G> loc(c);
  if (!status) status = loc.run();
  if (status) {
    if (lane == 0) {
      code[e] = status;
      if (first_failure) atomicMin(first_failure, (int32_t)e);
    }
    return;
  }
  condense<G>(c, want_tangent, force, tangent);
  if (lane == 0) {
    energy[e] = s.energy;
    iterations[e] = loc.iterations;
    code[e] = 0;
  }
  for (int i = lane; i < 9; i += G) alpha_out[e * 9 + i] = s.alpha[i];
}

template <int G>
__global__ void __launch_bounds__(256) element_kernel(const __grid_constant__ Params p, int64_t ne, bool batch,
                                                      const double* __restrict__ coords,
                                                      const int32_t* __restrict__ conn, const double* __restrict__ u,
                                                      const double* __restrict__ state,
                                                      const double* __restrict__ alpha_n, int want_tangent,
                                                      double* __restrict__ force, double* __restrict__ tangent,
                                                      double* __restrict__ energy, double* __restrict__ trial,
                                                      double* __restrict__ alpha_out, uint8_t* __restrict__ yield,
                                                      int32_t* __restrict__ iterations, int32_t* __restrict__ code,
                                                      int32_t* __restrict__ first_failure,
                                                      const int32_t* __restrict__ order) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int epb = blockDim.x / G;
  const int slot_in_block = threadIdx.x / G;
  const int lane = threadIdx.x % G;
  const int64_t slot = (int64_t)blockIdx.x * epb + slot_in_block;
  ElemShared<G>* sh = reinterpret_cast<ElemShared<G>*>(smem_raw) + slot_in_block;
  const unsigned lanes_mask = (G == 32) ? 0xffffffffu : ((1u << G) - 1u);
  const unsigned mask = lanes_mask << ((threadIdx.x % 32) / G * G);
  if (slot >= ne) return;  // whole groups leave together
  // The element of this slot: the schedule's order (elements of alike cost
  // side by side, so that the groups sharing a warp take alike paths), or
  // the mesh order. Every output is indexed by the element, so the order
  // changes no result.
  const int64_t e = order ? (int64_t)order[slot] : slot;
  element_body<G>(p, ne, batch, e, sh, lane, mask, coords, conn, u, state, alpha_n, want_tangent, force, tangent,
                  energy, trial, alpha_out, yield, iterations, code, first_failure);
}

// The single kernel over a device-counted list of elements (grid-stride):
// the tile kernel hands it the elements that leave its common road.
template <int G>
__global__ void __launch_bounds__(256) element_list_kernel(const __grid_constant__ Params p, int64_t ne, bool batch,
                                                           const double* __restrict__ coords,
                                                           const int32_t* __restrict__ conn,
                                                           const double* __restrict__ u,
                                                           const double* __restrict__ state,
                                                           const double* __restrict__ alpha_n, int want_tangent,
                                                           double* __restrict__ force, double* __restrict__ tangent,
                                                           double* __restrict__ energy, double* __restrict__ trial,
                                                           double* __restrict__ alpha_out,
                                                           uint8_t* __restrict__ yield,
                                                           int32_t* __restrict__ iterations,
                                                           int32_t* __restrict__ code,
                                                           int32_t* __restrict__ first_failure,
                                                           const int32_t* __restrict__ list,
                                                           const int32_t* __restrict__ count) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int epb = blockDim.x / G;
  const int slot_in_block = threadIdx.x / G;
  const int lane = threadIdx.x % G;
  ElemShared<G>* sh = reinterpret_cast<ElemShared<G>*>(smem_raw) + slot_in_block;
  const unsigned lanes_mask = (G == 32) ? 0xffffffffu : ((1u << G) - 1u);
  const unsigned mask = lanes_mask << ((threadIdx.x % 32) / G * G);
  const int64_t n = *count;
  for (int64_t i = (int64_t)blockIdx.x * epb + slot_in_block; i < n; i += (int64_t)gridDim.x * epb) {
    __syncwarp(mask);
    element_body<G>(p, ne, batch, (int64_t)list[i], sh, lane, mask, coords, conn, u, state, alpha_n, want_tangent,
                    force, tangent, energy, trial, alpha_out, yield, iterations, code, first_failure);
  }
}

// ---- the shape derivative: lambda . d f* / d X ---------------------------------
//
// For the condensed residual f*(u, X) of an IM Hex8 at fixed displacements
// and committed history, with the modes at their local equilibrium
// r_a(u, alpha, X) = 0: lambda^T d f*/dX = [lambda; mu]^T d r/dX |_alpha with
// mu = -K_aa^-T K_ua^T lambda, and r = sum_q w F S [G | G~] (nodes and
// modes). Per point the reverse chain runs r -> (w, F, S, [G | G~]);
// S -> E through the point's material tangent dS/dE; E -> F; F = I + U
// [G | G~]^T -> [G | G~]; G = dN J^-1, G~ = (det0/det)(-2 xi) J0^-1 and
// w = w_q det J -> (J, J0) -> X.

// One point's share: xb (24, node-major) and j0b (9, row-major) accumulate.
template <int G>
__device__ __noinline__ void vjp_point(const Ctx<G>& c, int q, const double* lam, const double* mu, double xb[24],
                                       double j0b[9]) {
  const ElemShared<G>& s = *c.s;
  const double* sl = s.slot[q];
  const double* Fp = sl + kSlotF;
  const double* Sv = sl + kSlotS;
  const double w = sl[kSlotW];
  const double* Ji = s.geo[q];  // J^-1, row-major
  const double ratio = s.geo[q][10];
  double S[9] = {Sv[0], Sv[3], Sv[5], Sv[3], Sv[1], Sv[4], Sv[5], Sv[4], Sv[2]};
  // Q = Lambda Ghat^T (3 x 3), FS = F S, phi = w sum Lambda . (F S Ghat).
  double Q[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  double dn[8][3];
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    shape_grad(a, c.p->qp[q][0], c.p->qp[q][1], c.p->qp[q][2], dn[a]);
    double g[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) g[i] = dn[a][0] * Ji[i] + dn[a][1] * Ji[3 + i] + dn[a][2] * Ji[6 + i];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int j = 0; j < 3; ++j) Q[k * 3 + j] += lam[3 * a + k] * g[j];
  }
  double gt[9];  // G~(i, m) at gt[i * 3 + m]
  mode_grads(c, q, gt);
#pragma unroll
  for (int m = 0; m < 3; ++m)
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int j = 0; j < 3; ++j) Q[k * 3 + j] += mu[3 * m + k] * gt[j * 3 + m];
  double FS[9];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int j = 0; j < 3; ++j) FS[k * 3 + j] = Fp[k * 3 + 0] * S[j] + Fp[k * 3 + 1] * S[3 + j] + Fp[k * 3 + 2] * S[6 + j];
  double phi = 0.0;
#pragma unroll
  for (int i = 0; i < 9; ++i) phi += FS[i] * Q[i];
  phi *= w;
  // Sbar = w sym(F^T Q) -> sbar (normal, 2 x shear) -> ebar = M^T sbar -> Ebar.
  double FtQ[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      FtQ[i * 3 + j] = w * (Fp[0 * 3 + i] * Q[0 * 3 + j] + Fp[1 * 3 + i] * Q[1 * 3 + j] + Fp[2 * 3 + i] * Q[2 * 3 + j]);
  const int vi[6] = {0, 1, 2, 0, 1, 2}, vj[6] = {0, 1, 2, 1, 2, 0};
  double sb[6];
#pragma unroll
  for (int cc = 0; cc < 6; ++cc) {
    const double sym = 0.5 * (FtQ[vi[cc] * 3 + vj[cc]] + FtQ[vj[cc] * 3 + vi[cc]]);
    sb[cc] = cc < 3 ? sym : 2.0 * sym;
  }
  double Eb[9];
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    double acc = 0.0;
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) acc += sl[cc * 6 + d] * sb[cc];
    Eb[vi[d] * 3 + vj[d]] = acc;
    Eb[vj[d] * 3 + vi[d]] = acc;
  }
  // Fbar = w Q S + F Ebar.
  double Fb[9];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      Fb[k * 3 + j] = w * (Q[k * 3 + 0] * S[j] + Q[k * 3 + 1] * S[3 + j] + Q[k * 3 + 2] * S[6 + j]) +
                      Fp[k * 3 + 0] * Eb[j] + Fp[k * 3 + 1] * Eb[3 + j] + Fp[k * 3 + 2] * Eb[6 + j];
  // Gbar = w (F S)^T Lambda + Fbar^T U, node by node; K1 = sum_a dN_a Gbar_a^T.
  double K1[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    double gb[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
      gb[j] = w * (FS[0 * 3 + j] * lam[3 * a + 0] + FS[1 * 3 + j] * lam[3 * a + 1] + FS[2 * 3 + j] * lam[3 * a + 2]) +
              Fb[0 * 3 + j] * s.U[3 * a + 0] + Fb[1 * 3 + j] * s.U[3 * a + 1] + Fb[2 * 3 + j] * s.U[3 * a + 2];
#pragma unroll
    for (int cc = 0; cc < 3; ++cc)
#pragma unroll
      for (int j = 0; j < 3; ++j) K1[cc * 3 + j] += dn[a][cc] * gb[j];
  }
  // Modes: Gbar~ (3 x 3), R and K2.
  double R = 0.0, K2[9];
  const double cm[3] = {-2.0 * c.p->qp[q][0], -2.0 * c.p->qp[q][1], -2.0 * c.p->qp[q][2]};
#pragma unroll
  for (int m = 0; m < 3; ++m)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double gbm = w * (FS[0 * 3 + i] * mu[3 * m + 0] + FS[1 * 3 + i] * mu[3 * m + 1] + FS[2 * 3 + i] * mu[3 * m + 2]) +
                         Fb[0 * 3 + i] * s.alpha[3 * m + 0] + Fb[1 * 3 + i] * s.alpha[3 * m + 1] +
                         Fb[2 * 3 + i] * s.alpha[3 * m + 2];
      R += gbm * cm[m] * s.jinv0[m * 3 + i];
      K2[m * 3 + i] = cm[m] * gbm;
    }
  // Jbar = (phi - ratio R) J^-T - J^-T K1 J^-T; J0bar += ratio R J0^-T - ratio J0^-T K2 J0^-T.
  const double* J0i = s.jinv0;
  double Jb[9];
#pragma unroll
  for (int pp = 0; pp < 3; ++pp)
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      double a1 = 0.0, a2 = 0.0;
#pragma unroll
      for (int cc = 0; cc < 3; ++cc)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          a1 += Ji[cc * 3 + pp] * K1[cc * 3 + j] * Ji[r * 3 + j];
          a2 += J0i[cc * 3 + pp] * K2[cc * 3 + j] * J0i[r * 3 + j];
        }
      Jb[pp * 3 + r] = (phi - ratio * R) * Ji[r * 3 + pp] - a1;
      j0b[pp * 3 + r] += ratio * R * J0i[r * 3 + pp] - ratio * a2;
    }
  // J = X dN: Xbar_ia += sum_c Jbar_ic dN_ac.
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int i = 0; i < 3; ++i)
      xb[3 * a + i] += Jb[i * 3 + 0] * dn[a][0] + Jb[i * 3 + 1] * dn[a][1] + Jb[i * 3 + 2] * dn[a][2];
}

template <int G>
__device__ __forceinline__ void vjp_element(const Params& p, int64_t ne, int64_t e, ElemShared<G>* sh, int lane,
                                            unsigned mask, const double* __restrict__ coords,
                                            const int32_t* __restrict__ conn, const double* __restrict__ u,
                                            const double* __restrict__ state, const double* __restrict__ alpha_n,
                                            const double* __restrict__ lambda, double* __restrict__ trial,
                                            uint8_t* __restrict__ yield, int32_t* __restrict__ code,
                                            int32_t* __restrict__ first_failure, double* __restrict__ out) {
  double hu_lane[9];
  double warm_lane[8];
  warm_lane[7] = 0.0;
  Ctx<G> c{&p, sh, lane, mask, e, ne * p.nq, state, trial, yield, hu_lane, warm_lane};
  ElemShared<G>& s = *sh;
  int bad_node = 0;
  double lam_a[3] = {0.0, 0.0, 0.0};
  if (lane < 8) {
    const int64_t node = conn[e * 8 + lane];
    if (p.num_nodes > 0 && (node < 0 || node >= p.num_nodes)) {
      bad_node = 1;
    } else {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        s.X[3 * lane + k] = coords[node * 3 + k];
        s.U[3 * lane + k] = u[node * 3 + k];
        lam_a[k] = lambda[node * 3 + k];
      }
    }
  }
  if (__any_sync(mask, bad_node)) {
    if (lane == 0) {
      code[e] = SBK_EL_BAD_NODE;
      atomicMin(first_failure, (int32_t)e);
    }
    return;
  }
  for (int i = lane; i < 9; i += G) s.alpha[i] = alpha_n ? alpha_n[e * 9 + i] : 0.0;
  c.sync();
  int status = set_up<G>(c);
  Local<G> loc(c);
  if (!status) status = loc.run();
  if (status) {
    if (lane == 0) {
      code[e] = status;
      atomicMin(first_failure, (int32_t)e);
    }
    return;
  }
  const bool geometric = p.kinematics != SBK_SMALL_STRAIN;
  // K_ua^T lambda, node by node (lane a), summed in node order by lane 0.
  double* part = s.work;  // 8 x 9 partial sums, then lambda (24) and mu (9)
  if (lane < 8) {
    const int a = lane;
    double kua[3][9];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int j = 0; j < 9; ++j) kua[k][j] = 0.0;
    for (int q = 0; q < p.nq; ++q) {
      double g[3], gt[9], V[27];
      node_grad(c, q, a, g);
      mode_grads(c, q, gt);
      vtensor(s.slot[q], g, false, geometric, V);
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int l = 0; l < 3; ++l)
            kua[k][3 * m + l] += V[(k * 3 + l) * 3 + 0] * gt[0 * 3 + m] + V[(k * 3 + l) * 3 + 1] * gt[1 * 3 + m] +
                                 V[(k * 3 + l) * 3 + 2] * gt[2 * 3 + m];
    }
#pragma unroll
    for (int j = 0; j < 9; ++j)
      part[a * 9 + j] = kua[0][j] * lam_a[0] + kua[1][j] * lam_a[1] + kua[2][j] * lam_a[2];
#pragma unroll
    for (int k = 0; k < 3; ++k) part[72 + 3 * a + k] = lam_a[k];
  }
  c.sync();
  if (lane == 0) {
    double b[9], y[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      double acc = 0.0;
      for (int a = 0; a < 8; ++a) acc += part[a * 9 + j];
      b[j] = acc;
    }
    fullpiv_solve9_t(s.lu, s.rowp, s.colp, b, y);
#pragma unroll
    for (int j = 0; j < 9; ++j) part[96 + j] = -y[j];
  }
  c.sync();
  // Every point's share, then the sums over the points (reduce-scatter of
  // 33 values: 24 of Xbar, 9 of J0bar), and J0 = X dN(0) folded in.
  double xb[24], j0b[9];
#pragma unroll
  for (int i = 0; i < 24; ++i) xb[i] = 0.0;
#pragma unroll
  for (int i = 0; i < 9; ++i) j0b[i] = 0.0;
  if (lane < p.nq) vjp_point<G>(c, lane, part + 72, part + 96, xb, j0b);
  double* red = s.kc;  // 33 sums
#pragma unroll
  for (int chunk = 0; chunk * G < 33; ++chunk) {
    double buf[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int idx = chunk * G + i;
      buf[i] = idx < 24 ? xb[idx < 24 ? idx : 0] : (idx < 33 ? j0b[idx - 24 < 9 && idx >= 24 ? idx - 24 : 0] : 0.0);
    }
    const double v = reduce_scatter<G>(buf, lane, mask);
    if (chunk * G + lane < 33) red[chunk * G + lane] = v;
  }
  c.sync();
  if (lane < 8) {
    const int a = lane;
    double dn0[3];
    shape_grad(a, 0.0, 0.0, 0.0, dn0);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      out[e * 24 + 3 * a + i] = red[3 * a + i] + red[24 + i * 3 + 0] * dn0[0] + red[24 + i * 3 + 1] * dn0[1] +
                                red[24 + i * 3 + 2] * dn0[2];
  }
  if (lane == 0) code[e] = 0;
}

// The elements the tile kernel handed on (grid-stride over its list).
template <int G>
__global__ void __launch_bounds__(256) vjp_kernel(const __grid_constant__ Params p, int64_t ne,
                                                  const double* __restrict__ coords, const int32_t* __restrict__ conn,
                                                  const double* __restrict__ u, const double* __restrict__ state,
                                                  const double* __restrict__ alpha_n,
                                                  const double* __restrict__ lambda, double* __restrict__ trial,
                                                  uint8_t* __restrict__ yield, int32_t* __restrict__ code,
                                                  int32_t* __restrict__ first_failure, double* __restrict__ out,
                                                  const int32_t* __restrict__ list,
                                                  const int32_t* __restrict__ count) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int epb = blockDim.x / G;
  const int slot_in_block = threadIdx.x / G;
  const int lane = threadIdx.x % G;
  ElemShared<G>* sh = reinterpret_cast<ElemShared<G>*>(smem_raw) + slot_in_block;
  const unsigned lanes_mask = (G == 32) ? 0xffffffffu : ((1u << G) - 1u);
  const unsigned mask = lanes_mask << ((threadIdx.x % 32) / G * G);
  const int64_t n = *count;
  for (int64_t i = (int64_t)blockIdx.x * epb + slot_in_block; i < n; i += (int64_t)gridDim.x * epb) {
    __syncwarp(mask);
    vjp_element<G>(p, ne, (int64_t)list[i], sh, lane, mask, coords, conn, u, state, alpha_n, lambda, trial, yield,
                   code, first_failure, out);
  }
}

template <int G>
int launch_g(const Params& p, int64_t ne, const double* coords, const int32_t* conn, const double* u,
             const double* state, const double* alpha_n, int want_tangent, double* force, double* tangent,
             double* energy, double* trial, double* alpha_out, uint8_t* yield, int32_t* iterations, int32_t* code,
             int32_t* first_failure, bool batch, int epb, const int32_t* order, cudaStream_t stream) {
  const int threads = epb * G;
  const size_t smem = sizeof(ElemShared<G>) * epb;
  const int64_t blocks = (ne + epb - 1) / epb;
  if (blocks == 0) return 0;
  auto kern = element_kernel<G>;
  static SmemLimit limit;
  const cudaError_t err = limit.allow(kern);
  if (err != cudaSuccess) return (int)err;
  kern<<<(unsigned)blocks, threads, smem, stream>>>(p, ne, batch, coords, conn, u, state, alpha_n, want_tangent,
                                                     force, tangent, energy, trial, alpha_out, yield, iterations,
                                                     code, first_failure, order);
  return (int)cudaGetLastError();
}

}  // namespace

namespace {

// The arrays of a launch's scratch at base (NULL: their bytes only).
size_t tile_layout(char* base, int64_t ne, int nq, int64_t chunk, TileScratch& s) {
  const int most = tile_most(nq);
  const size_t points = (size_t)(most * nq) | 1;
  const size_t blocks = (size_t)(ne < kTileBlocks ? ne : kTileBlocks);
  size_t at = 0;
  auto take = [&](size_t bytes) {
    char* here = base + at;
    at += (bytes + 255) / 256 * 256;
    return static_cast<void*>(here);
  };
  s.counts = static_cast<int32_t*>(take(2 * sizeof(int32_t)));
  s.fallback = static_cast<int32_t*>(take((size_t)ne * sizeof(int32_t)));
  s.geo = static_cast<double*>(take(blocks * kTileGeo * points * sizeof(double)));
  s.cond = static_cast<double*>(take((size_t)chunk * tile_record(nq) * sizeof(double)));
  s.chunk = chunk;
  return at;
}

}  // namespace

size_t tile_scratch_bytes(int64_t ne, int nq, int64_t chunk) {
  TileScratch s;
  return tile_layout(nullptr, ne, nq, chunk, s);
}

void tile_scratch_carve(void* base, int64_t ne, int nq, int64_t chunk, TileScratch& s) {
  tile_layout(static_cast<char*>(base), ne, nq, chunk, s);
}

namespace {

// The element's kernels over the elements of `a`, in launches of s.chunk, each
// followed by after(its arguments, its scratch).
template <class After>
int run_tiles(const Params& p, TileArgs a, const TileScratch& s, int elements_per_block, cudaStream_t stream,
              After after) {
  // As many elements a tile as make the waves of tiles full ones: n elements
  // in ceil(n / (148 most)) waves. Full tiles leave a last wave of a few that
  // takes as long as the others: 2,304 elements of 20 points, 379 us as 192
  // tiles of 12, 327 us as 288 of 8; 8,192 of 8 points 190 and 178 us. From
  // five waves on there is no difference (23,086 of 8 points: 975 us).
  const int most = tile_most(p.nq);
  for (a.begin = 0; a.begin < a.ne; a.begin += s.chunk) {
    a.end = a.ne - a.begin < s.chunk ? a.ne : a.begin + s.chunk;
    const int64_t n = a.end - a.begin, waves = (n + kTileBlocks * most - 1) / (kTileBlocks * most);
    a.elements = elements_per_block > 0 ? elements_per_block : (int)((n + kTileBlocks * waves - 1) / (kTileBlocks * waves));
    if (a.elements > most) a.elements = most;
    a.num_tiles = (int)((a.end - a.begin + a.elements - 1) / a.elements);
    const unsigned grid = (unsigned)(a.num_tiles < kTileBlocks ? a.num_tiles : kTileBlocks);
    cudaError_t err = cudaMemsetAsync(s.counts, 0, (a.begin == 0 ? 2 : 1) * sizeof(int32_t), stream);
    if (err != cudaSuccess) return (int)err;
    int rc;
    if (p.element == 1) rc = launch_standard(p, a, s, stream);
    else if (!p.general) rc = launch_tile_j2(p, a, s, grid, stream);
    else if (p.nterms == 0) rc = launch_tile_general0(p, a, s, grid, stream);
    else if (p.nterms == 1) rc = launch_tile_general1(p, a, s, grid, stream);
    else if (p.nterms == 2) rc = launch_tile_general2(p, a, s, grid, stream);
    else rc = launch_tile_general4(p, a, s, grid, stream);
    if (!rc) rc = after(a);
    if (rc) return rc;
  }
  return 0;
}

// The elements handed on, by a list kernel that starts each again with
// `record` bytes of shared memory an element (one block of it per SM).
template <class K, class... A>
int run_list(K kern, int64_t ne, int group, size_t record, SmemLimit& limit, cudaStream_t stream, const A&... args) {
  const int epb = group == 8 ? 16 : 8;
  const size_t smem = record * epb;
  const cudaError_t err = limit.allow(kern);
  if (err != cudaSuccess) return (int)err;
  const int64_t need = (ne + epb - 1) / epb;
  kern<<<(unsigned)(need < 148 * 2 ? need : 148 * 2), epb * group, smem, stream>>>(args...);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_elements_tile(const Params& p, int64_t ne, const double* coords, const int32_t* conn, const double* u,
                         const double* state, const double* alpha_n, int want_tangent, double* force,
                         double* tangent, double* energy, double* trial, double* alpha_out, uint8_t* yield,
                         int32_t* iterations, int32_t* code, int32_t* first_failure, bool batch,
                         const TileScratch& s, int elements_per_block, cudaStream_t stream) {
  if (ne <= 0) return 0;
  const TileArgs a{ne, coords, conn, u, state, alpha_n, force, tangent, energy, trial, alpha_out, yield, iterations,
                   code, first_failure, want_tangent, batch ? 1 : 0, 0, 0, 0, 0};
  const int rc = run_tiles(p, a, s, elements_per_block, stream, [&](const TileArgs& at) {
    return p.element == 1 ? 0 : launch_condense(p, at, s, stream);
  });
  if (rc || p.element == 1) return rc;
  static SmemLimit limit[2];
  if (p.nq <= 8)
    return run_list(element_list_kernel<8>, ne, 8, sizeof(ElemShared<8>), limit[0], stream, p, ne, batch, coords,
                    conn, u, state, alpha_n, want_tangent, force, tangent, energy, trial, alpha_out, yield,
                    iterations, code, first_failure, s.fallback, s.counts + 1);
  return run_list(element_list_kernel<32>, ne, 32, sizeof(ElemShared<32>), limit[1], stream, p, ne, batch, coords,
                  conn, u, state, alpha_n, want_tangent, force, tangent, energy, trial, alpha_out, yield, iterations,
                  code, first_failure, s.fallback, s.counts + 1);
}

int launch_vjp(const Params& p, int64_t ne, const double* coords, const int32_t* conn, const double* u,
               const double* state, const double* alpha_n, const double* lambda, double* energy, double* trial,
               double* alpha_out, uint8_t* yield, int32_t* iterations, int32_t* code, int32_t* first_failure,
               double* out, const TileScratch& s, int elements_per_block, cudaStream_t stream) {
  if (ne <= 0) return 0;
  const TileArgs a{ne, coords, conn, u, state, alpha_n, nullptr, nullptr, energy, trial, alpha_out, yield, iterations,
                   code, first_failure, 0, 0, 0, 0, 0, 0};
  const int rc = run_tiles(p, a, s, elements_per_block, stream,
                           [&](const TileArgs& at) { return launch_vjp_tile(p, at, s, lambda, out, stream); });
  if (rc) return rc;
  static SmemLimit limit[2];
  if (p.nq <= 8)
    return run_list(vjp_kernel<8>, ne, 8, sizeof(ElemShared<8>), limit[0], stream, p, ne, coords, conn, u, state,
                    alpha_n, lambda, trial, yield, code, first_failure, out, s.fallback, s.counts + 1);
  return run_list(vjp_kernel<32>, ne, 32, sizeof(ElemShared<32>), limit[1], stream, p, ne, coords, conn, u, state,
                  alpha_n, lambda, trial, yield, code, first_failure, out, s.fallback, s.counts + 1);
}

int launch_elements(const Params& p, int64_t ne, const double* coords, const int32_t* conn, const double* u,
                    const double* state, const double* alpha_n, int want_tangent, double* force, double* tangent,
                    double* energy, double* trial, double* alpha_out, uint8_t* yield, int32_t* iterations,
                    int32_t* code, int32_t* first_failure, bool batch, int elements_per_block,
                    const int32_t* order, cudaStream_t stream) {
  if (p.nq <= 8) {
    // At most what 227 KB of shared memory and 256 threads hold.
    const int most = (int)((227 * 1024) / sizeof(ElemShared<8>)) < 32 ? (int)((227 * 1024) / sizeof(ElemShared<8>)) : 32;
    // The default, 16 elements (4 warps) per block and so one block per SM:
    // the four warps of a block start together and, their elements being
    // alike under the schedule, stay close enough in the code to share its
    // instruction fetches (1.8x over one-warp blocks on the sheet
    // microbenchmark; 5 to 7 warps per block are slower).
    int epb = elements_per_block > 0 ? elements_per_block : 16;
    if (epb > most) epb = most;
    return launch_g<8>(p, ne, coords, conn, u, state, alpha_n, want_tangent, force, tangent, energy, trial,
                       alpha_out, yield, iterations, code, first_failure, batch, epb, order, stream);
  }
  // Rules of 9 to 32 points (the sheet rules 2 x 2 x 3..7, the 3 x 3 x 3
  // cube): a warp per element, lane = point. The default, 8 warps per block
  // (the most 256 threads allow), for the same shared instruction fetches:
  // 42 ms per 80,000 elements of the 2 x 2 x 5 rule, against 55 ms at 4
  // warps and 80 ms at 1.
  const int epb = elements_per_block > 0 ? (elements_per_block < 8 ? elements_per_block : 8) : 8;
  return launch_g<32>(p, ne, coords, conn, u, state, alpha_n, want_tangent, force, tangent, energy, trial,
                      alpha_out, yield, iterations, code, first_failure, batch, epb, order, stream);
}

}  // namespace sbk
