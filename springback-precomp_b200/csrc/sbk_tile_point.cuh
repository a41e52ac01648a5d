// The tile kernel's material point: the spectral log strain, the trial
// state, the J2 and the general return, the logarithmic map. The same
// algorithms as sbk_material.cuh (which cites the reference), arranged for a
// thread that reads and writes its point's record field by field in shared
// memory: nothing is indexed by a run-time value, so nothing of a point
// lives in a stack frame.
//
// NT is the number of kinematic terms known when the kernel is compiled: -1
// the J2 law, 0 to 2 the general law with that many, 4 the general law with
// up to four (their count read from the parameters).
#pragma once

#include "sbk_element_math.cuh"
#include "sbk_material.cuh"

namespace sbk {

// A field of one point: base[f * stride].
struct PointRecord {
  double* base;
  int stride;
  __device__ __forceinline__ double get(int f) const { return base[f * stride]; }
  __device__ __forceinline__ void put(int f, double v) const { base[f * stride] = v; }
};

// One rotation of the cyclic Jacobi iteration on the symmetric 3 x 3 (packed
// 00 11 22 01 12 20) with the axes as columns of v. tan(2 phi) = b / d with
// d = a_qq - a_pp, b = 2 a_pq: t = b / (d +- sqrt(d^2 + b^2)), one root, one
// quotient and one reciprocal root a rotation.
template <int P, int Q>
__device__ __forceinline__ void spectral_rotate(double a[6], double v[9]) {
  constexpr int R = 3 - P - Q;
  constexpr int PQ = (P + Q == 1) ? 3 : (P + Q == 3 ? 4 : 5);
  constexpr int PR = (P + R == 1) ? 3 : (P + R == 3 ? 4 : 5);
  constexpr int QR = (Q + R == 1) ? 3 : (Q + R == 3 ? 4 : 5);
  const double b = 2.0 * a[PQ];
  if (b * b == 0.0) return;
  const double d = a[Q] - a[P];
  const double h = sqrt(d * d + b * b);
  const double t = b / (d >= 0.0 ? d + h : d - h);
  const double c = rsqrt(1.0 + t * t);
  const double s = t * c;
  const double u = t * a[PQ];
  a[P] -= u;
  a[Q] += u;
  a[PQ] = 0.0;
  const double pr = a[PR], qr = a[QR];
  a[PR] = c * pr - s * qr;
  a[QR] = s * pr + c * qr;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double vp = v[k * 3 + P], vq = v[k * 3 + Q];
    v[k * 3 + P] = c * vp - s * vq;
    v[k * 3 + Q] = s * vp + c * vq;
  }
}

// Q^T A Q of a symmetric A (Voigt 00 11 22 01 12 20, tensorial).
__device__ __forceinline__ void rotate_in(const double q[9], const double a[6], double out[6]) {
  double b[9];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    b[0 + j] = a[0] * q[j] + a[3] * q[3 + j] + a[5] * q[6 + j];
    b[3 + j] = a[3] * q[j] + a[1] * q[3 + j] + a[4] * q[6 + j];
    b[6 + j] = a[5] * q[j] + a[4] * q[3 + j] + a[2] * q[6 + j];
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int i = k < 3 ? k : k - 3, j = k < 3 ? k : (k - 2) % 3;
    out[k] = q[i] * b[j] + q[3 + i] * b[3 + j] + q[6 + i] * b[6 + j];
  }
}
// Q A Q^T.
__device__ __forceinline__ void rotate_out(const double q[9], const double a[6], double out[6]) {
  double b[9];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    b[i * 3 + 0] = q[i * 3] * a[0] + q[i * 3 + 1] * a[3] + q[i * 3 + 2] * a[5];
    b[i * 3 + 1] = q[i * 3] * a[3] + q[i * 3 + 1] * a[1] + q[i * 3 + 2] * a[4];
    b[i * 3 + 2] = q[i * 3] * a[5] + q[i * 3 + 1] * a[4] + q[i * 3 + 2] * a[2];
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int i = k < 3 ? k : k - 3, j = k < 3 ? k : (k - 2) % 3;
    out[k] = b[i * 3] * q[j * 3] + b[i * 3 + 1] * q[j * 3 + 1] + b[i * 3 + 2] * q[j * 3 + 2];
  }
}

// E_log (engineering Voigt) of a Green-Lagrange strain (engineering Voigt)
// and its spectral data L. L.q holds the axes to start from: those of the
// element's last pass, in which the strain of the next is nearly diagonal (a
// sweep or two remain of four or five), or the identity. One step of Newton's
// iteration for the nearest orthogonal matrix, Q (3 - Q^T Q) / 2, first: each
// pass's rotations leave them off by some units in the last place, which
// would add up over an element's passes.
__device__ __forceinline__ int spectral_log(const double green[6], LogKin& L, double elog[6]) {
#pragma unroll
  for (int i = 0; i < 6; ++i)
    if (!isfinite(green[i])) return kFailNonFinite;
  double a[6];
  {
    double g[6], q[9];  // (3 - Q^T Q) / 2
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int i = k < 3 ? k : k - 3, j = k < 3 ? k : (k - 2) % 3;
      g[k] = (i == j ? 1.5 : 0.0) - 0.5 * (L.q[i] * L.q[j] + L.q[3 + i] * L.q[3 + j] + L.q[6 + i] * L.q[6 + j]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      q[3 * i] = L.q[3 * i] * g[0] + L.q[3 * i + 1] * g[3] + L.q[3 * i + 2] * g[5];
      q[3 * i + 1] = L.q[3 * i] * g[3] + L.q[3 * i + 1] * g[1] + L.q[3 * i + 2] * g[4];
      q[3 * i + 2] = L.q[3 * i] * g[5] + L.q[3 * i + 1] * g[4] + L.q[3 * i + 2] * g[2];
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) L.q[i] = q[i];
    const double e[6] = {green[0], green[1], green[2], 0.5 * green[3], 0.5 * green[4], 0.5 * green[5]};
    rotate_in(L.q, e, a);
  }
#pragma unroll 1
  for (int sweep = 0; sweep < 60; ++sweep) {
    const double off = a[3] * a[3] + a[4] * a[4] + a[5] * a[5];
    const double diag = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    if (off == 0.0 || off <= 1.0e-36 * diag) break;
    spectral_rotate<0, 1>(a, L.q);
    spectral_rotate<0, 2>(a, L.q);
    spectral_rotate<1, 2>(a, L.q);
  }
  // Ascending, the axes with their values.
  auto order = [&](int i, int j) {
    const bool swap = a[j] < a[i];
    const double lo = swap ? a[j] : a[i], hi = swap ? a[i] : a[j];
    a[i] = lo;
    a[j] = hi;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const double vi = L.q[r * 3 + i], vj = L.q[r * 3 + j];
      L.q[r * 3 + i] = swap ? vj : vi;
      L.q[r * 3 + j] = swap ? vi : vj;
    }
  };
  order(0, 1);
  order(0, 2);
  order(1, 2);
  bool bad = false;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double s2 = 1.0 + 2.0 * a[c];
    bad = bad || !(s2 > 0.0) || !isfinite(s2);
    L.mu[c] = a[c];
    L.first[c] = 1.0 / s2;
  }
  if (bad) return kFailDegenerate;
  // The principal log strains, and the first divided differences of ln
  // between the principal values (mu ascending): log1p(d / y) / d.
  double pr[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const double m = c == 0 ? a[0] : (c == 1 ? a[1] : a[2]);
    const double lo = c == 1 ? a[1] : a[0], hi = c == 0 ? a[1] : a[2];
    const double y = c == 0 ? L.first[1] : L.first[2];
    const double d = 2.0 * (lo - hi);
    const double v = 0.5 * log1p(2.0 * m);
    const double f = d == 0.0 ? y : log1p(d * y) / d;
    if (c == 0) pr[0] = v, L.first[3] = f;
    else if (c == 1) pr[1] = v, L.first[4] = f;
    else pr[2] = v, L.first[5] = f;
  }
  rotate_out(L.q, pr, elog);
#pragma unroll
  for (int i = 3; i < 6; ++i) elog[i] *= 2.0;
  return 0;
}

// Reference geometry of a point (set_up, IncompatibleModes.cpp:134-192) from its
// element's staged coordinates and displacements X, U (24 each): J^-1, w det
// J, det0 / det, J0^-1 and U G^T. False for an element inverted at rest.
struct PointGeometry {
  double ji[9], j0i[9], du[9], w, ratio;
};
__device__ __forceinline__ bool point_geometry(const Params& p, int q, const double* X, const double* U,
                                               PointGeometry& G) {
  double j0[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, jq[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  double uq[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  const double xi = p.qp[q][0], eta = p.qp[q][1], zeta = p.qp[q][2];
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const double sx = ((n + 1) >> 1) & 1 ? 1.0 : -1.0, sy = (n >> 1) & 1 ? 1.0 : -1.0, sz = n >> 2 ? 1.0 : -1.0;
    const double fx = 1.0 + xi * sx, fy = 1.0 + eta * sy, fz = 1.0 + zeta * sz;
    const double dn[3] = {0.125 * sx * fy * fz, 0.125 * sy * fx * fz, 0.125 * sz * fx * fy};
    const double d0[3] = {0.125 * sx, 0.125 * sy, 0.125 * sz};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double x = X[3 * n + i], u = U[3 * n + i];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        j0[i * 3 + c] += x * d0[c];
        jq[i * 3 + c] += x * dn[c];
        uq[i * 3 + c] += u * dn[c];
      }
    }
  }
  const double det0 = det3(j0), det = det3(jq);
  if (!(det0 > 0.0) || !(det > 0.0)) return false;
  inv3(j0, G.j0i);
  inv3(jq, G.ji);
  G.w = p.qp[q][3] * det;
  G.ratio = det0 / det;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      G.du[i * 3 + j] = uq[i * 3] * G.ji[j] + uq[i * 3 + 1] * G.ji[3 + j] + uq[i * 3 + 2] * G.ji[6 + j];
  return true;
}

// The strain the return takes at the displacement gradient h, with L (from the
// axes it holds) under logarithmic kinematics. 0 or the point's failure.
__device__ __forceinline__ int point_strain(const Params& p, const double h[9], LogKin& L, double strain[6]) {
  if (p.kinematics == SBK_SMALL_STRAIN) {
    strain[0] = h[0], strain[1] = h[4], strain[2] = h[8];
    strain[3] = h[1] + h[3], strain[4] = h[5] + h[7], strain[5] = h[6] + h[2];
    return 0;
  }
  double green[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int i = c < 3 ? c : c - 3, j = c < 3 ? c : (c - 2) % 3;
    const double e2 = h[i * 3 + j] + h[j * 3 + i] + h[i] * h[j] + h[3 + i] * h[3 + j] + h[6 + i] * h[6 + j];
    green[c] = c < 3 ? 0.5 * e2 : e2;
    strain[c] = green[c];
  }
  if (p.kinematics != SBK_FINITE_LOGARITHMIC) return 0;
  const double F[9] = {h[0] + 1.0, h[1], h[2], h[3], h[4] + 1.0, h[5], h[6], h[7], h[8] + 1.0};
  if (!(det3(F) > 0.0)) return SBK_EL_INVERTED_POINT;
  return spectral_log(green, L, strain);
}

// second(k, j, i), mu_k <= mu_j <= mu_i: the second divided difference of ln
// (log_div2 with the order of its arguments known).
__device__ __forceinline__ double spectral_second(const LogKin& L, int k, int j, int i) {
  const double fij = i == j ? L.first[i] : first_of(L.first, i, j);
  const double fjk = j == k ? L.first[j] : first_of(L.first, j, k);
  const double iy = L.first[j];  // 1 / (1 + 2 mu_j)
  const double spread = 2.0 * (L.mu[i] - L.mu[k]);
  if (spread * iy > 5.0e-3) return (fij - fjk) / spread;
  const double u = 2.0 * (L.mu[i] - L.mu[j]) * iy;
  const double w = 2.0 * (L.mu[k] - L.mu[j]) * iy;
  double h = 1.0, wn = 1.0, sum = -0.5;
#pragma unroll
  for (int n = 1; n <= 5; ++n) {
    wn *= w;
    h = u * h + wn;
    sum += (n % 2 == 1 ? 1.0 : -1.0) / (double)(n + 2) * h;
  }
  return sum * (iy * iy);
}

// The logarithmic map of a point's response: S = P^T T and the material
// block P^T C P + T : L in global axes, through the principal frame with
// 3 x 3 rotations (C's rows, then its columns, as symmetric tensors). T : L
// there has H(aa,aa) = 4 t_aa D_aaa, H(aa,ab) = 2 t_ab D_aab, H(ab,ab) =
// t_aa D_aab + t_bb D_abb, H(ab,bc) = t_ac D_abc and nothing else. An
// elastic point's C is isotropic, the same in every frame. C stays in the
// point's record and passes through row by row and column by column: 36
// values in registers would leave no room for more warps, and unrolled they
// are 20 KB of code that every tile fetches each round.
__device__ __forceinline__ double spectral_map(const Params& p, const LogKin& L, bool elastic, const PointRecord& rec,
                                               int fS, int fM) {
  double tp[6];
  {
    double t[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) t[i] = rec.get(fS + i);
    rotate_in(L.q, t, tp);
  }
  if (!elastic) {
#pragma unroll 1
    for (int i = 0; i < 6; ++i) {
      double row[6], r[6];
#pragma unroll
      for (int j = 0; j < 6; ++j) row[j] = rec.get(fM + i * 6 + j);
      rotate_in(L.q, row, r);
#pragma unroll
      for (int j = 0; j < 6; ++j) rec.put(fM + i * 6 + j, r[j]);
    }
  }
  // Pairs 3: (0,1), 4: (1,2), 5: (2,0).
  const double d001 = spectral_second(L, 0, 0, 1), d011 = spectral_second(L, 0, 1, 1);
  const double d112 = spectral_second(L, 1, 1, 2), d122 = spectral_second(L, 1, 2, 2);
  const double d002 = spectral_second(L, 0, 0, 2), d022 = spectral_second(L, 0, 2, 2);
  const double d012 = spectral_second(L, 0, 1, 2);
  // Column j of H: its diagonal entry and up to two others in each half.
  const double h03 = 2.0 * tp[3] * d001, h13 = 2.0 * tp[3] * d011, h14 = 2.0 * tp[4] * d112, h24 = 2.0 * tp[4] * d122;
  const double h05 = 2.0 * tp[5] * d002, h25 = 2.0 * tp[5] * d022;
  const double h33 = tp[0] * d001 + tp[1] * d011, h44 = tp[1] * d112 + tp[2] * d122, h55 = tp[0] * d002 + tp[2] * d022;
  const double h34 = tp[5] * d012, h45 = tp[3] * d012, h35 = tp[4] * d012;
  const double lame = p.K - 2.0 * p.G / 3.0;
#pragma unroll 1
  for (int j = 0; j < 6; ++j) {
    double col[6], r[6];
    if (elastic) {
#pragma unroll
      for (int i = 0; i < 6; ++i) r[i] = (i < 3 && j < 3 ? lame : 0.0) + (i == j ? (i < 3 ? 2.0 * p.G : p.G) : 0.0);
    } else {
#pragma unroll
      for (int i = 0; i < 6; ++i) col[i] = rec.get(fM + i * 6 + j);
      rotate_in(L.q, col, r);
    }
    double fj = L.first[0];
#pragma unroll
    for (int i = 1; i < 6; ++i) fj = j == i ? L.first[i] : fj;
#pragma unroll
    for (int i = 0; i < 6; ++i) r[i] *= L.first[i] * fj;
    switch (j) {
      case 0: r[0] -= 2.0 * tp[0] * (fj * fj), r[3] += h03, r[5] += h05; break;  // D_aaa = -1 / (2 y^2)
      case 1: r[1] -= 2.0 * tp[1] * (fj * fj), r[3] += h13, r[4] += h14; break;
      case 2: r[2] -= 2.0 * tp[2] * (fj * fj), r[4] += h24, r[5] += h25; break;
      case 3: r[0] += h03, r[1] += h13, r[3] += h33, r[4] += h34, r[5] += h35; break;
      case 4: r[1] += h14, r[2] += h24, r[3] += h34, r[4] += h44, r[5] += h45; break;
      default: r[0] += h05, r[2] += h25, r[3] += h35, r[4] += h45, r[5] += h55; break;
    }
    rotate_out(L.q, r, col);
#pragma unroll
    for (int i = 0; i < 6; ++i) rec.put(fM + i * 6 + j, col[i]);
  }
  double top = 0.0;
#pragma unroll 1
  for (int i = 0; i < 6; ++i) {
    double row[6], r[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) row[j] = rec.get(fM + i * 6 + j);
    rotate_out(L.q, row, r);
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      rec.put(fM + i * 6 + j, r[j]);
      top = fmax(top, fabs(r[j]));
    }
  }
  double t[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) tp[i] *= L.first[i];
  rotate_out(L.q, tp, t);
#pragma unroll
  for (int i = 0; i < 6; ++i) rec.put(fS + i, t[i]);
  return top;
}

// ---- the trial state ------------------------------------------------------------

template <int NT>
struct PointTrial {
  static constexpr int kTerms = NT > 0 ? NT : 1;
  double el[6], s[6], xi[6];  // elastic strain, trial deviator, relative stress
  double a[kTerms][6];        // the committed kinematic terms
  double vol, a_n, ey, sy, eq, f;  // ey = expm1(-delta a_n); f = overstress
  bool loading;
};

template <int NT>
__device__ __forceinline__ int term_count(const Params& p) {
  return NT < 0 ? 0 : (NT <= 2 ? NT : p.nterms);
}

__device__ __forceinline__ double deviatoric(const Params& p, const double el[6], double s[6]) {
  const double vol = el[0] + el[1] + el[2], mean = vol / 3.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) s[i] = 2.0 * p.G * (el[i] - mean);
#pragma unroll
  for (int i = 3; i < 6; ++i) s[i] = p.G * el[i];
  return vol;
}

template <int NT>
__device__ __forceinline__ void point_trial(const Params& p, const double strain[6], const double* state,
                                            int64_t stride, PointTrial<NT>& T) {
  const int nt = term_count<NT>(p);
#pragma unroll
  for (int i = 0; i < 6; ++i) T.el[i] = strain[i] - state[(kFieldEp + i) * stride];
  T.a_n = state[field_eqps(nt) * stride];
  T.loading = state[field_loading(nt) * stride] != 0.0;
  if (NT < 0) {
#pragma unroll
    for (int i = 0; i < 6; ++i) T.xi[i] = -state[(kFieldBeta + i) * stride];
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) T.xi[i] = 0.0;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        T.a[t][i] = (NT <= 2 || t < nt) ? state[(kFieldAlpha + 6 * t + i) * stride] : 0.0;
        T.xi[i] -= T.a[t][i];
      }
  }
  T.vol = deviatoric(p, T.el, T.s);
#pragma unroll
  for (int i = 0; i < 6; ++i) T.xi[i] += T.s[i];
  T.ey = expm1(-p.delta * T.a_n);
  T.sy = p.sy0 + p.H * T.a_n - p.Q * T.ey;
  if (NT < 0) {
    T.eq = tnorm(T.xi);
    T.sy *= 0.816496580927726;  // the radius sqrt(2/3) sigma_y
  } else {
    double q = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      double v = 0.0;
#pragma unroll
      for (int j = 0; j < 6; ++j) v += p.P[i * 6 + j] * T.xi[j];
      q += T.xi[i] * v;
    }
    T.eq = sqrt(q < 0.0 ? 0.0 : q);  // a NaN stays one (fmax would drop it): the return fails on it
  }
  T.f = T.eq - T.sy;
}

template <int NT>
__device__ __forceinline__ bool point_elastic(const Params& p, const PointTrial<NT>& T) {
  return !p.enabled || T.f <= 1.0e-12 * T.sy;
}
template <int NT>
__device__ __forceinline__ bool point_window(const Params& p, const PointTrial<NT>& T) {
  return p.enabled && T.loading && T.f > -1.0e-10 * T.sy && T.eq > 0.0;
}

// ---- the general return -----------------------------------------------------------
//
// The closest-point equations (Plasticity.cpp:246-311) in the coordinates of
// the yield matrix's generalised eigenvectors: P = S^-1 V L V^T S^-1 with V^T
// S^-1 V = I (S = diag(1, 1, 1, 1/2, 1/2, 1/2), found once on the host), xi =
// V y. There sigma_bar^2 = sum L y^2, the flow direction S m is V (L y /
// sigma_bar), and the equations are
//   r_k = y_k (1 + f L_k) - z_k(dl),  f = b / sigma_bar,
//   r_7 = sigma_bar - sigma_y(a_n + dl),
// with z(dl) the trial relative stress: no 6 x 6 product is left in the
// iteration. With n = L y / sigma_bar, d = 1 / (1 + f L), bm = d n and the
// Jacobian [[diag(1 + f L) - f n n^T, j], [n^T, -h]], j = back_rate + db n,
// the rank one term goes by Sherman-Morrison (kappa = 1 / (1 - f n.bm) = 1 /
// sum n y d / sigma_bar, as sum n^2 / L = 1), the border by its Schur
// complement s = kappa bm.j + h. The consistent tangent, from the stress as y
// plus the back stresses, closes to one diagonal and one rank-one term in
// which nothing of the elastic modulus's size cancels but their sum:
//   C_alg = lambda 1 1^T + 2 G V diag((1 + f_k L) d) V^T + 2 G (V w) (V bm)^T,
//   w = 2 G (kappa / s) d {g L back_rate + n [g (h + db_k L) - (1 + f_k L)]},
// with g = dl / sigma_bar and f_k, db_k the kinematic terms' shares of f, db.

struct ReturnPoint {
  double y[6], dl;
  double inv;          // 1 / sigma_bar
  double n[6];         // L y / sigma_bar
  double bk, b, db;    // 2/3 sum C chi; with 2G dl; its derivative
  double back_rate[6];
  double res[7];
  double slope;        // sigma_y'(a_n + dl)
};

// theta, chi and their derivatives of one kinematic term.
__device__ __forceinline__ void decay(const Params& p, int t, double dl, double& theta, double& chi, double& dtheta,
                                      double& dchi) {
  const double gamma = p.termG[t];
  if (gamma == 0.0) {
    theta = 1.0, chi = dl, dtheta = 0.0, dchi = 1.0;
  } else if (p.integration == 0) {
    const double em = expm1(-gamma * dl);
    theta = 1.0 + em;
    chi = -em * p.termGi[t];
    dtheta = -gamma * theta;
    dchi = theta;
  } else {
    theta = 1.0 / (1.0 + gamma * dl);
    chi = theta * dl;
    dtheta = -gamma * theta * theta;
    dchi = theta * theta;
  }
}

// V^T S^-1 t of a tensorial Voigt t.
__device__ __forceinline__ void to_basis(const Params& p, const double t[6], double y[6]) {
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double v = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) v += p.PV[i * 6 + k] * t[i];
    double w = 0.0;
#pragma unroll
    for (int i = 3; i < 6; ++i) w += p.PV[i * 6 + k] * t[i];
    y[k] = v + 2.0 * w;
  }
}
// V y.
__device__ __forceinline__ void from_basis(const Params& p, const double y[6], double t[6]) {
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < 6; ++k) v += p.PV[i * 6 + k] * y[k];
    t[i] = v;
  }
}

// The trial state in the basis: the deviator and the kinematic terms.
template <int NT>
struct ReturnTrial {
  double s[6], a[PointTrial<NT>::kTerms][6];
  double a_n;
};

template <int NT>
__device__ __forceinline__ bool return_evaluate(const Params& p, const ReturnTrial<NT>& T, ReturnPoint& e) {
  double q = 0.0;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    e.n[k] = p.PL[k] * e.y[k];
    q += e.n[k] * e.y[k];
  }
  if (!(q > 0.0) || !isfinite(q)) return false;
  e.inv = rsqrt(q);
  double eq = q * e.inv;
  eq += 0.5 * e.inv * fma(-eq, eq, q);
  double z[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    e.n[k] *= e.inv;
    z[k] = T.s[k];
    e.back_rate[k] = 0.0;
  }
  e.bk = 0.0;
  e.db = 2.0 * p.G;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    if (NT <= 2 || t < p.nterms) {
      double theta, chi, dtheta, dchi;
      decay(p, t, e.dl, theta, chi, dtheta, dchi);
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        z[k] -= theta * T.a[t][k];
        e.back_rate[k] += dtheta * T.a[t][k];
      }
      e.bk += 2.0 / 3.0 * p.termC[t] * chi;
      e.db += 2.0 / 3.0 * p.termC[t] * dchi;
    }
  }
  e.b = e.bk + 2.0 * p.G * e.dl;
#pragma unroll
  for (int k = 0; k < 6; ++k) e.res[k] = e.y[k] - z[k] + e.b * e.n[k];
  const double a = T.a_n + e.dl;
  const double ey = expm1(-p.delta * a);
  e.res[6] = eq - (p.sy0 + p.H * a - p.Q * ey);
  e.slope = p.H + p.Q * p.delta * (1.0 + ey);
  return true;
}

__device__ __forceinline__ double return_inf(const ReturnPoint& e) {
  double m = fabs(e.res[0]);
#pragma unroll
  for (int i = 1; i < 7; ++i) m = fmax(m, fabs(e.res[i]));
  return m;
}
__device__ __forceinline__ double return_norm2(const ReturnPoint& e) {
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < 7; ++i) s += e.res[i] * e.res[i];
  return s;
}

struct ReturnFactor {
  double d[6], bm[6], aj[6];
  double kappa, c, si;  // kappa, f kappa, 1 / s
};

__device__ __forceinline__ double dot6(const double a[6], const double b[6]) {
  return (a[0] * b[0] + a[1] * b[1]) + (a[2] * b[2] + a[3] * b[3]) + (a[4] * b[4] + a[5] * b[5]);
}

__device__ __forceinline__ void return_factor(const Params& p, const ReturnPoint& e, ReturnFactor& r) {
  const double f = e.b * e.inv;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    r.d[k] = 1.0 / (1.0 + f * p.PL[k]);
    r.bm[k] = r.d[k] * e.n[k];
  }
  r.kappa = 1.0 / (e.inv * dot6(r.bm, e.y));
  r.c = f * r.kappa;
  double j[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) j[k] = e.back_rate[k] + e.db * e.n[k];
  const double bj = dot6(r.bm, j);
#pragma unroll
  for (int k = 0; k < 6; ++k) r.aj[k] = r.d[k] * j[k] + r.c * bj * r.bm[k];
  r.si = 1.0 / (r.kappa * bj + e.slope);
}

// C_alg into the record.
__device__ __forceinline__ void return_tangent(const Params& p, const ReturnPoint& e, const ReturnFactor& r,
                                               const PointRecord& rec, int fM) {
  const double g = e.dl * e.inv, fk = e.bk * e.inv, dbk = e.db - 2.0 * p.G;
  const double g2 = 2.0 * p.G, ks = g2 * g2 * r.kappa * r.si;
  double u[6], w[6], vu[6], vb[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const double l = p.PL[k], kin = 1.0 + fk * l;
    w[k] = g2 * (kin * r.d[k]);
    u[k] = ks * r.d[k] * (g * l * e.back_rate[k] + e.n[k] * (g * (e.slope + dbk * l) - kin));
  }
  from_basis(p, u, vu);
  from_basis(p, r.bm, vb);
  const double lame = p.K - 2.0 * p.G / 3.0;
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = i; j < 6; ++j) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < 6; ++k) v += w[k] * p.PV[i * 6 + k] * p.PV[j * 6 + k];
      if (i < 3 && j < 3) v += lame;
      rec.put(fM + i * 6 + j, v + vu[i] * vb[j]);
      if (i != j) rec.put(fM + j * 6 + i, v + vu[j] * vb[i]);
    }
}

// The general law's return of a point that is not plainly elastic
// (general_plastic; in the loading window the elastic branch with the
// tangent at dl = 0): stress and tangent into the record, the closest point
// (y, dl) into its warm fields fW. `warm`: they hold the one of this
// element's last pass, from which the iteration starts where its residual
// is the smaller one; if that does not converge the return runs again from
// the trial state. One loop evaluates every candidate - start, Newton trial,
// polishing step - so that the equations and their factors are in the code
// once. TANGENT = false: the stress alone.
template <int NT, bool TANGENT = true>
__device__ __forceinline__ int return_general(const Params& p, const PointTrial<NT>& P, bool window, bool warm,
                                              const PointRecord& rec, int fS, int fM, int fW) {
  ReturnTrial<NT> T;
  double scale = P.sy;
#pragma unroll
  for (int i = 0; i < 6; ++i) scale = fmax(scale, fmax(fabs(P.s[i]), fabs(P.xi[i])));
  const double eps_scale = kEps * scale;
  const double tol = fmax(1.0e-13 * P.sy, 32.0 * eps_scale);
  to_basis(p, P.s, T.s);
#pragma unroll
  for (int t = 0; t < NT; ++t) to_basis(p, P.a[t], T.a[t]);
  T.a_n = P.a_n;
  // kBack: the last accepted point again, no step from it being accepted;
  // kFinal: again, the polishing step from it being no better.
  enum { kWarm, kTrial, kNewton, kBack, kPolish, kFinal };
  int mode = warm && !window ? kWarm : kTrial;
  bool warmed = mode == kWarm;
  ReturnPoint n;
  ReturnFactor r;
  double base[7], step[7], t = 1.0, r_inf = 0.0, norm2 = 0.0;
  int it = 0, ls = 0;
#pragma unroll
  for (int k = 0; k < 7; ++k) base[k] = warmed ? rec.get(fW + k) : 0.0, step[k] = 0.0;
#pragma unroll 1
  for (;;) {
    // The candidate: base + t step, or the trial state.
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      double trial = T.s[k];
#pragma unroll
      for (int q = 0; q < NT; ++q) trial -= T.a[q][k];
      n.y[k] = mode == kTrial ? trial : base[k] + t * step[k];
    }
    n.dl = mode == kTrial ? 0.0 : fmax(base[6] + t * step[6], 0.0);
    const bool ok = return_evaluate<NT>(p, T, n);
    const double got = return_norm2(n);
    bool restart = false;
    if (mode == kWarm) {
      // At the trial state the residual is the overstress, and 0 in the
      // other rows.
      if (!ok || !(got < P.f * P.f)) {
        mode = kTrial;
        warmed = false;
        continue;
      }
    } else if (mode == kNewton) {
      const double down = 1.0 - 1.0e-4 * t;
      if (!(ok && got <= down * down * norm2)) {
        t *= 0.5;
        if (++ls < 40) continue;
        if (r_inf > 4.0 * tol) {
          restart = true;
        } else {
          mode = kBack;
          t = 0.0;
          continue;
        }
      }
    } else if (mode == kPolish) {
      if (!(ok && return_inf(n) < r_inf)) {
        mode = kFinal;
        t = 0.0;
        continue;
      }
    }
    if (!restart) {
      r_inf = return_inf(n);
      norm2 = got;
      return_factor(p, n, r);
      if (mode >= kPolish || (mode == kTrial && window)) break;
      const bool converged = mode == kBack || r_inf <= tol;
      if (converged && !(r_inf > 4.0 * eps_scale)) break;
      restart = !converged && it++ == 50;
      if (!restart) {
        // Newton's step J step = -R; the one beyond convergence is the
        // polishing step (Plasticity.cpp:431-448).
        const double g = r.c * dot6(r.bm, n.res);
#pragma unroll
        for (int k = 0; k < 6; ++k) step[k] = -(r.d[k] * n.res[k] + g * r.bm[k]);
        step[6] = (dot6(n.n, step) + n.res[6]) * r.si;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          step[k] -= r.aj[k] * step[6];
          base[k] = n.y[k];
        }
        base[6] = n.dl;
        mode = converged ? kPolish : kNewton;
        t = 1.0;
        ls = 0;
        continue;
      }
    }
    if (!warmed) return kFailReturn;
    warmed = false;
    mode = kTrial;
    it = 0;
  }
  double m[6];
  from_basis(p, n.n, m);  // S m
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    if (!window) rec.put(fW + k, n.y[k]);
    rec.put(fS + k, P.s[k] - 2.0 * p.G * n.dl * m[k] + (k < 3 ? p.K * P.vol : 0.0));
  }
  if (!window) rec.put(fW + 6, n.dl);
  if (TANGENT) return_tangent(p, n, r, rec, fM);
  return 0;
}

// The J2 law's elastic branch inside the loading window.
__device__ __forceinline__ void return_window_radial(const Params& p, const PointTrial<-1>& P, const PointRecord& rec,
                                                     int fS, int fM) {
#pragma unroll
  for (int i = 0; i < 6; ++i) rec.put(fS + i, P.s[i] + (i < 3 ? p.K * P.vol : 0.0));
  const double slope = p.H + p.Q * p.delta * (1.0 + P.ey);
  const double f = 2.0 * p.G / (1.0 + (slope + p.Hkin) / (3.0 * p.G));
  const double inv = 1.0 / P.eq, lame = p.K - 2.0 * p.G / 3.0;
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const double el = i < 3 ? (j < 3 ? lame : 0.0) + (i == j ? 2.0 * p.G : 0.0) : (i == j ? p.G : 0.0);
      rec.put(fM + i * 6 + j, el - f * (P.xi[i] * inv) * (P.xi[j] * inv));
    }
}

// The plastic J2 return (radial_return): stress and tangent into the record,
// the flow direction and dgamma into its warm fields.
template <bool TANGENT = true>
__device__ __forceinline__ int return_radial(const Params& p, const PointTrial<-1>& T, const PointRecord& rec, int fS,
                                             int fM, int fW) {
  const double g = p.G, k = p.K, hk = p.Hkin;
  const double sq23 = 0.816496580927726;
  const double stiff = 2.0 * g + 2.0 / 3.0 * hk;
  double ey = T.ey;
  double dgamma = T.f / (stiff + 2.0 / 3.0 * (p.H + p.Q * p.delta * (1.0 + ey)));
  if (p.Q != 0.0) {
    dgamma = 0.0;
    bool converged = false;
#pragma unroll 1
    for (int it = 0; it <= 60; ++it) {
      const double a = T.a_n + sq23 * dgamma;
      ey = expm1(-p.delta * a);
      const double res = T.eq - stiff * dgamma - sq23 * (p.sy0 + p.H * a - p.Q * ey);
      if (fabs(res) <= 1.0e-13 * T.sy || (it == 60 && fabs(res) <= 8.0 * kEps * T.eq)) {
        converged = true;
        break;
      }
      if (it < 60) dgamma += res / (stiff + 2.0 / 3.0 * (p.H + p.Q * p.delta * (1.0 + ey)));
    }
    if (!converged) return kFailReturn;
  }
  const double slope = p.H + p.Q * p.delta * (1.0 + ey);
  double n[6];
  const double inv = 1.0 / T.eq;
#pragma unroll
  for (int i = 0; i < 6; ++i) n[i] = T.xi[i] * inv;
  const double drop = 2.0 * g * dgamma * inv;
  const double theta = 1.0 - drop;
  const double theta_bar = 1.0 / (1.0 + (slope + hk) / (3.0 * g)) - drop;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    rec.put(fS + i, T.s[i] - 2.0 * g * dgamma * n[i] + (i < 3 ? k * T.vol : 0.0));
    rec.put(fW + i, n[i]);
#pragma unroll
    for (int j = 0; j < (TANGENT ? 6 : 0); ++j) {
      const double el = i < 3 ? (j < 3 ? k - 2.0 * g * theta / 3.0 : 0.0) + (i == j ? 2.0 * g * theta : 0.0)
                              : (i == j ? g * theta : 0.0);
      rec.put(fM + i * 6 + j, el - 2.0 * g * theta_bar * (n[i] * n[j]));
    }
  }
  rec.put(fW + 6, dgamma);
  return 0;
}

// The converged point's state and energy: the committed state where it is
// elastic, the return's update from the closest point in the record.
// flag: 0 elastic, 1 plastic, 2 elastic inside the loading window.
template <int NT>
__device__ __forceinline__ double point_finish(const Params& p, const double strain[6], int flag,
                                               const PointRecord& rec, int fW, const double* state, double* trial,
                                               int64_t stride) {
  const int nt = term_count<NT>(p);
  double ep[6], beta[6], a[PointTrial<NT>::kTerms][6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    ep[i] = state[(kFieldEp + i) * stride];
    beta[i] = state[(kFieldBeta + i) * stride];
  }
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int i = 0; i < 6; ++i) a[t][i] = (NT <= 2 || t < nt) ? state[(kFieldAlpha + 6 * t + i) * stride] : 0.0;
  double eq = state[field_eqps(nt) * stride];
  if (flag == 1) {
    const double dl = rec.get(fW + 6);
    double xi[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) xi[i] = rec.get(fW + i);
    if (NT < 0) {
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        ep[i] += (i < 3 ? 1.0 : 2.0) * dl * xi[i];
        beta[i] += 2.0 / 3.0 * p.Hkin * dl * xi[i];
      }
      eq += 0.816496580927726 * dl;
    } else {
      double n[6], m[6], q = 0.0;  // the flow direction S m
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        n[k] = p.PL[k] * xi[k];
        q += n[k] * xi[k];
      }
      const double inv = 1.0 / sqrt(q);
      from_basis(p, n, m);
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        m[i] *= inv;
        ep[i] += (i < 3 ? 1.0 : 2.0) * dl * m[i];
        beta[i] = 0.0;
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        if (NT <= 2 || t < nt) {
          double theta, chi, dtheta, dchi;
          decay(p, t, dl, theta, chi, dtheta, dchi);
          const double f = 2.0 / 3.0 * p.termC[t] * chi;
#pragma unroll
          for (int i = 0; i < 6; ++i) {
            a[t][i] = theta * a[t][i] + f * m[i];
            beta[i] += a[t][i];
          }
        }
      }
      eq += dl;
    }
  }
  double el[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    el[i] = strain[i] - ep[i];
    trial[(kFieldEp + i) * stride] = ep[i];
    trial[(kFieldBeta + i) * stride] = beta[i];
  }
  const double vol = el[0] + el[1] + el[2];
  double energy = 0.5 * p.K * vol * vol + p.G * dev_norm2(el) + isotropic_energy_of(p, eq);
  if (NT < 0) {
    double o = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) o += (i < 3 ? 1.0 : 0.5) * ep[i] * ep[i];
    energy += p.Hkin / 3.0 * o;
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    if (NT <= 2 || t < nt) {
      const double n = tnorm(a[t]);
      energy += 0.75 * n * n / p.termC[t];
#pragma unroll
      for (int i = 0; i < 6; ++i) trial[(kFieldAlpha + 6 * t + i) * stride] = a[t][i];
    }
  }
  trial[field_eqps(nt) * stride] = eq;
  trial[field_loading(nt) * stride] = flag ? 1.0 : 0.0;
  return energy;
}

}  // namespace sbk
