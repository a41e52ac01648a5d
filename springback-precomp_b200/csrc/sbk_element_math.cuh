// What the element kernels share: the constants of the local iteration
// (src/fem/IncompatibleModes.hpp:98-127), 3 x 3 algebra and the group sum.
#pragma once

#include <cuda_runtime.h>

namespace sbk {

constexpr int kMaxLocal = 25;
constexpr double kFullStepReduction = 1.0 - 1.0e-4;
constexpr int kMaxLineSearch = 8;
constexpr double kLineSearchRatio = 0.5;
constexpr double kLocalShift = 1.0e-3;
constexpr double kLocalMarquardt = 1.0e-6;
constexpr double kLocalTolerance = 1.0e-8;
constexpr double kLocalRoundOff = 1.0e-13;

__device__ __forceinline__ double det3(const double m[9]) {
  return m[0] * (m[4] * m[8] - m[7] * m[5]) - m[3] * (m[1] * m[8] - m[7] * m[2]) +
         m[6] * (m[1] * m[5] - m[4] * m[2]);
}
__device__ __forceinline__ void inv3(const double m[9], double out[9]) {
  out[0] = m[4] * m[8] - m[5] * m[7];
  out[3] = m[5] * m[6] - m[3] * m[8];
  out[6] = m[3] * m[7] - m[4] * m[6];
  const double det = m[0] * out[0] + m[1] * out[3] + m[2] * out[6];
  const double inv = 1.0 / det;
  out[1] = m[2] * m[7] - m[1] * m[8];
  out[4] = m[0] * m[8] - m[2] * m[6];
  out[7] = m[1] * m[6] - m[0] * m[7];
  out[2] = m[1] * m[5] - m[2] * m[4];
  out[5] = m[2] * m[3] - m[0] * m[5];
  out[8] = m[0] * m[4] - m[1] * m[3];
#pragma unroll
  for (int i = 0; i < 9; ++i) out[i] *= inv;
}

// Reduce-scatter of G values over the G lanes of a group: lane l returns the
// group sum of v[l]. Fixed pairing, so the result is deterministic.
template <int G>
__device__ __forceinline__ double reduce_scatter(double (&v)[G], int lane, unsigned mask) {
  double cur[G];
#pragma unroll
  for (int i = 0; i < G; ++i) cur[i] = v[i];
#pragma unroll
  for (int half = G / 2; half >= 1; half >>= 1) {
    const bool upper = (lane & half) != 0;
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const double send = upper ? cur[j] : cur[half + j];
      const double keep = upper ? cur[half + j] : cur[j];
      cur[j] = keep + __shfl_xor_sync(mask, send, half, G);
    }
  }
  return cur[0];
}

// ---- 9 x 9 algebra of one lane ----

// Cholesky (lower, in place); false at the first non-positive pivot.
static __device__ __noinline__ bool llt9(double* a) {
  _Pragma("unroll 1") for (int k = 0; k < 9; ++k) {
    double x = a[k * 9 + k];
    _Pragma("unroll 1") for (int j = 0; j < k; ++j) x -= a[k * 9 + j] * a[k * 9 + j];
    if (x <= 0.0) return false;
    a[k * 9 + k] = sqrt(x);
    _Pragma("unroll 1") for (int i = k + 1; i < 9; ++i) {
      double v = a[i * 9 + k];
      _Pragma("unroll 1") for (int j = 0; j < k; ++j) v -= a[i * 9 + j] * a[k * 9 + j];
      a[i * 9 + k] = v / a[k * 9 + k];
    }
  }
  return true;
}

static __device__ __noinline__ void llt9_solve(const double* l, const double* b, double* x) {
  double y[9];
  _Pragma("unroll 1") for (int i = 0; i < 9; ++i) {
    double v = b[i];
    _Pragma("unroll 1") for (int j = 0; j < i; ++j) v -= l[i * 9 + j] * y[j];
    y[i] = v / l[i * 9 + i];
  }
  _Pragma("unroll 1") for (int i = 8; i >= 0; --i) {
    double v = y[i];
    _Pragma("unroll 1") for (int j = i + 1; j < 9; ++j) v -= l[j * 9 + i] * y[j];
    y[i] = v / l[i * 9 + i];
  }
  _Pragma("unroll 1") for (int i = 0; i < 9; ++i) x[i] = y[i];
}

// Smallest eigenvalue and largest |eigenvalue| of a symmetric 9x9 (cyclic
// Jacobi on a copy in `a`, destroyed).
static __device__ __noinline__ void sym_eig9(double* a, double* lo, double* top) {
  _Pragma("unroll 1") for (int sweep = 0; sweep < 60; ++sweep) {
    double off = 0.0, diag = 0.0;
    _Pragma("unroll 1") for (int p = 0; p < 9; ++p) {
      diag += a[p * 9 + p] * a[p * 9 + p];
      _Pragma("unroll 1") for (int q = p + 1; q < 9; ++q) off += a[p * 9 + q] * a[p * 9 + q];
    }
    if (off == 0.0 || off <= 1.0e-36 * diag) break;
    _Pragma("unroll 1") for (int p = 0; p < 8; ++p)
      _Pragma("unroll 1") for (int q = p + 1; q < 9; ++q) {
        const double apq = a[p * 9 + q];
        if (apq == 0.0) continue;
        const double theta = (a[q * 9 + q] - a[p * 9 + p]) / (2.0 * apq);
        const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        const double cs = 1.0 / sqrt(t * t + 1.0);
        const double sn = t * cs;
        _Pragma("unroll 1") for (int k = 0; k < 9; ++k) {
          const double akp = a[k * 9 + p], akq = a[k * 9 + q];
          a[k * 9 + p] = cs * akp - sn * akq;
          a[k * 9 + q] = sn * akp + cs * akq;
        }
        _Pragma("unroll 1") for (int k = 0; k < 9; ++k) {
          const double apk = a[p * 9 + k], aqk = a[q * 9 + k];
          a[p * 9 + k] = cs * apk - sn * aqk;
          a[q * 9 + k] = sn * apk + cs * aqk;
        }
      }
  }
  double mn = a[0], mx = fabs(a[0]);
  _Pragma("unroll 1") for (int i = 1; i < 9; ++i) {
    mn = fmin(mn, a[i * 9 + i]);
    mx = fmax(mx, fabs(a[i * 9 + i]));
  }
  *lo = mn;
  *top = mx;
}

// Partial-pivoting LU solve of a 9x9 (in place), x = A^-1 b.
static __device__ __noinline__ void plu9_solve(double* a, int* perm, const double* b, double* x) {
  _Pragma("unroll 1") for (int k = 0; k < 9; ++k) {
    int p = k;
    double big = fabs(a[k * 9 + k]);
    _Pragma("unroll 1") for (int i = k + 1; i < 9; ++i)
      if (fabs(a[i * 9 + k]) > big) {
        big = fabs(a[i * 9 + k]);
        p = i;
      }
    perm[k] = p;
    if (big != 0.0) {
      if (p != k)
        _Pragma("unroll 1") for (int j = 0; j < 9; ++j) {
          const double t = a[k * 9 + j];
          a[k * 9 + j] = a[p * 9 + j];
          a[p * 9 + j] = t;
        }
      const double inv = 1.0 / a[k * 9 + k];
      _Pragma("unroll 1") for (int i = k + 1; i < 9; ++i) a[i * 9 + k] *= inv;
    }
    _Pragma("unroll 1") for (int i = k + 1; i < 9; ++i)
      _Pragma("unroll 1") for (int j = k + 1; j < 9; ++j) a[i * 9 + j] -= a[i * 9 + k] * a[k * 9 + j];
  }
  double y[9];
  _Pragma("unroll 1") for (int i = 0; i < 9; ++i) y[i] = b[i];
  _Pragma("unroll 1") for (int k = 0; k < 9; ++k)
    if (perm[k] != k) {
      const double t = y[k];
      y[k] = y[perm[k]];
      y[perm[k]] = t;
    }
  _Pragma("unroll 1") for (int i = 1; i < 9; ++i)
    _Pragma("unroll 1") for (int j = 0; j < i; ++j) y[i] -= a[i * 9 + j] * y[j];
  _Pragma("unroll 1") for (int i = 8; i >= 0; --i) {
    _Pragma("unroll 1") for (int j = i + 1; j < 9; ++j) y[i] -= a[i * 9 + j] * y[j];
    y[i] /= a[i * 9 + i];
  }
  _Pragma("unroll 1") for (int i = 0; i < 9; ++i) x[i] = y[i];
}

}  // namespace sbk
