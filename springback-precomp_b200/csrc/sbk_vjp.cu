// The shape derivative lambda^T d f* / d X of the converged elements of a
// tile launch, from the records the tile kernel leaves for the condensation
// (the derivation is at vjp_point, sbk_element.cu): the modes' cotangent mu =
// -K_aa^-T K_ua^T lambda, then every point's reverse chain from r = w F S [G |
// G~] to X.
//
// Eight lanes an element, a lane the points l, l + 8, ...; sums over the
// points by shuffles. With the gradients as products of the Jacobians (Q =
// (Lambda dN^T) J^-1, K_ua^T lambda = w (F V + Q S) g) no node's gradient is
// formed. The local iteration is the tile kernel's; as one kernel a warp of
// four elements, it was 1,011 us for 8,192 frozen elements, of which the
// chain is now 30.
#include <cuda_runtime.h>

#include "sbk_element.h"
#include "sbk_element_math.cuh"
#include "sbk_tile.h"

namespace sbk {
namespace {

constexpr int kElements = 16;

__device__ __forceinline__ void mul33(const double a[9], const double b[9], double c[9]) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) c[i * 3 + j] = a[i * 3] * b[j] + a[i * 3 + 1] * b[3 + j] + a[i * 3 + 2] * b[6 + j];
}

__device__ __forceinline__ void node_dn(const Params& p, int q, int n, double dn[3]) {
  const double sx = ((n + 1) >> 1) & 1 ? 1.0 : -1.0, sy = (n >> 1) & 1 ? 1.0 : -1.0, sz = n >> 2 ? 1.0 : -1.0;
  const double fx = 1.0 + p.qp[q][0] * sx, fy = 1.0 + p.qp[q][1] * sy, fz = 1.0 + p.qp[q][2] * sz;
  dn[0] = 0.125 * sx * fy * fz;
  dn[1] = 0.125 * sy * fx * fz;
  dn[2] = 0.125 * sz * fx * fy;
}

// v dN^T: sum over the nodes of v_a (3) times dN_a.
__device__ __forceinline__ void nodes_dn(const Params& p, int q, const double* v, double out[9]) {
#pragma unroll
  for (int i = 0; i < 9; ++i) out[i] = 0.0;
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    double dn[3];
    node_dn(p, q, n, dn);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int c = 0; c < 3; ++c) out[i * 3 + c] += v[3 * n + i] * dn[c];
  }
}

struct Point {
  double F[9], S[9], Ji[9], gt[9];  // gt: G~(i, m) at i * 3 + m
  double w, ratio;
};

__device__ __forceinline__ void load_point(const Params& p, const double* R, const double* J0, int q, Point& x) {
  const int nq = p.nq;
  double s[6];
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    x.F[i] = R[(kCondH + i) * nq] + (i % 4 == 0 ? 1.0 : 0.0);
    x.Ji[i] = R[(kCondGeo + i) * nq];
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) s[i] = R[(kCondS + i) * nq];
  x.S[0] = s[0], x.S[1] = s[3], x.S[2] = s[5], x.S[3] = s[3], x.S[4] = s[1], x.S[5] = s[4], x.S[6] = s[5], x.S[7] = s[4],
  x.S[8] = s[2];
  x.w = R[kCondW * nq];
  x.ratio = R[(kCondGeo + 9) * nq];
#pragma unroll
  for (int m = 0; m < 3; ++m)
#pragma unroll
    for (int i = 0; i < 3; ++i) x.gt[i * 3 + m] = x.ratio * (-2.0 * p.qp[q][m]) * J0[m * 3 + i];
}

__global__ void __launch_bounds__(8 * kElements)
    vjp_tile_kernel(const __grid_constant__ Params p, const __grid_constant__ TileArgs a,
                    const double* __restrict__ cond, const double* __restrict__ lambda, double* __restrict__ out) {
  __shared__ double nodes[kElements][48];  // lambda, u
  __shared__ double modes[kElements][18];  // mu, alpha
  const int k = threadIdx.x >> 3, lane = threadIdx.x & 7, nq = p.nq;
  const int64_t at = (int64_t)blockIdx.x * kElements + k, e = a.begin + at;
  const bool live = e < a.end && a.code[e < a.end ? e : a.begin] == 0;
  const double* rec = cond + (size_t)(live ? at : 0) * cond_record(nq);
  const double* own = rec + kCondPoint * nq;
  if (live) {
    const int64_t node = a.conn[e * 8 + lane];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      nodes[k][3 * lane + i] = lambda[node * 3 + i];
      nodes[k][24 + 3 * lane + i] = a.u[node * 3 + i];
    }
    for (int i = lane; i < 9; i += 8) modes[k][9 + i] = a.alpha_out[e * 9 + i];
  }
  __syncwarp();
  double J0[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) J0[i] = live ? own[kCondJ0 + i] : 0.0;
  // K_ua^T lambda.
  double b[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) b[i] = 0.0;
#pragma unroll 1
  for (int q = live ? lane : nq; q < nq; q += 8) {
    const double* R = rec + q;
    Point x;
    load_point(p, R, J0, q, x);
    double L[9], Q[9], FtQ[9];
    nodes_dn(p, q, nodes[k], L);
    mul33(L, x.Ji, Q);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) FtQ[i * 3 + j] = x.F[i] * Q[j] + x.F[3 + i] * Q[3 + j] + x.F[6 + i] * Q[6 + j];
    const double en[6] = {FtQ[0], FtQ[4], FtQ[8], FtQ[1] + FtQ[3], FtQ[5] + FtQ[7], FtQ[2] + FtQ[6]};
    double v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
      for (int d = 0; d < 6; ++d) v[d] += en[c] * R[(kCondM + c * 6 + d) * nq];
    const double V[9] = {v[0], v[3], v[5], v[3], v[1], v[4], v[5], v[4], v[2]};
    double N[9], QS[9];
    mul33(x.F, V, N);
    mul33(Q, x.S, QS);
#pragma unroll
    for (int i = 0; i < 9; ++i) N[i] = x.w * (N[i] + QS[i]);
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        b[3 * m + i] += N[i * 3] * x.gt[m] + N[i * 3 + 1] * x.gt[3 + m] + N[i * 3 + 2] * x.gt[6 + m];
  }
#pragma unroll
  for (int i = 0; i < 9; ++i)
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) b[i] += __shfl_xor_sync(0xffffffffu, b[i], o, 8);
  if (live && lane == 0) {
    // mu = -K_aa^-T b with K_aa = L U in pivot order: U^T forward, L^T
    // backward.
    int row[9], col[9];
    double y[9];
#pragma unroll
    for (int s = 0; s < 9; ++s) {
      const int perm = (int)own[kCondPerm + s];
      row[s] = perm >> 4;
      col[s] = perm & 15;
    }
#pragma unroll
    for (int s = 0; s < 9; ++s) {
      double v = b[0];
#pragma unroll
      for (int i = 1; i < 9; ++i) v = col[s] == i ? b[i] : v;
#pragma unroll
      for (int j = 0; j < s; ++j) v -= own[kCondLu + j * 9 + s] * y[j];
      y[s] = v * own[kCondPiv + s];
    }
#pragma unroll
    for (int s = 8; s >= 0; --s) {
#pragma unroll
      for (int j = s + 1; j < 9; ++j) y[s] -= own[kCondLu + j * 9 + s] * y[j];
      modes[k][row[s]] = -y[s];
    }
  }
  __syncwarp();
  double xb[24], j0b[9];
#pragma unroll
  for (int i = 0; i < 24; ++i) xb[i] = 0.0;
#pragma unroll
  for (int i = 0; i < 9; ++i) j0b[i] = 0.0;
#pragma unroll 1
  for (int q = live ? lane : nq; q < nq; q += 8) {
    const double* R = rec + q;
    const double* mu = modes[k];
    Point x;
    load_point(p, R, J0, q, x);
    // Q = [Lambda | mu] [G | G~]^T, phi = w (F S) . Q.
    double L[9], Q[9], FS[9], phi = 0.0;
    nodes_dn(p, q, nodes[k], L);
    mul33(L, x.Ji, Q);
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Q[i * 3 + j] += mu[3 * m + i] * x.gt[j * 3 + m];
    mul33(x.F, x.S, FS);
#pragma unroll
    for (int i = 0; i < 9; ++i) phi += FS[i] * Q[i];
    phi *= x.w;
    // Sbar = w sym(F^T Q), Ebar = M^T Sbar, Fbar = w Q S + F Ebar.
    double FtQ[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        FtQ[i * 3 + j] = x.w * (x.F[i] * Q[j] + x.F[3 + i] * Q[3 + j] + x.F[6 + i] * Q[6 + j]);
    const double sb[6] = {FtQ[0], FtQ[4], FtQ[8], FtQ[1] + FtQ[3], FtQ[5] + FtQ[7], FtQ[2] + FtQ[6]};
    double v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
      for (int d = 0; d < 6; ++d) v[d] += sb[c] * R[(kCondM + c * 6 + d) * nq];
    const double Eb[9] = {v[0], v[3], v[5], v[3], v[1], v[4], v[5], v[4], v[2]};
    double Fb[9], QS[9];
    mul33(x.F, Eb, Fb);
    mul33(Q, x.S, QS);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      Fb[i] += x.w * QS[i];
      FS[i] *= x.w;
    }
    // Gbar_a = (w F S)^T lambda_a + Fbar^T u_a; K1 = sum_a dN_a Gbar_a^T =
    // (Lambda dN^T)^T (w F S) + (U dN^T)^T Fbar.
    double D[9], K1[9];
    nodes_dn(p, q, nodes[k] + 24, D);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        K1[c * 3 + j] = L[c] * FS[j] + L[3 + c] * FS[3 + j] + L[6 + c] * FS[6 + j] + D[c] * Fb[j] + D[3 + c] * Fb[3 + j] +
                        D[6 + c] * Fb[6 + j];
    double rr = 0.0, K2[9];
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double gbm = FS[i] * mu[3 * m] + FS[3 + i] * mu[3 * m + 1] + FS[6 + i] * mu[3 * m + 2] +
                           Fb[i] * mu[9 + 3 * m] + Fb[3 + i] * mu[9 + 3 * m + 1] + Fb[6 + i] * mu[9 + 3 * m + 2];
        const double cm = -2.0 * p.qp[q][m];
        rr += gbm * cm * J0[m * 3 + i];
        K2[m * 3 + i] = cm * gbm;
      }
    // Jbar = (phi - ratio R) J^-T - J^-T K1 J^-T, J0bar likewise.
    double T1[9], T2[9], Jb[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        T1[i * 3 + j] = x.Ji[i] * K1[j] + x.Ji[3 + i] * K1[3 + j] + x.Ji[6 + i] * K1[6 + j];
        T2[i * 3 + j] = J0[i] * K2[j] + J0[3 + i] * K2[3 + j] + J0[6 + i] * K2[6 + j];
      }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        Jb[i * 3 + c] = (phi - x.ratio * rr) * x.Ji[c * 3 + i] -
                        (T1[i * 3] * x.Ji[c * 3] + T1[i * 3 + 1] * x.Ji[c * 3 + 1] + T1[i * 3 + 2] * x.Ji[c * 3 + 2]);
        j0b[i * 3 + c] += x.ratio * rr * J0[c * 3 + i] -
                          x.ratio * (T2[i * 3] * J0[c * 3] + T2[i * 3 + 1] * J0[c * 3 + 1] + T2[i * 3 + 2] * J0[c * 3 + 2]);
      }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      double dn[3];
      node_dn(p, q, n, dn);
#pragma unroll
      for (int i = 0; i < 3; ++i) xb[3 * n + i] += Jb[i * 3] * dn[0] + Jb[i * 3 + 1] * dn[1] + Jb[i * 3 + 2] * dn[2];
    }
  }
  // Sums over the lanes: node n's three in lane n, J0bar in every lane.
  double mine[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double v[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) v[n] = xb[3 * n + i];
    mine[i] = reduce_scatter<8>(v, lane, 0xffffffffu);
  }
#pragma unroll
  for (int i = 0; i < 9; ++i)
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) j0b[i] += __shfl_xor_sync(0xffffffffu, j0b[i], o, 8);
  if (live) {
    const double d0[3] = {((lane + 1) >> 1) & 1 ? 0.125 : -0.125, (lane >> 1) & 1 ? 0.125 : -0.125,
                          lane >> 2 ? 0.125 : -0.125};
#pragma unroll
    for (int i = 0; i < 3; ++i)
      out[e * 24 + 3 * lane + i] = mine[i] + j0b[i * 3] * d0[0] + j0b[i * 3 + 1] * d0[1] + j0b[i * 3 + 2] * d0[2];
  }
}

}  // namespace

int launch_vjp_tile(const Params& p, const TileArgs& a, const TileScratch& s, const double* lambda, double* out,
                    cudaStream_t stream) {
  const int64_t n = a.end - a.begin;
  vjp_tile_kernel<<<(unsigned)((n + kElements - 1) / kElements), 8 * kElements, 0, stream>>>(p, a, s.cond, lambda, out);
  return (int)cudaGetLastError();
}

}  // namespace sbk
