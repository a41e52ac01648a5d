// Stress recovery at the end of a step (incompatible_elastoplastic_stress,
// IncompatibleModes.cpp:602-664; for the standard Hex8 elastoplastic_stress,
// Elastoplastic.cpp:342-430; called for every element by the forming driver,
// Forming.cpp:1266-1281): the kinematics at the committed modes without a local
// iteration, every point's return from its committed state (after a commit an
// elastic check that reproduces it), and per element the point averages of the
// Cauchy, second Piola-Kirchhoff and Kirchhoff stresses and the log strain,
// the von Mises stress of the average Cauchy stress, the largest accumulated
// plastic strain and strain component and the smallest det F.
//
// A thread a point, the points of up to 32 elements a block; the point values
// meet in shared memory, where a thread a field sums them in point order, as
// the reference does. Nothing of a point is indexed at run time and a point
// that yields is a call of its own, so that the common road fits 128 registers
// and two blocks of eight warps an SM. Measured (20,000 elements, Hill48 +
// two-term Chaboche): 329 us with a group of lanes and a 10 KB record an
// element, 50 us so (72 us with the return's registers on the common road).
#include <cuda_runtime.h>

#include "sbk_element.h"
#include "sbk_smem.h"
#include "sbk_tile_point.cuh"

namespace sbk {
namespace {

constexpr int kThreads = 256;
constexpr int kElements = 32;
constexpr int kOut = 27;   // cauchy 6, pk2 6, kirchhoff 6, log strain 6, max strain, det F, eqps
// F T F^T of a tensorial Voigt T.
__device__ __forceinline__ void push_forward(const double F[9], const double t[6], double out[6]) {
  const double T[9] = {t[0], t[3], t[5], t[3], t[1], t[4], t[5], t[4], t[2]};
  double A[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) A[i * 3 + j] = F[i * 3] * T[j] + F[i * 3 + 1] * T[3 + j] + F[i * 3 + 2] * T[6 + j];
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int i = c < 3 ? c : c - 3, j = c < 3 ? c : (c - 2) % 3;
    out[c] = A[i * 3] * F[j * 3] + A[i * 3 + 1] * F[j * 3 + 1] + A[i * 3 + 2] * F[j * 3 + 2];
  }
}

// A point's values into its record.
__device__ __forceinline__ void stress_values(const Params& p, const double h[9], const LogKin& L,
                                              const double strain[6], const double t[6], double own, double eqps,
                                              const PointRecord& rec) {
  const double F[9] = {h[0] + 1.0, h[1], h[2], h[3], h[4] + 1.0, h[5], h[6], h[7], h[8] + 1.0};
  double jac = 1.0;
  if (p.kinematics == SBK_FINITE_LOGARITHMIC) {
    double tp[6], pk[6], tau[6];
    rotate_in(L.q, t, tp);
#pragma unroll
    for (int i = 0; i < 6; ++i) tp[i] *= L.first[i];
    rotate_out(L.q, tp, pk);
    push_forward(F, pk, tau);
    const double volume = exp(strain[0] + strain[1] + strain[2]);
    jac = det3(F);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      rec.put(i, tau[i] / volume);
      rec.put(6 + i, pk[i]);
      rec.put(12 + i, tau[i]);
      rec.put(18 + i, i < 3 ? strain[i] : 0.5 * strain[i]);
    }
  } else {
    double cauchy[6];
    if (p.kinematics == SBK_FINITE) {
      push_forward(F, t, cauchy);
      jac = det3(F);
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      rec.put(i, p.kinematics == SBK_FINITE ? cauchy[i] / jac : t[i]);
      rec.put(6 + i, t[i]);
      rec.put(12 + i, 0.0);
      rec.put(18 + i, 0.0);
    }
  }
  rec.put(24, own);
  rec.put(25, jac);
  rec.put(26, eqps);
}

// The displacement gradient of a point at its element's staged nodes and modes.
__device__ __forceinline__ bool stress_gradient(const Params& p, int q, const double* nodes, double h[9], double& w) {
  PointGeometry G;
  if (!point_geometry(p, q, nodes, nodes + 24, G)) return false;
  w = G.w;
#pragma unroll
  for (int i = 0; i < 9; ++i) h[i] = G.du[i];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const double f = G.ratio * (-2.0 * p.qp[q][m]);
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) h[i * 3 + j] += nodes[48 + 3 * m + i] * (f * G.j0i[m * 3 + j]);
  }
  return true;
}

// A point that yields from its committed state, start to finish, so that the
// common road keeps nothing across a call.
template <int NT>
__device__ __noinline__ int stress_plastic(const Params& p, int q, const double* nodes, double shift, double own,
                                           const double* state, int64_t stride, const PointRecord rec) {
  constexpr int kWarm = 6;  // the return's record, over the outputs: stress 6, closest point 7
  double h[9], strain[6], w;
  stress_gradient(p, q, nodes, h, w);
  LogKin L;
#pragma unroll
  for (int i = 0; i < 9; ++i) L.q[i] = i % 4 == 0 ? 1.0 : 0.0;
  point_strain(p, h, L, strain);
#pragma unroll
  for (int i = 0; i < 3; ++i) strain[i] += shift;
  PointTrial<NT> T;
  point_trial<NT>(p, strain, state, stride, T);
  int code;
  double eqps = T.a_n;
  if constexpr (NT < 0) {
    code = return_radial<false>(p, T, rec, 0, 0, kWarm);
    eqps += 0.816496580927726 * rec.get(kWarm + 6);
  } else {
    code = return_general<NT, false>(p, T, false, false, rec, 0, 0, kWarm);
    eqps += rec.get(kWarm + 6);
  }
  if (code) return code;
  double t[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) t[i] = rec.get(i);
  stress_values(p, h, L, strain, t, own, eqps, rec);
  return 0;
}

template <int NT>
__global__ void __launch_bounds__(kThreads, 2)
    stress_kernel(const __grid_constant__ Params p, int64_t ne, int elements, const double* __restrict__ coords,
                  const int32_t* __restrict__ conn, const double* __restrict__ u, const double* __restrict__ state,
                  const double* __restrict__ alpha_n, double* __restrict__ out, int32_t* __restrict__ code,
                  int32_t* __restrict__ first_failure) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int fail[kElements];
  const int tid = threadIdx.x, nq = p.nq, np = (elements * nq) | 1;
  double* nodes = smem;  // coordinates 24, displacements 24, modes 9 an element
  double* values = smem + 57 * elements;  // kOut x np
  const int64_t e0 = (int64_t)blockIdx.x * elements;
  const int here = (int)(ne - e0 < elements ? ne - e0 : elements);
  for (int k = tid; k < here; k += kThreads) fail[k] = 0x7fffffff;
  __syncthreads();
  for (int i = tid; i < here * 8; i += kThreads) {
    const int k = i >> 3, n = i & 7;
    const int64_t node = conn[(e0 + k) * 8 + n];
    double* X = nodes + 57 * k + 3 * n;
    if (p.num_nodes > 0 && (node < 0 || node >= p.num_nodes)) {
      fail[k] = SBK_EL_BAD_NODE;
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        X[c] = coords[node * 3 + c];
        X[24 + c] = u[node * 3 + c];
      }
    }
  }
  // The standard Hex8 has no modes: its kinematics are at zero modes.
  for (int i = tid; i < here * 9; i += kThreads)
    nodes[57 * (i / 9) + 48 + i % 9] = (alpha_n && !p.element) ? alpha_n[e0 * 9 + i] : 0.0;
  __syncthreads();
  const int k = tid / nq, q = tid - k * nq, pt = tid;
  bool live = k < here && fail[k < here ? k : 0] != SBK_EL_BAD_NODE;
  double h[9], strain[6], w = 0.0, shift = 0.0;
  LogKin L;
  if (live && !stress_gradient(p, q, nodes + 57 * k, h, w)) {
    atomicMin(&fail[k], SBK_EL_MESH_INVERTED);
    live = false;
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < 9; ++i) L.q[i] = i % 4 == 0 ? 1.0 : 0.0;
    const int bad = point_strain(p, h, L, strain);
    if (bad) {
      atomicMin(&fail[k], (1 << 16) | (q << 8) | bad);
      live = false;
    }
  }
  // The standard Hex8 with mean dilatation (kinematics_of,
  // Elastoplastic.cpp:140-167): every point's trace replaced by the volume
  // average; the largest strain component stays the point's own.
  double own = 0.0;
  if (live)
#pragma unroll
    for (int i = 0; i < 6; ++i) own = fmax(own, fabs(i < 3 ? strain[i] : 0.5 * strain[i]));
  if (p.averaged) {
    if (live) {
      values[pt] = w;
      values[np + pt] = w * (strain[0] + strain[1] + strain[2]);
    }
    __syncthreads();
    live = live && fail[k] == 0x7fffffff;
    if (live) {
      double volume = 0.0, trace = 0.0;
      for (int j = 0; j < nq; ++j) {
        volume += values[k * nq + j];
        trace += values[np + k * nq + j];
      }
      shift = (trace / volume - (strain[0] + strain[1] + strain[2])) / 3.0;
      strain[0] += shift;
      strain[1] += shift;
      strain[2] += shift;
    }
    __syncthreads();
  }
  if (live) {
    const int64_t at = (e0 + k) * nq + q;
    const PointRecord rec{values + pt, np};
    PointTrial<NT> T;
    point_trial<NT>(p, strain, state + at, ne * nq, T);
    int bad = 0;
    if (NT >= 0 && !isfinite(T.f)) {
      bad = kFailReturn;
    } else if (point_elastic<NT>(p, T)) {
      // (The loading window changes the tangent alone.)
      double t[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) t[i] = T.s[i] + (i < 3 ? p.K * T.vol : 0.0);
      stress_values(p, h, L, strain, t, own, T.a_n, rec);
    } else {
      bad = stress_plastic<NT>(p, q, nodes + 57 * k, shift, own, state + at, ne * nq, rec);
    }
    if (bad) atomicMin(&fail[k], (2 << 16) | (q << 8) | bad);
  }
  __syncthreads();
  for (int i = tid; i < here; i += kThreads) {
    const int failed = fail[i];
    code[e0 + i] = failed == 0x7fffffff ? 0 : failed & 0xff;
    if (failed != 0x7fffffff) atomicMin(first_failure, (int32_t)(e0 + i));
  }
  // A thread a field of an element; the von Mises stress by the thread of the
  // first, from its own sums.
  const double count = (double)nq;
  for (int i = tid; i < here * kOut; i += kThreads) {
    const int j = i / kOut, f = i - j * kOut;
    if (fail[j] != 0x7fffffff) continue;
    const double* v = values + f * np + j * nq;
    double* res = out + (e0 + j) * 28;
    if (f < 24) {
      double sum = 0.0;
      for (int n = 0; n < nq; ++n) sum += v[n];
      res[f < 12 ? f : f + 4] = sum / count;
    } else {
      double m = f == 25 ? __longlong_as_double(0x7ff0000000000000LL) : 0.0;
      for (int n = 0; n < nq; ++n) m = f == 25 ? fmin(m, v[n]) : fmax(m, v[n]);
      res[f == 24 ? 14 : (f == 25 ? 15 : 13)] = m;
    }
  }
  for (int j = tid; j < here; j += kThreads) {
    if (fail[j] != 0x7fffffff) continue;
    double c[6];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const double* v = values + f * np + j * nq;
      double sum = 0.0;
      for (int n = 0; n < nq; ++n) sum += v[n];
      c[f] = sum / count;
    }
    const double a0 = c[0] - c[1], a1 = c[1] - c[2], a2 = c[2] - c[0];
    out[(e0 + j) * 28 + 12] =
        sqrt(0.5 * (a0 * a0 + a1 * a1 + a2 * a2) + 3.0 * (c[3] * c[3] + c[4] * c[4] + c[5] * c[5]));
  }
}

template <int NT>
int launch(const Params& p, int64_t ne, const double* coords, const int32_t* conn, const double* u, const double* state,
           const double* alpha_n, double* out, int32_t* code, int32_t* first_failure, cudaStream_t stream) {
  static SmemLimit limit;
  const cudaError_t err = limit.allow(stress_kernel<NT>);
  if (err != cudaSuccess) return (int)err;
  const int elements = kThreads / p.nq < kElements ? kThreads / p.nq : kElements;
  const size_t np = (size_t)(elements * p.nq) | 1;
  const size_t smem = (kOut * np + 57u * elements) * sizeof(double);
  const unsigned grid = (unsigned)((ne + elements - 1) / elements);
  stress_kernel<NT><<<grid, kThreads, smem, stream>>>(p, ne, elements, coords, conn, u, state, alpha_n, out, code,
                                                      first_failure);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_stress(const Params& p, int64_t ne, const double* coords, const int32_t* conn, const double* u,
                  const double* state, const double* alpha_n, double* out, int32_t* code, int32_t* first_failure,
                  cudaStream_t stream) {
  if (ne <= 0) return 0;
  const auto run = !p.general ? launch<-1>
                              : (p.nterms == 0 ? launch<0> : (p.nterms == 1 ? launch<1> : (p.nterms == 2 ? launch<2> : launch<4>)));
  return run(p, ne, coords, conn, u, state, alpha_n, out, code, first_failure, stream);
}

}  // namespace sbk
