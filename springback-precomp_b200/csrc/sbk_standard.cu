// K1s: the standard Hex8 (elastoplastic_element for an element without internal
// modes, Elastoplastic.cpp:226-340, kinematics_of :104-168), with mean dilatation
// (B-bar) or without, for small, finite and logarithmic strain.
//
// Two kernels, as for the incompatible-mode element: standard_points_kernel, a
// thread a point over a tile of elements (kinematics, the averaged dilatation,
// returns, the logarithmic maps, states and energies), and
// standard_tangent_kernel, a warp an element, whose contraction goes through
// the FP64 tensor instruction. The mean-dilatation terms fit its padding: with
// s = mean_row - d (d = B_NL^T P^T m the point's dilatation row) as a seventh
// strain component,
//   K = sum w [B_NL; s]^T [[M, U1 / 3], [U2^T / 3, m.C m / 9]] [B_NL; s] + geometric,
// M and S the logarithmic map at the pressure-shifted stress, U1 = P^T C m, U2 =
// P^T C^T m; for finite strain the geometric part takes S + (mean p - p) 1.
//
// Measured (7,200 J2 elements with mean dilatation): 479 us for the element
// kernel that had a group of lanes and 12 KB of shared memory an element, and
// 49 us for its schedule; 51 + 64 us so.
#include <cuda_runtime.h>

#include "sbk_element.h"
#include "sbk_mma.cuh"
#include "sbk_point_table.cuh"
#include "sbk_smem.h"
#include "sbk_tile_point.cuh"

namespace sbk {
namespace {

// ---- points ------------------------------------------------------------------

constexpr int kThreads = kTileThreads;
// A point's record in shared memory.
constexpr int kM = 0, kS = 36, kL = 42, kStrain = 60, kWarm = 66, kW = 73, kSum = 74, kRec = 75;

// One element of a tile: its failure, as the tile kernel keeps it.
__device__ __forceinline__ void fail_point(int* fail, int stage, int q, int code) {
  atomicMin(fail, (stage << 16) | (q << 8) | code);
}

__device__ __forceinline__ void load_spectral(const PointRecord& r, LogKin& L) {
#pragma unroll
  for (int i = 0; i < 9; ++i) L.q[i] = r.get(kL + i);
#pragma unroll
  for (int i = 0; i < 3; ++i) L.mu[i] = r.get(kL + 9 + i);
#pragma unroll
  for (int i = 0; i < 6; ++i) L.first[i] = r.get(kL + 12 + i);
}

// P^T t: the second Piola-Kirchhoff stress of a stress work-conjugate to the
// log strain (LogarithmicStrain.cpp:144-149).
__device__ __forceinline__ void pull_back(const LogKin& L, const double t[6], double out[6]) {
  double tp[6];
  rotate_in(L.q, t, tp);
#pragma unroll
  for (int i = 0; i < 6; ++i) tp[i] *= L.first[i];
  rotate_out(L.q, tp, out);
}

// The mean over element k's points of field f's sums, weighted by w.
__device__ __forceinline__ double element_mean(const double* rec, int np, int nq, int k) {
  double volume = 0.0, sum = 0.0;
#pragma unroll 1
  for (int j = k * nq; j < (k + 1) * nq; ++j) {
    volume += rec[kW * np + j];
    sum += rec[kSum * np + j];
  }
  return sum / volume;
}

template <int NT>
__global__ void __launch_bounds__(kThreads, 1)
    standard_points_kernel(const __grid_constant__ Params p, const __grid_constant__ TileArgs a,
                           double* __restrict__ records) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int fail[kTileMostElements], listed;
  __shared__ int16_t yields[kThreads];
  __shared__ uint8_t flag[kThreads];
  const int tid = threadIdx.x, nq = p.nq, elements = a.elements, np = (elements * nq) | 1;
  double* rec = smem;
  double* nodes = smem + kRec * np;  // coordinates 24, displacements 24 an element
  const int64_t e0 = a.begin + (int64_t)blockIdx.x * elements;
  const int here = (int)(a.end - e0 < elements ? a.end - e0 : elements);
  const bool averaged = p.averaged != 0, log = p.kinematics == SBK_FINITE_LOGARITHMIC;
  for (int k = tid; k < here; k += kThreads) fail[k] = 0x7fffffff;
  if (tid == 0) listed = 0;
  __syncthreads();
  for (int i = tid; i < here * 8; i += kThreads) {
    const int k = i >> 3, n = i & 7;
    const int64_t node = a.conn[(e0 + k) * 8 + n];
    double* X = nodes + 48 * k + 3 * n;
    if (p.num_nodes > 0 && (node < 0 || node >= p.num_nodes)) {
      fail[k] = SBK_EL_BAD_NODE;
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        X[c] = a.coords[node * 3 + c];
        X[24 + c] = a.u[node * 3 + c];
      }
    }
  }
  __syncthreads();
  const int pt = tid, k = tid / nq, q = tid - k * nq;
  const bool mine = k < here;
  const PointRecord r{rec + pt, np};
  double* out = records + (size_t)(e0 - a.begin + (mine ? k : 0)) * kStdPoint * nq + q;
  if (mine && fail[k] != SBK_EL_BAD_NODE) {
    PointGeometry G;
    if (!point_geometry(p, q, nodes + 48 * k, nodes + 48 * k + 24, G)) {
      atomicMin(&fail[k], SBK_EL_MESH_INVERTED);
    } else {
      LogKin L;
#pragma unroll
      for (int i = 0; i < 9; ++i) L.q[i] = i % 4 == 0 ? 1.0 : 0.0;
      double strain[6];
      const int code = point_strain(p, G.du, L, strain);
      if (code) {
        fail_point(&fail[k], 1, q, code);
      } else {
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          out[(kCondH + i) * nq] = G.du[i];
          out[(kCondGeo + i) * nq] = G.ji[i];
        }
        out[kCondW * nq] = G.w;
        r.put(kW, G.w);
        r.put(kSum, G.w * (strain[0] + strain[1] + strain[2]));
#pragma unroll
        for (int i = 0; i < 6; ++i) r.put(kStrain + i, strain[i]);
        if (log) {
#pragma unroll
          for (int i = 0; i < 9; ++i) r.put(kL + i, L.q[i]);
#pragma unroll
          for (int i = 0; i < 3; ++i) r.put(kL + 9 + i, L.mu[i]);
#pragma unroll
          for (int i = 0; i < 6; ++i) r.put(kL + 12 + i, L.first[i]);
        }
        if (averaged) {
          // P^T m: the variation of the trace.
          double pv[6] = {1.0, 1.0, 1.0, 0.0, 0.0, 0.0};
          if (log) {
            const double f[6] = {L.first[0], L.first[1], L.first[2], 0.0, 0.0, 0.0};
            rotate_out(L.q, f, pv);
          }
#pragma unroll
          for (int i = 0; i < 6; ++i) out[(kStdPv + i) * nq] = pv[i];
        }
      }
    }
  }
  __syncthreads();
  const bool live = mine && fail[mine ? k : 0] == 0x7fffffff;
  const int64_t at = (e0 + (mine ? k : 0)) * nq + q;
  if (live) {
    double strain[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) strain[i] = r.get(kStrain + i);
    if (averaged) {
      const double shift = (element_mean(rec, np, nq, k) - (strain[0] + strain[1] + strain[2])) / 3.0;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        strain[i] += shift;
        r.put(kStrain + i, strain[i]);
      }
    }
    PointTrial<NT> T;
    point_trial<NT>(p, strain, a.state + at, a.ne * nq, T);
    flag[pt] = 0;
    if (NT >= 0 && !isfinite(T.f)) {
      fail_point(&fail[k], 2, q, kFailReturn);
    } else if (point_elastic<NT>(p, T) && !point_window<NT>(p, T)) {
#pragma unroll
      for (int i = 0; i < 6; ++i) r.put(kS + i, T.s[i] + (i < 3 ? p.K * T.vol : 0.0));
    } else {
      yields[atomicAdd(&listed, 1)] = (int16_t)pt;
    }
  }
  __syncthreads();
  if (tid < listed) {
    const int y = yields[tid], ky = y / nq, qy = y - ky * nq;
    const PointRecord ry{rec + y, np};
    double strain[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) strain[i] = ry.get(kStrain + i);
    PointTrial<NT> T;
    point_trial<NT>(p, strain, a.state + (e0 + ky) * nq + qy, a.ne * nq, T);
    const bool window = point_elastic<NT>(p, T);
    int code = 0;
    if constexpr (NT < 0) {
      if (window) return_window_radial(p, T, ry, kS, kM);
      else code = return_radial(p, T, ry, kS, kM, kWarm);
    } else {
      code = return_general<NT>(p, T, window, false, ry, kS, kM, kWarm);
    }
    if (code) fail_point(&fail[ky], 2, qy, code);
    else flag[y] = window ? 2 : 1;
  }
  __syncthreads();
  const bool whole = mine && fail[mine ? k : 0] == 0x7fffffff;
  double trace = 0.0, energy = 0.0;
  if (whole) {
    trace = r.get(kS) + r.get(kS + 1) + r.get(kS + 2);
    r.put(kSum, r.get(kW) * trace / 3.0);
  }
  __syncthreads();
  if (whole) {
    const int fl = flag[pt];
    const bool elastic = fl == 0;
    const double shift = averaged ? element_mean(rec, np, nq, k) - trace / 3.0 : 0.0;
    LogKin L;
    if (log) load_spectral(r, L);
    if (!log && elastic) {
      double C[36];
      elastic_C(p, C);
#pragma unroll
      for (int i = 0; i < 36; ++i) r.put(kM + i, C[i]);
    }
    if (averaged) {
      double cm[6], mc[6], st[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        st[i] = r.get(kS + i);
        if (elastic) {
          cm[i] = mc[i] = i < 3 ? 3.0 * p.K : 0.0;
        } else {
          cm[i] = r.get(kM + i * 6) + r.get(kM + i * 6 + 1) + r.get(kM + i * 6 + 2);
          mc[i] = r.get(kM + i) + r.get(kM + 6 + i) + r.get(kM + 12 + i);
        }
      }
      out[kStdMcm * nq] = (cm[0] + cm[1] + cm[2]) / 9.0;
      out[kStdTr * nq] = trace / 3.0;
      double v[6];
#pragma unroll 1
      for (int j = 0; j < 3; ++j) {
        double t[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) t[i] = j == 0 ? st[i] : (j == 1 ? cm[i] : mc[i]);
        if (log) {
          pull_back(L, t, v);
        } else {
#pragma unroll
          for (int i = 0; i < 6; ++i) v[i] = t[i];
        }
        const double scale = j == 0 ? 1.0 : 1.0 / 3.0;
#pragma unroll
        for (int i = 0; i < 6; ++i) out[(kStdSt + 6 * j + i) * nq] = scale * v[i];
      }
      // The geometric part's stress: shifted before the logarithmic map; for
      // finite strain as it is.
      if (p.kinematics != SBK_SMALL_STRAIN)
#pragma unroll
        for (int i = 0; i < 3; ++i) r.put(kS + i, st[i] + shift);
    }
    if (log) spectral_map(p, L, elastic, r, kS, kM);
#pragma unroll 6
    for (int i = 0; i < 36; ++i) out[(kCondM + i) * nq] = r.get(kM + i);
#pragma unroll
    for (int i = 0; i < 6; ++i) out[(kCondS + i) * nq] = r.get(kS + i);
    double strain[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) strain[i] = r.get(kStrain + i);
    energy = r.get(kW) * point_finish<NT>(p, strain, fl, r, kWarm, a.state + at, a.trial + at, a.ne * nq);
    a.yield[at] = fl == 1 ? 1 : 0;
  }
  __syncthreads();
  if (whole) r.put(kSum, energy);
  __syncthreads();
  for (int j = tid; j < here; j += kThreads) {
    const int64_t e = e0 + j;
    const int failed = fail[j];
    if (failed != 0x7fffffff) {
      a.code[e] = failed & 0xff;
      if (a.first_failure) atomicMin(a.first_failure, (int32_t)e);
      continue;
    }
    double en = 0.0;
    for (int n = 0; n < nq; ++n) en += rec[kSum * np + j * nq + n];
    a.energy[e] = en;
    a.iterations[e] = 0;
    a.code[e] = 0;
  }
  for (int i = tid; i < here * 9; i += kThreads) a.alpha_out[e0 * 9 + i] = 0.0;
}

// ---- force and tangent ---------------------------------------------------------

constexpr int kWarps = 4;
// Per point of the table (sbk_point_table.cuh): eight gradients, the rows of
// F, three zeros.
constexpr int kTabF = 40, kTabZero = 55, kTab = 58;
constexpr int kExtra = 8 * kTab + 64;

__host__ __device__ inline int warp_doubles(int nq) {
  return (kStdPoint * nq > 576 ? kStdPoint * nq : 576) + kExtra;
}

template <bool SYM, bool AVERAGED>
__global__ void __launch_bounds__(kWarps * 32, 4)
    standard_tangent_kernel(const __grid_constant__ Params p, int64_t begin, int64_t end,
                            const double* __restrict__ records, const int32_t* __restrict__ code,
                            double* __restrict__ force, double* __restrict__ tangent, int want) {
  extern __shared__ __align__(16) double smem[];
  const int lane = threadIdx.x & 31, nq = p.nq;
  const int64_t at = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5), e = begin + at;
  if (e >= end || code[e] != 0) return;
  double* rec = smem + (threadIdx.x >> 5) * warp_doubles(nq);
  double* tab = rec + warp_doubles(nq) - kExtra;
  {
    const double2* src = reinterpret_cast<const double2*>(records + (size_t)at * kStdPoint * nq);
    double2* dst = reinterpret_cast<double2*>(rec);
    const int n = (AVERAGED ? kStdPoint : kCondPoint) * nq / 2;
#pragma unroll 8
    for (int i = lane; i < n; i += 32) dst[i] = __ldcs(src + i);
  }
  const int g = lane >> 2, t = lane & 3;
  const bool small = p.kinematics == SBK_SMALL_STRAIN;
  double uu[3][3][2], geo[2] = {0.0, 0.0}, fl[3] = {0.0, 0.0, 0.0}, mean[3] = {0.0, 0.0, 0.0}, volume = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) uu[i][j][0] = uu[i][j][1] = 0.0;
  // The lane's strain components (t, t) and (t + 1, t + 2); lane t = 3 the
  // dilatation row and nothing.
  const int c0 = t < 3 ? t : 0, c1 = t < 3 ? 3 + (t + 1) % 3 : 0;
  const int gc = g < 6 ? ((g & 1) ? 3 + ((g >> 1) + 1) % 3 : g >> 1) : 0;  // component of D's column g
  // D's entries (column g; rows of the lane): a field of the record, or none.
  int m0 = -1, m1 = -1;
  if (g < 6) {
    if (t < 3) m0 = kCondM + gc * 6 + c0, m1 = kCondM + gc * 6 + c1;
    else if (AVERAGED) m0 = kStdU1 + gc;
  } else if (AVERAGED && g == 6) {
    if (t < 3) m0 = kStdU2 + c0, m1 = kStdU2 + c1;
    else m0 = kStdMcm;
  }
  const bool has0 = m0 >= 0, has1 = m1 >= 0;
  m0 = has0 ? m0 * nq : 0;
  m1 = has1 ? m1 * nq : 0;
  const int s0 = ((AVERAGED ? kStdSt : kCondS) + c0) * nq, s1 = ((AVERAGED ? kStdSt : kCondS) + c1) * nq;
  const int r0 = (kCondS + (t == 0 ? 0 : (t == 1 ? 3 : 5))) * nq, r1 = (kCondS + (t == 0 ? 3 : (t == 1 ? 1 : 4))) * nq,
            r2 = (kCondS + (t == 0 ? 5 : (t == 1 ? 4 : 2))) * nq;
  int fo[3], go[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int dof = 8 * i + g;
    fo[i] = t < 3 ? kTabF + 5 * (dof % 3) + t : kTabZero;
    go[i] = t < 3 ? 5 * (dof / 3) + t : 0;
  }
  __syncwarp();
  // First (mean dilatation) the volume average of the dilatation rows, then
  // the sums: two walks over the points in groups of eight.
#pragma unroll 1
  for (int pass = AVERAGED ? 0 : 1; pass < 2; ++pass) {
#pragma unroll 1
    for (int q0 = 0; q0 < nq; q0 += 8) {
      const int count = min(8, nq - q0);
      if (!AVERAGED || nq > 8 || pass == 0) {
        __syncwarp();
        if (g < count)
          point_table<false>(p, q0 + g, t, small, rec + q0 + g, nq, nullptr, tab + g * kTab, kTabF, kTabZero);
        __syncwarp();
      }
#pragma unroll 1
      for (int qq = 0; qq < count; ++qq) {
        const double* T = tab + qq * kTab;
        const double* R = rec + q0 + qq;
        const double w = R[kCondW * nq];
        double bf[3][2], row[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double* F = T + fo[i];
          const double* G = T + go[i];
          bf[i][0] = F[0] * G[0];
          bf[i][1] = F[1] * G[2] + F[2] * G[1];
        }
        if (AVERAGED) {
          const double v0 = R[(kStdPv + c0) * nq], v1 = R[(kStdPv + c1) * nq];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            row[i] = bf[i][0] * v0 + bf[i][1] * v1;
            if (pass == 1) {
              row[i] += __shfl_xor_sync(0xffffffffu, row[i], 1);
              row[i] += __shfl_xor_sync(0xffffffffu, row[i], 2);
            }
          }
          if (pass == 0) {
            volume += w;
#pragma unroll
            for (int i = 0; i < 3; ++i) mean[i] += w * row[i];
            continue;
          }
#pragma unroll
          for (int i = 0; i < 3; ++i) bf[i][0] = t < 3 ? bf[i][0] : mean[i] - row[i];
        }
        const double f0 = w * (t < 3 ? R[s0] : (AVERAGED ? R[kStdTr * nq] : 0.0)), f1 = t < 3 ? w * R[s1] : 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) fl[i] += bf[i][0] * f0 + bf[i][1] * f1;
        if (!want) continue;
        const double d0 = has0 ? w * R[m0] : 0.0, d1 = has1 ? w * R[m1] : 0.0;
        double db[3][2];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          db[i][0] = db[i][1] = 0.0;
          mma884(db[i], bf[i][0], d0);
          mma884(db[i], bf[i][1], d1);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = SYM ? i : 0; j < 3; ++j) {
            mma884(uu[i][j], bf[i][0], db[j][0]);
            mma884(uu[i][j], bf[i][1], db[j][1]);
          }
        if (!small) {
          const double w0 = t < 3 ? w * R[r0] : 0.0, w1 = t < 3 ? w * R[r1] : 0.0, w2 = t < 3 ? w * R[r2] : 0.0;
          const double* gb = T + 5 * g;
          mma884(geo, t < 3 ? T[5 * g + t] : 0.0, w0 * gb[0] + w1 * gb[1] + w2 * gb[2]);
        }
      }
    }
    if (AVERAGED && pass == 0) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        mean[i] += __shfl_xor_sync(0xffffffffu, mean[i], 1);
        mean[i] += __shfl_xor_sync(0xffffffffu, mean[i], 2);
        mean[i] /= volume;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    fl[i] += __shfl_xor_sync(0xffffffffu, fl[i], 1);
    fl[i] += __shfl_xor_sync(0xffffffffu, fl[i], 2);
    if (t == 0) force[e * 24 + 8 * i + g] = fl[i];
  }
  if (!want) return;
  double* x = rec;
  double* gs = tab + 8 * kTab;
  gs[g * 8 + 2 * t] = geo[0];
  gs[g * 8 + 2 * t + 1] = geo[1];
  __syncwarp();
  // The tangent in node blocks through shared memory, so that it leaves
  // coalesced; a symmetric one from its upper triangle.
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int row = 8 * i + g, a3 = row / 3, k3 = row - 3 * a3;
#pragma unroll
    for (int c = SYM ? i : 0; c < 3; ++c)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int col = 8 * c + 2 * t + s, b3 = col / 3, l3 = col - 3 * b3;
        const double v = uu[i][c][s] + (k3 == l3 ? gs[a3 * 8 + b3] : 0.0);
        if (!SYM || c > i || 2 * t + s >= g) {
          x[72 * a3 + 9 * b3 + 3 * k3 + l3] = v;
          if (SYM) x[72 * b3 + 9 * a3 + 3 * l3 + k3] = v;
        }
      }
  }
  __syncwarp();
  double* out = tangent + e * 576;
#pragma unroll
  for (int i = 0; i < 18; ++i) out[lane + 32 * i] = x[lane + 32 * i];
}

template <int NT>
int launch_points(const Params& p, const TileArgs& a, const TileScratch& s, cudaStream_t stream) {
  static SmemLimit limit;
  const size_t np = (size_t)(a.elements * p.nq) | 1;
  const size_t smem = (kRec * np + 48u * a.elements) * sizeof(double);
  const cudaError_t err = limit.allow(standard_points_kernel<NT>);
  if (err != cudaSuccess) return (int)err;
  standard_points_kernel<NT><<<(unsigned)a.num_tiles, kThreads, smem, stream>>>(p, a, s.cond);
  return (int)cudaGetLastError();
}

template <bool SYM, bool AVERAGED>
int launch_tangent(const Params& p, const TileArgs& a, const TileScratch& s, cudaStream_t stream) {
  static SmemLimit limit;
  const size_t smem = (size_t)kWarps * warp_doubles(p.nq) * sizeof(double);
  const cudaError_t err = limit.allow(standard_tangent_kernel<SYM, AVERAGED>);
  if (err != cudaSuccess) return (int)err;
  const int64_t n = a.end - a.begin;
  standard_tangent_kernel<SYM, AVERAGED><<<(unsigned)((n + kWarps - 1) / kWarps), kWarps * 32, smem, stream>>>(
      p, a.begin, a.end, s.cond, a.code, a.force, a.tangent, a.want_tangent);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_standard(const Params& p, const TileArgs& a, const TileScratch& s, cudaStream_t stream) {
  int rc;
  if (!p.general) rc = launch_points<-1>(p, a, s, stream);
  else if (p.nterms == 0) rc = launch_points<0>(p, a, s, stream);
  else if (p.nterms == 1) rc = launch_points<1>(p, a, s, stream);
  else if (p.nterms == 2) rc = launch_points<2>(p, a, s, stream);
  else rc = launch_points<4>(p, a, s, stream);
  if (rc) return rc;
  if (p.symmetric) return p.averaged ? launch_tangent<true, true>(p, a, s, stream) : launch_tangent<true, false>(p, a, s, stream);
  return p.averaged ? launch_tangent<false, true>(p, a, s, stream) : launch_tangent<false, false>(p, a, s, stream);
}

}  // namespace sbk
