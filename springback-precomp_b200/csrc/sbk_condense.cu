// The condensation of the incompatible-mode Hex8 (IncompatibleModes.cpp:
// 549-561): with K_aa factorised by the local iteration's last pass, f* = f_u
// - K_ua K_aa^-1 r_a and K* = K_uu - K_ua K_aa^-1 K_au.
//
// A warp takes an element. Over the augmented gradients (eight nodes, three
// modes: 33 degrees of freedom) K = sum_q B^T (w D) B + the geometric part is
// a chain of small contractions, and goes in 8 x 8 tiles through the FP64
// tensor instruction: at a quarter of the instructions of the same products
// in FMAs it is the one form that keeps the FP64 pipe, not the issue slots,
// the limit. The 33rd degree of freedom and the stress (f_u) would each open
// a tile of one column or row: they go as FMAs, four lanes an entry. Measured
// on 1,000,000 elements (2 x 2 x 2 points, non-symmetric): 17.8 ms as FMAs of
// 8 lanes an element, 12.4 ms all in tiles, 11.4 ms so, 9.2 ms with the
// table filled straight through (sbk_point_table.cuh); the tensor instructions
// alone are 5.5 ms of it. Four blocks an SM (spilling at 128 registers) or two
// points unrolled took 5 % longer.
#include <cuda_runtime.h>

#include "sbk_element_math.cuh"
#include "sbk_mma.cuh"
#include "sbk_point_table.cuh"
#include "sbk_smem.h"
#include "sbk_tile.h"

namespace sbk {
namespace {

constexpr int kWarps = 4;
// Per point of the table (sbk_point_table.cuh): 11 gradients, the rows of F,
// three zeros.
constexpr int kTabF = 55, kTabZero = 70, kTab = 73;
constexpr int kKua = 0;    // 24 x 10: K_ua and f_u (over the record's points)
constexpr int kC = 240;    // 9 x 25: K_au and r_a, then their solutions
constexpr int kGeo = 8 * kTab;  // 8 x 11 behind the table
constexpr int kExtra = 8 * kTab + 88;

// The record's points and, behind at least what K_ua and C take over them,
// the element's own values; then the table.
__host__ __device__ inline int own_at(int nq) { return kCondPoint * nq > 466 ? kCondPoint * nq : 466; }
__host__ __device__ inline int warp_doubles(int nq) { return own_at(nq) + kCondElement + kExtra; }

template <bool SYM, bool TANGENT>
__global__ void __launch_bounds__(kWarps * 32, SYM || !TANGENT ? 4 : 3)
    condense_kernel(const __grid_constant__ Params p, int64_t begin, int64_t end, const double* __restrict__ cond,
                    const int32_t* __restrict__ code, double* __restrict__ force, double* __restrict__ tangent) {
  extern __shared__ __align__(16) double smem[];
  const int lane = threadIdx.x & 31, nq = p.nq;
  const int64_t at = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5), e = begin + at;
  if (e >= end || code[e] != 0) return;
  const int record = (int)cond_record(nq);
  double* rec = smem + (threadIdx.x >> 5) * warp_doubles(nq);
  double* tab = rec + warp_doubles(nq) - kExtra;
  {
    const double2* src = reinterpret_cast<const double2*>(cond + (size_t)at * record);
    double2* dst = reinterpret_cast<double2*>(rec);
    const int points = kCondPoint * nq / 2, shift = own_at(nq) / 2 - points;
#pragma unroll 8
    for (int i = lane; i < record / 2; i += 32) dst[i < points ? i : i + shift] = __ldcs(src + i);
  }
  const double* own = rec + own_at(nq);
  const int g = lane >> 2, t = lane & 3;
  const bool small = p.kinematics == SBK_SMALL_STRAIN;
  // Column 32 of K_ua, f_u and row 32 of K_au beyond the tiles: a lane's
  // share over its components, four lanes an entry.
  double uu[3][3][2], ua[3][2], au[3][2], last[3], fu[3], lastrow[3], geo[2][2];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 3; ++j) uu[i][j][0] = uu[i][j][1] = 0.0;
    ua[i][0] = ua[i][1] = au[i][0] = au[i][1] = last[i] = fu[i] = lastrow[i] = 0.0;
  }
  geo[0][0] = geo[0][1] = geo[1][0] = geo[1][1] = 0.0;
  // The lane's strain components: c(t, 0) the normal one t, c(t, 1) the
  // shear (t + 1, t + 2). It forms B's entries of both in the columns 8 i +
  // g: the left operands of the two steps of a contraction over the
  // components (k = t). With D's rows in the same order the product D B
  // leaves its right operands in this lane.
  const int c0 = t, c1 = 3 + (t + 1) % 3;
  const int gc = (g & 1) ? 3 + ((g >> 1) + 1) % 3 : g >> 1;  // component of D's column g
  const bool in = g < 6 && t < 3;
  const int m0 = in ? (kCondM + gc * 6 + c0) * nq : 0, m1 = in ? (kCondM + gc * 6 + c1) * nq : 0;
  const int s0 = t < 3 ? (kCondS + c0) * nq : 0, s1 = t < 3 ? (kCondS + c1) * nq : 0;
  // Row t of the stress.
  const int r0 = (kCondS + (t == 0 ? 0 : (t == 1 ? 3 : 5))) * nq, r1 = (kCondS + (t == 0 ? 3 : (t == 1 ? 1 : 4))) * nq,
            r2 = (kCondS + (t == 0 ? 5 : (t == 1 ? 4 : 2))) * nq;
  int fo[5], go[5];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const int dof = i < 4 ? 8 * i + g : 32;  // the last in every row
    const bool live = t < 3;
    fo[i] = live ? kTabF + 5 * (dof % 3) + t : kTabZero;
    go[i] = live ? 5 * (dof / 3) + t : 0;
  }
  __syncwarp();
#pragma unroll 1
  for (int q0 = 0; q0 < nq; q0 += 8) {
    const int count = min(8, nq - q0);
    __syncwarp();
    if (g < count)
      point_table<true>(p, q0 + g, t, small, rec + q0 + g, nq, own + kCondJ0, tab + g * kTab, kTabF, kTabZero);
    __syncwarp();
#pragma unroll 1
    for (int qq = 0; qq < count; ++qq) {
      const double* T = tab + qq * kTab;
      const double* R = rec + q0 + qq;
      const double w = R[kCondW * nq];
      const double d0 = in ? w * R[m0] : 0.0, d1 = in ? w * R[m1] : 0.0;
      double bf[5][2], db[5][2];
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const double* F = T + fo[i];
        const double* G = T + go[i];
        bf[i][0] = F[0] * G[0];
        bf[i][1] = F[1] * G[2] + F[2] * G[1];
        db[i][0] = db[i][1] = 0.0;
        mma884(db[i], bf[i][0], d0);
        mma884(db[i], bf[i][1], d1);
      }
      const double sn = t < 3 ? w * R[s0] : 0.0, ss = t < 3 ? w * R[s1] : 0.0;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        mma884(ua[i], bf[i][0], db[3][0]);
        mma884(ua[i], bf[i][1], db[3][1]);
        last[i] = fma(bf[i][1], db[4][1], fma(bf[i][0], db[4][0], last[i]));
        fu[i] = fma(bf[i][1], ss, fma(bf[i][0], sn, fu[i]));
      }
      if (TANGENT) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = SYM ? i : 0; j < 3; ++j) {
            mma884(uu[i][j], bf[i][0], db[j][0]);
            mma884(uu[i][j], bf[i][1], db[j][1]);
          }
        if (!SYM) {
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            mma884(au[j], bf[3][0], db[j][0]);
            mma884(au[j], bf[3][1], db[j][1]);
            lastrow[j] = fma(bf[4][1], db[j][1], fma(bf[4][0], db[j][0], lastrow[j]));
          }
        }
      }
      if (!small) {
        // g_a . w S g_b: rows a = g, columns the nodes and the modes.
        const double w0 = t < 3 ? w * R[r0] : 0.0, w1 = t < 3 ? w * R[r1] : 0.0, w2 = t < 3 ? w * R[r2] : 0.0;
        const double ga = t < 3 ? T[5 * g + t] : 0.0;
        const double* gb = T + 5 * g;
        if (TANGENT) mma884(geo[0], ga, w0 * gb[0] + w1 * gb[1] + w2 * gb[2]);
        const double* gm = T + 40 + 5 * (g < 3 ? g : 0);
        mma884(geo[1], ga, g < 3 ? w0 * gm[0] + w1 * gm[1] + w2 * gm[2] : 0.0);
      }
    }
  }
  // The geometric part to its entries (k, l alike); K_ua, f_u and K_au over
  // the record's points, which are done with.
  double* x = rec;
  double* gs = tab + kGeo;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    gs[g * 11 + 2 * t + s] = geo[0][s];
    if (2 * t + s < 3) gs[g * 11 + 8 + 2 * t + s] = geo[1][s];
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int row = 8 * i + g, a3 = row / 3, k3 = row - 3 * a3;
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
      last[i] += __shfl_xor_sync(0xffffffffu, last[i], o);
      fu[i] += __shfl_xor_sync(0xffffffffu, fu[i], o);
      if (!SYM && TANGENT) lastrow[i] += __shfl_xor_sync(0xffffffffu, lastrow[i], o);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int col = 2 * t + s;
      const double v = ua[i][s] + (col % 3 == k3 ? gs[a3 * 11 + 8 + col / 3] : 0.0);
      x[kKua + row * 10 + col] = v;
      if (SYM && TANGENT) x[kC + col * 25 + row] = v;
    }
    const double mode = k3 == 2 ? gs[a3 * 11 + 10] : 0.0;  // entry 32's
    if (t == 0) {
      x[kKua + row * 10 + 8] = last[i] + mode;
      if (SYM && TANGENT) x[kC + 8 * 25 + row] = last[i] + mode;
    } else if (t == 1) {
      x[kKua + row * 10 + 9] = fu[i];
    } else if (t == 2 && !SYM && TANGENT) {
      x[kC + 8 * 25 + row] = lastrow[i] + mode;
    }
  }
  if (!SYM && TANGENT) {
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int col = 8 * j + 2 * t + s, a3 = col / 3, k3 = col - 3 * a3;
        x[kC + g * 25 + col] = au[j][s] + (g % 3 == k3 ? gs[a3 * 11 + 8 + g / 3] : 0.0);
      }
  }
  if (lane < 9) x[kC + lane * 25 + 24] = own[kCondR + lane];
  __syncwarp();
  // K_aa^-1 [K_au, r_a], a column per lane.
  if (TANGENT ? lane < 25 : lane == 24) {
    double y[9];
#pragma unroll
    for (int s = 0; s < 9; ++s) {
      double v = x[kC + ((int)own[kCondPerm + s] >> 4) * 25 + lane];
#pragma unroll
      for (int j = 0; j < s; ++j) v -= own[kCondLu + s * 9 + j] * y[j];
      y[s] = v;
    }
#pragma unroll
    for (int s = 8; s >= 0; --s) {
      double v = y[s];
#pragma unroll
      for (int j = s + 1; j < 9; ++j) v -= own[kCondLu + s * 9 + j] * y[j];
      y[s] = v * own[kCondPiv + s];
    }
#pragma unroll
    for (int s = 0; s < 9; ++s) x[kC + ((int)own[kCondPerm + s] & 15) * 25 + lane] = y[s];
  }
  __syncwarp();
  if (lane < 24) {
    double v = x[kKua + lane * 10 + 9];
#pragma unroll
    for (int j = 0; j < 9; ++j) v -= x[kKua + lane * 10 + j] * x[kC + j * 25 + 24];
    force[e * 24 + lane] = v;
  }
  if (!TANGENT) return;
#pragma unroll
  for (int kk = 0; kk < 3; ++kk) {
    const int j = 4 * kk + t;
    double left[3], right[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      left[i] = j < 9 ? -x[kKua + (8 * i + g) * 10 + j] : 0.0;
      right[i] = j < 9 ? x[kC + j * 25 + 8 * i + g] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int c = SYM ? i : 0; c < 3; ++c) mma884(uu[i][c], left[i], right[c]);
  }
  __syncwarp();
  // K* in node blocks through shared memory, so that it leaves coalesced.
  // A symmetric one from its upper triangle.
  int cpos[3][2], cnode[3][2], ccomp[3][2];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int col = 8 * c + 2 * t + s;
      cnode[c][s] = col / 3;
      ccomp[c][s] = col - 3 * cnode[c][s];
      cpos[c][s] = 9 * cnode[c][s] + ccomp[c][s];
    }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int row = 8 * i + g, a3 = row / 3, k3 = row - 3 * a3;
#pragma unroll
    for (int c = SYM ? i : 0; c < 3; ++c)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const double v = uu[i][c][s] + (k3 == ccomp[c][s] ? gs[a3 * 11 + cnode[c][s]] : 0.0);
        if (!SYM || c > i || 2 * t + s >= g) {
          x[72 * a3 + 3 * k3 + cpos[c][s]] = v;
          if (SYM) x[72 * cnode[c][s] + 3 * ccomp[c][s] + 9 * a3 + k3] = v;
        }
      }
  }
  __syncwarp();
  double* out = tangent + e * 576;
#pragma unroll
  for (int i = 0; i < 18; ++i) out[lane + 32 * i] = x[lane + 32 * i];
}

template <bool SYM, bool TANGENT>
int launch(const Params& p, const TileArgs& a, const TileScratch& s, cudaStream_t stream) {
  static SmemLimit limit;
  const size_t smem = (size_t)kWarps * warp_doubles(p.nq) * sizeof(double);
  auto kern = condense_kernel<SYM, TANGENT>;
  const cudaError_t err = limit.allow(kern);
  if (err != cudaSuccess) return (int)err;
  const int64_t n = a.end - a.begin;
  kern<<<(unsigned)((n + kWarps - 1) / kWarps), kWarps * 32, smem, stream>>>(p, a.begin, a.end, s.cond, a.code,
                                                                             a.force, a.tangent);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_condense(const Params& p, const TileArgs& a, const TileScratch& s, cudaStream_t stream) {
  if (p.symmetric) return a.want_tangent ? launch<true, true>(p, a, s, stream) : launch<true, false>(p, a, s, stream);
  return a.want_tangent ? launch<false, true>(p, a, s, stream) : launch<false, false>(p, a, s, stream);
}

}  // namespace sbk
