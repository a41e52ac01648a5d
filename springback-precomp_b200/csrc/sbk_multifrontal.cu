// The multifrontal Cholesky: where the reference takes CHOLMOD's supernodal
// one (src/fem/Forming.cpp:100-160).
//
// The elimination tree of the groups (nodes) is cut into fronts: subtrees of
// at most kLeafRows rows become one dense front each (below that size a
// sparse elimination is all launches and latency), above them columns whose
// patterns nest join. A front is a dense lower matrix of its columns and the
// rows they reach; level by level from the leaves, every front of a level at
// once,
//
//   extend_add_kernel  adds the children's remainders (a warp a column, the
//                      children in order: the same sums on every run);
//   panel_kernel       factorises the next kPanel columns' diagonal block and
//                      solves the rows below (every block factorises the
//                      small block for itself rather than wait for one);
//   tile_kernel        takes the panel's product off the front's own columns
//                      in 64 x 64 tiles on the FP64 tensor instruction and,
//                      after the last panel, all its columns' product off
//                      the remainder, which is so read and written once;
//
// and the solves walk the same levels with a block a front. What bounds it is
// the chain of levels and panels, some hundred launches of a few microseconds
// for a sheet of 13,689 rows. Measured there (41 x 41 x 3 nodes, clamped):
// factorisation and one solve 44.7 ms with the level-scheduled sparse Cholesky
// of the library, 1.5 ms so (2.0 ms with the refinement a symmetric solve takes,
// sbk_partition.cu).
#include "sbk_multifrontal.h"

#include <algorithm>
#include <numeric>

#include "sbk_mma.cuh"

namespace sbk {
namespace {

constexpr int kLeafRows = 96;  // rows of a leaf front's columns, at most (48 to 192: within 4 %, 1.27 ms busy here)
constexpr int kPanel = 32;
constexpr int kTile = 64;
constexpr int kRowChunk = 128;  // rows of a panel task
constexpr int kAddColumns = 8;  // columns of an extend-add task

struct Fronts {
  const int4* front;
  const int64_t* offset;
  double* arena;
};

__global__ void scatter_values_kernel(const double* __restrict__ values, const int32_t* __restrict__ src,
                                      const int64_t* __restrict__ dst, int64_t n, double* __restrict__ arena) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    arena[dst[i]] = values[src[i]];
}

// A warp a column of the front: the children's remainders' columns that land
// there, child after child.
__global__ void __launch_bounds__(32 * kAddColumns)
    extend_add_kernel(Fronts f, const int2* __restrict__ tasks, const int2* __restrict__ children,
                      const int32_t* __restrict__ child, const int32_t* __restrict__ place) {
  const int2 task = tasks[blockIdx.x];
  const int4 me = f.front[task.x];
  const int column = task.y + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (column >= me.z) return;
  double* to = f.arena + f.offset[task.x] + (int64_t)column * me.z;
  const int2 list = children[task.x];
  for (int i = 0; i < list.y; ++i) {
    const int c = child[list.x + i];
    const int4 it = f.front[c];
    const int rest = it.z - it.y;
    const int32_t* at = place + it.w;
    // The child's row that is this column (places ascend).
    int lo = 0, hi = rest;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (at[mid] < column) lo = mid + 1;
      else hi = mid;
    }
    if (lo == rest || at[lo] != column) continue;
    const double* from = f.arena + f.offset[c] + (int64_t)(it.y + lo) * it.z + it.y;
    // Four rows at once: the places differ, which the compiler cannot know.
    for (int r0 = lo + lane; r0 < rest; r0 += 128) {
      double* at4[4];
      double sum[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = min(r0 + 32 * u, rest - 1);
        at4[u] = to + at[r];
        sum[u] = *at4[u] + from[r];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r0 + 32 * u < rest) *at4[u] = sum[u];
    }
    __syncwarp();
  }
}

// The panel of columns [p0, p0 + nb): its diagonal block's Cholesky factor
// (into diag, by the first task of the front), and L21 = A21 L11^-T for the
// task's rows, a thread a row.
__global__ void __launch_bounds__(kRowChunk)
    panel_kernel(Fronts f, const int2* __restrict__ tasks, int p0, const int32_t* __restrict__ diag_offset,
                 double* __restrict__ diag, int32_t* __restrict__ failed) {
  __shared__ double L[kPanel][kPanel + 1];
  __shared__ double inv[kPanel];
  const int2 task = tasks[blockIdx.x];
  const int4 me = f.front[task.x];
  const int m = me.z, nb = min(kPanel, me.y - p0), tid = threadIdx.x;
  double* A = f.arena + f.offset[task.x];
  const int row = task.y + tid;
  double x[kPanel];
#pragma unroll
  for (int j = 0; j < kPanel; ++j) x[j] = j < nb && row < m ? A[(int64_t)(p0 + j) * m + row] : 0.0;
  {
    // Every warp the whole block for itself, lane r the row r (identity
    // beyond nb): no barrier in the 32 steps.
    const int r = tid & 31;
    double d_row[kPanel];
#pragma unroll
    for (int c = 0; c < kPanel; ++c)
      d_row[c] = r < nb && c <= r ? A[(int64_t)(p0 + c) * m + p0 + r] : (r == c ? 1.0 : 0.0);
    int bad = 0x7fffffff;
    double mine = 1.0;
#pragma unroll
    for (int j = 0; j < kPanel; ++j) {
      double d = __shfl_sync(0xffffffffu, d_row[j], j);
      if (!(d > 0.0)) {
        bad = min(bad, j);
        d = 1.0;
      }
      const double scale = rsqrt(d);
      const double l = d_row[j] * scale;
      if (r == j) mine = scale;
      d_row[j] = r == j ? d * scale : l;
#pragma unroll
      for (int c = j + 1; c < kPanel; ++c) d_row[c] -= l * __shfl_sync(0xffffffffu, l, c);
    }
    if (bad < nb && tid == 0) atomicMin(failed, me.x + p0 + bad);
    if (tid < 32) {
#pragma unroll
      for (int c = 0; c < kPanel; ++c) L[r][c] = c <= r ? d_row[c] : 0.0;
      inv[r] = mine;
    }
    __syncthreads();
  }
  if (task.y == p0 + nb) {  // the front's first task
    double* D = diag + (int64_t)(diag_offset[task.x] + p0 / kPanel) * kPanel * kPanel;
    for (int i = tid; i < kPanel * kPanel; i += kRowChunk) D[i] = L[i % kPanel][i / kPanel];
  }
  if (row >= m) return;
#pragma unroll
  for (int j = 0; j < kPanel; ++j) {
    if (j < nb) {
      x[j] *= inv[j];
#pragma unroll
      for (int i = j + 1; i < kPanel; ++i) x[i] -= x[j] * L[i][j];
    }
  }
#pragma unroll
  for (int j = 0; j < kPanel; ++j)
    if (j < nb) A[(int64_t)(p0 + j) * m + row] = x[j];
}

// C -= P_i P_j^T of one 64 x 64 tile of the lower matrix below the columns P:
// four warps a quadrant of 4 x 4 tensor tiles each. P is the panel at p0 and C
// the front's own columns, or (p0 < 0) P all its columns and C the remainder.
__global__ void __launch_bounds__(128)
    tile_kernel(Fronts f, const int4* __restrict__ tasks, int p0) {
  __shared__ double P[2][kPanel][kTile + 4];
  const int4 task = tasks[blockIdx.x];
  const int4 me = f.front[task.x];
  const int m = me.z, first = p0 < 0 ? 0 : p0, base = p0 < 0 ? me.y : min(p0 + kPanel, me.y);
  const int columns = p0 < 0 ? m : me.y;
  double* A = f.arena + f.offset[task.x];
  const int r0 = base + task.y * kTile, c0 = base + task.z * kTile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int wr = (warp & 1) * 32, wc = (warp >> 1) * 32;
  const bool lower = r0 + wr + 31 >= c0 + wc;
  // C first, all of it in flight at once: added at the end instead, each entry
  // waits for the store before it (17 us a tile for 6).
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int row = r0 + wr + 8 * i + g, col = c0 + wc + 8 * j + 2 * t + s;
        acc[i][j][s] = row < m && col < columns && col <= row ? A[(int64_t)col * m + row] : 0.0;
      }
#pragma unroll 1
  for (int k0 = first; k0 < base; k0 += kPanel) {
    if (k0 > first) __syncthreads();
#pragma unroll
    for (int i = threadIdx.x; i < kPanel * kTile; i += 128) {
      const int r = i % kTile, j = i / kTile;
      const double* col = A + (int64_t)(k0 + j) * m;
      P[0][j][r] = k0 + j < base && r0 + r < m ? col[r0 + r] : 0.0;
      P[1][j][r] = k0 + j < base && c0 + r < m ? col[c0 + r] : 0.0;
    }
    __syncthreads();
    if (!lower) continue;
#pragma unroll
    for (int k = 0; k < kPanel; k += 4) {
      double a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = -P[0][k + t][wr + 8 * i + g];
        b[i] = P[1][k + t][wc + 8 * i + g];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma884(acc[i][j], a[i], b[j]);
    }
  }
  if (!lower) return;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int row = r0 + wr + 8 * i + g, col = c0 + wc + 8 * j + 2 * t + s;
        if (row < m && col < columns && col <= row) A[(int64_t)col * m + row] = acc[i][j][s];
      }
}

constexpr int kSolveThreads = 256;

// L y = b for the fronts of a level: y starts from b and the children's
// remainders; panel after panel the small triangle by one warp, then its
// product off the rows below.
__global__ void __launch_bounds__(kSolveThreads)
    forward_kernel(Fronts f, const int32_t* __restrict__ order, const int2* __restrict__ children,
                   const int32_t* __restrict__ child, const int32_t* __restrict__ place,
                   const int64_t* __restrict__ y_offset, const int32_t* __restrict__ diag_offset,
                   const double* __restrict__ diag, const double* __restrict__ b, double* y_all) {
  __shared__ double x[kPanel];
  const int s = order[blockIdx.x], tid = threadIdx.x;
  const int4 me = f.front[s];
  const int k = me.y, m = me.z;
  double* y = y_all + y_offset[s];
  const double* A = f.arena + f.offset[s];
  for (int i = tid; i < m; i += kSolveThreads) y[i] = i < k ? b[me.x + i] : 0.0;
  __syncthreads();
  const int2 list = children[s];
  for (int c = 0; c < list.y; ++c) {
    const int it = child[list.x + c];
    const int4 that = f.front[it];
    const double* yc = y_all + y_offset[it] + that.y;
    const int32_t* at = place + that.w;
    for (int i = tid; i < that.z - that.y; i += kSolveThreads) y[at[i]] += yc[i];
    __syncthreads();
  }
  // Everything a panel reads but y is on its way before the barrier it waits
  // for: the next triangle, the thread's first row.
  double l[kPanel], inv = 0.0;
  auto triangle = [&](int p0) {
    if (tid >= 32) return;
    const double* D = diag + (int64_t)(diag_offset[s] + p0 / kPanel) * kPanel * kPanel;
#pragma unroll
    for (int j = 0; j < kPanel; ++j) l[j] = D[j * kPanel + tid];  // L(tid, j)
    inv = 1.0 / D[tid * kPanel + tid];
  };
  triangle(0);
  for (int p0 = 0; p0 < k; p0 += kPanel) {
    const int nb = min(kPanel, k - p0), first = p0 + nb + tid;
    const double* row = A + (int64_t)p0 * m + first;
    double a[kPanel];
#pragma unroll
    for (int j = 0; j < kPanel; ++j) a[j] = j < nb && first < m ? row[(int64_t)j * m] : 0.0;
    if (tid < 32) {
      double v = tid < nb ? y[p0 + tid] : 0.0;
#pragma unroll
      for (int j = 0; j < kPanel; ++j) {
        const double xj = __shfl_sync(0xffffffffu, v * inv, j);
        v = tid == j ? xj : v - (tid > j ? l[j] * xj : 0.0);
      }
      x[tid] = v;
      if (tid < nb) y[p0 + tid] = v;
    }
    if (p0 + kPanel < k) triangle(p0 + kPanel);
    __syncthreads();
    for (int i = first; i < m; i += kSolveThreads) {
      if (i > first) {
        row += kSolveThreads;
#pragma unroll
        for (int j = 0; j < kPanel; ++j) a[j] = j < nb ? row[(int64_t)j * m] : 0.0;
      }
      double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int j = 0; j < kPanel; ++j) v[j & 3] += a[j] * x[j];
      y[i] -= (v[0] + v[1]) + (v[2] + v[3]);
    }
    __syncthreads();
  }
}

// L^T x = y for the fronts of a level: the rows below from x, then the panels
// from the last, a warp a column's product.
__global__ void __launch_bounds__(kSolveThreads)
    backward_kernel(Fronts f, const int32_t* __restrict__ order, const int32_t* __restrict__ rows,
                    const int64_t* __restrict__ y_offset, const int32_t* __restrict__ diag_offset,
                    const double* __restrict__ diag, double* y_all, double* x) {
  __shared__ double part[kPanel];
  const int s = order[blockIdx.x], tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int4 me = f.front[s];
  const int k = me.y, m = me.z;
  double* y = y_all + y_offset[s];
  const double* A = f.arena + f.offset[s];
  for (int i = k + tid; i < m; i += kSolveThreads) y[i] = x[rows[me.w + i - k]];
  __syncthreads();
  for (int p0 = (k - 1) / kPanel * kPanel; p0 >= 0; p0 -= kPanel) {
    const int nb = min(kPanel, k - p0);
    // Four columns a warp at once (beyond nb the last one again).
    constexpr int kWarps = kSolveThreads / 32, kEach = kPanel / kWarps;
    double v[kEach];
    const double* col[kEach];
#pragma unroll
    for (int c = 0; c < kEach; ++c) {
      v[c] = 0.0;
      col[c] = A + (int64_t)(p0 + min(warp + c * kWarps, nb - 1)) * m;
    }
#pragma unroll 2
    for (int i = p0 + nb + lane; i < m; i += 32) {
      const double yi = y[i];
#pragma unroll
      for (int c = 0; c < kEach; ++c) v[c] += col[c][i] * yi;
    }
#pragma unroll
    for (int c = 0; c < kEach; ++c) {
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
      if (lane == 0) part[warp + c * kWarps] = v[c];
    }
    __syncthreads();
    if (tid < 32) {
      const double* D = diag + (int64_t)(diag_offset[s] + p0 / kPanel) * kPanel * kPanel;
      double l[kPanel], v = tid < nb ? y[p0 + tid] - part[tid] : 0.0;
      const double inv = 1.0 / D[tid * kPanel + tid];
#pragma unroll
      for (int j = 0; j < kPanel; ++j) l[j] = D[tid * kPanel + j];  // L(j, tid)
#pragma unroll
      for (int j = kPanel - 1; j >= 0; --j) {
        const double xj = __shfl_sync(0xffffffffu, v * inv, j);
        v = tid == j ? xj : v - (tid < j ? l[j] * xj : 0.0);
      }
      if (tid < nb) {
        y[p0 + tid] = v;
        x[me.x + p0 + tid] = v;
      }
    }
    __syncthreads();
  }
}

}  // namespace

void front_order(const std::vector<int32_t>& fill_order, const std::vector<std::vector<int32_t>>& members,
                 const std::vector<int32_t>& group_ptr, const std::vector<int32_t>& group_adj, FrontOrder& order) {
  const int32_t n = (int32_t)fill_order.size();
  std::vector<int32_t> at((size_t)n);
  for (int32_t i = 0; i < n; ++i) at[(size_t)fill_order[(size_t)i]] = i;
  // The elimination tree (Liu's algorithm, ancestors compressed).
  std::vector<int32_t> parent((size_t)n, -1), ancestor((size_t)n, -1);
  for (int32_t i = 0; i < n; ++i) {
    const int32_t g = fill_order[(size_t)i];
    for (int32_t q = group_ptr[(size_t)g]; q < group_ptr[(size_t)g + 1]; ++q) {
      int32_t j = at[(size_t)group_adj[(size_t)q]];
      while (j != -1 && j < i) {
        const int32_t next = ancestor[(size_t)j];
        ancestor[(size_t)j] = i;
        if (next == -1) parent[(size_t)j] = i;
        j = next;
      }
    }
  }
  // Its postorder, children in their order.
  std::vector<int32_t> head((size_t)n, -1), next((size_t)n, -1), post;
  post.reserve((size_t)n);
  for (int32_t i = n - 1; i >= 0; --i)
    if (parent[(size_t)i] >= 0) {
      next[(size_t)i] = head[(size_t)parent[(size_t)i]];
      head[(size_t)parent[(size_t)i]] = i;
    }
  std::vector<int32_t> stack;
  for (int32_t root = 0; root < n; ++root) {
    if (parent[(size_t)root] >= 0) continue;
    stack.push_back(root);
    while (!stack.empty()) {
      const int32_t v = stack.back();
      const int32_t c = head[(size_t)v];
      if (c >= 0) {
        head[(size_t)v] = next[(size_t)c];
        stack.push_back(c);
      } else {
        post.push_back(v);
        stack.pop_back();
      }
    }
  }
  std::vector<int32_t> where((size_t)n);  // fill place -> postorder place
  for (int32_t i = 0; i < n; ++i) where[(size_t)post[(size_t)i]] = i;
  order.parent.assign((size_t)n, -1);
  order.offsets.assign((size_t)n + 1, 0);
  order.ptr.assign((size_t)n + 1, 0);
  order.perm.clear();
  order.adj.clear();
  for (int32_t i = 0; i < n; ++i) {
    const int32_t v = post[(size_t)i], g = fill_order[(size_t)v];
    if (parent[(size_t)v] >= 0) order.parent[(size_t)i] = where[(size_t)parent[(size_t)v]];
    for (int32_t row : members[(size_t)g]) order.perm.push_back(row);
    order.offsets[(size_t)i + 1] = (int32_t)order.perm.size();
    for (int32_t q = group_ptr[(size_t)g]; q < group_ptr[(size_t)g + 1]; ++q) {
      const int32_t j = where[(size_t)at[(size_t)group_adj[(size_t)q]]];
      if (j > i) order.adj.push_back(j);
    }
    std::sort(order.adj.begin() + order.ptr[(size_t)i], order.adj.end());
    order.ptr[(size_t)i + 1] = (int32_t)order.adj.size();
  }
}

Multifrontal::~Multifrontal() {
  for (void* p : owned_) cudaFree(p);
}

template <class T>
cudaError_t Multifrontal::upload(T** out, const std::vector<T>& in) {
  void* p = nullptr;
  cudaError_t err = cudaMalloc(&p, std::max<size_t>(1, in.size()) * sizeof(T));
  if (err != cudaSuccess) return err;
  owned_.push_back(p);
  *out = static_cast<T*>(p);
  if (in.empty()) return cudaSuccess;
  return cudaMemcpy(p, in.data(), in.size() * sizeof(T), cudaMemcpyHostToDevice);
}

cudaError_t Multifrontal::build(const FrontOrder& order, const std::vector<int32_t>& rowptr,
                                const std::vector<int32_t>& col, size_t most) {
  const int32_t ng = (int32_t)order.parent.size();
  n_ = order.offsets.back();
  auto width = [&](int32_t a, int32_t b) { return order.offsets[(size_t)b] - order.offsets[(size_t)a]; };
  // Subtrees: rows in them and their first group (postorder: contiguous).
  std::vector<int32_t> rows_under((size_t)ng), first((size_t)ng);
  for (int32_t v = 0; v < ng; ++v) {
    rows_under[(size_t)v] += width(v, v + 1);
    if (rows_under[(size_t)v] == width(v, v + 1)) first[(size_t)v] = v;
    const int32_t p = order.parent[(size_t)v];
    if (p >= 0) {
      if (rows_under[(size_t)p] == 0) first[(size_t)p] = first[(size_t)v];
      rows_under[(size_t)p] += rows_under[(size_t)v];
    }
  }
  // Fronts in postorder: groups [g0, g1), the groups below them.
  struct Front {
    int32_t g0, g1;
    std::vector<int32_t> below;
    std::vector<int32_t> kids;
    int parent = -1, level = 0;
  };
  std::vector<Front> fronts;
  std::vector<int32_t> front_of((size_t)ng, -1), mark((size_t)ng, -1);
  // The groups after `last` reached from groups [a, last] and the fronts kids.
  auto reach = [&](int32_t a, int32_t last, const std::vector<int32_t>& kids, int32_t stamp) {
    std::vector<int32_t> out;
    auto take = [&](int32_t g) {
      if (g > last && mark[(size_t)g] != stamp) {
        mark[(size_t)g] = stamp;
        out.push_back(g);
      }
    };
    for (int32_t g = a; g <= last; ++g)
      for (int32_t q = order.ptr[(size_t)g]; q < order.ptr[(size_t)g + 1]; ++q) take(order.adj[(size_t)q]);
    for (int32_t c : kids)
      for (int32_t g : fronts[(size_t)c].below) take(g);
    std::sort(out.begin(), out.end());
    return out;
  };
  auto weight = [&](const std::vector<int32_t>& groups) {
    int64_t w = 0;
    for (int32_t g : groups) w += width(g, g + 1);
    return w;
  };
  std::vector<std::vector<int32_t>> waiting((size_t)ng);  // fronts whose parent group is this one
  auto attach = [&](int32_t f) {
    const Front& fr = fronts[(size_t)f];
    if (!fr.below.empty()) waiting[(size_t)fr.below.front()].push_back(f);
  };
  int32_t stamp = 0;
  for (int32_t v = 0; v < ng; ++v) {
    const int32_t p = order.parent[(size_t)v];
    if (rows_under[(size_t)v] <= kLeafRows) {
      if (p >= 0 && rows_under[(size_t)p] <= kLeafRows) continue;  // inside a leaf
      Front fr;
      fr.g0 = first[(size_t)v];
      fr.g1 = v + 1;
      fr.below = reach(fr.g0, v, {}, stamp++);
      fronts.push_back(std::move(fr));
      attach((int32_t)fronts.size() - 1);
      continue;
    }
    // A group above the leaves: joined to the front that ends before it when
    // that is its child and their patterns (nearly) nest, else a front.
    std::vector<int32_t> kids = std::move(waiting[(size_t)v]);
    Front* prev = fronts.empty() ? nullptr : &fronts.back();
    const bool child_before = prev && prev->g1 == v && !prev->below.empty() && prev->below.front() == v &&
                              rows_under[(size_t)v - 1] > kLeafRows;
    std::vector<int32_t> below = reach(v, v, kids, stamp++);
    if (child_before) {
      const int64_t had = weight(prev->below) - width(v, v + 1), now = weight(below);
      const int64_t columns = width(prev->g0, prev->g1);
      if (now <= had || (now - had) * columns <= (had + columns) * (columns < kPanel ? columns : columns / 8)) {
        const int32_t self = (int32_t)fronts.size() - 1;
        prev->g1 = v + 1;
        prev->below = std::move(below);
        for (int32_t c : kids)
          if (c != self) prev->kids.push_back(c);
        attach(self);
        continue;
      }
    }
    Front fr;
    fr.g0 = v;
    fr.g1 = v + 1;
    fr.below = std::move(below);
    fr.kids = std::move(kids);
    fronts.push_back(std::move(fr));
    attach((int32_t)fronts.size() - 1);
  }
  const int nf = (int)fronts.size();
  for (int f = 0; f < nf; ++f)
    for (int32_t g = fronts[(size_t)f].g0; g < fronts[(size_t)f].g1; ++g) front_of[(size_t)g] = f;
  int levels = 0;
  for (int f = 0; f < nf; ++f) {
    Front& fr = fronts[(size_t)f];
    std::sort(fr.kids.begin(), fr.kids.end());
    for (int32_t c : fr.kids) {
      fronts[(size_t)c].parent = f;
      fr.level = std::max(fr.level, fronts[(size_t)c].level + 1);
    }
    levels = std::max(levels, fr.level + 1);
  }
  // The tables.
  std::vector<int4> front((size_t)nf);
  std::vector<int64_t> offset((size_t)nf), y_offset((size_t)nf);
  std::vector<int32_t> diag_offset((size_t)nf), rows, place;
  std::vector<int2> children((size_t)nf);
  std::vector<int32_t> child;
  int64_t at = 0, y_at = 0;
  int32_t diag_at = 0;
  for (int f = 0; f < nf; ++f) {
    const Front& fr = fronts[(size_t)f];
    int4& t = front[(size_t)f];
    t.x = order.offsets[(size_t)fr.g0];
    t.y = width(fr.g0, fr.g1);
    t.w = (int)rows.size();
    for (int32_t g : fr.below)
      for (int32_t r = order.offsets[(size_t)g]; r < order.offsets[(size_t)g + 1]; ++r) rows.push_back(r);
    t.z = t.y + (int)rows.size() - t.w;
    offset[(size_t)f] = at;
    at += (int64_t)t.z * t.z;
    y_offset[(size_t)f] = y_at;
    y_at += t.z;
    diag_offset[(size_t)f] = diag_at;
    diag_at += (t.y + kPanel - 1) / kPanel;
    children[(size_t)f] = make_int2((int)child.size(), (int)fr.kids.size());
    child.insert(child.end(), fr.kids.begin(), fr.kids.end());
  }
  arena_ = (size_t)at;
  // A front's place of a row: its own columns first, then its rows below.
  auto place_in = [&](int f, int32_t row) {
    const int4& t = front[(size_t)f];
    if (row < t.x + t.y) return row - t.x;
    const auto lo = rows.begin() + t.w, hi = lo + (t.z - t.y);
    return (int32_t)(t.y + (std::lower_bound(lo, hi, row) - lo));
  };
  place.assign(rows.size(), 0);
  for (int f = 0; f < nf; ++f) {
    const int p = fronts[(size_t)f].parent;
    if (p < 0) continue;
    const int4& t = front[(size_t)f];
    for (int i = 0; i < t.z - t.y; ++i) place[(size_t)(t.w + i)] = place_in(p, rows[(size_t)(t.w + i)]);
  }
  std::vector<int32_t> src;
  std::vector<int64_t> dst;
  {
    std::vector<int32_t> front_of_row((size_t)n_);
    for (int32_t g = 0; g < ng; ++g)
      for (int32_t r = order.offsets[(size_t)g]; r < order.offsets[(size_t)g + 1]; ++r)
        front_of_row[(size_t)r] = front_of[(size_t)g];
    src.reserve(col.size() / 2 + (size_t)n_);
    dst.reserve(col.size() / 2 + (size_t)n_);
    for (int32_t i = 0; i < n_; ++i)
      for (int32_t q = rowptr[(size_t)i]; q < rowptr[(size_t)i + 1]; ++q) {
        const int32_t j = col[(size_t)q];  // entry (i, j), row i
        if (j > i) break;
        const int f = front_of_row[(size_t)j];
        const int4& t = front[(size_t)f];
        src.push_back(q);
        dst.push_back(offset[(size_t)f] + (int64_t)(j - t.x) * t.z + place_in(f, i));
      }
  }
  entries_ = (int64_t)src.size();
  // What the lists of tasks take is known before they are made: the tiles',
  // one list a panel, grow with the cube of a front (a tenth of its own
  // bytes at 40,000 rows).
  int64_t num_adds = 0, num_panels = 0, num_tiles = 0;
  for (int f = 0; f < nf; ++f) {
    const int4& t = front[(size_t)f];
    auto up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
    if (children[(size_t)f].y > 0) num_adds += up(t.z, kAddColumns);
    for (int p0 = 0; p0 < t.y; p0 += kPanel) {
      const int base = std::min(p0 + kPanel, t.y);
      const int64_t tiles = up(t.z - base, kTile), own = up(t.y - base, kTile);
      num_panels += std::max<int64_t>(1, up(t.z - base, kRowChunk));
      num_tiles += own * (own + 1) / 2 + (tiles - own) * own;
    }
    const int64_t rest = up(t.z - t.y, kTile);
    num_tiles += rest * (rest + 1) / 2;
  }
  auto some = [](int64_t n) { return (size_t)std::max<int64_t>(1, n); };  // as upload and room allocate
  const size_t bytes =
      (some(at) + some((int64_t)diag_at * kPanel * kPanel) + some(y_at)) * sizeof(double) +
      some(nf) * (sizeof(int4) + sizeof(int2) + 2 * sizeof(int64_t) + 2 * sizeof(int32_t)) +
      (some((int64_t)child.size()) + 2 * some((int64_t)rows.size()) + some(entries_)) * sizeof(int32_t) +
      some(entries_) * sizeof(int64_t) + (some(num_adds) + some(num_panels)) * sizeof(int2) + some(num_tiles) * sizeof(int4);
  if (bytes > most || std::max(num_tiles, std::max(num_panels, num_adds)) > INT32_MAX)
    return cudaErrorMemoryAllocation;
  // Tasks, level by level.
  std::vector<int32_t> by_level;
  std::vector<int2> adds, panel_tasks;
  std::vector<int4> tile_tasks;
  levels_.assign((size_t)levels, Level());
  std::vector<std::vector<int>> members((size_t)levels);
  for (int f = 0; f < nf; ++f) members[(size_t)fronts[(size_t)f].level].push_back(f);
  for (int l = 0; l < levels; ++l) {
    Level& L = levels_[(size_t)l];
    L.front0 = (int)by_level.size();
    L.fronts = (int)members[(size_t)l].size();
    L.adds0 = (int)adds.size();
    int steps = 0;
    for (int f : members[(size_t)l]) {
      by_level.push_back(f);
      const int4& t = front[(size_t)f];
      if (children[(size_t)f].y > 0)
        for (int c = 0; c < t.z; c += kAddColumns) adds.push_back(make_int2(f, c));
      steps = std::max(steps, (t.y + kPanel - 1) / kPanel);
    }
    L.adds = (int)adds.size() - L.adds0;
    for (int s = 0; s < steps; ++s) {
      const int p0 = s * kPanel;
      L.panel0.push_back((int)panel_tasks.size());
      L.tile0.push_back((int)tile_tasks.size());
      for (int f : members[(size_t)l]) {
        const int4& t = front[(size_t)f];
        if (p0 >= t.y) continue;
        const int base = std::min(p0 + kPanel, t.y);
        int r = base;
        do {
          panel_tasks.push_back(make_int2(f, r));
          r += kRowChunk;
        } while (r < t.z);
        const int tiles = (t.z - base + kTile - 1) / kTile, own = (t.y - base + kTile - 1) / kTile;
        for (int i = 0; i < tiles; ++i)
          for (int j = 0; j <= i && j < own; ++j) tile_tasks.push_back(make_int4(f, i, j, 0));
      }
      L.panels.push_back((int)panel_tasks.size() - L.panel0.back());
      L.tiles.push_back((int)tile_tasks.size() - L.tile0.back());
    }
    L.rest0 = (int)tile_tasks.size();
    for (int f : members[(size_t)l]) {
      const int4& t = front[(size_t)f];
      const int tiles = (t.z - t.y + kTile - 1) / kTile;
      for (int i = 0; i < tiles; ++i)
        for (int j = 0; j <= i; ++j) tile_tasks.push_back(make_int4(f, i, j, 0));
    }
    L.rest = (int)tile_tasks.size() - L.rest0;
  }
  cudaError_t err = upload(&front_, front);
  auto next = [&](cudaError_t e) {
    if (err == cudaSuccess) err = e;
  };
  if (err == cudaSuccess) next(upload(&offset_, offset));
  if (err == cudaSuccess) next(upload(&y_offset_, y_offset));
  if (err == cudaSuccess) next(upload(&diag_offset_, diag_offset));
  if (err == cudaSuccess) next(upload(&children_, children));
  if (err == cudaSuccess) next(upload(&child_, child));
  if (err == cudaSuccess) next(upload(&rows_, rows));
  if (err == cudaSuccess) next(upload(&place_, place));
  if (err == cudaSuccess) next(upload(&src_, src));
  if (err == cudaSuccess) next(upload(&dst_, dst));
  if (err == cudaSuccess) next(upload(&order_, by_level));
  if (err == cudaSuccess) next(upload(&adds_, adds));
  if (err == cudaSuccess) next(upload(&panel_tasks_, panel_tasks));
  if (err == cudaSuccess) next(upload(&tile_tasks_, tile_tasks));
  auto room = [&](double** p, size_t n) {
    void* q = nullptr;
    const cudaError_t e = cudaMalloc(&q, std::max<size_t>(1, n) * sizeof(double));
    if (e == cudaSuccess) {
      owned_.push_back(q);
      *p = static_cast<double*>(q);
    }
    return e;
  };
  if (err == cudaSuccess) next(room(&arena_dev_, arena_));
  if (err == cudaSuccess) next(room(&diag_, (size_t)diag_at * kPanel * kPanel));
  if (err == cudaSuccess) next(room(&y_, (size_t)y_at));
  // The uploads have landed before any other stream reads them.
  if (err == cudaSuccess) next(cudaStreamSynchronize(cudaStreamLegacy));
  return err;
}

cudaError_t Multifrontal::factor(const double* values, int32_t* failed, cudaStream_t stream) {
  const Fronts f{front_, offset_, arena_dev_};
  cudaError_t err = cudaMemsetAsync(arena_dev_, 0, arena_ * sizeof(double), stream);
  if (err != cudaSuccess) return err;
  err = cudaMemsetAsync(failed, kAllPositive & 0xff, sizeof(int32_t), stream);
  if (err != cudaSuccess) return err;
  const int64_t blocks = std::min<int64_t>((entries_ + 255) / 256, 148 * 16);
  scatter_values_kernel<<<(unsigned)std::max<int64_t>(1, blocks), 256, 0, stream>>>(values, src_, dst_, entries_,
                                                                                   arena_dev_);
  for (const Level& L : levels_) {
    if (L.adds)
      extend_add_kernel<<<L.adds, 32 * kAddColumns, 0, stream>>>(f, adds_ + L.adds0, children_, child_, place_);
    for (size_t s = 0; s < L.panels.size(); ++s) {
      const int p0 = (int)s * kPanel;
      panel_kernel<<<L.panels[s], kRowChunk, 0, stream>>>(f, panel_tasks_ + L.panel0[s], p0, diag_offset_, diag_,
                                                          failed);
      if (L.tiles[s]) tile_kernel<<<L.tiles[s], 128, 0, stream>>>(f, tile_tasks_ + L.tile0[s], p0);
    }
    if (L.rest) tile_kernel<<<L.rest, 128, 0, stream>>>(f, tile_tasks_ + L.rest0, -1);
  }
  return cudaGetLastError();
}

cudaError_t Multifrontal::solve(const double* b, double* x, cudaStream_t stream) {
  const Fronts f{front_, offset_, arena_dev_};
  for (const Level& L : levels_)
    forward_kernel<<<L.fronts, kSolveThreads, 0, stream>>>(f, order_ + L.front0, children_, child_, place_, y_offset_,
                                                           diag_offset_, diag_, b, y_);
  for (auto L = levels_.rbegin(); L != levels_.rend(); ++L)
    backward_kernel<<<L->fronts, kSolveThreads, 0, stream>>>(f, order_ + L->front0, rows_, y_offset_, diag_offset_,
                                                             diag_, y_, x);
  return cudaGetLastError();
}

}  // namespace sbk
