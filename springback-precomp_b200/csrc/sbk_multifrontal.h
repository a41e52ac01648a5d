// A multifrontal Cholesky of the partition's block on the device
// (sbk_multifrontal.cu): the analysis on the host, once per partition; the
// factorisation and the solves as a few launches per level of the tree.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace sbk {

// The rows of a symmetric pattern, grouped (a group: the free DOFs of one
// node), in an order that eliminates it: perm[i] is the row at place i, the
// rows of a group together; offsets[g] the first place of the group at g.
struct FrontOrder {
  std::vector<int32_t> perm;
  std::vector<int32_t> offsets;
  // The groups' lower patterns in that order: group g's neighbours after it.
  std::vector<int32_t> ptr, adj;
  std::vector<int32_t> parent;  // the elimination tree, postordered (-1: a root)
};

// Completes `order` from a fill-reducing order of the groups (place ->
// group): the elimination tree and its postorder. members[g]: the rows of
// group g; group_ptr / group_adj: the groups' pattern (symmetric, without
// the diagonal).
void front_order(const std::vector<int32_t>& fill_order, const std::vector<std::vector<int32_t>>& members,
                 const std::vector<int32_t>& group_ptr, const std::vector<int32_t>& group_adj, FrontOrder& order);

class Multifrontal {
 public:
  Multifrontal() = default;
  ~Multifrontal();
  Multifrontal(const Multifrontal&) = delete;
  Multifrontal& operator=(const Multifrontal&) = delete;

  // The fronts of the matrix whose CSR pattern (rowptr, col; in `order`) is
  // given, and their device storage. cudaErrorMemoryAllocation when that
  // takes more than `most` bytes, all tables counted, or is not to be had.
  cudaError_t build(const FrontOrder& order, const std::vector<int32_t>& rowptr, const std::vector<int32_t>& col,
                    size_t most);
  // A = L L^T of the CSR values (device). *failed (device): the first column
  // of non-positive pivot, or kAllPositive.
  static constexpr int32_t kAllPositive = 0x7f7f7f7f;  // four bytes alike: a memset's
  cudaError_t factor(const double* values, int32_t* failed, cudaStream_t stream);
  // x = A^-1 b (device, in `order`; x and b may not alias).
  cudaError_t solve(const double* b, double* x, cudaStream_t stream);

 private:
  struct Level {
    int front0 = 0, fronts = 0;         // of the fronts in level order
    int adds = 0, adds0 = 0;            // extend-add tasks
    std::vector<int> panel0, panels, tile0, tiles;  // per panel step
    int rest = 0, rest0 = 0;            // tiles of the remainders
  };
  template <class T>
  cudaError_t upload(T** out, const std::vector<T>& in);

  int32_t n_ = 0;
  int64_t entries_ = 0;    // lower entries of A
  size_t arena_ = 0;       // doubles of all fronts
  std::vector<Level> levels_;
  std::vector<void*> owned_;
  // device
  int4* front_ = nullptr;        // per front: first column, columns, rows, first row index
  int64_t* offset_ = nullptr;    // its place in the arena
  int64_t* y_offset_ = nullptr;  // of its vector in the solves
  int32_t* diag_offset_ = nullptr;  // its first diagonal block
  int2* children_ = nullptr;     // per front: first child, children (of child_)
  int32_t* child_ = nullptr;     // fronts
  int32_t* rows_ = nullptr;      // per front: the rows below its columns
  int32_t* place_ = nullptr;     // and their places in the parent's front
  int32_t* src_ = nullptr;       // lower entries: position in the values
  int64_t* dst_ = nullptr;       // and in the arena
  int32_t* order_ = nullptr;     // fronts by level
  int2* adds_ = nullptr;         // (front, first column)
  int2* panel_tasks_ = nullptr;  // (front, first row)
  int4* tile_tasks_ = nullptr;   // (front, row tile, column tile)
  double* arena_dev_ = nullptr;
  double* diag_ = nullptr;       // factorised diagonal blocks
  double* y_ = nullptr;
};

}  // namespace sbk
