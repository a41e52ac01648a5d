"""The bound on the device memory of the multifrontal Cholesky: everything
that build() allocates counts, and what exceeds the bound is refused before
anything is allocated. The analysis is host code; it is linked here with a
CUDA runtime that counts bytes."""
from __future__ import annotations

import ctypes
import importlib
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "springback-precomp_b200", "csrc")

HARNESS = """
#include "sbk_multifrontal.h"
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <numeric>
static size_t allocated;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { allocated += n; *p = std::malloc(16); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 1; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaErrorUnknown; }
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
char __cudaInitModule(void**) { return 0; }

// A grid of nx x ny x nz nodes of three rows each, in the grid's own order.
// Returns build's status; *bytes: what it allocated.
int build(int nx, int ny, int nz, size_t most, size_t* bytes) {
  const int n = nx * ny * nz;
  std::vector<std::vector<int32_t>> members(n);
  std::vector<int32_t> fill(n), ptr{0}, adj;
  std::iota(fill.begin(), fill.end(), 0);
  for (int k = 0; k < nz; ++k)
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i) {
        const int g = (k * ny + j) * nx + i;
        members[g] = {3 * g, 3 * g + 1, 3 * g + 2};
        for (int c = -1; c <= 1; ++c)
          for (int b = -1; b <= 1; ++b)
            for (int a = -1; a <= 1; ++a) {
              const int x = i + a, y = j + b, z = k + c;
              if (x < 0 || y < 0 || z < 0 || x >= nx || y >= ny || z >= nz || (!a && !b && !c)) continue;
              adj.push_back((z * ny + y) * nx + x);
            }
        ptr.push_back((int32_t)adj.size());
      }
  sbk::FrontOrder order;
  sbk::front_order(fill, members, ptr, adj, order);
  std::vector<int32_t> place(3 * n);
  for (int i = 0; i < 3 * n; ++i) place[order.perm[i]] = i;
  std::vector<int32_t> rowptr{0}, col;
  for (int i = 0; i < 3 * n; ++i) {
    const int g = order.perm[i] / 3;
    const size_t from = col.size();
    for (int c = 0; c < 3; ++c) col.push_back(place[3 * g + c]);
    for (int q = ptr[g]; q < ptr[g + 1]; ++q)
      for (int c = 0; c < 3; ++c) col.push_back(place[3 * adj[q] + c]);
    std::sort(col.begin() + from, col.end());
    rowptr.push_back((int32_t)col.size());
  }
  allocated = 0;
  sbk::Multifrontal fronts;
  const int status = (int)fronts.build(order, rowptr, col, most);
  *bytes = allocated;
  return status;
}
}
"""


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    builder = importlib.import_module("springback-precomp_b200.build")
    d = tmp_path_factory.mktemp("fronts")
    (d / "harness.cpp").write_text(HARNESS)
    lib, obj = str(d / "fronts.so"), str(d / "fronts.o")
    subprocess.run([builder.nvcc()] + builder.flags() + ["-c", os.path.join(CSRC, "sbk_multifrontal.cu"), "-o", obj],
                   check=True)
    cuda = os.path.join(os.path.dirname(os.path.dirname(builder.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + CSRC, "-I" + cuda,
                    str(d / "harness.cpp"), obj, "-o", lib], check=True)
    f = ctypes.CDLL(lib).build
    f.argtypes = [ctypes.c_int] * 3 + [ctypes.c_size_t, ctypes.POINTER(ctypes.c_size_t)]
    return f


# A leaf alone, a few fronts, fronts of over a thousand rows, whose lists of tiles weigh most.
@pytest.mark.parametrize("shape", [(1, 1, 1), (5, 3, 2), (14, 13, 3), (20, 20, 14)])
def test_everything_allocated_counts(build, shape):
    bytes_ = ctypes.c_size_t()
    assert build(*shape, 1 << 50, ctypes.byref(bytes_)) == 0
    whole = bytes_.value
    assert build(*shape, whole, ctypes.byref(bytes_)) == 0 and bytes_.value == whole
    assert build(*shape, whole - 1, ctypes.byref(bytes_)) == 2 and bytes_.value == 0  # cudaErrorMemoryAllocation
