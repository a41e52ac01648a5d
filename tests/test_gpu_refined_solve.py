"""The symmetric solve to the last bits on blocks of thin sheets, where a plain
Cholesky solve in 64 bits loses three to four digits.

The reference solution is kept as a sum of two doubles and refined on exact
residuals. One step of refinement on a residual of twice the precision leaves
the rounding of the sum x + d, 2^-53 of every entry, and the first solve's
error squared, below 1e-20: the error is at most 1.2e-16 of the solution's
norm. Twice that is asked, whatever the right-hand side."""
from __future__ import annotations

import math

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla
import torch

pytestmark = pytest.mark.gpu


def two_product(a, b):
    """a b = p + e exactly (Dekker)."""
    def split(v):
        t = 134217729.0 * v
        hi = t - (t - v)
        return hi, v - hi
    p = a * b
    (ah, al), (bh, bl) = split(a), split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def exact_solution(K, b):
    """K^-1 b as hi + lo (K CSR)."""
    lu = spla.splu(K.tocsc())
    hi, lo = lu.solve(b), np.zeros_like(b)
    for _ in range(4):
        p, e = two_product(K.data, hi[K.indices])
        q = K.data * lo[K.indices]
        parts = [p, e, q]
        r = np.array([math.fsum([b[i]] + [-v for t in parts for v in t[K.indptr[i]:K.indptr[i + 1]]])
                      for i in range(len(b))])
        d = lu.solve(r) + lo
        s = hi + d
        z = s - hi
        hi, lo = s, (hi - (s - z)) + (d - z)
    return hi, lo


# One element through the thickness and two; a block of one front, one of several levels.
@pytest.mark.parametrize("nx,ny,nz", [(5, 4, 1), (9, 9, 2), (40, 40, 1), (23, 17, 2)])
@pytest.mark.parametrize("load", ["corner", "random", "zero"])
def test_symmetric_solve_is_exact_to_rounding(pkg, cuda, nx, ny, nz, load):
    cell = 1.0e-3
    mesh = pkg.structured_hex_mesh(nx, ny, nz, nx * cell, ny * cell, nz * 0.5 * cell)
    s = pkg.NonlinearSystem(mesh, pkg.material.aluminium_swift(), kinematics="logarithmic")
    values = s.evaluate(torch.zeros(mesh.num_dofs, dtype=torch.float64, device=cuda), 0.0, True).tangent.clone()
    x, y = mesh.coords[:, 0], mesh.coords[:, 1]
    free = np.flatnonzero(np.repeat(~(np.isclose(x, x.min()) | np.isclose(y, y.min())), 3)).astype(np.int32)
    n = s.num_dofs
    full = sp.csc_matrix((values.cpu().numpy(), s.inner.cpu().numpy(), s.outer.cpu().numpy()), shape=(n, n))
    K = full[free][:, free].tocsr()
    b = np.zeros(len(free))
    if load == "corner":
        b[-1] = 1.0
    elif load == "random":
        b = np.random.default_rng(nx).standard_normal(len(free))
    part = pkg.PartitionedFactor.for_system(s, free)
    assert part.factorize(values, symmetric=True) == 1
    got = part.solve(torch.tensor(b, device=cuda)).cpu().numpy()
    if load == "zero":
        assert not got.any()
        return
    hi, lo = exact_solution(K, b)
    assert np.linalg.norm((got - hi) - lo) <= 2.4e-16 * np.linalg.norm(hi)
