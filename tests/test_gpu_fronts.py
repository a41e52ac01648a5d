"""The multifrontal Cholesky at the sizes where its fronts, panels (32
columns) and tiles (64 rows) end: blocks of 1 row up to several levels of
fronts, odd free sets, parts that do not touch, against a dense solve.

The values are random, symmetric and diagonally dominant: the condition
number is at most 2 * rowsum + 1 < 500, a front has fewer than 500 rows, so a
Cholesky's relative error is below 500 * 500 * 2^-53 * 2 < 1e-10 and, with
its roundings unaligned, near the root of that; 1e-12 is asked."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def grid_matrix(shape, seed, parts=1):
    """CSC of a node grid's 3 x 3 blocks (neighbours within one step in every
    direction), `parts` such grids that do not touch."""
    rng = np.random.default_rng(seed)
    ijk = np.stack(np.meshgrid(*[np.arange(k) for k in shape], indexing="ij"), -1).reshape(-1, 3)
    near = (np.abs(ijk[:, None] - ijk[None]).max(-1) <= 1).astype(float)
    near = sp.kron(sp.identity(parts), sp.csr_matrix(near))
    pattern = sp.kron(near, np.ones((3, 3))).tocoo()
    n = pattern.shape[0]
    upper = np.triu(rng.uniform(-1.0, 1.0, (n, n)), 1)
    dense = np.zeros((n, n))
    dense[pattern.row, pattern.col] = (upper + upper.T)[pattern.row, pattern.col]
    np.fill_diagonal(dense, np.abs(dense).sum(1) + 1.0)
    csc = sp.csc_matrix((np.ones(len(pattern.row)), (pattern.row, pattern.col)), shape=(n, n))
    csc.sort_indices()
    col = np.repeat(np.arange(n), np.diff(csc.indptr))
    return csc.indptr.astype(np.int32), csc.indices.astype(np.int32), dense[csc.indices, col], dense


# (nodes, parts, free): free is how many DOFs stay, or the fraction of them.
@pytest.mark.parametrize("shape,parts,free", [
    ((1, 1, 1), 1, 1), ((1, 1, 1), 1, 3), ((2, 1, 1), 1, 5), ((4, 2, 2), 1, 31), ((4, 2, 2), 1, 32),
    ((4, 2, 2), 1, 33), ((11, 3, 1), 1, 95), ((11, 3, 1), 1, 96), ((11, 3, 1), 1, 97), ((40, 1, 1), 1, 1.0),
    ((17, 13, 2), 1, 1.0), ((17, 13, 2), 1, 0.4), ((9, 9, 9), 1, 0.8), ((5, 5, 2), 5, 0.9)])
@pytest.mark.parametrize("definite", [True, False])
def test_solves_at_the_edges_of_fronts(pkg, cuda, shape, parts, free, definite):
    outer, inner, values, dense = grid_matrix(shape, 5, parts)
    n = len(outer) - 1
    rng = np.random.default_rng(9)
    count = free if isinstance(free, int) else int(free * n)
    keep = np.sort(rng.choice(n, count, replace=False)).astype(np.int32)
    if not definite:  # one pivot negative, dominance kept
        at = int(keep[count // 2])
        dense[at, at] = -dense[at, at]
        values[(inner == at) & (np.repeat(np.arange(n), np.diff(outer)) == at)] *= -1.0
    part = pkg.PartitionedFactor(torch.tensor(outer, device=cuda), torch.tensor(inner, device=cuda), keep)
    v = torch.tensor(values, device=cuda)
    b = rng.standard_normal(count)
    want = np.linalg.solve(dense[np.ix_(keep, keep)], b)
    for _ in range(2):  # the second factorisation takes the first one's analysis
        assert part.factorize(v, symmetric=True) == (1 if definite else 4)
        for transpose in (False, True):
            got = part.solve(torch.tensor(b, device=cuda), transpose=transpose).cpu().numpy()
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
