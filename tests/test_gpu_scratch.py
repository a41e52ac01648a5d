"""The tile kernels' scratch where device memory is short."""
from __future__ import annotations

import gc
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
MB = 1 << 20


def sheet(pkg, cuda, element="incompatible_modes"):
    """20,000 elements of 20 points (282 MB of records) and a displacement at which points yield."""
    mesh = pkg.structured_hex_mesh(100, 100, 2, 0.1, 0.1, 0.002)
    s = pkg.NonlinearSystem(mesh, pkg.material.hill_chaboche_sheet(), "logarithmic", 2, 5, 2, element=element)
    gen = torch.Generator(device=cuda).manual_seed(5)
    u = 4.0e-6 * torch.randn(mesh.num_dofs, generator=gen, device=cuda, dtype=torch.float64)
    return s, u


def free_bytes():
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def leave(cuda, n):
    """Takes the device's memory but n bytes."""
    return torch.empty(max(0, free_bytes() - n), dtype=torch.uint8, device=cuda)


def test_an_element_refused_for_memory_is_not_taken(pkg, cuda):
    system = importlib.import_module("springback-precomp_b200.system")
    system.set_local_iteration("single")
    try:
        s, u = sheet(pkg, cuda)
    finally:
        system.set_local_iteration("phases")
    want = s.evaluate(u, 0.0, True).internal.cpu()
    taken = leave(cuda, 8 * MB)
    with pytest.raises(pkg.SbkError):
        s.set_element("standard")
    assert torch.equal(s.evaluate(u, 0.0, True).internal.cpu(), want)
    s.commit()
    del taken
    free_bytes()
    s.set_element("standard")
    t, _ = sheet(pkg, cuda, "standard")
    t.set_committed(s.committed_all())
    assert torch.equal(s.evaluate(u, 0.0, True).internal.cpu(), t.evaluate(u, 0.0, True).internal.cpu())
