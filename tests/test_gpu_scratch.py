"""The tile kernels' scratch where device memory is short: a mesh whose own
arrays fit is taken, its elements in more and smaller launches, with the
same results to the bit."""
from __future__ import annotations

import contextlib
import gc
import importlib

import numpy as np
import pytest
import torch

from conftest import X_DISTORTED, deformation, oracle_to_device

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


@contextlib.contextmanager
def only(cuda, n):
    """Takes the device's memory but n bytes for a while."""
    taken = [torch.empty(max(0, free_bytes() - n), dtype=torch.uint8, device=cuda)]
    try:
        yield
    finally:
        taken.clear()
        free_bytes()


def test_an_element_refused_for_memory_is_not_taken(pkg, cuda):
    system = importlib.import_module("springback-precomp_b200.system")
    system.set_local_iteration("single")
    try:
        s, u = sheet(pkg, cuda)
    finally:
        system.set_local_iteration("phases")
    want = s.evaluate(u, 0.0, True).internal.cpu()
    with only(cuda, 8 * MB):
        with pytest.raises(pkg.SbkError):
            s.set_element("standard")
        assert torch.equal(s.evaluate(u, 0.0, True).internal.cpu(), want)
        s.commit()
    s.set_element("standard")
    t, _ = sheet(pkg, cuda, "standard")
    t.set_committed(s.committed_all())
    assert torch.equal(s.evaluate(u, 0.0, True).internal.cpu(), t.evaluate(u, 0.0, True).internal.cpu())


def results(s, u, standard):
    ev = s.evaluate(u, 0.0, True)
    out = [ev.internal.cpu(), ev.tangent.cpu(), torch.tensor([ev.energy, ev.gross, ev.yielding_points])]
    out += [torch.tensor(s.trial_states()), torch.tensor(s.trial_modes())]
    if not standard:
        lam = torch.linspace(-1.0, 1.0, s.num_dofs, device=u.device, dtype=torch.float64)
        out.append(s.vjp_x(u, lam, frozen=False).cpu())
    return out


@pytest.mark.parametrize("element", ["incompatible_modes", "standard"])
def test_a_system_takes_smaller_launches(pkg, cuda, element):
    s, u = sheet(pkg, cuda, element)
    want = results(s, u, element == "standard")
    assert 0 < want[2][2] < 20 * s.mesh.num_elements
    before = free_bytes()
    del s
    whole = free_bytes() - before
    assert whole > 300 * MB
    with only(cuda, whole - 200 * MB):
        s, _ = sheet(pkg, cuda, element)
        got = results(s, u, element == "standard")
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_a_batch_takes_smaller_launches(pkg, cuda):
    n, mat = 20000, pkg.material.hill_chaboche_sheet()
    mesh = pkg.structured_hex_mesh(n, 1, 1, n * 1.0e-3, 1.0e-3, 1.0e-3)
    x = torch.tensor(mesh.element_coordinates().reshape(n, 24), device=cuda)
    gen = torch.Generator(device=cuda).manual_seed(6)
    u = 4.0e-6 * torch.randn((n, 24), generator=gen, device=cuda, dtype=torch.float64)
    state = torch.zeros((mat.state_fields, n, 20), device=cuda, dtype=torch.float64)

    def run():
        r = pkg.element_batch(mat, x, u, state, kinematics="logarithmic", thickness_points=5)
        return [getattr(r, k).cpu() for k in ("force", "tangent", "energy", "states", "alpha", "code", "iterations")]

    want = run()
    assert (want[5] == 0).all() and (want[6] > 0).any()
    outputs = sum(t.numel() * t.element_size() for t in want)
    with only(cuda, outputs + 150 * MB):
        got = run()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", ["chaboche_steel", "perfectly_plastic"])
def test_elements_handed_on_in_every_launch(pkg, orc, cuda, name):
    """The list of the elements handed to the single kernel runs on over the
    launches: reversals that search and that turn K_aa indefinite and elements
    that fail, spread over all of them."""
    n, mat = 20000, getattr(pkg.material, name)()
    kw = dict(kinematics="logarithmic", in_plane=2, thickness=5)
    X = X_DISTORTED.reshape(1, 24)
    first = orc.elements(mat.as_dict(), X, deformation(X_DISTORTED, 0.02).reshape(1, 24), want_tangent=False, **kw)
    kinds = np.stack([deformation(X_DISTORTED, 0.02 * f) for f in (-6.0, -10.0, -15.0, 1.3, 1.0)])
    kinds[4, 10] = np.nan
    m = len(kinds)
    states, alpha = np.repeat(first["states"], m, axis=0), np.repeat(first["alpha"].reshape(1, 9), m, axis=0)
    ref = orc.elements(mat.as_dict(), np.repeat(X, m, axis=0), kinds, states, alpha, **kw)
    at = np.random.default_rng(8).integers(0, m, n)
    dev = np.ascontiguousarray(oracle_to_device(states, mat.kinematic_terms)[:, at])
    args = [torch.tensor(v, device=cuda) for v in (np.repeat(X, n, axis=0), kinds[at], dev, alpha[at])]

    def run():
        r = pkg.element_batch(mat, *args, kinematics="logarithmic", thickness_points=5)
        return [getattr(r, k).cpu() for k in ("force", "tangent", "energy", "alpha", "code", "iterations", "states")]

    want = run()
    np.testing.assert_array_equal(want[4].numpy(), ref["status"][at])
    outputs = sum(t.numel() * t.element_size() for t in want)
    with only(cuda, outputs + 150 * MB):
        got = run()
    assert torch.equal(got[4], want[4])
    ok = want[4] == 0
    for a, b in zip(got[:6], want[:6]):
        assert torch.equal(a[ok], b[ok])
    assert torch.equal(got[6][:, ok], want[6][:, ok])
