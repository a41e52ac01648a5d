"""Elements that fail, search or are handed on, in one tile with elements that
converge: the status of each is the oracle's, and no element's results depend
on what shares its tile. Non-finite displacements are refused as the oracle
refuses them, whatever the law and the kinematics."""
from __future__ import annotations

import importlib

import numpy as np
import pytest
import torch

from conftest import X_DISTORTED, deformation, oracle_to_device

pytestmark = pytest.mark.gpu

LAWS = {"elastic": "elastic_steel", "j2": "j2_steel", "hill": "hill_sheet", "chaboche": "chaboche_steel",
        "perfect": "perfectly_plastic"}
SCALE = {"small": 4e-3, "finite": 0.02, "logarithmic": 0.1}


def law(pkg, name):
    return getattr(pkg.material, LAWS[name])()


def run(pkg, mat, X, ue, states, alpha, cuda, kin, rule):
    return pkg.element_batch(mat, torch.tensor(X, device=cuda), torch.tensor(ue, device=cuda),
                             torch.tensor(np.ascontiguousarray(states), device=cuda),
                             torch.tensor(np.ascontiguousarray(alpha), device=cuda), kinematics=kin,
                             stiffness_points=rule[0], thickness_points=rule[1])


def same_bits(a, i, b, j):
    """Element i of the batch a (code 0) has the results of element j of b."""
    for name in ("force", "tangent", "energy", "alpha", "yielding", "iterations"):
        assert torch.equal(getattr(a, name)[i], getattr(b, name)[j]), name
    assert torch.equal(a.states[:, i], b.states[:, j])


def bad_displacements(u):
    """u with a value that is no number, all of them, an infinite one of either sign."""
    out = np.tile(u, (4, 1))
    out[0, 4], out[1], out[2, 7], out[3, 22] = np.nan, np.nan, np.inf, -np.inf
    return out


# Full tiles (32, 12 elements) and an element a tile.
@pytest.mark.parametrize("rule,n", [((2, 0), 148 * 32), ((2, 5), 148 * 12), ((2, 0), 6)])
@pytest.mark.parametrize("kin", list(SCALE))
@pytest.mark.parametrize("name", ["elastic", "j2", "hill", "chaboche"])
def test_nonfinite_displacements_fail(pkg, orc, cuda, name, kin, rule, n):
    mat, X = law(pkg, name), X_DISTORTED.reshape(1, 24)
    good = [deformation(X_DISTORTED, SCALE[kin]), deformation(X_DISTORTED, -0.4 * SCALE[kin])]
    kinds = np.concatenate([good, bad_displacements(good[0])])
    m, kw = len(kinds), dict(kinematics=kin, in_plane=rule[0], thickness=rule[1])
    ref = orc.elements(mat.as_dict(), np.tile(X, (m, 1)), kinds, **kw)
    assert (ref["status"][:2] == 0).all() and (ref["status"][2:] != 0).all()
    at = np.arange(n) % m
    states, alpha = np.zeros((mat.state_fields, n, orc.rule_size(*rule, 2))), np.zeros((n, 9))
    r = run(pkg, mat, np.tile(X, (n, 1)), kinds[at], states, alpha, cuda, kin, rule)
    np.testing.assert_array_equal(r.code.cpu().numpy(), ref["status"][at])
    alone = run(pkg, mat, np.tile(X, (n, 1)), kinds[at % 2], states, alpha, cuda, kin, rule)
    assert (alone.code == 0).all()
    ok = torch.tensor(at < 2, device=cuda)
    same_bits(r, ok, alone, ok)


@pytest.mark.parametrize("kin", list(SCALE))
@pytest.mark.parametrize("name,frozen", [("elastic", False), ("j2", False), ("j2", True), ("chaboche", False)])
def test_nonfinite_evaluation_is_refused(pkg, orc, cuda, name, frozen, kin):
    """One node of a strip: the call names the first element at it and the
    oracle's reason, leaves nothing to commit, and a captured evaluation's
    summary says so too. (A frozen J2 law is the elastic one.)"""
    batch = importlib.import_module("springback-precomp_b200.batch")
    mat = law(pkg, name)
    mesh = pkg.structured_hex_mesh(6, 2, 1, 6.0e-3, 2.0e-3, 1.0e-3)
    good = torch.tensor(1.0e-6 * np.random.default_rng(3).standard_normal(mesh.num_dofs), device=cuda)
    s, t = (pkg.NonlinearSystem(mesh, mat, kin) for _ in range(2))
    for each in (s, t):
        each.set_frozen(frozen)
    s.evaluate(good, 0.0, True)
    s.commit()
    node = int(mesh.connectivity[7, 6])
    first = int(np.nonzero((mesh.connectivity == node).any(1))[0][0])
    graph = batch.GraphedEvaluation(t, good.clone())
    for value in (np.nan, np.inf):
        u = good.clone()
        u[3 * node + 1] = value
        ref = orc.system_evaluate(law(pkg, "elastic" if frozen else name).as_dict(), mesh.coords, mesh.connectivity,
                                  u.cpu().numpy(), kinematics=kin)
        assert ref["failed_element"] == first and ref["code"] != 0
        with pytest.raises(pkg.SolverError) as e:
            s.evaluate(u, 0.0, True)
        assert e.value.element == first and e.value.code == ref["code"]
        with pytest.raises(pkg.SbkError):
            s.commit()
        graph.u.copy_(u)
        summary = graph.replay().cpu().numpy()
        assert summary[3] == first and summary[4] == ref["code"]
        with pytest.raises(pkg.SbkError):
            s.vjp_x(u, torch.ones_like(u), frozen=False)


@pytest.mark.parametrize("kin", list(SCALE))
@pytest.mark.parametrize("name", list(LAWS))
def test_nonfinite_points_without_modes(pkg, orc, cuda, name, kin):
    """The standard element and the stress recovery, where a point's return
    is all that can refuse: as the oracle's do (a radial return without
    saturation has nothing to refuse with)."""
    mat = law(pkg, name)
    mesh = pkg.structured_hex_mesh(6, 2, 1, 6.0e-3, 2.0e-3, 1.0e-3)
    u = 1.0e-6 * np.random.default_rng(3).standard_normal(mesh.num_dofs)
    u[40] = np.nan
    with orc.element(True, True):
        ref = orc.system_evaluate(mat.as_dict(), mesh.coords, mesh.connectivity, u, kinematics=kin)
    _, status = orc.element_stress(mat.as_dict(), mesh.element_coordinates(), mesh.gather(u), kinematics=kin)
    t = pkg.NonlinearSystem(mesh, mat, kin, element="standard")
    s = pkg.NonlinearSystem(mesh, mat, kin)
    v = torch.tensor(u, device=cuda)
    if ref["code"]:
        with pytest.raises(pkg.SolverError) as e:
            t.evaluate(v, 0.0, True)
        assert e.value.element == ref["failed_element"] and e.value.code == ref["code"]
    else:
        t.evaluate(v, 0.0, True)
    if status.any():
        with pytest.raises(pkg.SbkError):
            s.stress(v)
    else:
        s.stress(v)


# Reversals that search and that turn K_aa indefinite, a mild step, an element
# inverted at rest, one crushed through itself, one that is no number.
@pytest.mark.parametrize("rule,n", [((2, 0), 148 * 32 + 5), ((2, 5), 148 * 12 + 5)])
@pytest.mark.parametrize("name", ["j2", "hill", "chaboche", "perfect"])
def test_a_tile_of_every_outcome(pkg, orc, cuda, name, rule, n):
    mat, nt = law(pkg, name), law(pkg, name).kinematic_terms
    kw = dict(kinematics="logarithmic", in_plane=rule[0], thickness=rule[1])
    X = np.tile(X_DISTORTED.reshape(1, 24), (7, 1))
    first = orc.elements(mat.as_dict(), X[:1], deformation(X_DISTORTED, 0.02).reshape(1, 24), want_tangent=False, **kw)
    ue = np.stack([deformation(X_DISTORTED, 0.02 * f) for f in (-6.0, -10.0, -15.0, 1.3, 1.0, 1.0, 1.0)])
    X[4] = X_DISTORTED[[4, 5, 6, 7, 0, 1, 2, 3]].reshape(24)
    for k in range(4, 8):
        ue[5, 3 * k + 2] = -2.5 * X_DISTORTED[k, 2]
    ue[6, 10] = np.nan
    m = len(ue)
    states, alpha = np.repeat(first["states"], m, axis=0), np.repeat(first["alpha"].reshape(1, 9), m, axis=0)
    ref = orc.elements(mat.as_dict(), X, ue, states, alpha, **kw)
    assert (ref["status"][[0, 2, 3]] == 0).all() and (ref["status"][4:] != 0).all() and ref["iterations"][:3].max() > 4
    at = np.random.default_rng(n).integers(0, m, n)
    dev = oracle_to_device(states, nt)
    r = run(pkg, mat, X[at], ue[at], dev[:, at], alpha[at], cuda, "logarithmic", rule)
    code = r.code.cpu().numpy()
    np.testing.assert_array_equal(code, ref["status"][at])
    np.testing.assert_array_equal(r.iterations.cpu().numpy()[code == 0], ref["iterations"][at][code == 0])
    one = run(pkg, mat, X, ue, dev, alpha, cuda, "logarithmic", rule)  # an element a tile
    ok = torch.tensor(code == 0, device=cuda)
    same_bits(r, ok, one, torch.tensor(at, device=cuda)[ok])
