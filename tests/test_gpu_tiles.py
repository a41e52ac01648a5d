"""The kernels that take elements in tiles, at the sizes where a tile, a warp
or a block ends: batches of one element up to 148 full tiles and one element
more, rules of 8 to 28 points, every count of backstress terms, against the
oracle within the parity bounds of the element tests (1e-11 relative; the
shape derivative 1e-10 of its largest entry). A batch repeats a few dozen
elements, so that every place in a tile is checked against the oracle's few."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest
import torch

from conftest import X_DISTORTED, deformation, dense_from_blocks, device_to_oracle, oracle_to_device

pytestmark = pytest.mark.gpu
KINDS = 37  # different elements of a batch; prime, so that they meet every place


def law(pkg, name):
    m = pkg.material
    if name in ("j2", "hill"):
        return m.j2_steel() if name == "j2" else m.hill_sheet()
    base = m.chaboche_steel()
    terms = ((40.0e9, 400.0), (5.0e9, 20.0), (2.0e9, 5.0), (1.0e9, 1.0))[:int(name[0])]
    return dataclasses.replace(base, backstresses=terms, criterion="hill48" if "h" in name else "von_mises", r0=1.9,
                               r45=1.5, r90=2.3, kinematic_integration="backward_euler" if "b" in name else
                               "exponential")


# (law, kinematics, rule, elements): full tiles of 32, 12 and 9 elements and
# one element more; less than a tile per SM; a single element.
@pytest.mark.parametrize("name,kin,rule,n", [
    ("j2", "logarithmic", (2, 0), 148 * 32 + 1), ("j2", "small", (2, 5), 148 * 12 + 1), ("j2", "finite", (3, 0), 1),
    ("hill", "logarithmic", (2, 0), 148 * 32), ("hill", "finite", (2, 3), 149), ("1", "logarithmic", (2, 0), 147),
    ("1h", "small", (2, 0), 299), ("2h", "logarithmic", (2, 5), 148 * 12 + 5), ("2b", "logarithmic", (2, 0), 31),
    ("2h", "finite", (2, 7), 148 * 9 + 1), ("3h", "logarithmic", (2, 0), 33), ("4", "logarithmic", (3, 0), 150),
    ("4hb", "finite", (2, 0), 5), ("4h", "logarithmic", (2, 0), 148 * 32 + 31)])
@pytest.mark.parametrize("want_tangent", [True, False])
def test_batches_at_the_edges_of_tiles(pkg, orc, cuda, name, kin, rule, n, want_tangent):
    mat = law(pkg, name)
    rng = np.random.default_rng(n)
    kinds = min(n, KINDS)
    X = np.tile(X_DISTORTED.reshape(1, 24), (kinds, 1)) + 0.03 * rng.uniform(-1, 1, (kinds, 24))
    s = {"small": 4e-3, "finite": 0.02, "logarithmic": 0.05}[kin]
    amount = s * rng.uniform(0.01, 1.0, kinds)  # some elastic, most yielding
    first = np.stack([deformation(x.reshape(8, 3), a) for x, a in zip(X, amount)])
    second = 1.2 * first + 0.02 * s * rng.uniform(-1, 1, (kinds, 24))
    kw = dict(kinematics=kin, in_plane=rule[0], thickness=rule[1])
    one = orc.elements(mat.as_dict(), X, first, want_tangent=False, **kw)
    ref = orc.elements(mat.as_dict(), X, second, one["states"], one["alpha"], **kw)
    assert (one["status"] == 0).all() and (ref["status"] == 0).all()
    assert ref["yield_flags"].any() and (kinds < KINDS or not ref["yield_flags"].all())
    nt = mat.kinematic_terms
    at = np.arange(n) % kinds
    r = pkg.element_batch(mat, torch.tensor(X[at], device=cuda), torch.tensor(second[at], device=cuda),
                          torch.tensor(np.ascontiguousarray(oracle_to_device(one["states"], nt)[:, at]), device=cuda),
                          torch.tensor(one["alpha"][at], device=cuda), kinematics=kin, want_tangent=want_tangent,
                          stiffness_points=rule[0], thickness_points=rule[1])
    assert (r.code == 0).all()
    got = [(r.force.cpu().numpy(), ref["force"]), (r.energy.cpu().numpy()[:, None], ref["energy"][:, None])]
    if want_tangent:
        got.append((dense_from_blocks(r.tangent.cpu().numpy()).reshape(n, -1), ref["tangent"].reshape(kinds, -1)))
    for mine, theirs in got:
        err = np.linalg.norm(mine - theirs[at], axis=1) / np.linalg.norm(theirs[at], axis=1)
        assert err.max() <= 1e-11, err.max()
    np.testing.assert_array_equal(r.yielding.cpu().numpy().astype(bool), ref["yield_flags"][at])
    np.testing.assert_array_equal(r.iterations.cpu().numpy(), ref["iterations"][at])
    st = device_to_oracle(r.states.cpu().numpy(), nt)
    scale = np.abs(ref["states"]).max(axis=(0, 1))
    assert (np.abs(st - ref["states"][at]).max(axis=(0, 1))[:39] <= 1e-10 * scale + 1e-40).all()


def strip(pkg, n):
    """n elements in a row, their nodes moved, and two displacements."""
    mesh = pkg.structured_hex_mesh(n, 1, 1, n * 1.0e-3, 1.0e-3, 1.0e-3)
    rng = np.random.default_rng(n)
    mesh.coords[:] = mesh.coords + 3.0e-5 * rng.uniform(-1, 1, mesh.coords.shape)
    x = mesh.coords / 1.0e-3
    field = np.stack([np.sin(x[:, 0] + x[:, 2]), 0.5 * np.cos(1.3 * x[:, 0]) * x[:, 1], 0.7 * np.sin(x[:, 1] - x[:, 0])], 1)
    return mesh, 1.0e-5 * field.reshape(-1), 2.5e-5 * field.reshape(-1)


# One element, a block of 16 (the shape derivative's and the condensation's
# multiples) and one more; rules of 8, 20 and 27 points.
@pytest.mark.parametrize("n", [1, 16, 17])
@pytest.mark.parametrize("rule", [(2, 0), (2, 5), (3, 0)])
@pytest.mark.parametrize("name", ["j2", "2h", "4hb"])
def test_systems_at_the_edges_of_blocks(pkg, orc, cuda, n, rule, name):
    mat, (mesh, u1, u2) = law(pkg, name), strip(pkg, n)
    kw = dict(kinematics="logarithmic", in_plane=rule[0], thickness=rule[1])
    nt, X = mat.kinematic_terms, mesh.element_coordinates()
    s = pkg.NonlinearSystem(mesh, mat, "logarithmic", rule[0], rule[1], 2)
    s.evaluate(torch.tensor(u1, device=cuda), 0.0, False)
    s.commit()
    st, al = s.committed_views()
    committed, alpha = device_to_oracle(st.cpu().numpy(), nt), al.cpu().numpy()
    # Stress at a displacement where points yield beyond the committed one.
    got = s.stress(torch.tensor(u2, device=cuda))
    ref, status = orc.element_stress(mat.as_dict(), X, mesh.gather(u2), committed, alpha, **kw)
    assert (status == 0).all()
    packed = torch.cat([got.cauchy, got.piola_kirchhoff, got.von_mises[:, None], got.max_plastic_strain[:, None],
                        got.max_strain[:, None], got.min_jacobian[:, None], got.kirchhoff, got.log_strain],
                       dim=1).cpu().numpy()
    for lo, hi in [(0, 6), (6, 12), (12, 13), (13, 14), (14, 15), (15, 16), (16, 22), (22, 28)]:
        assert np.abs(packed[:, lo:hi] - ref[:, lo:hi]).max() <= 1e-11 * np.abs(ref[:, lo:hi]).max() + 1e-40
    # The shape derivative with the returns.
    lam = np.random.default_rng(5).standard_normal(mesh.num_dofs)
    gx = s.vjp_x(torch.tensor(u2, device=cuda), torch.tensor(lam, device=cuda), frozen=False).cpu().numpy()
    per, status = orc.vjp_x(mat.as_dict(), X, mesh.gather(u2), mesh.gather(lam), committed, alpha, **kw)
    assert (status == 0).all()
    want = np.zeros(mesh.num_dofs)
    for e in range(n):
        for a in range(8):
            want[3 * mesh.connectivity[e, a]:3 * mesh.connectivity[e, a] + 3] += per[e, 3 * a:3 * a + 3]
    assert np.abs(gx - want).max() <= 1e-10 * np.abs(want).max()
    # The standard element of the same rule.
    t = pkg.NonlinearSystem(mesh, mat, "logarithmic", rule[0], rule[1], 2, element="standard")
    t.set_committed(s.committed_all())
    ev = t.evaluate(torch.tensor(u2, device=cuda), 0.0, True)
    with orc.element(True, True):
        ref = orc.system_evaluate(mat.as_dict(), mesh.coords, mesh.connectivity, u2, committed, None, **kw)
    assert ref["code"] == 0 and ev.yielding_points == ref["yielding_points"] > 0
    assert np.abs(ev.internal.cpu().numpy() - ref["internal"]).max() <= 1e-11 * ref["gross"]
    assert np.linalg.norm(ev.tangent.cpu().numpy() - ref["values"]) <= 1e-11 * np.linalg.norm(ref["values"])
