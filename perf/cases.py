"""The calls a forming run makes of this library, at the sizes it makes them.

A sheet of Hex8 cells, formed towards a bump in committed increments, is
evaluated once more with the tool a little further on: part of the sheet
loads, the rest unloads elastically. A pass is one call (or the calls of one
Newton iteration) of the public interface on that state.

`prepare` does what a program has done before: the mesh, the system with its
committed history, the displacement of the iteration on the device. `exact`
restates the element in plain torch: the logarithm by its series, its
derivatives by forward differentiation, the returns by Newton's method on
their equations, everything in 64 bits and dense.
"""
from __future__ import annotations

import ctypes
import importlib
import math
import random

import numpy as np
import torch

pkg = importlib.import_module("springback-precomp_b200")
system_mod = importlib.import_module("springback-precomp_b200.system")
workload = importlib.import_module("springback-precomp_b200.workload")
capi = importlib.import_module("springback-precomp_b200._capi")

F64 = torch.float64
MM = 1.0e-3


def listed():
    return [
        # A Newton iteration of a bending strip, the smallest model that is
        # run in earnest: 80 elements, all latency.
        dict(name="strip", kind="evaluate", law="swift", nx=20, ny=1, nz=4, thick=0, cell=1.0, height=0.25, tangent=True),
        # A line-search trial of the CPU-runnable forming run's sheet: the
        # residual alone.
        dict(name="dome_residual", kind="evaluate", law="swift", nx=40, ny=40, nz=2, thick=0, cell=0.5, height=0.5,
             tangent=False),
        # The first Newton iteration of an increment of the same sheet under
        # a ball: candidates, tangent, contact, node blocks.
        dict(name="dome_newton", kind="newton", law="swift", nx=40, ny=40, nz=2, thick=0, cell=0.5, height=0.5,
             tangent=True),
        # The linear solve of that iteration: factorise, solve, update.
        dict(name="dome_solve", kind="solve", law="swift", nx=40, ny=40, nz=2, thick=0, cell=0.5, height=0.5,
             tangent=True),
        # The kinematic-hardening forming run: one layer, the production
        # rule of five points through the thickness.
        dict(name="kin_sheet", kind="evaluate", law="hill_chaboche", nx=48, ny=48, nz=1, thick=5, cell=1.0, height=1.0,
             tangent=True),
        # The same rule on a part of the design sweep's least size.
        dict(name="thick_part", kind="evaluate", law="hill_chaboche", nx=150, ny=149, nz=1, thick=5, cell=0.25,
             height=1.0, tangent=True),
        # A two-layer part of the design sweep, odd sides.
        dict(name="part", kind="evaluate", law="hill_chaboche", nx=119, ny=97, nz=2, thick=0, cell=0.2, height=0.5,
             tangent=True),
        # The four-layer fine mesh of the cone.
        dict(name="four_layers", kind="evaluate", law="hill_chaboche", nx=224, ny=224, nz=4, thick=0, cell=0.107,
             height=0.25, tangent=True),
        # The element microbenchmark's sheet, a million elements.
        dict(name="sheet_1m", kind="evaluate", law="hill_chaboche", nx=1000, ny=500, nz=2, thick=0, cell=0.04,
             height=0.5, tangent=True),
        # The standard Hex8 with mean dilatation, the default element of the
        # cone quarter.
        dict(name="standard", kind="standard", law="swift", nx=60, ny=60, nz=2, thick=0, cell=0.5, height=0.5,
             tangent=True),
        # Stress recovery at the end of a step.
        dict(name="stress", kind="stress", law="hill_chaboche", nx=100, ny=100, nz=2, thick=0, cell=0.2, height=0.5,
             tangent=True),
        # The shape derivative of the release step's adjoint.
        dict(name="shape_derivative", kind="vjp", law="hill_chaboche", nx=64, ny=64, nz=2, thick=0, cell=0.25,
             height=0.5, tangent=True),
    ]


def draw(rng: random.Random):
    kind = rng.choice(["evaluate"] * 7 + ["newton", "standard", "stress", "vjp", "solve"])
    law = rng.choice(["swift", "hill_chaboche"]) if kind != "vjp" else "hill_chaboche"
    thick = rng.choice([0, 0, 0, 5, 5, 7]) if kind in ("evaluate", "newton") else 0
    most = {"evaluate": 250000, "newton": 60000, "standard": 250000, "stress": 60000, "vjp": 40000, "solve": 2000}[kind]
    if thick:
        most = min(most, 60000)
    nz = rng.choice([1, 2, 3, 4]) if not thick else rng.choice([1, 2])
    ne = math.exp(rng.uniform(math.log(80.0), math.log(float(most))))
    aspect = math.exp(rng.uniform(0.0, math.log(2.5)))
    ny = max(3, int(round(math.sqrt(ne / nz / aspect))))
    nx = max(4, int(round(ne / nz / ny)))
    side = rng.uniform(18.0, 48.0)
    return dict(kind=kind, law=law, nx=nx, ny=ny, nz=nz, thick=thick, cell=side / nx, height=rng.uniform(0.8, 1.2) / nz,
                tangent=True if kind != "evaluate" else rng.random() < 0.75)


def material(case):
    return pkg.material.aluminium_swift() if case["law"] == "swift" else pkg.material.hill_chaboche_sheet()


# ---- the sheet and its displacements ------------------------------------------


def sheet(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    cell, t = case["cell"] * MM, case["height"] * MM
    lx, ly, lz = nx * cell, ny * cell, nz * t
    return pkg.structured_hex_mesh(nx, ny, nz, lx, ly, lz, x0=-0.5 * lx, y0=-0.5 * ly, z0=-lz)


def bump(case, x, y, at):
    """Height and its gradient of a smooth bump over the sheet: `at` its
    centre; along x alone for a strip."""
    cell = case["cell"] * MM
    rx, ry = 0.45 * case["nx"] * cell, 0.45 * case["ny"] * cell
    strip = case["ny"] < 3
    radius = rx if strip else min(rx, ry)
    depth = 0.05 * 2.0 * radius / math.pi
    dx, dy = (x - at[0]) / rx, torch.zeros_like(y) if strip else (y - at[1]) / ry
    r = torch.sqrt(dx * dx + dy * dy)
    inside = r < 1.0
    safe = torch.where(r > 1.0e-12, r, torch.ones_like(r))
    h = torch.where(inside, -0.5 * depth * (1.0 + torch.cos(math.pi * r)), torch.zeros_like(r))
    slope = torch.where(inside & (r > 1.0e-12), 0.5 * depth * math.pi * torch.sin(math.pi * r) / safe,
                        torch.zeros_like(r))
    return h, slope * dx / rx, torch.zeros_like(h) if strip else slope * dy / ry


def laid(case, coords, scale, at):
    """The displacement of the sheet laid on scale x bump, every fibre along
    the surface's normal and thinned by the wall's cosine."""
    x, y, z = coords[:, 0], coords[:, 1], coords[:, 2]
    mid = -0.5 * case["nz"] * case["height"] * MM
    h, hx, hy = bump(case, x, y, at)
    h, hx, hy = scale * h, scale * hx, scale * hy
    n2 = 1.0 + hx * hx + hy * hy
    off = (z - mid) / n2
    return torch.stack([-off * hx, -off * hy, h + off - (z - mid)], dim=1)


def inputs(case, seed):
    """The mesh on the host, its nodes, the displacements of the committed
    increments and of the evaluated state on the device."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    pick = torch.rand(4, generator=gen, device="cuda", dtype=F64).tolist()
    mesh = sheet(case)
    coords = torch.tensor(mesh.coords, device="cuda")
    cell = case["cell"] * MM
    at = ((pick[0] - 0.5) * 2.0 * cell, (pick[1] - 0.5) * 2.0 * cell)
    depth = 0.9 + 0.2 * pick[2]
    if case["kind"] == "solve":
        depth *= 0.1  # early in the forming, where the tangent is safely definite
    small = min(case["cell"], case["height"]) * MM
    noise = 2.0 * torch.rand(coords.shape, generator=gen, device="cuda", dtype=F64) - 1.0
    full = laid(case, coords, depth, at) + 1.0e-3 * small * noise
    steps = [laid(case, coords, depth * k / 4.0, at) + 1.0e-3 * small * (k / 4.0) * noise for k in range(1, 4)] + [full]
    # The tool's neighbourhood goes on (a quarter of the sheet's width around
    # a point of the wall); the rest springs back a little.
    wx = 0.25 * case["nx"] * cell
    wy = 0.25 * case["ny"] * cell if case["ny"] >= 3 else 1.0
    tx, ty = at[0] + 0.2 * case["nx"] * cell * math.cos(6.28 * pick[3]), at[1] + (
        0.2 * case["ny"] * cell * math.sin(6.28 * pick[3]) if case["ny"] >= 3 else 0.0)
    near = torch.exp(-((coords[:, 0] - tx) / wx) ** 2 - ((coords[:, 1] - ty) / wy) ** 2)
    fresh = 2.0 * torch.rand(coords.shape, generator=gen, device="cuda", dtype=F64) - 1.0
    u = full * (1.0 - 0.01 + 0.04 * near[:, None]) + 2.0e-4 * small * fresh
    return mesh, coords, [s.reshape(-1).contiguous() for s in steps], u.reshape(-1).contiguous(), at


def make_system(case, mesh):
    return pkg.NonlinearSystem(mesh, material(case), "logarithmic", 2, case["thick"], 2,
                               element="standard" if case["kind"] == "standard" else "incompatible_modes")


def formed(case, seed):
    """The system with its committed history, and the evaluated displacement."""
    mesh, coords, steps, u, at = inputs(case, seed)
    sysm = make_system(case, mesh)
    for s in steps:
        sysm.evaluate(s, 0.0, False)
        sysm.commit()
    return sysm, mesh, coords, steps[-1], u, at


def held(mesh):
    """The free DOFs of the sheet clamped on its outer edge."""
    x, y = mesh.coords[:, 0], mesh.coords[:, 1]
    edge = np.isclose(x, x.min()) | np.isclose(x, x.max()) | np.isclose(y, y.min()) | np.isclose(y, y.max())
    free = np.repeat(~edge, 3)
    return np.flatnonzero(free).astype(np.int32)


def ball(case, mesh, u0, u1, at):
    """A ball on the bump's floor, pressed a twentieth of a cell deeper in
    the increment."""
    r = 3.0 * MM
    nodes, area, kappa = workload.slave_faces(mesh, True)
    pts = []
    for u, pen in ((u0, 0.05), (u1, 0.1)):
        z = mesh.coords[nodes] + u.reshape(-1, 3).cpu().numpy()[nodes]
        k = int(np.argmin((z[:, 0] - at[0]) ** 2 + (z[:, 1] - at[1]) ** 2))
        pts.append((float(z[k, 0]), float(z[k, 1]), float(z[k, 2]) + r - pen * case["cell"] * MM))
    return pkg.Tool(shape="sphere", times=[0.0, 1.0], points=pts, nodes=nodes, area=area, kappa=kappa, radius=r,
                    friction=0.1, tangential_ratio=1.0, name="ball")


def trial_views(sysm):
    """The trial points and modes of the last evaluate, on the device."""
    p = [ctypes.c_void_p() for _ in range(4)]
    capi.check(capi.lib().sbk_system_buffers(sysm._h, *[ctypes.byref(v) for v in p]))
    ne = sysm.mesh.num_elements
    return (system_mod.device_view(p[2].value, (sysm.nfields, ne, sysm.nq)),
            system_mod.device_view(p[3].value, (ne, 9)))


def prepare(case, seed):
    sysm, mesh, coords, u0, u, at = formed(case, seed)
    state = dict(case=case, system=sysm, u=u)
    if case["kind"] == "newton":
        state["contact"] = pkg.ToolContact(mesh, [ball(case, mesh, u0, u, at)])
        state["u0"], state["margin"] = u0, 2.0 * case["cell"] * MM
    elif case["kind"] == "solve":
        ev = sysm.evaluate(u, 0.0, True)
        part = pkg.PartitionedFactor.for_system(sysm, held(mesh))
        state.update(part=part, values=ev.tangent.clone(), residual=ev.residual.clone(), symmetric=sysm.symmetric())
    elif case["kind"] == "stress":
        sysm.evaluate(u, 0.0, False)
        sysm.commit()
    elif case["kind"] == "vjp":
        sysm.set_frozen(True)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(seed) + 77)
        state["lam"] = torch.randn(sysm.num_dofs, generator=gen, device="cuda", dtype=F64)
    return state


def run(state):
    out = call(state)
    for v in out.values():
        if isinstance(v, torch.Tensor):
            v.owner = state  # views of the system's buffers live as long as they do
    return out


def call(state):
    case, sysm, u = state["case"], state["system"], state["u"]
    kind = case["kind"]
    if kind in ("evaluate", "standard"):
        ev = sysm.evaluate(u, 0.0, case["tangent"])
        points, modes = trial_views(sysm)
        out = dict(internal=ev.internal, energy=ev.energy, gross=ev.gross, yielding=ev.yielding_points, points=points,
                   modes=modes)
        if case["tangent"]:
            out["tangent"] = ev.tangent
        return out
    if kind == "newton":
        contact = state["contact"]
        contact.begin_increment(state["u0"], 0.0, 1.0, [True], state["margin"])
        ev = sysm.evaluate(u, 0.0, True)
        ce = contact.evaluate(u, 1.0, True)
        sysm.add_node_blocks(ce.nodes, ce.blocks)
        points, modes = trial_views(sysm)
        return dict(residual=ev.residual + ce.residual, tangent=ev.tangent, energy=ev.energy, gross=ev.gross,
                    yielding=ev.yielding_points, points=points, modes=modes, contact_gross=ce.gross,
                    force_norm=ce.force_norm, tools=ce.tools)
    if kind == "solve":
        part = state["part"]
        part.factorize(state["values"], state["symmetric"])
        du = part.solve(-part.restrict(state["residual"]))
        return dict(du=du, u=part.add_to(u.clone(), du, 1.0))
    if kind == "stress":
        s = sysm.stress(u)
        return dict(cauchy=s.cauchy, piola=s.piola_kirchhoff, mises=s.von_mises, plastic=s.max_plastic_strain,
                    strain=s.max_strain, jacobian=s.min_jacobian, kirchhoff=s.kirchhoff, log_strain=s.log_strain)
    return dict(gx=sysm.vjp_x(u, state["lam"], frozen=True))


# Operations of one point's kinematics, return and material block, and of the
# tangent and the condensation, per element evaluation at its least: two
# passes of the points (the start and the converged state).
def work(case):
    ne = case["nx"] * case["ny"] * case["nz"]
    nn = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    nq = 4 * case["thick"] if case["thick"] else 8
    fields = 14 + (12 if case["law"] == "hill_chaboche" else 0)
    blocks = (3 * case["nx"] + 1) * (3 * case["ny"] + 1) * (3 * case["nz"] + 1)  # node pairs of the pattern
    mesh = 8.0 * 6 * nn + 32.0 * ne
    if case["kind"] == "solve":
        nf = 3 * (case["nx"] - 1) * (case["ny"] - 1) * (case["nz"] + 1)
        # Nested dissection of a plate: the separators' dense factors.
        top = 3.0 * (case["nz"] + 1) * min(case["nx"], case["ny"])
        return dict(bytes=72.0 * blocks + 16.0 * nf * top / 4 + 16.0 * nf, flops=top ** 3 * 3.0 + 4.0 * nf * top)
    if case["kind"] == "stress":
        return dict(bytes=mesh + ne * (8.0 * nq * fields + 72 + 28 * 8), flops=ne * nq * 1500.0)
    if case["kind"] == "vjp":
        return dict(bytes=mesh + 48.0 * nn + ne * (8.0 * nq * fields + 72), flops=ne * nq * 12000.0)
    per_point = 9000.0 if case["kind"] == "standard" else 20000.0
    per_tangent = 12000.0 * case["tangent"]
    return dict(bytes=mesh + 24.0 * nn + ne * (16.0 * nq * fields + 144) + 72.0 * blocks * case["tangent"],
                flops=ne * nq * (per_point + per_tangent))


# ---- the same in plain torch, 64 bits -------------------------------------------

CORNER = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                       [-1, 1, 1]], dtype=F64)
VOIGT = ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0))


def gauss(case):
    g2, w2 = np.polynomial.legendre.leggauss(2)
    gt, wt = np.polynomial.legendre.leggauss(case["thick"]) if case["thick"] else (g2, w2)
    return torch.tensor([[g2[i], g2[j], gt[k], w2[i] * w2[j] * wt[k]] for k in range(len(gt)) for j in range(2)
                         for i in range(2)], dtype=F64, device="cuda")


def shape_gradients(at):
    c = CORNER.to(at.device)
    f = 1.0 + at[None, :] * c
    return 0.125 * torch.stack([c[:, 0] * f[:, 1] * f[:, 2], c[:, 1] * f[:, 0] * f[:, 2], c[:, 2] * f[:, 0] * f[:, 1]],
                               dim=1)  # (8, 3)


def geometry(case, X):
    """X (n, 8, 3): the gradient operators G (n, q, 3, 11) of the eight nodes
    and three modes, and the weights w (n, q)."""
    pts = gauss(case)
    d0 = shape_gradients(torch.zeros(3, dtype=F64, device=X.device))
    j0 = torch.einsum("nai,ak->nik", X, d0)
    i0, det0 = torch.linalg.inv(j0), torch.linalg.det(j0)
    ops, ws = [], []
    for p in pts:
        dn = shape_gradients(p[:3])
        j = torch.einsum("nai,ak->nik", X, dn)
        ji, det = torch.linalg.inv(j), torch.linalg.det(j)
        g = torch.einsum("ac,nci->nia", dn, ji)
        gm = (det0 / det)[:, None, None] * (-2.0 * p[:3])[None, None, :] * i0.transpose(1, 2)
        ops.append(torch.cat([g, gm], dim=2))
        ws.append(p[3] * det)
    return torch.stack(ops, dim=1), torch.stack(ws, dim=1)


def inverse(A):
    """The inverse of symmetric 3 x 3 matrices by their cofactors."""
    a, b, c = A[..., 0, 0], A[..., 0, 1], A[..., 0, 2]
    d, e, f = A[..., 1, 1], A[..., 1, 2], A[..., 2, 2]
    k0, k1, k2 = d * f - e * e, c * e - b * f, b * e - c * d
    rows = [k0, k1, k2, k1, a * f - c * c, b * c - a * e, k2, b * c - a * e, a * d - b * b]
    return torch.stack(rows, dim=-1).reshape(A.shape) / (a * k0 + b * k1 + c * k2)[..., None, None]


def log_strain(F):
    """E_log (..., 6; engineering shears) of F (..., 3, 3): log C by the
    series of the inverse hyperbolic tangent."""
    eye = torch.eye(3, dtype=F64, device=F.device)
    C = F.transpose(-1, -2) @ F
    Y = (C - eye) @ inverse(C + eye)
    Y2 = Y @ Y
    acc = torch.zeros_like(Y)
    for k in range(16, -1, -1):
        acc = acc @ Y2 + eye / (2 * k + 1)
    E = Y @ acc
    return torch.stack([E[..., i, j] * (1.0 if i == j else 2.0) for i, j in VOIGT], dim=-1)


def log_derivatives(F, T):
    """dE_log / dF (N, 6, 9) and d2 (T . E_log) / dF2 (N, 9, 9)."""
    basis = torch.eye(9, dtype=F64, device=F.device).reshape(9, 1, 3, 3)

    def along(at, v):
        return torch.func.jvp(log_strain, (at,), (v.expand_as(at),))[1]

    def twice(v):
        return torch.func.vmap(lambda d: torch.func.jvp(lambda at: along(at, d), (F,), (v.expand_as(F),)))(basis)

    first, second = torch.func.vmap(lambda v: twice(v))(basis)
    return first[0].permute(1, 2, 0), torch.einsum("nc,ijnc->nij", T, second)


def respond(mat, strain, old, elastic_only=False):
    """The return of N points: stress (N, 6), C (N, 6, 6), energy, the new
    state (N, fields) and whether it yields."""
    dev = strain.device
    G = mat.youngs_modulus / (2 * (1 + mat.poisson_ratio))
    K = mat.youngs_modulus / (3 * (1 - 2 * mat.poisson_ratio))
    m = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=F64, device=dev)
    half = torch.tensor([1.0, 1, 1, 0.5, 0.5, 0.5], dtype=F64, device=dev)
    D = 2 * G * (torch.diag(half) - torch.outer(m, m) / 3.0)  # strain -> deviator
    nt = mat.kinematic_terms
    if mat.criterion == "hill48":  # rolling direction x, sheet normal z
        g, h = 1 / (1 + mat.r0), mat.r0 / (1 + mat.r0)
        f = mat.r0 / (mat.r90 * (1 + mat.r0))
        n = (mat.r0 + mat.r90) * (1 + 2 * mat.r45) / (2 * mat.r90 * (1 + mat.r0))
        P = torch.zeros(6, 6, dtype=F64, device=dev)
        P[:3, :3] = torch.tensor([[g + h, -h, -g], [-h, f + h, -f], [-g, -f, f + g]], dtype=F64, device=dev)
        P[3, 3], P[4, 4], P[5, 5] = 2 * n, 2 * mat.shear_l, 2 * mat.shear_m
    else:
        P = torch.diag(torch.tensor([1.5, 1.5, 1.5, 3.0, 3.0, 3.0], dtype=F64, device=dev))
        P[:3, :3] -= 0.5
    ep, eq_n = old[:, :6], old[:, 12 + 6 * nt]
    terms = [old[:, 12 + 6 * t:18 + 6 * t] for t in range(nt)]
    cg = [tuple(b) for b in mat.backstresses][:nt]

    def sigma_y(a):
        return mat.yield_stress + mat.hardening_modulus * a - mat.saturation_stress * torch.expm1(-mat.saturation_rate * a)

    def residual(y, eps):
        xi, dl = y[:, :6], y[:, 6]
        pxi = xi @ P
        eq = torch.sqrt((xi * pxi).sum(-1))
        flow = half * pxi / eq[:, None]
        r = xi - (eps - ep) @ D + 2 * G * dl[:, None] * flow
        for (c, gam), a in zip(cg, terms):
            th = torch.exp(-gam * dl)
            chi = -torch.expm1(-gam * dl) / gam
            r = r + th[:, None] * a + (2.0 / 3.0 * c * chi)[:, None] * flow
        return torch.cat([r, (eq - sigma_y(eq_n + dl))[:, None]], dim=1)

    eye7 = torch.eye(7, dtype=F64, device=dev)

    def jac(fn, at):
        return torch.stack([torch.func.jvp(fn, (at,), (eye7[k][:at.shape[1]].expand_as(at),))[1]
                            for k in range(at.shape[1])], dim=-1)

    xi0 = (strain - ep) @ D - sum(terms, torch.zeros_like(ep))
    eq0 = torch.sqrt((xi0 * (xi0 @ P)).sum(-1))
    yields = (eq0 - sigma_y(eq_n) > 1e-12 * sigma_y(eq_n)) & (not elastic_only)
    idx = torch.nonzero(yields).reshape(-1)
    stress = (strain - ep) @ D + K * (strain - ep)[:, :3].sum(-1, keepdim=True) * m
    C = (D + K * torch.outer(m, m)).expand(len(strain), 6, 6).clone()
    new = old.clone()
    new[:, -1] = 0.0
    if len(idx):
        full = (ep, eq_n, terms)
        ep, eq_n, terms = ep[idx], eq_n[idx], [a[idx] for a in terms]
        eps = strain[idx]
        y = torch.cat([xi0[idx], torch.zeros(len(idx), 1, dtype=F64, device=dev)], dim=1)
        norm = residual(y, eps).abs().amax(-1)
        for _ in range(40):
            r = residual(y, eps)
            step = -torch.linalg.solve(jac(lambda v: residual(v, eps), y), r)
            t = torch.ones(len(idx), 1, dtype=F64, device=dev)
            for _ in range(12):
                trial = y + t * step
                trial = torch.cat([trial[:, :6], trial[:, 6:].clamp_min(0.0)], dim=1)
                rn = residual(trial, eps).abs().amax(-1)
                worse = ~(rn <= norm * (1 + 1e-9)) & (norm > 1e-9 * mat.yield_stress)
                if not bool(worse.any()):
                    break
                t = torch.where(worse[:, None], 0.5 * t, t)
            y, norm = trial, rn
            if float(step[:, :6].abs().max()) < 1e-11 * mat.yield_stress:
                break
        J = jac(lambda v: residual(v, eps), y)
        dR = jac(lambda e: residual(y, e), eps)
        dy = -torch.linalg.solve(J, dR)  # (n, 7, 6)

        def plastic_strain(v):
            pxi = v[:, :6] @ P
            return v[:, 6:] * pxi / torch.sqrt((v[:, :6] * pxi).sum(-1, keepdim=True))

        dep = plastic_strain(y)
        Jp = jac(plastic_strain, y)
        elastic = D + K * torch.outer(m, m)
        stress[idx] = (eps - ep - dep) @ D + K * (eps - ep)[:, :3].sum(-1, keepdim=True) * m
        C[idx] = elastic - elastic @ (Jp @ dy)
        pxi = y[:, :6] @ P
        flow = half * pxi / torch.sqrt((y[:, :6] * pxi).sum(-1, keepdim=True))
        dl = y[:, 6]
        beta = torch.zeros_like(dep)
        for t, ((c, gam), a) in enumerate(zip(cg, terms)):
            a1 = torch.exp(-gam * dl)[:, None] * a + (2.0 / 3.0 * c * -torch.expm1(-gam * dl) / gam)[:, None] * flow
            new[idx, 12 + 6 * t:18 + 6 * t] = a1
            beta = beta + a1
        new[idx, :6] = ep + dep
        new[idx, 6:12] = beta
        new[idx, 12 + 6 * nt] = eq_n + dl
        new[idx, -1] = 1.0
        ep, eq_n, terms = full
    el = strain - new[:, :6]
    dev_el = el - el[:, :3].sum(-1, keepdim=True) * m / 3.0
    w2 = torch.tensor([1.0, 1, 1, 0.5, 0.5, 0.5], dtype=F64, device=dev)
    a = new[:, 12 + 6 * nt]
    energy = 0.5 * K * el[:, :3].sum(-1) ** 2 + G * (w2 * dev_el ** 2).sum(-1) + 0.5 * mat.hardening_modulus * a * a
    if mat.saturation_stress:
        energy = energy + mat.saturation_stress * (a + torch.expm1(-mat.saturation_rate * a) / mat.saturation_rate)
    for t, (c, _) in enumerate(cg):
        b = new[:, 12 + 6 * t:18 + 6 * t]
        energy = energy + 0.75 / c * (b * b / w2).sum(-1)
    return stress, C, energy, new, yields


def element_pass(case, mat, G, w, U, alpha, old, tangent=True):
    """Residual (n, 33) and its derivative, energy, states of n elements at
    the nodal displacements U (n, 8, 3) and modes alpha (n, 9)."""
    n, nq = w.shape
    D = torch.cat([U, alpha.reshape(n, 3, 3)], dim=1)  # augmented nodes (n, 11, 3)
    F = torch.einsum("nai,nqja->nqij", D, G).reshape(-1, 3, 3) + torch.eye(3, dtype=F64, device=U.device)
    E = log_strain(F)
    wf = w.reshape(-1)
    bbar = case["kind"] == "standard"
    m = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=F64, device=U.device)
    if bbar:
        tr = E[:, :3].sum(-1).reshape(n, nq)
        mean = (w * tr).sum(1, keepdim=True) / w.sum(1, keepdim=True)
        E = E + ((mean - tr) / 3.0).reshape(-1, 1) * m
    T, C, energy, new, yields = respond(mat, E, old, case["kind"] == "vjp")
    Tg = T
    if bbar:
        p = (T[:, :3].sum(-1) / 3.0).reshape(n, nq)
        mean = (w * p).sum(1, keepdim=True) / w.sum(1, keepdim=True)
        Tg = T + (mean - p).reshape(-1, 1) * m
    first, second = log_derivatives(F, Tg)
    # dF_ij / dq_(a i) = G_j a: the chain onto the 33 augmented DOFs.
    B = torch.einsum("ncij,nja->ncai", first.reshape(-1, 6, 3, 3), G.reshape(-1, 3, 11)).reshape(-1, 6, 33)
    if bbar:
        row = B[:, :3].sum(1).reshape(n, nq, 33)
        mean = (w[:, :, None] * row).sum(1, keepdim=True) / w.sum(1)[:, None, None]
        B = B + m[None, :, None] * ((mean - row) / 3.0).reshape(-1, 1, 33)
    r = torch.einsum("n,nc,ncd->nd", wf, T, B).reshape(n, nq, 33).sum(1)
    CB = torch.einsum("ncd,nde->nce", C, B) * wf[:, None, None]
    Kt = torch.bmm(B.transpose(1, 2), CB)
    Gf = G.reshape(-1, 3, 11)
    H = torch.einsum("nijkl,nja->naikl", second.reshape(-1, 3, 3, 3, 3), Gf)
    H = torch.einsum("naikl,nlb->naikb", H, Gf).transpose(-1, -2).reshape(-1, 33, 33)
    Kt = (Kt + wf[:, None, None] * H).reshape(n, nq, 33, 33).sum(1)
    return r, Kt, (wf * energy).reshape(n, nq).sum(1), new, yields


def equilibrate(case, mat, G, w, U, alpha, old):
    if case["kind"] != "standard":
        for _ in range(15):
            r, Kt, _, _, _ = element_pass(case, mat, G, w, U, alpha, old)
            step = torch.linalg.solve(Kt[:, 24:, 24:], r[:, 24:])
            alpha = alpha - step
            if float(step.abs().max()) < 1e-10 * float(alpha.abs().max() + 1e-300):
                break
    return alpha, element_pass(case, mat, G, w, U, alpha, old)


def assemble_csc(conn, Ke, ndof):
    dofs = (3 * conn[:, :, None] + torch.arange(3, device=conn.device)).reshape(len(conn), 24)
    key = (dofs[:, None, :] * ndof + dofs[:, :, None]).reshape(-1)  # column-major: entry (row, col)
    uniq, inv = torch.unique(key, return_inverse=True)
    return torch.zeros(len(uniq), dtype=F64, device=conn.device).index_add_(0, inv, Ke.reshape(-1))


def exact(case, seed):
    ne = case["nx"] * case["ny"] * case["nz"]
    most = dict(evaluate=50000, standard=100000, stress=200000, vjp=70000, solve=200000).get(case["kind"], 0)
    if ne * (4 * case["thick"] or 8) > most:
        return None  # the contact has no restatement here; the large ones take too long
    state = prepare(case, seed)
    sysm, u, mat = state["system"], state["u"], material(case)
    if case["kind"] == "solve":
        part = state["part"]
        free = torch.tensor(part.free, device="cuda").long()
        outer, inner = sysm.outer.long(), sysm.inner.long()
        cols = torch.repeat_interleave(torch.arange(sysm.num_dofs, device="cuda"), outer[1:] - outer[:-1])
        place = torch.full((sysm.num_dofs,), -1, device="cuda").index_put_((free,), torch.arange(len(free), device="cuda"))
        keep = (place[cols] >= 0) & (place[inner] >= 0)
        A = torch.zeros(len(free), len(free), dtype=F64, device="cuda")
        A[place[inner[keep]], place[cols[keep]]] = state["values"][keep]
        b = -state["residual"][free]
        lu = torch.linalg.lu_factor(A)
        x = torch.linalg.lu_solve(*lu, b[:, None])[:, 0]
        x = x + torch.linalg.lu_solve(*lu, (b - A @ x)[:, None])[:, 0]
        return dict(du=x, u=u.index_add(0, free, x))
    conn = torch.tensor(sysm.mesh.connectivity, device="cuda").long()
    X = torch.tensor(sysm.mesh.coords, device="cuda")[conn]
    U = u.reshape(-1, 3)[conn]
    points, modes = (v.clone() for v in sysm.committed_views())
    old = points.permute(1, 2, 0).reshape(-1, sysm.nfields)
    nq = sysm.nq
    parts = []
    chunk = max(1, 20000 // nq)
    for lo in range(0, ne, chunk):
        hi = min(ne, lo + chunk)
        parts.append(exact_chunk(case, mat, X[lo:hi], U[lo:hi], modes[lo:hi], old[lo * nq:hi * nq], sysm.nfields,
                                 state["lam"].reshape(-1, 3)[conn[lo:hi]] if case["kind"] == "vjp" else None))
    cat = {k: torch.cat([p[k] for p in parts], dim=1 if k == "points" else 0) for k in parts[0]}
    if case["kind"] == "stress":
        return cat
    dofs = (3 * conn[:, :, None] + torch.arange(3, device="cuda")).reshape(-1)
    if case["kind"] == "vjp":
        return dict(gx=torch.zeros_like(u).index_add_(0, dofs, cat["gx"].reshape(-1)))
    fe = cat["force"].reshape(-1)
    out = dict(internal=torch.zeros_like(u).index_add_(0, dofs, fe), energy=float(cat["energy"].sum()),
               gross=float(torch.linalg.norm(torch.zeros_like(u).index_add_(0, dofs, fe.abs()))),
               yielding=int(cat["yields"].sum()), points=cat["points"], modes=cat["modes"])
    if case["tangent"]:
        out["tangent"] = assemble_csc(conn, cat["tangent"], sysm.num_dofs)
    return out


def exact_chunk(case, mat, X, U, alpha, old, fields, lam):
    n = len(X)
    G, w = geometry(case, X)
    nq = w.shape[1]
    if case["kind"] == "stress":
        D = torch.cat([U, alpha.reshape(n, 3, 3)], dim=1)
        F = torch.einsum("nai,nqja->nqij", D, G) + torch.eye(3, dtype=F64, device=U.device)
        E = log_strain(F)
        T = respond(mat, E.reshape(-1, 6), old)[0]
        first, _ = log_derivatives(F.reshape(-1, 3, 3), T)
        # T . dE = (F S) . dF, tau = F S F^T.
        FS = torch.einsum("nc,ncf->nf", T, first).reshape(n, nq, 3, 3)
        S, tau = torch.linalg.solve(F, FS), FS @ F.transpose(-1, -2)
        el = torch.stack([E[..., k] * (1.0 if k < 3 else 0.5) for k in range(6)], dim=-1)

        def mean6(A):
            return torch.stack([A[..., i, j] for i, j in VOIGT], dim=-1).mean(1)

        cauchy = mean6(tau / torch.exp(el[..., :3].sum(-1))[..., None, None])
        d = cauchy[:, :3] - cauchy[:, [1, 2, 0]]
        return dict(cauchy=cauchy, piola=mean6(S),
                    mises=torch.sqrt(0.5 * (d * d).sum(-1) + 3.0 * (cauchy[:, 3:] ** 2).sum(-1)),
                    plastic=old.reshape(n, nq, fields)[..., -2].amax(1), strain=el.abs().amax((1, 2)),
                    jacobian=torch.linalg.det(F).amin(1), kirchhoff=mean6(tau), log_strain=el.mean(1))
    alpha, (r, Kt, energy, new, yields) = equilibrate(case, mat, G, w, U, alpha, old)
    if case["kind"] == "vjp":
        mu = -torch.linalg.solve(Kt[:, 24:, 24:].transpose(1, 2),
                                 torch.einsum("nij,ni->nj", Kt[:, :24, 24:], lam.reshape(n, 24)))
        v = torch.cat([lam, mu.reshape(n, 3, 3)], dim=1)
        D = torch.cat([U, alpha.reshape(n, 3, 3)], dim=1)

        def work_of(Xv):  # the virtual work of (lam, mu) in the frozen elements
            Gv, wv = geometry(case, Xv)
            F = torch.einsum("nai,nqja->nqij", D, Gv) + torch.eye(3, dtype=F64, device=U.device)
            dF = torch.einsum("nai,nqja->nqij", v, Gv)
            E, dE = torch.func.jvp(log_strain, (F,), (dF,))
            T = respond(mat, E.reshape(-1, 6), old, True)[0].reshape(E.shape)
            return (wv * (T * dE).sum(-1)).sum()

        return dict(gx=torch.func.grad(work_of)(X).reshape(n, 24))
    out = dict(force=r[:, :24], energy=energy, yields=yields.reshape(n, nq), modes=alpha if case["kind"] != "standard"
               else torch.zeros_like(alpha), points=new.reshape(n, nq, fields).permute(2, 0, 1))
    if case["kind"] != "standard":
        A = torch.linalg.solve(Kt[:, 24:, 24:], torch.cat([Kt[:, 24:, :24], r[:, 24:, None]], dim=2))
        out["force"] = r[:, :24] - torch.einsum("nij,nj->ni", Kt[:, :24, 24:], A[:, :, 24])
        Kt = Kt[:, :24, :24] - Kt[:, :24, 24:] @ A[:, :, :24]
    else:
        Kt = Kt[:, :24, :24]
    if case["tangent"]:
        out["tangent"] = Kt
    return out
