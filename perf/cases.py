"""Workloads whose speed matters to a user of this library, with the inputs, the calls and
an independent 64-bit evaluation of each.

A case is one of:

  force    one internal-force evaluation on device arrays: what a host code that keeps its
           own time integration calls once per step
  run      a stretch of a simulation between two output frames: set the state, form the
           initial acceleration, advance `steps` central-difference steps, read the state back
  adjoint  loss at sensor nodes after `steps` steps and its gradient with respect to every
           element's shear and bulk modulus

on one of these discretizations of a box of nx x ny x nz lattice cells:

  tet4         six tets per cell on jittered nodes (1-point Gauss)
  scattered    the same tets with some left out and nodes and elements numbered at random:
               a mesh as an unstructured mesher numbers it
  hex8         2x2x2 Gauss hexes on jittered nodes
  smoothed     strain-smoothed tets (element smoothing cells)
  rkpm         reproducing-kernel nodal cells, one pass
  fbar         reproducing-kernel nodal subcells with F-bar over each node
  two_pass     reproducing-kernel element cells, two-pass coupling

A mixed-precision run carries its forces in 32 bits; its frames are kept as 32-bit fields.
"""
from __future__ import annotations

import functools
import math
from types import SimpleNamespace

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from aperi_mech_b200 import capi, mesh
from aperi_mech_b200.model import BoundaryCondition, ExplicitDynamics, Material, Part

JITTER = 0.15  # of the lattice spacing, interior nodes


def _case(name, call, mesh_kind, nx, ny, nz, precision, material="neo_hookean", steps=100, fields=False, semi=0, ckpt=0):
    case = {"call": call, "mesh": mesh_kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "material": material, "steps": steps, "fields": fields, "semi": semi, "ckpt": ckpt}
    return case if name is None else {"name": name, **case}


def listed():
    return [
        # a host solver's call on a small part: the latency of one evaluation
        _case("force_tet4_12_fp64", "force", "tet4", 12, 12, 12, "fp64", steps=1),
        # a small component model, 8,000 hexes: the launches of each step
        _case("run_hex8_le_20_fp64", "run", "hex8", 20, 20, 20, "fp64", material="linear_elastic"),
        # two million tets, the usual production size, mixed precision
        _case("run_tet4_70_mixed", "run", "tet4", 70, 70, 70, "mixed"),
        # the same path in FP64 (the precision users come from) on a ragged box
        _case("run_tet4_57x41x83_fp64", "run", "tet4", 57, 41, 83, "fp64"),
        # an unstructured tet mesh
        _case("run_scattered_61x47x53_fp64", "run", "scattered", 61, 47, 53, "fp64"),
        # impact-style runs: semi-Lagrangian, reference update every 10 steps
        _case("run_semi_tet4_45x45x61_fp64", "run", "tet4", 45, 45, 61, "fp64", semi=10),
        # the largest hex model, with a modulus field per element
        _case("run_hex8_nh_128_mixed", "run", "hex8", 128, 128, 128, "mixed", fields=True),
        # gradients for material identification
        _case("adjoint_hex8_64_fp64", "adjoint", "hex8", 64, 64, 64, "fp64", steps=50, fields=True, ckpt=10),
        # strain-smoothed tets, the default treatment of tet meshes near incompressibility
        _case("run_smoothed_46_mixed", "run", "smoothed", 46, 46, 92, "mixed"),
        # meshfree nodal integration
        _case("run_rkpm_32_mixed", "run", "rkpm", 32, 32, 64, "mixed"),
        # meshfree with F-bar over nodal subcells
        _case("run_fbar_20_fp64", "run", "fbar", 20, 20, 40, "fp64", steps=60),
        # meshfree element cells with the two-pass coupling
        _case("run_two_pass_32_fp64", "run", "two_pass", 32, 32, 64, "fp64"),
    ]


# largest lattice cell count drawn per discretization (the listed sizes' neighbourhood)
_MOST = {"tet4": 343000, "scattered": 160000, "hex8": 900000, "smoothed": 194000, "rkpm": 65000, "fbar": 16000,
         "two_pass": 65000}
_LEAST = {"tet4": 60, "scattered": 400, "hex8": 100, "smoothed": 400, "rkpm": 400, "fbar": 250, "two_pass": 400}


def draw(rng):
    kind = rng.choice(["force", "run", "run", "run", "run", "adjoint"])
    lattice = "hex8" if kind == "adjoint" else rng.choice(list(_MOST))
    most = 130000 if kind == "adjoint" else _MOST[lattice]
    cells = math.exp(rng.uniform(math.log(_LEAST[lattice]), math.log(most)))
    a, b = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
    nx = max(3, round(cells ** (1 / 3) * a))
    ny = max(3, round(cells ** (1 / 3) * b))
    nz = max(3, round(cells / (nx * ny)))
    gauss = lattice in ("tet4", "scattered", "hex8")
    material = rng.choice(["neo_hookean", "neo_hookean", "linear_elastic", "elastic"]) if gauss else "neo_hookean"
    semi = rng.choice([0, 0, 1, 10]) if kind == "run" and lattice in ("tet4", "scattered") else 0
    precision = "fp64" if semi or kind == "adjoint" else rng.choice(["fp64", "mixed"])
    steps = 1 if kind == "force" else rng.randint(10, 50) if kind == "adjoint" else rng.randint(20, 120)
    return _case(None, kind, lattice, nx, ny, nz, precision, material, steps,
                 fields=kind == "adjoint" or (gauss and rng.random() < 0.3), semi=semi,
                 ckpt=rng.randint(4, 15) if kind == "adjoint" else 0)


# ---- the model: mesh, cells, material (from the case alone) -----------------------------

def _thin_out(coords, conn, rng):
    """Leaves out 3% of the tets whose nodes all lie inside, and numbers nodes and tets at random."""
    inside = ~mesh.boundary_mask(coords)
    gone = inside[conn].all(axis=1) & (rng.random(conn.shape[0]) < 0.03)
    conn = conn[~gone]
    pn = rng.permutation(coords.shape[0])
    new = np.empty_like(pn)
    new[pn] = np.arange(pn.size)
    return coords[pn].copy(), new[conn[rng.permutation(conn.shape[0])]].astype(np.int32)


@functools.lru_cache(maxsize=2)
def _model(mesh_kind, nx, ny, nz, material):
    rng = np.random.default_rng(7)
    h = 1.0 / max(nx, ny, nz)
    coords, hexes = mesh.box_hex(nx, ny, nz, nx * h, ny * h, nz * h)
    coords = mesh.jitter_interior(coords, JITTER * h, rng)
    mat = Material.create(material, 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    M = SimpleNamespace(h=h, mat=mat, mass=None, rk=None, conn=None, part=None, length=0.6 * h)
    if mesh_kind == "hex8":
        M.conn = hexes
    else:
        conn = mesh.hex_to_tets(hexes)
        if mesh_kind == "scattered":
            coords, conn = _thin_out(coords, conn, rng)
        M.length = float(mesh.tet_char_length(coords, conn).min())
        M.conn = conn
        if mesh_kind == "smoothed":
            from aperi_mech_b200.smoothing import element_smoothing_part
            M.part, M.mass = element_smoothing_part(coords, conn, mat)
        elif mesh_kind in ("rkpm", "fbar", "two_pass"):
            from aperi_mech_b200 import rkpm
            build = {"rkpm": rkpm.nodal_cells, "fbar": rkpm.nodal_subcells, "two_pass": rkpm.two_pass_element_cells}
            radius = (1.1 * rkpm.tet_max_edge_length(coords, conn) if mesh_kind == "two_pass"
                      else np.full(coords.shape[0], 1.8 * h))
            cells = build[mesh_kind](coords, conn, mat, radius)
            M.part, M.mass = cells.part, cells.mass
            M.rk = cells.functions() if mesh_kind == "two_pass" else None
    M.coords = coords
    M.fixed = mesh.side_sets(coords)["surface_5"]
    return M


def _model_of(case):
    return _model(case["mesh"], case["nx"], case["ny"], case["nz"], case["material"])


def _inputs(case, seed):
    """The initial state, modulus fields, time increment and sensors a simulation starts from:
    a smooth displacement of up to a percent that respects the support, a shear velocity with
    noise, lognormal moduli."""
    M = _model_of(case)
    rng = np.random.default_rng(seed)
    X = M.coords
    n = X.shape[0]
    z = X[:, 2] / X[:, 2].max()
    u = np.zeros((n, 3))
    if not case["semi"]:  # semi-Lagrangian runs start from the undeformed body
        for i in range(3):
            for _ in range(2):
                k = rng.uniform(-1.0, 1.0, 3)
                u[:, i] += 0.004 * z * np.cos(math.pi * (X @ k) + rng.uniform(0, math.pi))
    v = rng.uniform(-0.01, 0.01, (n, 3))
    v[:, 0] += X[:, 2]
    u[M.fixed] = 0.0
    v[M.fixed] = 0.0
    I = SimpleNamespace(u=u, v=v, mu=None, kappa=None, sensors=None)
    lam, mu = M.mat.lam, M.mat.mu
    speed2 = lam + 2 * mu
    if case["fields"]:
        ne = M.conn.shape[0]
        I.mu = 3.85e8 * np.exp(0.3 * rng.standard_normal(ne))
        I.kappa = 8.33e8 * np.exp(0.3 * rng.standard_normal(ne))
        speed2 = float((I.kappa + 4.0 / 3.0 * I.mu).max())
    I.dt = 0.5 * M.length / math.sqrt(speed2 / M.mat.density)
    if case["call"] == "adjoint":
        free = np.setdiff1d(np.arange(n), M.fixed)
        I.sensors = np.sort(rng.choice(free, min(512, free.size), replace=False)).astype(np.int32)
    return M, I


# ---- the library's calls ----------------------------------------------------------------

def prepare(case, seed):
    M, I = _inputs(case, seed)
    part = M.part or Part("hex8" if case["mesh"] == "hex8" else "tet4", M.mat, conn=M.conn, mu_field=I.mu,
                          kappa_field=I.kappa)
    S = SimpleNamespace(call=case["call"], precision=case["precision"], steps=case["steps"], ckpt=case["ckpt"], dt=I.dt,
                        sensors=I.sensors, stream=torch.cuda.Stream())
    S.model = ExplicitDynamics(M.coords, [part], [BoundaryCondition.fixed(M.fixed)], mass=M.mass, rk=M.rk,
                               stream=S.stream.cuda_stream, formulation=("semi", case["semi"]) if case["semi"] else None)
    S.u0 = None if case["semi"] else torch.from_numpy(I.u).cuda()
    S.v0 = torch.from_numpy(I.v).cuda()
    names = {"force": ("f",), "run": ("u", "v", "a"), "adjoint": ()}[case["call"]]
    S.out = {k: torch.empty(M.coords.shape, dtype=torch.float64, device="cuda") for k in names}
    S.frame = None
    if case["precision"] == "mixed":
        S.frame = {k: torch.empty(M.coords.shape, dtype=torch.float32, device="cuda") for k in names}
    torch.cuda.synchronize()
    return S


def run(S):
    m = S.model
    if S.call == "adjoint":
        m.set_state(S.u0, S.v0, None, where=capi.AM_DEVICE)
        loss, gmu, gkappa = m.adjoint(S.steps, S.dt, S.ckpt, S.sensors)
        return {"loss": loss, "gmu": gmu, "gkappa": gkappa}
    if S.call == "force":
        m.internal_force(S.u0, S.precision, out=S.out["f"])
    else:
        m.set_state(S.u0, S.v0, None, where=capi.AM_DEVICE)
        m.init_acceleration(S.precision)
        m.run(S.steps, S.dt, S.precision)
        m.get_state_into(S.out["u"], S.out["v"], S.out["a"])
    if S.frame is None:
        return S.out
    with torch.cuda.stream(S.stream):
        for k, x in S.out.items():
            S.frame[k].copy_(x)
    return S.frame


# ---- what a pass cannot do without ------------------------------------------------------

def work(case):
    """Per force evaluation: connectivity (or cell entries: an index and a gradient of three
    reals), moduli, volumes and function values once, X and u read and f written per node; per
    step also v read and written, u written and the mass; flops of the element formulas in
    their shape-function-free forms."""
    M = _model_of(case)
    n = M.coords.shape[0]
    real = 4 if case["precision"] == "mixed" else 8
    if M.part is None:
        e, nn = M.conn.shape
        nbytes = 4 * nn * e + (16 * e if case["fields"] else 0) + 72 * n
        flops = (450 if nn == 4 else 3900) * e
    else:
        entries, cells = int(M.part.cell_ptr[-1]), M.part.num_elems
        nbytes = entries * (4 + 3 * real) + 8 * cells + 48 * n
        flops = 36 * entries + 150 * cells
        if M.rk is not None:
            nbytes += 12 * M.rk[1].size
            flops += 12 * M.rk[1].size
    if case["semi"]:
        nbytes += 144 * M.conn.shape[0]
        flops += 150 * M.conn.shape[0]
    if case["call"] == "force":
        return {"bytes": nbytes, "flops": flops}
    step = nbytes + 80 * n
    if case["call"] == "run":
        return {"bytes": case["steps"] * step, "flops": case["steps"] * flops}
    # adjoint: the forward steps, their recomputation, and a transposed step of about twice the arithmetic
    return {"bytes": 3 * case["steps"] * step, "flops": 4 * case["steps"] * flops}


# ---- the same in plain torch, 64 bits ---------------------------------------------------

def _stress(kind, lam, mu, H):
    eye = torch.eye(3, dtype=H.dtype, device=H.device)
    Ht = H.transpose(-1, -2)
    if kind == "linear_elastic":
        return lam * torch.einsum("...ii->...", H)[..., None, None] * eye + mu * (H + Ht)
    F = eye + H
    if kind == "elastic":
        E = 0.5 * (H + Ht + Ht @ H)
        return F @ (lam * torch.einsum("...ii->...", E)[..., None, None] * eye + 2 * mu * E)
    Finv_t = _cofactor(F)
    J = (F[..., 0, :] * Finv_t[..., 0, :]).sum(-1)[..., None, None]
    Finv_t = Finv_t / J
    return ((mu * (H @ Ht + H + Ht)) + lam * torch.log(J) * eye) @ Finv_t


def _cofactor(F):
    a, b, c = F.unbind(-2)
    return torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], -2)


def _gauss_geometry(X, conn):
    """Gradients (E, points, nodes, 3) and weights (E, points) of Tet4 or Hex8 elements."""
    if conn.shape[1] == 4:
        dN = X.new_tensor([[[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]])
        w = 1.0 / 6.0
    else:
        s = X.new_tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                          [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])
        g = s / math.sqrt(3.0)
        t = 1 + s[None, :, :] * g[:, None, :]
        dN = torch.stack([s[:, 0] * t[..., 1] * t[..., 2], s[:, 1] * t[..., 0] * t[..., 2],
                          s[:, 2] * t[..., 0] * t[..., 1]], -1) / 8.0
        w = 1.0
    J = torch.einsum("eai,gaj->egij", X[conn], dN)
    cof = _cofactor(J)
    det = (J[..., 0, :] * cof[..., 0, :]).sum(-1)
    return torch.einsum("gaj,egij->egai", dN, cof / det[..., None, None]), w * det


def _physics(case, M, I):
    """The nodal force as a function of (u, mu, kappa), and the lumped mass, on the GPU."""
    def dev(a, dtype=torch.float64):
        return torch.as_tensor(np.ascontiguousarray(a)).to("cuda", dtype)

    kind, n = M.mat.kind, M.coords.shape[0]
    mu0 = dev(I.mu) if I.mu is not None else torch.full((1,), M.mat.mu, dtype=torch.float64, device="cuda")
    ka0 = dev(I.kappa) if I.kappa is not None else torch.full((1,), M.mat.kappa, dtype=torch.float64, device="cuda")
    if M.part is None:
        conn = dev(M.conn, torch.int64)
        B, w = _gauss_geometry(dev(M.coords), conn)
        share = (M.mat.density * w.sum(1) / conn.shape[1])[:, None].expand(conn.shape).reshape(-1)
        mass = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, conn.reshape(-1), share)

        def force(u, mu, kappa):
            mu_, lam_ = mu[:, None, None, None], (kappa - 2 * mu / 3)[:, None, None, None]
            H = torch.einsum("eai,egaj->egij", u[conn], B)
            P = _stress(kind, lam_, mu_, H) * w[..., None, None]
            f = torch.einsum("egij,egaj->eai", P, B)
            return torch.zeros_like(u).index_add(0, conn.reshape(-1), -f.reshape(-1, 3))

        return force, mass, mu0, ka0
    part = M.part
    counts = np.diff(part.cell_ptr)
    cell = dev(np.repeat(np.arange(counts.size), counts), torch.int64)
    node, grad, vol = dev(part.cell_nodes, torch.int64), dev(part.cell_grads), dev(part.cell_volumes)
    mass = dev(M.mass)
    group = None
    if part.cell_groups is not None:
        size = np.diff(part.cell_groups)
        group = dev(np.repeat(np.arange(size.size), size), torch.int64)
    if M.rk is not None:
        reach = np.diff(M.rk[0])
        row, nbr, val = dev(np.repeat(np.arange(reach.size), reach), torch.int64), dev(M.rk[1], torch.int64), dev(M.rk[2])[:, None]

    def force(u, mu, kappa):
        lam_, mu_ = (kappa - 2 * mu / 3)[:, None, None], mu[:, None, None]
        d = torch.zeros_like(u).index_add_(0, row, val * u[nbr]) if M.rk is not None else u
        H = d.new_zeros(counts.size, 3, 3).index_add_(0, cell, d[node][:, :, None] * grad[:, None, :])
        if group is None:
            P = _stress(kind, lam_, mu_, H)
        else:
            eye = torch.eye(3, dtype=u.dtype, device=u.device)
            F = H + eye
            cof = _cofactor(F)
            J = (F[:, 0] * cof[:, 0]).sum(-1)

            def over_cell(x):
                return x.new_zeros(size.size).index_add_(0, group, x)[group]

            total = over_cell(vol)
            Jbar = over_cell(J * vol) / total
            s = (Jbar / J) ** (1.0 / 3.0)
            Pb = _stress(kind, lam_, mu_, s[:, None, None] * F - eye)
            PF = (Pb * F).sum((-1, -2))
            p = over_cell(s / (3 * Jbar) * vol * PF) / total
            P = s[:, None, None] * Pb + (p - s / (3 * J) * PF)[:, None, None] * cof
        f = torch.einsum("eij,ej->ei", (P * -vol[:, None, None])[cell], grad)
        f = torch.zeros_like(u).index_add_(0, node, f)
        return f if M.rk is None else torch.zeros_like(u).index_add_(0, nbr, val * f[row])

    return force, mass, mu0, ka0


def exact(case, seed):
    M, I = _inputs(case, seed)
    force, mass, mu, kappa = _physics(case, M, I)
    u, v = torch.from_numpy(I.u).cuda(), torch.from_numpy(I.v).cuda()
    if case["call"] == "force":
        return {"f": force(u, mu, kappa)}
    grads = case["call"] == "adjoint"
    if grads:
        mu.requires_grad_(True)
        kappa.requires_grad_(True)
    fixed = torch.from_numpy(M.fixed.astype(np.int64)).cuda()
    free = torch.ones_like(mass)
    free[fixed] = 0.0
    free, mass = free[:, None], mass[:, None]

    def accel(u):
        f = checkpoint(force, u, mu, kappa, use_reentrant=False) if grads else force(u, mu, kappa)
        return f / mass

    # semi-Lagrangian Tet4 steps are the total formulation's up to rounding
    a = accel(u)
    for _ in range(case["steps"]):
        v = free * (v + 0.5 * I.dt * a)
        u = u + I.dt * v
        a = free * accel(u)
        v = v + 0.5 * I.dt * a
    if not grads:
        return {"u": u, "v": v, "a": a}
    loss = (u[torch.from_numpy(I.sensors.astype(np.int64)).cuda()] ** 2).sum()
    loss.backward()
    return {"loss": float(loss.detach()), "gmu": mu.grad, "gkappa": kappa.grad}
