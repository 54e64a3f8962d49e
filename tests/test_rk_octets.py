"""The two-pass coupling's octet rows (weights apart from indices) where they can go wrong:
octets aligned by offset and not, in one field and across it, rows of length zero, one and
many, zero weights, a node count that leaves the last octet partly empty. The force against
the oracle's, at the parity tests' 1e-12 (sums of a few dozen FP64 terms in another order)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


def _functions(n, kind, rng):
    rows = []
    for i in range(n):
        if kind == "banded" or (kind == "mixed" and (i // 8) % 2 == 0):
            near = np.array([j for j in (i - 9, i - 1, i, i + 1, i + 9) if 0 <= j < n])
        else:
            near = rng.choice(n, size=rng.integers(0, min(n, 23)), replace=False)
        if i % 11 == 10:
            near = near[:0]
        elif i % 13 == 12:
            near = near[:1]
        rows.append(rng.permutation(near))
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    nbr = np.concatenate(rows).astype(np.int32)
    val = rng.uniform(-0.2, 1.0, nbr.size)
    val[::17] = 0.0
    return ptr, nbr, val


@pytest.mark.parametrize("dims", [(2, 2, 1), (4, 3, 3), (6, 5, 4)])  # 18, 80, 210 nodes
@pytest.mark.parametrize("kind", ["banded", "random", "mixed"])
def test_coupled_force_matches_oracle(gpu, oracle_lib, dims, kind):
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import ExplicitDynamics, Material
    from aperi_mech_b200.smoothing import element_smoothing_part

    rng = np.random.default_rng(sum(dims) + len(kind))
    coords, hexes = mesh.box_hex(*dims)
    conn = mesh.hex_to_tets(hexes)
    mat = Material.create("neo_hookean", 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    part, mass = element_smoothing_part(coords, conn, mat)
    rk = _functions(coords.shape[0], kind, rng)
    d = 1e-3 * rng.standard_normal(coords.shape)
    want = oracle_lib.OracleProblem(coords, [part], mass=mass, rk=rk)
    with ExplicitDynamics(coords, [part], mass=mass, rk=rk) as m:
        assert rel_err(m.internal_force(d, "fp64"), want.internal_force(d)) < 1e-12


@pytest.mark.parametrize("octets", ["1", "0"])
@pytest.mark.parametrize("dims", [(2, 2, 1), (6, 5, 4)])
def test_coupled_steps_match_oracle(gpu, oracle_lib, monkeypatch, dims, octets):
    """Steps whose nodes the columns' kernel advances (and, with the octets off, the node
    kernel), one at a time and 40 in a run (past the first graph replay), with a held face and
    gravity, against the oracle's steps: u and v at the parity tests' 1e-12, the acceleration, a
    residual of larger stresses, at 1e-11 as in the full-size tests."""
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import BoundaryCondition, ExplicitDynamics, Material
    from aperi_mech_b200.smoothing import element_smoothing_part

    monkeypatch.setenv("APERI_B200_RK_OCTETS", octets)
    rng = np.random.default_rng(sum(dims))
    coords, hexes = mesh.box_hex(*dims)
    conn = mesh.hex_to_tets(hexes)
    mat = Material.create("neo_hookean", 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    part, mass = element_smoothing_part(coords, conn, mat)
    ptr, nbr, val = _functions(coords.shape[0], "mixed", rng)
    val = np.where(val == 0.0, 0.0, 0.05 * val)  # weak coupling: the step stays stable
    bcs = [BoundaryCondition.fixed(mesh.side_sets(coords)["surface_5"])]
    v0 = rng.uniform(-0.1, 0.1, coords.shape)
    v0[bcs[0].nodes] = 0.0
    dt = 0.2 * float(mesh.tet_char_length(coords, conn).min()) / np.sqrt((mat.lam + 2 * mat.mu) / 1000.0)
    g = (0.0, 0.3, -9.81)
    z = np.zeros_like(coords)
    op = oracle_lib.OracleProblem(coords, [part], bcs, mass=mass, body_accel=g, rk=(ptr, nbr, val))
    a0 = op.init_acceleration(z)
    with ExplicitDynamics(coords, [part], bcs, body_accel=g, mass=mass, rk=(ptr, nbr, val)) as m:
        for runs in ([3], [1, 1, 1], [40], [40]):
            want = op.steps(z, v0, a0, np.full(sum(runs), dt))
            m.set_state(z, v0)
            m.init_acceleration()
            for k, r in enumerate(runs):
                m.run(r, dt, t0=sum(runs[:k]) * dt)
            for got, ref, tol in zip(m.get_state(), want, (1e-12, 1e-12, 1e-11)):
                assert rel_err(got, ref) < tol
