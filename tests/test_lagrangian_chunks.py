"""The warp-chunked Tet4 kernel of the updated / semi formulations where it can go wrong: a
last chunk that is not full, and element gradients kept only for the step that reads them,
with runs split at every step. Against the oracle at the 1e-12 of the Lagrangian tests (the
same FP64 operations; sums of up to a few dozen terms in another order)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


def _problem(dims, material="neo_hookean"):
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import BoundaryCondition, Material, Part

    rng = np.random.default_rng(sum(dims))
    coords, hexes = mesh.box_hex(*dims)
    coords = mesh.jitter_interior(coords, 0.1 / max(dims), rng)
    conn = mesh.hex_to_tets(hexes)
    mat = Material.create(material, 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    fixed = mesh.side_sets(coords)["surface_5"]
    v0 = rng.uniform(-1.0, 1.0, coords.shape)
    v0[fixed] = 0.0
    dt = 0.3 * float(mesh.tet_char_length(coords, conn).min()) / np.sqrt((mat.lam + 2 * mat.mu) / 1000.0)
    return coords, [Part("tet4", mat, conn=conn)], [BoundaryCondition.fixed(fixed)], v0, dt


@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 1, 1), (4, 4, 1), (11, 1, 1)])  # 6, 30, 96, 66 tets
@pytest.mark.parametrize("form, k", [("updated", 1), ("semi", 1), ("semi", 2), ("semi", 5)])
def test_steps_match_oracle_however_split(gpu, oracle_lib, dims, form, k):
    from aperi_mech_b200.model import ExplicitDynamics

    coords, parts, bcs, v0, dt = _problem(dims)
    n = 12
    op = oracle_lib.OracleProblem(coords, parts, bcs)
    st = op.lagrangian_state(form, k)
    z = np.zeros_like(coords)
    want = op.lagrangian_steps(st, z, v0, op.lagrangian_init(st), np.full(n, dt))
    with ExplicitDynamics(coords, parts, bcs, formulation=(form, k)) as m:
        for runs in ([n], [1] * n, [3, 4, 5]):
            m.set_state(z, v0)
            m.init_acceleration()
            done = 0
            for r in runs:
                m.run(r, dt, t0=done * dt)
                done += r
            for g, w in zip(m.get_state(), want):
                assert rel_err(g, w) < 1e-12


@pytest.mark.parametrize("material", ["linear_elastic", "neo_hookean", "elastic"])
def test_chunks_agree_with_per_tet_slots(gpu, monkeypatch, material):
    """20 semi steps with and without warp chunks: the same sums in another order (1e-12)."""
    from aperi_mech_b200.model import ExplicitDynamics

    coords, parts, bcs, v0, dt = _problem((7, 3, 5), material)
    got = []
    for chunks in ("1", "0"):
        monkeypatch.setenv("APERI_B200_WARP_CHUNKS", chunks)
        with ExplicitDynamics(coords, parts, bcs, formulation=("semi", 4)) as m:
            slots = m.layout()["used_slots"]
            m.set_state(None, v0)
            m.init_acceleration()
            m.run(20, dt)
            got.append(m.get_state())
        assert (slots == parts[0].conn.size) == (chunks == "0")
    for a, b in zip(*got):
        assert rel_err(a, b) < 1e-12
