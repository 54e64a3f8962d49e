"""Element smoothing cells grouped as split hexes, whose gradients and volumes are read from the
half-patch tables: one patch, a warp of half patches not filled, exactly filled and passed, with
and without warp chunks and modulus fields. FP64 against the oracle at the parity tests' 1e-12,
mixed at their 5e-5 (FP32 element arithmetic)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", ["1", "0"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (15, 1, 1), (4, 4, 1), (17, 1, 1), (5, 4, 7)])  # 2, 30, 32, 34, 280 units
@pytest.mark.parametrize("material", ["linear_elastic", "neo_hookean", "elastic"])
def test_force_matches_oracle(gpu, oracle_lib, monkeypatch, dims, chunks, material):
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import ExplicitDynamics, Material
    from aperi_mech_b200.smoothing import element_smoothing_part

    monkeypatch.setenv("APERI_B200_WARP_CHUNKS", chunks)
    rng = np.random.default_rng(sum(dims))
    coords, hexes = mesh.box_hex(*dims)
    coords = mesh.jitter_interior(coords, 0.1 / max(dims), rng)
    conn = mesh.hex_to_tets(hexes)
    mat = Material.create(material, 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    mu = 3.85e8 * np.exp(0.3 * rng.standard_normal(conn.shape[0])) if dims[0] == 5 else None
    part, mass = element_smoothing_part(coords, conn, mat, mu_field=mu)
    h = 1.0 / max(dims)
    u = 1e-2 * h * rng.standard_normal(coords.shape) + 1e-3 * coords @ rng.standard_normal((3, 3))
    want = oracle_lib.OracleProblem(coords, [part], mass=mass).internal_force(u)
    with ExplicitDynamics(coords, [part], mass=mass) as m:
        assert rel_err(m.internal_force(u, "fp64"), want) < 1e-12
        assert rel_err(m.internal_force(u, "mixed"), want) < 5e-5
