"""The Hex8 force and VJP kernels with four and eight rounds a warp (meshes from 4 and 8 x
3 x 148 x 16 x 8 elements on), the last block's rounds and the last element group partly
filled, against the oracle at the parity tests' 1e-12 (force) and 1e-11 (VJP)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(61, 61, 62), (77, 77, 77)])
def test_many_rounds_match_oracle(gpu, oracle_lib, dims):
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import ExplicitDynamics, Material, Part

    rng = np.random.default_rng(dims[0])
    coords, conn = mesh.box_hex(*dims)
    coords = mesh.jitter_interior(coords, 0.1 / max(dims), rng)
    mat = Material.create("neo_hookean", 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    parts = [Part("hex8", mat, conn=conn, mu_field=3.85e8 * np.exp(0.3 * rng.standard_normal(conn.shape[0])))]
    u = 2e-3 / max(dims) * rng.standard_normal(coords.shape) + 1e-3 * coords @ rng.standard_normal((3, 3))
    lam = rng.standard_normal(coords.shape)
    op = oracle_lib.OracleProblem(coords, parts)
    with ExplicitDynamics(coords, parts) as m:
        assert rel_err(m.internal_force(u, "fp64"), op.internal_force(u)) < 1e-12
        for g, w in zip(m.vjp_force(u, lam), op.vjp_force(u, lam)):
            assert rel_err(g, w) < 1e-11
