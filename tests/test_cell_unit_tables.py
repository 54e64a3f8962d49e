"""Element smoothing cells grouped as split hexes keep their gradients and volumes in the
half-patch tables alone: a mesh of more patches than one staging slice (65,536) at set-up, force
and VJP against the oracle, and the device memory the model takes."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


def _problem(dims):
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import Material
    from aperi_mech_b200.smoothing import element_smoothing_part

    rng = np.random.default_rng(sum(dims))
    coords, hexes = mesh.box_hex(*dims)
    coords = mesh.jitter_interior(coords, 0.1 / max(dims), rng)
    conn = mesh.hex_to_tets(hexes)
    mat = Material.create("neo_hookean", 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    part, mass = element_smoothing_part(coords, conn, mat)
    u = 1e-2 / max(dims) * rng.standard_normal(coords.shape) + 1e-3 * coords @ rng.standard_normal((3, 3))
    return coords, part, mass, u, rng.standard_normal(coords.shape)


@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 4, 7), (60, 60, 60)])  # 1, 140, 216,000 patches
def test_force_vjp_and_memory(gpu, oracle_lib, dims):
    """FP64 at the parity tests' 1e-12 (force) and 1e-11 (VJP), mixed at their 5e-5. Memory, in
    bytes: 172 a cell (what the CSR arrays of both precisions take: the tables' 160 and some), 24
    for the plan and the patch nodes, 300 a node, 32 a slot, and up to one 2 MB page of each of
    the context's arrays. Tables beside CSR gradients would take 264 a cell."""
    import torch

    from aperi_mech_b200.model import ExplicitDynamics

    coords, part, mass, u, lam = _problem(dims)
    op = oracle_lib.OracleProblem(coords, [part], mass=mass)
    with ExplicitDynamics(*_problem((2, 2, 2))[0:1], [_problem((2, 2, 2))[1]], mass=_problem((2, 2, 2))[2]):
        pass  # the kernels of the set-up are loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with ExplicitDynamics(coords, [part], mass=mass) as m:
        torch.cuda.synchronize()
        used = free - torch.cuda.mem_get_info()[0]
        assert used < (172 + 24) * part.num_elems + 300 * coords.shape[0] + 32 * m.layout()["used_slots"] + 22 * 2**21
        assert rel_err(m.internal_force(u, "fp64"), op.internal_force(u)) < 1e-12
        assert rel_err(m.internal_force(u, "mixed"), op.internal_force(u)) < 5e-5
        for g, w in zip(m.vjp_force(u, lam), op.vjp_force(u, lam)):
            assert rel_err(g, w) < 1e-11
