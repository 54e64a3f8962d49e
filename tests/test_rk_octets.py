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
