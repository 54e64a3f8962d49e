"""The four-lanes-per-element Hex8 force kernel (FP64) where its grouping can go wrong: element
counts around the eight elements of a warp and the 32 of a block, and blocks of several
rounds (two from 2 x 3 x 148 x 16 x 8 elements on), with a last round that is not full.

FP64 is held to the 1e-12 of the parity tests. In the mixed path each element force carries
FP32 rounding (6e-8) through about a hundred operations on values up to 8 times the nodal
sum: 5e-5, the bar of the parity tests."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu


def _problem(dims, material, fields):
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import Material, Part

    rng = np.random.default_rng(dims[0] + 7 * dims[1] + 49 * dims[2])
    coords, conn = mesh.box_hex(*dims)
    coords = mesh.jitter_interior(coords, 0.1 / max(dims), rng)
    mat = (Material.create(material, 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8) if material == "neo_hookean"
           else Material.create(material, 1000.0, youngs_modulus=1e9, poissons_ratio=0.3))
    mu = 3.85e8 * np.exp(0.3 * rng.standard_normal(conn.shape[0])) if fields else None
    u = 2e-3 / max(dims) * rng.standard_normal(coords.shape) + 1e-3 * coords @ rng.standard_normal((3, 3))
    return coords, [Part("hex8", mat, conn=conn, mu_field=mu)], u


@pytest.mark.parametrize("material", ["linear_elastic", "neo_hookean", "elastic"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (7, 1, 1), (2, 2, 2), (3, 3, 1), (31, 1, 1), (4, 4, 2), (11, 3, 1)])
def test_group_edges(gpu, oracle_lib, dims, material):
    from aperi_mech_b200.model import ExplicitDynamics

    coords, parts, u = _problem(dims, material, fields=dims[0] == 11)
    want = oracle_lib.OracleProblem(coords, parts).internal_force(u)
    with ExplicitDynamics(coords, parts) as m:
        assert rel_err(m.internal_force(u, "fp64"), want) < 1e-12
        assert rel_err(m.internal_force(u, "mixed"), want) < 5e-5


@pytest.mark.parametrize("dims", [(49, 48, 49), (57, 55, 55)])  # two and three rounds, partly filled
def test_several_rounds(gpu, oracle_lib, dims):
    from aperi_mech_b200.model import ExplicitDynamics

    coords, parts, u = _problem(dims, "neo_hookean", fields=True)
    want = oracle_lib.OracleProblem(coords, parts).internal_force(u)
    with ExplicitDynamics(coords, parts) as m:
        assert rel_err(m.internal_force(u, "fp64"), want) < 1e-12
        assert rel_err(m.internal_force(u, "mixed"), want) < 5e-5


def test_inverted_element_is_named(gpu):
    """The element reported is the inverted one, whichever of a quad's lanes sees it."""
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.capi import AmError
    from aperi_mech_b200.model import ExplicitDynamics, Material, Part

    coords, conn = mesh.box_hex(5, 3, 2)
    mat = Material.create("neo_hookean", 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    far = int(np.argmax(coords.sum(axis=1)))  # a corner node: one element holds it
    u = np.zeros_like(coords)
    u[far] = -0.9
    for precision in ("fp64", "mixed"):
        with ExplicitDynamics(coords, [Part("hex8", mat, conn=conn)]) as m:
            with pytest.raises(AmError, match=f"element/cell {int(np.nonzero((conn == far).any(axis=1))[0][0])}$"):
                m.internal_force(u, precision)


@pytest.mark.parametrize("dims, material", [(d, m) for d in [(1, 1, 1), (7, 1, 1), (3, 3, 1), (11, 3, 1)]
                                            for m in ("linear_elastic", "neo_hookean", "elastic")]
                         + [((49, 48, 49), "neo_hookean")])
def test_vjp_group_edges(gpu, oracle_lib, dims, material):
    """The VJP runs in the same quads and rounds: against the oracle at the parity tests' 1e-11
    (nodal) and, for the modulus gradients, contractions of eight points whose terms cancel to
    the strain's order (1e-3 here, so 1e-16 / 1e-3 a term and a few terms), 1e-11 of the largest."""
    from aperi_mech_b200.model import ExplicitDynamics

    coords, parts, u = _problem(dims, material, fields=dims[0] >= 11)
    lam = np.random.default_rng(5).standard_normal(coords.shape)
    want = oracle_lib.OracleProblem(coords, parts).vjp_force(u, lam)
    with ExplicitDynamics(coords, parts) as m:
        for g, w in zip(m.vjp_force(u, lam), want):
            assert rel_err(g, w) < 1e-11
