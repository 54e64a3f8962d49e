"""VJP of thin, sheared neo-Hookean hexes at small strains, where the shear-modulus sensitivity
L : (F - F^-T) is a small difference of large terms: separate hexes of aspect ratio k, turned
before and after they are flattened, under displacement gradients of the strain's size.

Tolerance, against the oracle and relative to the largest value. An element's gradients of u and
lambda carry the rounding of nodal values over its thickness, a few tens of operations of eps k
each. The oracle forms L : (F - F^-T) entry by entry: F and F^-T round at eps, so its sum of nine
products over the eight Gauss points is off by up to 27 eps against a value of the strain's size.
Together 30 eps (k + 1 / strain)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import rel_err

EPS = 2.0**-52
CASES = [(k, s) for k in (1, 10, 100) for s in (1e-2, 1e-4)]


def _rotation(rng):
    q = np.linalg.qr(rng.standard_normal((3, 3)))[0]
    return q if np.linalg.det(q) > 0 else q[:, ::-1]


def _problem(k, strain):
    from aperi_mech_b200 import mesh

    rng = np.random.default_rng(k)
    cube, conn1 = mesh.box_hex(1, 1, 1)
    X, U, W, conn = [], [], [], []
    for e in range(27):
        x = (cube + 0.1 * rng.uniform(-1.0, 1.0, cube.shape)) @ (_rotation(rng) @ np.diag([1, 1, 1 / k]) @ _rotation(rng)).T
        X.append(x)
        U.append(x @ (strain * rng.uniform(-1.0, 1.0, (3, 3))).T)
        W.append(x @ rng.uniform(-1.0, 1.0, (3, 3)).T)
        conn.append(conn1 + 8 * e)
    return np.concatenate(X), np.concatenate(conn).astype(np.int32), np.concatenate(U), np.concatenate(W)


def _tolerance(k, strain):
    return 30 * EPS * (k + 1 / strain)


@pytest.mark.gpu
@pytest.mark.parametrize("k, strain", CASES)
def test_thin_sheared_hexes_match_oracle(gpu, oracle_lib, k, strain):
    from aperi_mech_b200.model import ExplicitDynamics, Material, Part

    coords, conn, u, lam = _problem(k, strain)
    mat = Material.create("neo_hookean", 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    parts = [Part("hex8", mat, conn=conn)]
    want = oracle_lib.OracleProblem(coords, parts).vjp_force(u, lam)
    with ExplicitDynamics(coords, parts) as m:
        for got, ref in zip(m.vjp_force(u, lam), want):
            assert rel_err(got, ref) < _tolerance(k, strain)
