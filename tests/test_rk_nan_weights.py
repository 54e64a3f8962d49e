"""A NaN among the two-pass coupling's function values reaches the force whatever its bits, those
of the octet rows' padding mark among them."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("octets", ["1", "0"])
@pytest.mark.parametrize("bits", [0x7FF8000000000000, 0x7FF8DEAD00000000, 0x7FF8DEAD12345678])
def test_nan_weight_is_not_padding(gpu, monkeypatch, bits, octets):
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import ExplicitDynamics, Material
    from aperi_mech_b200.smoothing import element_smoothing_part

    monkeypatch.setenv("APERI_B200_RK_OCTETS", octets)
    coords, hexes = mesh.box_hex(3, 2, 2)
    n = coords.shape[0]
    mat = Material.create("linear_elastic", 1000.0, youngs_modulus=1e9, poissons_ratio=0.3)
    part, mass = element_smoothing_part(coords, mesh.hex_to_tets(hexes), mat)
    val = np.ones(n)
    val[5] = np.array([bits], dtype=np.uint64).view(np.float64)[0]
    rk = (np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), val)
    d = 1e-3 * np.random.default_rng(0).standard_normal(coords.shape)
    with ExplicitDynamics(coords, [part], mass=mass, rk=rk) as m:
        f = m.internal_force(d, "fp64")
    assert np.isnan(f[5]).all()
