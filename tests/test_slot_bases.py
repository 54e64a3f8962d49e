"""Models whose first block has a slot count that is no multiple of four, followed by hexes,
whose kernels read their slot positions two (FP64) and four (mixed) at a time: every block must
begin at a multiple of four. The host rule is checked alone; the force, its VJP and a few steps
of such models against the oracle."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import rel_err

ROOT = Path(__file__).resolve().parent.parent


def test_blocks_begin_at_multiples_of_four(tmp_path):
    exe = tmp_path / "slot_bases"
    res = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror",
                          f"-I{ROOT / 'aperi_mech_b200' / 'csrc'}", str(ROOT / "tests" / "cxx" / "slot_bases_dump.cpp"),
                          "-o", str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    rng = np.random.default_rng(3)
    for counts in ([5, 8], [1, 2, 3, 4], [0, 7, 0, 64], [8, 16], list(rng.integers(0, 1000, 50))):
        out = subprocess.run([str(exe), *map(str, counts)], capture_output=True, text=True, check=True).stdout
        base = [int(x) for x in out.split()]
        assert len(base) == len(counts) + 1 and base[0] == 0
        for k, c in enumerate(counts):
            assert base[k] % 4 == 0
            assert 0 <= base[k + 1] - base[k] - c < 4


def _first_block(kind, coords, conn, mat):
    """A block with an odd slot count before the hexes, and its nodal mass."""
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import Part

    tets = mesh.hex_to_tets(conn[:1])
    if kind.startswith("tet4"):  # warp-chunked: one slot per distinct node
        n = int(kind[4:])
        return Part("tet4", mat, conn=tets[:n])
    rng = np.random.default_rng(11)
    sizes = (3, 4, 6) if kind == "entries" else (9, 12)  # one slot per entry / per touched node
    nodes = [rng.choice(coords.shape[0], size=s, replace=False) for s in sizes]
    grads = [rng.uniform(-1.0, 1.0, (s, 3)) for s in sizes]
    grads = [g - g.mean(axis=0) for g in grads]  # a constant field has no gradient
    return Part("cells", mat, cell_ptr=np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64),
                cell_nodes=np.concatenate(nodes).astype(np.int32), cell_grads=np.concatenate(grads),
                cell_volumes=rng.uniform(0.005, 0.01, len(sizes)))


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["tet41", "tet42", "tet43", "tet44", "entries", "touched"])
@pytest.mark.parametrize("material", ["linear_elastic", "neo_hookean"])
def test_hexes_after_an_odd_block_match_oracle(gpu, oracle_lib, first, material):
    """FP64 at the parity tests' 1e-12 (force, steps) and 1e-11 (VJP), mixed at their 5e-5."""
    from aperi_mech_b200 import mesh
    from aperi_mech_b200.model import ExplicitDynamics, Material, Part

    coords, conn = mesh.box_hex(3, 3, 3)
    rng = np.random.default_rng(5)
    coords = mesh.jitter_interior(coords, 0.03, rng)
    mat = Material.create(material, 1000.0, shear_modulus=3.85e8, bulk_modulus=8.33e8)
    parts = [_first_block(first, coords, conn, mat), Part("hex8", mat, conn=conn)]
    mass = np.full(coords.shape[0], 1000.0 / coords.shape[0])
    u = 2e-3 * rng.standard_normal(coords.shape) + 1e-3 * coords @ rng.standard_normal((3, 3))
    lam = rng.standard_normal(coords.shape)
    v0 = rng.uniform(-1.0, 1.0, coords.shape)
    z = np.zeros_like(coords)
    dt = 2e-6  # well below h / c = 0.2 / 1150 s
    op = oracle_lib.OracleProblem(coords, parts, mass=mass)
    want = op.internal_force(u)
    with ExplicitDynamics(coords, parts, mass=mass) as m:
        assert rel_err(m.internal_force(u, "fp64"), want) < 1e-12
        assert rel_err(m.internal_force(u, "mixed"), want) < 5e-5
        for g, w in zip(m.vjp_force(u, lam), op.vjp_force(u, lam)):
            assert rel_err(g, w) < 1e-11
        m.set_state(z, v0)
        m.init_acceleration()
        m.run(5, dt)
        for g, w in zip(m.get_state(), op.steps(z, v0, op.init_acceleration(z), np.full(5, dt))):
            assert rel_err(g, w) < 1e-11
