"""Mesh collider with vertex thicknesses of any sign: the skip tests drop only
triangles that the reference's own test (segment to centroid against the square
of 1.5 radius + thickness) drops, so positions are the oracle's, which tests every
triangle.  Colliders with several lanes per vertex and with one."""
import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntris", [200, 1280])
@pytest.mark.parametrize("thickness", [0.004, -0.02, -0.1, -0.2])
def test_positions_match_oracle(oracle_lib, ntris, thickness):
    sc = scenes.config2(n=24, subdiv=3)
    sc["thickness"] = thickness
    sc["self_collision"] = False
    tris = sc["mesh"]["triangles"]
    order = np.argsort(-tris[:, :, 1].mean(1), kind="stable")  # the side the cloth falls on
    sc["mesh"]["triangles"] = np.ascontiguousarray(tris[order[:ntris]])
    v = np.zeros_like(sc["positions"])
    v[:, 1] = -8.0
    g = scenes.build(ClothSimulator, sc)
    o = scenes.build(oracle_lib.OracleSim, sc)
    g.set_positions_and_velocities(sc["positions"], v)
    o.set_state(sc["positions"], v)
    moved = False
    for _ in range(2):
        g.step(sc["dt"], 8, 2)
        o.step(sc["dt"], 8, 2)
        xg, xo = g.get_state()[0], o.get_state()[0]
        ext = np.linalg.norm(np.ptp(sc["positions"], axis=0))
        assert np.abs(xg.astype(np.float64) - xo).max() <= 1e-5 * ext
        moved = moved or np.ptp(xo[:, 1]) > 0.02
    assert moved  # the body stopped part of the cloth
