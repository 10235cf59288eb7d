"""Which mesh-collider kernel a frame launches, by vertices and triangles: 8 or
16 lanes per vertex up to 20,480 vertices and 256 triangles or more, above that
(up to 32,768) only against 4,096 triangles or more.  In the default shape the
pass is a launch of its own on both sides of the line, with the bits of the
persistent solver's thread-per-vertex walk."""
import re

import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ntris,kernel", [
    (40, 256, "k_collision_lanesILj16E"), (101, 1280, "k_collision_lanesILj8E"),  # 3,200 and 20,402 vertices
    (102, 1280, "k_collisionILb0E"), (102, 4095, "k_collisionILb0E"),             # 20,808
    (102, 4096, "k_collision_lanesILj8E"), (128, 5120, "k_collision_lanesILj8E"), (129, 5120, "k_collisionILb0E")])
def test_lanes_by_size(tmp_path, n, ntris, kernel):
    sc = scenes.config2(n=n, subdiv=4 if ntris > 1280 else 3)
    tris = np.ascontiguousarray(sc["mesh"]["triangles"][:ntris])
    out = []
    for mode in (1, 4):
        s = scenes.build(ClothSimulator, sc)
        s.set_launch_config(mode, 1)
        s.set_enable_self_collision(False)
        s.set_auto_coupled_on_low_substeps(False)
        s.set_mesh_collider_triangles(tris, friction=0.4, thickness=0.004, restitution=0.1)
        x, _, v = [a.copy() for a in s.get_state()]
        v[:, 1] -= np.float32(8.0)
        s.set_positions_and_velocities(x, v)
        for _ in range(2):
            s.step(sc["dt"], 4, 2)
        out.append([a.copy() for a in s.get_state()])
    s.write_frame_graph(tmp_path / "frame.dot")
    found = set(re.findall(r"k_collision(?:_lanes)?IL[bj]\d+E", (tmp_path / "frame.dot").read_text()))
    assert found == {kernel}
    for a, b in zip(*out):
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a, b)
