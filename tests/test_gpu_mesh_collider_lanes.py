"""The mesh-collider pass with several lanes per vertex (up to 32,768 vertices,
256 triangles and more) against the thread-per-vertex walk of the persistent
solver: the same triangles in the same order, so the same bits.  Vertex counts
on both sides of the lane rule's lines, triangle counts at the edges of the
runs of 16, 256 and 4,096, one- and two-sided triangles, with and without
self-collision, and the default shape, where the pass leaves the resident
launch."""
import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ntris,single,self_collision", [
    (3, 320, True, False), (33, 255, True, True), (33, 256, False, True), (33, 257, True, False),
    (64, 1279, True, False), (64, 4097, False, False), (65, 1280, True, True), (65, 20480, False, False),
    (128, 5120, True, False), (129, 5120, False, False)])
def test_lanes_match_the_serial_walk(n, ntris, single, self_collision):
    sc = scenes.config2(n=n, subdiv=5 if ntris > 5120 else 4 if ntris > 1280 else 3)
    tris = np.ascontiguousarray(sc["mesh"]["triangles"][:ntris])
    assert len(tris) == ntris
    out = []
    for mode in (1, 0, 4):
        s = scenes.build(ClothSimulator, sc)
        s.set_launch_config(mode, 1)
        s.set_enable_self_collision(self_collision)
        s.set_mesh_collider_triangles(tris, friction=0.4, thickness=0.004, restitution=0.1, single_sided=single)
        s.set_pin(1, np.asarray(sc["positions"][1], np.float32) + np.float32(0.01), 0.5)
        # into the body within the frame: contacts that move p many times in one walk
        x, _, v = [a.copy() for a in s.get_state()]
        v[:, 1] -= np.float32(8.0)
        s.set_positions_and_velocities(x, v)
        for _ in range(3):
            s.step(sc["dt"], 4, 2)
        out.append([a.copy() for a in s.get_state()])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.isfinite(b).all()
            np.testing.assert_array_equal(a, b)
