"""A coupled mesh collider (a pass per iteration) in the default launch shape.
With 256 triangles or more the pass has several lanes per vertex, which the
resident launch cannot give it, so the frame takes a launch per colour; with
fewer the resident launch keeps it.  The same bits as with the other shapes."""
import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ntris,resident", [(3, 255, True), (3, 256, False), (40, 255, True), (40, 256, False),
                                              (64, 1280, False), (65, 5120, False)])
def test_coupled_collider_leaves_the_resident_launch(n, ntris, resident):
    sc = scenes.config2(n=n, subdiv=4 if ntris > 1280 else 3)
    tris = np.ascontiguousarray(sc["mesh"]["triangles"][:ntris])
    out, kernels = [], []
    for mode in (1, 0, 4):
        s = scenes.build(ClothSimulator, sc)
        s.set_launch_config(mode, 1)
        s.set_enable_self_collision(False)
        s.set_coupled_collider(True)
        s.set_mesh_collider_triangles(tris, friction=0.4, thickness=0.004, restitution=0.1)
        s.set_pin(1, np.asarray(sc["positions"][1], np.float32) + np.float32(0.01), 0.5)
        x, _, v = [a.copy() for a in s.get_state()]
        v[:, 1] -= np.float32(8.0)
        s.set_positions_and_velocities(x, v)
        for _ in range(3):
            s.step(sc["dt"], 4, 2)
        out.append([a.copy() for a in s.get_state()])
        kernels.append(s.frame_kernel_count())
    assert (kernels[2] == 1) == resident
    assert resident or kernels[2] == kernels[1]
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.isfinite(b).all()
            np.testing.assert_array_equal(a, b)
    # uncoupled again, the iterations are resident and the pass is a launch of its own
    s.set_coupled_collider(False)
    s.set_auto_coupled_on_low_substeps(False)
    s.step(sc["dt"], 4, 2)
    assert s.frame_kernel_count() <= 4 * 4
