"""Many sphere and capsule colliders in the default launch shape.  From 128 on,
where a thread of the resident launch would have more than one vertex, the
collider pass is a launch of its own, and coupled (a pass per iteration) the
frame takes a launch per colour; otherwise the resident launch keeps it.  The
same bits as with a launch per colour."""
import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


def _frames(s, coupled, x0):
    s.set_enable_self_collision(False)
    s.set_coupled_collider(coupled)
    s.set_auto_coupled_on_low_substeps(False)
    v0 = np.zeros_like(x0)
    v0[:, 1] = -2.0
    out, kernels = [], []
    for mode in (0, 4):
        s.set_launch_config(mode)
        s.set_positions_and_velocities(x0, v0)
        for _ in range(2):
            s.step(1.0 / 60.0, 4, 2)
        out.append([a.copy() for a in s.get_state()])
        kernels.append(s.frame_kernel_count())
    for a, b in zip(*out):
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a, b)
    return kernels


def _spheres(k, side, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0.0, side, (k, 3))
    c[:, 1] = -0.05 * side
    return [("sphere", tuple(map(float, q)), 0.04 * side, 0.2) for q in c]


@pytest.mark.parametrize("coupled", [False, True])
@pytest.mark.parametrize("n,k,resident", [(64, 128, True), (72, 127, True), (72, 128, False), (98, 300, False)])
def test_many_spheres(n, k, resident, coupled):
    pos, edges, faces, idx = scenes.poke_grid(n, 1.0, seed=n)  # 8,065, 10,225 and 19,013 vertices
    s = ClothSimulator(pos, edges, faces, scenes.areal_inv_masses(pos, faces, 0.15))
    s.set_pin(int(idx[0, 0]), pos[idx[0, 0]] + np.float32(0.01), 0.5)
    for _, c, r, f in _spheres(k, 1.0, k):
        s.add_sphere_collider(c, r, friction=f)
    kernels = _frames(s, coupled, pos)
    assert (kernels[1] == 1) == resident
    if coupled and not resident:
        assert kernels[1] == kernels[0]


@pytest.mark.parametrize("k,resident", [(127, True), (128, False)])
def test_batch_goes_by_its_fullest_cloth(k, resident):
    sc = scenes.config4(3, seed=2, side_range=(58, 64))  # more than 8,192 vertices in all
    for i, inst in enumerate(sc["instances"]):
        inst["colliders"] = _spheres(k if i == 1 else 40, 0.6, i)
    s = scenes.build_batch(sc)
    pos = np.concatenate([inst["positions"] for inst in sc["instances"]])
    assert len(pos) > 8192
    kernels = _frames(s, False, pos)
    assert (kernels[1] == 1) == resident
