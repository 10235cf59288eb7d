"""The resident solver (one thread-block cluster with the cloth on chip)
against one launch per colour: the same per-element arithmetic in the same
order, so the same bits.  Sizes at the edges of its range: a cloth smaller than
a warp, one and two CTAs, the full cluster, vertices too many for x and v to
stay on chip, and one that no longer fits."""
import numpy as np
import pytest

from oracle import warmstart_ref as W
from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


def _sheet(n, damped, coupled):
    pos, edges, faces, idx = scenes.poke_grid(n, 1.0, seed=n)
    s = ClothSimulator(pos, edges, faces, scenes.areal_inv_masses(pos, faces, 0.15))
    s.set_gravity(0.0, -9.81, 0.0)
    s.set_compliance_all(1e-8, 1e-6, 1e-6, 1e10 if n == 17 else 1e-5)  # 17: bending off
    if damped:
        s.set_damping_all(5.0, 3.0, 2.0, 0.5)
    s.set_enable_self_collision(False)
    s.set_coupled_collider(coupled)
    s.set_pin(int(idx[n - 1, 0]), pos[idx[n - 1, 0]], 1.0)
    s.set_pin(int(idx[n - 1, n - 1]), pos[idx[n - 1, n - 1]] + np.float32(0.01), 0.5)  # compliant
    s.add_sphere_collider((0.5, -0.2501, 0.5), 0.25, friction=0.3)
    return s


def _both(s, frames, substeps, iterations, dt=1.0 / 60.0):
    x0, _, v0 = s.get_state()
    out, kernels = [], []
    for mode in (0, 4):
        s.set_launch_config(mode)
        s.set_positions_and_velocities(x0.copy(), v0.copy())
        for _ in range(frames):
            s.step(dt, substeps, iterations)
        out.append([a.copy() for a in s.get_state()])
        kernels.append(s.frame_kernel_count())
    for a, b in zip(*out):
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a, b)
    return kernels


@pytest.mark.parametrize("n,fits", [(2, True), (3, True), (16, True), (17, True), (64, True), (98, True), (140, False)])
@pytest.mark.parametrize("damped,coupled,iterations", [(False, False, 3), (True, True, 1)])
def test_matches_colour_launches(n, fits, damped, coupled, iterations):
    kernels = _both(_sheet(n, damped, coupled), 2, 6, iterations)
    assert (kernels[1] == 1) == fits


@pytest.mark.parametrize("n", [9, 40, 96])
def test_sewn_garment_matches_colour_launches(n):
    # sewing colours, seam-gated bending, the final sewing pass, self-collision
    sc = scenes.sewn_garment(n=n)
    s = scenes.build(ClothSimulator, sc)
    rest = np.array(s.get_sewing_current_rest_lengths())
    x0, _, v0 = s.get_state()
    out = []
    for mode in (0, 4):
        s.set_launch_config(mode)
        s.set_positions_and_velocities(x0.copy(), v0.copy())
        s.set_sewing_current_rest_lengths(rest)
        for _ in range(5):
            s.step(sc["dt"], sc["substeps"])
        out.append((s.get_state()[0].copy(), np.array(s.get_sewing_current_rest_lengths())))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


def test_follows_changed_pins_and_stiffness():
    s = _sheet(24, False, False)
    _both(s, 1, 5, 2)
    s.set_compliance_all(1e-7, 1e10, 1e-5, 1e-4)
    s.set_pin(100, (0.1, 0.2, 0.3), 1.0)
    s.release_pin(23 * 24)
    _both(s, 1, 5, 2)


def test_mesh_without_triangles_and_single_step():
    # a strand: two colours, no bending; and one edge: a single step
    for k in (2, 40):
        pos = np.zeros((k, 3), np.float32)
        pos[:, 0] = np.arange(k) * 0.1
        e = np.stack([np.arange(k - 1), np.arange(1, k)], 1).astype(np.uint32)
        s = ClothSimulator(pos, e, None)
        s.set_enable_self_collision(False)
        s.set_pin(0, pos[0], 1.0)
        kernels = _both(s, 2, 4, 3)
        assert kernels[1] == 1


@pytest.mark.parametrize("threshold", [None, float("inf"), 1e-4, -1.0])
def test_chosen_persistent_solver_matches_the_default(threshold):
    # without and with the warm start (never, as the residual says, always falling back)
    out, stats = [], []
    for mode in (1, 4):
        s = _sheet(32, False, False)
        s.set_launch_config(mode, 1)
        s.set_solver_iterations(4)
        if threshold is not None:
            s.ws_set_params(W.random_params(np.random.default_rng(3), scale_head=0.05))
            s.ws_enable(2, threshold)
        for _ in range(2):
            s.step(1.0 / 60.0, 6)
        out.append([a.copy() for a in s.get_state()])
        stats.append(s.ws_stats() if threshold is not None else None)
    for a, b in zip(*out):
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a, b)
    assert stats[0] == stats[1]
