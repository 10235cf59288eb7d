"""State to and from the simulator (set_positions_and_velocities, get_state)
beside other calls, below and above the size up to which it crosses the bus in
one copy (16,384 vertices)."""
import threading

import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu

SIDES = [40, 121]  # two layers: 3,200 and 29,282 vertices


def _held(n):
    """Layers with self-collision on and every vertex immovable: no call
    changes the state."""
    sc = scenes.config2(n=n, subdiv=2)
    s = ClothSimulator(sc["positions"], sc["edges"], sc["faces"], np.zeros(len(sc["positions"]), np.float32),
                       layer_ids=sc["layer_ids"], thickness=sc["thickness"])
    s.set_gravity(0.0, 0.0, 0.0)
    s.set_enable_self_collision(True)
    s.set_solver_iterations(1)
    return s, sc["positions"]


@pytest.mark.parametrize("n", SIDES)
@pytest.mark.parametrize("busy", ["frames", "seeks"])
def test_a_second_thread_reads_a_whole_state(n, busy):
    s, pos = _held(n)
    still = np.zeros_like(pos)
    s.set_positions_and_velocities(pos, still)
    s.step(1.0 / 60.0, 4)  # the frame is recorded before the threads start
    bad, stop = [], threading.Event()

    def read():
        while not stop.is_set():
            for name, got, want in zip("xpv", s.get_state(), (pos, pos, still)):
                if not np.array_equal(got, want):
                    bad.append(name)

    t = threading.Thread(target=read)
    t.start()
    try:
        for _ in range(150):
            if busy == "frames":
                s.step(1.0 / 60.0, 4)
            else:
                s.set_positions_and_velocities(pos, still)
    finally:
        stop.set()
        t.join()
    assert not bad, (len(bad), bad[:3])


@pytest.mark.parametrize("n", SIDES)
def test_masses_follow_pins_and_settings_through_seeks(n):
    """Inverse masses cross with the state only when they may have changed: a
    simulator that was seeked before its pins and masses changed goes the same
    way as one that had them from the start."""
    sc = scenes.config2(n=n, subdiv=2)
    rng = np.random.default_rng(3)
    held = rng.choice(len(sc["positions"]), 6, replace=False)
    v = rng.uniform(-0.1, 0.1, sc["positions"].shape).astype(np.float32)

    def masses(s):
        for k in held[:3]:
            s.set_pin(int(k), sc["positions"][k], 1.0)
        s.set_pin(int(held[3]), sc["positions"][held[3]], 0.5)
        s.set_vertex_inv_masses(held[4:], np.array([0.0, 3.0], np.float32))

    a, b = (scenes.build(ClothSimulator, sc) for _ in range(2))
    masses(a)
    b.set_positions_and_velocities(sc["positions"], v)
    b.step(1.0 / 60.0, 4)
    b.set_pin(int(held[5]), sc["positions"][held[5]], 1.0)
    b.set_positions_and_velocities(sc["positions"], v)
    b.release_pin(int(held[5]))
    masses(b)
    for _ in range(2):  # with the masses, then without
        for s in (a, b):
            s.set_positions_and_velocities(sc["positions"], v)
            s.step(1.0 / 60.0, 4)
        for x, y in zip(a.get_state(), b.get_state()):
            np.testing.assert_array_equal(x, y)
