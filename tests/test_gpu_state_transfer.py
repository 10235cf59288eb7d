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
