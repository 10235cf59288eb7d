"""Crowded cloth: layers pressed together until an edge has some tens of counted
edge-edge pairs, more than a cluster's pair buffer or a short pair list would
hold.  The default list takes them all, and the pairs and positions are those of
the search that works each edge's pairs in its own warp."""
import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


# 2, 4 and 8 edges per warp
@pytest.mark.parametrize("n,squeeze", [(40, 0.45), (70, 0.48), (121, 0.55), (121, 0.5)])
def test_default_list_holds_crowded_pairs(n, squeeze):
    sc = scenes.config2(n=n, subdiv=2)
    rng = np.random.default_rng(n)
    pos = sc["positions"].astype(np.float64)
    mid = pos.mean(0)
    x = mid + (pos - mid) * np.array([squeeze, 1.0, squeeze])
    x = (x + rng.normal(0.0, float(np.mean(sc["thickness"])), x.shape)).astype(np.float32)
    v = rng.normal(0.0, 0.02, x.shape).astype(np.float32)
    out, lists = [], []
    for variant in (0, 2):
        s = scenes.build(ClothSimulator, sc)
        s.clear_colliders()
        s.set_self_collision_variant(variant)
        s.set_pair_recording(True, 1 << 23, 1 << 23)
        s.set_positions_and_velocities(x, v)
        s.step(1.0 / 600.0, 1, 1)
        lists.append(s.get_pair_lists()["ee"])
        if variant == 0:
            listed, past = s.get_ee_pair_list()
            assert listed > 24 * len(sc["edges"]) + 1024
            assert past == 0
        s.step(1.0 / 600.0, 1, 1)
        out.append([a.copy() for a in s.get_state()])
    assert listed == len(lists[0])
    np.testing.assert_array_equal(*lists)
    for a, b in zip(*out):
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a, b)


def test_pairs_past_a_short_list_are_counted():
    sc = scenes.config2(n=40, subdiv=2)
    s = scenes.build(ClothSimulator, sc)
    s.set_ee_pair_list_capacity(256)
    s.step(sc["dt"], 6, 2)
    for _ in range(6):
        s.step(sc["dt"], 6, 2)
    listed, past = s.get_ee_pair_list()
    assert 0 < past < listed
    s.set_ee_pair_list_capacity(0)
    s.step(sc["dt"], 6, 2)
    assert s.get_ee_pair_list()[1] == 0
