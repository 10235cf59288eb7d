"""Runaway geometry beside cloth in contact: loose edges, neighbours of the cloth
in the searches' working order, whose positions lie beyond the range of the
hash cells on both sides.  The cloth's own pairs and positions are those it has
beside edges that lie within the range.  1, 4 and 8 vertices and 2, 4 and 8
edges per warp."""
import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


def _scene(n, where):
    sc = scenes.config2(n=n, subdiv=1)
    pos, edges = sc["positions"], sc["edges"].astype(np.int64)
    rng = np.random.default_rng(n)
    at = rng.choice(len(pos), len(pos) // 16, replace=False)
    a = pos[at] + np.float32(2e-4)
    b = a + np.array([1e-3, 0, 0], np.float32)
    far = np.zeros((2 * len(at), 3), np.float32)
    far[:, 0] = np.repeat(np.where(np.arange(len(at)) % 2, where, -where), 2)
    loose = np.stack([a, b], 1).reshape(-1, 3).astype(np.float32)
    k = np.arange(len(at))
    sc["edges"] = np.concatenate([edges, len(pos) + np.stack([2 * k, 2 * k + 1], 1)]).astype(np.uint32)
    sc["positions"] = np.concatenate([pos, loose])
    sc["inv_masses"] = np.concatenate([sc["inv_masses"], np.ones(len(loose), np.float32)])
    sc["layer_ids"] = np.concatenate([sc["layer_ids"], np.zeros(len(loose), np.uint32)])
    sc["mesh"] = None
    x = sc["positions"].copy()
    # the two layers into contact
    x[:len(pos), 1] = 0.45 + (x[:len(pos), 1] - 0.45) * 0.2
    far[:, 1:] = loose[:, 1:]  # beside the cloth but for x
    x[len(pos):] = far
    return sc, x, len(pos)


@pytest.mark.parametrize("n", [20, 90, 150])
def test_cloth_keeps_its_contacts(n):
    out = []
    for where in (1e4, 1e30):
        sc, x, n_cloth = _scene(n, where)
        s = scenes.build(ClothSimulator, sc)
        s.set_pair_recording(True, 1 << 22, 1 << 22)
        s.set_positions_and_velocities(x, np.zeros_like(x))
        s.step(1.0 / 600.0, 1, 1)
        lists = s.get_pair_lists()
        vt, ee = np.asarray(lists["vt"]), np.asarray(lists["ee"])
        cloth = (np.asarray(s.get_edges()[0]).reshape(-1, 2) < n_cloth).all(1)
        out.append((vt[(vt < n_cloth).all(1)], ee[cloth[ee].all(1)], s.get_state()[0][:n_cloth].copy()))
    assert len(out[0][0]) > n_cloth // 2 and len(out[0][1]) > n_cloth // 2
    for a, b in zip(*out):
        assert np.isfinite(b).all()
        np.testing.assert_array_equal(a, b)
