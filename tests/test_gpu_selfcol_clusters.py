"""The cluster searches of the self-collision passes where they can go wrong:
vertices that are neighbours in the working order but far apart in space,
crowds that outgrow the queues and the pair buffer, stars of more than 8
triangles, hash buckets of several cells, a small cap on counted pairs, sizes
around a cluster and a block.  Pair lists, positions and the untangled layers
against the oracle, which searches element by element: integer accumulators
and the same float operations, so the same bits."""
import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


def _fan(k, centre, radius, rng):
    """One vertex with a star of k triangles."""
    t = np.linspace(0.0, 2.0 * np.pi, k, endpoint=False)
    p = np.zeros((k + 1, 3))
    p[1:, 0], p[1:, 2] = radius * np.cos(t), radius * np.sin(t)
    p += np.asarray(centre) + rng.uniform(-1e-4, 1e-4, p.shape)
    f = [(0, 1 + i, 1 + (i + 1) % k) for i in range(k)]
    return p, f


def _scene(kind, seed):
    rng = np.random.default_rng(seed)
    parts = []
    if kind == "one":                       # fewer vertices than a cluster
        parts.append(_fan(3, (0, 0, 0), 0.01, rng))
        parts.append(_fan(3, (0, 0.003, 0), 0.01, rng))
    elif kind == "fans":                    # large stars over each other, an odd count
        for i in range(9):
            parts.append(_fan(5 + 3 * i, (0.012 * (i % 3), 0.0025 * i, 0.012 * (i // 3)), 0.015, rng))
    elif kind == "scattered":               # pairs of triangles metres apart
        for i in range(75):
            c = rng.uniform(-3.0, 3.0, 3)
            parts.append(_fan(3, c, 0.008, rng))
            parts.append(_fan(4, c + (0.001, 0.003, 0.0), 0.008, rng))
    elif kind == "crowd":                   # everything within a few cells
        for i in range(150):
            parts.append(_fan(6, rng.uniform(-0.02, 0.02, 3), 0.008, rng))
    elif kind == "wide":                    # coordinates far from the origin, shared buckets
        for i in range(400):
            c = np.round(rng.uniform(-60.0, 60.0, 3), 0)
            parts.append(_fan(3, c, 0.006, rng))
            parts.append(_fan(3, c + (0.0, 0.002, 0.0), 0.006, rng))
    pos, faces, layers, off = [], [], [], 0
    for i, (p, f) in enumerate(parts):
        pos.append(p)
        faces += [(a + off, b + off, c + off) for a, b, c in f]
        layers += [i % 3] * len(p)
        off += len(p)
    pos = np.concatenate(pos).astype(np.float32)
    # a shuffled numbering: index order says nothing about space
    perm = rng.permutation(len(pos))
    inv = np.argsort(perm)
    pos, layers = pos[perm], np.asarray(layers, np.uint32)[perm]
    faces = inv[np.asarray(faces)].astype(np.uint32)
    e = {tuple(sorted((int(f[i]), int(f[(i + 1) % 3])))) for f in faces for i in range(3)}
    return pos, np.asarray(sorted(e), np.uint32), faces, layers


def _build(cls, kind, seed, max_iterations=None):
    pos, edges, faces, layers = _scene(kind, seed)
    s = cls(pos, edges, faces, scenes.areal_inv_masses(pos, faces, 0.15), layer_ids=layers, thickness=0.002)
    s.set_gravity(0.0, -9.81, 0.0)
    s.set_compliance_all(1e-8, 1e-8, 1e-6, 1e-5)
    s.set_enable_self_collision(True)
    if max_iterations is not None:
        s.set_self_collision_options(0.2, 0.2, True, True, max_iterations)
    s.set_pin(0, pos[0], 1.0)
    v = np.random.default_rng(seed + 1).uniform(-0.5, 0.5, pos.shape).astype(np.float32)
    return s, pos, v


@pytest.mark.parametrize("kind,cap", [("one", None), ("fans", None), ("fans", 3), ("scattered", None),
                                      ("crowd", None), ("crowd", 7), ("wide", None)])
def test_pairs_and_positions_match_oracle(oracle_lib, kind, cap):
    g, pos, v = _build(ClothSimulator, kind, 5, cap)
    o, _, _ = _build(oracle_lib.OracleSim, kind, 5, cap)
    g.set_positions_and_velocities(pos, v)
    o.set_state(pos, v)
    g.set_pair_recording(True, 4 << 20, 4 << 20)
    o.set_pair_recording(True)
    for _ in range(3):
        g.step(1.0 / 600.0, 1, 2)
        o.step(1.0 / 600.0, 1, 2)
        a, b = g.get_pair_lists(), o.get_pair_lists()
        np.testing.assert_array_equal(a["vt"], b["vt"])
        np.testing.assert_array_equal(a["ee"], b["ee"])
        assert len(b["ee"]) > 0
        xg, xo = g.get_state()[0], o.get_state()[0]
        ext = np.linalg.norm(pos.max(0) - pos.min(0))
        assert np.abs(xg.astype(np.float64) - xo).max() <= 1e-5 * ext


@pytest.mark.parametrize("kind", ["crowd", "fans"])
@pytest.mark.parametrize("variant", [1, 2])
def test_edge_search_variants_agree(kind, variant):
    out = []
    for k in (0, variant):
        s, pos, v = _build(ClothSimulator, kind, 9)
        s.set_self_collision_variant(k)
        s.set_positions_and_velocities(pos, v)
        for _ in range(4):
            s.step(1.0 / 600.0, 1, 2)
        out.append(s.get_state()[0].copy())
    np.testing.assert_array_equal(out[0], out[1])
