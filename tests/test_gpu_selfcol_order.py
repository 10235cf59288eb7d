"""Order of the self-collision pass's launches: the two sides run on streams of
their own, and everything that may do contact work comes after the kernel
that writes the vertex normals.  The edge filter does contact work on the
pairs that its list does not hold, so a list too small for the scene changes
nothing."""
import re

import numpy as np
import pytest

from taremincloth_b200 import ClothSimulator, scenes

pytestmark = pytest.mark.gpu


def _graph(sim, path):
    """(node -> kernel name, node -> its direct successors) of the recorded frame."""
    sim.write_frame_graph(path)
    text = path.read_text()
    names = {m.group(1): m.group(2) for m in re.finditer(r'"(\w+_node_\d+)"\s*\[(.*?)\];', text, flags=re.S)}
    after = {k: set() for k in names}
    for a, b in re.findall(r'"(\w+_node_\d+)"\s*->\s*"(\w+_node_\d+)"', text):
        after[a].add(b)
    return names, after


def _nodes(names, kernel):
    return [k for k, label in names.items() if re.search(r"\d%s[IEv]" % kernel, label)]


def _reached(after, start):
    seen, todo = set(), [start]
    while todo:
        for b in after[todo.pop()] - seen:
            seen.add(b)
            todo.append(b)
    return seen


@pytest.mark.parametrize("variant,edge_kernels", [(0, ("k_ee_cluster", "k_ee_pairs", "k_ee_ccd")),
                                                  (1, ("k_ee_grouped", "k_ee_ccd")), (2, ("k_ee", "k_ee_ccd"))])
def test_contact_work_comes_after_the_normals(tmp_path, variant, edge_kernels):
    sc = scenes.config2(n=24, subdiv=2)
    s = scenes.build(ClothSimulator, sc)
    s.set_self_collision_variant(variant)
    s.step(sc["dt"] / sc["substeps"], 1)
    names, after = _graph(s, tmp_path / "frame.dot")
    (normals,) = _nodes(names, "k_star_box")
    reached = _reached(after, normals)
    for kernel in ("k_sc_solve", "k_untangle", "k_apply") + edge_kernels:
        found = _nodes(names, kernel)
        assert len(found) == 1, kernel
        assert found[0] in reached, kernel


@pytest.mark.parametrize("n", [20, 40])  # 800 and 3,200 vertices
@pytest.mark.parametrize("entries", [256 * 4, 256])
def test_overflowing_pair_list_changes_nothing(n, entries):
    """Two layers, untangling on, frames with the layers in contact: a list of
    4 pairs or 1 per segment against one that holds every pair; the contacts go
    through integer accumulators, so the same bits."""
    sc = scenes.config2(n=n, subdiv=2)
    sims = [scenes.build(ClothSimulator, sc) for _ in range(2)]
    for s, cap in zip(sims, (1 << 20, entries)):
        s.set_ee_pair_list_capacity(cap)
        s.set_pair_recording(True, 1 << 22, 1 << 22)
    most = 0
    for _ in range(12):
        for s in sims:
            s.step(sc["dt"], 6, 2)
        a, b = (s.get_pair_lists() for s in sims)
        np.testing.assert_array_equal(a["ee"], b["ee"])
        np.testing.assert_array_equal(a["vt"], b["vt"])
        most = max(most, len(a["ee"]))
        for u, w in zip(sims[0].get_state(), sims[1].get_state()):
            np.testing.assert_array_equal(u, w)
    assert most > 2 * entries  # most pairs did not fit
