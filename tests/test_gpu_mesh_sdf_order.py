"""The single-mesh bake walks a tree over reordered triangles; the first of
equally near triangles still has to win.  Against the oracle's scan in triangle
order, texel for texel: one triangle, fewer than a run, ragged last runs on
every level, coincident and degenerate triangles, ties across shared edges."""
import numpy as np
import pytest

from taremincloth_b200.simulator import bake_mesh_sdf_gpu

pytestmark = pytest.mark.gpu


def _mesh(nt, seed):
    rng = np.random.default_rng(seed)
    if nt >= 64:  # a bumpy sheet of quads: every inner edge and vertex is shared
        m = int(np.ceil(np.sqrt(nt / 2))) + 1
        g = np.stack(np.meshgrid(np.arange(m), np.arange(m), indexing="ij"), -1).reshape(-1, 2) / (m - 1) * 0.3
        v = np.c_[g, np.round(rng.uniform(0.0, 0.05, len(g)), 2)]
        i = np.arange(m * m).reshape(m, m)
        a, b, c, d = i[:-1, :-1].ravel(), i[:-1, 1:].ravel(), i[1:, 1:].ravel(), i[1:, :-1].ravel()
        t = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)])[:nt]
    else:
        v = rng.uniform(0.0, 0.3, (nt + 2, 3))
        t = np.stack([np.arange(nt), np.arange(nt) + 1, np.arange(nt) + 2], 1)
    t = t[rng.permutation(len(t))]
    if nt > 2:
        t[-1] = t[0][[1, 2, 0]]      # the same triangle again, turned round
        t[-2] = [t[1][0]] * 3        # a point
    return v.astype(np.float32), t.astype(np.int32)


@pytest.mark.parametrize("nt", [1, 3, 8, 9, 64, 65, 513, 1000])
def test_matches_scan_in_triangle_order(oracle_lib, nt):
    v, t = _mesh(nt, nt)
    g = bake_mesh_sdf_gpu(v, t, voxel_size=0.015, close_open_boundaries=False)
    dims, info, tex = oracle_lib.bake_mesh_sdf(v, t, 0.015)
    assert (g["width"], g["height"], g["depth"]) == tuple(int(x) for x in dims)
    np.testing.assert_array_equal(g["bone_info"], info)
    np.testing.assert_array_equal(np.frombuffer(g["texture_bytes"], np.uint32), np.asarray(tex).ravel())
