"""Training gradients at the edges of the row and tile loops: fewer rows than a
warp, ragged last tiles, a vertex without neighbours, one with more than 32.
Against the numpy reference with its bf16 rounding points, tolerances as for
the grid graphs (2e-2 of each tensor's norm: bf16 operands, fp32 sums)."""
import numpy as np
import pytest

from oracle import warmstart_ref as W
from taremincloth_b200 import warmstart

pytestmark = pytest.mark.gpu


def _graph(n, rng):
    """A ring, a hub joined to up to 50 vertices, and the last vertex alone."""
    pairs = set()
    for i in range(n - 2):
        pairs.add((i, i + 1))
    for j in rng.choice(n - 1, size=min(50, n - 1), replace=False) if n > 2 else []:
        if j:
            pairs.add((0, int(j)))
    nb = [[] for _ in range(n)]
    for a, b in pairs:
        nb[a].append(b)
        nb[b].append(a)
    off = np.concatenate([[0], np.cumsum([len(v) for v in nb])]).astype(np.uint32)
    idx = np.asarray([j for v in nb for j in sorted(v)], np.uint32)
    return off, idx


@pytest.mark.parametrize("n", [2, 15, 17, 127, 129, 1000, 40001])
def test_gradients_match_reference(n):
    rng = np.random.default_rng(n)
    off, idx = _graph(n, rng)
    feat = rng.normal(0, 1, (n, 16)).astype(np.float32)
    target = rng.normal(0, 0.3, (n, 3)).astype(np.float32)
    mask = (rng.random(n) > 0.1).astype(np.float32)
    mask[0] = 1.0
    blob = W.random_params(rng)
    loss_g, grad_g, y_g = warmstart.mlp_grad(feat, off, idx, target, mask, blob)
    loss_r, grad_r, y_r = W.forward_backward(feat, off, idx, target, mask, blob)
    assert abs(loss_g - loss_r) <= 1e-3 * abs(loss_r)
    assert np.linalg.norm(y_g - y_r) <= 5e-3 * np.linalg.norm(y_r)
    for name, o, shape in W.LAYOUT:
        k = int(np.prod(shape))
        a, b = grad_g[o:o + k].astype(np.float64), np.asarray(grad_r[o:o + k], np.float64)
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b), name
