"""Subtree nodes by a lane each: trees of sizes around the lane limit and the
subtree limit against the oracle, bit for bit, with cells that coincide (a node
turned to the other dimension, or left a leaf), with bounds that tie and differ
only in the sign of a zero, and with split costs too close for float32."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("child", "Lmax", "Rmin", "ptr", "size", "dim")


def _triangles(kind, n, rng):
    """n separate triangles: vertices and faces."""
    if kind == "random":
        c, s = rng.uniform(0.0, 10.0, (n, 2)), rng.uniform(0.05, 2.0, (n, 1, 1))
    elif kind == "same":  # few distinct cells
        c, s = rng.integers(0, 3, (n, 2)).astype(float), 0.25
    elif kind == "line":  # nothing to split in y
        c, s = np.stack([np.arange(n, dtype=float), np.zeros(n)], 1), 0.5
    elif kind == "even":  # equal costs on either side of the middle
        k = int(np.ceil(np.sqrt(n)))
        c, s = np.stack(np.meshgrid(np.arange(k), np.arange(k)), -1).reshape(-1, 2)[rng.permutation(k * k)[:n]] * 1.0, 0.5
    else:  # zeros of either sign among the bounds
        c, s = rng.integers(-1, 2, (n, 2)).astype(float), 1.0
    t = c[:, None, :] + s * np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
    if kind == "zeros":
        t[(t == 0.0) & (rng.random(t.shape) < 0.5)] = -0.0
    return t.reshape(-1, 2), np.arange(3 * n).reshape(n, 3)


@pytest.mark.parametrize("kind", ["random", "same", "line", "even", "zeros"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 31, 32, 33, 64, 65, 127, 128, 129, 700])
@pytest.mark.parametrize("nb,cpl", [(4, 1), (4, 2), (4, 31), (4, 33), (3, 2)])
def test_small_trees(oracle, kind, n, nb, cpl):
    from numba_celltree_gb300 import CellTree2d

    xy, f = _triangles(kind, n, np.random.default_rng(n))
    g = CellTree2d(xy, f, -1, nb, cpl)
    o = oracle.OracleCellTree2d(xy, f, -1, nb, cpl)
    assert np.array_equal(g.bb_indices, o.bb_indices)
    assert len(g.nodes) == len(o.nodes)
    for k in FIELDS:
        a, b = np.ascontiguousarray(g.nodes[k]), np.ascontiguousarray(o.nodes[k])
        assert a.tobytes() == b.tobytes(), k
