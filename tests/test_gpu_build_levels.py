"""The level passes of the builder (nodes above the subtree size) against the
oracle, bit for bit: cell numbers around the tile lengths, meshes whose nodes
need their other dimension on every level or on some, bounds that are zeros of
either sign, and numbers of buckets with and without the 4-bucket form."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cells(kind, n, rng):
    if kind == "strip":  # one row: nothing to split in y
        c = np.stack([rng.permutation(n).astype(float), np.zeros(n)], 1)
    elif kind == "columns":  # few columns, far apart: x splits at first only
        c = np.stack([100.0 * rng.integers(0, 3, n), rng.permutation(n).astype(float)], 1)
    elif kind == "heap":  # a third of the cells coincide
        c = rng.uniform(-50.0, 50.0, (n, 2))
        c[::3] = [7.0, -3.0]
    else:  # many bounds are zeros
        c = rng.integers(-40, 40, (n, 2)).astype(float)
    t = c[:, None, :] + np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
    t[(t == 0.0) & (rng.random(t.shape) < 0.5)] = -0.0
    return t.reshape(-1, 2), np.arange(3 * n).reshape(n, 3)


@pytest.mark.parametrize("kind", ["strip", "columns", "heap", "zeros"])
@pytest.mark.parametrize("n", [130, 511, 512, 513, 2049, 40961])
@pytest.mark.parametrize("nb", [4, 3])
def test_levels(oracle, kind, n, nb):
    from numba_celltree_gb300 import CellTree2d

    xy, f = _cells(kind, n, np.random.default_rng(n))
    g = CellTree2d(xy, f, -1, nb, 2)
    o = oracle.OracleCellTree2d(xy, f, -1, nb, 2)
    assert np.array_equal(g.bb_indices, o.bb_indices)
    assert len(g.nodes) == len(o.nodes)
    for k in ("child", "Lmax", "Rmin", "ptr", "size", "dim"):
        assert np.ascontiguousarray(g.nodes[k]).tobytes() == np.ascontiguousarray(o.nodes[k]).tobytes(), k
