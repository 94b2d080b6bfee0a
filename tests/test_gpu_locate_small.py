"""Small batches of points on both sides of the warp-per-point limit, and grid
cells that list more than a warp's worth of cells, against the oracle."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 20, 45])  # of one mesh, shifted a little: any number of cells hold a point
@pytest.mark.parametrize("n", [1, 5, 32768, 32769])
def test_small_batches(oracle, copies, n):
    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.mixed_mesh(9, 7, seed=copies, extent=(9.0, 7.0))
    shift = 0.01 * np.arange(copies)[:, None, None]
    faces = np.where(f[None] >= 0, f[None] + len(xy) * np.arange(copies)[:, None, None], -1).reshape(-1, f.shape[1])
    xy = (xy[None] + shift).reshape(-1, 2)
    g, o = CellTree2d(xy, faces, -1), oracle.OracleCellTree2d(xy, faces, -1)
    rng = np.random.default_rng(n)
    p = rng.uniform(-0.5, 9.5, (max(n, 40), 2))
    p[::3] = xy[rng.integers(0, len(xy), len(p[::3]))]  # on vertices
    p = p[-n:]
    assert np.array_equal(g.locate_points(p), o.locate_points(p))
