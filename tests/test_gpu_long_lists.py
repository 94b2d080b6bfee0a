"""Open points in grid cells with long candidate lists: vertices and edge points
of a mesh whose cells grow by a factor of thousands, by a warp, by a lane and
in the staged form, against the oracle."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["triangle", "quad"])
@pytest.mark.parametrize("n", [2000, 40_000, 120_000])
def test_vertices_of_a_graded_mesh(oracle, kind, n):
    from numba_celltree_gb300 import CellTree2d

    make = syn.triangle_mesh if kind == "triangle" else syn.quad_mesh
    xy, f = make(150, seed=71)
    xy = np.exp(8.0 * xy)
    rng = np.random.default_rng(72)
    pts = xy[rng.integers(0, len(xy), n)].copy()
    a, b = xy[f[rng.integers(0, len(f), n // 4), 0]], xy[f[rng.integers(0, len(f), n // 4), 1]]
    pts[: n // 4] = a + rng.random((n // 4, 1)) * (b - a)
    t = CellTree2d(xy, f, -1)
    longest = int((t._tree.cand_off[1:] - t._tree.cand_off[:-1]).max())
    assert longest > 1000
    want = oracle.OracleCellTree2d(xy, f, -1).locate_points(pts)
    assert np.array_equal(t.locate_points(pts), want)
