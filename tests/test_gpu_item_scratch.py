"""Segments cut into work items whose counting pass keeps their first
candidates: against the oracle with scratches that hold all, some and almost
none of an item's candidates, and without one."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap,limit", [(128, 1 << 31), (8, 1 << 31), (1, 1 << 31), (128, 1 << 19), (128, 0)])
@pytest.mark.parametrize("n", [1, 5, 300])
def test_items(oracle, cap, limit, n):
    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.mixed_mesh(60, 60, seed=2, extent=(60.0, 60.0))
    g, o = CellTree2d(xy, f, -1), oracle.OracleCellTree2d(xy, f, -1)
    t = g._tree
    t.SEG_SPEC_CAP, t.SEG_SPEC_MAX_BYTES, t.SPLIT_CELLS = cap, limit, 256
    assert t.edge_cut({}, n) is not None
    rng = np.random.default_rng(n)
    segs = rng.uniform(-5.0, 65.0, (n, 2, 2))
    segs[0] = [[0.0, 30.0], [60.0, 30.0]]
    for a, b in zip(g.intersect_edges(segs), o.intersect_edges(segs)):
        assert np.array_equal(a, b, equal_nan=True)
