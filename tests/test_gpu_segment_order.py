"""Segments run in spatial order and finished per segment: results against the
oracle for hit counts on both sides of the warp (128) and shared-memory (1024)
sorts, with ties in t, with and without the spatial order."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _same(a, b):
    for x, y in zip(a, b):
        x = x.cpu().numpy() if hasattr(x, "cpu") else x
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("work_order", [None, True])
@pytest.mark.parametrize("cells", [30, 127, 128, 129, 1023, 1024, 1025, 2500])
def test_hits_per_segment(oracle, cells, work_order):
    import torch

    from numba_celltree_gb300 import CellTree2d

    # a strip of `cells` quads: a segment along it crosses them all, one on
    # the shared line of two strips touches both (ties in t)
    xy, f = syn.quad_mesh(cells, 2, seed=cells, extent=(float(cells), 2.0), jitter=0.0)
    rng = np.random.default_rng(cells)
    y = rng.uniform(0.05, 1.95, 40)
    segs = np.stack([np.stack([np.full(40, -0.5), y], 1), np.stack([np.full(40, cells + 0.5), y[::-1]], 1)], 1)
    segs[:3, :, 1] = 1.0
    segs[5:20] = segs[5:20, ::-1]
    segs[20:30, 1, 0] = rng.uniform(0, cells, 10)
    segs[30:, :, 0] = rng.uniform(-1, cells + 1, (10, 2))
    t = CellTree2d(xy, f, -1)
    got = t._tree.locate_edges(torch.as_tensor(segs, device="cuda"), 1, {"work_order": work_order})
    _same(got, oracle.OracleCellTree2d(xy, f, -1).intersect_edges(segs))


@pytest.mark.parametrize("n", [65535, 65536, 70001])
def test_spatial_order_of_large_batches(oracle, n, monkeypatch):
    import torch

    from numba_celltree_gb300 import CellTree2d, EdgeCellTree2d
    from numba_celltree_gb300.celltree_base import _GpuTree

    monkeypatch.setattr(_GpuTree, "ORDER_MIN_CELLS", 0)
    xy, f = syn.mixed_mesh(60, seed=5, extent=(60.0, 60.0))
    rng = np.random.default_rng(n)
    a = rng.uniform(-3.0, 63.0, (n, 2))
    segs = np.stack([a, a + rng.uniform(-2.0, 2.0, (n, 2))], 1)
    segs[::1000] = rng.uniform(-10.0, 70.0, (len(segs[::1000]), 2, 2))
    segs[7] = segs[7, :1]
    t = CellTree2d(xy, f, -1)
    _same(t.intersect_edges(torch.as_tensor(segs, device="cuda")),
          oracle.OracleCellTree2d(xy, f, -1).intersect_edges(segs))
    e = np.unique(np.sort(np.concatenate([f[:, [0, 1]], f[:, [1, 2]]]), axis=1), axis=0)
    _same(EdgeCellTree2d(xy, e).intersect_edges(torch.as_tensor(segs, device="cuda")),
          oracle.OracleEdgeCellTree2d(xy, e).intersect_edges(segs))
    # ranges of segments (counts come back in segment order)
    chunks = list(t.iter_intersect_edges(segs, max_candidates=20000))
    _same([np.concatenate([c[k] for c in chunks]) for k in range(3)],
          oracle.OracleCellTree2d(xy, f, -1).intersect_edges(segs))
    res = t._tree.locate_edges(torch.as_tensor(segs, device="cuda"), 1, budget=10)
    assert res is None
    assert torch.equal(t._tree.last_counts, t._tree.count_edge_candidates(torch.as_tensor(segs, device="cuda"), 1))
