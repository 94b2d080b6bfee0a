"""Box queries by warps: pairs and their order against the oracle for boxes from
smaller than a cell to the whole mesh, on trees with leaves of 1 to 40 cells,
for batches on both sides of the tasks-per-warp steps, in and out of spatial
order, with and without the box index, and by a thread per box."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells_per_leaf", [1, 2, 33, 40])
@pytest.mark.parametrize("n", [1, 7, 9729, 38913])
def test_boxes_of_every_size(oracle, cells_per_leaf, n):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.mixed_mesh(50, 40, seed=cells_per_leaf, extent=(50.0, 40.0))
    t = CellTree2d(xy, f, -1, 4, cells_per_leaf)._tree
    rng = np.random.default_rng(n)
    c = rng.uniform(-2.0, 52.0, (n, 2))
    s = np.exp(rng.uniform(np.log(0.05), np.log(6.0), (n, 2)))
    s[:: max(1, n // 20)] *= 12.0
    boxes = np.stack([c[:, 0], c[:, 0] + s[:, 0], c[:, 1], c[:, 1] + s[:, 1]], 1)
    boxes[0] = [-1.0, 51.0, -1.0, 41.0]  # every cell
    if n > 5:
        boxes[1] = [3.0, 3.0, 2.0, 5.0]  # no area
        boxes[2] = [7.0, 5.0, 2.0, 5.0]  # inverted
        boxes[3] = [np.nan, 5.0, 2.0, 5.0]
        boxes[4] = [-np.inf, np.inf, 10.0, 11.0]
    i, j = oracle.OracleCellTree2d(xy, f, -1, 4, cells_per_leaf).locate_boxes(boxes)
    bd = torch.as_tensor(boxes, device="cuda")
    for config, small, spec in (({}, False, True), ({"work_order": True}, False, True), ({}, True, True),
                                ({}, False, False), ({"work_order": True}, False, False)):
        t.SPEC_MAX_BOXES = type(t).SPEC_MAX_BOXES if spec else 0
        gi, gj = t.locate_boxes(bd, config, small=small)
        assert np.array_equal(gi.cpu().numpy(), i) and np.array_equal(gj.cpu().numpy(), j), (config, small, spec)
    nbx, t.desc.node_box = t.desc.node_box, None  # no box index: cells tested one by one
    import ctypes

    from numba_celltree_gb300 import _device, _lib

    counts = torch.empty(n, dtype=torch.int64, device="cuda")
    _lib.check(_lib.load().ct_count_boxes(ctypes.byref(t.desc), bd.data_ptr(), n, None, counts.data_ptr(),
                                          _device.stream()))
    t.desc.node_box = nbx
    assert np.array_equal(counts.cpu().numpy(), np.bincount(i, minlength=n))
