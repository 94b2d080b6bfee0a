"""Box pairs from the counting pass's records: against the oracle's pairs and
order, with room for all records, for few and for one (the boxes are then
walked again), on leaves of 1 to 40 cells."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells_per_leaf", [1, 2, 33, 40])
@pytest.mark.parametrize("n,room", [(1, 4096), (33, 4096), (33, 8), (2000, 4096), (2000, 1)])
def test_records(oracle, cells_per_leaf, n, room):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.mixed_mesh(50, 40, seed=cells_per_leaf, extent=(50.0, 40.0))
    t = CellTree2d(xy, f, -1, 4, cells_per_leaf)._tree
    rng = np.random.default_rng(n)
    c, s = rng.uniform(-2.0, 52.0, (n, 2)), np.exp(rng.uniform(np.log(0.05), np.log(30.0), (n, 2)))
    boxes = np.stack([c[:, 0], c[:, 0] + s[:, 0], c[:, 1], c[:, 1] + s[:, 1]], 1)
    boxes[0] = [-1.0, 51.0, -1.0, 41.0]  # every cell
    if n > 5:
        boxes[1:5] = [[3.0, 3.0, 2.0, 5.0], [7.0, 5.0, 2.0, 5.0], [np.nan, 5.0, 2.0, 5.0], [-np.inf, np.inf, 10.0, 11.0]]
    i, j = oracle.OracleCellTree2d(xy, f, -1, 4, cells_per_leaf).locate_boxes(boxes)
    t.BOX_RECORDS, t.BOX_RECORDS_MIN, t.lengths_once = room, 1, lambda *_: True
    gi, gj, inside = (x.cpu().numpy() for x in t.locate_boxes(torch.as_tensor(boxes, device="cuda"), inside=True))
    assert np.array_equal(gi, i) and np.array_equal(gj, j)
    bb, flag = t.bb_coords.cpu().numpy()[gj], inside.astype(bool)
    b = boxes[gi]
    assert np.isin(inside, (0, 1)).all() and flag[gi == 0].all()
    held = (b[:, 0] < bb[:, 0]) & (bb[:, 1] < b[:, 1]) & (b[:, 2] < bb[:, 2]) & (bb[:, 3] < b[:, 3])
    assert held[flag].all()
