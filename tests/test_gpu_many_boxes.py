"""A batch of more than 2^31 boxes: pairs carry the 64-bit box index."""

import ctypes

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def test_box_index_beyond_32_bits(oracle):
    import torch

    from numba_celltree_gb300 import CellTree2d, _device, _lib

    n = (1 << 31) + 5
    if torch.cuda.mem_get_info()[0] < 48 * n + (8 << 30):
        pytest.skip("not enough device memory")
    xy, f = syn.mixed_mesh(20, seed=31, extent=(20.0, 20.0))
    xy = xy + 100.0  # away from the boxes at the origin
    t = CellTree2d(xy, f, -1)._tree
    t.ensure_box_index()
    at = [0, (1 << 31) - 1, 1 << 31, n - 1]
    some = np.array([[101.0, 104.5, 102.0, 109.0], [99.0, 121.0, 99.0, 121.0], [105.0, 105.2, 105.0, 105.2],
                     [110.0, 117.0, 103.0, 104.0]])
    boxes = torch.zeros((n, 4), dtype=torch.float64, device="cuda")
    boxes[at] = torch.as_tensor(some, device="cuda")
    counts = t.count_boxes(boxes)
    wi, wj = oracle.OracleCellTree2d(xy, f, -1).locate_boxes(some)
    assert np.array_equal(counts[at].cpu().numpy(), np.bincount(wi, minlength=4))
    offsets, total = t.scan(counts)
    del counts
    assert total == len(wi)
    ii = torch.full((total,), -7, dtype=torch.int64, device="cuda")
    jj = torch.full((total,), -7, dtype=torch.int64, device="cuda")
    P = _device.ptr
    _lib.check(_lib.load().ct_write_boxes(ctypes.byref(t.desc), P(boxes), n, None, P(offsets), P(ii), P(jj),
                                          _device.stream()), "write_boxes")
    assert np.array_equal(ii.cpu().numpy(), np.array(at)[wi]) and np.array_equal(jj.cpu().numpy(), wj)
    del boxes, offsets
    torch.cuda.empty_cache()
