"""Boxes around much of a mesh: whole subtrees written in parts, from the
counting pass's records, from the writing pass's when those did not fit, with
room for some of these or none, and from the job workspace; pairs and order
against the oracle, on leaves of fewer and more cells than a part."""

import ctypes

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

BOXES = np.array([[-1.0, 121.0, -1.0, 121.0], [2.3, 117.1, 3.1, 118.2], [60.2, 110.0, -3.0, 60.0],
                  [5.0, 5.4, 5.0, 5.4], [-9.0, -8.0, 0.0, 1.0], [10.0, 75.0, 10.0, 90.0]])


@pytest.fixture(scope="module", params=[1, 2, 40, 300, 20_000])
def case(request):
    import torch

    from numba_celltree_gb300 import CellTree2d
    from oracle import oracle as O

    O.build()
    xy, f = syn.triangle_mesh(120, seed=51, extent=(120.0, 120.0))
    t = CellTree2d(xy, f, -1, 4, request.param)._tree
    i, j = O.OracleCellTree2d(xy, f, -1, 4, request.param).locate_boxes(BOXES)
    return t, torch.as_tensor(BOXES, device="cuda"), i, j


def check(got, case):
    ii, jj = (x.cpu().numpy() for x in got[:2])
    assert np.array_equal(ii, case[2]) and np.array_equal(jj, case[3])


def test_tree(case):
    check(case[0].locate_boxes(case[1]), case)


@pytest.mark.parametrize("room", [1, 20, 100, 1000, 100_000])
def test_records(case, room):
    import torch

    from numba_celltree_gb300 import _device, _lib

    t, b, i, j = case
    lib, P, d, st = _lib.load(), _device.ptr, ctypes.byref(t.desc), _device.stream()
    n = len(BOXES)
    t.ensure_box_index()
    recs = torch.full((int(lib.ct_box_records_size(room)),), 255, dtype=torch.uint8, device="cuda")
    counts = torch.empty(n, dtype=torch.int64, device="cuda")
    _lib.check(lib.ct_count_boxes_records(d, P(b), n, None, P(counts), P(recs), room, st))
    offsets, total = t.scan(counts)
    assert total == len(i)
    for _ in range(2):  # the writing call may be repeated
        ii = torch.full((total,), -7, dtype=torch.int64, device="cuda")
        jj, inside = ii.clone(), torch.full((total,), 7, dtype=torch.uint8, device="cuda")
        _lib.check(lib.ct_write_boxes_records(d, P(b), n, None, P(offsets), P(recs), room, total, P(ii), P(jj),
                                              P(inside), st))
        check((ii, jj), case)
        assert (inside[ii == 0] == 1).all() and not inside[ii == 3].any()


@pytest.mark.parametrize("cells", [0, 8, 256, 400, 5000])
def test_jobs(case, cells):
    import torch

    from numba_celltree_gb300 import _device, _lib

    t, b, i, j = case
    lib, P, d, st = _lib.load(), _device.ptr, ctypes.byref(t.desc), _device.stream()
    n, cap = len(BOXES), 4
    counts = t.count_boxes(b)
    offsets, total = t.scan(counts)
    size = int(lib.ct_write_boxes_workspace_size(total, cells))
    ws = torch.full((size,), 255, dtype=torch.uint8, device="cuda")
    ii = torch.full((total,), -7, dtype=torch.int64, device="cuda")
    jj = ii.clone()
    _lib.check(lib.ct_write_boxes_ws(d, P(b), n, None, P(offsets), total, cells, P(ii), P(jj), P(ws), size, st))
    check((ii, jj), case)
    spec = torch.full((n, cap), -7, dtype=torch.int32, device="cuda")
    _lib.check(lib.ct_count_boxes_spec(d, P(b), n, None, P(counts), P(spec), cap, st))
    ii.fill_(-7), jj.fill_(-7), ws.fill_(255)
    _lib.check(lib.ct_write_boxes_spec(d, P(b), n, None, P(counts), P(offsets), P(spec), cap, total, cells, P(ii), P(jj),
                                       P(ws), size, st))
    check((ii, jj), case)
