"""Entry points for C callers that the Python classes do not use: the four-call
form from segment candidates to results, against the classes' results, and the
work order by size."""

import ctypes

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 700, 40_000])
def test_edge_results_in_four_calls(mode, n):
    import torch

    from numba_celltree_gb300 import CellTree2d, EdgeCellTree2d, _device, _lib

    lib, P, st = _lib.load(), _device.ptr, _device.stream()
    xy, f = syn.mixed_mesh(40, seed=101, extent=(40.0, 40.0))
    edges = np.stack([f[:, 0], f[:, 1]], 1)
    t = (CellTree2d(xy, f, -1) if mode else EdgeCellTree2d(xy, edges))._tree
    rng = np.random.default_rng(102)
    a = rng.uniform(-1, 41, (n, 2))
    segs = torch.as_tensor(np.stack([a, a + rng.normal(0, 9.0, (n, 2))], 1), device="cuda")
    want = t.locate_edges(segs, mode)
    d = ctypes.byref(t.desc)
    new = lambda m, dtype=torch.int64: torch.full((max(m, 1),), -7, dtype=dtype, device="cuda")  # noqa: E731
    ccnt = new(n)
    _lib.check(lib.ct_count_edge_candidates(d, mode, P(segs), n, None, P(ccnt), st))
    coff, nc = t.scan(ccnt)
    cseg, cpos = new(nc, torch.int32), new(nc, torch.int32)
    _lib.check(lib.ct_write_edge_candidates(d, mode, P(segs), n, None, P(coff), P(cseg), P(cpos), st))
    keep, xyc = new(nc), torch.empty((max(nc, 1), 2, 2), dtype=torch.float64, device="cuda")
    _lib.check(lib.ct_test_edge_candidates(d, mode, P(segs), P(cseg), P(cpos), nc, P(keep), P(xyc), st))
    pos, total = t.scan(keep[:nc])
    assert total == len(want[0])
    ii, jj, j2 = new(total), new(total), new(total)
    p, p2 = (torch.empty((max(total, 1), 2, 2), dtype=torch.float64, device="cuda") for _ in range(2))
    off, cnt = new(n), new(n)
    _lib.check(lib.ct_compact_edge_hits(d, P(keep), P(pos), nc, P(cseg), P(cpos), P(xyc), P(coff), P(ccnt), n, P(ii),
                                        P(jj), P(p), P(off), P(cnt), st))
    size = int(lib.ct_sort_workspace_size(total))
    ws = new(size, torch.uint8)
    _lib.check(lib.ct_sort_intersections(P(segs), n, P(off), P(cnt), P(ii), P(jj), P(p), total, P(j2), P(p2), P(ws),
                                         size, st))
    assert torch.equal(ii[:total], want[0]) and torch.equal(j2[:total], want[1])
    assert torch.equal(torch.nan_to_num(p2[:total]), torch.nan_to_num(want[2]))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("n", [1, 5000, 70_000])
def test_work_order(kind, n):
    import torch

    from numba_celltree_gb300 import CellTree2d, _device, _lib

    lib, P, st = _lib.load(), _device.ptr, _device.stream()
    xy, f = syn.mixed_mesh(30, seed=103, extent=(30.0, 30.0))
    t = CellTree2d(xy, f, -1)._tree
    t.ensure_box_index()
    rng = np.random.default_rng(104)
    size = np.exp(rng.uniform(-3, 2, n))
    a = rng.uniform(0, 30, (n, 2))
    q = np.stack([a[:, 0], a[:, 0] + size, a[:, 1], a[:, 1] + size], 1) if kind == 0 else np.concatenate(
        [a, a + size[:, None]], 1)
    q_d = torch.as_tensor(q, device="cuda")
    nbytes = int(lib.ct_work_order_workspace_size(n))
    ws = torch.empty((nbytes,), dtype=torch.uint8, device="cuda")
    order = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    _lib.check(lib.ct_work_order(P(q_d), n, kind, 1.0, P(order), P(ws), nbytes, st))
    o = order.cpu().numpy()
    assert np.array_equal(np.sort(o), np.arange(n))
    # weight: area of the box widened by a cell, or length and a cell; classes of a quarter of an octave
    w = ((size + 1.0) ** 2 if kind == 0 else size * np.sqrt(2.0) + 1.0)[o]
    assert (np.maximum.accumulate(w) <= w * 2.0**0.25 * (1 + 1e-5)).all()
    counts = [torch.empty((n,), dtype=torch.int64, device="cuda") for _ in range(2)]
    for c, ord_d in zip(counts, (None, order)):
        call = lib.ct_count_boxes if kind == 0 else lib.ct_count_edge_candidates
        args = (P(q_d), n, P(ord_d), P(c), st)
        _lib.check(call(ctypes.byref(t.desc), *args) if kind == 0 else call(ctypes.byref(t.desc), 1, *args))
    assert torch.equal(*counts)
