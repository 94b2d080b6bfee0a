"""Optional scratch of the box and segment queries: kept within a quarter of
the free memory, and not taken where the traversal does not use it; the results
stay the same."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

FREE = 320 << 20


def peak(fn):
    """fn's result and the most memory it held beyond what was held before."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out = fn()
    torch.cuda.synchronize()
    return out, torch.cuda.max_memory_allocated() - base


def small_device(monkeypatch):
    """A device with FREE bytes left and nothing cached."""
    import torch

    total = torch.cuda.mem_get_info()[1]
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (FREE, total))
    monkeypatch.setattr(torch.cuda, "memory_reserved", torch.cuda.memory_allocated)


@pytest.mark.parametrize("n", [40_000, 100_000])  # fewer records a box; none
def test_box_records(monkeypatch, n):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.quad_mesh(60, seed=41)
    t = CellTree2d(xy, f, -1)._tree
    b = torch.as_tensor(syn.random_boxes(n, (0, 0), (1, 1), 0.01, 0.03, seed=42), device="cuda")
    t.locate_boxes(b[:100])  # the box index
    want = t.locate_boxes(b)
    with monkeypatch.context() as m:
        small_device(m)
        got, most = peak(lambda: t.locate_boxes(b))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    # pairs, counts and offsets, order and scans, and the scratch
    assert most <= 16 * len(want[0]) + 64 * n + FREE // 4 + (4 << 20)


def test_no_box_records_for_deep_trees():
    import torch

    from numba_celltree_gb300 import CellTree2d
    from test_gpu_deep import nested_triangles

    xy, f = nested_triangles(200)
    t = CellTree2d(xy, f, -1, n_buckets=2, cells_per_leaf=1)._tree
    n = 50_000
    b = torch.as_tensor(syn.random_boxes(n, (0, 0), (1, 1), 0.01, 0.03, seed=43), device="cuda")
    t.locate_boxes(b[:100])
    got, most = peak(lambda: t.locate_boxes(b))
    assert most <= 16 * len(got[0]) + 64 * n + n * t.SPEC_CAP * 4 + (4 << 20)


def test_work_items(monkeypatch):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.quad_mesh(300, seed=44)
    t = CellTree2d(xy, f, -1)._tree
    rng = np.random.default_rng(45)
    s = torch.as_tensor(rng.uniform(0, 1, (8000, 2, 2)), device="cuda")
    cfg = {"split": 16}  # many items
    want = t.locate_edges(s, 1, cfg)
    cut = t.edge_cut(cfg, len(s))
    ni = t.edge_candidate_ranges(s, 1, None, cut)[3][2]
    assert ni * t.SEG_SPEC_CAP * 4 > FREE // 4  # the scratch would not fit
    taken = []
    empty = torch.empty
    with monkeypatch.context() as m:
        small_device(m)
        m.setattr(torch, "empty", lambda *a, **k: (taken.append(x := empty(*a, **k)), x)[1])
        got = t.locate_edges(s, 1, cfg)
    assert all(torch.equal(torch.nan_to_num(a), torch.nan_to_num(b)) for a, b in zip(got, want))
    spec = [x for x in taken if x.dtype == torch.int32 and x.ndim == 2]
    assert spec and all(x.numel() * 4 <= FREE // 4 for x in spec)
