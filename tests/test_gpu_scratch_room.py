"""Optional scratch of the box and segment queries: left out where the device
has no room for it, and not taken where the traversal does not use it; the
results stay the same."""

import contextlib

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def room(nbytes):
    """This process may hold nbytes more than it holds now."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.mem_get_info()[1]
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + nbytes) / total)
    try:
        yield
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


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


def test_box_records():
    import torch

    from numba_celltree_gb300 import CellTree2d

    n = 100_000
    xy, f = syn.quad_mesh(60, seed=41)
    t = CellTree2d(xy, f, -1)._tree
    b = torch.as_tensor(syn.random_boxes(n, (0, 0), (1, 1), 0.01, 0.03, seed=42), device="cuda")
    want = t.locate_boxes(b)
    assert t.box_records(n, False) * 16 > 300 << 20
    with room(200 << 20):
        got = t.locate_boxes(b)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


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


def test_work_items():
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.quad_mesh(300, seed=44)
    t = CellTree2d(xy, f, -1)._tree
    rng = np.random.default_rng(45)
    s = torch.as_tensor(rng.uniform(0, 1, (4000, 2, 2)), device="cuda")
    cfg = {"split": 1}  # an item for about every candidate
    want = t.locate_edges(s, 1, cfg)
    ni = t.edge_candidate_ranges(s, 1, None, t.edge_cut(cfg, 4000))[3][2]
    assert ni * t.SEG_SPEC_CAP * 4 > 300 << 20
    with room(200 << 20):
        got = t.locate_edges(s, 1, cfg)
    assert all(torch.equal(torch.nan_to_num(a), torch.nan_to_num(b)) for a, b in zip(got, want))
