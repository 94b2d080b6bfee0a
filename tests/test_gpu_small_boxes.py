"""Large batches of small boxes: by a thread each, with and without the scratch
and the spatial order, and the choice by their sizes; pairs and order against
the oracle."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh():
    return syn.mixed_mesh(40, 30, seed=61, extent=(40.0, 30.0))


def batch(n, side):
    rng = np.random.default_rng(n)
    c = rng.uniform(-1.0, 41.0, (n, 2))
    b = np.stack([c[:, 0], c[:, 0] + side, c[:, 1], c[:, 1] + side], 1)
    b[7] = [-1.0, 41.0, -1.0, 31.0]  # every cell
    b[8] = [np.nan, 5.0, 2.0, 5.0]
    b[9] = [-np.inf, np.inf, 10.0, 11.0]
    b[10] = [7.0, 5.0, 2.0, 5.0]  # inverted
    return b


@pytest.mark.parametrize("cells_per_leaf", [2, 40])
@pytest.mark.parametrize("n", [20, 70_001])
@pytest.mark.parametrize("scratch", [True, False])
@pytest.mark.parametrize("order", [None, True])
def test_thread_per_box(oracle, mesh, cells_per_leaf, n, scratch, order):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = mesh
    t = CellTree2d(xy, f, -1, 4, cells_per_leaf)._tree
    b = batch(n, 0.7)
    i, j = oracle.OracleCellTree2d(xy, f, -1, 4, cells_per_leaf).locate_boxes(b)
    if not scratch:
        t.SPEC_MAX_BYTES = 1
    t.SMALL_LOOK_MIN = 1
    for small, beside in ((None, 0.0), (None, 1.0), (True, 0.0)):
        t.box_sample = lambda _: (1.0, beside)
        gi, gj = t.locate_boxes(torch.as_tensor(b, device="cuda"), {"work_order": order}, small=small)
        assert np.array_equal(gi.cpu().numpy(), i) and np.array_equal(gj.cpu().numpy(), j)


@pytest.mark.parametrize("n,side,small", [((1 << 19) - 1, 0.5, False), (1 << 19, 0.5, True), (1 << 19, 9.0, False)])
def test_choice(mesh, monkeypatch, n, side, small):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = mesh
    t = CellTree2d(xy, f, -1)._tree
    b = torch.as_tensor(batch(n, side), device="cuda")
    seen = []
    inner = t._locate_boxes
    monkeypatch.setattr(t, "_locate_boxes", lambda *a: (seen.append((bool(a[3]), a[4])), inner(*a))[1])
    got = t.locate_boxes(b)
    assert seen == [(small, True)]
    want = t.locate_boxes(b, small=not small)
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    o = torch.argsort((b[:, 2] / 0.5).floor() * 100 + b[:, 0])  # beside one another
    t.locate_boxes(b[o].contiguous())
    assert seen[2] == (small, not small)


def test_sample(mesh):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = mesh
    t = CellTree2d(xy, f, -1)._tree
    W, H = xy.max(0) - xy.min(0)
    c = np.sqrt(W * H / len(f))
    for n in (11, 1024, 1025, 100_000):
        b = batch(n, 0.7)
        m = min(n, 1024)
        at = (n / m * np.arange(m)).astype(np.int64)
        s, d = b[at], b[np.minimum(at + 1, n - 1)]
        with np.errstate(invalid="ignore"):
            w, h = (np.clip(np.nan_to_num(s[:, k + 1] - s[:, k], nan=0.0), 0.0, e) for k, e in ((0, W), (2, H)))
            x, y = (np.abs((d[:, k] + d[:, k + 1] - s[:, k] - s[:, k + 1]) / 2) <= 16 * c for k in (0, 2))
        cells, beside = t.box_sample(torch.as_tensor(b, device="cuda"))
        want = ((w / c + 1) * (h / c + 1)).mean()
        # float32 terms of seven roundings and a sum of eleven levels
        assert abs(cells - want) <= 20 * 2.0**-24 * want
        assert abs(beside - (x & y).mean()) <= 2.0 / m  # one at the limit either way
