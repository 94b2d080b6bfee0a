"""The launch shapes of the box and segment traversals: `threads` reaches the
walks by warps, `work_order` is on, off or by the rule, an entry of a cache
file written when it meant the order by size is not read, and no shape changes
a result."""

import numpy as np
import pytest

from numba_celltree_gb300 import autotune as at
from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def tree():
    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.mixed_mesh(80, seed=81, extent=(80.0, 80.0))
    return CellTree2d(xy, f, -1)


@pytest.mark.parametrize("n", [1, 9, 5000, 70_000])
def test_threads(n):
    import torch

    t = tree()._tree
    b = torch.as_tensor(syn.random_boxes(n, (0, 0), (80, 80), 0.2, 9.0, seed=82), device="cuda")
    rng = np.random.default_rng(83)
    a = rng.uniform(0, 80, (n, 2))
    s = torch.as_tensor(np.stack([a, a + rng.uniform(-20, 20, (n, 2))], 1), device="cuda")
    for run in (lambda c: t.locate_boxes(b, c, small=False), lambda c: t.locate_edges(s, 1, c),
                lambda c: t.locate_edges(s, 1, dict(c, split=16))):
        base = run({})
        for threads in (64, 128, 256):
            for order in (False, True):
                got = run({"threads": threads, "work_order": order})
                assert all(torch.equal(torch.nan_to_num(x), torch.nan_to_num(y)) for x, y in zip(got, base))


def test_work_order():
    t = tree()._tree
    n = t.WORK_ORDER_MIN
    for cells, rule in ((t.ORDER_MIN_CELLS, True), (t.ORDER_MIN_CELLS - 1, False)):
        t.n = cells
        assert t.in_spatial_order(n, {}) is rule and t.in_spatial_order(n, {"work_order": None}) is rule
        assert t.in_spatial_order(n, {"work_order": True}) and not t.in_spatial_order(n, {"work_order": False})
        assert not t.in_spatial_order(n - 1, {}) and not t.in_spatial_order(0, {"work_order": True})


def test_old_entries_are_not_read(tmp_path, monkeypatch):
    monkeypatch.setenv(at.CACHE_ENV, str(tmp_path / "t.json"))
    at._cache = None
    t = tree()._tree
    for kind in ("boxes", "segments"):
        at.cache().put(at.cache_key(kind, t.gpu(), t.n, 70_000, K=t.K), {"config": {"threads": 64, "work_order": True}})
        assert t.cached(kind, 70_000) == at.DEFAULTS[kind]
        key = t.tune_key(kind, 70_000)
        at.cache().put(key, {"config": {"threads": 64, "work_order": False}})
        t._tuned.clear()
        assert t.cached(kind, 70_000) == dict(at.DEFAULTS[kind], threads=64, work_order=False)
