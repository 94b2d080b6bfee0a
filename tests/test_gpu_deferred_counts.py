"""ct_locate_deferred_count reports the last float32 pass, whatever the
workspace held before: bytes of 0xff, or the counts of a larger batch."""

import ctypes

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bits", [(0, 0), (0, 16), (1, 0), (1000, 0), (32768, 0), (32769, 0), (65536, 0),
                                    (65537, 0), (1000, 16)])
@pytest.mark.parametrize("before", ["ff", "batch"])
def test_counts(n, bits, before):
    import torch

    from numba_celltree_gb300 import CellTree2d, _device, _lib

    lib = _lib.load()
    xy, f = syn.triangle_mesh(60, seed=21)
    tree = CellTree2d(xy, f, -1)
    t, tol = tree._tree, tree.default_tolerance()
    m = 100_000
    pts = syn.uniform_points(m, (0, 0), (1, 1), seed=22)
    pts[::10] = syn.near_edge_points(xy, f, m // 10, dist=1e-12, seed=23)
    p = torch.as_tensor(pts, device="cuda")
    out = torch.empty((m,), dtype=torch.int64, device="cuda")
    size = int(lib.ct_locate_workspace_size(m, 16))
    ws = torch.full((size,), 255, dtype=torch.uint8, device="cuda")
    P = _device.ptr

    def locate(k, b):
        _lib.check(lib.ct_locate_points_batched(ctypes.byref(t.desc), P(p), k, tol, b, P(out), P(ws), size,
                                                _device.stream()), "locate")

    def counts(k, b):
        c = (ctypes.c_int64 * 4)()
        _lib.check(lib.ct_locate_deferred_count(P(ws), k, b, c, _device.stream()), "counts")
        return list(c)

    if before == "batch":
        locate(m, bits)
        assert counts(m, bits)[3] >= m // 20  # points on edges are left open by the lists
    locate(n, bits)
    c = counts(n, bits)
    staged = n > 65536 or (bits and n)
    assert c[1] == c[2] == 0 and 0 <= c[0] <= c[3] <= n
    assert (c[3] >= n // 20) if staged else c == [0, 0, 0, 0]
    assert np.array_equal(out[:n].cpu().numpy(), tree.locate_points(pts[:n]))
