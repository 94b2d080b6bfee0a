"""Faces that repeat a vertex -- closed rings (the first vertex again at the
end), a vertex twice in a row -- in the candidate lists of the batched locate:
same answers as the oracle, for trees built alone and in a batch."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

FORMS = {
    "closed": lambda t: np.stack([t[:, 0], t[:, 1], t[:, 2], t[:, 0]], 1),
    "closed_cw": lambda t: np.stack([t[:, 2], t[:, 1], t[:, 0], t[:, 2]], 1),
    "last_twice": lambda t: np.stack([t[:, 0], t[:, 1], t[:, 2], t[:, 2]], 1),
    "first_twice": lambda t: np.stack([t[:, 0], t[:, 0], t[:, 1], t[:, 2]], 1),
    "closed_k6": lambda t: np.stack([t[:, 0], t[:, 1], t[:, 2], t[:, 0], t[:, 0] * 0 - 1, t[:, 0] * 0 - 1], 1),
}


def inputs(form, offset):
    xy, t = syn.triangle_mesh(40, seed=11, extent=(40.0, 40.0), offset=offset)
    pts = syn.uniform_points(70_000, xy.min(0), xy.max(0), seed=12, margin=0.02)
    pts[::50] = syn.near_edge_points(xy, t, len(pts[::50]), dist=1e-9, seed=13)
    return xy, FORMS[form](t), pts


@pytest.mark.parametrize("n", [1000, 40_000, 70_000])  # a warp a point, a lane a point, sorted
@pytest.mark.parametrize("offset", [(0.0, 0.0), (5.0e5, 4.2e6)])
@pytest.mark.parametrize("form", FORMS)
def test_locate(oracle, form, offset, n):
    from numba_celltree_gb300 import CellTree2d

    xy, f, pts = inputs(form, offset)
    want = oracle.OracleCellTree2d(xy, f, -1).locate_points(pts[:n])
    assert np.array_equal(CellTree2d(xy, f, -1).locate_points(pts[:n]), want)


@pytest.mark.parametrize("form", FORMS)
def test_batch(oracle, form):
    from numba_celltree_gb300.batch import CellTreeBatch

    xy, f, pts = inputs(form, (0.0, 0.0))
    x2, f2 = syn.quad_mesh(20, seed=14)
    p2 = syn.uniform_points(3000, (0, 0), (1, 1), seed=15)
    got = CellTreeBatch([(xy, f), (x2, f2)]).locate_points([pts[:5000], p2])
    for g, (v, e, p) in zip(got, ((xy, f, pts[:5000]), (x2, f2, p2))):
        g = g.cpu().numpy() if hasattr(g, "cpu") else np.asarray(g)
        assert np.array_equal(g, oracle.OracleCellTree2d(v, e, -1).locate_points(p))


@pytest.mark.parametrize("form", FORMS)
def test_weights(oracle, form):
    from numba_celltree_gb300 import CellTree2d

    xy, f, pts = inputs(form, (0.0, 0.0))
    wi, ww = oracle.OracleCellTree2d(xy, f, -1).compute_barycentric_weights(pts[:5000])
    gi, gw = CellTree2d(xy, f, -1).compute_barycentric_weights(pts[:5000])
    assert np.array_equal(gi, wi) and np.array_equal(gw, ww, equal_nan=True)
