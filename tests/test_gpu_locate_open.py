"""Points the candidate lists leave open -- on and within the tolerance of edges
and vertices, inside several overlapping cells, off the mesh by less and more
than the tolerance, not finite -- against the oracle, by the one-launch form of
small batches and the staged form of large ones."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _mesh(name):
    if name == "tri":
        return syn.triangle_mesh(24, 17, seed=1, extent=(24.0, 17.0))
    if name == "utm":
        return syn.triangle_mesh(24, 17, seed=1, extent=(24.0, 17.0), offset=(5.0e5, 4.2e6))
    if name == "lattice":  # edges on the split planes and on each other's lines
        return syn.quad_mesh(24, 17, seed=1, extent=(24.0, 17.0), jitter=0.0)
    if name == "mixed":
        return syn.mixed_mesh(24, 17, seed=2, extent=(24.0, 17.0))
    xy, f = syn.quad_mesh(24, 17, seed=1, extent=(24.0, 17.0))  # overlapping: the mesh twice, shifted
    return np.concatenate([xy, xy + 0.37]), np.concatenate([f, f + len(xy)])


def _points(xy, f, n, rng, tol):
    lo, hi = xy.min(0), xy.max(0)
    p = lo + (hi - lo) * rng.uniform(-0.1, 1.1, (n, 2))
    m = n // 3
    g = f[rng.integers(0, len(f), m)]
    k = rng.integers(0, 3, m)
    a, b = xy[g[np.arange(m), k]], xy[g[np.arange(m), (k + 1) % 3]]
    t = rng.choice([0.0, 1.0, 0.5, -1e-13, 1.0 + 1e-13, 0.3], m) * (rng.random(m) < 0.7) + 0.0
    p[:m] = a + t[:, None] * (b - a) + rng.choice([0.0, 1.0], m)[:, None] * rng.uniform(-3, 3, (m, 2)) * tol
    c = slice(m, m + m // 4)  # around the bounding box
    side = rng.integers(0, 4, m // 4)
    p[c, 0] = np.where(side == 0, lo[0], np.where(side == 1, hi[0], p[c, 0]))
    p[c, 1] = np.where(side == 2, lo[1], np.where(side == 3, hi[1], p[c, 1]))
    p[c] += rng.choice([0.0, 0.5, 2.0, 1e6], m // 4)[:, None] * tol * rng.choice([-1, 1], (m // 4, 2))
    p[-6:] = [[np.nan, 1], [1, np.nan], [np.inf, 1], [1, -np.inf], [1e300, 1], [-1e30, -1e30]]
    return p


@pytest.mark.parametrize("name", ["tri", "utm", "lattice", "mixed", "twice"])
@pytest.mark.parametrize("cells_per_leaf", [1, 2, 9])
@pytest.mark.parametrize("tol", [None, 1e-9, 1e-3])
def test_open_points(oracle, name, cells_per_leaf, tol):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = _mesh(name)
    g, o = CellTree2d(xy, f, -1, 4, cells_per_leaf), oracle.OracleCellTree2d(xy, f, -1, 4, cells_per_leaf)
    assert g._tree.desc.bounds_finite == 3
    rng = np.random.default_rng(cells_per_leaf)
    width = g.default_tolerance() if tol is None else tol
    for n, bits in ((1, 0), (997, 0), (65536, 0), (65537, 0), (70001, 16)):
        p = _points(xy, f, max(n, 40), rng, width)[-n:] if n < 40 else _points(xy, f, n, rng, width)
        ref = o.locate_points(p, tol)
        pd = torch.as_tensor(np.ascontiguousarray(p), device="cuda")
        out = torch.full((len(p),), -7, dtype=torch.int64, device="cuda")
        g._tree.reset_error()
        g._tree.locate(pd, out, width, "fp32", sort_bits=bits)
        g._tree.raise_on_device_error()
        got = out.cpu().numpy()
        bad = np.nonzero(got != ref)[0]
        assert len(bad) == 0, (n, bits, len(bad), p[bad[:3]], got[bad[:3]], ref[bad[:3]])
