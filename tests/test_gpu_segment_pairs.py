"""Segments against single cells, bit for bit with the oracle: cell lengths on
both sides of the float32 path's limits, segments that end on edges and
vertices, run along edges, lie inside a cell or have no length, and
coordinates at both ends of float32's range."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cells(K, n, rng, kind):
    """n x n separate cells of 3..K vertices, one per unit square."""
    verts, faces = [], []
    for i in range(n):
        for j in range(n):
            k = int(rng.integers(3, K + 1)) if K > 3 else 3
            if kind == "round":
                ang = np.sort(rng.uniform(0, 2 * np.pi, k))
                p = 0.5 + 0.45 * np.stack([np.cos(ang), np.sin(ang)], 1)
            else:  # vertices on a coarse lattice: axis-parallel and repeated ones
                p = rng.integers(0, 4, (k, 2)) / 4.0
                p[0], p[2] = 0.0, 0.75  # no cell of zero width: upstream builds no tree over some of those
            faces.append(list(range(len(verts), len(verts) + k)) + [-1] * (K - k))
            verts.extend(p + [i, j])
    return np.array(verts), np.array(faces)


def _segments(v, f, n, rng):
    a, b = rng.uniform(-1, 9, (n, 2)), rng.uniform(-1, 9, (n, 2))
    m = n // 8
    b[:m] = a[:m] + rng.uniform(-0.3, 0.3, (m, 2))  # short
    pick = f[rng.integers(0, len(f), n)]
    p, q = v[pick[:, 0]], v[pick[:, 1]]
    s = slice(m, 2 * m)
    a[s] = p[s]  # from a vertex
    s = slice(2 * m, 3 * m)
    a[s], b[s] = p[s], q[s]  # an edge itself
    s = slice(3 * m, 4 * m)
    a[s], b[s] = p[s] - (q[s] - p[s]), q[s] + (q[s] - p[s])  # along an edge
    s = slice(4 * m, 5 * m)
    a[s] = p[s] + rng.random((m, 1)) * (q[s] - p[s])  # from an edge
    s = slice(5 * m, 6 * m)
    b[s] = p[s] * 2 - a[s]  # through a vertex
    a[6 * m:7 * m, 1] = b[6 * m:7 * m, 1]  # parallel to an axis
    b[7 * m:7 * m + 5] = a[7 * m:7 * m + 5]  # no length
    return np.stack([a, b], 1)


@pytest.mark.parametrize("kind", ["round", "coarse"])
@pytest.mark.parametrize("K", [3, 4, 8, 9])
@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1.0, 4.2e6), (1e-12, 0.0), (1e16, 0.0)])
def test_segment_cells(oracle, kind, K, scale, offset):
    from numba_celltree_gb300 import CellTree2d

    rng = np.random.default_rng(10 * K + len(kind))
    v, f = _cells(K, 8, rng, kind)
    segs = _segments(v, f, 1600, rng)
    v, segs = scale * (v + offset), scale * (segs + offset)
    ref = oracle.OracleCellTree2d(v, f, -1).intersect_edges(segs)
    got = CellTree2d(v, f, -1).intersect_edges(segs)
    for x, y in zip(got, ref):
        assert np.array_equal(x, y, equal_nan=True)
