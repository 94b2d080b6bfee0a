"""Segments against single network edges, bit for bit with the oracle: proper
crossings, shared endpoints, collinear and parallel ones, edges touched within
the tolerance, and coordinates at both ends of float32's range."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1.0, 4.2e6), (1e-12, 0.0), (1e16, 0.0), (1e-25, 0.0)])
def test_segment_edges(oracle, scale, offset):
    from numba_celltree_gb300 import EdgeCellTree2d

    rng = np.random.default_rng(3)
    n = 150
    p = rng.uniform(0, 10, (n, 2))
    p[:60] = np.round(p[:60])  # lattice points: shared vertices, parallel and collinear edges
    q = p + rng.uniform(-2, 2, (n, 2))
    # no axis-parallel edges far from the origin: upstream builds no tree over some of their flat boxes
    steps = [[1, 1], [2, 1], [1, 2], [2, 2]] if offset else [[1, 0], [0, 1], [1, 1], [2, 0]]
    q[:60] = p[:60] + rng.choice(steps, 60)
    v = np.stack([p, q], 1).reshape(-1, 2)
    e = np.arange(2 * n).reshape(n, 2)
    m = 2000
    a, b = rng.uniform(-1, 11, (m, 2)), rng.uniform(-1, 11, (m, 2))
    k = rng.integers(0, n, m)
    s = slice(0, 250)
    a[s], b[s] = p[k[s]], q[k[s]]  # the edge itself
    s = slice(250, 500)
    a[s] = p[k[s]]  # from its vertex
    s = slice(500, 750)
    a[s] = p[k[s]] + rng.random((250, 1)) * (q - p)[k[s]]  # from a point on it
    s = slice(750, 1000)
    w = (q - p)[k[s]]
    a[s], b[s] = p[k[s]] - 0.3 * w, q[k[s]] + 0.2 * w  # along it
    s = slice(1000, 1250)  # along it at distances around the tolerance
    w = (q - p)[k[s]]
    off = np.stack([-w[:, 1], w[:, 0]], 1) * 10.0 ** rng.uniform(-14, -9, (250, 1))
    a[s], b[s] = p[k[s]] - 0.3 * w + off, q[k[s]] + off * rng.choice([-1, 1], (250, 1))
    s = slice(1250, 1400)
    b[s] = 2 * p[k[s]] - a[s]  # through its vertex
    b[1400:1500, 0] = a[1400:1500, 0]
    b[1500:1510] = a[1500:1510]
    segs = scale * (np.stack([a, b], 1) + offset)
    v = scale * (v + offset)
    ref = oracle.OracleEdgeCellTree2d(v, e).intersect_edges(segs)
    got = EdgeCellTree2d(v, e).intersect_edges(segs)
    for x, y in zip(got, ref):
        assert np.array_equal(x, y, equal_nan=True)
