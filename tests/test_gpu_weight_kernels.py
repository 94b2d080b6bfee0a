"""Barycentric weights of the register kernels against the oracle, bit for bit:
face lengths on both sides of their limits, points on edges and vertices and
just off them, and coordinates whose products leave the normal float64 range."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [3, 4, 5, 8, 9])
@pytest.mark.parametrize("scale,offset", [(1.0, 0.0), (1.0, 4.2e6), (2.0**-500, 0.0), (2.0**-1040, 0.0), (2.0**340, 0.0)])
def test_weights_of_single_faces(oracle, K, scale, offset):
    import torch

    from numba_celltree_gb300 import _lib

    rng = np.random.default_rng(K)
    n = 400
    ang = np.sort(rng.uniform(0.0, 2 * np.pi, (n, K)), axis=1)
    poly = np.stack([np.cos(ang), np.sin(ang)], 2) * rng.uniform(0.3, 1.0, (n, 1, 1))
    t = rng.random((n, K))
    p = np.einsum("nk,nkd->nd", t / t.sum(1, keepdims=True), poly)
    k = rng.integers(0, K - 1, n)
    r, at = np.arange(n), rng.random(n)[:, None]
    on = poly[r, k] + at * (poly[r, k + 1] - poly[r, k])  # on an edge, off it by little, on a vertex
    p[:80] = on[:80]
    p[80:160] = on[80:160] + rng.uniform(-1, 1, (80, 2)) * 10.0 ** rng.uniform(-17, -9, (80, 1))
    p[160:200] = poly[r, k][160:200]
    poly, p = scale * (poly + offset), scale * (p + offset)
    lens = np.full(n, K)
    faces = np.arange(n * K).reshape(n, K)
    if K > 4:  # shorter faces padded with -1
        lens = rng.integers(3, K + 1, n)
        faces = np.where(np.arange(K) < lens[:, None], faces, -1)
    fi = np.where(rng.random(n) < 0.05, -1, r)
    tol = 1e-12 * scale * max(1.0, offset)
    d = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    v, f, pts, idx = d(poly.reshape(-1, 2)), d(faces), d(p), d(fi)
    out = torch.empty((n, K), dtype=torch.float64, device="cuda")
    desc = _lib.CtTree()
    desc.vertices, desc.elements, desc.n_max_vert = v.data_ptr(), f.data_ptr(), K
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().ct_barycentric_weights(ctypes.byref(desc), pts.data_ptr(), idx.data_ptr(), n, tol,
                                                  out.data_ptr(), st))
    L = oracle.lib()
    ref = np.empty((n, K))
    fn = L.cto_barycentric_wachspress if K > 3 else L.cto_barycentric_triangle
    args = [np.ascontiguousarray(x) for x in (p, fi, faces)]
    verts = np.ascontiguousarray(poly.reshape(-1, 2))
    ptr = [x.ctypes.data for x in args]
    if K > 3:
        fn(ptr[0], ptr[1], ptr[2], K, verts.ctypes.data, n, tol, ref.ctypes.data)
    else:
        fn(ptr[0], ptr[1], ptr[2], K, verts.ctypes.data, n, ref.ctypes.data)
    assert np.array_equal(out.cpu().numpy(), ref, equal_nan=True)
