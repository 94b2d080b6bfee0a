"""Clip areas of single polygon pairs against the oracle, bit for bit: polygon
lengths on both sides of the shared-memory clip's limits, polygons whose
vertices lie on each other's edge lines, concave ones, and coordinates whose
products leave the normal float64 range."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _polygons(kind, n, k, rng):
    if kind == "convex":
        ang = np.sort(rng.uniform(0.0, 2 * np.pi, (n, k)), axis=1)
        rad = rng.uniform(0.2, 1.0, (n, 1))
        p = rad[:, :, None] * np.stack([np.cos(ang), np.sin(ang)], 2) + rng.uniform(-0.5, 0.5, (n, 1, 2))
    elif kind == "any":  # concave and self-crossing ones: any number of crossings
        p = rng.uniform(-1.0, 1.0, (n, k, 2))
    elif kind == "coarse":  # shared vertices, collinear and zero-length edges
        p = rng.integers(-2, 3, (n, k, 2)).astype(float)
    else:  # axis-parallel rectangles, extra vertices repeated
        a, b = rng.integers(-4, 4, (n, 2)) / 4.0, rng.integers(1, 6, (n, 2)) / 4.0
        c = np.stack([a, a + b * [1, 0], a + b, a + b * [0, 1]], 1)
        p = c[:, np.minimum(np.arange(k) * 4 // k, 3)] if k > 4 else c[:, :k]
    return p


def _areas(pa, pb):
    import torch

    from numba_celltree_gb300 import _lib

    n, ka, kb = len(pa), pa.shape[1], pb.shape[1]
    d = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    va, vb = d(pa.reshape(-1, 2)), d(pb.reshape(-1, 2))
    fa, fb = d(np.arange(n * ka).reshape(n, ka)), d(np.arange(n * kb).reshape(n, kb))
    i = d(np.arange(n))
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().ct_area_of_intersection(va.data_ptr(), fa.data_ptr(), ka, vb.data_ptr(), fb.data_ptr(), kb,
                                                   i.data_ptr(), i.data_ptr(), n, out.data_ptr(), err.data_ptr(), st))
    assert int(err.item()) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("kind", ["convex", "any", "coarse", "rect"])
@pytest.mark.parametrize("ka,kb", [(3, 3), (3, 4), (4, 3), (4, 4), (4, 6), (6, 5), (8, 8), (8, 9), (9, 3)])
def test_pair_areas(oracle, kind, ka, kb):
    rng = np.random.default_rng(ka * 100 + kb)
    n = 150
    pa, pb = _polygons(kind, n, ka, rng), _polygons(kind, n, kb, rng)
    moves = [(1.0, 0.0), (1.0, 4.2e6), (2.0**-520, 0.0), (2.0**-1040, 0.0), (2.0**300, 0.0), (1e-3, 1e12)]
    pa = np.concatenate([s * (pa + o) for s, o in moves])
    pb = np.concatenate([s * (pb + o) for s, o in moves])
    got = _areas(pa, pb)
    ref = np.array([oracle.polygon_polygon_clip_area(p, q) for p, q in zip(pa, pb)])
    assert np.array_equal(got, ref, equal_nan=True)


def test_non_finite_vertices(oracle):
    rng = np.random.default_rng(3)
    pa, pb = _polygons("convex", 60, 4, rng), _polygons("convex", 60, 3, rng)
    for k, bad in enumerate([np.nan, np.inf, -np.inf, 1e308, 1e200, 5e-324]):
        pa[10 * k: 10 * k + 5, k % 4, k % 2] = bad
        pb[10 * k + 5: 10 * k + 10, k % 3, k % 2] = bad
    ref = np.array([oracle.polygon_polygon_clip_area(p, q) for p, q in zip(pa, pb)])
    assert np.array_equal(_areas(pa, pb), ref, equal_nan=True)
