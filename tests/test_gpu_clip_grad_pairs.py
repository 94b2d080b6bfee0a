"""The two kernels of the clip area's gradient against each other: the edge
integrals of polygons of up to 8 vertices and the tape, which faces padded to 9
columns take.  Polygons on each other's edge lines, concave ones and repeated
vertices included, where the subgradient must be the tape's."""

import numpy as np
import pytest

from test_gpu_clip_pairs import _polygons

pytestmark = pytest.mark.gpu


def _grad(pa, pb, g, pad):
    import torch

    from numba_celltree_gb300 import _device, _lib

    n, ka, kb = len(pa), pa.shape[1], pb.shape[1]
    d = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    fa, fb = np.arange(n * ka).reshape(n, ka), np.arange(n * kb).reshape(n, kb)
    fa = np.concatenate([fa, np.full((n, max(0, pad - ka)), -1)], 1)
    fb = np.concatenate([fb, np.full((n, max(0, pad - kb)), -1)], 1)
    va, vb, fa, fb, i, gd = d(pa.reshape(-1, 2)), d(pb.reshape(-1, 2)), d(fa), d(fb), d(np.arange(n)), d(g)
    ga, gb = torch.zeros_like(va), torch.zeros_like(vb)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    P = _device.ptr
    _lib.check(_lib.load().ct_area_of_intersection_grad(P(va), P(fa), fa.shape[1], P(vb), P(fb), fb.shape[1], P(i), P(i),
                                                        n, P(gd), P(ga), P(gb), P(err), _device.stream()))
    assert int(err.item()) == 0
    return ga.cpu().numpy().reshape(n, -1), gb.cpu().numpy().reshape(n, -1)


@pytest.mark.parametrize("kind", ["convex", "any", "coarse", "rect"])
@pytest.mark.parametrize("ka,kb", [(3, 3), (3, 4), (4, 4), (5, 6), (8, 8)])
def test_edge_integrals_equal_the_tape(kind, ka, kb):
    rng = np.random.default_rng(ka * 100 + kb)
    n = 600
    pa, pb = _polygons(kind, n, ka, rng), _polygons(kind, n, kb, rng)
    if kind == "convex":
        pa[::2] = pa[::2, ::-1]  # clockwise subjects
        pa[300:] += 4.2e6
        pb[300:] += 4.2e6
    g = rng.normal(size=n)
    g[:10] = 0.0
    small, tape = _grad(pa, pb, g, 0), _grad(pa, pb, g, 9)
    for x, y in zip(small, tape):
        # entries are lengths (a few units) times g, from coordinates rounded
        # to 2^-53 of 4.2e6 (5e-10) and lines that cross at angles of 1e-3 and more
        assert np.allclose(x, y, rtol=0.0, atol=2e-9 if kind != "convex" else 2e-6)
        far = slice(None, 300) if kind == "convex" else slice(None)
        assert np.allclose(x[far], y[far], rtol=0.0, atol=2e-9)
