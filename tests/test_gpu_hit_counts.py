"""Hits per segment at the edges of the counting kernel's groups: candidates
from none to past the eight-lane limit and the warp's steps, batches that end
within a warp's four segments, with and without another result order."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 33, 5000])
@pytest.mark.parametrize("ordered", [False, True])
def test_counts(n, ordered):
    import torch

    from numba_celltree_gb300 import _device, _lib

    lib, P = _lib.load(), _device.ptr
    rng = np.random.default_rng(n)
    m = rng.choice([0, 1, 7, 8, 9, 31, 255, 256, 257, 384, 385, 1000], n).astype(np.int64)
    off = np.concatenate([[0], np.cumsum(m)])
    keep = (rng.random(max(off[-1], 1)) < 0.6).astype(np.uint8) * 3
    order = rng.permutation(n).astype(np.int32)
    ref = np.zeros(n, dtype=np.int64)
    ref[order if ordered else np.arange(n)] = [np.count_nonzero(keep[off[i]:off[i + 1]]) for i in range(n)]
    d = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    kd, od, md, rd = d(keep), d(off[:-1]), d(m), d(order)
    counts, offsets = (torch.full((n,), -1, dtype=torch.int64, device="cuda") for _ in range(2))
    size = int(lib.ct_edge_hit_counts_workspace_size(n))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    total, most = ctypes.c_int64(-1), ctypes.c_int64(-1)
    _lib.check(lib.ct_edge_hit_counts(P(kd), P(od), P(md), P(rd) if ordered else None, n, P(counts), P(offsets), P(ws),
                                      size, ctypes.byref(total), ctypes.byref(most), _device.stream()), "counts")
    assert np.array_equal(counts.cpu().numpy(), ref)
    assert np.array_equal(offsets.cpu().numpy(), np.cumsum(ref) - ref)
    assert total.value == ref.sum() and most.value == ref.max()
