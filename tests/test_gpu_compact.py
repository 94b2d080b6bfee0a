"""Compaction of pairs at the edges of its tiles (2048 pairs) and of the number
of tiles whose counts are summed without a scan (1024), by area and by flag."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 31, 33, 2047, 2048, 2049, 5000, 2048 * 1024, 2048 * 1024 + 1, 2048 * 3000 + 7])
@pytest.mark.parametrize("by", ["area", "flag"])
@pytest.mark.parametrize("share", [0.0, 0.3, 1.0])
def test_kept_pairs(n, by, share):
    import torch

    from numba_celltree_gb300 import _device, _lib

    lib = _lib.load()
    gen = torch.Generator("cuda").manual_seed(n)
    rnd = lambda: torch.rand(n, device="cuda", dtype=torch.float64, generator=gen)
    keep = rnd() < share
    i, j = torch.arange(n, device="cuda"), torch.arange(n, device="cuda") * 7 - 3
    area = torch.where(keep, rnd() + 0.1, torch.where(rnd() < 0.5, -rnd(), torch.zeros_like(rnd())))
    area[~keep & (rnd() < 0.1)] = float("nan")
    flag = keep.to(torch.uint8) * 5
    out_i, out_j, out_a = torch.full_like(i, -9), torch.full_like(j, -9), torch.full_like(area, -9.0)
    ws = torch.empty(int(lib.ct_compact_workspace_size(n)), dtype=torch.uint8, device="cuda")
    total = ctypes.c_int64(-1)
    P = _device.ptr
    a = by == "area"
    _lib.check(lib.ct_compact_pairs(P(area) if a else None, None if a else P(flag), n, P(i), P(j), P(out_i), P(out_j),
                                    P(out_a) if a else None, P(ws), ws.numel(), ctypes.byref(total),
                                    _device.stream()), "compact")
    m = int(total.value)
    assert m == int(keep.sum())
    assert torch.equal(out_i[:m], i[keep]) and torch.equal(out_j[:m], j[keep])
    assert not a or torch.equal(out_a[:m], area[keep])
    assert (out_i[m:] == -9).all() and (out_j[m:] == -9).all()
