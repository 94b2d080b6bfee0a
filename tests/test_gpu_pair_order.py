"""Processing order of (box, face) pairs from the faces' lengths: a permutation
by the classes that the pairs' rows give, for every polygon length and around
the class limit (the order within a class is any)."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [3, 4, 8, 11, 13])
@pytest.mark.parametrize("n", [1, 255, 1000, 1_300_007])
def test_same_order(k, n):
    import torch

    from numba_celltree_gb300 import _device, _lib

    lib, P = _lib.load(), _device.ptr
    gen = torch.Generator("cuda").manual_seed(n + k)
    m = 257
    length = torch.randint(3, k + 1, (m, 1), device="cuda", generator=gen)
    faces = torch.where(torch.arange(k, device="cuda") < length, 7, -1)
    jb = torch.randint(0, m, (n,), device="cuda", generator=gen)
    ib = torch.zeros_like(jb)
    got = []
    for rows in (False, True):
        order = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        size = lib.ct_pair_order_workspace_size(n) if rows else lib.ct_box_pair_order_workspace_size(n, m)
        ws = torch.empty(int(size), dtype=torch.uint8, device="cuda")
        st = _device.stream()
        if rows:
            _lib.check(lib.ct_pair_order(None, 4, P(ib), P(faces), k, P(jb), n, P(order), P(ws), int(size), st), "order")
        else:
            _lib.check(lib.ct_box_pair_order(P(faces), k, m, P(jb), None, n, P(order), P(ws), int(size), st), "order")
        got.append(order)
    inside = (torch.rand(n, device="cuda", generator=gen) < 0.5).to(torch.uint8)
    order = torch.empty(n, dtype=torch.int32, device="cuda")
    size = int(lib.ct_box_pair_order_workspace_size(n, m))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    _lib.check(lib.ct_box_pair_order(P(faces), k, m, P(jb), P(inside), n, P(order), P(ws), size, _device.stream()), "order")
    classes = (length.flatten()[jb] - 3).clamp(max=7)
    halves = 2 * classes + inside
    assert torch.equal(halves[order.long()], torch.sort(halves).values)
    for order in got:
        assert torch.equal(torch.sort(order).values, torch.arange(n, dtype=torch.int32, device="cuda"))
        assert torch.equal(classes[order.long()], torch.sort(classes).values)
