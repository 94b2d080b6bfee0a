"""The differentiable intersect_faces at its edges: no overlapping pair, no
candidate pair, faces given as a CUDA or host tensor (which stays as it was),
and a batch of boxes past the room for records through the public calls."""

import numpy as np
import pytest

from numba_celltree_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def setup(shift):
    import torch

    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.quad_mesh(20, seed=91)
    qx, qf = syn.triangle_mesh(10, seed=92)
    tree = CellTree2d(xy, f, -1)
    v = torch.tensor(qx * 0.8 + shift, device="cuda", requires_grad=True)
    tv = torch.tensor(xy, device="cuda", requires_grad=True)
    return tree, v, qf, tv


@pytest.mark.parametrize("shift", [5.0, 1.0])  # away from the mesh; touching its corner at most
def test_no_overlap(shift):
    import torch

    from numba_celltree_gb300 import autodiff

    tree, v, qf, tv = setup(shift)
    i, j, a = autodiff.intersect_faces(tree, v, qf, tree_vertices=tv)
    assert len(i) == len(j) == len(a) == 0
    for t, g in zip((v, tv), torch.autograd.grad(a.sum(), [v, tv])):
        assert g.shape == t.shape and not g.any()


@pytest.mark.parametrize("where", ["cuda", "cpu", "int32", "fill"])
def test_faces_as_tensors(where):
    import torch

    from numba_celltree_gb300 import autodiff

    tree, v, qf, tv = setup(0.05)
    cw = qf[:, ::-1].copy()  # turned counter-clockwise on the way
    want = autodiff.intersect_faces(tree, v, cw, tree_vertices=tv)
    fill = -1
    f = torch.tensor(cw, device="cpu" if where == "cpu" else "cuda")
    if where == "int32":
        f = f.to(torch.int32)
    if where == "fill":
        fill = 99_999
        f = torch.cat([f, torch.full_like(f[:, :1], fill)], 1)
    before = f.clone()
    got = autodiff.intersect_faces(tree, v, f, fill, tree_vertices=tv)
    assert torch.equal(f, before)
    assert all(torch.equal(x, y) for x, y in zip(got, want))


def test_boxes_past_the_records(oracle):
    from numba_celltree_gb300 import CellTree2d

    xy, f = syn.mixed_mesh(40, seed=93, extent=(40.0, 40.0))
    tree, o = CellTree2d(xy, f, -1), oracle.OracleCellTree2d(xy, f, -1)
    tree._tree.BOX_RECORDS = tree._tree.BOX_RECORDS_MIN = tree._tree.BOX_RECORDS_BOXES = 1
    b = syn.random_boxes(3000, (0, 0), (40, 40), 0.3, 12.0, seed=94)
    for got, want in ((tree.locate_boxes(b), o.locate_boxes(b)), (tree.intersect_boxes(b), o.intersect_boxes(b))):
        assert all(np.array_equal(x, y) for x, y in zip(got, want))
