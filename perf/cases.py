"""The work a program has this package do, as cases whose speed is measured.

Every case is one call sequence of the public classes on GPU tensors: point
location, tree construction, zonal statistics over boxes, cross-sections,
regridding, its adjoint, interpolation weights, and cross-sections of an edge
network.  Meshes are jittered lattices (triangles, quads, or a mix of 3- to
6-gons), made on the GPU from a seed.  Where the number of results depends on
the geometry, a seed poses one geometry (mirrored, axes swapped) and orders
its queries and draws its values anew, so that every seed has as many results.
`exact` gives computed outputs from the lattice itself, in float64, without a
tree.
"""

import math

import numpy as np
import torch

from numba_celltree_gb300 import CellTree2d, EdgeCellTree2d, autodiff
from numba_celltree_gb300.regrid import WeightMatrix

DEVICE = "cuda"
JITTER = 0.2  # of a cell width: every quad stays convex
UTM = (5.0e5, 4.2e6)
CHUNK = 1 << 22  # rows per step of the float64 evaluations


def listed():
    return [
        # a map click or a model probe: a handful of points, once per event
        {"name": "locate_1k", "kind": "locate", "mesh": "tri", "nx": 200, "ny": 200, "h": 0.005, "utm": False,
         "points": 1000},
        # particle tracking / raster sampling on a national grid, in projected coordinates
        {"name": "locate_268m", "kind": "locate", "mesh": "tri", "nx": 4000, "ny": 2000, "h": 1.0, "utm": True,
         "points": 268435456},
        # a tree made for one model grid, then one point per cell located in it
        {"name": "build_80k", "kind": "build", "mesh": "tri", "nx": 200, "ny": 200, "h": 0.005, "utm": False,
         "points": 80000},
        {"name": "build_16m", "kind": "build", "mesh": "tri", "nx": 4000, "ny": 2000, "h": 1.0, "utm": True,
         "points": 16000000},
        # zonal means over a few small windows of a grid
        {"name": "zonal_10k", "kind": "zonal", "mesh": "tri", "nx": 200, "ny": 200, "h": 0.005, "boxes": 10000,
         "side_lo": 0.2, "side_hi": 4.0},
        # zonal means over windows of very different sizes on a mixed mesh
        {"name": "zonal_250k", "kind": "zonal", "mesh": "mixed", "nx": 2000, "ny": 2000, "h": 0.5, "boxes": 250000,
         "side_lo": 0.2, "side_hi": 100.0},
        # a million line pieces (tracks, rivers) cut by a mixed mesh
        {"name": "segments_1m", "kind": "segments", "mesh": "mixed", "nx": 2000, "ny": 2000, "h": 0.5,
         "segments": 1000000, "reach": 40.0},
        # cross-sections through the whole model
        {"name": "sections_1k", "kind": "segments", "mesh": "mixed", "nx": 2000, "ny": 2000, "h": 0.5,
         "segments": 1000, "reach": 0.0},
        # conservative regridding between two unrelated meshes
        {"name": "regrid_1m", "kind": "regrid", "nx": 1000, "ny": 500, "qnx": 1000, "qny": 500, "h": 0.1},
        # the same overlap areas inside an optimisation: forward and backward
        {"name": "adjoint_250k", "kind": "adjoint", "nx": 500, "ny": 250, "qnx": 500, "qny": 250, "h": 0.1},
        # interpolation weights of a million points in a rotated quad grid
        {"name": "weights_1m", "kind": "weights", "nx": 1000, "ny": 500, "h": 0.1, "points": 1000000},
        # a channel network cut by cross-sections
        {"name": "network_100k", "kind": "network", "nx": 500, "ny": 500, "h": 1.0, "segments": 100000,
         "reach": 20.0},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def lattice(lo, hi):
        n = size(lo, hi)
        nx = max(2, int(math.sqrt(n * rng.uniform(0.5, 2.0))))
        return {"nx": nx, "ny": max(2, n // nx)}

    kind = rng.choice(["locate", "locate", "build", "zonal", "segments", "regrid", "adjoint", "weights", "network"])
    mesh = rng.choice(["tri", "quad", "mixed"])
    if kind == "locate":
        return {"kind": kind, "mesh": mesh, **lattice(2e3, 4e6), "h": 1.0, "utm": rng.random() < 0.5,
                "points": size(1e3, 6e7)}
    if kind == "build":
        grid = lattice(2e3, 4e6)
        return {"kind": kind, "mesh": mesh, **grid, "h": 1.0, "utm": rng.random() < 0.5,
                "points": grid["nx"] * grid["ny"]}
    if kind == "zonal":
        return {"kind": kind, "mesh": mesh, **lattice(4e4, 4e6), "h": 0.5, "boxes": size(1e3, 2e5), "side_lo": 0.2,
                "side_hi": rng.choice([4.0, 20.0, 80.0])}
    if kind == "segments":
        grid = lattice(4e4, 4e6)
        if rng.random() < 0.5:
            return {"kind": kind, "mesh": mesh, **grid, "h": 0.5, "segments": size(1e3, 9e5), "reach": 40.0}
        return {"kind": kind, "mesh": mesh, **grid, "h": 0.5, "segments": size(50, 1e3), "reach": 0.0}
    if kind in ("regrid", "adjoint"):
        top = 4.5e5 if kind == "regrid" else 1.2e5
        q = lattice(2e3, top)
        return {"kind": kind, **lattice(2e3, top), "qnx": q["nx"], "qny": q["ny"], "h": 0.1}
    if kind == "weights":
        return {"kind": kind, **lattice(2e3, 5e5), "h": 0.1, "points": size(1e3, 4e6)}
    return {"kind": kind, **lattice(2e3, 2.5e5), "h": 1.0, "segments": size(1e3, 9e4), "reach": 20.0}


# -- meshes -------------------------------------------------------------------


def _rng(seed, stream):
    return torch.Generator(DEVICE).manual_seed(int(seed) * 64 + stream)


def _rand(shape, gen):
    return torch.rand(shape, dtype=torch.float64, device=DEVICE, generator=gen)


def _pose(xy, seed):
    """xy (..., 2) mirrored and its axes swapped as the seed says (no rounding)."""
    sign = torch.tensor([-1.0 if seed & 1 else 1.0, -1.0 if seed & 2 else 1.0], dtype=torch.float64, device=DEVICE)
    return ((xy * sign).flip(-1) if seed & 4 else xy * sign).contiguous()


def _lattice(nx, ny, h, gen):
    """Jittered lattice vertices in units of length and its quads (row-major)."""
    i = torch.arange(nx + 1, device=DEVICE, dtype=torch.float64).repeat(ny + 1)
    j = torch.arange(ny + 1, device=DEVICE, dtype=torch.float64).repeat_interleave(nx + 1)
    inner = (i > 0) & (i < nx) & (j > 0) & (j < ny)
    u = (2.0 * _rand((i.shape[0], 2), gen) - 1.0) * JITTER * inner[:, None]
    xy = (torch.stack([i, j], 1) + u) * h
    qi = torch.arange(nx, device=DEVICE).repeat(ny)
    qj = torch.arange(ny, device=DEVICE).repeat_interleave(nx)
    v0 = qj * (nx + 1) + qi
    return xy, torch.stack([v0, v0 + 1, v0 + nx + 2, v0 + nx + 1], 1)


def _convex(p):
    """Whether polygons p (m, k, 2) turn left or go straight at every corner."""
    d = p.roll(-1, 1) - p
    e = d.roll(-1, 1)
    return (d[..., 0] * e[..., 1] - d[..., 1] * e[..., 0] >= 0).all(1)


def _mesh(kind, nx, ny, h, gen):
    """(vertices, faces, cover): cover (n_quads, 2) is the face that holds each
    quad's triangles (0, 1, 2) and (0, 2, 3)."""
    xy, q = _lattice(nx, ny, h, gen)
    n = q.shape[0]
    ids = torch.arange(n, device=DEVICE)
    if kind == "quad":
        return xy, q, torch.stack([ids, ids], 1)
    if kind == "tri":
        f = torch.stack([q[:, [0, 1, 2]], q[:, [0, 2, 3]]], 1).reshape(-1, 3)
        return xy, f, torch.stack([2 * ids, 2 * ids + 1], 1)
    # mixed: a fifth of the quads merged in pairs into a convex hexagon or a
    # pentagon and a triangle, a third of the rest split, the others whole
    left = (ids % nx % 2 == 0) & (ids % nx + 1 < nx)
    roll = _rand((n,), gen)
    a = ids[left & (roll < 0.2)]
    fill = -1
    hexa = torch.stack([q[a, 0], q[a, 1], q[a + 1, 1], q[a + 1, 2], q[a, 2], q[a, 3]], 1)
    penta = hexa[:, :5]
    want = roll[a] < 0.1
    as_p = want & _convex(xy[penta])
    as_h = ~as_p & _convex(xy[hexa])
    pa, ha = a[as_p], a[as_h]
    used = torch.zeros(n, dtype=torch.bool, device=DEVICE)
    for m in (pa, ha):
        used[m] = True
        used[m + 1] = True
    rest = ids[~used]
    split = _rand((n,), gen)[rest] < 0.3
    s, w = rest[split], rest[~split]
    cover = torch.empty((n, 2), dtype=torch.int64, device=DEVICE)
    parts, base = [], 0

    def add(rows):
        nonlocal base
        pad = torch.full((rows.shape[0], 6 - rows.shape[1]), fill, dtype=torch.int64, device=DEVICE)
        parts.append(torch.cat([rows, pad], 1))
        base += rows.shape[0]
        return torch.arange(base - rows.shape[0], base, device=DEVICE)

    k = add(hexa[as_h])
    cover[ha] = k[:, None]
    cover[ha + 1] = k[:, None]
    k = add(penta[as_p])
    cover[pa, 0] = k
    cover[pa + 1] = k[:, None]
    cover[pa, 1] = add(q[pa][:, [0, 2, 3]])
    cover[w] = add(q[w])[:, None]
    cover[s, 0] = add(q[s][:, [0, 1, 2]])
    cover[s, 1] = add(q[s][:, [0, 2, 3]])
    order = torch.randperm(base, device=DEVICE, generator=gen)
    place = torch.empty_like(order)
    place[order] = torch.arange(base, device=DEVICE)
    return xy, torch.cat(parts)[order], place[cover]


def _edges(nx, ny):
    """The lattice's horizontal and vertical edges as a network."""
    v = torch.arange((nx + 1) * (ny + 1), device=DEVICE).reshape(ny + 1, nx + 1)
    return torch.cat([torch.stack([v[:, :-1], v[:, 1:]], 2).reshape(-1, 2),
                      torch.stack([v[:-1], v[1:]], 2).reshape(-1, 2)])


TURN = math.radians(7.0)


def _turned(xy, nx, ny, h, back=False):
    """Rotated by 7 degrees about the lattice's centre and shifted by 0.37 cell."""
    c, s = math.cos(TURN), math.sin(TURN)
    mid = torch.tensor([0.5 * nx * h, 0.5 * ny * h], dtype=torch.float64, device=DEVICE)
    if back:
        d = xy - 0.37 * h - mid
        return torch.stack([c * d[..., 0] + s * d[..., 1], -s * d[..., 0] + c * d[..., 1]], -1) + mid
    d = xy - mid
    return torch.stack([c * d[..., 0] - s * d[..., 1], s * d[..., 0] + c * d[..., 1]], -1) + mid + 0.37 * h


# -- inputs -------------------------------------------------------------------


def _points(case, xy, faces, gen):
    """99 of 100 points uniform in the mesh's box widened by a hundredth, one
    within 1e-9 of a vertex or an edge (grid nodes and faces sampled in place)."""
    n = int(case["points"])
    lo, hi = xy.amin(0), xy.amax(0)
    p = lo + (hi - lo) * (1.02 * _rand((n, 2), gen) - 0.01)
    near = p[::100]
    m = near.shape[0]
    f = torch.randint(0, faces.shape[0], (m,), device=DEVICE, generator=gen)
    k = torch.randint(0, 3, (m,), device=DEVICE, generator=gen)
    a, b = xy[faces[f, k]], xy[faces[f, (k + 1) % 3]]
    t = _rand((m,), gen)
    t = torch.where(_rand((m,), gen) < 0.2, torch.zeros_like(t), t)
    near.copy_(a + t[:, None] * (b - a) + (2.0 * _rand((m, 2), gen) - 1.0) * 1e-9)
    return p


def _segments(case, gen, order):
    n, h = int(case["segments"]), case["h"]
    size = torch.tensor([case["nx"] * h, case["ny"] * h], dtype=torch.float64, device=DEVICE)
    a = _rand((n, 2), gen) * size
    if case["reach"] == 0.0:  # both ends anywhere
        b = _rand((n, 2), gen) * size
    else:  # any direction, length up to `reach` cells
        ang = _rand((n,), gen) * (2.0 * math.pi)
        b = a + (_rand((n,), gen) * case["reach"] * h)[:, None] * torch.stack([ang.cos(), ang.sin()], 1)
    return torch.stack([a, b], 1)[torch.randperm(n, device=DEVICE, generator=order)]


def _inputs(case, seed):
    """Everything a case is made from, before any tree and before its pose."""
    kind, nx, ny, h = case["kind"], int(case["nx"]), int(case["ny"]), float(case["h"])
    gm, gq = _rng(seed, 0), _rng(seed, 1)
    if kind not in ("locate", "build", "weights"):  # one geometry, see the module's docstring
        gm, gs = _rng(0, 2), _rng(0, 3)
    if kind in ("locate", "build"):
        xy, f, _ = _mesh(case["mesh"], nx, ny, h, gm)
        if case["utm"]:
            xy = xy + torch.tensor(UTM, dtype=torch.float64, device=DEVICE)
        return {"xy": xy, "faces": f, "points": _points(case, xy, f, gq)}
    if kind == "zonal":
        xy, f, cover = _mesh(case["mesh"], nx, ny, h, gm)
        n = int(case["boxes"])
        size = torch.tensor([nx * h, ny * h], dtype=torch.float64, device=DEVICE)
        c = _rand((n, 2), gs) * size
        lo, hi = math.log(case["side_lo"] * h), math.log(case["side_hi"] * h)
        s = torch.exp(lo + (hi - lo) * _rand((n, 2), gs))
        corners = torch.stack([c, c + s], 1)[torch.randperm(n, device=DEVICE, generator=gq)]
        return {"xy": xy, "faces": f, "cover": cover, "corners": corners, "values": 1.0 + _rand((f.shape[0],), gq)}
    if kind == "segments":
        xy, f, cover = _mesh(case["mesh"], nx, ny, h, gm)
        return {"xy": xy, "faces": f, "cover": cover, "segments": _segments(case, gs, gq)}
    if kind == "network":
        xy, _ = _lattice(nx, ny, h, gm)
        return {"xy": xy, "edges": _edges(nx, ny), "segments": _segments(case, gs, gq)}
    xy, f, _ = _mesh("quad", nx, ny, h, gm)
    xy = _turned(xy, nx, ny, h)
    if kind == "weights":
        lo, hi = xy.amin(0), xy.amax(0)
        return {"xy": xy, "faces": f, "points": lo + (hi - lo) * _rand((int(case["points"]), 2), gq)}
    qnx, qny = int(case["qnx"]), int(case["qny"])
    qh = math.sqrt(nx * ny / (qnx * qny)) * h  # both meshes cover the same area
    qxy, qf, _ = _mesh("tri", qnx, qny, qh, gs)
    qf = qf.roll(int(torch.randint(0, qf.shape[0], (1,), device=DEVICE, generator=gq)), 0)
    out = {"xy": xy, "faces": f, "qxy": qxy, "qfaces": qf, "values": 1.0 + _rand((f.shape[0],), gq)}
    if kind == "adjoint":
        out["qvalues"] = 1.0 + _rand((qf.shape[0],), gq)
    return out


def prepare(case, seed):
    s = _inputs(case, seed)
    s["kind"] = case["kind"]
    s.pop("cover", None)
    if case["kind"] not in ("locate", "build", "weights"):
        for k in ("xy", "qxy", "segments", "corners"):
            if k in s:
                s[k] = _pose(s[k], seed)
    if case["kind"] == "zonal":
        c = s.pop("corners")
        lo, hi = c.amin(1), c.amax(1)
        s["boxes"] = torch.stack([lo[:, 0], hi[:, 0], lo[:, 1], hi[:, 1]], 1)
    if case["kind"] == "network":
        s["tree"] = EdgeCellTree2d(s["xy"], s["edges"])
    elif case["kind"] != "build":
        s["tree"] = CellTree2d(s["xy"], s["faces"], -1)
    if case["kind"] == "adjoint":
        s["xy"].requires_grad_(True)
        s["qxy"].requires_grad_(True)
    return s


def run(s):
    kind = s["kind"]
    if kind == "locate":
        return s["tree"].locate_points(s["points"])
    if kind == "build":
        return CellTree2d(s["xy"], s["faces"], -1).locate_points(s["points"])
    if kind == "zonal":
        i, j, area = s["tree"].intersect_boxes(s["boxes"])
        w = WeightMatrix.from_intersections(i, j, area, s["boxes"].shape[0], s["faces"].shape[0])
        return {"box": i, "face": j, "area": area, "mean": w.mean(s["values"])}
    if kind in ("segments", "network"):
        return s["tree"].intersect_edges(s["segments"])
    if kind == "regrid":
        i, j, area = s["tree"].intersect_faces(s["qxy"], s["qfaces"], -1)
        w = WeightMatrix.from_intersections(i, j, area, s["qfaces"].shape[0], s["faces"].shape[0])
        return {"target": i, "face": j, "area": area, "mean": w.mean(s["values"])}
    if kind == "adjoint":
        i, j, area = autodiff.intersect_faces(s["tree"], s["qxy"], s["qfaces"], -1, tree_vertices=s["xy"])
        loss = (area * s["qvalues"][i] * s["values"][j]).sum()
        gq, gt = torch.autograd.grad(loss, [s["qxy"], s["xy"]])
        return {"target": i, "face": j, "area": area.detach(), "grad_target": gq, "grad_tree": gt}
    return s["tree"].compute_barycentric_weights(s["points"])


# -- work ---------------------------------------------------------------------


def work(case):
    kind, cells = case["kind"], float(case["nx"] * case["ny"])
    per = {"tri": 2.0, "quad": 1.0, "mixed": 1.25}.get(case.get("mesh", "quad"), 1.0)
    corners = {"tri": 3, "quad": 4, "mixed": 6}.get(case.get("mesh", "quad"), 4)
    faces = cells * per
    mesh = 16.0 * cells + 8.0 * corners * faces  # vertices and faces, read once
    if kind == "locate":  # per point: coordinates in, index out
        return {"bytes": 24.0 * case["points"], "flops": 30.0 * case["points"]}
    if kind == "build":  # mesh in; boxes, leaf order and packed nodes out; points as above
        return {"bytes": mesh + faces * (32.0 + 8.0 + 1.14 * 16.0) + 24.0 * case["points"],
                "flops": faces * math.log2(faces + 1) * 8.0}
    if kind == "zonal":  # boxes in, (box, face, area) per pair and a mean per box out
        lo, hi = math.log(case["side_lo"]), math.log(case["side_hi"])
        side = (case["side_hi"] - case["side_lo"]) / (hi - lo)
        pairs = case["boxes"] * (side * side + 2.0 * side + 1.0) * per
        return {"bytes": 40.0 * case["boxes"] + 24.0 * pairs + min(mesh, 8.0 * (corners + 2 * corners) * pairs),
                "flops": 10.0 * corners * pairs}
    if kind in ("segments", "network"):  # segments in, (segment, element, xy) per result out
        if case["reach"] == 0.0:
            length = 0.52 * math.sqrt(case["nx"] * case["ny"])
        else:
            length = 0.5 * case["reach"]
        hits = case["segments"] * (length * 4.0 / math.pi + 1.0) * math.sqrt(per if kind == "segments" else 1.0)
        out = 48.0 if kind == "segments" else 32.0
        return {"bytes": 32.0 * case["segments"] + out * hits, "flops": 40.0 * hits}
    if kind == "weights":  # point in, index and four weights out
        return {"bytes": (16.0 + 8.0 + 32.0) * case["points"] + min(mesh, 96.0 * case["points"]),
                "flops": 60.0 * case["points"]}
    q = 2.0 * case["qnx"] * case["qny"]
    pairs = q + cells + 2.5 * math.sqrt(q * cells)
    both = mesh + 16.0 * case["qnx"] * case["qny"] + 24.0 * q
    if kind == "regrid":  # both meshes in, (face, face, area) per pair and a mean per face out
        return {"bytes": both + 8.0 * cells + 24.0 * pairs + 8.0 * q, "flops": 100.0 * pairs}
    return {"bytes": both + 24.0 * pairs + 16.0 * (cells + q / 2) + 8.0 * (cells + q), "flops": 400.0 * pairs}


# -- float64 values -----------------------------------------------------------


def _cross(a, b):
    return a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]


def _span(a, b, poly):
    """Parameters [t0, t1] of segments a -> b (m, 2) inside convex polygons
    poly (m, k, 2) (t1 <= t0 where they miss)."""
    t0 = torch.zeros_like(a[..., 0])
    t1 = torch.ones_like(t0)
    d = b - a
    for k in range(poly.shape[1]):
        p = poly[:, k]
        e = poly[:, (k + 1) % poly.shape[1]] - p
        num, den = _cross(e, a - p), _cross(e, d)
        t = -num / den
        t0 = torch.where(den > 0, torch.maximum(t0, t), t0)
        t1 = torch.where(den < 0, torch.minimum(t1, t), t1)
        t1 = torch.where((den == 0) & (num < 0), -torch.ones_like(t1), t1)
    return t0, t1


def _overlap(a, b, grads=False):
    """Area of the overlap of convex counter-clockwise polygons a (m, ka, 2)
    and b (m, kb, 2) as the integral along its outline, and its gradients."""
    base = a[:, :1]
    a, b = a - base, b - base
    area = torch.zeros_like(a[:, 0, 0])
    ga, gb = (torch.zeros_like(a), torch.zeros_like(b)) if grads else (None, None)
    for p, other, g in ((a, b, ga), (b, a, gb)):
        k = p.shape[1]
        for c in range(k):
            u, v = p[:, c], p[:, (c + 1) % k]
            t0, t1 = _span(u, v, other)
            t1 = torch.maximum(t0, t1)
            d = v - u
            area = area + 0.5 * _cross(u + t0[:, None] * d, u + t1[:, None] * d)
            if grads:
                out = torch.stack([d[:, 1], -d[:, 0]], 1)
                second = 0.5 * (t1 * t1 - t0 * t0)
                g[:, c] += out * ((t1 - t0) - second)[:, None]
                g[:, (c + 1) % k] += out * second[:, None]
    return area, ga, gb


def _windows(lo, hi, nx, ny):
    """(query, quad) for every lattice quad in each query's index window."""
    lo = lo.floor().long() - 1
    hi = hi.floor().long() + 1
    top = torch.tensor([nx - 1, ny - 1], device=DEVICE)
    lo = torch.minimum(lo.clamp(min=0), top + 1)
    hi = torch.minimum(hi.clamp(min=-1), top)
    w = (hi - lo + 1).clamp(min=0)
    n = w[:, 0] * w[:, 1]
    for s, e in _chunks(n):
        m = n[s:e]
        q = torch.repeat_interleave(torch.arange(s, e, device=DEVICE), m)
        r = torch.arange(q.shape[0], device=DEVICE) - torch.repeat_interleave(m.cumsum(0) - m, m)
        yield q, (lo[q, 1] + r // w[q, 0]) * nx + lo[q, 0] + r % w[q, 0]


def _chunks(n):
    """Ranges of queries with about CHUNK candidates each."""
    total = n.cumsum(0).cpu().numpy()
    s = 0
    while s < len(total):
        e = int(np.searchsorted(total, (total[s - 1] if s else 0) + CHUNK, side="right"))
        e = min(max(e, s + 1), len(total))
        yield s, e
        s = e


def _exact_zonal(case, d):
    nx, ny, h = int(case["nx"]), int(case["ny"]), float(case["h"])
    _, quads = _lattice(nx, ny, h, _rng(0, 0))
    b = d["corners"].transpose(1, 2).reshape(-1, 4)
    n = b.shape[0]
    num = torch.zeros(n, dtype=torch.float64, device=DEVICE)
    den = torch.zeros_like(num)
    for q, c in _windows(b[:, [0, 2]] / h, b[:, [1, 3]] / h, nx, ny):
        box = b[q]
        for half, corner in enumerate(([0, 1, 2], [0, 2, 3])):
            tri = d["xy"][quads[c][:, corner]]
            lo, hi = tri.amin(1), tri.amax(1)
            inside = (lo[:, 0] >= box[:, 0]) & (hi[:, 0] <= box[:, 1]) & (lo[:, 1] >= box[:, 2]) & (hi[:, 1] <= box[:, 3])
            area = 0.5 * _cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]) * inside
            cut = (~inside & (lo[:, 0] < box[:, 1]) & (hi[:, 0] > box[:, 0]) & (lo[:, 1] < box[:, 3])
                   & (hi[:, 1] > box[:, 2])).nonzero()[:, 0]
            x = box[cut]
            rect = torch.stack([x[:, [0, 2]], x[:, [1, 2]], x[:, [1, 3]], x[:, [0, 3]]], 1)
            area[cut] = _overlap(tri[cut], rect)[0]
            num.index_add_(0, q, area * d["values"][d["cover"][c, half]])
            den.index_add_(0, q, area)
    return {"box": None, "face": None, "area": None, "mean": num / den}


def _regrid_pairs(case, d):
    """Candidate (query triangle, tree quad) pairs of the two meshes, in chunks."""
    nx, ny, h = int(case["nx"]), int(case["ny"]), float(case["h"])
    tri = _turned(d["qxy"], nx, ny, h, back=True)[d["qfaces"]] / h
    yield from _windows(tri.amin(1), tri.amax(1), nx, ny)


def _exact_regrid(case, d):
    n = d["qfaces"].shape[0]
    num = torch.zeros(n, dtype=torch.float64, device=DEVICE)
    den = torch.zeros_like(num)
    for q, c in _regrid_pairs(case, d):
        area = _overlap(d["qxy"][d["qfaces"][q]], d["xy"][d["faces"][c]])[0].clamp(min=0.0)
        num.index_add_(0, q, area * d["values"][c])
        den.index_add_(0, q, area)
    return {"target": None, "face": None, "area": None, "mean": num / den}


def _exact_adjoint(case, d):
    gq, gt = torch.zeros_like(d["qxy"]), torch.zeros_like(d["xy"])
    for q, c in _regrid_pairs(case, d):
        qf, tf = d["qfaces"][q], d["faces"][c]
        _, ga, gb = _overlap(d["qxy"][qf], d["xy"][tf], grads=True)
        g = (d["qvalues"][q] * d["values"][c])[:, None, None]
        gq.index_add_(0, qf.reshape(-1), (ga * g).reshape(-1, 2))
        gt.index_add_(0, tf.reshape(-1), (gb * g).reshape(-1, 2))
    return {"target": None, "face": None, "area": None, "grad_target": gq, "grad_tree": gt}


def _exact_weights(case, d):
    """Wachspress weights of each point in the quad that holds it."""
    nx, ny, h = int(case["nx"]), int(case["ny"]), float(case["h"])
    p = d["points"]
    cell = _turned(p, nx, ny, h, back=True) / h
    w = torch.zeros((p.shape[0], 4), dtype=torch.float64, device=DEVICE)
    for q, c in _windows(cell, cell, nx, ny):
        v = d["xy"][d["faces"][c]] - p[q][:, None]
        a = _cross(v, v.roll(-1, 1))  # twice the areas (p, v_k, v_k+1)
        held = ((a > 0).all(1)).nonzero()[:, 0]
        v, a = v[held], a[held]
        e = v.roll(-1, 1) - v
        corner = _cross(e.roll(1, 1), e)
        x = corner / (a.roll(1, 1) * a)
        w[q[held]] = x / x.sum(1, keepdim=True)
    return [None, w]


def _stepped(a, b, nx, ny, h):
    """(segment, quad) candidates: the quads around points a quarter cell apart."""
    n = ((b - a).norm(dim=1) / (0.5 * h)).ceil().long() + 1
    around = torch.arange(9, device=DEVICE)
    for s, e in _chunks(n * 9):
        m = n[s:e]
        q = torch.repeat_interleave(torch.arange(s, e, device=DEVICE), m)
        r = torch.arange(q.shape[0], device=DEVICE) - torch.repeat_interleave(m.cumsum(0) - m, m)
        t = r.double() / (n[q] - 1).clamp(min=1).double()
        c = ((a[q] + t[:, None] * (b[q] - a[q])) / h).floor().long()
        i = c[:, :1] + around % 3 - 1
        j = c[:, 1:] + around // 3 - 1
        ok = (i >= 0) & (i < nx) & (j >= 0) & (j < ny)
        key = torch.unique((q[:, None] * (nx * ny) + j * nx + i)[ok])
        yield key // (nx * ny), key % (nx * ny)


def _in_order(seg, t):
    """Permutation by segment, then by t."""
    first = torch.argsort(t, stable=True)
    return first[torch.argsort(seg[first], stable=True)]


def _exact_segments(case, d):
    nx, ny, h = int(case["nx"]), int(case["ny"]), float(case["h"])
    _, quads = _lattice(nx, ny, h, _rng(0, 0))
    a, b = d["segments"][:, 0], d["segments"][:, 1]
    faces, out = d["faces"].shape[0], []
    for q, c in _stepped(a, b, nx, ny, h):
        keys, lows, highs = [], [], []
        for half, corner in enumerate(([0, 1, 2], [0, 2, 3])):
            t0, t1 = _span(a[q], b[q], d["xy"][quads[c][:, corner]])
            hit = t1 > t0
            keys.append((q * faces + d["cover"][c, half])[hit])
            lows.append(t0[hit])
            highs.append(t1[hit])
        key, at = torch.unique(torch.cat(keys), return_inverse=True)
        t0 = torch.full(key.shape, 2.0, dtype=torch.float64, device=DEVICE)
        t1 = torch.full(key.shape, -1.0, dtype=torch.float64, device=DEVICE)
        t0.scatter_reduce_(0, at, torch.cat(lows), "amin")
        t1.scatter_reduce_(0, at, torch.cat(highs), "amax")
        seg = key // faces
        o = _in_order(seg, t0)
        seg, t = seg[o], torch.stack([t0[o], t1[o]], 1)
        out.append(a[seg][:, None] + t[:, :, None] * (b[seg] - a[seg])[:, None])
    return [None, None, torch.cat(out)]


def _exact_network(case, d):
    nx, ny, h = int(case["nx"]), int(case["ny"]), float(case["h"])
    _, quads = _lattice(nx, ny, h, _rng(0, 0))
    a, b = d["segments"][:, 0], d["segments"][:, 1]
    n, out = d["xy"].shape[0], []
    for q, c in _stepped(a, b, nx, ny, h):
        sides = torch.stack([quads[c], quads[c].roll(-1, 1)], 2)  # (m, 4, 2)
        key = (q[:, None] * n + sides.amin(2)) * 2 + (sides[..., 1] - sides[..., 0]).abs().gt(1)
        key = torch.unique(key)
        up, key = key % 2, key // 2
        seg, v = key // n, key % n
        p = d["xy"][v]
        e = d["xy"][v + 1 + up * nx] - p
        s = b[seg] - a[seg]
        den = _cross(s, e)
        t = _cross(p - a[seg], e) / den
        u = _cross(p - a[seg], s) / den
        hit = (t >= 0) & (t <= 1) & (u >= 0) & (u <= 1)
        seg, t = seg[hit], t[hit]
        o = _in_order(seg, t)
        seg, t = seg[o], t[o]
        out.append(a[seg] + t[:, None] * (b[seg] - a[seg]))
    return [None, None, torch.cat(out)]


def exact(case, seed):
    """The computed outputs of `run` in 64 bits (None for indices, and for the
    areas of single pairs, whose order is the tree's)."""
    kind = case["kind"]
    if kind in ("locate", "build"):
        return None
    fn = {"zonal": _exact_zonal, "segments": _exact_segments, "network": _exact_network, "regrid": _exact_regrid,
          "adjoint": _exact_adjoint, "weights": _exact_weights}[kind]
    out = fn(case, _inputs(case, seed))
    if kind in ("segments", "network"):
        out[2] = _pose(out[2], seed)
    if kind == "adjoint":
        out["grad_target"], out["grad_tree"] = _pose(out["grad_target"], seed), _pose(out["grad_tree"], seed)
    return out
