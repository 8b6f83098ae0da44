"""Workloads that a user of the library runs, through its public entry points.

Each case is a dict of plain values with a ``kind``:

* ``build``    bulk load of an R-tree (bottom-up or top-down) from boxes in
               device memory, every coordinate type; the leaf order and the
               root level are read back;
* ``counts``   per-query window counts against a resident tree;
* ``join``     all intersecting (leaf entry, query) pairs of a resident tree,
               in (query, leaf entry) order;
* ``overlay``  filter and refine of two polygon layers: MBRs, tree, join, clip
               of every candidate pair, contours in host memory;
* ``area``     differentiable intersection area of polygon pairs, forward and
               backward;
* ``align``    one step of a map-alignment fit: moved layer's MBRs, tree, join,
               areas, gradient of the vertices and of the 6 parameters.

Inputs have the distributions of the benchmark configurations (boxes and
layers around a 64-Gaussian mixture, star polygons, jittered parcels).
"""
from __future__ import annotations

import math

import torch

import parlllelrtree_b200 as prt
from parlllelrtree_b200 import alignment
from parlllelrtree_b200 import datagen as dg

F64 = torch.float64


def listed():
    return [
        # one map tile's boxes: launches and host work are all there is
        dict(name="build_tile", kind="build", n=4_001, method="bottomup", keys="morton32", coord="f32", fanout=16),
        # the build configuration at its full size, Z-order
        dict(name="build_bottomup_10m", kind="build", n=10_000_000, method="bottomup", keys="morton32", coord="f32",
             fanout=16),
        # and top-down (the better tree for repeated queries)
        dict(name="build_topdown_10m", kind="build", n=10_000_000, method="topdown", keys="", coord="f32", fanout=16),
        # the reference's own integer boxes, 4-D keys and node size (m = 10)
        dict(name="build_ref64_1m", kind="build", n=1_000_003, method="bottomup", keys="ref64", coord="i64",
             fanout=10),
        # the reference's top-down build of the same boxes
        dict(name="build_topdown_i64_300k", kind="build", n=300_007, method="topdown", keys="", coord="i64",
             fanout=10),
        # the query configuration: one million windows counted against ten million boxes
        dict(name="counts_1m_windows", kind="counts", n=10_000_000, q=1_000_000, coord="f32", fanout=16),
        # window join of a city-sized layer, pairs in query order
        dict(name="join_100k_windows", kind="join", n=1_000_003, q=100_003, coord="f32", fanout=16),
        # the small overlay configuration (two layers of 10,000 stars, 8-32 vertices)
        dict(name="overlay_stars_10k", kind="overlay", layer="stars", n=10_000, op="int"),
        # uneven polygons (4 to 4,096 vertices, holes), four candidate pairs per polygon
        dict(name="overlay_uneven_10k", kind="overlay", layer="uneven", n=10_007, op="int"),
        # the differentiable configuration at its full size
        dict(name="area_1m_pairs", kind="area", n=1_000_000, nv_lo=16, nv_hi=64),
        # fewer, more uneven polygons, some above every staging size
        dict(name="area_ragged_50k", kind="area", n=50_021, nv_lo=4, nv_hi=160),
        # one full-resolution step of the alignment configuration
        dict(name="align_step_200k", kind="align", n=200_000, fanout=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "counts", "join", "overlay", "overlay", "area", "align"])
    if kind == "build":
        coord = rng.choice(["f32", "f32", "f64", "i64", "i32"])
        method = rng.choice(["bottomup", "topdown"])
        keys = "" if method == "topdown" else rng.choice(["morton32", "ref64"]) if coord == "i64" else "morton32"
        return dict(kind=kind, n=_log(rng, 1_000, 10_000_000), method=method, keys=keys, coord=coord,
                    fanout=rng.choice([8, 10, 16, 16, 32]))
    if kind == "counts":
        return dict(kind=kind, n=_log(rng, 10_000, 10_000_000), q=_log(rng, 1_000, 1_000_000),
                    coord=rng.choice(["f32", "f64", "i64"]), fanout=rng.choice([8, 10, 16, 32]))
    if kind == "join":
        return dict(kind=kind, n=_log(rng, 10_000, 2_000_000), q=_log(rng, 1_000, 300_000),
                    coord=rng.choice(["f32", "f64", "i64", "i32"]), fanout=rng.choice([8, 10, 16, 32]))
    if kind == "overlay":
        op = rng.choice(["int", "int", "int", "diff", "union", "xor"])
        if rng.random() < 0.5:
            return dict(kind=kind, layer="stars", n=_log(rng, 300, 20_000), op=op)
        return dict(kind=kind, layer="uneven", n=_log(rng, 300, 5_000), op=op)
    if kind == "area":
        hi = rng.randint(24, 160)
        n = _log(rng, 1_000, 500_000)
        return dict(kind=kind, n=min(n, 8_000_000 // hi), nv_lo=rng.randint(4, 16), nv_hi=hi)
    return dict(kind=kind, n=_log(rng, 2_000, 200_000), fanout=rng.choice([8, 16, 32]))


# ------------------------------------------------------------------ inputs

def _typed(v, coord):
    """Boxes in the unit square in the case's coordinates; integers on the
    grids the reference reads (1e6 for its R-tree programs, 1e5 for its
    polygon files)."""
    if coord == "f32":
        return v.to(torch.float32)
    if coord == "i64":
        return torch.round(v * 1e6).to(torch.int64)
    if coord == "i32":
        return (v * 1e5).to(torch.int32)
    return v


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _mixture_boxes(n, seed, coord, mean_side=1e-4, sigma=0.02):
    g = _generator(seed)
    means = torch.from_numpy(dg.mixture_means()).cuda()
    comp = torch.randint(0, len(means), (n,), generator=g, device="cuda")
    c = (means[comp] + sigma * torch.randn((n, 2), generator=g, device="cuda", dtype=F64)).clamp_(0.0, 1.0)
    half = -0.5 * mean_side * torch.log1p(-torch.rand((n, 2), generator=g, device="cuda", dtype=F64))
    return _typed(torch.cat([c - half, c + half], 1), coord)


def _windows(n, seed, coord, lo=1e-4, hi=1e-2):
    g = _generator(seed)
    c = torch.rand((n, 2), generator=g, device="cuda", dtype=F64)
    half = 0.5 * (lo + (hi - lo) * torch.rand((n, 1), generator=g, device="cuda", dtype=F64))
    return _typed(torch.cat([c - half, c + half], 1), coord)


def _tree_inputs(case, seed):
    """Boxes and windows of the case in the seed's order: every seed finds as
    many pairs, so the joins of two seeds have outputs of the same size."""
    boxes = _mixture_boxes(case["n"], 1, case["coord"])
    queries = _windows(case["q"], 2, case["coord"])
    g = _generator(seed)
    pick = lambda x: x[torch.randperm(len(x), generator=g, device="cuda")]
    return pick(boxes), pick(queries)


def _overlay_layers(case, seed):
    """Both layers, their polygons in the seed's order (the same contours for
    every seed, elsewhere in the result)."""
    n = case["n"]
    if case["layer"] == "stars":
        args = dict(nv_lo=8, nv_hi=32, zipf=None, hole_frac=0.0, centres="uniform")
        # the configuration's radii at 10,000 polygons, scaled to keep its two pairs per polygon
        s = math.sqrt(10_000 / n)
        args.update(r_lo=1e-3 * s, r_hi=1e-2 * s)
    else:
        # the configuration's radii at 1M polygons, scaled to keep its four pairs per polygon
        s = math.sqrt(1_000_000 / n)
        args = dict(r_lo=6.5e-5 * s, r_hi=6.5e-4 * s)
    g = _generator(seed)
    return [_reordered(dg.star_layer_device(n, k, **args), torch.randperm(n, generator=g, device="cuda"))
            for k in (101, 102)]


def _spread(first, count):
    """The ranges [first, first + count) one after another, and their offsets."""
    off = torch.zeros(len(count) + 1, dtype=torch.int64, device=count.device)
    torch.cumsum(count, 0, out=off[1:])
    owner = torch.repeat_interleave(torch.arange(len(count), device=count.device), count)
    return first[owner] + torch.arange(len(owner), device=count.device) - off[owner], off


def _reordered(d, perm):
    pr, rv = d["poly_ring"], d["ring_vert"]
    rings, poly_ring = _spread(pr[perm], (pr[1:] - pr[:-1])[perm])
    verts, ring_vert = _spread(rv[rings], (rv[1:] - rv[:-1])[rings])
    return {"poly_ring": poly_ring, "ring_vert": ring_vert, "ring_hole": d["ring_hole"][rings], "xy": d["xy"][verts]}


def _pair_layers(case, seed):
    """The configuration's overlapping pairs, each turned, scaled and moved by
    the seed; vertex counts go by the case alone."""
    n = case["n"]
    A, B = dg.overlapping_pairs_device(n, seed=7, nv_lo=case["nv_lo"], nv_hi=case["nv_hi"])
    g = _generator(seed)
    u = torch.rand((n, 4), generator=g, device="cuda", dtype=F64)
    ang, scale, to = 2 * math.pi * u[:, 0], 0.7 + 0.6 * u[:, 1], u[:, 2:]
    cos, sin = scale * torch.cos(ang), scale * torch.sin(ang)
    at = A["xy"][A["ring_vert"][:-1]]
    for d in (A, B):
        owner = torch.repeat_interleave(torch.arange(n, device="cuda"), d["ring_vert"][1:] - d["ring_vert"][:-1])
        v = d["xy"] - at[owner]
        c, s = cos[owner], sin[owner]
        d["xy"] = torch.stack([c * v[:, 0] - s * v[:, 1], s * v[:, 0] + c * v[:, 1]], 1) + to[owner]
    return A, B


def _parcels(case, seed):
    """Parcels and the same parcels moved by at most half a cell, where the
    last stage of a fit works; shapes and motion by the seed, vertex counts
    by the case alone."""
    n = case["n"]
    h = 1.0 / math.ceil(math.sqrt(n))
    A, _, _ = alignment.parcel_layers(n, seed=5)
    A = {k: torch.from_numpy(v).cuda() for k, v in A.items()}
    g = _generator(seed)
    noise = lambda s: s * torch.randn(A["xy"].shape, generator=g, device="cuda", dtype=F64)
    A["xy"] = A["xy"] + noise(0.01 * h)
    motion = 2 * torch.rand(6, generator=g, device="cuda", dtype=F64) - 1
    scale = torch.tensor([0.2, 0.2, 0.2, 0.2, 0.15, 0.15], dtype=F64, device="cuda")
    return A, dict(A, xy=_moved(motion * scale * h, A["xy"]) + noise(0.045 * h))


def _shoelace(xy, ring_vert):
    nv = ring_vert[1:] - ring_vert[:-1]
    owner = torch.repeat_interleave(torch.arange(len(nv), device=xy.device), nv)
    nxt = torch.arange(len(xy), device=xy.device) + 1
    nxt = torch.where(nxt == ring_vert[owner + 1], ring_vert[owner], nxt)
    d = xy - xy[ring_vert[owner]]
    e = xy[nxt] - xy[ring_vert[owner]]
    return 0.5 * float((d[:, 0] * e[:, 1] - e[:, 0] * d[:, 1]).sum())


def _moved(theta, xy):
    m = torch.eye(2, dtype=F64, device=xy.device) + theta[:4].reshape(2, 2)
    return (xy - 0.5) @ m.T + 0.5 + theta[4:]


def _build(case, boxes):
    if case["method"] == "topdown":
        return prt.build_topdown(boxes, fanout=case["fanout"])
    return prt.build_bottomup(boxes, fanout=case["fanout"], key_mode=case["keys"])


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "build":
        st["boxes"] = _mixture_boxes(case["n"], seed, case["coord"])
    elif kind in ("counts", "join"):
        boxes, st["queries"] = _tree_inputs(case, seed)
        st["tree"] = prt.build_bottomup(boxes, fanout=case["fanout"])
    elif kind == "overlay":
        A, B = _overlay_layers(case, seed)
        st["base"], st["over"] = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
    elif kind == "area":
        A, B = _pair_layers(case, seed)
        st["base"], st["over"] = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
        st["ids"] = torch.arange(case["n"], dtype=torch.int32, device="cuda")
        st["xa"] = st["base"].xy.requires_grad_(True)
        st["xb"] = st["over"].xy.requires_grad_(True)
    else:
        A, B = _parcels(case, seed)
        st["base"], st["over"] = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
        st["xb"] = st["over"].xy
        st["queries"] = st["base"].mbr()  # the fixed layer's boxes are the join's queries
        st["total"] = _shoelace(A["xy"], A["ring_vert"])
    return st


# ------------------------------------------------------------------ passes

def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "build":
        tree = _build(case, st["boxes"])
        return tree.leaf_order(), tree.level_mbr(tree.levels - 1)
    if kind == "counts":
        return st["tree"].query_counts(st["queries"])
    if kind == "join":
        return st["tree"].join(st["queries"], sorted=True)
    if kind == "overlay":
        base, over = st["base"], st["over"]
        tree = prt.build_bottomup(base.mbr(), fanout=16)
        pairs = tree.join(over.mbr(), sorted=True)
        ids = tree.leaf_order()
        off, nverts, hole, xy = prt.overlay(pairs, base, over, leaf_to_poly=ids, op=case["op"]).to_host()
        return pairs, ids, off, nverts, hole, xy
    if kind == "area":
        xa, xb = st["xa"], st["xb"]
        xa.grad = xb.grad = None
        area = prt.intersection_area(st["base"], st["over"], st["ids"], st["ids"], base_xy=xa, over_xy=xb)
        area.sum().backward()
        return area.detach(), xa.grad, xb.grad
    base, over = st["base"], st["over"]
    theta = torch.zeros(6, dtype=F64, device="cuda", requires_grad=True)
    xb = _moved(theta, st["xb"])
    xb.retain_grad()
    over.xy = xb.detach()
    tree = prt.build_bottomup(over.mbr(), fanout=case["fanout"])
    pairs = tree.join(st["queries"])
    pb = tree.leaf_order()[pairs[:, 0].long()]
    area = prt.intersection_area(base, over, pairs[:, 1].contiguous(), pb, base_xy=base.xy, over_xy=xb)
    loss = -area.sum() / st["total"]
    loss.backward()
    return loss.detach(), theta.grad, xb.grad


def work(case):
    """Bytes a pass cannot do without: inputs read once, outputs written once."""
    kind = case["kind"]
    box = {"f32": 16, "i32": 16, "f64": 32, "i64": 32}.get(case.get("coord"), 32)
    if kind == "build":
        n = case["n"]
        # boxes in; leaf order and the levels' boxes out
        return {"bytes": n * (box + 4 + box * (1 + 1 / (case["fanout"] - 1))), "flops": 0}
    if kind in ("counts", "join"):
        n, q = case["n"], case["q"]
        # at most the whole tree, at least a path of nodes per window
        levels = max(1, math.ceil(math.log(n, case["fanout"])))
        tree = min(n * box * (1 + 1 / (case["fanout"] - 1)), q * levels * case["fanout"] * box)
        if kind == "counts":
            return {"bytes": tree + q * (box + 24), "flops": 0}
        # E[(s + w)(s + h)] of uniform windows s in [1e-4, 1e-2] and boxes of mean side 1e-4
        pairs = n * q * (3.367e-5 + 2 * 5.05e-3 * 1e-4 + 1e-8)
        return {"bytes": tree + q * box + 8 * pairs, "flops": 0}
    if kind == "overlay":
        n = case["n"]
        # vertices of both layers in; pairs and contours out (per pair, as the configurations give them)
        per_poly, pairs, out = (20, 2.1 * n, 14) if case["layer"] == "stars" else (870, 4 * n, 395)
        return {"bytes": 2 * n * per_poly * 16 + pairs * (8 + 8 + 16 * out), "flops": 0}
    if kind == "area":
        n, nv = case["n"], 0.5 * (case["nv_lo"] + case["nv_hi"])
        # both polygons read by each direction, gradients and areas written
        return {"bytes": n * (2 * nv * 48 + 32), "flops": 0}
    n, nv = case["n"], 5
    # moved layer written and read, fixed layer read, gradient out, about 2.4 pairs per parcel
    return {"bytes": n * (nv * 16 * 5 + 2.4 * 16 + 2 * 32), "flops": 0}


# ------------------------------------------------------------------ 64-bit values

def _padded(xy, ring_vert, ids):
    """Vertices of polygons `ids` and their successors, [P, n, 2], the mask of
    real ones and their indices."""
    v0 = ring_vert[ids]
    nv = ring_vert[ids + 1] - v0
    k = torch.arange(int(nv.max()), device=xy.device)
    ok = k < nv[:, None]
    i = v0[:, None] + torch.where(ok, k, 0)
    j = v0[:, None] + torch.where(k + 1 < nv[:, None], k + 1, 0)
    return xy[i], xy[j], ok, i, j


def _inside(px, py, a, s, ok):
    """Even-odd test of points [P, n] against edges a -> a + s [P, m]."""
    ay, by = a[:, None, :, 1], (a + s)[:, None, :, 1]
    straddle = ((ay > py[..., None]) != (by > py[..., None])) & ok[:, None, :]
    x = a[:, None, :, 0] + (py[..., None] - ay) * s[:, None, :, 0] / torch.where(straddle, s[:, None, :, 1], 1.0)
    return ((straddle & (px[..., None] < x)).sum(-1) & 1).to(F64)


def _areas(xa, rva, xb, rvb, pa, pb, budget=20_000_000):
    """Areas of A[pa] ∩ B[pb] of counter-clockwise simple polygons and the
    gradients of their sum, by the boundary integral with every pair of edges
    intersected: an edge's inside length is what it starts with plus the rest
    of the edge after every entering crossing less that after every leaving one."""
    area = torch.zeros(len(pa), dtype=F64, device=xa.device)
    ga, gb = torch.zeros_like(xa), torch.zeros_like(xb)
    most = int((rva[1:] - rva[:-1]).max()) * int((rvb[1:] - rvb[:-1]).max())
    step = max(1, budget // most)
    for c in range(0, len(pa), step):
        p, q, oka, ia, ja = _padded(xa, rva, pa[c:c + step])
        a, b, okb, ib, jb = _padded(xb, rvb, pb[c:c + step])
        r, s = q - p, b - a
        rx, ry = r[:, :, None, 0], r[:, :, None, 1]
        sx, sy = s[:, None, :, 0], s[:, None, :, 1]
        dx = a[:, None, :, 0] - p[:, :, None, 0]
        dy = a[:, None, :, 1] - p[:, :, None, 1]
        den = rx * sy - ry * sx
        safe = torch.where(den != 0, den, 1.0)
        t, u = (dx * sy - dy * sx) / safe, (dx * ry - dy * rx) / safe
        hit = (den != 0) & oka[:, :, None] & okb[:, None, :] & (t > 0) & (t < 1) & (u > 0) & (u < 1)
        sign = torch.where(hit, torch.sign(den), 0.0)  # > 0: A's edge leaves B, B's edge enters A
        o = p[:, :1]
        total = 0.0
        for (v, e, ok, idx, jdx, w, ew, okw, sg, par, dim, grad) in (
                (p, r, oka, ia, ja, a, s, okb, -sign, t, 2, ga), (a, s, okb, ib, jb, p, r, oka, sign, u, 1, gb)):
            start = _inside(v[..., 0], v[..., 1], w, ew, okw)
            length = torch.where(ok, start + (sg * (1 - par)).sum(dim), 0.0)
            first = torch.where(ok, 0.5 * start + (0.5 * sg * (1 - par * par)).sum(dim), 0.0)
            d = v - o
            total = total + (length * (d[..., 0] * e[..., 1] - d[..., 1] * e[..., 0])).sum(1)
            normal = torch.stack([e[..., 1], -e[..., 0]], -1)
            grad.index_add_(0, jdx.reshape(-1), (normal * first[..., None]).reshape(-1, 2))
            grad.index_add_(0, idx.reshape(-1), (normal * (length - first)[..., None]).reshape(-1, 2))
        area[c:c + step] = 0.5 * total
    return area, ga, gb


def exact(case, seed):
    kind = case["kind"]
    if kind == "area":
        A, B = _pair_layers(case, seed)
        ids = torch.arange(case["n"], device="cuda")
        return _areas(A["xy"], A["ring_vert"], B["xy"], B["ring_vert"], ids, ids)
    if kind == "align":
        A, B = _parcels(case, seed)
        n, g = case["n"], math.ceil(math.sqrt(case["n"]))
        theta = torch.zeros(6, dtype=F64, device="cuda", requires_grad=True)
        xb = _moved(theta, B["xy"])
        cell = torch.arange(n, device="cuda")
        i, j = cell // g, cell % g
        # a parcel moved by less than a cell meets its neighbours only
        pa, pb = [], []
        for di in (-1, 0, 1):
            for dj in (-1, 0, 1):
                k = (i + di) * g + j + dj
                ok = (i + di >= 0) & (j + dj >= 0) & (j + dj < g) & (k < n)
                pa.append(cell[ok])
                pb.append(k[ok])
        total = _shoelace(A["xy"], A["ring_vert"])
        area, _, grad = _areas(A["xy"], A["ring_vert"], xb.detach(), B["ring_vert"], torch.cat(pa), torch.cat(pb))
        grad = -grad / total
        xb.backward(grad)
        return -area.sum() / total, theta.grad, grad
    return None
