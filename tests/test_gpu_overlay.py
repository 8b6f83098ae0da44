"""GPC clipping on the GPU: contours, hole flags and vertex order bit-exact
against the oracle and the reference's golden fixtures."""
import os

import numpy as np
import pytest
import torch

import oracle
from conftest import GOLDEN
from helpers import rings_of, same_contours
from parlllelrtree_b200 import datagen as dg

pytestmark = pytest.mark.gpu

OPS = ["diff", "int", "xor", "union"]


def golden():
    g = np.load(os.path.join(GOLDEN, "gpc.npz"))
    A = {k[2:]: g[k] for k in g.files if k.startswith("a_")}
    B = {k[2:]: g[k] for k in g.files if k.startswith("b_")}
    return g, A, B


@pytest.mark.parametrize("sched", ["plain", "batched"])
@pytest.mark.parametrize("op", [0, 1, 2, 3])
def test_golden_pairs(cuda, sched, op):
    import parlllelrtree_b200 as prt

    g, A, B = golden()
    pairs = g["pairs"].astype(np.int32)
    res = prt.overlay(torch.from_numpy(pairs).cuda(), prt.Layer.from_dict(A), prt.Layer.from_dict(B),
                      op=OPS[op], sched=sched)
    got = res.contours()
    nc, nv, hole, xy = g[f"op{op}_ncont"], g[f"op{op}_nverts"], g[f"op{op}_hole"], g[f"op{op}_xy"]
    c = v = 0
    for k in range(len(pairs)):
        ref = []
        for _ in range(nc[k]):
            ref.append((int(hole[c]), xy[v:v + nv[c]]))
            v += nv[c]
            c += 1
        assert same_contours(got[k], ref), f"pair {k}"


def small_config(n=2500, seed=0):
    """The small plain config's shape: stars of 8-32 vertices, radius
    log-uniform 1e-3..1e-2; denser (fewer polygons per unit area) to keep the
    oracle fast."""
    A = dg.star_layer(n, seed=seed, r_lo=5e-3, r_hi=3e-2)
    B = dg.star_layer(n, seed=seed + 1, r_lo=5e-3, r_hi=3e-2)
    return A, B


@pytest.mark.parametrize("sched", ["plain", "batched"])
def test_join_then_clip_pipeline(cuda, sched):
    """Tree over layer A's MBRs -> join layer B -> clip every candidate pair,
    remapped through the leaf order like Execute (GPC:89-90)."""
    import parlllelrtree_b200 as prt

    A, B = small_config()
    LA, LB = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
    t = prt.build_bottomup(LA.mbr(), fanout=16)
    pairs = t.join(LB.mbr(), sorted=True)
    l2p = t.leaf_order()
    res = prt.overlay(pairs, LA, LB, leaf_to_poly=l2p, sched=sched)
    got = res.contours()
    p = pairs.cpu().numpy()
    perm = l2p.cpu().numpy()
    # candidate set == brute-force MBR intersections
    ba, bb = dg.layer_bboxes(A), dg.layer_bboxes(B)
    exp = set()
    for j in range(len(bb)):
        m = (ba[:, 0] <= bb[j, 2]) & (bb[j, 0] <= ba[:, 2]) & (ba[:, 1] <= bb[j, 3]) & (bb[j, 1] <= ba[:, 3])
        exp.update((int(i), j) for i in np.nonzero(m)[0])
    assert {(int(perm[a]), int(b)) for a, b in p} == exp
    for k, (leaf, q) in enumerate(p):
        ref = oracle.gpc_clip(rings_of(A, perm[leaf]), rings_of(B, q), 1)
        assert same_contours(got[k], ref), k
    assert res.nonempty > 0


def test_plain_equals_batched_with_holes(cuda):
    import parlllelrtree_b200 as prt

    A = dg.star_layer(300, seed=5, nv_lo=4, nv_hi=200, r_lo=0.02, r_hi=0.1, hole_frac=0.3, zipf=1.2)
    B = dg.star_layer(300, seed=6, nv_lo=4, nv_hi=200, r_lo=0.02, r_hi=0.1, hole_frac=0.3, zipf=1.2)
    LA, LB = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
    t = prt.build_bottomup(LA.mbr(), fanout=16)
    pairs = t.join(LB.mbr(), sorted=True)
    l2p = t.leaf_order()
    r1 = prt.overlay(pairs, LA, LB, leaf_to_poly=l2p, sched="plain").contours()
    r2 = prt.overlay(pairs, LA, LB, leaf_to_poly=l2p, sched="batched").contours()
    p = pairs.cpu().numpy()
    perm = l2p.cpu().numpy()
    for k, (leaf, q) in enumerate(p):
        ref = oracle.gpc_clip(rings_of(A, perm[leaf]), rings_of(B, q), 1)
        assert same_contours(r1[k], ref), k
        assert same_contours(r2[k], ref), k


def comb(k, x0, y0, w, h, vertical=False):
    """A comb polygon with k teeth (4k vertices)."""
    pts = []
    for i in range(k):
        pts += [(x0 + (2 * i) * w, y0), (x0 + (2 * i + 1) * w, y0), (x0 + (2 * i + 1) * w, y0 + h),
                (x0 + (2 * i + 2) * w, y0 + h)]
    pts += [(x0 + 2 * k * w, y0 - h), (x0, y0 - h)]
    a = np.array(pts, float)
    if vertical:
        a = a[:, ::-1].copy()[::-1].copy()
    return a


def test_many_intersections_retry_path(cuda):
    """Two crossing combs give O(k^2) output vertices: more than the first
    arena slice holds, so the pair is retried with a larger slice."""
    import parlllelrtree_b200 as prt

    s = [comb(40, 0.0, 0.0, 0.01, 0.9)]
    c = [comb(40, -0.05, -0.05, 0.0101, 0.95, vertical=True)]
    for op in OPS:
        got = prt.clip_pair(s, c, op)
        ref = oracle.gpc_clip(s, c, OPS.index(op))
        assert same_contours(got, ref), op


def test_clip_pair_degenerate(cuda):
    import parlllelrtree_b200 as prt

    sq = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], float)
    cases = [([sq], [sq]), ([sq], [sq + [1, 0]]), ([sq], [sq + [1, 1]]), ([sq], [sq * 0.5 + 0.25]),
             ([sq], [sq + [5, 5]]), ([sq], []), ([], [sq]), ([sq, sq * 0.5 + 0.25], [sq + [0.5, 0.5]]),
             ([np.array([[0, 0], [2, 0], [2, 0], [1, 1]], float)], [sq]),
             ([np.array([[0, 0], [1, 0], [2, 0], [1, 1]], float)], [sq])]
    for s, c in cases:
        for op in OPS:
            assert same_contours(prt.clip_pair(s, c, op), oracle.gpc_clip(s, c, OPS.index(op))), (op,)


def test_reference_csr_entry_point(cuda):
    """run() with the reference's num/prefix/vertex/hole arrays."""
    import parlllelrtree_b200 as prt

    A, B = small_config(800, seed=9)
    LA, LB = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
    t = prt.build_bottomup(LA.mbr(), fanout=10)
    pairs = t.join(LB.mbr(), sorted=True)
    l2p = t.leaf_order()
    numA = np.diff(A["ring_vert"]).astype(np.int32)
    numB = np.diff(B["ring_vert"]).astype(np.int32)
    r1 = prt.overlay_ref(pairs, numA, A["ring_vert"][:-1], A["xy"], A["ring_hole"], numB, B["ring_vert"][:-1],
                         B["xy"], B["ring_hole"], leaf_to_poly=l2p).contours()
    r2 = prt.overlay(pairs, LA, LB, leaf_to_poly=l2p, sched="plain").contours()
    assert all(same_contours(x, y) for x, y in zip(r1, r2))


def test_results_area_matches_oracle(cuda):
    import parlllelrtree_b200 as prt

    g, A, B = golden()
    pairs = g["pairs"].astype(np.int32)
    res = prt.overlay(torch.from_numpy(pairs).cuda(), prt.Layer.from_dict(A), prt.Layer.from_dict(B))
    area = res.area().cpu().numpy()
    for k, (i, j) in enumerate(pairs):
        # same contours, same centred shoelace in the same order as the oracle
        ref = oracle.result_area(oracle.gpc_clip(rings_of(A, i), rings_of(B, j), 1))
        assert abs(area[k] - ref) <= 1e-12 * abs(ref) + 1e-24


def layer_of(polys):
    rings = [np.asarray(r, dtype=np.float64).reshape(-1, 2) for p in polys for r in p]
    return {"poly_ring": np.cumsum([0] + [len(p) for p in polys]).astype(np.int64),
            "ring_vert": np.cumsum([0] + [len(r) for r in rings]).astype(np.int64),
            "ring_hole": np.zeros(len(rings), dtype=np.int32),
            "xy": np.concatenate(rings)}


def clip_all(A, B, n):
    import parlllelrtree_b200 as prt

    ids = np.arange(n, dtype=np.int32)
    pairs = torch.from_numpy(np.stack([ids, ids], axis=1)).cuda()
    return prt.overlay(pairs, prt.Layer.from_dict(A), prt.Layer.from_dict(B), op="int").contours()


@pytest.mark.parametrize("na,nb,hole_frac", [
    (3, 3, 0.0), (4, 5, 0.0), (16, 15, 0.9), (17, 16, 0.0), (63, 64, 0.0), (64, 64, 0.0), (64, 65, 0.0),
    (124, 4, 0.0), (60, 50, 0.9), (511, 512, 0.0), (512, 512, 0.0), (512, 513, 0.9), (1020, 4, 0.0), (1025, 3, 0.0),
    (2000, 2223, 0.0), (4096, 128, 0.0), (4096, 129, 0.9), (4096, 4096, 0.0), (4352, 4096, 0.0), (4353, 4096, 0.0)])
def test_traced_intersections(cuda, na, nb, hole_frac):
    """Stars around the edges of the tracing classes' sizes (128, 1,024, 4,224 and
    8,448 vertices a pair), apart, overlapping in one and in several contours, and
    one inside the other."""
    n = 64 if na + nb < 200 else 12 if na + nb < 2000 else 5
    rng = np.random.default_rng(na * 10007 + nb)
    c = rng.random((n, 2))
    r = np.full(n, 0.01)
    A = dg.star_layer(n, seed=na, nv_lo=na, nv_hi=na, centre_xy=c, radii=r, hole_frac=hole_frac)
    B = dg.star_layer(n, seed=nb + 1, nv_lo=nb, nv_hi=nb, centre_xy=c + rng.uniform(-0.012, 0.012, (n, 2)),
                      radii=r * rng.uniform(0.2, 1.5, n), hole_frac=hole_frac)
    got = clip_all(A, B, n)
    for i in range(n):
        assert same_contours(got[i], oracle.gpc_clip(rings_of(A, i), rings_of(B, i), 1)), f"pair {i}"


def test_pairs_that_are_not_traced(cuda):
    """Pairs outside general position: shared vertices and edges,
    vertices on edges, polygons that cross or touch themselves, equal polygons,
    crossings at one y, slivers of an ulp, rings of under three vertices, more rings
    than are kept, coordinates of very different sizes."""
    sq = [(0, 0), (4, 0), (4, 4), (0, 4)]
    tri = [(0.0, 0.0), (4.0, 0.5), (1.0, 4.0)]
    bow = [(0, 0.1), (4, 4), (4, 0), (0.3, 3.9)]
    star = [tuple(p) for p in dg.star_layer(1, seed=5, nv_lo=21, nv_hi=21, centre_xy=np.array([[2.0, 2.0]]),
                                            radii=np.array([2.0]))["xy"]]
    ulp = [(x, float(np.nextafter(y, 9.0))) for x, y in star]
    dots = [[(0.3 + 0.11 * k, 0.3 + 0.107 * k), (0.35 + 0.11 * k, 0.33 + 0.107 * k), (0.31 + 0.11 * k, 0.38 + 0.107 * k)]
            for k in range(33)]
    cases = [([sq], [sq]), ([sq], [[(2, 2), (6, 2), (6, 6), (2, 6)]]), ([tri], [tri]), ([tri], [sq]),
             ([bow], [tri]), ([tri], [bow]), ([bow], [bow]), ([star], [star]), ([star], [ulp]), ([star], [sq]),
             ([tri], [[(2.0, 0.25), (5.0, 1.0), (3.0, 3.0)]]),           # a vertex on an edge
             ([tri], [[(4.0, 0.5), (6.0, 1.5), (5.0, 3.0)]]),            # a shared vertex
             ([tri], [[(0.0, 0.0), (4.0, 0.5), (2.0, -3.0)]]),           # a shared edge
             ([[(0, 0), (2, 3), (4, 0.5), (2, 1)]], [[(0, 0.25), (4, 0.25), (2, -1)]]),
             ([[(-1, -3), (1, 3.5), (1.5, 3)]], [[(1, -3.25), (-1, 3.25), (-1.5, 2.75)]]),
             ([tri, [(1.0, 1.0)]], [sq]), ([tri, [(1.0, 1.0), (2.0, 1.5)]], [star]),
             (dots, [star]), ([star], dots + [sq]), (dots[:16], dots[16:32] + [star]),
             ([[(1e12 * x, 1e12 * y) for x, y in star]], [tri]), ([tri], [[(1e-12 * x, 1e-12 * y) for x, y in star]]),
             ([[(0.0, 0.0), (4.0, 0.5), (4.0, 0.5), (1.0, 4.0)]], [star])]
    A, B = layer_of([a for a, _ in cases]), layer_of([b for _, b in cases])
    got = clip_all(A, B, len(cases))
    for i in range(len(cases)):
        assert same_contours(got[i], oracle.gpc_clip(rings_of(A, i), rings_of(B, i), 1)), f"pair {i}"


def test_traced_on_a_grid(cuda):
    """Rectangles, Ls, combs and stars on whole numbers: equal ys, horizontal and
    vertical edges, crossings on horizontal edges; many pairs share points too."""
    rng = np.random.default_rng(12)

    def rect():
        x, y = np.sort(rng.integers(0, 40, 2)) + [0, 1], np.sort(rng.integers(0, 40, 2)) + [0, 1]
        return np.array([(x[0], y[0]), (x[1], y[0]), (x[1], y[1]), (x[0], y[1])], float)[::rng.choice([1, -1])]

    def ell():
        a, b = np.sort(rng.choice(40, 3, replace=False)), np.sort(rng.choice(40, 3, replace=False))
        r = np.array([(a[0], b[0]), (a[2], b[0]), (a[2], b[1]), (a[1], b[1]), (a[1], b[2]), (a[0], b[2])], float)
        return np.roll(np.abs(40.0 * rng.integers(0, 2, 2) - r), rng.integers(6), 0)

    def comb():
        k = int(rng.integers(2, 6))
        x = np.sort(rng.choice(60, 2 * k, replace=False)).astype(float)
        p = [(x[0], 0.0)]
        for t in range(k):
            p += [(x[2 * t], h := float(rng.integers(10, 45))), (x[2 * t + 1], h)]
            if t < k - 1:
                p += [(x[2 * t + 1], g := float(rng.integers(1, 9))), (x[2 * t + 2], g)]
        p = np.array(p + [(x[-1], 0.0)])
        return np.abs([0.0, 45.0 * rng.integers(0, 2)] - p)[:, ::rng.choice([1, -1])]

    def star():
        t = np.sort(rng.random(int(rng.integers(4, 16)))) * 2 * np.pi
        r = rng.uniform(5, 20, len(t))
        return np.round(np.stack([20 + r * np.cos(t), 20 + r * np.sin(t)], 1) + rng.uniform(-5, 5, 2))

    def polygon():
        return [[rect, ell, comb, star][rng.integers(4)]() for _ in range(rng.choice([1, 1, 2]))]

    n = 3000
    A, B = layer_of([polygon() for _ in range(n)]), layer_of([polygon() for _ in range(n)])
    got = clip_all(A, B, n)
    for i in range(n):
        assert same_contours(got[i], oracle.gpc_clip(rings_of(A, i), rings_of(B, i), 1)), f"pair {i}"


@pytest.mark.parametrize("op", [0, 2, 3])
@pytest.mark.parametrize("na,nb,hole_frac", [(3, 3, 0.0), (16, 15, 0.9), (64, 64, 0.9), (64, 65, 0.0), (512, 513, 0.9),
                                             (4096, 129, 0.9), (4352, 4096, 0.0)])
def test_traced_other_operations(cuda, op, na, nb, hole_frac):
    """The same pairs' difference, exclusive or and union, and polygons on a grid."""
    import parlllelrtree_b200 as prt

    n = 64 if na + nb < 200 else 6
    rng = np.random.default_rng(na + 7919 * nb)
    c = rng.random((n, 2))
    r = np.full(n, 0.01)
    A = dg.star_layer(n, seed=na, nv_lo=na, nv_hi=na, centre_xy=c, radii=r, hole_frac=hole_frac)
    B = dg.star_layer(n, seed=nb + 1, nv_lo=nb, nv_hi=nb, centre_xy=c + rng.uniform(-0.012, 0.012, (n, 2)),
                      radii=r * rng.uniform(0.2, 1.5, n), hole_frac=hole_frac)
    if na < 200:  # the second half on a grid that a few of their points share
        for L in (A, B):
            half = L["ring_vert"][L["poly_ring"][n // 2]]
            L["xy"][half:] = np.round(L["xy"][half:] * 3000) / 3000
    ids = np.arange(n, dtype=np.int32)
    got = prt.overlay(torch.from_numpy(np.stack([ids, ids], axis=1)).cuda(), prt.Layer.from_dict(A),
                      prt.Layer.from_dict(B), op=OPS[op]).contours()
    for i in range(n):
        assert same_contours(got[i], oracle.gpc_clip(rings_of(A, i), rings_of(B, i), op)), f"pair {i}"


@pytest.mark.parametrize("op", [0, 1, 2, 3])
@pytest.mark.parametrize("sx,sy", [(1.0, 1e9), (1e9, 1.0), (1e6, 1e6), (1e-9, 1.0), (1.0, 1e18), (1e-18, 1e-18)])
def test_traced_scales(cuda, op, sx, sy):
    """Polygons much wider or taller than the other way, very large and very small."""
    import parlllelrtree_b200 as prt

    n = 48
    rng = np.random.default_rng(17)
    c = rng.random((n, 2))
    r = np.full(n, 0.01)
    A = dg.star_layer(n, seed=3, nv_lo=4, nv_hi=30, centre_xy=c, radii=r, hole_frac=0.3)
    B = dg.star_layer(n, seed=4, nv_lo=4, nv_hi=30, centre_xy=c + rng.uniform(-0.01, 0.01, (n, 2)), radii=r, hole_frac=0.3)
    for L in (A, B):
        L["xy"] = L["xy"] * np.array([sx, sy])
    ids = np.arange(n, dtype=np.int32)
    got = prt.overlay(torch.from_numpy(np.stack([ids, ids], axis=1)).cuda(), prt.Layer.from_dict(A),
                      prt.Layer.from_dict(B), op=OPS[op]).contours()
    for i in range(n):
        assert same_contours(got[i], oracle.gpc_clip(rings_of(A, i), rings_of(B, i), op)), f"pair {i}"


def check_all(A, B, n, op):
    import parlllelrtree_b200 as prt

    ids = np.arange(n, dtype=np.int32)
    got = prt.overlay(torch.from_numpy(np.stack([ids, ids], axis=1)).cuda(), prt.Layer.from_dict(A),
                      prt.Layer.from_dict(B), op=OPS[op]).contours()
    for i in range(n):
        assert same_contours(got[i], oracle.gpc_clip(rings_of(A, i), rings_of(B, i), op)), f"pair {i}"


@pytest.mark.parametrize("op", [0, 1, 2, 3])
@pytest.mark.parametrize("na,nb,sx,sy", [(60, 40, 1e-9, 1e-307), (300, 40, 1e-9, 1e-307), (1500, 100, 1e-9, 1e-306),
                                         (4500, 300, 1e-9, 1e-306), (30, 20, 1e140, 1e-150), (30, 20, 1.0, 1e-131)])
def test_ys_next_to_zero(cuda, op, na, nb, sx, sy):
    """Pairs of every tracing class whose y extent is next to nothing, where
    vertices per unit of y are beyond the largest double."""
    n = 24 if na < 100 else 4
    rng = np.random.default_rng(na)
    c = np.zeros((n, 2))
    A = dg.star_layer(n, seed=na, nv_lo=na, nv_hi=na, centre_xy=c, radii=np.ones(n))
    B = dg.star_layer(n, seed=nb, nv_lo=nb, nv_hi=nb, centre_xy=rng.uniform(-1, 1, (n, 2)), radii=np.ones(n))
    for L in (A, B):
        L["xy"] = L["xy"] * np.array([sx, sy])
    check_all(A, B, n, op)


@pytest.mark.parametrize("op", [0, 1, 2, 3])
def test_both_zeros_on_a_scanline(cuda, op):
    """Horizontal edges between y = +0.0 and y = -0.0, as rounding to whole numbers
    gives them, alone and in polygons on a grid around the origin."""
    a = [(-1, 1), (2, 1), (2, -0.0), (-1, 0.0)]
    cases = [([a], [[(0, -2), (1, -2), (0.5, 0.5)]]), ([a], [[(0, -2), (1, -2), (0.5, -0.5)]]),
             ([a[::-1]], [[(0, -2), (1, -2), (0.5, 0.5)]]), ([[(x, -y) for x, y in a]], [[(0, -2), (1, -2), (0.5, 0.5)]]),
             ([[(-1, 1), (2, 1), (2, 0.0), (-1, -0.0)]], [[(0, -2), (1, -2), (0.5, 0.5)]]),
             ([[(-1, 1), (2, 1), (2, -0.0), (-1, -0.0)]], [[(0, -2), (1, -2), (0.5, 0.5)]]),
             ([[(-1, 1), (2, 1), (2, 0.0), (-1, 0.0)]], [[(0.2, -0.0), (1, -2), (0.5, 0.5)]])]
    rng = np.random.default_rng(31)

    def star():
        t = np.sort(rng.random(int(rng.integers(4, 17)))) * 2 * np.pi
        r = rng.uniform(2, 6, len(t))
        return np.round(np.stack([r * np.cos(t), r * np.sin(t)], 1) + rng.uniform(-2, 2, 2))

    cases += [([star() for _ in range(1 + k % 2)], [star()]) for k in range(3000)]
    assert any((np.signbit(p) & (p == 0)).any() for s, _ in cases[7:] for p in s)
    check_all(layer_of([s for s, _ in cases]), layer_of([c for _, c in cases]), len(cases), op)


@pytest.mark.parametrize("op", [0, 1, 2, 3])
@pytest.mark.parametrize("scale", [1e149, 1e155, 1e160, 1e290])
def test_products_that_overflow(cuda, op, scale):
    """Coordinates whose products of differences are within, and beyond, the
    largest double; pairs with holes and inside each other, which are told apart
    by such products."""
    n = 300
    rng = np.random.default_rng(23)
    c, r = np.zeros((n, 2)), np.full(n, 1.0)
    A = dg.star_layer(n, seed=5, nv_lo=4, nv_hi=12, centre_xy=c, radii=r, hole_frac=0.5)
    B = dg.star_layer(n, seed=6, nv_lo=4, nv_hi=12, centre_xy=rng.uniform(-0.8, 0.8, (n, 2)),
                      radii=rng.uniform(0.2, 1.2, n), hole_frac=0.3)
    for L in (A, B):
        L["xy"] = L["xy"] * scale
    check_all(A, B, n, op)


def stars_across(n, na, nb):
    """Stars, each with a smaller one across its boundary: a few crossings, general
    position."""
    rng = np.random.default_rng(na * 31 + nb)
    c = rng.random((n, 2))
    A = dg.star_layer(n, seed=na, nv_lo=na, nv_hi=na, centre_xy=c, radii=np.full(n, 0.01))
    B = dg.star_layer(n, seed=nb + 1, nv_lo=nb, nv_hi=nb, centre_xy=c + [0.006, 0.003], radii=np.full(n, 0.004))
    return A, B


def ids_of(n):
    ids = np.arange(n, dtype=np.int32)
    return torch.from_numpy(np.stack([ids, ids], axis=1)).cuda()


@pytest.mark.parametrize("na,nb,left", [(64, 64, 0), (124, 5, 0), (1020, 4, 0), (1020, 5, 0), (4096, 64, 0), (4096, 65, 0),
                                        (4352, 4096, 0), (4353, 4096, 4)])
def test_class_limits(cuda, na, nb, left):
    """Pairs at and one above the tracing classes' 128, 1,024, 4,160 and 8,448
    vertices are traced, up to the last."""
    import parlllelrtree_b200 as prt

    A, B = stars_across(4, na, nb)
    r = prt.overlay(ids_of(4), prt.Layer.from_dict(A), prt.Layer.from_dict(B))
    assert r.left == left
    for i, got in enumerate(r.contours()):
        assert same_contours(got, oracle.gpc_clip(rings_of(A, i), rings_of(B, i), 1)), f"pair {i}"


def test_pairs_left_are_counted(cuda):
    """Equal polygons are left; every pair counts where nothing is traced."""
    import parlllelrtree_b200 as prt

    A, B = stars_across(40, 12, 9)
    LA, LB = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
    for op in OPS:
        assert prt.overlay(ids_of(40), LA, LB, op=op).left == 0
        assert prt.overlay(ids_of(40), LA, LA, op=op).left == 40
    assert prt.overlay(ids_of(40), LA, LB, sched="plain").left == 40
    with prt.schedule(dict(prt.get_schedule(), sweep_only=1)):
        assert prt.overlay(ids_of(40), LA, LB).left == 40
    assert prt.overlay(ids_of(0), LA, LB).left == 0


@pytest.mark.parametrize("op", ["int", "xor"])
@pytest.mark.parametrize("equal", [0, 1000, 56_800, 56_832, 60_000])
def test_many_small_pairs_left(cuda, op, equal):
    """62,000 small pairs, too many for a warp each, of which tracing leaves a few, some
    1,776 warps of one pair per thread (the line between the two launches), and most."""
    import parlllelrtree_b200 as prt

    n = 62_000
    A, B = stars_across(n, 8, 8)
    B["xy"][: 8 * equal] = A["xy"][: 8 * equal]
    LA, LB = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
    r = prt.overlay(ids_of(n), LA, LB, op=op)
    assert r.left == equal
    got, ref = r.to_host(), prt.overlay(ids_of(n), LA, LB, op=op, sched="plain").to_host()
    assert all(np.array_equal(g, e) for g, e in zip(got, ref))
    c = r.contours_of(range(0, n, 500))
    for k, i in enumerate(range(0, n, 500)):
        assert same_contours(c[k], oracle.gpc_clip(rings_of(A, i), rings_of(B, i), OPS.index(op))), f"pair {i}"


@pytest.mark.parametrize("op", OPS)
def test_traced_bits(cuda, op):
    """Traced results are those of the clippers bit for bit, zeros' signs too."""
    import parlllelrtree_b200 as prt

    rng = np.random.default_rng(41)
    A = dg.star_layer(3000, seed=1, nv_lo=4, nv_hi=40, r_lo=2.0, r_hi=8.0, centre_xy=rng.uniform(-6, 6, (3000, 2)), hole_frac=0.2)
    B = dg.star_layer(3000, seed=2, nv_lo=4, nv_hi=40, r_lo=2.0, r_hi=8.0, centre_xy=rng.uniform(-6, 6, (3000, 2)), hole_frac=0.2)
    for L in (A, B):  # a third on whole numbers
        v = L["ring_vert"][L["poly_ring"][1000]]
        L["xy"][:v] = np.round(L["xy"][:v])
    LA, LB = prt.Layer.from_dict(A), prt.Layer.from_dict(B)
    r = prt.overlay(ids_of(3000), LA, LB, op=op)
    assert 0 < r.left < 1000
    with prt.schedule(dict(prt.get_schedule(), sweep_only=1)):
        ref = prt.overlay(ids_of(3000), LA, LB, op=op).to_host()
    assert all(np.array_equal(g.view(np.int64) if g.dtype == np.float64 else g,
                              e.view(np.int64) if e.dtype == np.float64 else e) for g, e in zip(r.to_host(), ref))


def test_large_results_leave_in_pieces(cuda):
    """Results above the 64 MiB of vertices that a copy-out puts into order at a time,
    and the same without device memory to do it in."""
    import parlllelrtree_b200 as prt
    from parlllelrtree_b200 import _lib

    n = 12_000
    A, B = stars_across(n, 500, 400)
    B["xy"] = A["xy"][np.arange(n * 500).reshape(n, 500)[:, :400].reshape(-1)] + [0.0004, 0.0003]
    r = prt.overlay(ids_of(n), prt.Layer.from_dict(A), prt.Layer.from_dict(B), op="union")
    assert r.n_vertices * 16 > 64 << 20
    off, nv, hole, xy = r.to_host()
    assert off[-1] == len(nv) == r.n_contours and nv.sum() == len(xy) == r.n_vertices
    L = _lib.lib()
    try:
        L.prt_debug_alloc_limit(1 << 16)
        host = r.to_host()
        with pytest.raises(prt.PrtError) as e:
            prt.overlay(ids_of(n), prt.Layer.from_dict(A), prt.Layer.from_dict(B))
        assert e.value.code == _lib.PRT_ERR_NOMEM
    finally:
        L.prt_debug_alloc_limit(0)
    assert all(np.array_equal(a, b) for a, b in zip((off, nv, hole, xy), host))
    vo = np.concatenate([[0], np.cumsum(nv)])
    for i in range(0, n, 600):
        got = [(int(hole[c]), xy[vo[c]:vo[c + 1]]) for c in range(off[i], off[i + 1])]
        assert same_contours(got, oracle.gpc_clip(rings_of(A, i), rings_of(B, i), 3)), f"pair {i}"
