"""R-tree build / join / query counters on the GPU, checked bit-exactly
against the oracle (and through it against the reference's fixtures)."""
import os

import numpy as np
import pytest
import torch

import oracle
from conftest import GOLDEN
from helpers import brute_pairs, compare_bu, compare_td, levels_to_bu, levels_to_td
from parlllelrtree_b200 import datagen as dg

pytestmark = pytest.mark.gpu

DT = {"i64": torch.int64, "f32": torch.float32, "f64": torch.float64, "i32": torch.int32}


def boxes_of(kind, n, seed, side=2e-3):
    b = dg.mixture_boxes(n, seed=seed, mean_side=side)
    if kind == "f32":
        return b
    if kind == "f64":
        return b.astype(np.float64) + np.float64(1e-9) * np.arange(4)
    if kind == "i64":
        return dg.quantise(b)
    return dg.quantise(b).astype(np.int32)


def check_levels(tree, ref_levels):
    assert tree.levels == len(ref_levels)
    for l in range(tree.levels):
        got = tree.level_mbr(l)
        assert np.array_equal(got, ref_levels[l]), f"level {l}"


@pytest.mark.parametrize("kind", ["f32", "f64", "i64", "i32"])
@pytest.mark.parametrize("F", [10, 16, 32])
@pytest.mark.parametrize("n", [1, 7, 16, 17, 1000, 70001])
def test_bottomup_morton32(cuda, kind, F, n):
    import parlllelrtree_b200 as prt

    b = boxes_of(kind, n, seed=n + F)
    keys, _ = oracle.keys_morton32(b)
    perm = oracle.stable_argsort(keys)
    lv = oracle.pack(b, F, perm)
    t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=F, key_mode="morton32")
    check_levels(t, lv)
    assert np.array_equal(t.leaf_order().cpu().numpy(), perm)


@pytest.mark.parametrize("F", [10, 16, 32])
def test_bottomup_ref64_golden(cuda, F):
    """The reference's own BU node array (golden fixture) from the device build."""
    import parlllelrtree_b200 as prt

    g = np.load(os.path.join(GOLDEN, f"bu_m{F}.npz"))
    rects = g["rects"]
    t = prt.build_bottomup(torch.from_numpy(rects).cuda(), fanout=F, key_mode="ref64")
    assert np.array_equal(t.leaf_order().cpu().numpy(), g["sorted_ids"])
    ex = t.export_bu()
    sx, sy = rects[:, 0].min(), rects[:, 1].min()
    ex["mbr"] = ex["mbr"] - np.array([sx, sy, sx, sy], np.float64)  # the reference stores shifted boxes
    compare_bu(ex, {k: g[k] for k in ("flag", "num", "mbr", "children", "data")} | {"root": int(g["root"])})
    sh = rects - np.array([sx, sy, sx, sy])
    d = t.digests(torch.from_numpy(rects).cuda())
    assert d == tuple(int(x) for x in g["digests"][:4])


@pytest.mark.parametrize("F", [10, 16, 32])
def test_topdown_golden(cuda, F):
    import parlllelrtree_b200 as prt

    g = np.load(os.path.join(GOLDEN, f"td_m{F}.npz"))
    rects = g["rects"]
    t = prt.build_topdown(torch.from_numpy(rects).cuda(), fanout=F)
    compare_td(t.export_td(), {k: g[k] for k in ("nodes_index", "nodes_mbr", "offsets")})
    d = t.digests(torch.from_numpy(rects).cuda(), td_slots=True)
    assert d == tuple(int(x) for x in g["digests"][:4])


@pytest.mark.parametrize("kind", ["f32", "f64", "i64", "i32"])
@pytest.mark.parametrize("F", [10, 16, 32])
@pytest.mark.parametrize("n", [1, 10, 11, 5000, 40000])
def test_topdown(cuda, kind, F, n):
    import parlllelrtree_b200 as prt

    b = boxes_of(kind, n, seed=7 * n + F)
    perm = oracle.td_order(b, F)
    lv = oracle.pack(b, F, perm)
    t = prt.build_topdown(torch.from_numpy(b).cuda(), fanout=F)
    check_levels(t, lv)
    assert np.array_equal(t.leaf_order().cpu().numpy(), perm)
    compare_td(t.export_td(), levels_to_td(lv, F))
    compare_bu(t.export_bu(), levels_to_bu(lv, F, perm))


@pytest.mark.parametrize("kind", ["f32", "i64"])
@pytest.mark.parametrize("F", [2, 4, 8])
@pytest.mark.parametrize("n", [1, 5000, 40000])
def test_small_fanouts(cuda, kind, F, n):
    """Fanouts below 10: many short-run levels (at F=2 more than one
    shared-memory launch holds), the last level's runs of F records sorted by
    counting ranks; bottom-up and top-down both bit-exact against the oracle."""
    import parlllelrtree_b200 as prt

    b = boxes_of(kind, n, seed=11 * n + F)
    perm = oracle.td_order(b, F)
    lv = oracle.pack(b, F, perm)
    t = prt.build_topdown(torch.from_numpy(b).cuda(), fanout=F)
    check_levels(t, lv)
    assert np.array_equal(t.leaf_order().cpu().numpy(), perm)
    compare_td(t.export_td(), levels_to_td(lv, F))
    modes = [("morton32", oracle.keys_morton32(b)[0])]
    if kind == "i64":
        modes.append(("ref64", oracle.keys_ref64(b)[0]))
    for mode, keys in modes:
        perm_bu = oracle.stable_argsort(keys)
        tb = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=F, key_mode=mode)
        assert np.array_equal(tb.leaf_order().cpu().numpy(), perm_bu)
        check_levels(tb, oracle.pack(b, F, perm_bu))


def test_sort_stability_many_ties(cuda):
    """Heavy key ties: the leaf order must keep input order inside each tie."""
    import parlllelrtree_b200 as prt

    rng = np.random.default_rng(3)
    c = rng.integers(0, 8, size=(300000, 2)).astype(np.float32)
    b = np.concatenate([c, c + 1], axis=1).astype(np.float32)
    keys, _ = oracle.keys_morton32(b)
    perm = oracle.stable_argsort(keys)
    t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=16)
    assert np.array_equal(t.leaf_order().cpu().numpy(), perm)


@pytest.mark.parametrize("kind", ["f32", "i64"])
@pytest.mark.parametrize("F", [10, 16, 32])
@pytest.mark.parametrize("build", ["bottomup", "topdown"])
def test_join_pairs_exact(cuda, kind, F, build):
    import parlllelrtree_b200 as prt

    b = boxes_of(kind, 20000, seed=F, side=4e-3)
    q = boxes_of(kind, 3000, seed=F + 100, side=8e-3)
    fn = prt.build_bottomup if build == "bottomup" else prt.build_topdown
    t = fn(torch.from_numpy(b).cuda(), fanout=F)
    pairs = t.join(torch.from_numpy(q).cuda(), sorted=True).cpu().numpy()
    lv = t.levels_mbr()
    ref = oracle.join_pairs(lv, F, q)
    # sorted by (query, leaf); the oracle's DFS order per query is increasing leaf
    ref = ref[np.lexsort((ref[:, 0], ref[:, 1]))]
    assert np.array_equal(pairs.astype(np.int64), ref)
    # and the candidate set equals the brute-force box intersection set
    perm = t.leaf_order().cpu().numpy()
    got = {(int(perm[a]), int(qq)) for a, qq in pairs}
    assert got == brute_pairs(b, q)


def test_join_empty_and_edge(cuda):
    import parlllelrtree_b200 as prt

    b = np.array([[0, 0, 1, 1], [2, 2, 3, 3]], np.float32)
    t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=16)
    q = np.array([[1, 1, 2, 2], [5, 5, 6, 6], [-1, -1, -0.5, -0.5]], np.float32)  # touching both, none, none
    p = t.join(torch.from_numpy(q).cuda(), sorted=True).cpu().numpy()
    assert p.tolist() == [[0, 0], [1, 0]] or p.tolist() == [[1, 0], [0, 0]]
    assert len(t.join(torch.zeros((0, 4), dtype=torch.float32).cuda())) == 0


@pytest.mark.parametrize("F", [10, 16, 32])
def test_query_counts_match_oracle(cuda, F):
    import parlllelrtree_b200 as prt

    b = boxes_of("i64", 30000, seed=F + 5, side=3e-3)
    for build, td in (("bottomup", False), ("topdown", True)):
        fn = prt.build_bottomup if build == "bottomup" else prt.build_topdown
        t = fn(torch.from_numpy(b).cuda(), fanout=F)
        got = t.query_counts(torch.from_numpy(b).cuda(), td_slots=td).cpu().numpy()
        ref = oracle.query_counts(t.levels_mbr(), F, b, td_slots=td)
        assert np.array_equal(got, ref)


def test_large_build_parity(cuda):
    """2M float32 boxes: levels and leaf order bit-exact, bottom-up and top-down."""
    import parlllelrtree_b200 as prt

    b = dg.mixture_boxes(2_000_000, seed=0)
    keys, _ = oracle.keys_morton32(b)
    perm = oracle.stable_argsort(keys)
    t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=16)
    assert np.array_equal(t.leaf_order().cpu().numpy(), perm)
    check_levels(t, oracle.pack(b, 16, perm))
    perm = oracle.td_order(b, 32)
    t = prt.build_topdown(torch.from_numpy(b).cuda(), fanout=32)
    assert np.array_equal(t.leaf_order().cpu().numpy(), perm)


@pytest.mark.parametrize("kind", ["f32", "f64", "i64", "i32"])
@pytest.mark.parametrize("F", [2, 3, 10, 16, 32])
@pytest.mark.parametrize("n", [1, 33, 4097, 30011])
def test_windows_that_contain_nodes(cuda, kind, F, n):
    """Windows from a point to more than the whole extent, so that nodes of
    every level lie inside some: pairs (one call, and into a given capacity)
    and counters against the oracle; then with records that intersect nothing
    (an empty polygon's box) inside their parents' boxes."""
    import parlllelrtree_b200 as prt

    rng = np.random.default_rng(n + F)
    scale = 1.0 if kind in ("f32", "f64") else 1e4
    dt = {"f32": np.float32, "f64": np.float64, "i64": np.int64, "i32": np.int32}[kind]
    c, h = rng.random((n, 2)), rng.random((n, 2)) * 0.01
    b = (np.concatenate([c - h, c + h], 1) * scale).astype(dt)
    m = 300
    c, h = rng.random((m, 2)), rng.random((m, 1)) ** 3 * 1.2
    q = (np.concatenate([c - h, c + h], 1) * scale).astype(dt)
    for improper in (False, True):
        if improper:
            big = np.finfo(dt).max if dt in (np.float32, np.float64) else np.iinfo(dt).max
            b[:: max(1, n // 5)] = np.array([big, big, -big, -big], dt)
        t = prt.build_topdown(torch.from_numpy(b).cuda(), fanout=F)
        lv = t.levels_mbr()
        qd = torch.from_numpy(q).cuda()
        ref = oracle.join_pairs(lv, F, q)
        ref = ref[np.lexsort((ref[:, 0], ref[:, 1]))]
        for got in (t.join(qd), t.join(qd, sorted=True), t.join(qd, cap=len(ref) + 7, sorted=True)):
            assert np.array_equal(got.cpu().numpy().astype(np.int64).reshape(-1, 2), ref.reshape(-1, 2))
        un = t.join(qd, cap=len(ref) + 7).cpu().numpy().astype(np.int64).reshape(-1, 2)
        assert np.array_equal(un[np.lexsort((un[:, 0], un[:, 1]))], ref.reshape(-1, 2))
        for td in (False, True):
            assert np.array_equal(t.query_counts(qd, td_slots=td).cpu().numpy(), oracle.query_counts(lv, F, q, td_slots=td))


@pytest.mark.parametrize("kind", ["f32", "f64", "i64", "i32"])
@pytest.mark.parametrize("F,n", [(10, 4097), (10, 20001), (17, 4914), (17, 83522), (16, 65537), (3, 50000),
                                 (10, 200001), (31, 30000)])
def test_topdown_run_lengths(cuda, kind, F, n):
    """Levels whose runs are no multiple of the sort's tiles, and sizes at the
    edges of its tile sizes; integers below zero and with the range of the
    whole type, so that the keys take every number of passes."""
    import parlllelrtree_b200 as prt

    rng = np.random.default_rng(F * n)
    dt = {"f32": np.float32, "f64": np.float64, "i64": np.int64, "i32": np.int32}[kind]
    c = rng.random((n, 2)) - 0.3
    for scale in (1.0, 300.0, 1e6) if dt in (np.int64, np.int32) else (1.0,):
        b = np.concatenate([c, c + 0.01], 1) * scale
        b = np.floor(b).astype(dt) if dt in (np.int64, np.int32) else b.astype(dt)
        if scale == 1e6:  # one record far away: 63 (31) significant bits
            b[n // 2, :2] = np.iinfo(dt).min // 2
            b[n // 3, 2:] = np.iinfo(dt).max // 2
            b[n // 3, :2] = np.iinfo(dt).max // 2
        perm = oracle.td_order(b, F)
        t = prt.build_topdown(torch.from_numpy(b).cuda(), fanout=F)
        assert np.array_equal(t.leaf_order().cpu().numpy(), perm)
        check_levels(t, oracle.pack(b, F, perm))


@pytest.mark.parametrize("kind", ["f32", "f64", "i64", "i32"])
@pytest.mark.parametrize("F", [2, 10, 16, 31, 32])
@pytest.mark.parametrize("shape", ["even", "32 equal", "33 equal", "skewed", "one value"])
def test_topdown_buckets(cuda, kind, F, shape):
    """Short runs whose keys fill the buckets evenly, with the largest bucket at the
    limit and one above it, almost all in one bucket, and equal."""
    import parlllelrtree_b200 as prt

    rng = np.random.default_rng(F)
    n = 9001
    if shape == "even":
        c = np.stack([rng.permutation(n), rng.permutation(n)], 1).astype(np.float64)
    elif shape == "one value":
        c = np.full((n, 2), 7.0)
    elif shape == "skewed":
        c = np.round(np.exp(rng.uniform(0, 20, (n, 2))))
    else:
        k = int(shape.split()[0])
        c = np.stack([rng.permutation(n), rng.permutation(n)], 1).astype(np.float64)
        c[rng.choice(n, k, replace=False)] = 4000.0
    dt = {"f32": np.float32, "f64": np.float64, "i64": np.int64, "i32": np.int32}[kind]
    b = np.concatenate([c, c + 1], 1).astype(dt)
    perm = oracle.td_order(b, F)
    t = prt.build_topdown(torch.from_numpy(b).cuda(), fanout=F)
    assert np.array_equal(t.leaf_order().cpu().numpy(), perm)
    check_levels(t, oracle.pack(b, F, perm))


@pytest.mark.parametrize("kind", ["f32", "f64", "i64", "i32"])
@pytest.mark.parametrize("F", [2, 3, 16, 32])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 1024, 1025, 4096, 6143, 6144, 6145, 8191, 8192, 8193])
def test_one_block_build(cuda, kind, F, n):
    """Sizes at the edges of the one-block build (rows of 1,024 records, its
    largest sizes for 32- and 64-bit coordinates), with ties and given ids."""
    import parlllelrtree_b200 as prt

    b = boxes_of(kind, n, seed=n + F)
    b[n // 3: n // 2] = b[n // 3]  # a run of equal boxes keeps its order
    keys, _ = oracle.keys_morton32(b)
    perm = oracle.stable_argsort(keys)
    ids = np.arange(n, dtype=np.int32)[::-1].copy()
    t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=F, ids=ids)
    assert np.array_equal(t.leaf_order().cpu().numpy(), ids[perm])
    check_levels(t, oracle.pack(b, F, perm))


@pytest.mark.parametrize("kind", ["f32", "f64", "i64"])
@pytest.mark.parametrize("equal", [32, 33, 5000])
@pytest.mark.parametrize("n", [40, 5000, 6144, 8192])
def test_one_block_buckets(cuda, kind, equal, n):
    """One-block builds whose largest bucket is at the limit of the counting, one
    above it, and almost all of the boxes."""
    import parlllelrtree_b200 as prt

    b = boxes_of(kind, n, seed=n + equal)
    rng = np.random.default_rng(n * equal)
    b[rng.choice(n, min(n, equal), replace=False)] = b[0]
    t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=16)
    perm = oracle.stable_argsort(oracle.keys_morton32(b)[0])
    assert np.array_equal(t.leaf_order().cpu().numpy(), perm)
    check_levels(t, oracle.pack(b, 16, perm))


def windows(kind, n, seed):
    """Small windows, some points, a hundred large ones and one around everything."""
    rng = np.random.default_rng(seed)
    c, half = rng.random((n, 2)), 10.0 ** rng.uniform(-5, -2, (n, 1))
    half[: n // 100] = 0.0
    half[n // 100: n // 100 + 100] = 0.2
    half[n // 2] = 2.0
    q = np.concatenate([c - half, c + half], 1)
    return q.astype(np.float32) if kind == "f32" else q if kind == "f64" else np.rint(q * 1e6).astype(
        np.int64 if kind == "i64" else np.int32)


@pytest.mark.parametrize("kind", ["f32", "f64", "i64", "i32"])
@pytest.mark.parametrize("F,n", [(9, 9), (9, 10), (10, 5000), (16, 16), (16, 17), (16, 4097), (17, 3000), (32, 33),
                                 (32, 20000)])
def test_counts_of_many_windows(cuda, kind, F, n):
    """Just under and just over the number of windows from which warps take batches of
    them, trees of one level and more, with and without a record that intersects
    nothing, against the oracle."""
    import parlllelrtree_b200 as prt

    q = windows(kind, 131_072 + 77, F)
    b = boxes_of(kind, n, seed=F + n, side=3e-3)
    for improper in (False, True):
        if improper:
            b[n // 2, 0], b[n // 2, 2] = b[n // 2, 2] + 1, b[n // 2, 0] - 1
        t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=F)
        lv = t.levels_mbr()
        for td in (False, True):
            ref = oracle.query_counts(lv, F, q, td_slots=td)
            for m in (131_071, 131_072, len(q)):
                got = t.query_counts(torch.from_numpy(q[:m]).cuda(), td_slots=td).cpu().numpy()
                assert np.array_equal(got, ref[:m]), (improper, td, m)


@pytest.mark.parametrize("kind", ["f32", "i64"])
@pytest.mark.parametrize("F", [10, 16, 32])
@pytest.mark.parametrize("nq", [1, 300, 443, 444, 591, 592, 700])
def test_counts_of_few_long_windows(cuda, kind, F, nq):
    """Windows across the whole extent and around everything, on a tree that cannot be
    pruned and on one that can, around the numbers of windows up to which long walks
    are handed on early: what a launch leaves, once and again."""
    import parlllelrtree_b200 as prt

    n = 60_000
    rng = np.random.default_rng(nq)
    y = rng.random(nq)
    q = np.stack([np.full(nq, -1.0), y, np.full(nq, 2.0), y + 1e-3], 1)
    q[nq // 2] = [-1, -1, 2, 2]
    q[:: 7, 3] += 0.05
    q = q.astype(np.float32) if kind == "f32" else np.rint(q * 1e6).astype(np.int64)
    b = boxes_of(kind, n, seed=F, side=1e-3)
    for improper in (True, False):
        if not improper:
            b[n // 2] = b[0]
        else:
            b[n // 2, 0], b[n // 2, 2] = b[n // 2, 2] + 1, b[n // 2, 0] - 1
        t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=F)
        got = t.query_counts(torch.from_numpy(q).cuda()).cpu().numpy()
        assert np.array_equal(got, oracle.query_counts(t.levels_mbr(), F, q)), improper


@pytest.mark.parametrize("F", [2, 4, 5])
@pytest.mark.parametrize("nq", [65_535, 65_536])
def test_unsorted_joins_of_small_nodes(cuda, F, nq):
    """The line between one traversal in order and two in none, with and without
    pairs, against the oracle."""
    import parlllelrtree_b200 as prt

    b = boxes_of("f32", 3000, seed=F, side=3e-3)
    q = windows("f32", nq, 3)
    t = prt.build_bottomup(torch.from_numpy(b).cuda(), fanout=F)
    ref = oracle.join_pairs(t.levels_mbr(), F, q)
    ref = ref[np.lexsort((ref[:, 0], ref[:, 1]))]
    for srt in (False, True):
        got = t.join(torch.from_numpy(q).cuda(), sorted=srt).cpu().numpy().astype(np.int64)
        if not srt:
            got = got[np.lexsort((got[:, 0], got[:, 1]))]
        assert np.array_equal(got, ref), srt
    assert len(t.join(torch.from_numpy(q + np.float32(9)).cuda())) == 0
