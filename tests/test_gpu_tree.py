"""GPU tree build against the oracle: bit-exact node arrays, leaf lists and point order."""
import numpy as np
import pytest

from conftest import assert_same_tree, make_scan
from oracle import orc

pytestmark = pytest.mark.gpu


def build_both(xyz, st, **params):
    import kd_slam2_b200 as kds
    O = orc.OTree.build(xyz, st, orc.tree_params(**params))
    G = kds.TreeGeneratorB2003D(**params).make_tree(xyz, st)
    return O, G


@pytest.mark.parametrize("seed,beams,params", [
    (2000, 16, dict(leaf_max_points=16)),
    (2001, 16, dict(leaf_max_points=16, propagate_normal=1)),
    (2002, 32, dict()),
    (2003, 64, dict(leaf_max_points=16)),  # 65k points: large-node path
    (2004, 16, dict(leaf_max_points=100, leaf_min_points=5, leaf_min_normal_incidence=0.2, propagate_normal=1,
                    tree_min_good_leaves=50)),
])
def test_tree_build_bit_exact(scene, seed, beams, params):
    xyz, st = make_scan(scene, seed, beams=beams, elev=(-15.0, 15.0) if beams <= 32 else (-22.5, 22.5))
    O, G = build_both(xyz, st, **params)
    assert O.accepted and G is not None
    assert_same_tree(O, G)


def test_forest_build_equals_single_builds(scene):
    """One batched pass over uneven clouds gives each tree bit-identical to its own build."""
    import kd_slam2_b200 as kds
    from kd_slam2_b200 import synth
    clouds = []
    for i, beams in enumerate([16, 32, 16, 64]):
        xyz, st = make_scan(scene, 2300 + i, beams=beams, elev=(-15.0, 15.0),
                            vel=[5.0 * i, 0, 0, 0, 0, 0.1 * i])
        clouds.append((xyz, st + 10.0 * i))
    clouds.insert(2, (np.zeros((3, 3), np.float32), None))  # rejected: fewer than leaf_min_points
    gen = kds.TreeGeneratorB2003D(leaf_max_points=16, propagate_normal=1)
    trees = gen.make_trees(clouds)
    assert trees[2] is None
    for (xyz, st), T in zip(clouds, trees):
        if len(xyz) < 5:
            continue
        O = orc.OTree.build(xyz, st, orc.tree_params(leaf_max_points=16, propagate_normal=1))
        assert_same_tree(O, T)
    # the packed form (kds_tree_build_batch: one array, offsets) gives the same trees
    import ctypes as C
    from kd_slam2_b200 import abi as L
    xyz = np.ascontiguousarray(np.concatenate([c[0] for c in clouds]))
    st = np.ascontiguousarray(np.concatenate([np.zeros(len(c[0])) if c[1] is None else c[1] for c in clouds]))
    off = np.zeros(len(clouds) + 1, np.int64)
    off[1:] = np.cumsum([len(c[0]) for c in clouds])
    hs = (C.c_void_p * len(clouds))()
    status = (C.c_int32 * len(clouds))()
    rc = kds.lib().kds_tree_build_batch(xyz.ctypes.data, st.ctypes.data, off.ctypes.data, len(clouds),
                                        L.KDS_MEM_HOST, C.byref(gen.params), None, hs, status)
    assert rc == L.KDS_OK and status[2] == L.KDS_ERR_TREE_REJECTED
    for i, T in enumerate(trees):
        if T is None:
            continue
        P = kds.Tree(hs[i])
        a, b = T.export(), P.export()
        for k in ("mean", "dir", "dts_mean", "left", "right", "leaves", "perm"):
            assert np.array_equal(a[k], b[k]), (i, k)


def test_tree_build_skewed_scan_with_stamps(scene):
    from kd_slam2_b200 import synth
    xyz, st = make_scan(scene, 2010, beams=32, vel=[10.0, 0, 0, 0, 0, np.deg2rad(30.0)])
    st = st + 1234.5  # absolute stamps: dts relative to the first point
    O, G = build_both(xyz, st, leaf_max_points=16)
    assert_same_tree(O, G)


def test_tree_without_stamps(scene):
    xyz, _ = make_scan(scene, 2011)
    O, G = build_both(xyz, None, leaf_max_points=16)
    assert_same_tree(O, G)


def test_rejected_trees_match_makeTree_nullptr(scene):
    import kd_slam2_b200 as kds
    # fewer points than leaf_min_points
    xyz = np.zeros((3, 3), np.float32)
    assert kds.TreeGeneratorB2003D().make_tree(xyz) is None
    # a tiny patch: too few good leaves for tree_min_good_leaves
    rng = np.random.default_rng(0)
    xyz = (rng.normal(size=(200, 3)) * [1.0, 1.0, 0.01] + [10.0, 0, 0]).astype(np.float32)
    O = orc.OTree.build(xyz, None, orc.tree_params(tree_min_good_leaves=50))
    G = kds.TreeGeneratorB2003D(tree_min_good_leaves=50).make_tree(xyz)
    assert not O.accepted and G is None


def test_degenerate_inputs(scene):
    """duplicated points and collinear runs: deterministic, same as the oracle"""
    xyz, st = make_scan(scene, 2012)
    dup = np.concatenate([xyz, xyz[:3000], np.repeat(xyz[:5], 40, axis=0)]).astype(np.float32)
    std = np.concatenate([st, st[:3000], np.repeat(st[:5], 40)])
    line = np.stack([np.linspace(5, 15, 500), np.full(500, 3.0), np.full(500, 0.5)], 1).astype(np.float32)
    allp = np.concatenate([dup, line]).astype(np.float32)
    alls = np.concatenate([std, np.zeros(500)])
    O, G = build_both(allp, alls, leaf_max_points=16)
    assert_same_tree(O, G)


@pytest.mark.parametrize("clouds,points,extra", [(3000, 9, 0), (4000, 20, 300), (290, 20, 300)])
def test_many_tiny_clouds(clouds, points, extra):
    """Subtree passes whose sums, or whose counts, have no room in the build's workspace (very
    many very small subtrees): the trees equal the oracle's all the same."""
    import kd_slam2_b200 as kds
    rng = np.random.default_rng(clouds)
    sizes = [points] * clouds + ([extra] if extra else [])
    made = [((rng.normal(size=(n, 3)) * [2.0, 2.0, 0.02] + [12.0, 0, 1.0]).astype(np.float32),
             np.sort(rng.uniform(0, 0.1, n))) for n in sizes]
    prm = dict(leaf_max_points=8, leaf_min_points=3, tree_min_good_leaves=1)
    trees = kds.TreeGeneratorB2003D(**prm).make_trees(made)
    for i in sorted(set(rng.integers(0, len(made), 60)) | {0, len(made) - 1}):
        O = orc.OTree.build(*made[i], orc.tree_params(**prm))
        assert O.accepted == (trees[i] is not None)
        if O.accepted:
            assert_same_tree(O, trees[i])


@pytest.mark.parametrize("clusters,pile,fits", [
    (60, 0, True),        # a subtree pass from the first level
    (60, 3000, True),     # the pile of equal points keeps the level kernels running to the last level
    (200, 0, False),      # too many nodes: in the subtree pass by blocks
    (30000, 0, False),    # ... by warps
    (40000, 600, False),  # in the level kernels of small nodes, some levels before the host looks
    (2000, 3000, False),  # ... with a large node beside them
    (5000, 70000, False),
])
def test_clouds_of_equal_points(clusters, pile, fits):
    """More than leaf_max_points equal points split at every level down to max_level, with one
    empty child each: the trees equal the oracle's while their nodes fit the build's arrays,
    and the build reports KDS_ERR_CAPACITY (and goes on to work) where they don't."""
    import kd_slam2_b200 as kds
    rng = np.random.default_rng(clusters + pile)
    xyz = np.repeat(rng.uniform(-40.0, 40.0, (clusters, 3)).astype(np.float32), 20, axis=0)
    xyz = np.concatenate([rng.permutation(xyz), np.zeros((pile, 3), np.float32)])
    gen = kds.TreeGeneratorB2003D(leaf_max_points=16, tree_min_good_leaves=1)
    if fits:
        O = orc.OTree.build(xyz, None, orc.tree_params(leaf_max_points=16, tree_min_good_leaves=1))
        G = gen.make_tree(xyz)
        assert O.accepted == (G is not None)
        if G is not None:
            assert_same_tree(O, G)
        return
    with pytest.raises(kds.KdsError) as ei:
        gen.make_tree(xyz)
    assert ei.value.code == kds.abi.KDS_ERR_CAPACITY
    assert gen.make_tree(rng.uniform(-40.0, 40.0, (5000, 3)).astype(np.float32)) is not None


def test_out_of_range_input_is_rejected_with_status():
    import kd_slam2_b200 as kds
    xyz = np.zeros((100, 3), np.float32)
    xyz[5] = [1e6, 0, 0]
    with pytest.raises(kds.KdsError) as ei:
        kds.TreeGeneratorB2003D().make_tree(xyz)
    assert ei.value.code == kds.abi.KDS_ERR_RANGE


def test_import_export_roundtrip(scene):
    import kd_slam2_b200 as kds
    xyz, st = make_scan(scene, 2013)
    O = orc.OTree.build(xyz, st, orc.tree_params(leaf_max_points=16))
    e = O.export()
    T = kds.Tree.import_nodes(e["mean"], e["dir"], e["left"], e["right"], e["dts_mean"], e["dts_cov"], e["start"],
                              e["end"], ts_start=e["ts_start"])
    g = T.export()
    for k in ("mean", "dir", "left", "right", "dts_mean", "dts_cov", "start", "end", "leaves"):
        assert np.array_equal(e[k], g[k]), k
    # malformed: child index pointing backwards
    bad = e["left"].copy()
    bad[5] = 1
    with pytest.raises(kds.KdsError) as ei:
        kds.Tree.import_nodes(e["mean"], e["dir"], bad, e["right"])
    assert ei.value.code == kds.abi.KDS_ERR_BAD_TREE


def test_morph_and_isometry_match_oracle(scene):
    import kd_slam2_b200 as kds
    xyz, st = make_scan(scene, 2014, vel=[5.0, 0.5, 0, 0.01, 0, 0.4])
    G = kds.TreeGeneratorB2003D(leaf_max_points=16).make_tree(xyz, st)
    e0 = G.export()
    v = np.array([5.0, 0.5, 0.1, 0.01, -0.02, 0.4], np.float32)
    G.apply_velocities_in_place(v)
    e1 = G.export()
    for i in range(0, len(e0["mean"]), 7):
        mo, no = orc.warp_leaf(v, np.float32(e0["dts_mean"][i]), e0["mean"][i], e0["dir"][i])
        assert np.array_equal(mo.view(np.uint32), e1["mean"][i].view(np.uint32))
        assert np.array_equal(no.view(np.uint32), e1["dir"][i].view(np.uint32))
    # leaves only skipped when asked
    G2 = kds.TreeGeneratorB2003D(leaf_max_points=16).make_tree(xyz, st)
    G2.apply_velocities_in_place(v, skip_leaves=True)
    e2 = G2.export()
    assert np.array_equal(e2["mean"][e2["leaves"]], e0["mean"][e0["leaves"]])
    # rigid transform: applyIsometry_ row loop
    from kd_slam2_b200 import synth
    X = synth.pose((1.0, -2.0, 0.3), (0.1, 0.2, -0.3)).astype(np.float32)
    G3 = kds.TreeGeneratorB2003D(leaf_max_points=16).make_tree(xyz, st)
    G3.apply_isometry_in_place(X)
    e3 = G3.export()
    m = e0["mean"][10]
    ref = np.float32(X[:, 3])
    for c in range(3):
        ref = (ref + (X[:, c] * m[c]).astype(np.float32)).astype(np.float32)
    assert np.array_equal(ref.view(np.uint32), e3["mean"][10].view(np.uint32))
    L = G3.extract_compressed_leaves()
    assert np.array_equal(L[:, :3], e3["mean"][e3["leaves"]])
    # into a device buffer: the same values, with and without a morph
    import torch
    D = torch.empty((G3.num_leaves, 6), dtype=torch.float32, device="cuda")
    G3.extract_compressed_leaves_device(D)
    torch.cuda.synchronize()
    assert np.array_equal(D.cpu().numpy(), L)
    G3.extract_compressed_leaves_device(D, v=v)
    torch.cuda.synchronize()
    assert np.array_equal(D.cpu().numpy(), G3.extract_compressed_leaves(v))


def test_tree_build_bit_exact_on_stream_scans():
    """Scans of the served-registration trace (moving sensors, skewed stamps)."""
    from kd_slam2_b200 import streams
    tr = streams.make_trace(7, num_streams=4, scans_per_stream=2, saturate=True, beam_mix=(16, 32), map_scans=2)
    for r in tr.requests:
        O, G = build_both(r.xyz, r.stamps, leaf_max_points=16)
        assert O.accepted and G is not None
        assert_same_tree(O, G)
    for s in tr.streams:  # the initial maps, world frame, no stamps
        O, G = build_both(s.map_xyz, None, leaf_max_points=16)
        assert_same_tree(O, G)


def test_tree_build_bit_exact_near_the_origin():
    """Many tiny products of mixed sign: the fixed-point floor of small negative values
    (where 1 - |v| does not fit a double) must agree between the GPU and the oracle."""
    rng = np.random.default_rng(21)
    n = 20000
    xyz = np.empty((n, 3), np.float32)
    xyz[:, 0] = rng.uniform(-0.05, 0.05, n)
    xyz[:, 1] = rng.uniform(-0.05, 0.05, n)
    xyz[:, 2] = -1.0 + rng.normal(scale=1e-4, size=n)  # a plane 1 m below the sensor
    st = rng.uniform(0.0, 0.1, n)
    O, G = build_both(xyz, st, leaf_max_points=16, leaf_density=0.0)
    assert O.accepted and G is not None
    assert_same_tree(O, G)


@pytest.mark.parametrize("sizes", [
    [1024, 1025, 2048, 2049, 1023] * 60,   # 300 roots around one and two chunks: several list batches per block
    [300_001, 7, 1025, 65_537],            # one root of many chunks beside ragged small ones
])
def test_large_node_chunk_lists(scene, sizes):
    """The large-node lists at their edges: roots of one chunk and one point more, more large
    roots than a block has threads, and chunk counts far above a block's threads."""
    import kd_slam2_b200 as kds
    xyz, st = make_scan(scene, 2450, beams=128, cols=4096, elev=(-22.5, 22.5))
    rng = np.random.default_rng(7)
    clouds = []
    for n in sizes:
        k = np.sort(rng.choice(len(xyz), n, replace=False))
        clouds.append((np.ascontiguousarray(xyz[k]), np.ascontiguousarray(st[k])))
    trees = kds.TreeGeneratorB2003D(leaf_max_points=16).make_trees(clouds)
    for (x, s), T in zip(clouds, trees):
        if len(x) < 100:
            assert T is None
            continue
        assert_same_tree(orc.OTree.build(x, s, orc.tree_params(leaf_max_points=16)), T)


@pytest.mark.parametrize("n", [1000, 1025, 40_000])
def test_exact_sums_off_the_grid(n):
    """Coordinates on both sides of the sums' 2^-40 grid (nonzero below 2^-17, down to
    denormals), exact zeros and values up to the range limit, with and without stamps: every
    node equals the oracle's bit for bit."""
    import kd_slam2_b200 as kds
    rng = np.random.default_rng(n)
    xyz = (rng.normal(size=(n, 3)) * [20.0, 8.0, 0.01]).astype(np.float32)
    k = rng.integers(0, n, n // 8)
    xyz[k, 2] = np.ldexp(rng.uniform(-1, 1, len(k)), rng.integers(-150, -14, len(k))).astype(np.float32)
    xyz[rng.integers(0, n, n // 16), 1] = 0.0
    xyz[rng.integers(0, n, n // 16), 0] = np.float32(2.0**-17)
    xyz[rng.integers(0, n, 5)] = [32767.996, -32767.0, 30000.5]
    st = np.sort(rng.uniform(0, 40_000.0, n))
    st[: n // 2] *= 1e-9
    prm = dict(leaf_max_points=16, tree_min_good_leaves=1)
    for s in (None, st, np.full(n, 7.25)):
        O, G = build_both(xyz, s, **prm)
        assert_same_tree(O, G)


@pytest.mark.parametrize("n", [2047, 2048, 2049, 4096])
def test_stamp_prefix_tiles(scene, n):
    """Point counts at the edges of the stamp prefix's tiles, in one forest with differing
    first stamps."""
    import kd_slam2_b200 as kds
    xyz, st = make_scan(scene, 2460, beams=32, vel=[8.0, 0, 0, 0, 0, 0.2])
    clouds = [(xyz[:n], st[:n] + 5.0), (xyz[n:2 * n + 1], st[n:2 * n + 1])]
    for (x, s), T in zip(clouds, kds.TreeGeneratorB2003D(leaf_max_points=16).make_trees(clouds)):
        assert_same_tree(orc.OTree.build(x, s, orc.tree_params(leaf_max_points=16)), T)
    assert_same_tree(*build_both(xyz[:n], st[:n], leaf_max_points=16))


@pytest.mark.parametrize("n,params", [
    (255, {}), (256, {}), (257, {}), (1024, {}), (2047, {}), (2048, {}), (2049, {}), (4097, {}),
    (2048, dict(leaf_max_points=3, leaf_min_points=3, leaf_density=1e9, tree_min_good_leaves=1)),
    (2048, dict(leaf_max_points=16, propagate_normal=1, max_level=5, tree_min_good_leaves=1)),
])
def test_subtree_pass_sizes(scene, n, params):
    """Clouds at the edges of the shared-memory subtree passes (256 and 2,048 points), down to
    leaves of three points (the most nodes per depth) and with a level limit inside the pass."""
    xyz, st = make_scan(scene, 2470, beams=64, elev=(-22.5, 22.5), vel=[5.0, 0, 0, 0, 0, 0.1])
    k = np.sort(np.random.default_rng(n).choice(len(xyz), n, replace=False))
    prm = dict(dict(leaf_max_points=16, tree_min_good_leaves=1), **params)
    O, G = build_both(np.ascontiguousarray(xyz[k]), np.ascontiguousarray(st[k]), **prm)
    assert_same_tree(O, G)


@pytest.mark.parametrize("clouds", [295, 296, 297, 330])
def test_subtree_pass_roots(scene, clouds):
    """Forests at the edge of the block form's number of subtrees (296)."""
    import kd_slam2_b200 as kds
    xyz, st = make_scan(scene, 2471, beams=32)
    rng = np.random.default_rng(clouds)
    cs = []
    for i in range(clouds):
        k = np.sort(rng.choice(len(xyz), int(rng.integers(300, 1200)), replace=False))
        cs.append((np.ascontiguousarray(xyz[k]), np.ascontiguousarray(st[k])))
    prm = dict(leaf_max_points=16, tree_min_good_leaves=1)
    for (x, s), T in zip(cs, kds.TreeGeneratorB2003D(**prm).make_trees(cs)):
        assert_same_tree(orc.OTree.build(x, s, orc.tree_params(**prm)), T)
