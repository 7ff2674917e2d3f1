"""Batched bundle-adjustment pairs (kds_batch_run) and the launch autotuner.

* Every pair of the batch -- rigid and CT-ICP, uneven sizes, one graph-captured launch
  sequence -- gives the result of its own kds_aligner_compute, bit for bit.
* The autotuner's configurations (tree-top staging, job order, per-iteration launches
  with one or two tiles per block, or one persistent launch over a device work queue)
  change the launch shape only:
  results are identical under the chosen one and under every other one.
"""
import numpy as np
import pytest

import kd_slam2_b200 as kds
from kd_slam2_b200 import synth

pytestmark = pytest.mark.gpu

TREE = dict(leaf_max_points=16)
ICP = dict(max_error=0.5, max_iterations=10)
CT = dict(max_error=0.5, max_iterations=15, velocity_damping=10.0)


@pytest.fixture(scope="module")
def workload():
    from kd_slam2_b200 import ba
    wl = ba.make_workload(seed=9, num_keyframes=10, min_pts=8000, max_pts=40000, beams=64, cols=1024)
    trees = ba.build_trees(wl, TREE)
    assert all(t is not None for t in trees)
    return wl, trees


def outputs(arr):
    return [(int(j.result), np.array(j.X[:]), np.array(j.v[:]), j.stats.num_inliers) for j in arr]


def same(a, b):
    for (ra, Xa, va, na), (rb, Xb, vb, nb) in zip(a, b):
        assert ra == rb and na == nb
        assert np.array_equal(Xa, Xb)
        assert np.array_equal(va, vb)


def test_batch_equals_per_pair_compute(workload):
    from kd_slam2_b200 import ba
    wl, trees = workload
    jobs = ba.jobs(wl, trees, ICP, CT)
    assert len(jobs) >= 8 and {p.kind for p in wl.pairs} == {0, 1}
    res = outputs(kds.Batch().run(jobs, use_graph=True))
    for p, (r, X, v, n) in zip(wl.pairs, res):
        a = kds.CTICPB2003D(**CT) if p.kind == 1 else kds.ICPB2003D(**ICP)
        a.set_fixed(trees[p.i])
        a.set_moving(trees[p.j])
        a.set_x(p.X0)
        if p.kind == 1:
            a.set_fixed_velocities(wl.keyframes[p.i].vel)
            a.set_velocities(wl.keyframes[p.j].vel)
        assert a.compute() == r
        assert np.array_equal(np.asarray(a.get_x()).reshape(12), X)
        if p.kind == 1:
            assert np.array_equal(a.velocities(), v)


def test_autotune_keeps_results(workload):
    from kd_slam2_b200 import ba
    wl, trees = workload
    jobs = ba.jobs(wl, trees, ICP, CT)
    ref = outputs(kds.Batch().run(jobs))
    b = kds.Batch()
    chosen, ms = b.autotune(jobs)
    assert 0 <= chosen < 18 and np.all(ms > 0)
    same(ref, outputs(b.run(jobs)))
    same(ref, outputs(b.run(jobs)))  # graph replay


@pytest.mark.parametrize("config", list(range(18)))
def test_every_configuration_gives_identical_results(workload, config):
    """Each launch configuration -- the persistent one included, whose blocks wait for a
    job's previous iteration on the device, and the two-tile blocks -- gives every job
    bit-identical results, run directly and replayed from its graph."""
    from kd_slam2_b200 import ba
    wl, trees = workload
    jobs = ba.jobs(wl, trees, ICP, CT)
    ref = outputs(kds.Batch().run(jobs, use_graph=False))
    b = kds.Batch()
    b.configure(config)
    for _ in range(3):  # direct, graph capture, graph replay
        same(ref, outputs(b.run(jobs, use_graph=True)))


@pytest.mark.parametrize("first,then", [((2, 2), (3, 1)), ((3, 1), (2, 2)), ((3, 3, 1), (4, 2, 1))])
@pytest.mark.parametrize("kind", ["icp", "ct"])
def test_two_tile_blocks_of_another_split_of_the_same_tiles(workload, first, then, kind):
    """With two tiles per block, batches of as many jobs, tiles and iterations can need different
    numbers of blocks: the graph of one must not be replayed for the other."""
    _, trees = workload
    cls, code = (kds.CTICPB2003D, kds.abi.KDS_CTICP) if kind == "ct" else (kds.ICPB2003D, kds.abi.KDS_ICP)
    prm = CT if kind == "ct" else ICP
    fixed, e = trees[0], trees[1].export()
    leaf = e["leaves"]

    def moving(tiles):  # a left-deep chain of 128 surfels a tile, the last one not full
        n = 128 * tiles - 5
        m, d = np.zeros((2 * n - 1, 3), np.float32), np.tile(np.float32([0, 0, 1]), (2 * n - 1, 1))
        left, right = np.full(2 * n - 1, -1, np.int32), np.full(2 * n - 1, -1, np.int32)
        inner = np.arange(0, 2 * n - 2, 2)
        left[inner], right[inner] = inner + 1, inner + 2
        m[left < 0], d[left < 0] = e["mean"][np.resize(leaf, n)], e["dir"][np.resize(leaf, n)]
        return kds.Tree.import_nodes(m, d, left, right)
    made = {t: moving(t) for t in set(first + then)}
    a = cls(**prm)
    X0 = [synth.pose((0.03 * k, 0.02, 0.0), (0.0, 0.0, 0.004 * k)) for k in range(len(first))]
    alone = {}
    for t in made:
        for k, X in enumerate(X0):
            a.set_fixed(fixed)
            a.set_moving(made[t])
            a.set_x(X)
            a.set_velocities(np.zeros(6))
            r = a.compute()
            alone[t, k] = (r, a.get_x().reshape(12), a.velocities(), a.stats["num_inliers"])
    b = kds.Batch()
    b.configure(12)  # two tiles per block
    for tiles in (first, first, first, then, then, then):  # direct, captured, replayed
        out = b.run([kds.make_job(code, fixed, made[t], a.params, X=X) for t, X in zip(tiles, X0)])
        same([alone[t, k] for k, t in enumerate(tiles)], outputs(out))


def test_batches_on_streams_of_other_priorities(workload):
    """A mixed batch's second stream follows the priority of the caller's: the same results on
    streams of either priority in turn, and on the default stream."""
    import torch

    from kd_slam2_b200 import ba
    wl, trees = workload
    jobs = ba.jobs(wl, trees, ICP, CT)
    ref = outputs(kds.Batch().run(jobs, use_graph=False))
    b = kds.Batch()
    streams = [torch.cuda.Stream(priority=p).cuda_stream for p in (0, -1)] + [None]
    for k in range(7):
        same(ref, outputs(b.run(jobs, use_graph=k % 2 == 1, stream=streams[k % 3])))


def test_autotune_as_first_use_of_the_library(tmp_path):
    """In a fresh process, the autotuner's staged configurations opt the kernels into their
    shared memory themselves (no earlier launch did it)."""
    import subprocess
    import sys

    from conftest import ROOT
    code = (
        "import sys; sys.path.insert(0, %r)\n"
        "import kd_slam2_b200 as kds\n"
        "from kd_slam2_b200 import ba\n"
        "wl = ba.make_workload(seed=3, num_keyframes=4, min_pts=8000, max_pts=20000, beams=64, cols=1024)\n"
        "trees = ba.build_trees(wl, dict(leaf_max_points=16))\n"
        "jobs = ba.jobs(wl, trees, dict(max_iterations=5), dict(max_iterations=5))\n"
        "b = kds.Batch()\n"
        "c, ms = b.autotune(jobs)\n"
        "print('chosen', c)\n" % ROOT)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "chosen" in r.stdout
