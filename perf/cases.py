"""Performance cases of the registration path: what a user of this framework runs, through
its public entry points, from one small scan to a map of millions of points.

listed() names the cases, draw() makes further ones of the same ranges, prepare() builds
what a program holds before the call, run() makes one pass, work() states the bytes and
operations a pass cannot do without, and exact() gives the values in 64 bits from numpy
alone.  Inputs are the package's seeded synthetic spinning-LiDAR scans (box scene, 2 cm
range noise, 1-60 m), the stand-in for recorded sequences that its benchmark uses too.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import kd_slam2_b200 as kds
from kd_slam2_b200 import abi, ba, streams, synth

ICP = dict(max_error=0.5, max_iterations=10)
CT = dict(max_error=0.5, max_iterations=15, velocity_damping=10.0)
VEL = np.array([10.0, 0.0, 0.0, 0.0, 0.0, np.deg2rad(30.0)])  # a vehicle's speed and yaw rate
RETURNS = 0.69      # share of the rays that come back in these scenes
LEAF_POINTS = 13.0  # points per surfel at 16 points per leaf


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one sweep of a small 16-beam sensor to a tree: the call an odometry loop makes per frame
        dict(name="tree_scan_16", kind="tree", beams=16, cols=1024, scans=1, source="device", stamps=True, leaf=16,
             propagate=False),
        # one sweep of a 128-beam sensor from host arrays, with normals handed down to sparse leaves
        dict(name="tree_scan_128_host", kind="tree", beams=128, cols=2048, scans=1, source="host", stamps=True,
             leaf=16, propagate=True),
        # a map of many accumulated scans, no stamps (odd column count): the largest build
        dict(name="tree_map", kind="tree", beams=128, cols=8191, scans=16, source="device", stamps=False, leaf=16,
             propagate=False),
        # the keyframe trees of a bundle-adjustment window in one pass, ragged sizes
        dict(name="forest_keyframes", kind="forest", keyframes=32, cols=2048, leaf=16),
        # scan-to-scan rigid registration of small scans: the shortest alignment
        dict(name="icp_scan_16", kind="align", ct=False, beams=16, cols=1024, map_beams=16, map_cols=1024,
             map_scans=1, leaf=16),
        # continuous-time registration of a moving 64-beam sensor against a large map
        dict(name="ct_scan_64_map", kind="align", ct=True, beams=64, cols=1024, map_beams=128, map_cols=8192,
             map_scans=12, leaf=16),
        # every overlapping pair of a window aligned, rigid and continuous-time, in one batch
        dict(name="batch_pairs", kind="batch", keyframes=64, cols=1024, leaf=16),
        # one solver step of the same graph: all factors linearized and assembled into blocks
        dict(name="factor_step", kind="factors", keyframes=24, cols=1024, leaf=16),
        # odometry: sweeps from the sensor driver's host arrays through tree build and tracker
        dict(name="odometry_64", kind="odometry", ct=True, beams=64, cols=1024, frames=4, leaf=16),
        # served registration: many streams, maps rebuilt on the way, every request at once
        dict(name="served_streams", kind="served", streams=8, scans=10, map_scans=3, leaf=16),
        # the voxel filter in front of the build
        dict(name="voxel_128", kind="voxel", beams=128, cols=2048, space_res=0.1, time_res=0.0, stamps=True),
        # a tree message from a recording to the device and back
        dict(name="message_64", kind="message", beams=64, cols=1024, scans=1, leaf=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tree", "tree", "forest", "align", "align", "batch", "factors", "odometry", "served", "voxel",
                       "message"])
    c = dict(kind=kind)
    if kind != "voxel":
        c["leaf"] = rng.choice([16, 16, 30])
    if kind == "tree":
        beams = rng.choice([16, 32, 64, 128])
        scans = _log(rng, 1, 16) if beams == 128 else 1
        c.update(beams=beams, scans=scans, cols=_log(rng, 500, 8191), source=rng.choice(["device", "device", "host"]),
                 stamps=rng.random() < 0.7, propagate=rng.random() < 0.3)
    elif kind in ("forest", "batch", "factors"):
        c.update(keyframes=_log(rng, 4, {"forest": 32, "batch": 64, "factors": 24}[kind]), cols=_log(rng, 400, 2048 if kind == "forest" else 1024))
    elif kind == "align":
        c.update(ct=rng.random() < 0.6, beams=rng.choice([16, 32, 64, 128]), cols=_log(rng, 700, 1900),
                 map_beams=rng.choice([32, 64, 128]), map_cols=_log(rng, 1000, 8000), map_scans=_log(rng, 1, 12))
    elif kind == "odometry":
        c.update(ct=rng.random() < 0.7, beams=rng.choice([16, 32, 64]), cols=_log(rng, 700, 1100),
                 frames=rng.randint(2, 4))
    elif kind == "served":
        c.update(streams=rng.randint(2, 8), scans=rng.randint(3, 10), map_scans=rng.randint(1, 3))
    elif kind == "voxel":
        c.update(beams=rng.choice([16, 32, 64, 128]), cols=_log(rng, 500, 2048), space_res=rng.choice([0.1, 0.25, 0.5]),
                 time_res=rng.choice([0.0, 0.0, 0.02]), stamps=rng.random() < 0.7)
    else:
        c.update(beams=rng.choice([16, 32, 64, 128]), cols=_log(rng, 700, 2000), scans=1)
    return c


# ------------------------------------------------------------------------------ inputs
def _elev(beams):
    return (-15.0, 15.0) if beams <= 32 else (-22.5, 22.5)


def _boxes(seed):
    return synth.scene(1001 + seed % 64)


def _sweep(case, seed, k=0, vel=None, pose=None, t_start=0.0):
    return synth.scan(_boxes(seed), synth.pose((0.0, 0.0, 1.8)) if pose is None else pose, vel=vel,
                      beams=case["beams"], cols=case["cols"], elev=_elev(case["beams"]), t_start=t_start,
                      seed=seed * 1009 + 17 + k, threads=16)


def _map(seed, beams, cols, scans):
    """The union of static scans 1 m apart, in the world frame."""
    out = []
    for k in range(scans):
        P = synth.pose((k - scans // 2, 0.0, 1.8))
        xyz, _ = synth.scan(_boxes(seed), P, beams=beams, cols=cols, elev=_elev(beams), seed=seed * 1009 + 500 + k,
                            threads=16)
        out.append(synth.transform(xyz, P))
    return np.ascontiguousarray(np.concatenate(out))


def _cloud(case, seed):
    """(points, stamps or None) of a tree or voxel case."""
    if case.get("scans", 1) > 1:
        xyz = _map(seed, case["beams"], case["cols"], case["scans"])
        return xyz, (np.linspace(0.0, 0.1 * case["scans"], len(xyz)) if case["stamps"] else None)
    xyz, st = _sweep(case, seed, vel=VEL)
    return xyz, (st if case.get("stamps", True) else None)


def _align_inputs(case, seed):
    """(map points, scan points, stamps, initial pose, initial velocity)."""
    m = _map(seed, case["map_beams"], case["map_cols"], case["map_scans"])
    true = synth.pose((0.0, 0.0, 1.8))
    xyz, st = _sweep(case, seed, vel=VEL if case["ct"] else None)
    rng = np.random.default_rng(seed)
    d, a = rng.normal(size=3), rng.normal(size=3)
    X0 = streams.compose(true, synth.pose(0.1 * d / np.linalg.norm(d), np.deg2rad(1.0) * a / np.linalg.norm(a)))
    v0 = VEL + rng.normal(size=6) * np.array([0.5, 0.5, 0.1, 0.01, 0.01, 0.05]) if case["ct"] else np.zeros(6)
    return m, xyz, st, X0, v0


def _workload(case, seed):
    full = 128 * case["cols"]
    return ba.make_workload(seed=seed % 100003, num_keyframes=case["keyframes"], cols=case["cols"],
                            min_pts=full // 13, max_pts=full)


def _frames(case, seed):
    """(time, points, stamps) of consecutive sweeps of a slowly driven sensor."""
    v = np.array([2.0, 0.1, 0.0, 0.0, 0.0, 0.1])
    P, out = synth.pose((0.0, 0.0, 1.8)), []
    for k in range(case["frames"]):
        xyz, st = _sweep(case, seed, k=k, vel=v, pose=P, t_start=0.1 * k)
        out.append((0.1 * k, xyz, st))
        P = streams.compose(P, streams.motion(v, 0.1))
    return out


def _gpu(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _capacity(case):
    """Surfels or nodes to make room for, whatever the scan returns."""
    return case.get("beams", 128) * case["cols"] * case.get("scans", 1) // 4


def _leaf_buffer(case):
    """Device memory that a program keeps for the surfels of one tree, or of each tree of a window."""
    shape = (_capacity(case), 6) if case["kind"] == "tree" else (case["keyframes"], _capacity(case), 6)
    return torch.zeros(shape, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    tree = dict(leaf_max_points=case["leaf"]) if "leaf" in case else {}
    if kind == "tree":
        xyz, st = _cloud(case, seed)
        if case["source"] == "device":
            xyz, st = _gpu(xyz), _gpu(st)
        return dict(kind=kind, xyz=xyz, st=st, device=case["source"] == "device", out=_leaf_buffer(case),
                    gen=kds.TreeGeneratorB2003D(propagate_normal=int(case["propagate"]), **tree))
    if kind == "forest":
        return dict(kind=kind, inputs=ba.device_inputs(_workload(case, seed)), tree=tree, out=_leaf_buffer(case))
    if kind == "align":
        m, xyz, st, X0, v0 = _align_inputs(case, seed)
        gen = kds.TreeGeneratorB2003D(**tree)
        a = kds.CTICPB2003D(**CT) if case["ct"] else kds.ICPB2003D(**ICP)
        fixed, moving = gen.make_tree(_gpu(m), device=True), gen.make_tree(_gpu(xyz), _gpu(st), device=True)
        a.set_fixed(fixed)
        a.set_moving(moving)
        return dict(kind=kind, aligner=a, X0=X0, v0=v0)
    if kind in ("batch", "factors"):
        wl = _workload(case, seed)
        trees = ba.build_trees(wl, tree, inputs=ba.device_inputs(wl))
        s = dict(kind=kind, trees=trees, batch=kds.Batch())
        if kind == "batch":
            s["jobs"] = ba.jobs(wl, trees, ICP, CT)
        else:
            s["jobs"], s["factors"], s["vars"] = ba.factor_jobs(wl, trees, ICP, CT)
        return s
    if kind == "odometry":
        a = kds.CTICPB2003D(**CT) if case["ct"] else kds.ICPB2003D(**ICP)
        trk = kds.Tracker3D(odom_aligner=a, motion_model=kds.ConstVelMotionModel3D(), max_kf_trans=0.5,
                            min_inlier_frac=0.3)
        return dict(kind=kind, frames=_frames(case, seed), tracker=trk, gen=kds.TreeGeneratorB2003D(**tree))
    if kind == "served":
        tr = streams.make_trace(seed % 100003, num_streams=case["streams"], scans_per_stream=case["scans"],
                                map_scans=case["map_scans"], scene_seed=1001 + seed % 64, saturate=True, threads=16)
        return dict(kind=kind, trace=tr, tree=tree, inputs=[(_gpu(r.xyz), _gpu(r.stamps)) for r in tr.requests])
    if kind == "voxel":
        xyz, st = _cloud(case, seed)
        rays = case["beams"] * case["cols"]
        return dict(kind=kind, xyz=_gpu(xyz), st=_gpu(st), duration=0.0 if st is not None else 0.1,
                    out_xyz=torch.zeros((rays, 3), device="cuda"),
                    out_st=torch.zeros(rays, dtype=torch.float64, device="cuda"),
                    params=dict(range_min=1.0, range_max=100.0, space_res=case["space_res"],
                                time_res=case["time_res"]))
    xyz, st = _sweep(case, seed, vel=VEL)
    return dict(kind=kind, msg=kds.TreeGeneratorB2003D(**tree).make_tree(xyz, st).to_msg(),
                out=np.zeros((_capacity(case), abi.KDNODE3F_DTYPE.itemsize), np.uint8))


# ------------------------------------------------------------------------------ one pass
def _leaves(tree, out):
    """The surfels' means and normals into the caller's buffer; returns their number."""
    n = tree.num_leaves
    tree.extract_compressed_leaves_device(out[:n])
    return n


def _job_outputs(arr):
    a = np.frombuffer(arr, dtype=np.dtype(abi.Job))
    return {k: a[k].copy() for k in ("X", "v", "H", "b", "result", "iterations")}


def run(state):
    kind = state["kind"]
    if kind == "tree":
        n = _leaves(state["gen"].make_tree(state["xyz"], state["st"], device=state["device"]), state["out"])
        return state["out"], n
    if kind == "forest":
        trees = ba.build_trees(None, state["tree"], inputs=state["inputs"])
        return state["out"], np.array([_leaves(t, state["out"][i]) for i, t in enumerate(trees)])
    if kind == "align":
        a = state["aligner"]
        a.set_x(state["X0"])
        a.set_velocities(state["v0"])
        result = a.compute()
        return dict(X=a.get_x(), v=a.velocities(), H=a.H, b=a.b, result=result,
                    counts=[s["num_inliers"] for s in a.stats_log])
    if kind == "batch":
        return _job_outputs(state["batch"].run(state["jobs"]))
    if kind == "factors":
        state["batch"].run(state["jobs"])
        rc, H, b, enabled = state["batch"].assemble(state["factors"], state["vars"], 0.3)
        return dict(blocks=rc, H=H, b=b, enabled=enabled)
    if kind == "odometry":
        trk = state["tracker"]
        trk.reset()
        res = [trk.add_frame(state["gen"].make_tree(xyz, st), ts) for ts, xyz, st in state["frames"]]
        return dict(pose=np.stack([r["pose_in_world"] for r in res]),
                    velocity=np.stack([r["ct_velocity"] for r in res]), keyframes=res[-1]["keyframe_count"])
    if kind == "served":
        res, _, _ = streams.serve(state["trace"], tree=state["tree"], icp=ICP, ct=CT, inputs=state["inputs"])
        return dict(X=np.stack([r["X"] for r in res]), v=np.stack([r["v"] for r in res]),
                    result=np.array([r["result"] for r in res]), map_version=np.array([r["map_version"] for r in res]))
    if kind == "voxel":
        xyz, st = kds.voxelize(state["xyz"], state["st"], scan_duration=state["duration"], **state["params"])
        state["out_xyz"][:len(xyz)] = xyz
        state["out_st"][:len(xyz)] = st
        return state["out_xyz"], state["out_st"], len(xyz)
    m = kds.Tree.from_msg(state["msg"]).to_msg()
    state["out"][:len(m["nodes"])] = m["nodes"].view(np.uint8).reshape(len(m["nodes"]), -1)
    return dict(nodes=state["out"], root_mean=m["root_mean"], root_eigenvalues=m["root_eigenvalues"],
                root_eigenvectors=m["root_eigenvectors"])


# ------------------------------------------------------------------------------ what a pass needs
def _tree_work(points, clouds=1, stamps=True):
    """Points and stamps in; nodes (72 B: record, stamps, range, level), leaves and point order out.
    Per point and level the split test (9 operations) and the second moments (20)."""
    leaves = points / LEAF_POINTS
    levels = max(1.0, math.log2(max(2.0, leaves / clouds)))
    return points * (20.0 if stamps else 12.0) + leaves * (2 * 72.0 + 36.0) + 4.0 * points, points * levels * 29.0


def _align_work(leaves, fixed_leaves, ct, iterations):
    """Moving surfels and the fixed nodes that their descents reach, 32 B each, read once; per surfel
    and iteration the descent (about 12 per level), the terms and the outer products."""
    depth = math.log2(max(2.0, fixed_leaves))
    nodes = min(2.0 * fixed_leaves, leaves * 6.0)
    return 32.0 * (leaves + nodes), iterations * leaves * (12.0 * depth + (1300.0 if ct else 200.0))


def work(case):
    kind = case["kind"]
    per = 16.0 / case.get("leaf", 16)  # leaves scale with the points per leaf
    if kind in ("tree", "message", "voxel"):
        n = RETURNS * case["beams"] * case["cols"] * case.get("scans", 1)
        if kind == "tree":
            by, fl = _tree_work(n, stamps=case["stamps"])
        elif kind == "message":
            by, fl = n / LEAF_POINTS * per * 2 * 2 * 56.0, n / LEAF_POINTS * per * 2
        else:
            by, fl = n * (20.0 if case["stamps"] else 12.0) + 0.6 * n * 20.0, n * 20.0
        return {"bytes": by, "flops": fl}
    if kind in ("forest", "batch", "factors"):
        points = 0.36 * 128 * case["cols"]  # mean of a log-uniform size between 1/13 and 1 of a sweep, capped
        k = case["keyframes"]
        if kind == "forest":
            by, fl = _tree_work(points * k, clouds=k)
            return {"bytes": by, "flops": fl}
        leaves = points / LEAF_POINTS * per
        pairs = max(1, 2 * k - 3)
        it = (10, 15) if kind == "batch" else (1, 1)
        a, b = _align_work(leaves, leaves, False, it[0]), _align_work(leaves, leaves, True, it[1])
        return {"bytes": k * 3.0 * 32.0 * leaves, "flops": pairs * (a[1] + b[1])}
    if kind == "align":
        leaves = RETURNS * case["beams"] * case["cols"] / LEAF_POINTS * per
        fixed = RETURNS * case["map_beams"] * case["map_cols"] * case["map_scans"] / LEAF_POINTS * per
        by, fl = _align_work(leaves, fixed, case["ct"], 15 if case["ct"] else 10)
        return {"bytes": by, "flops": fl}
    if kind == "odometry":
        n = RETURNS * case["beams"] * case["cols"]
        t = _tree_work(n)
        a = _align_work(n / LEAF_POINTS * per, n / LEAF_POINTS * per, case["ct"], 15 if case["ct"] else 10)
        return {"bytes": case["frames"] * (t[0] + a[0]), "flops": case["frames"] * (t[1] + a[1])}
    by = fl = 0.0
    for s in range(case["streams"]):
        beams = streams.BEAM_MIX[s % 4]
        n = RETURNS * beams * streams.beam_layout(beams)[0]
        rebuilt = case["map_scans"] + case["scans"]  # every scan becomes part of a map once
        t, m = _tree_work(n), _tree_work(n * rebuilt, stamps=False)
        a = _align_work(n / LEAF_POINTS * per, n * 5 / LEAF_POINTS * per, True, 13.6)
        by += case["scans"] * (t[0] + a[0]) + m[0]
        fl += case["scans"] * (t[1] + a[1]) + m[1]
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------------------ 64-bit values
def _dot32(a, b):
    """Three-term dot product in float32, x + (y + z), each operation rounded once: the split
    test is defined in 32 bits, so the sets of points are only the same if it is taken there."""
    p = a.astype(np.float32) * b.astype(np.float32)
    return p[:, 0] + (p[:, 1] + p[:, 2])


def _tree64(xyz, st, leaf, propagate=False):
    """The surfel tree of one cloud, level by level, statistics in 64 bits: means, directions,
    stamps, children of the nodes kept after pruning, breadth first, and the list of leaves."""
    p, t = xyz.astype(np.float64), np.zeros(len(xyz)) if st is None else st - st.min()
    order, seg, k = np.arange(len(xyz)), np.zeros(len(xyz), np.int64), 1
    has_par, prop_par = np.zeros(1, bool), np.zeros((1, 3))
    levels = []
    while k:
        q = p[order]
        n = np.bincount(seg, minlength=k).astype(np.float64)
        dn = np.maximum(n, 1.0)
        mean = np.stack([np.bincount(seg, q[:, i], k) for i in range(3)], 1) / dn[:, None]
        d = q - mean[seg]
        C = np.empty((k, 3, 3))
        for i in range(3):
            for j in range(i, 3):
                C[:, i, j] = C[:, j, i] = np.bincount(seg, d[:, i] * d[:, j], k) / dn
        dts = np.bincount(seg, t[order], k) / dn
        lam, V = np.linalg.eigh(C)
        e0, e2 = V[:, :, 0], V[:, :, 2]
        e0 = np.where(((mean * e0).sum(1) > 0)[:, None], -e0, e0)
        e2 = np.where(((mean * e2).sum(1) > 0)[:, None], -e2, e2)
        bad, few = n < 3, n < 5
        with np.errstate(divide="ignore", invalid="ignore"):
            flat = ~few & (lam[:, 0] / lam[:, 2] < np.float32(0.1)) & \
                (np.abs((mean * e0).sum(1)) > np.float32(0.1))
            split = ~few & ((n > leaf) | (n / (lam[:, 1] * lam[:, 2]) < 100.0))
        has = has_par & propagate
        prop = np.where((mean * prop_par).sum(1)[:, None] > 0, -prop_par, prop_par)
        use = has & ~split & ~flat
        direction = np.where(bad[:, None], 0.0, np.where(split[:, None], e2, e0))
        direction = np.where(use[:, None], prop, direction)
        mean[n == 0] = 0.0
        side = _dot32(direction[seg], xyz[order] - mean.astype(np.float32)[seg]) > 0
        levels.append((mean, direction, dts, split))
        handed, handed_prop = has | flat, np.where(flat[:, None], e0, prop_par)
        keep = split[seg]
        child = 2 * (np.cumsum(split) - 1)
        key = child[seg[keep]] + ~side[keep]
        o = np.argsort(key, kind="stable")
        order, seg, k = order[keep][o], key[o], 2 * int(split.sum())
        has_par, prop_par = np.repeat(handed[split], 2), np.repeat(handed_prop[split], 2, axis=0)
    alive = [None] * len(levels)
    for i in reversed(range(len(levels))):
        mean, direction, _, split = levels[i]
        a = (_dot32(direction, direction) > 0) & (np.abs(_dot32(mean, direction)) > np.float32(0.1)) & ~split
        if split.any():
            a[split] = alive[i + 1].reshape(-1, 2).any(1)
        alive[i] = a
    base = np.cumsum([0] + [int(a.sum()) for a in alive])
    left, right = [], []
    for i, a in enumerate(alive):
        kids = np.full((len(a), 2), -1)
        if levels[i][3].any():
            r = np.where(alive[i + 1], base[i + 1] + np.cumsum(alive[i + 1]) - 1, -1)
            kids[levels[i][3]] = r.reshape(-1, 2)
        left.append(kids[a, 0])
        right.append(kids[a, 1])
    m, d, s = (np.concatenate([lv[j][a] for lv, a in zip(levels, alive)]) for j in range(3))
    left, right = np.concatenate(left), np.concatenate(right)
    return dict(mean=m, dir=d, dts=s, left=left, right=right, leaves=np.nonzero((left < 0) & (right < 0))[0])


def _leaves64(t):
    return np.concatenate([t["mean"], t["dir"]], 1)[t["leaves"]]


def _padded(a, n):
    return np.concatenate([a, np.zeros((n - len(a),) + a.shape[1:])])


def _stored(t):
    """The tree as it is kept: nodes in 32 bits."""
    return dict(t, **{k: t[k].astype(np.float32).astype(np.float64) for k in ("mean", "dir", "dts")})


def _skew(u):
    S = np.zeros(u.shape[:-1] + (3, 3))
    S[..., 0, 1], S[..., 0, 2], S[..., 1, 2] = -u[..., 2], u[..., 1], -u[..., 0]
    S[..., 1, 0], S[..., 2, 0], S[..., 2, 1] = u[..., 2], -u[..., 1], u[..., 0]
    return S


def _rot(w):
    """Rotation matrices of rotation vectors (..., 3)."""
    a = np.linalg.norm(w, axis=-1)[..., None, None]
    S = _skew(w / np.maximum(a[..., 0], 1e-300))
    return np.eye(3) + np.sin(a) * S + (1.0 - np.cos(a)) * (S @ S)


def _drot(w, u):
    """Derivative of R(w) u by w: -R skew(u) Q."""
    a = np.maximum(np.linalg.norm(w, axis=-1)[..., None, None], 1e-300)
    R, n = _rot(w), w / a[..., 0]
    Q = n[..., :, None] * n[..., None, :] + (np.swapaxes(R, -1, -2) - np.eye(3)) @ _skew(n) / a
    Q = np.where(a < 1e-9, np.eye(3), Q)
    return -R @ _skew(u) @ Q


def _terms64(fixed, moving, X, v, Xf, prm, dual=False):
    """Jacobian rows, errors, weights and counts of one linearization (fixed velocity zero)."""
    m, n, dt = (moving[k][moving["leaves"]] for k in ("mean", "dir", "dts"))
    ct = v is not None
    mw, nw = m, n
    if ct:
        R = _rot(v[3:] * dt[:, None])
        mw, nw = np.einsum("nij,nj->ni", R, m) + v[:3] * dt[:, None], np.einsum("nij,nj->ni", R, n)
    pm, nm = mw @ X[:, :3].T + X[:, 3], nw @ X[:, :3].T
    q = (pm - Xf[:, 3]) @ Xf[:, :3]
    idx, live = np.zeros(len(m), np.int64), np.full(len(m), len(fixed["mean"]) > 0)
    while True:
        l, r = fixed["left"][idx], fixed["right"][idx]
        go = live & ((l >= 0) | (r >= 0))
        if not go.any():
            break
        side = (fixed["dir"][idx] * (q - fixed["mean"][idx])).sum(1) > 0
        nxt = np.where(side, l, r)
        live &= ~(go & (nxt < 0))
        idx = np.where(go & live, nxt, idx)
    pf, nf = fixed["mean"][idx] @ Xf[:, :3].T + Xf[:, 3], fixed["dir"][idx] @ Xf[:, :3].T
    ns, dp = nm + nf, pm - pf
    e = (dp * ns).sum(1)
    ok = live & ((nf * nm).sum(1) >= np.float32(math.cos(25.0 / 180.0 * math.pi))) & (np.abs(e) <= prm["max_error"])
    J = [ns, np.cross(pm, nf) + np.cross(pf, nm)]
    if ct:
        w = v[3:] * dt[:, None]
        A, B = X[:, :3] @ _drot(w, m), X[:, :3] @ _drot(w, n)
        J += [ns @ X[:, :3] * dt[:, None],
              (np.einsum("ni,nij->nj", ns, A) + np.einsum("ni,nij->nj", dp, B)) * dt[:, None]]
    if dual:
        db = fixed["dts"][idx][:, None]
        A, B = -Xf[:, :3] @ _skew(fixed["mean"][idx]), -Xf[:, :3] @ _skew(fixed["dir"][idx])
        J += [-ns @ Xf[:, :3] * db, (np.einsum("ni,nij->nj", -ns, A) + np.einsum("ni,nij->nj", dp, B)) * db]
    chi2 = e * e
    g = np.where(chi2 > np.float32(0.1), np.sqrt(np.float32(0.1) / np.maximum(chi2, 1e-300)), 1.0)
    J = np.concatenate(J, 1)[ok]
    return J, e[ok], g[ok], int((ok & (chi2 <= np.float32(0.1))).sum()), len(m)


def _align64(fixed, moving, X0, v0, prm):
    """Gauss-Newton as compute() runs it, all in 64 bits: (X, v, H, b, inlier share)."""
    X, v = np.array(X0), None if v0 is None else np.array(v0)
    D = 6 if v0 is None else 12
    lam = np.array([1.0] * 6 + [prm.get("velocity_damping", 0.0)] * (D - 6))
    for _ in range(prm["max_iterations"]):
        J, e, g, inliers, total = _terms64(fixed, moving, X, v, np.eye(3, 4), prm)
        H, b = (J * g[:, None]).T @ J, J.T @ (g * e)
        if len(e) < 10:
            break
        dx = np.linalg.solve(H + np.diag(lam), -b)
        X = streams.compose(synth.pose(dx[:3], dx[3:6]), X)
        if v is not None:
            v = v + dx[6:]
    return X, v, H, b, inliers / max(1, total)


def _factors64(case, seed):
    """The assembled blocks of a solver step."""
    wl = _workload(case, seed)
    trees = [_stored(_tree64(k.xyz, k.stamps, case["leaf"])) for k in wl.keyframes]
    blocks, b = {}, np.zeros((2 * len(trees), 6))
    enabled = []
    for p in wl.pairs:
        Xi, Xj = wl.keyframes[p.i].X, wl.keyframes[p.j].X
        J, e, g, inliers, total = _terms64(trees[p.i], trees[p.j], Xj, None if p.kind == 0 else np.zeros(6), Xi,
                                           ICP if p.kind == 0 else CT, dual=p.kind == 1)
        # rows by variable: the fixed pose moves against the moving one
        cols = [(2 * p.i, -J[:, :6]), (2 * p.j, J[:, :6])]
        if p.kind == 1:
            cols = [cols[0], (2 * p.i + 1, J[:, 12:]), cols[1], (2 * p.j + 1, J[:, 6:12])]
        enabled.append(inliers / total > 0.3)
        for x, (vx, Jx) in enumerate(cols):
            for vy, Jy in cols[x:]:
                A = blocks.setdefault((min(vx, vy), max(vx, vy)), np.zeros((6, 6)))
                if enabled[-1]:
                    A += (Jx * g[:, None]).T @ Jy if vx <= vy else (Jy * g[:, None]).T @ Jx
            if enabled[-1]:
                b[vx] -= Jx.T @ (g * e)
    keys = sorted(blocks)
    return dict(blocks=None, H=np.stack([blocks[k] for k in keys]), b=b, enabled=None)


def _morph(t, v):
    """Every node moved by the body velocity v over its stamp, as the tree is kept."""
    R = _rot(v[3:] * t["dts"][:, None])
    return _stored(dict(t, mean=np.einsum("nij,nj->ni", R, t["mean"]) + v[:3] * t["dts"][:, None],
                        dir=np.einsum("nij,nj->ni", R, t["dir"])))


def _log6(X):
    c = min(1.0, max(-1.0, 0.5 * (np.trace(X[:, :3]) - 1.0)))
    a = math.acos(c)
    f = 0.5 if a < 1e-7 else a / (2.0 * math.sin(a))
    return np.concatenate([X[:, 3], f * np.array([X[2, 1] - X[1, 2], X[0, 2] - X[2, 0], X[1, 0] - X[0, 1]])])


def _odometry64(case, seed):
    kf, world, rel, delta, last = None, np.eye(3, 4), np.eye(3, 4), np.zeros(6), None
    poses, vels = [], []
    for ts, xyz, st in _frames(case, seed):
        t = _stored(_tree64(xyz, st, case["leaf"]))
        if last is not None and np.any(delta):
            t = _morph(t, delta / (ts - last))
        last, cv = ts, np.zeros(6)
        if kf is None:
            kf = t
        else:
            X0 = streams.compose(rel, synth.pose(delta[:3], delta[3:]))
            X, v, _, _, share = _align64(kf, t, X0, np.zeros(6) if case["ct"] else None, CT if case["ct"] else ICP)
            inv = np.concatenate([rel[:, :3].T, -rel[:, :3].T @ rel[:, 3:]], 1)
            alpha = float(np.float32(0.9))
            delta = alpha * delta + (1.0 - alpha) * _log6(streams.compose(inv, X))
            rel = X
            if case["ct"]:
                cv, t = v, _morph(t, v)
            if share < 0.3 or np.linalg.norm(rel[:, 3]) > 0.5:
                kf, world, rel = t, streams.compose(world, rel), np.eye(3, 4)
        poses.append(streams.compose(world, rel))
        vels.append(cv)
    return dict(pose=np.stack(poses), velocity=np.stack(vels), keyframes=None)


def _voxel64(case, seed):
    """Voxels in the order of their integer index; cells in 32 bits (they define the sets)."""
    xyz, st = _cloud(case, seed)
    if st is None:
        st = (np.arctan2(xyz[:, 1].astype(np.float64), xyz[:, 0].astype(np.float64)) + np.pi) / (2 * np.pi) * 0.1
    cell = (xyz * (np.float32(1.0) / np.float32(case["space_res"]))).astype(np.int64)
    if case["time_res"] > 0:
        inv = float(np.float32(1.0) / np.float32(case["time_res"]))
        cell = np.concatenate([cell, ((st - st.min()) * inv).astype(np.int64)[:, None]], 1)
    _, inv, n = np.unique(cell, axis=0, return_inverse=True, return_counts=True)
    inv = inv.reshape(-1)
    mean = np.stack([np.bincount(inv, xyz[:, i].astype(np.float64)) for i in range(3)], 1) / n[:, None]
    return mean, np.bincount(inv, st) / n


def exact(case, seed):
    """None where it takes too long (maps of millions of points, the big batch, the served trace)
    and for messages, which are copied and not computed."""
    kind = case["kind"]
    if kind == "tree":
        xyz, st = _cloud(case, seed)
        if len(xyz) >= 1_000_000:
            return None
        return _padded(_leaves64(_tree64(xyz, st, case["leaf"], case["propagate"])), _capacity(case)), None
    if kind == "forest":
        wl = _workload(case, seed)
        if sum(len(k.xyz) for k in wl.keyframes) > 3_000_000:
            return None
        return np.stack([_padded(_leaves64(_tree64(k.xyz, k.stamps, case["leaf"])), _capacity(case))
                         for k in wl.keyframes]), None
    if kind == "align":
        m, xyz, st, X0, v0 = _align_inputs(case, seed)
        if len(m) > 1_000_000:
            return None
        fixed, moving = (_stored(_tree64(p, s, case["leaf"])) for p, s in ((m, None), (xyz, st)))
        X, v, H, b, _ = _align64(fixed, moving, X0, v0 if case["ct"] else None, CT if case["ct"] else ICP)
        # a rigid alignment has settled: what is left of b is rounding, of no value of its own
        return dict(X=X, v=np.zeros(6) if v is None else v, H=H, b=b if case["ct"] else None, result=None, counts=None)
    if kind == "factors":
        return _factors64(case, seed)
    if kind == "odometry":
        return _odometry64(case, seed)
    if kind == "voxel":
        rays = case["beams"] * case["cols"]
        return tuple(_padded(a, rays) for a in _voxel64(case, seed)) + (None,)
    return None
