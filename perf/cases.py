"""The work this framework is used for, as measurable cases.

Every case is one call (or the few calls that belong together) a program makes through the public
Python API, on inputs it already holds: a map and a sensor set up once, poses and observations on the
GPU or, where the caller works in host memory, on the host.  A case is a dict of plain values:

    kind      scan | batch | scene | build | refit | correct | grad | icp
    scene     room (a closed box room, size = boxes in it) or terrain (a heightfield with boxes on it,
              size = grid points per side)
    sensor    spherical (rows x cols), pinhole (rows x cols), o1dn / ondn (cols directions scattered
              over the sphere)

listed() spans the range from one scan of one sensor to millions of rays per call; draw() spreads
cases over the same ranges.  exact() restates a case in binary64 with plain torch (every ray against
every triangle, so only where rays x triangles stays small).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import scenes, sensors, statistics
from rmagine_gb300.batched import BatchPlan
from rmagine_gb300.grad import range_pose_grad
from rmagine_gb300.noise import GaussianNoise, NoiseOptions

ALL = "hits,ranges,points,normals,face_ids"
SEVEN = ALL + ",geom_ids,object_ids"
BYTES = {"hits": 1, "ranges": 4, "points": 12, "normals": 12, "face_ids": 4, "geom_ids": 4, "object_ids": 4}
# rays x triangles of the largest brute-force restatement (a few seconds of binary64 on the GPU)
EXACT_TESTS = 4e10


def listed():
    return [
        # one scan of a VLP-16 in a room: a robot simulation's step, where latency counts
        dict(name="scan_room", kind="scan", scene="room", size=200, sensor="spherical", rows=16, cols=900, poses=1,
             attrs="hits,ranges", where="device", noise=False),
        # noisy scans of a fleet of robots in one room: data generation, multi-robot simulation
        dict(name="fleet_room", kind="scan", scene="room", size=200, sensor="spherical", rows=16, cols=360, poses=500,
             attrs="hits,ranges", where="device", noise=True),
        # full attributes of a 128-row lidar along a trajectory over a large outdoor map
        dict(name="lidar_terrain", kind="scan", scene="terrain", size=708, sensor="spherical", rows=128, cols=1024,
             poses=200, attrs=ALL, where="device", noise=False),
        # depth camera frames over a 2.1M-triangle map
        dict(name="camera_terrain", kind="scan", scene="terrain", size=1025, sensor="pinhole", rows=480, cols=640,
             poses=60, attrs=ALL, where="device", noise=False),
        # a sensor given as a table of scattered directions, results wanted in host memory
        dict(name="directions_host", kind="scan", scene="terrain", size=512, sensor="o1dn", rows=1, cols=10000,
             poses=64, attrs="hits,ranges,points", where="host", noise=False),
        # many small sensors of different kinds in one planned launch
        dict(name="sensors_batch", kind="batch", scene="terrain", size=512, sensors=512, poses=8,
             attrs="hits,ranges"),
        # a lidar over a map made of one big mesh and many instances of a small one
        dict(name="scene_instances", kind="scene", scene="terrain", size=708, boxes=2000, sensor="spherical", rows=64,
             cols=1024, poses=100, attrs=SEVEN),
        # a map arrives (a file read, a reconstruction step) and is scanned at once
        dict(name="map_build", kind="build", scene="terrain", size=513, sensor="spherical", rows=16, cols=900, poses=1,
             attrs="ranges,face_ids"),
        # a deforming mesh: new vertices for the same faces, then a scan
        dict(name="map_refit", kind="refit", scene="terrain", size=361, sensor="spherical", rows=32, cols=513, poses=3,
             attrs="ranges,face_ids"),
        # one correction step of a particle set against its scans (simulate, match point to plane, solve)
        dict(name="correct_room", kind="correct", scene="room", size=200, sensor="spherical", rows=16, cols=360,
             poses=256, shared=False),
        # pose gradients of a range loss: the backward direction of the ray cast
        dict(name="grad_terrain", kind="grad", scene="terrain", size=708, sensor="spherical", rows=64, cols=1024,
             poses=150),
        # correspondence statistics, Umeyama and its backward over a batch of ragged clouds
        dict(name="icp_batch", kind="icp", batches=400, points=10007, masked=True, p2l=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scene(rng, grid_hi):
    if rng.random() < 0.4:
        return dict(scene="room", size=_log(rng, 5, 400))
    return dict(scene="terrain", size=_log(rng, 40, grid_hi))


def _draw_sensor(rng):
    kind = rng.choice(["spherical", "spherical", "pinhole", "o1dn", "ondn"])
    if kind == "spherical":
        return dict(sensor=kind, rows=rng.choice([1, 16, 32, 64, 128, rng.randint(2, 100)]), cols=_log(rng, 90, 2048))
    if kind == "pinhole":
        return dict(sensor=kind, rows=_log(rng, 24, 480), cols=_log(rng, 32, 640))
    return dict(sensor=kind, rows=1, cols=_log(rng, 100, 10000))


def _draw_poses(rng, sensor, rays_lo, rays_hi, poses_hi=60000):
    per = sensor["rows"] * sensor["cols"]
    return max(1, min(poses_hi, int(_log(rng, rays_lo, rays_hi) / per)))


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan", "batch", "scene", "build", "refit", "correct", "grad", "icp"])
    if kind == "batch":
        return dict(kind=kind, **_draw_scene(rng, 708), sensors=_log(rng, 8, 600), poses=rng.randint(1, 8),
                    attrs=rng.choice(["hits,ranges", "ranges", "hits,ranges,face_ids"]))
    if kind == "icp":
        batches = _log(rng, 1, 600)
        return dict(kind=kind, batches=batches, points=max(16, min(40000, int(_log(rng, 3000, 4_000_000) / batches))),
                    masked=rng.random() < 0.7, p2l=rng.random() < 0.4)
    sensor = _draw_sensor(rng)
    if kind == "scan":
        host = rng.random() < 0.2
        return dict(kind=kind, **_draw_scene(rng, 1025), **sensor,
                    poses=_draw_poses(rng, sensor, 5000, 2_000_000 if host else 18_000_000),
                    attrs=rng.choice(["ranges", "hits,ranges", "hits,ranges,face_ids", "hits,points,normals", ALL]),
                    where="host" if host else "device", noise=not host and rng.random() < 0.2)
    if kind == "scene":
        return dict(kind=kind, scene="terrain", size=_log(rng, 60, 708), boxes=_log(rng, 10, 2000), **sensor,
                    poses=_draw_poses(rng, sensor, 10000, 6_000_000), attrs=rng.choice(["ranges", ALL, SEVEN]))
    if kind == "build":
        return dict(kind=kind, **_draw_scene(rng, 513), **sensor, poses=_draw_poses(rng, sensor, 3000, 100_000),
                    attrs="ranges,face_ids")
    if kind == "refit":
        return dict(kind=kind, **_draw_scene(rng, 513), **sensor, poses=_draw_poses(rng, sensor, 3000, 300_000),
                    attrs="ranges,face_ids")
    if kind == "correct":
        return dict(kind=kind, **_draw_scene(rng, 512), **sensor, poses=_draw_poses(rng, sensor, 10000, 4_000_000, 4000),
                    shared=rng.random() < 0.3)
    return dict(kind=kind, **_draw_scene(rng, 708), **sensor, poses=_draw_poses(rng, sensor, 10000, 9_000_000, 4000))


# ---- inputs ---------------------------------------------------------------------------------------
_last_mesh: dict = {}  # the mesh of the latest (scene, size, boxes, seed): cases share maps


def _mesh(case, seed):
    """(vertices, faces, height or None) of the case's map."""
    key = (case["scene"], case["size"], seed)
    if key not in _last_mesh:
        _last_mesh.clear()
        if case["scene"] == "room":
            s = scenes.box_room(seed=seed, n_boxes=case["size"])
        else:
            s = scenes.terrain(grid=case["size"], size=500.0 * case["size"] / 708.0, n_boxes=2 * case["size"], seed=seed)
        _last_mesh[key] = s
    return _last_mesh[key]


def _free_room_poses(mesh, n, seed):
    """Poses in a room whose sensor stands outside its boxes, by at least 0.3 m."""
    boxes = _cuda(mesh.vertices[8:].reshape(-1, 8, 3))
    lo, hi = boxes.amin(1) - 0.3, boxes.amax(1) + 0.3
    found, have = [], 0
    while have < n:
        p = scenes.room_poses(2 * (n - have) + 256, seed=seed)
        at = _cuda(p[:, 4:7])
        inside = torch.zeros(len(p), dtype=torch.bool, device="cuda")
        for i in range(len(lo)):
            inside |= ((at > lo[i]) & (at < hi[i])).all(1)
        found.append(p[~inside.cpu().numpy()])
        have += len(found[-1])
        seed += 1000003
    return np.concatenate(found)[:n]


def _poses(case, mesh, n, seed):
    if case["scene"] == "room":
        return _free_room_poses(mesh, n, seed + 1)
    return scenes.terrain_poses(mesh, n, seed=seed + 2, size=500.0 * case["size"] / 708.0)


def _model(case, seed):
    rows, cols = case["rows"], case["cols"]
    if case["sensor"] == "pinhole":
        return rm.depth_camera(cols, rows)
    if case["sensor"] == "spherical":
        if rows <= 16:  # a VLP-16's rows
            m = rm.vlp16_360()
            m.phi.size = rows
            m.theta = rm.DiscreteInterval(sensors.f32(-math.pi), sensors.f32(2.0 * math.pi / cols), cols)
            return m
        return rm.ouster_like(rows, cols)
    dirs = sensors.sphere_directions(cols, seed=seed + 3)
    if case["sensor"] == "o1dn":
        return rm.O1DnModel(width=cols, height=1, range=rm.Interval(0.3, 130.0), orig=(0.1, 0.0, 0.2), dirs=dirs)
    origs = (0.2 * sensors.sphere_directions(cols, seed=seed + 4)).astype(np.float32)
    return rm.OnDnModel(width=cols, height=1, range=rm.Interval(0.3, 130.0), origs=origs, dirs=dirs)


def _attrs(case):
    return tuple(case["attrs"].split(","))


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _instances(case, seed):
    """The terrain (identity) and its boxes, turned about the vertical and scaled, as instances."""
    mesh = scenes.terrain(grid=case["size"], size=500.0 * case["size"] / 708.0, n_boxes=0, seed=seed)
    half = 0.45 * 500.0 * case["size"] / 708.0
    rng = np.random.default_rng(seed + 5)
    n = case["boxes"]
    xy = rng.uniform(-half, half, (n, 2)).astype(np.float32)
    z = mesh.height_at(xy[:, 0], xy[:, 1]) - np.float32(0.1)
    yaw = rng.uniform(-math.pi, math.pi, n)
    scale = rng.uniform(0.2, 2.0, (n, 3)).astype(np.float32)
    inst = [rm.Instance(0, geom_id=0, object_id=0)]
    for i in range(n):
        T = [0.0, 0.0, math.sin(yaw[i] / 2), math.cos(yaw[i] / 2), xy[i, 0], xy[i, 1], z[i], 0.0]
        inst.append(rm.Instance(1, T=T, scale=scale[i], geom_id=1, object_id=1 + i))
    return mesh, inst


def _correspondences(case, seed):
    """Noisy, partly masked correspondences of clouds that a small motion apart from one another."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, N = case["batches"], case["points"]
    dev = dict(device="cuda", dtype=torch.float32)
    centre = 40.0 * torch.rand((B, 1, 3), generator=g, **dev) - 20.0
    data = centre + torch.randn((B, N, 3), generator=g, **dev) * torch.tensor([8.0, 6.0, 2.0], device="cuda")
    w = 0.05 * torch.randn((B, 3), generator=g, **dev)
    t = 0.2 * torch.randn((B, 1, 3), generator=g, **dev)
    model = data + torch.cross(w[:, None, :].expand_as(data), data, dim=2) + t
    model = model + 0.02 * torch.randn((B, N, 3), generator=g, **dev)
    nrm = torch.nn.functional.normalize(torch.randn((B, N, 3), generator=g, **dev), dim=2)
    mask = (torch.rand((B, N), generator=g, **dev) < 0.8).to(torch.uint8) if case["masked"] else None
    pre = torch.zeros((B, 8), **dev)
    pre[:, :3] = 0.01 * torch.randn((B, 3), generator=g, **dev)
    pre[:, 3] = 1.0
    pre[:, :4] = torch.nn.functional.normalize(pre[:, :4], dim=1)
    pre[:, 4:7] = 0.1 * torch.randn((B, 3), generator=g, **dev)
    gR = torch.randn((B, 3, 3), generator=g, **dev)
    gt = torch.randn((B, 3), generator=g, **dev)
    return dict(data=data, model=model, normals=nrm, mask=mask, pre=pre, gR=gR, gt=gt)


# the fused and plain statistics' gate: beyond the clouds' own spread, so noise never decides a pair
MAX_DIST = 30.0


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": seed}
    if kind == "icp":
        s.update(_correspondences(case, seed))
        s["params"] = statistics.UmeyamaReductionConstraints(max_dist=MAX_DIST)
        return s
    if kind == "scene":
        mesh, inst = _instances(case, seed)
        ub = scenes.box_mesh([-0.5, -0.5, 0.0], [0.5, 0.5, 1.0])
        s["map"] = rm.Scene([rm.Map(mesh.vertices, mesh.faces), rm.Map(*ub)], inst)
    else:
        mesh = _mesh(case, seed)
        if kind != "build":
            s["map"] = rm.Map(mesh.vertices, mesh.faces)
    if kind == "batch":
        # every sensor's results in its part of one buffer per attribute
        small = _small_sensors(case, seed)
        counts = [n for _, n in small]
        poses = _cuda(_poses(case, mesh, sum(counts), seed))
        s["bundle"] = rm.resize_memory_bundle(rm.Bundle(*_attrs(case)), 256, 1, sum(counts))
        jobs, at = [], 0
        for model, n in small:
            b = rm.Bundle(*_attrs(case))
            for a, t in s["bundle"].tensors().items():
                setattr(b, a, t[256 * at:256 * (at + n)])
            jobs.append((rm.Sensor(model), poses[at:at + n], b))
            at += n
        s["plan"] = BatchPlan(s["map"], jobs)
        return s
    model = _model(case, seed)
    sim = rm.make_simulator(model, s.get("map"))
    s["sim"] = sim
    poses = _poses(case, mesh, case["poses"], seed)
    s["poses"] = _cuda(poses)
    if kind in ("scan", "scene"):
        host = case.get("where") == "host"
        s["bundle"] = rm.resize_memory_bundle(rm.Bundle(*_attrs(case)), model.getWidth(), model.getHeight(),
                                              case["poses"], device="cpu" if host else "cuda", pin_memory=host)
        if host:
            s["poses"] = torch.from_numpy(poses).pin_memory()
    if kind == "build":
        s["vertices"], s["faces"] = mesh.vertices, mesh.faces
    if kind == "refit":
        rng = np.random.default_rng(seed + 6)
        ph = rng.uniform(0.0, 6.28, 2)
        v = mesh.vertices.copy()
        v[:, 2] += (0.2 * np.sin(0.3 * v[:, 0] + ph[0]) * np.cos(0.2 * v[:, 1] + ph[1])).astype(np.float32)
        s["vertices"] = v
    if kind in ("correct", "grad"):
        est = scenes.perturb_poses(poses, seed + 7, sigma_t=0.05, sigma_r_deg=1.0)
        truth = sim.simulate(s["poses"][:1] if case.get("shared") else s["poses"], attrs=("hits", "ranges", "points"))
        if kind == "grad":
            g = torch.Generator(device="cuda").manual_seed(seed + 8)
            s["obs"] = truth.ranges + 0.02 * torch.randn(truth.ranges.shape, generator=g, device="cuda")
        else:
            per = model.getWidth() * model.getHeight()
            one = case["shared"]
            s["scan"] = truth.points.nan_to_num(0.0).reshape((per, 3) if one else (-1, per, 3))
            s["mask"] = truth.hits.reshape(per if one else (-1, per)).contiguous()
            s["params"] = statistics.UmeyamaReductionConstraints(max_dist=1.0)
            if one:  # every estimate near the pose that the one scan was taken at
                est = scenes.perturb_poses(np.tile(poses[:1], (case["poses"], 1)), seed + 7, 0.05, 1.0)
        s["poses"] = _cuda(est)
    return s


def _small_sensors(case, seed):
    """Small sensors of two kinds with 1 .. case["poses"] poses each."""
    out = []
    for i in range(case["sensors"]):
        n = 1 + (5 * i // 2) % case["poses"]
        if i % 2 == 0:
            m = rm.O1DnModel(width=256, height=1, range=rm.Interval(0.3, 130.0), orig=(0.05, 0.0, 0.1),
                             dirs=sensors.sphere_directions(256, seed=seed + 1000 + i))
        else:
            m = rm.depth_camera(32, 8, 60.0)
        out.append((m, n))
    return out


# ---- one pass -------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("scan", "scene"):
        s["sim"].simulate(s["poses"], s["bundle"])
        if case.get("noise"):
            GaussianNoise(0.0, 0.02, NoiseOptions(seed=s["seed"])).apply(s["bundle"].ranges)
        return s["bundle"].tensors()
    if kind == "batch":
        s["plan"].launch()
        return s["bundle"].tensors()
    if kind == "build":
        s["sim"].setMap(rm.Map(s["vertices"], s["faces"]))
        return s["sim"].simulate(s["poses"], attrs=_attrs(case)).tensors()
    if kind == "refit":
        s["map"].refit(s["vertices"])
        return s["sim"].simulate(s["poses"], attrs=_attrs(case)).tensors()
    if kind == "correct":
        stats, T = s["sim"].simulate_statistics(s["poses"], s["scan"], dataset_mask=s["mask"], params=s["params"])
        return {"stats": stats, "T": T}
    if kind == "grad":
        grad, loss, ranges, faces = range_pose_grad(s["sim"], s["poses"], s["obs"], want_sim=True)
        return {"grad": grad, "loss": loss, "ranges": ranges, "face_ids": faces}
    # icp
    kw = dict(pre=s["pre"], params=s["params"], dataset_mask=s["mask"])
    if case["p2l"]:
        stats, T = statistics.statistics_p2l(s["data"], s["model"], s["normals"], **kw)
        return {"stats": stats, "T": T}
    stats, T = statistics.statistics_p2p(s["data"], s["model"], **kw)
    gd, gm = statistics.umeyama_backward(s["data"], s["model"], stats, s["gR"], s["gt"], **kw)
    return {"stats": stats, "T": T, "grad_dataset": gd, "grad_model": gm}


# ---- what a pass cannot do without ----------------------------------------------------------------
def _mesh_bytes(case):
    if case["scene"] == "room":
        return 12 * (8 * (case["size"] + 1)) + 12 * (12 * (case["size"] + 1))
    g = case["size"]
    boxes = 0 if case["kind"] == "scene" else 2 * g
    return 12 * (g * g + 8 * boxes) + 12 * (2 * (g - 1) ** 2 + 12 * boxes)


def work(case):
    """Inputs read once and outputs written once; per ray the arithmetic of its set-up, one triangle
    test and its attributes (a search structure's own traffic is the implementation's)."""
    kind = case["kind"]
    if kind == "icp":
        n = case["batches"] * case["points"]
        read = 24 + (1 if case["masked"] else 0) + (12 if case["p2l"] else 0)
        if case["p2l"]:
            return {"bytes": read * n, "flops": 75.0 * n}
        return {"bytes": (2 * read + 24) * n, "flops": 150.0 * n}
    if kind == "batch":
        rays = 256 * sum(1 + (5 * i // 2) % case["poses"] for i in range(case["sensors"]))
        out = sum(BYTES[a] for a in _attrs(case))
        return {"bytes": min(_mesh_bytes(case), 36 * rays) + out * rays + 12 * 256 * case["sensors"], "flops": 200.0 * rays}
    per = case["rows"] * case["cols"]
    rays = per * case["poses"]
    mesh = _mesh_bytes(case)
    table = per * (24 if case["sensor"] == "ondn" else 12) + 32 * case["poses"]
    if kind == "correct":
        scan = 13 * (per if case["shared"] else rays)
        return {"bytes": min(mesh, 36 * rays) + table + scan + 96 * case["poses"], "flops": 300.0 * rays}
    if kind == "grad":
        return {"bytes": min(mesh, 36 * rays) + table + 12 * rays + 28 * case["poses"], "flops": 300.0 * rays}
    out = sum(BYTES[a] for a in _attrs(case))
    if kind in ("build", "refit"):  # the whole mesh is read, and a tree over it written and read
        return {"bytes": mesh + table + out * rays, "flops": 200.0 * rays}
    return {"bytes": min(mesh, 36 * rays) + table + out * rays, "flops": 200.0 * rays}


# ---- binary64 restatements ------------------------------------------------------------------------
def _rot(q, v):
    """Rotation of v [..., 3] by unit quaternions q [..., 4] (x, y, z, w) in binary64."""
    u, w = q[..., :3], q[..., 3:]
    t = 2.0 * torch.linalg.cross(u.expand_as(v), v, dim=-1)
    return v + w * t + torch.linalg.cross(u.expand_as(v), t, dim=-1)


def _rays64(case, seed):
    """Sensor-frame directions and origins [per, 3] in binary64."""
    m = _model(case, seed)
    if case["sensor"] == "spherical":
        phi = m.phi.min + np.arange(m.phi.size) * np.float64(np.float32(m.phi.inc))
        th = m.theta.min + np.arange(m.theta.size) * np.float64(np.float32(m.theta.inc))
        d = np.stack([np.cos(phi)[:, None] * np.cos(th)[None], np.cos(phi)[:, None] * np.sin(th)[None],
                      np.repeat(np.sin(phi)[:, None], th.size, 1)], -1).reshape(-1, 3)
        o = np.zeros_like(d)
    elif case["sensor"] == "pinhole":
        u, v = np.meshgrid(np.arange(m.width), np.arange(m.height))
        px, py = (u - m.c[0]) / m.f[0], (v - m.c[1]) / m.f[1]
        d = np.stack([np.ones_like(px), -px, -py], -1).reshape(-1, 3)
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        o = np.zeros_like(d)
    else:
        d = m.dirs.astype(np.float64)
        o = m.origs.astype(np.float64) if case["sensor"] == "ondn" else np.tile(np.float64(m.orig), (len(d), 1))
    return torch.from_numpy(d).cuda(), torch.from_numpy(o).cuda(), m.range


def _cast64(v, f, org, dirs, tmax):
    """Closest hits of rays [n, 3] on triangles in binary64: (t or inf [n], face [n])."""
    tri = v[f.long()]
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    best = torch.full((len(org),), math.inf, dtype=torch.float64, device="cuda")
    face = torch.zeros(len(org), dtype=torch.long, device="cuda")
    step = max(1, int(3e7 / len(a)))
    for i in range(0, len(org), step):
        o, d = org[i:i + step], dirs[i:i + step]
        # scalar triple products of the Moeller-Trumbore test, as matrix products over the triangles
        det = -(d @ n.T)
        s_n = o @ n.T - (a * n).sum(1)
        m = torch.linalg.cross(d, o)
        u = -(m @ e2.T) - d @ torch.linalg.cross(e2, a).T
        w = (m @ e1.T) + d @ torch.linalg.cross(e1, a).T
        u, w, t = u / det, w / det, s_n / det
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0) & (t <= tmax)
        t = torch.where(ok, t, math.inf)
        best[i:i + step], face[i:i + step] = t.min(1)
    return best, face


def _scan64(case, seed, poses, vertices, faces):
    """(dirs [per, 3], t [n, per], unit normals towards the sensor [n, per, 3], range) in binary64."""
    d, o, rng = _rays64(case, seed)
    q, tr = poses[:, :4].double(), poses[:, 4:7].double()
    q = q[:, None, :]
    D = _rot(q.expand(-1, len(d), -1), d[None].expand(len(q), -1, -1))
    O = _rot(q.expand(-1, len(d), -1), o[None].expand(len(q), -1, -1)) + tr[:, None]
    v = torch.from_numpy(vertices).cuda().double()
    f = torch.from_numpy(faces.astype(np.int64)).cuda()
    t, face = _cast64(v, f, O.reshape(-1, 3), D.reshape(-1, 3), rng.max)
    tri = v[f[face]]
    nrm = torch.nn.functional.normalize(torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]), dim=1)
    nrm = _rot((q * torch.tensor([-1.0, -1.0, -1.0, 1.0], device="cuda")).expand(-1, len(d), -1).reshape(-1, 4), nrm)
    nrm = nrm.reshape(len(q), len(d), 3)
    nrm = torch.where((nrm * d[None]).sum(-1, keepdim=True) > 0, -nrm, nrm)
    return d, o, t.reshape(len(q), len(d)), nrm, rng


def _umeyama64(dm, mm, C):
    U, _, Vh = torch.linalg.svd(C)
    sign = torch.ones(C.shape[:-1], dtype=torch.float64, device=C.device)
    sign[..., 2] = torch.sign(torch.linalg.det(U) * torch.linalg.det(Vh))
    R = U @ torch.diag_embed(sign) @ Vh
    return R, mm - (R @ dm[..., None])[..., 0]


def _quat64(R):
    """(x, y, z, w) with w >= 0 (the motions here are small)."""
    w = 0.5 * torch.sqrt(1.0 + R[:, 0, 0] + R[:, 1, 1] + R[:, 2, 2])
    return torch.stack([R[:, 2, 1] - R[:, 1, 2], R[:, 0, 2] - R[:, 2, 0], R[:, 1, 0] - R[:, 0, 1], 4.0 * w * w], 1) / (4.0 * w[:, None])


def _stats64(D, M, ok):
    """Means and covariance E[m d^T] - E[m] E[d]^T of the kept pairs, per batch."""
    k = ok.double()[..., None]
    D, M = torch.where(ok[..., None], D, 0.0), torch.where(ok[..., None], M, 0.0)
    n = k.sum(1).clamp_min(1.0)
    dm, mm = (D * k).sum(1) / n, (M * k).sum(1) / n
    C = ((M - mm[:, None]) * k).transpose(1, 2) @ (D - dm[:, None]) / n[..., None]
    return dm, mm, C, k.sum((1, 2))


def _records64(dm, mm, C, n):
    count = torch.from_numpy(n.cpu().numpy().astype(np.uint32).view(np.float32).astype(np.float64)).cuda()
    return torch.cat([dm, mm, C.transpose(1, 2).reshape(-1, 9), count[:, None]], 1)


def _transforms64(R, t):
    return torch.cat([_quat64(R), t, torch.zeros((len(t), 1), dtype=torch.float64, device="cuda")], 1)


def _match64(D, M, N, max_dist):
    if N is None:
        return M, ((M - D) ** 2).sum(-1) < max_dist * max_dist
    dist = ((M - D) * N).sum(-1)
    return D + N * dist[..., None], dist.abs() < max_dist


def exact(case, seed):
    kind = case["kind"]
    if kind == "icp":
        return _exact_icp(case, seed)
    if kind not in ("scan", "correct") or case.get("noise"):
        return None
    tests = float(case["rows"] * case["cols"] * case["poses"])
    tests *= 12 * (case["size"] + 1) if case["scene"] == "room" else 2 * case["size"] ** 2
    if tests > EXACT_TESTS:
        return None
    mesh = _mesh(case, seed)
    if kind == "scan":
        poses = _cuda(_poses(case, mesh, case["poses"], seed))
        d, o, t, nrm, rng = _scan64(case, seed, poses, mesh.vertices, mesh.faces)
        miss = torch.isinf(t)
        nan = torch.where(miss, math.nan, 0.0)[..., None]
        got = {"hits": None, "face_ids": None, "ranges": torch.where(miss, rng.max + 1.0, t).reshape(-1),
               "points": (d[None] * torch.where(miss, 0.0, t)[..., None] + o[None] + nan).reshape(-1, 3),
               "normals": (nrm + nan).reshape(-1, 3)}
        return {a: got[a] for a in _attrs(case)}
    s = prepare(case, seed)
    d, o, t, nrm, rng = _scan64(case, seed, s["poses"], mesh.vertices, mesh.faces)
    hit = torch.isfinite(t) & (t >= rng.min)
    I = d[None] * torch.where(hit, t, 0.0)[..., None] + o[None]
    D = s["scan"].double().expand(len(I), -1, -1)
    M, near = _match64(D, I, nrm, s["params"].max_dist)
    ok = hit & near & (s["mask"] != 0)
    dm, mm, C, n = _stats64(D, M, ok)
    return {"stats": _records64(dm, mm, C, n), "T": _transforms64(*_umeyama64(dm, mm, C))}


def _exact_icp(case, seed):
    s = prepare(case, seed)
    x, y = s["data"].double().requires_grad_(), s["model"].double().requires_grad_()
    pre = s["pre"].double()
    D = _rot(pre[:, None, :4].expand(-1, x.shape[1], -1), x) + pre[:, None, 4:7]
    M, ok = _match64(D, y, s["normals"].double() if case["p2l"] else None, s["params"].max_dist)
    if s["mask"] is not None:
        ok = ok & (s["mask"] != 0)
    dm, mm, C, n = _stats64(D, M, ok)
    R, t = _umeyama64(dm, mm, C)
    out = {"stats": _records64(dm, mm, C, n).detach(), "T": _transforms64(R, t).detach()}
    if not case["p2l"]:
        ((R * s["gR"].double()).sum() + (t * s["gt"].double()).sum()).backward()
        out["grad_dataset"], out["grad_model"] = x.grad, y.grad
    return out
