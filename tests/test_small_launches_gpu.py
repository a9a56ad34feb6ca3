"""Launches of few rays use warps of 4, 8 or 16 rays: every result equals the same rays' results in a
launch large enough for whole warps, at the sizes where the number of rays per warp changes and for
sensors narrower, shorter or smaller than a tile.  The pose gradient and the fused correction sum
over a warp's rays; a pose's result is the same bits in a launch of any size."""
import numpy as np
import pytest
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import scenes, sensors
from rmagine_gb300.batched import BatchPlan
from rmagine_gb300.grad import range_pose_grad

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world(built):
    torch.cuda.set_device(0)
    s = scenes.terrain(grid=120, size=60.0, n_boxes=60, seed=3)
    m = rm.Map(s.vertices, s.faces)
    scene = rm.Scene([m, rm.Map(*scenes.gen_cube())],
                     [rm.Instance(0)] + [rm.Instance(1, T=[0, 0, 0.6, 0.8, 3.0 * i, 2.0, 3.0], object_id=i) for i in range(5)])
    return s, m, scene


def models():
    d = sensors.sphere_directions(77, seed=4)
    return {"1x1": rm.depth_camera(1, 1), "3x5": rm.depth_camera(5, 3), "1x40": rm.depth_camera(40, 1),
            "40x1": rm.depth_camera(1, 40), "16x90": rm.ouster_like(16, 90), "33x65": rm.ouster_like(33, 65),
            "table": rm.O1DnModel(width=77, height=1, range=rm.Interval(0.1, 100.0), orig=(0.1, 0.0, 0.2), dirs=d)}


@pytest.mark.parametrize("name", list(models()))
@pytest.mark.parametrize("kind", ["map", "scene"])
def test_few_rays_equal_the_same_rays_among_many(world, name, kind):
    s, m, scene = world
    model = models()[name]
    per = model.getWidth() * model.getHeight()
    many = 1 + 250000 // per  # 42 warps of 32 rays on each of 152 SMs are 204,288 rays
    poses = torch.from_numpy(scenes.terrain_poses(s, many, seed=5, size=60.0)).cuda()
    sim = rm.make_simulator(model, m if kind == "map" else scene)
    whole = sim.simulate(poses).tensors()
    for n in sorted({1, 2, max(1, 25000 // per), max(1, 51000 // per), max(1, 102000 // per), max(1, 204000 // per)}):
        part = sim.simulate(poses[:n].contiguous()).tensors()
        for a, t in part.items():
            assert torch.equal(t.contiguous().view(torch.uint8), whole[a][:n * per].contiguous().view(torch.uint8)), (n, a)


@pytest.mark.parametrize("poses", [1, 9, 60])
def test_batch_of_few_rays_equals_plain_launches(world, poses):
    s, m, _ = world
    jobs, want = [], []
    for i, (name, model) in enumerate(models().items()):
        n = poses + i
        T = torch.from_numpy(scenes.terrain_poses(s, n, seed=7 + i, size=60.0)).cuda()
        b = rm.resize_memory_bundle(rm.Bundle("hits", "ranges", "normals"), model.getWidth(), model.getHeight(), n)
        sim = rm.make_simulator(model, m)
        sim.launch_config = rm.launch_config(bvh_width=2, packet=0)  # whole warps, the binary walk
        jobs.append((sim, T, b))
        want.append(sim.simulate(T, attrs=("hits", "ranges", "normals")).tensors())
    plan = BatchPlan(m, jobs)
    for _ in range(2):
        plan.launch()
        for (_, _, b), w in zip(jobs, want):
            for a, t in b.tensors().items():
                assert torch.equal(t.contiguous().view(torch.uint8), w[a].contiguous().view(torch.uint8)), a


@pytest.mark.parametrize("name", ["1x1", "3x5", "40x1", "33x65", "table"])
def test_gradient_and_correction_of_few_rays(world, name):
    s, m, _ = world
    model = models()[name]
    per = model.getWidth() * model.getHeight()
    many = min(60000, 1 + 250000 // per)  # the gradient takes at most 65,535 poses
    poses = torch.from_numpy(scenes.terrain_poses(s, many, seed=5, size=60.0)).cuda()
    sim = rm.make_simulator(model, m)
    truth = sim.simulate(poses, attrs=("hits", "ranges", "points"))
    obs = truth.ranges + 0.05
    scan, mask = truth.points.nan_to_num(0.0).reshape(many, per, 3) + 0.02, truth.hits.reshape(many, per).contiguous()
    g0, l0, r0, f0 = range_pose_grad(sim, poses, obs, want_sim=True)
    st0, _ = sim.simulate_statistics(poses, scan, dataset_mask=mask)
    for n in sorted({1, 3, min(many, max(1, 51000 // per))}):
        g, l, r, f = range_pose_grad(sim, poses[:n].contiguous(), obs[:n * per], want_sim=True)
        assert torch.equal(r, r0[:n * per]) and torch.equal(f, f0[:n * per])
        assert torch.equal(g, g0[:n]) and torch.equal(l, l0[:n])
        st, _ = sim.simulate_statistics(poses[:n].contiguous(), scan[:n].contiguous(), dataset_mask=mask[:n].contiguous())
        assert torch.equal(st.view(torch.int32), st0[:n].view(torch.int32))


@pytest.mark.parametrize("poses", [14, 40, 41])
def test_walk_by_launch_size_gives_the_same_bytes(poses):
    """On a small map, launches of 16 rays a warp, just inside and just outside of 48 warps per SM
    (152 SMs, 180 tiles a pose): the walk that the library picks, the binary and the 4-wide one."""
    sc = scenes.box_room(seed=6, n_boxes=60)
    sim = rm.make_simulator(sensors.vlp16_360(), rm.Map(sc.vertices, sc.faces))
    T = torch.from_numpy(scenes.room_poses(poses, seed=3)).cuda()
    got = []
    for cfg in (None, rm.launch_config(bvh_width=2, packet=0), rm.launch_config(bvh_width=4)):
        sim.launch_config = cfg
        got.append(sim.simulate(T, attrs=("hits", "ranges", "points", "normals", "face_ids")).tensors())
    for other in got[1:]:
        for a, t in got[0].items():
            assert torch.equal(t.view(torch.uint8), other[a].view(torch.uint8)), a
