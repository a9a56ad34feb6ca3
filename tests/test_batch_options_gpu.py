"""A batch plan's set options are taken literally: tiles of 32 rays, `grab` tiles per fetch (also where
the last fetch is cut short), and the walk that the stack depth names; left at their defaults, small
plans take smaller tiles."""
import numpy as np
import pytest
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import _lib, batched, scenes, sensors

pytestmark = pytest.mark.gpu
ATTRS = ("ranges", "face_ids")


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    torch.cuda.set_device(0)


def plan_of(m, models, n_poses, **cfg):
    jobs, want = [], []
    for i, model in enumerate(models):
        sim = rm.make_simulator(model, m)
        poses = torch.from_numpy(scenes.room_poses(n_poses, seed=i)).cuda()
        want.append(sim.simulate(poses, attrs=ATTRS))
        b = rm.Bundle(*ATTRS)
        rm.resize_memory_bundle(b, sim.sensor.width, sim.sensor.height, n_poses)
        jobs.append((sim, poses, b))
    return batched.BatchPlan(m, jobs, batched.batch_config(**cfg) if cfg else None), jobs, want


def same(jobs, want):
    torch.cuda.synchronize()
    return all(torch.equal(getattr(b, a).view(torch.uint8), getattr(w, a).view(torch.uint8))
               for (_, _, b), w in zip(jobs, want) for a in ATTRS)


def tiles(models, n_poses, w, h):
    return sum(-(-m.getWidth() // w) * -(-m.getHeight() // h) for m in models) * n_poses


@pytest.fixture(scope="module")
def room():
    s = scenes.box_room(seed=3, n_boxes=40)
    return rm.Map(s.vertices, s.faces)


def test_set_tiles_and_grab_are_literal(room):
    models = [sensors.vlp16_900(), sensors.ouster_like(32, 65)]
    for cfg in (dict(tile_w=16, tile_h=2), dict(tile_w=4, tile_h=8), dict(grab=1), dict(grab=7, ctas_per_sm=1)):
        plan, jobs, want = plan_of(room, models, 3, **cfg)
        assert plan.info()["tiles"] == tiles(models, 3, cfg.get("tile_w", 8), cfg.get("tile_h", 4)), cfg
        plan.launch()
        assert same(jobs, want), cfg
    for cfg in (dict(), dict(block_warps=2), dict(stack_depth=16)):  # left to the library: 8 rays a warp
        plan, jobs, want = plan_of(room, models, 3, **cfg)
        assert plan.info()["tiles"] > 3 * tiles(models, 3, 8, 4), cfg
        plan.launch()
        assert same(jobs, want), cfg


@pytest.mark.parametrize("grab", [2, 3, 64])
def test_several_tiles_per_fetch_with_a_cut_short_last_one(room, grab):
    """Many tiles for each of the warps, no multiple of grab: in twos the library's own choice."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    models = [sensors.ouster_like(32, 129)]
    n = (32 * sms // 136 + 1) | 1  # 136 tiles a pose, one warp on each SM: more than 16 twos per warp
    plan, jobs, want = plan_of(room, models, n, grab=grab, ctas_per_sm=1, block_warps=1)
    total = plan.info()["tiles"]
    assert total >= 32 * sms and total % 2 == 0
    plan.launch()
    assert same(jobs, want)
    plan, jobs, want = plan_of(room, models + [sensors.depth_camera(5, 3)], n, grab=grab, ctas_per_sm=1, block_warps=1)
    assert plan.info()["tiles"] % 2 == 1  # one tile a pose more, an odd number of poses
    plan.launch()
    assert same(jobs, want)


def test_the_stack_depth_names_the_walk():
    """A leaf in place of a subtree of the 4-wide tree: the default's walk misses what was below it, the
    binary walks do not."""
    s = scenes.box_room(seed=3, n_boxes=40)
    m = rm.Map(s.vertices, s.faces)
    models = [sensors.vlp16_900()]
    plans = {d: plan_of(m, models, 2, stack_depth=d) for d in (0, 8, 16)}
    for d, (plan, jobs, want) in plans.items():
        plan.launch()
        assert same(jobs, want), d
    _lib.call("rmg_map_debug_set_child", m.handle, 0, 2, -1)
    for d, (plan, jobs, want) in plans.items():
        plan.launch()
        assert same(jobs, want) == (d != 8), d
    assert m.status() == 0
