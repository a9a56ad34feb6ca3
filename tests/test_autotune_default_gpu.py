"""The tuner knows the default launch: a launch is no slower tuned than left alone; and the default
configuration given explicitly is the same launch as none."""
import numpy as np
import pytest
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import _lib, scenes, sensors

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scan(built):
    torch.cuda.set_device(0)
    s = scenes.box_room(seed=0, n_boxes=200)
    sim = rm.make_simulator(sensors.vlp16_900(), rm.Map(s.vertices, s.faces))
    poses = torch.from_numpy(scenes.room_poses(1, seed=2)).cuda()
    b = rm.resize_memory_bundle(rm.Bundle("ranges", "face_ids"), 900, 16, 1, device="cuda")
    return sim, poses, b


def median_us(sim, poses, b, cfg, n=40):
    """Of launches queued behind a long kernel, so that the host's time does not count."""
    sim.launch_config = cfg
    for _ in range(3):
        sim.simulate(poses, b)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(n + 1)]
    torch.cuda._sleep(5_000_000)
    ev[0].record()
    for i in range(n):
        sim.simulate(poses, b)
        ev[i + 1].record()
    torch.cuda.synchronize()
    return float(np.median([a.elapsed_time(c) * 1e3 for a, c in zip(ev, ev[1:])]))


def fields(c):
    return [getattr(c, f) for f, _ in c._fields_]


def test_a_small_launch_is_no_slower_when_tuned(scan):
    sim, poses, b = scan
    none = median_us(sim, poses, b, None)
    default = _lib.LaunchConfigC()
    _lib.call("rmg_default_launch_config", sim._map.handle, sim.sensor.handle, default)
    whole = rm.launch_config(bvh_width=4)  # 32 rays a warp: 1.4 times as long
    assert median_us(sim, poses, b, default) < 0.5 * (none + median_us(sim, poses, b, whole))
    sim.launch_config = None
    tuned = sim.autotune(poses, b, reps=9)
    assert median_us(sim, poses, b, tuned) < 0.5 * (none + median_us(sim, poses, b, whole)), fields(tuned)


def test_the_default_given_explicitly_changes_no_byte(scan):
    sim, poses, b = scan
    got = []
    default = _lib.LaunchConfigC()
    _lib.call("rmg_default_launch_config", sim._map.handle, sim.sensor.handle, default)
    for cfg in (None, default, rm.launch_config(), rm.launch_config(bvh_width=2), rm.launch_config(bvh_width=2, chunk=0),
                rm.launch_config(bvh_width=4, chunk=0, tile_w=4, tile_h=8), rm.launch_config(packet=1, chunk=0)):
        sim.launch_config = cfg
        got.append([t.clone() for t in sim.simulate(poses, attrs=("ranges", "face_ids")).tensors().values()])
    for g in got[1:]:
        assert all(torch.equal(x.view(torch.uint8), y.view(torch.uint8)) for x, y in zip(g, got[0]))
