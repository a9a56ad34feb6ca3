"""The 4-wide walk visits a node's children from near to far: where many boxes stand behind one
another it gives the binary walk's bytes and is no slower than it."""
import numpy as np
import pytest
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import scenes, sensors

pytestmark = pytest.mark.gpu
ATTRS = ("ranges", "face_ids")


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    torch.cuda.set_device(0)


@pytest.mark.parametrize("half,boxes", [(10.0, 1700), (40.0, 1700), (10.0, 200)])
@pytest.mark.parametrize("model,n", [(sensors.vlp16_360(), 35), (sensors.depth_camera(360, 1), 560)])
def test_many_boxes_in_each_others_way(half, boxes, model, n):
    s = scenes.box_room(seed=0, n_boxes=boxes, half=half)
    sim = rm.make_simulator(model, rm.Map(s.vertices, s.faces))
    poses = torch.from_numpy(scenes.room_poses(n, seed=3, half=half)).cuda()
    out, us = {}, {}
    for width in (2, 4):
        sim.launch_config = rm.launch_config(bvh_width=width, packet=0)
        b = sim.simulate(poses, attrs=ATTRS)
        t = []
        for _ in range(7):
            torch.cuda._sleep(300_000)  # the host's time does not count
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(8):
                sim.simulate(poses, b)
            e1.record()
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1))
        us[width] = min(t)
        out[width] = b
    for a in ATTRS:
        assert torch.equal(getattr(out[2], a).view(torch.uint8), getattr(out[4], a).view(torch.uint8)), a
    assert us[4] <= us[2], us  # 0.6 to 0.8 of it; as the children came up to 1.4


@pytest.mark.parametrize("n", [17, 35])
def test_launches_of_one_wave_take_the_faster_walk(n):
    """20 and 41 warps per SM on 2,412 triangles: 25 and 33 us with the 4-wide walk, 45 and 52 binary."""
    s = scenes.box_room(seed=0, n_boxes=200)
    sim = rm.make_simulator(sensors.vlp16_360(), rm.Map(s.vertices, s.faces))
    poses = torch.from_numpy(scenes.room_poses(n, seed=3)).cuda()
    b = sim.simulate(poses, attrs=ATTRS)
    us = {}
    for cfg in (None, rm.launch_config(bvh_width=2, packet=0, chunk=0), rm.launch_config(bvh_width=4, packet=0, chunk=0)):
        sim.launch_config = cfg
        t = []
        for _ in range(7):
            torch.cuda._sleep(300_000)
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(8):
                sim.simulate(poses, b)
            e1.record()
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1))
        us[None if cfg is None else cfg.bvh_width] = min(t)
    assert us[None] <= 1.15 * min(us[2], us[4]), us
