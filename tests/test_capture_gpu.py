"""Calls under CUDA graph capture: a process whose first use of the library's memory pool is captured;
maps destroyed while another thread captures, or in a relaxed capture, leave the capture whole."""
import subprocess
import sys
import threading
from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

FIRST = """
import torch
from rmagine_gb300 import statistics as rs
torch.cuda.set_device(0)
d = torch.randn(2, 50000, 3, generator=torch.Generator('cuda').manual_seed(1), device='cuda')
m = d + 0.01
st = torch.zeros(2, 16, device='cuda')
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    s, T = rs.statistics(d, m)
    gd, gm = rs.umeyama_backward(d, m, s, torch.ones(2, 9, device='cuda'))
for _ in range(2):
    g.replay()
torch.cuda.synchronize()
s2, T2 = rs.statistics(d, m)
gd2, gm2 = rs.umeyama_backward(d, m, s2, torch.ones(2, 9, device='cuda'))
for a, b in ((s, s2), (T, T2), (gd, gd2), (gm, gm2)):
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
"""


def test_the_first_call_of_a_process_may_be_captured(built):
    r = subprocess.run([sys.executable, "-c", FIRST], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-1500:]


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
@pytest.mark.parametrize("last", [False, True])
def test_a_map_destroyed_during_a_capture(built, mode, last):
    """thread_local: destroyed by another thread; relaxed: by the capturing one."""
    import rmagine_gb300 as rm
    from rmagine_gb300 import scenes, sensors

    torch.cuda.set_device(0)
    s = scenes.box_room(seed=0, n_boxes=20)
    poses = torch.from_numpy(scenes.room_poses(3, seed=1)).cuda()
    m = rm.Map(s.vertices, s.faces)
    keep = None if last else rm.Map(s.vertices, s.faces)
    sim = rm.make_simulator(sensors.vlp16_360(), m)
    b = sim.simulate(poses, attrs=("ranges",))
    want = b.ranges.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):  # work that still needs the map when it is destroyed
        torch.cuda._sleep(20_000_000)
        b.ranges.zero_()
        sim.simulate(poses, b)
    x = torch.zeros(4, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        y = x + 1
        if mode == "relaxed":
            m.destroy()
        else:
            t = threading.Thread(target=m.destroy)
            t.start()
            t.join()
        y = y + 1
    g.replay()
    torch.cuda.synchronize()
    assert y.tolist() == [2.0] * 4
    other = rm.Map(s.vertices * np.float32(2), s.faces)  # may take the destroyed map's memory
    assert torch.equal(b.ranges, want)
    del other, keep
