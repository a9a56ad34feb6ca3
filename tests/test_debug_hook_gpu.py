"""After a link of the binary tree is overwritten every walk of the map is the binary one's."""
import pytest
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import _lib, scenes, sensors

pytestmark = pytest.mark.gpu


def test_the_changed_binary_tree_is_the_one_walked(built):
    torch.cuda.set_device(0)
    s = scenes.box_room(seed=8, n_boxes=20)
    m = rm.Map(s.vertices, s.faces).build_wide8()
    sim = rm.make_simulator(sensors.vlp16_360(), m)
    poses = torch.from_numpy(scenes.room_poses(2, seed=9)).cuda()

    def faces(width):
        sim.launch_config = rm.launch_config(bvh_width=width)
        return sim.simulate(poses, attrs=("face_ids",)).face_ids

    before = [faces(w) for w in (0, 2, 4, 8)]
    assert all(torch.equal(b, before[0]) for b in before)
    _lib.call("rmg_map_debug_set_child", m.handle, 0, 0, -1)  # a leaf in place of the root's left subtree
    after = [faces(w) for w in (0, 2, 4, 8)]
    assert not torch.equal(after[1], before[0])
    assert all(torch.equal(a, after[1]) for a in after)
    assert m.status() == 0
