"""The 4-wide walk (the default) against the binary walk, bit for bit, where its nodes have empty
slots or only leaves (meshes of 1 to 17 triangles) and its rays are degenerate: zero, tiny, huge,
infinite and NaN direction components, an unbounded range, origins at infinity."""
import numpy as np
import pytest
import torch

import rmagine_gb300 as rm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    torch.cuda.set_device(0)


def odd_directions():
    c = [0.0, -0.0, 1.0, -1.0, 1e-25, 1e25, -1e25, np.inf, np.nan]
    g = np.array([[x, y, z] for x in c for y in c for z in c], np.float32)
    r = np.random.default_rng(3).standard_normal((500, 3)).astype(np.float32)
    return np.concatenate([g, r])


@pytest.mark.parametrize("n_tris", [1, 2, 3, 4, 5, 6, 9, 17])
@pytest.mark.parametrize("max_range", [50.0, np.inf])
def test_default_walk_equals_the_binary_walk(n_tris, max_range):
    rng = np.random.default_rng(n_tris)
    v = rng.uniform(-3, 3, (3 * n_tris, 3)).astype(np.float32)
    m = rm.Map(v, np.arange(3 * n_tris, dtype=np.uint32).reshape(-1, 3))
    dirs = odd_directions()
    model = rm.O1DnModel(width=len(dirs), height=1, range=rm.Interval(0.1, max_range), orig=(0.0, 0.0, 0.0), dirs=dirs)
    sim = rm.make_simulator(model, m)
    poses = rm.identity_transforms(4)
    poses[1, 4:7] = torch.tensor([0.5, -1.0, 2.0])
    poses[2, 4] = float("inf")
    poses[3, 5] = float("nan")
    got = {}
    for name, cfg in (("default", None), ("binary", rm.launch_config(bvh_width=2, packet=0))):
        sim.launch_config = cfg
        got[name] = sim.simulate(poses.cuda()).tensors()
    for a, t in got["default"].items():
        assert np.array_equal(t.cpu().numpy().view(np.uint8), got["binary"][a].cpu().numpy().view(np.uint8)), a
    assert m.status() == 0
