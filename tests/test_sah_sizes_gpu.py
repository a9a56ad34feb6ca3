"""The SAH builder at the sizes where its work changes hands: subtrees of up to 32 triangles (one
lane each), up to 512 (one CTA), chunks of 1,024 positions of a larger range; the same sizes with
coinciding centres, where every range is halved by position; vertices that are NaN or infinite."""
import numpy as np
import pytest
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import scenes, sensors
from test_sah_build import _check_tree

pytestmark = pytest.mark.gpu
SIZES = [2, 3, 31, 32, 33, 63, 65, 511, 512, 513, 1023, 1024, 1025, 2049, 4500]


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    torch.cuda.set_device(0)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["soup", "same", "half_same", "line"])
def test_tree_is_valid_exact_and_deterministic(n, kind):
    rng = np.random.default_rng(n)
    c = rng.standard_normal((n, 1, 3)) * [30.0, 10.0, 1.0]
    if kind == "same":
        c[:] = 1.0
    if kind == "half_same":
        c[: n // 2] = 0.25
    if kind == "line":
        c = np.arange(n, dtype=np.float64)[:, None, None] * [1.0, 0.0, 0.0]
    v = (c + rng.standard_normal((n if kind != "same" else 1, 3, 3))).reshape(-1, 3).astype(np.float32)
    v = np.broadcast_to(v.reshape(-1, 3, 3), (n, 3, 3)).reshape(-1, 3).copy()
    f = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    g = _check_tree(rm.Map(v, f), v, f)
    g2 = rm.Map(v, f).export()
    for k in g:
        assert np.array_equal(g[k].view(np.uint32), g2[k].view(np.uint32)), k


@pytest.mark.parametrize("n", [40, 700, 3000])
def test_vertices_that_are_not_finite(n):
    rng = np.random.default_rng(n)
    v = (rng.standard_normal((n, 1, 3)) * 5 + rng.standard_normal((n, 3, 3))).astype(np.float32)
    v[::17, 1, 0] = np.nan
    v[::23, 2, 1] = np.inf
    f = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    poses = torch.from_numpy(scenes.room_poses(4, seed=1)).cuda()
    got = []
    for builder in ("sah", "lbvh"):
        m = rm.Map(v.reshape(-1, 3), f, builder=builder)
        sim = rm.SphereSimulator(m)
        sim.setModel(sensors.vlp16_360())
        got.append(sim.simulate(poses, attrs=("hits", "ranges", "face_ids")).tensors())
        assert m.status() == 0
    for a, t in got[0].items():
        assert torch.equal(t.view(torch.uint8), got[1][a].view(torch.uint8)), a


@pytest.mark.parametrize("n", [600, 1500, 6000])
@pytest.mark.parametrize("builder", ["sah", "lbvh"])
def test_trees_with_more_levels_than_a_balanced_one(n, builder):
    """A dense cluster and 80 triangles at growing distances from it: splits take off a few distant
    triangles each, so the cluster stays large, and nodes stay to be collapsed, for many levels."""
    rng = np.random.default_rng(n)
    c = rng.standard_normal((n, 1, 3)) * 0.1
    c[:80, 0, 0] = 1.3 ** np.arange(80)
    c[40:80, 0, 1] = 1.2 ** np.arange(40)
    v = (c + 0.05 * rng.standard_normal((n, 3, 3))).reshape(-1, 3).astype(np.float32)
    f = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    m = rm.Map(v, f, builder=builder)
    if builder == "sah":
        _check_tree(m, v, f)
    sim = rm.SphereSimulator(m)
    sim.setModel(sensors.vlp16_360())
    poses = torch.from_numpy(scenes.room_poses(4, seed=1)).cuda()
    got = []
    for width in (0, 2):
        sim.launch_config = rm.launch_config(bvh_width=width, packet=0)
        got.append(sim.simulate(poses, attrs=("hits", "ranges", "face_ids")).tensors())
    assert m.status() == 0
    for a, t in got[0].items():
        assert torch.equal(t.view(torch.uint8), got[1][a].view(torch.uint8)), a
