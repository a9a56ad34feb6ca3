"""SAH builds of meshes in which whole triangles are NaN (depth images with invalid pixels), in one
coordinate or in all: the boxes are those a refit computes, and queries agree with the LBVH."""
import numpy as np
import pytest
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import scenes, sensors

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    torch.cuda.set_device(0)


def mesh(n, kind, which, coord):
    rng = np.random.default_rng(n)
    v = rng.standard_normal((n, 1, 3)) * 5 + rng.standard_normal((n, 3, 3))
    if kind == "wall":  # equal centres on x: every triangle in bin 0 there
        v[..., 0] = 3.0
    bad = {"one": [n // 2], "tenth": slice(0, None, 10), "half": slice(0, None, 2), "end": slice(n // 2, None)}[which]
    v[bad, :, coord] = np.nan
    return v.astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("n", [2, 40, 700, 3000])
@pytest.mark.parametrize("kind", ["cloud", "wall"])
@pytest.mark.parametrize("which", ["one", "tenth", "half", "end"])
@pytest.mark.parametrize("coord", [0, 2, slice(None)])
def test_whole_triangles_that_are_nan(n, kind, which, coord):
    v, f = mesh(n, kind, which, coord)
    m = rm.Map(v, f)
    got, bounds = m.export()["boxes"], m.info()
    poses = torch.from_numpy(scenes.room_poses(4, seed=1)).cuda()
    out = []
    for mp in (m, rm.Map(v, f, builder="lbvh")):
        sim = rm.SphereSimulator(mp)
        sim.setModel(sensors.vlp16_360())
        for width in (0, 2):
            sim.launch_config = rm.launch_config(bvh_width=width)
            out.append(sim.simulate(poses, attrs=("hits", "ranges", "face_ids")).tensors())
        assert mp.status() == 0
    for o in out[1:]:
        for a, t in o.items():
            assert torch.equal(t.view(torch.uint8), out[0][a].view(torch.uint8)), a
    m.refit(v)
    assert np.array_equal(got.view(np.uint32), m.export()["boxes"].view(np.uint32))
    after = m.info()
    for k in ("bounds_lo", "bounds_hi"):
        assert np.array_equal(bounds[k], after[k], equal_nan=True)
