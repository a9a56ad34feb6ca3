"""The scene kernel's three combinations of walks against the brute-force oracle: 4-wide trees on both
levels (the rule), a top tree too deep for its 4-wide walk over 4-wide geometries, and binary walks
on both levels where a geometry's 4-wide tree cannot be walked; with a geometry large enough to be
opened into pieces."""
import numpy as np
import pytest
import torch

import oracle
import rmagine_gb300 as rm
from oracle.scene import InstancedScene
from rmagine_gb300 import _lib, scenes, sensors
from test_scene import ALL, IDENT, pose, quat

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    torch.cuda.set_device(0)


def chain_centres():
    """Centres at powers of two on each axis, and many more in one place: a top tree that stays
    unbalanced to its depth limit."""
    pts = [np.eye(3)[a] * 2.0 ** i for i in range(10) for a in range(3)]
    return np.array(pts + [pts[3]] * 600, np.float32)


@pytest.mark.parametrize("deep_top", [False, True])
@pytest.mark.parametrize("binary", [False, True])
def test_scene_walks_match_the_oracle(deep_top, binary):
    ter = scenes.terrain(grid=140, size=60.0, n_boxes=0, seed=3)  # 38,642 triangles: opened into two pieces or more
    cube = scenes.gen_cube()
    maps = [rm.Map(ter.vertices, ter.faces), rm.Map(*cube)]
    if binary:  # the same link again: the tree is unchanged, its 4-wide form no longer walked
        left = int(maps[1].export()["links"][0][0])
        _lib.call("rmg_map_debug_set_child", maps[1].handle, 0, 0, left)
    rng = np.random.default_rng(5)
    if deep_top:
        c = chain_centres()
        insts = [dict(geometry=1, T=pose(quat(rng.standard_normal(3), 0.3 * i), p), scale=(0.6, 0.5, 0.4), geom_id=1,
                      object_id=i) for i, p in enumerate(c)]
    else:
        insts = [dict(geometry=1, T=pose(quat(rng.standard_normal(3), 0.3 * i), [*rng.uniform(-20, 20, 2), rng.uniform(5, 12)]),
                      scale=rng.uniform(0.5, 3.0, 3).astype(np.float32), geom_id=1, object_id=i) for i in range(60)]
    insts.append(dict(geometry=0, T=pose(quat([0, 0, 1], 0.4), [1.0, 2.0, -15.0]), geom_id=0, object_id=5000))
    insts.append(dict(geometry=0, T=IDENT.copy(), geom_id=0, object_id=5001))
    meshes = [(ter.vertices, ter.faces), cube]
    scene = rm.Scene(maps, [rm.Instance(i["geometry"], T=i["T"], scale=i.get("scale", (1, 1, 1)), geom_id=i["geom_id"],
                                        object_id=i["object_id"]) for i in insts])
    n = 160
    model = sensors.O1DnModel(width=n, height=1, range=sensors.Interval(0.1, 2000.0), orig=(0.0, 0.0, 0.0),
                              dirs=sensors.sphere_directions(n, seed=9))
    poses = np.stack([pose(IDENT[:4], [0.3, -0.2, 14.0]), pose(IDENT[:4], [5.0, 3.0, 2.0])])
    sim = rm.make_simulator(model, scene)
    got = sim.simulate(torch.from_numpy(poses).cuda()).tensors()
    want = InstancedScene(meshes, insts).simulate(model, IDENT, poses)
    assert scene.status() == 0
    for a in ALL:
        g = got[a].cpu().numpy()
        g = g.view(np.uint32) if a.endswith("_ids") else g
        w = np.asarray(want[a]).reshape(g.shape)
        assert np.array_equal(g, w, equal_nan=not a.endswith("_ids") and g.dtype.kind == "f"), a
