"""Maps and workspaces share the library's memory pool: maps built, scanned and destroyed by several
threads on their own streams, right after one another, give what they give alone; a face index
outside the vertices is refused at every size, and the next build is unharmed; the pool is given
back with the last map and on demand."""
import gc
import threading

import numpy as np
import pytest
import torch

import rmagine_gb300 as rm
from rmagine_gb300 import _lib, scenes, sensors
from rmagine_gb300.grad import range_pose_grad

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built):
    torch.cuda.set_device(0)


def scan(grid, seed, stream=None):
    s = scenes.terrain(grid=grid, size=60.0, n_boxes=20, seed=seed)
    poses = torch.from_numpy(scenes.terrain_poses(s, 5, seed=seed, size=60.0)).cuda()
    m = rm.Map(s.vertices, s.faces)
    sim = rm.make_simulator(sensors.ouster_like(16, 128), m)
    out = sim.simulate(poses, attrs=("ranges", "face_ids"))
    g, loss = range_pose_grad(sim, poses, out.ranges + 0.05)
    m.destroy()  # while the work above may still be on its way
    return [t.cpu().numpy() for t in (out.ranges, out.face_ids, g, loss)]


def test_maps_come_and_go_on_several_threads():
    jobs = [[(20 + 17 * i + j, 10 * i + j) for j in range(6)] for i in range(4)]
    want = {job: scan(*job) for row in jobs for job in row}
    errors = []

    def work(row):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for job in row:
                    for a, b in zip(scan(*job), want[job]):
                        assert np.array_equal(a, b), job
        except Exception as e:  # noqa: BLE001 - handed to the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(row,)) for row in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("n", [1, 2, 40, 600, 5000])
@pytest.mark.parametrize("builder", ["sah", "lbvh"])
def test_face_index_out_of_range_is_refused(n, builder):
    v = np.random.default_rng(n).standard_normal((3 * n, 3)).astype(np.float32)
    f = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    for at, bad in ((0, 3 * n), (n - 1, 0xFFFFFFFF)):
        g = f.copy()
        g[at, 1] = bad
        with pytest.raises(rm.RmgError) as e:
            rm.Map(v, g, builder=builder)
        assert e.value.status == _lib.RMG_ERR_INVALID_ARG
    with pytest.raises(rm.RmgError):
        rm.Map(np.zeros((0, 3), np.float32), f, builder=builder)
    assert rm.Map(v, f, builder=builder).info()["n_faces"] == n


def test_the_pool_is_given_back():
    gc.collect()
    _lib.call("rmg_host_staging_trim")
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    s = scenes.terrain(grid=300, size=100.0, n_boxes=0, seed=1)
    maps = [rm.Map(s.vertices, s.faces) for _ in range(2)]
    maps[0].destroy()  # kept for the next map while another lives
    maps[1].destroy()
    gc.collect()
    _lib.call("rmg_host_staging_trim")
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= free0 - (8 << 20)
