"""A map file whose parent fields do not agree with its links: the links count, so that a refit of the
loaded map (which climbs from the leaves) ends and gives the boxes of the map that was saved."""
import numpy as np
import pytest

from test_meshio import map_file

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["leaves", "nodes", "both"])
def test_parents_come_from_the_links(built, tmp_path, how):
    import torch

    import rmagine_gb300 as rm
    from rmagine_gb300 import scenes

    torch.cuda.set_device(0)
    s = scenes.box_room(seed=4, n_boxes=10)
    m = rm.Map(s.vertices, s.faces)
    m.save(tmp_path / "a.rmgmap")
    g = m.export()
    n = len(s.faces)
    rng = np.random.default_rng(1)
    parents = np.zeros(n, np.int32)
    for side in (0, 1):
        c = g["links"][:, side]
        parents[~c[c < 0]] = np.nonzero(c < 0)[0]
    links = g["links"].copy()
    if how != "nodes":
        parents = rng.permutation(parents)
    if how != "leaves":
        links[1:, 2] = rng.integers(0, n - 1, n - 2)
    nodes = np.concatenate([g["boxes"], links.view(np.float32)], 1)
    data = map_file(nodes, g["tris"], s.faces, s.vertices, g["leaf_order"], parents, depth=m.info()["depth"])
    assert len(data) == (tmp_path / "a.rmgmap").stat().st_size
    (tmp_path / "b.rmgmap").write_bytes(data)
    got = rm.Map.load(tmp_path / "b.rmgmap")
    got.save(tmp_path / "c.rmgmap")
    assert (tmp_path / "c.rmgmap").read_bytes() == (tmp_path / "a.rmgmap").read_bytes()
    moved = s.vertices + np.float32(0.25) * rng.standard_normal(s.vertices.shape).astype(np.float32)
    for x in (m, got):
        x.refit(moved)
    a, b = m.export(), got.export()
    for k in a:
        assert np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)), k
