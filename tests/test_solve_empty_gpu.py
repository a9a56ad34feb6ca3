"""Umeyama transforms where some problems of a warp have no correspondences: those give the identity,
their neighbours what they give alone."""
import numpy as np
import pytest
import torch

from test_solve_lanes_gpu import matrices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("empty", [[0], [7], [1, 2, 6], list(range(8)), [3, 8, 9, 31, 32]])
def test_problems_without_correspondences(built, empty):
    from rmagine_gb300 import statistics as rs

    torch.cuda.set_device(0)
    n = 40
    st = np.zeros((n, 16), np.float32)
    st[:, 0:3] = np.random.default_rng(1).standard_normal((n, 3))
    st[:, 3:6] = 2.0
    st[:, 6:15] = np.repeat(matrices(12, seed=3)[[0, 2, 4, 7]], 10, 0).transpose(0, 2, 1).reshape(n, 9)
    st[:, 15:16].view(np.uint32)[:] = 10
    want = rs.umeyama_transform(torch.from_numpy(st)).cpu().numpy()
    st[empty, 15] = 0.0
    got = rs.umeyama_transform(torch.from_numpy(st)).cpu().numpy()
    want[empty, :7] = [0, 0, 0, 1, 0, 0, 0]
    assert np.array_equal(got[:, :7], want[:, :7])
