"""The four-lane solve where C^T C is diagonal: the same rotations as the one-thread solve (bit for bit
up to the quaternion's rounding), in warps of such problems alone and among others; and large calls of
them take no longer than the general problems do."""
import numpy as np
import pytest
import torch

from test_solve_alone_gpu import records
from test_solve_lanes_gpu import matrices, to_matrix

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rs(built):
    torch.cuda.set_device(0)
    from rmagine_gb300 import statistics
    return statistics


def diagonal_ones():
    """Signed permutations times every pattern of (0, 1e-15, 0.5, 1, 1e15) on the diagonal, and zero."""
    out = []
    for perm in ([0, 1, 2], [1, 2, 0], [1, 0, 2], [2, 1, 0]):
        for sign in ((1, 1, 1), (1, -1, 1), (-1, 1, -1), (-1, -1, -1)):
            for d in ((0, 0, 0), (1, 0, 0), (0, 1e-15, 0), (0, 0, 1e15), (1, .5, 0), (0, 1, 1), (1, 1, 1), (.5, 1, .25),
                      (1e15, 1, 1e-15)):
                m = np.zeros((3, 3))
                m[np.arange(3), perm] = np.multiply(sign, d)
                out.append(m)
    return np.array(out, np.float32)


def rotations(rs, C):
    return to_matrix(rs.umeyama_transform(torch.from_numpy(records(C))).cpu().numpy()[:, :4])


def test_diagonal_problems_take_the_one_thread_choices(rs):
    C = diagonal_ones()
    U, _, V = (x.cpu().numpy().astype(np.float64) for x in rs.svd(torch.from_numpy(C), rotations=True))
    want = U @ V.transpose(0, 2, 1)
    got = rotations(rs, C)
    assert np.abs(got - want).max() <= 4 * 2.0 ** -24  # a binary32 quaternion's rounding
    # among problems that are not: the same
    other = matrices(len(C), seed=5)
    both = np.stack([C, other, other], 1).reshape(-1, 3, 3)
    assert np.array_equal(rotations(rs, both)[::3], got)


@pytest.mark.parametrize("kind", ["zero", "axis"])
def test_large_calls_are_no_slower_than_general_ones(rs, kind):
    n = 400_000
    C = np.zeros((n, 3, 3), np.float32)
    if kind == "axis":
        C[:, 0, 0] = 1.0
    general = np.tile(np.diag([1.0, .5, .2]).astype(np.float32) + np.float32(.1), (n, 1, 1))

    def best(C):
        st = torch.from_numpy(records(C)).cuda()
        t = []
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            rs.umeyama_transform(st)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return min(t[1:])

    assert best(C) <= 1.0 * best(general)
