"""The four-lane solve: a problem's result does not depend on what else is in the call, and on graded
covariances its rotation is as close to the binary64 one as the one-thread solve's."""
import numpy as np
import pytest
import torch

from test_solve_lanes_gpu import rotation, to_matrix

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rs(built):
    torch.cuda.set_device(0)
    from rmagine_gb300 import statistics
    return statistics


def records(C):
    st = np.zeros((len(C), 16), np.float32)
    st[:, 6:15] = C.transpose(0, 2, 1).reshape(-1, 9)
    st[:, 15:16].view(np.uint32)[:] = 10
    return st


def graded(n, spectra, seed):
    rng = np.random.default_rng(seed)
    return np.array([rotation(rng) @ np.diag(spectra[i % len(spectra)]) @ rotation(rng).T for i in range(n)], np.float32)


def test_a_problem_stands_alone(rs):
    """Bytes of every problem in a shuffled call and next to itself only."""
    C = graded(800, [(1, .5, .2), (1, .999999, .2), (1, 1e-4, 9e-5), (1, 1e-6, 1e-7), (1, 1, 1), (1, 0, 0), (0, 0, 0)], 1)
    C[3, 0, 1] = np.nan
    st = records(C)
    want = rs.umeyama_transform(torch.from_numpy(st)).cpu().numpy().view(np.uint32)
    for seed in range(3):
        p = np.random.default_rng(seed).permutation(len(st))
        got = rs.umeyama_transform(torch.from_numpy(st[p])).cpu().numpy().view(np.uint32)
        assert np.array_equal(got, want[p])
    for i in range(0, 40):
        alone = rs.umeyama_transform(torch.from_numpy(st[i:i + 1].repeat(9, 0))).cpu().numpy().view(np.uint32)
        assert np.array_equal(alone, want[i:i + 1].repeat(9, 0)), i
    # the backward's coefficients: each batch of four points in a call of its own
    rng = np.random.default_rng(2)
    d = torch.from_numpy(rng.standard_normal((9, 4, 3)).astype(np.float32)).cuda()
    m = torch.from_numpy(rng.standard_normal((9, 4, 3)).astype(np.float32)).cuda()
    s9 = torch.from_numpy(st[:9]).cuda()
    gR = torch.from_numpy(rng.standard_normal((9, 9)).astype(np.float32)).cuda()
    whole = rs.umeyama_backward(d, m, s9, gR)
    for i in range(9):
        for a, b in zip(whole, rs.umeyama_backward(d[i:i + 1], m[i:i + 1], s9[i:i + 1], gR[i:i + 1])):
            assert torch.equal(a[i:i + 1].view(torch.int32), b.view(torch.int32)), i


@pytest.mark.parametrize("a", [1e-1, 1e-3, 1e-5, 1e-6, 1e-7])
@pytest.mark.parametrize("b", [1.0, .999, .5, 1e-2, 0.0, -.5])
def test_graded_spectra_against_binary64(rs, a, b):
    """Singular values 1, a, a b.  Both solves form C^T C, whose rounding of some 2^-53 turns the
    rotation by that over its eigenvalues, (a + a b) a at the least, times the few sums in it; and
    a binary32 quaternion has 2^-24 per component, up to 4 in a matrix element."""
    C = graded(400, [(1, a, a * b)], 7)
    u, s, vt = np.linalg.svd(C.astype(np.float64))
    u[:, :, 2] *= np.sign(np.linalg.det(u) * np.linalg.det(vt))[:, None]
    R = u @ vt
    err = np.abs(to_matrix(rs.umeyama_transform(torch.from_numpy(records(C))).cpu().numpy()[:, :4]) - R).max((1, 2))
    assert err.mean() <= 2.0 ** -24 * 4 + 16 * 2.0 ** -53 / (a * (a + a * b))
    U, _, V = (x.cpu().numpy().astype(np.float64) for x in rs.svd(torch.from_numpy(C), rotations=True))
    one = np.abs(U @ V.transpose(0, 2, 1) - R).max((1, 2))
    # binary32 factors of the one-thread solve: 2^-24 of each of six products
    assert err.mean() <= 1.25 * one.mean() + 2.0 ** -24 * 4
