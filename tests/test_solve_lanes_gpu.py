"""The Umeyama step solved with four lanes per problem against the one-thread solve (svd) and the
property that defines its rotation, over matrices where one warp holds easy and hard problems: equal
singular values, graded and tiny and huge ones, reflections, ranks two to zero, NaN."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rs(built):
    torch.cuda.set_device(0)
    from rmagine_gb300 import statistics
    return statistics


def rotation(rng):
    q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
    return q * np.sign(np.linalg.det(q))


def matrices(n, seed):
    rng = np.random.default_rng(seed)
    spectra = [(1, .5, .2), (1, 1, 1), (1, 1, .3), (1, .3, .3), (1, .02, .01), (1, 1e-3, 5e-4), (1, .9999999, .5), (1, .4, -.1),
               (1, .4, 0), (1, 0, 0), (0, 0, 0), (1, 1e-5, 1e-6)]
    out = []
    for i in range(n):
        s = np.array(spectra[i % len(spectra)]) * 10.0 ** rng.integers(-15, 16)
        u, v = (np.eye(3), np.eye(3)) if i % 5 == 4 else (rotation(rng), rotation(rng))
        out.append(u @ np.diag(s) @ v.T)
    return np.array(out, np.float32).reshape(n, 3, 3)


def to_matrix(q):
    x, y, z, w = q.astype(np.float64).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 2 * (x * y + z * w),
                     1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 2 * (x * z - y * w), 2 * (y * z + x * w),
                     1 - 2 * (x * x + y * y)], -1).reshape(-1, 3, 3)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 1203])
def test_solve_is_the_best_rotation(rs, n):
    C = matrices(n, seed=n)
    nan = n > 8
    if nan:
        C[5, 1, 2] = np.nan
    stats = np.zeros((n, 16), np.float32)
    stats[:, 0:3] = np.random.default_rng(n).standard_normal((n, 3))
    stats[:, 3:6] = 2.0
    stats[:, 6:15] = C.transpose(0, 2, 1).reshape(n, 9)
    stats[:, 15:16].view(np.uint32)[:] = 10
    T = rs.umeyama_transform(torch.from_numpy(stats)).cpu().numpy()
    if nan:
        assert np.array_equal(T[5, :4], np.array([0, 0, 0, 1], np.float32))
        T, C, stats = np.delete(T, 5, 0), np.delete(C, 5, 0), np.delete(stats, 5, 0)
    # binary32 quaternions: 2^-24 per component, up to 4 in a matrix element
    assert np.abs(np.linalg.norm(T[:, :4].astype(np.float64), axis=1) - 1).max() < 3e-7
    R = to_matrix(T[:, :4])
    u, s, vt = np.linalg.svd(C.astype(np.float64))
    sign = np.sign(np.linalg.det(u) * np.linalg.det(vt))
    best = s[:, 0] + s[:, 1] + sign * s[:, 2]
    got = np.einsum("nij,nij->n", R, C.astype(np.float64))  # trace(R^T C): largest for the rotation sought
    assert np.all(np.abs(got - best) <= 1.5e-6 * s[:, 0])
    # where the rotation is unique it is the one-thread solve's
    sure = s[:, 1] + sign * s[:, 2] > 1e-2 * s[:, 0]
    U, _, V = (x.cpu().numpy().astype(np.float64) for x in rs.svd(torch.from_numpy(C), rotations=True))
    assert np.abs(R - U @ V.transpose(0, 2, 1))[sure].max() < 2e-6 if sure.any() else True
    t = stats[:, 3:6] - np.einsum("nij,nj->ni", R, stats[:, 0:3].astype(np.float64))
    assert np.abs(T[:, 4:7] - t).max() < 1e-5
