"""Statistics of batches whose sizes are no multiple of the four correspondences a thread loads at a
time: groups shared by neighbouring batches and CTAs, a cut-short last group of the whole array,
arrays that start off a 16-byte boundary (the one-by-one path), masks and ids; and the pose
gradient's final sum where its warps do not fill the summing threads."""
import numpy as np
import pytest
import torch

from oracle import stats as ost
from test_statistics import gpu_stats, icp_batches

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rs(built):
    from rmagine_gb300 import statistics as rs_

    torch.cuda.set_device(0)
    return rs_


def shifted(a, by):
    """A CUDA copy of `a` that starts `by` elements behind a 16-byte boundary."""
    t = torch.from_numpy(np.ascontiguousarray(a))
    buf = torch.zeros(t.numel() + by, dtype=t.dtype, device="cuda")
    buf[by:] = t.reshape(-1).cuda()
    return buf[by:].view(t.shape)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("B,N", [(1, 1), (1, 2), (3, 3), (5, 5), (2, 1023), (7, 4097), (3, 8193), (2, 20011)])
def test_ragged_batches_match_the_oracle(rs, B, N, shift):
    src, tgt, _, _ = icp_batches(B, N, seed=B + N, outliers=0.0)
    rng = np.random.default_rng(N)
    dm, mm = (rng.random((2, B, N)) < 0.8).astype(np.uint8)
    di, mi = rng.integers(0, 2, (2, B, N)).astype(np.uint32)
    P = rs.UmeyamaReductionConstraints(dataset_id=1, model_id=0)
    ids = dict(dids=di, mids=mi, dataset_id=1, model_id=0)
    d, m = shifted(src, shift), shifted(tgt, shift)
    for dmask, use_ids in ((None, False), (dm, False), (dm, True)):
        kw = {}
        if dmask is not None:
            kw = dict(dataset_mask=shifted(dm, shift), model_mask=shifted(mm, shift))
        if use_ids:
            kw.update(dataset_ids=shifted(di.view(np.int32), shift), model_ids=shifted(mi.view(np.int32), shift))
        got, _ = gpu_stats(rs, d, m, params=P if use_ids else None, **kw)
        want = ost.stats(*ost.correspondences(src, tgt, dmask=dmask, mmask=None if dmask is None else mm,
                                              **(ids if use_ids else {})))
        # the kernels sum binary32 products of offsets of up to E = 100 m around the batch's first
        # pair: 2^-24 E^2 for a product's offsets and its rounding each, in runs of at most 32 and
        # a 5-level sum, whatever the size of the covariance itself (zero for a single pair)
        assert np.array_equal(got["n"], want["n"])
        assert np.abs(got["covariance"] - want["covariance"]).max() <= 16 * 2.0 ** -24 * 100.0 ** 2
        for k in ("dataset_mean", "model_mean"):
            assert np.abs(got[k] - want[k]).max() <= 16 * 2.0 ** -24 * 100.0


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 33), (4, 8), (5, 129), (33, 65)])
def test_gradient_sum_over_any_number_of_warps(built, rows, cols):
    import rmagine_gb300 as rm
    from rmagine_gb300 import scenes
    from rmagine_gb300.grad import range_pose_grad

    s = scenes.box_room(seed=0, n_boxes=20)
    sim = rm.make_simulator(rm.ouster_like(rows, cols) if rows > 1 else rm.depth_camera(cols, rows), rm.Map(s.vertices, s.faces))
    n = 3
    poses = torch.from_numpy(scenes.room_poses(n, seed=2)).cuda()
    obs = sim.simulate(poses, attrs=("ranges",)).ranges + 0.05
    grad, loss = range_pose_grad(sim, poses, obs)
    # the same observations one ray at a time: per-ray losses and gradients summed in binary64
    per = rows * cols
    want_g, want_l, mag = np.zeros((n, 6)), np.zeros(n), np.zeros((n, 6))
    for i in range(per):
        far = torch.full((n, per), -1.0, device="cuda")  # below range.min: no part of the loss
        far[:, i] = obs.reshape(n, per)[:, i]
        g1, l1 = range_pose_grad(sim, poses, far.reshape(-1))
        want_g += g1.double().cpu().numpy()
        mag += np.abs(g1.double().cpu().numpy())
        want_l += l1.double().cpu().numpy()
    # a warp adds 32 rays in binary32 (5 levels, 2^-24 each), the rest is binary64 and one rounding
    assert (np.abs(grad.cpu().numpy() - want_g) <= 8 * 2.0 ** -24 * mag + 1e-12).all()
    assert (np.abs(loss.cpu().numpy() - want_l) <= 8 * 2.0 ** -24 * want_l + 1e-12).all()
