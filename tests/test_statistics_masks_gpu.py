"""Statistics whose points start on 16 bytes and whose masks and ids do not (carved out of one buffer):
read four correspondences at a time all the same, with the sums of aligned masks bit for bit."""
import numpy as np
import pytest
import torch

from test_statistics import icp_batches
from test_statistics_ragged_gpu import shifted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p2l", [False, True])
@pytest.mark.parametrize("B,N", [(1, 4), (5, 64), (3, 4096), (2, 20012), (3, 4099)])
def test_masks_off_their_boundary(built, B, N, p2l):
    from rmagine_gb300 import statistics as rs

    torch.cuda.set_device(0)
    src, tgt, _, _ = icp_batches(B, N, seed=B + N)
    rng = np.random.default_rng(N)
    dm, mm = (rng.random((2, B, N)) < 0.8).astype(np.uint8)
    di, mi = rng.integers(0, 2, (2, B, N)).astype(np.int32)
    nrm = rng.standard_normal((B, N, 3)).astype(np.float32)
    P = rs.UmeyamaReductionConstraints(dataset_id=1, model_id=0, max_dist=20.0)
    kw = dict(params=P, model_normals=torch.from_numpy(nrm).cuda() if p2l else None)
    d, m = torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda()

    def run(shift):
        s, T = rs.statistics(d, m, dataset_mask=shifted(dm, shift), model_mask=shifted(mm, shift),
                             dataset_ids=shifted(di, shift), model_ids=shifted(mi, shift), **kw)
        return s.view(torch.int32).cpu(), T.view(torch.int32).cpu()

    want = run(0)
    for shift in (1, 2, 3):
        for a, b in zip(run(shift), want):
            assert torch.equal(a, b), shift
