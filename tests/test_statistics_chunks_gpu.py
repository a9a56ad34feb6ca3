"""Statistics of one large batch whose equal parts, rounded up to four correspondences, need fewer
CTAs than parts: every correspondence counts once, on the vector path and on the one-by-one path
(arrays off a 16-byte boundary), forward and backward."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rs(built):
    torch.cuda.set_device(0)
    from rmagine_gb300 import statistics
    return statistics


def sizes():
    """Batch sizes for which the last of the most parts would start far behind the batch's end."""
    most = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    found = [n for n in range(4096 * most, 4096 * most + 2_000_000, 13)
             if (most - 1) * (-(-(-(-n // most)) // 4) * 4) > n + 255]
    return [found[0], found[len(found) // 2], found[-1]]


@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("shift", [0, 1])
def test_every_correspondence_counts_once(rs, which, shift):
    n = sizes()[which]
    gen = torch.Generator("cuda").manual_seed(n)
    # multiples of 1/8 below 4: their binary32 runs and sums are exact, whatever the order
    d = torch.randint(-31, 32, (n + shift, 3), generator=gen, device="cuda").float()[shift:] / 8
    m = torch.randint(-31, 32, (n + shift, 3), generator=gen, device="cuda").float()[shift:] / 8
    st, _ = rs.statistics_p2p(d[None], m[None])
    got = rs.decode_stats(st)
    assert got["n"][0] == n
    dd, mm = d.double(), m.double()
    # one rounding to binary32 of numbers below 8
    for k, want in (("dataset_mean", dd.mean(0)), ("model_mean", mm.mean(0)),
                    ("covariance", mm.T @ dd / n - torch.outer(mm.mean(0), dd.mean(0)))):
        assert np.abs(got[k][0] - want.cpu().numpy()).max() <= 2.0 ** -24 * 8, k
    # the backward of each part, given the whole batch's statistics, is that part's of the whole
    gR, gt = torch.randn(9, generator=gen, device="cuda"), torch.randn(3, generator=gen, device="cuda")
    whole = rs.umeyama_backward(d[None], m[None], st, gR, gt)
    for part in (slice(0, n // 3), slice(n // 3, n)):
        for a, b in zip(whole, rs.umeyama_backward(d[None, part], m[None, part], st, gR, gt)):
            assert torch.equal(a[:, part], b)


def test_backward_of_more_than_it_can_count_is_refused(rs):
    """Within a CTA's width of 2^32 the stream kernel's count would not come to an end."""
    from rmagine_gb300 import _lib as L

    x = torch.zeros(64, device="cuda")
    pc = rs.UmeyamaReductionConstraints().to_c()
    import ctypes as C

    for n in (0xFFFFFF01, 0xFFFFFFFF):
        st = L.load().rmg_umeyama_backward(None, 0, rs._ptr(x), None, None, rs._ptr(x), None, None, C.byref(pc), 1, n,
                                           rs._ptr(x), None, None, rs._ptr(x), rs._ptr(x), rs._stream())
        assert st == L.RMG_ERR_INVALID_ARG
