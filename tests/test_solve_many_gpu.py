"""Umeyama transforms of more problems than a quarter of 2^32 (four lanes each)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_more_than_a_quarter_of_four_billion_problems(built):
    from rmagine_gb300 import _lib as L
    from rmagine_gb300 import statistics as rs

    torch.cuda.set_device(0)
    n = (1 << 30) + 5
    if torch.cuda.mem_get_info()[0] < 112 << 30:
        pytest.skip("needs 97 GB of device memory")
    one = torch.zeros(16, device="cuda")
    one[6], one[10], one[14] = 1.0, 0.5, 0.25
    one[15:].view(torch.int32)[:] = 10
    stats = one.expand(n, 16).contiguous()
    at = [0, 4, (1 << 30) - 1, 1 << 30, n - 1]
    for k, i in enumerate(at):
        stats[i, 3] = float(k + 1)  # model mean: the translation
    out = torch.full((n, 8), float("nan"), device="cuda")
    L.call("rmg_umeyama_transform", rs._ptr(stats), n, rs._ptr(out), rs._stream())
    assert out[at, 4].cpu().tolist() == [1.0, 2.0, 3.0, 4.0, 5.0]
    assert out[at, 3].cpu().tolist() == [1.0] * 5
    del stats, out
    torch.cuda.empty_cache()
