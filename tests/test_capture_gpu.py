"""Calls under CUDA graph capture: a process whose first use of the library's memory pool is captured."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

FIRST = """
import torch
from rmagine_gb300 import statistics as rs
torch.cuda.set_device(0)
d = torch.randn(2, 50000, 3, generator=torch.Generator('cuda').manual_seed(1), device='cuda')
m = d + 0.01
st = torch.zeros(2, 16, device='cuda')
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    s, T = rs.statistics(d, m)
    gd, gm = rs.umeyama_backward(d, m, s, torch.ones(2, 9, device='cuda'))
for _ in range(2):
    g.replay()
torch.cuda.synchronize()
s2, T2 = rs.statistics(d, m)
gd2, gm2 = rs.umeyama_backward(d, m, s2, torch.ones(2, 9, device='cuda'))
for a, b in ((s, s2), (T, T2), (gd, gd2), (gm, gm2)):
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
"""


def test_the_first_call_of_a_process_may_be_captured(built):
    r = subprocess.run([sys.executable, "-c", FIRST], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-1500:]
