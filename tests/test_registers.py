"""The statistics kernels keep a thread's correspondences in registers: none of their variants spills
at the registers that its launch bounds leave it (read from the assembler's report)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

from rmagine_gb300 import build as lib_build


def test_statistics_kernels_do_not_spill(tmp_path):
    if shutil.which("nvcc") is None and not Path("/usr/local/cuda/bin/nvcc").exists():
        pytest.skip("no nvcc")
    cmd = [lib_build.nvcc(), *lib_build.ARCH, *lib_build.NVCC_FLAGS, "-Xptxas", "-v", "-c",
           str(lib_build.CSRC / "stats.cu"), "-o", str(tmp_path / "stats.o")]
    out = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    spills = {}
    for name, report in re.findall(r"Function properties for (\S+)\n\s*(.*)", out):
        if "7k_stats" in name:
            spills[name] = re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", report).groups()
    assert len(spills) >= 8
    assert all(v == ("0", "0") for v in spills.values()), spills
