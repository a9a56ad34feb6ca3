"""The host forms' pose chunks (csrc/chunks.h, compiled for the CPU): they cover all poses in order,
fit the staging memory, and hold the least number of poses, the last one a quarter of it, wherever the
staging memory allows it."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "rmagine_gb300" / "csrc"
MAIN = r"""
#include <cstdio>
#include "chunks.h"
int main() {
  unsigned n; size_t want, least;
  while (std::scanf("%u %zu %zu", &n, &want, &least) == 3) {
    const size_t chunk = rmg::chunk_poses(n, want, least);
    std::printf("%zu", chunk);
    for (uint32_t p : rmg::chunk_schedule(n, chunk, least)) std::printf(" %u", p);
    std::printf("\n");
  }
}
"""


@pytest.fixture(scope="module")
def schedule(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("chunks")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", str(CSRC), str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def run(cases):
        text = "\n".join(" ".join(map(str, c)) for c in cases)
        out = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True, check=True).stdout
        rows = [list(map(int, line.split())) for line in out.splitlines()]
        assert len(rows) == len(cases)
        return [(r[0], r[1:]) for r in rows]

    return run


def test_chunks_cover_the_poses_and_keep_their_bounds(schedule):
    cases = [(n, want, least) for n in list(range(1, 140)) + [200, 299, 300, 1000, 1001, 4097]
             for want in (0, 1, 2, 7, 49, 50, 97, 98, 128, 789) for least in (0, 1, 7, 16, 49) if least <= max(1, want)]
    for (n, want, least), (chunk, first) in zip(cases, schedule(cases)):
        sizes = [b - a for a, b in zip(first, first[1:])]
        assert first[0] == 0 and first[-1] == n and min(sizes) >= 1 and max(sizes) <= chunk <= max(1, want), (n, want, least)
        if chunk >= min(n, least + least // 4):  # room for a rest to go with the chunk before it
            assert min(sizes[:-1] + [n]) >= min(n, least) and sizes[-1] >= min(n, least // 4), (n, want, least, sizes)
        if n >= least + max(1, least // 4) and n >= 2 and want >= 1:  # two chunks overlap
            assert len(sizes) >= 2, (n, want, least)


def test_the_quoted_calls(schedule):
    (_, a), (_, b), (_, c) = schedule([(200, 789, 49), (50, 789, 49), (64, 789, 49)])
    assert a == [0, 100, 150, 200] and b == [0, 50] and c == [0, 49, 64]
