"""The launch-shape rule (batch_shape.cuh, compiled here): empty blocks for batches of many small events are what it
must not launch, and too few blocks for uneven or large ones."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cms-julia_b200" / "csrc"
MAIN = """
#include <cstdio>
#include <cstdlib>
#include "batch_shape.cuh"
int main(int, char** v) { std::printf("%d", pxl::blocks_per_event(std::atoi(v[1]), std::strtoull(v[2], nullptr, 10))); }
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return lambda e, words: int(subprocess.run([str(d / "main"), str(e), str(e * words)], capture_output=True).stdout)


# events, words per event (0: unknown), blocks: 100 tracks are 2000 words, pileup 10 some 11 000, pileup 50 37 000
@pytest.mark.parametrize("events,words,blocks", [(1, 2000, 256), (1, 130000, 256), (37, 0, 256), (38, 37000, 249),
                                                 (111, 70000, 85), (296, 2000, 32), (512, 37000, 32), (512, 2000, 18),
                                                 (2368, 2000, 4), (4096, 2000, 4), (4096, 0, 4), (2048, 11000, 10),
                                                 (4096, 4000000, 32), (100000, 0, 4)])
def test_blocks_per_event(rule, events, words, blocks):
    assert rule(events, words) == blocks
