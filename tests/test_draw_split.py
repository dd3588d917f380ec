"""The split of a draw list's samples over the raster's warps, on the CPU: every
sample once, whatever the items' sizes, and with more than 2^32 samples (a tree
past an arena overflow)."""
import os
import subprocess

import pytest

from remobench_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("draw") / "probe")
    subprocess.check_call([build._nvcc(), "-O1", "-std=c++17", *build.ARCH, "-x", "cu",
                           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "remobench_b200", "csrc"),
                           "-o", exe, os.path.join(ROOT, "tests", "host_draw_probe.cpp")])
    return exe


@pytest.mark.parametrize("warps,items", [
    (9472, [(1, 1)]), (9472, [(3, 0), (1, 31), (2, 0), (1, 33)]), (7, [(100, 1000)]), (9472, [(2000, 25_001)]),
    (9472, [(1, 4_000_000_000), (10, 7), (3, 0), (1, 4_294_967_295)]), (9472, [(1000, 3_000_000), (500, 3_000_001)]),
    (7104, [(100_000, 50_000)])])
def test_every_sample_once(probe, warps, items):
    out = subprocess.run([probe, str(warps), *[str(v) for pair in items for v in pair]], capture_output=True, text=True,
                         check=True).stdout
    total, drawn, bad = (int(v) for v in out.split())
    assert total == sum(n * c for n, c in items) == drawn and bad == 0
