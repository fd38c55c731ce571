"""bench.py's mirror of the library's bin-size choice (bin_edge): the automatic size on both sides of each of
its limits, and a requested one."""
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_for_bins", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("width,height,ntris,tile,edge", [
    (800, 600, 12, 0, 16), (1920, 1080, 8191, 0, 16), (1920, 1080, 8192, 0, 32),  # by triangles
    (2048, 2048, 12, 0, 16), (2049, 2048, 12, 0, 32), (16384, 16384, 100, 0, 32),  # by bins of one counting pass
    (1920, 1080, 100_000, 16, 16), (256, 256, 100, 32, 32), (64, 64, 10, 8, 8), (16384, 16384, 100, 8, 8),  # asked for
    (640, 480, 100, 12, 16)])  # not a bin size
def test_bin_edge(bench, width, height, ntris, tile, edge):
    assert bench.bin_edge(width, height, ntris, tile) == edge
