"""Bins filled from the tiles' side (small frames, k_bin_gather) and from the chunks' side (the others),
at the sizes where either can go wrong: one triangle, a partial warp and chunk, the largest small
frame and one triangle more, blocks of 8 and of 4 bins cut by the image edge, quadrant masks, triangles over many
bins, several draws, bins over more than one counting band, and the raster queue's classes at heavy
limits on and between their steps. Binning decides nothing about a pixel, so samples, image and
counts equal the oracle's bit for bit.
"""
import numpy as np
import pytest

from parity import assert_parity
from rusterizer_gb300 import scenes

pytestmark = pytest.mark.gpu

SMALL = 8160  # kGatherTris


def soup(ntris, w, h, seed, msaa=4, min_px=1.0, max_px=64.0):
    rng = np.random.default_rng(seed)
    s = scenes.soup_scene(2, w, h, msaa, rng, 32)
    s["draws"] = [dict(scenes.soup(ntris, w, h, rng, min_px=min_px, max_px=max_px), world=s["draws"][0]["world"], fs=0)]
    return s


@pytest.mark.parametrize("ntris,tile,w,h", [
    (1, 16, 33, 17), (31, 8, 257, 131), (33, 32, 300, 200), (97, 0, 1366, 769), (4097, 8, 517, 389),
    (SMALL, 16, 640, 360), (SMALL + 1, 16, 640, 360), (SMALL, 32, 333, 221), (SMALL + 1, 8, 333, 221),
    (SMALL + 1, 8, 2101, 1100)])
def test_sizes(ntris, tile, w, h):
    assert_parity(soup(ntris, w, h, ntris + tile), tile=tile, log=False, nthreads=8)


@pytest.mark.parametrize("tile", [8, 16, 32])
def test_triangles_over_many_bins(tile):
    assert_parity(soup(300, 700, 500, tile, min_px=64.0, max_px=700.0), tile=tile, log=False, nthreads=8)


@pytest.mark.parametrize("msaa", [1, 4])
def test_several_draws(msaa):
    s = soup(70, 400, 300, 5, msaa=msaa)
    more = [soup(n, 400, 300, 6 + n)["draws"][0] for n in (1, 64, 333)]
    s["draws"] += [dict(d, fs=k % 3) for k, d in enumerate(more)]
    assert_parity(s, log=False, nthreads=8)


@pytest.mark.parametrize("heavy", [1, 2, 4, 8, 32, 100, 4096, 8192])
def test_heavy_limits(heavy):
    assert_parity(soup(9000, 96, 80, 3), tile=16, log=False, nthreads=8, heavy_entries=heavy)
