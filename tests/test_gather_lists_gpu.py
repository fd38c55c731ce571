"""Bins of small frames filled from a block's list (k_bin_gather): images of few bins, where a block
of 4 x 4 bins lists most of the mesh and its warps share the list from 256 entries on. Lists just below, at
and above that, with a partial last group, one group per warp and one more, and the longest; blocks cut
by the image, quadrant masks, triangles over one bin and over all. Samples, image and counts equal the
oracle's bit for bit."""
import numpy as np
import pytest

from parity import assert_parity
from rusterizer_gb300 import math as rm
from rusterizer_gb300 import scenes

pytestmark = pytest.mark.gpu


def inside(n, w, h, reach, seed, msaa=4):
    """n triangles inside the view, corners up to `reach` of it apart, most of them clockwise."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-0.9, 0.9, (n, 1, 2))
    xy = np.clip(c + rng.uniform(-reach, reach, (n, 3, 2)), -0.99, 0.99)
    e1, e2 = xy[:, 1] - xy[:, 0], xy[:, 2] - xy[:, 0]
    ccw = (e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0] > 0) & (rng.random(n) < 0.9)
    xy[ccw, 1], xy[ccw, 2] = xy[ccw, 2].copy(), xy[ccw, 1].copy()
    pos = np.concatenate([xy, rng.uniform(-0.9, 0.9, (n, 3, 1))], 2).reshape(-1, 3).astype(np.float32)
    return {"name": "inside", "width": w, "height": h, "msaa": msaa, "clear_depth": float(np.finfo(np.float32).max),
            "view": rm.identity(), "proj": rm.identity(), "textures": [scenes.noise_texture(16, rng)],
            "draws": [{"pos": pos, "uv": rng.random((3 * n, 2), dtype=np.float32),
                       "rgba": rng.random((3 * n, 4), dtype=np.float32),
                       "idx": np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), "world": rm.identity(), "fs": 0}]}


# one block: the list is the whole mesh
@pytest.mark.parametrize("n", [31, 255, 256, 257, 511, 512, 513, 1000, 8160])
@pytest.mark.parametrize("tile,reach", [(8, 0.1), (16, 0.6), (32, 0.2)])
def test_one_block(n, tile, reach):
    assert_parity(inside(n, 4 * tile, 4 * tile - 3, reach, n + tile), tile=tile, log=False, nthreads=8)


@pytest.mark.parametrize("tile,w,h", [(8, 67, 35), (16, 200, 150), (32, 161, 290), (16, 70, 7)])
@pytest.mark.parametrize("msaa,reach", [(4, 0.05), (1, 1.0)])
def test_blocks_cut_by_the_image(tile, w, h, msaa, reach):
    assert_parity(inside(3001, w, h, reach, w + h, msaa), tile=tile, log=False, nthreads=8)


def test_all_in_one_bin():
    s = inside(5000, 64, 64, 0.02, 3)
    s["draws"][0]["pos"][:, :2] = s["draws"][0]["pos"][:, :2] * 0.2 + 0.25  # within one 16-pixel bin
    assert_parity(s, tile=16, log=False, nthreads=8)
