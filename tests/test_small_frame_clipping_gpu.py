"""Clipping in small frames (k_front), where one warp classifies up to four triangles, one per
lane, and then clips those that straddle a plane with all its lanes: straddlers in every lane's place, alone
and together, among triangles inside, culled and clipped away, in full and partial warps. The box and
the polygon offset of every triangle have one writer each, its lane or the clipping warp's first lane;
samples, image and counts equal the oracle's bit for bit (src/rasterizer/clipping.rs:62-190)."""
import numpy as np
import pytest

from parity import assert_parity
from rusterizer_gb300 import math as rm
from rusterizer_gb300 import scenes

pytestmark = pytest.mark.gpu

INSIDE, STRADDLES, CLIPPED_AWAY, OUTSIDE = range(4)


def triangle(kind, rng):
    """Clip-space corners (w = 1), clockwise on the screen."""
    z = rng.uniform(-0.8, 0.8, 3)
    if kind == CLIPPED_AWAY:  # past a corner of the view: outside no single plane, nothing left of it
        s = rng.choice([-1.0, 1.0], 2)
        xy = np.array([(2.5, 0.0), (0.0, 2.5), (2.5, 2.5)]) * s + rng.uniform(-0.1, 0.1, (3, 2))
    else:
        xy = rng.uniform(-0.6, 0.6, 2) + rng.uniform(-0.3, 0.3, (3, 2))
        if kind == OUTSIDE:
            xy[:, 0] += 2.0
        elif kind == STRADDLES:
            if rng.random() < 0.5:
                xy[rng.integers(3)] *= 6.0
                xy[0, 0] = 1.0 + rng.uniform(0.1, 1.0)
            else:
                z[0], z[1] = -1.0 - rng.uniform(0.1, 1.0), rng.uniform(-0.8, 0.8)
    v = np.concatenate([xy, z[:, None]], 1).astype(np.float32)
    a = np.cross(np.append(v[1, :2] - v[0, :2], 0), np.append(v[2, :2] - v[0, :2], 0))[2]
    return v if a < 0 else v[[0, 2, 1]]


def scene(kinds, seed, msaa=4, fs=scenes.FS_COLOR):
    rng = np.random.default_rng(seed)
    pos = np.concatenate([triangle(k, rng) for k in kinds])
    n = len(pos)
    return {"name": "kinds", "width": 96, "height": 64, "msaa": msaa, "clear_depth": float(np.finfo(np.float32).max),
            "view": rm.identity(), "proj": rm.identity(), "textures": [scenes.noise_texture(16, rng)],
            "draws": [{"pos": pos, "uv": rng.random((n, 2), dtype=np.float32),
                       "rgba": rng.random((n, 4), dtype=np.float32),
                       "idx": np.arange(n, dtype=np.uint32).reshape(-1, 3), "world": rm.identity(), "fs": fs}]}


@pytest.mark.parametrize("mask", range(16))
def test_straddlers_in_each_lane(mask):
    """Four triangles, one warp: those in `mask` straddle a plane."""
    kinds = [STRADDLES if mask >> t & 1 else INSIDE for t in range(4)]
    _, stats = assert_parity(scene(kinds, mask), log=False)
    assert stats["shaded_samples"] > 0


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 32, 33, 67, 128, 1001])
@pytest.mark.parametrize("fs,msaa", [(scenes.FS_COLOR, 4), (scenes.FS_TEXTURE, 1)])
def test_all_straddle(n, fs, msaa):
    assert_parity(scene([STRADDLES] * n, n, msaa=msaa, fs=fs), log=False, nthreads=4)


@pytest.mark.parametrize("n", [4, 7, 61, 300])
def test_mixed_with_clipped_away_and_culled(n):
    kinds = np.random.default_rng(n).integers(0, 4, n)
    assert_parity(scene(kinds, 100 + n), log=False, nthreads=4)


def test_nothing_left_of_any():
    img, stats = assert_parity(scene([CLIPPED_AWAY] * 37, 9), log=False)
    assert stats["shaded_samples"] == 0
