"""The raster queue's classes at heavy limits with bins on both sides of each: bins of one entry less
than the limit, exactly the limit, one more and other counts, empty ones among them, binned from the tiles'
side (at most 8 160 triangles) and from the chunks' side. Whichever kernel rasters a bin, samples, image
and counts equal the oracle's bit for bit. On the CPU: a bin's class is heavy exactly from the limit on."""
import os
import subprocess

import numpy as np
import pytest

from parity import assert_parity
from rusterizer_gb300 import math as rm
from rusterizer_gb300 import scenes

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "rusterizer_gb300", "csrc")
EDGE = 16


def counts_for(limit, chunked):
    """Entries per bin: around the limit's power of two, others below and above, empty bins between."""
    p = 1 << (limit.bit_length() - 1)
    c = [0, 1, 2, 3, p - 1, 0, p, p + 1, 0, 5, 17, 40]
    if 3 * p < 4000:
        c += [2 * p - 1, 2 * p, max(p // 2, 1)]
    if chunked:
        c += [8161]  # more than a small frame holds
    assert (sum(c) > 8160) == chunked
    assert any(x >= p for x in c) and (p == 1 or any(0 < x < p for x in c))
    return c


def scene(counts, msaa, seed):
    """One bin per count, its triangles inside it, clockwise; bins in rows of five, submission order mixed."""
    rng = np.random.default_rng(seed)
    cols = 5
    rows = -(-len(counts) // cols)
    W, H = cols * EDGE - 3, rows * EDGE
    tri = []
    for b, c in enumerate(counts):
        o = np.array([b % cols, b // cols]) * EDGE
        p = rng.uniform(1.0, EDGE - 4.0, (c, 3, 2)) + o  # whole pixels inside the bin, also in the cut last column
        a = np.cross(np.pad(p[:, 1] - p[:, 0], ((0, 0), (0, 1))), np.pad(p[:, 2] - p[:, 0], ((0, 0), (0, 1))))[:, 2]
        thin = np.abs(a) < 1.0
        p[thin] = o + np.array([(2.0, 2.0), (9.0, 3.0), (3.0, 10.0)])
        a[thin] = 1.0
        p[a < 0] = p[a < 0][:, ::-1]
        tri.append(p)
    v = np.concatenate(tri)[rng.permutation(sum(counts))]
    n = len(v)
    pos = np.concatenate([v[..., :1] / (W / 2) - 1, 1 - v[..., 1:] / (H / 2), rng.uniform(-0.9, 0.9, (n, 3, 1))], 2)
    return {"name": "stacks", "width": W, "height": H, "msaa": msaa, "clear_depth": float(np.finfo(np.float32).max),
            "view": rm.identity(), "proj": rm.identity(), "textures": [scenes.noise_texture(16, rng)],
            "draws": [{"pos": pos.reshape(-1, 3).astype(np.float32), "uv": rng.random((3 * n, 2), dtype=np.float32),
                       "rgba": rng.random((3 * n, 4), dtype=np.float32),
                       "idx": np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), "world": rm.identity(), "fs": 0}]}


def stacked(s):
    """Triangles whose pixel box lies in each bin (all in one each)."""
    W, H = s["width"], s["height"]
    p = s["draws"][0]["pos"].reshape(-1, 3, 3)
    x, y = W * (p[..., 0] + 1) / 2, H * (1 - (p[..., 1] + 1) / 2)
    x0, x1 = np.floor(x.min(1)) // EDGE, (np.ceil(x.max(1)) - 1) // EDGE
    y0, y1 = np.floor(y.min(1)) // EDGE, (np.ceil(y.max(1)) - 1) // EDGE
    assert (x0 == x1).all() and (y0 == y1).all()
    return np.bincount((y0 * 5 + x0).astype(int), minlength=5 * -(-H // EDGE))


LIMITS = [(p, False) for p in (1, 2, 4, 8, 16, 32, 64, 100, 128, 256, 512, 1024, 2048)] + \
         [(p, True) for p in (1, 2, 8, 32, 512, 4096, 8192)]


@pytest.mark.parametrize("limit,chunked", LIMITS)
def test_stacks_hold_what_they_say(limit, chunked):
    c = counts_for(limit, chunked)
    got = stacked(scene(c, 4, limit))
    assert got[:len(c)].tolist() == c and not got[len(c):].any()


@pytest.mark.gpu
@pytest.mark.parametrize("limit,chunked", LIMITS)
@pytest.mark.parametrize("msaa", [4, 1])
def test_bins_on_both_sides_of_the_limit(limit, chunked, msaa):
    assert_parity(scene(counts_for(limit, chunked), msaa, limit), tile=EDGE, log=False, nthreads=8, heavy_entries=limit)


def test_heavy_classes_are_the_counts_from_the_limit_on(tmp_path):
    exe = str(tmp_path / "classes")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, os.path.join(HERE, "c", "classes.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    assert out == ["ok"], out[:10]
